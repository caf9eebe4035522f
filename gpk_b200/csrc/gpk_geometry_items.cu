// gpk_geometry_items.cu — the direct Gaussian-Hessian geometry, sm_100a.
//
// Same result, bit for bit, as the direct masked tensor stencil of the
// reference (src/gpk_geometry.cpp:88-183): for every interface cell the nine
// sums Ix..Iyz run over the (2R+1)^d taps in z -> y -> x order, each tap
// adding its precomputed product (formed on the host exactly as (a*b)*c)
// when the tap's label equals the cell's label.  Here that test is one bit of
// a per-label bitmap, so every sum is the reference's sequence of correctly
// rounded additions.
//
// Zero products: the Gaussian factor w0(o) is exactly 0 for |o| in {R-1, R}
// (the Gaussian has radius R-2), so some products of those taps are +-0.
// Each sum starts at +0, and in round-to-nearest a sum that starts at +0
// never becomes -0, so adding +-0 to it is an exact no-op and such products
// are skipped.
//
// Two kernels:
//   k_geo_prepare  one CTA per tile of TX x TY x TZ cells, TX = 32 - 2R, so
//     that a halo row of the tile is exactly 32 cells: one 32-bit word per
//     halo row and label of the tile's interface cells, written to global
//     memory, and the tile's interface cells sorted by (label, octant of the
//     boundary's normal) into items of 64 cells;
//   k_geo_sum      a persistent CTA per SM holds the whole tap table in
//     shared memory and its warps take items: no barrier, every warp busy.
//     A warp skips each pair of taps that none of a slot's 32 cells matches
//     (sorted cells of one side of one boundary match much the same taps).
// The sums are bound by instruction issue (FP32) or the FP64 pipe.  One
// kernel per tile, with the table streamed plane by plane through shared
// memory and a barrier per plane, took 9.81 ms (FP32) for 256^3 cells and
// 4096 grains; it issued additions for 0.9 of the taps (0.35 match) from 3.3
// warps per scheduler.
#include <cuda_runtime.h>

#include <cub/cub.cuh>

#include <algorithm>
#include <type_traits>
#include <vector>

#include "gpk_grid.h"
#include "gpk_pool.h"

namespace gpk_dev {

// ---- conditional additions: acc_k += w_k when b != 0 ------------------------
// FP32: one predicate for a tap's additions.  FP64: acc_k = fma(w_k, m, acc_k)
// with m = 1 or 0; the product is exact, so it is the conditional addition
// bit for bit (a sum here is never -0).  A predicated FP64 addition takes 4.6
// issue cycles of a scheduler, an unpredicated FMA 2.1 (measured, 16
// independent sums per thread).
template <int N>
__device__ __forceinline__ void add_if(uint32_t b, float* const (&a)[N], const float* w) {
    static_assert(N >= 1, "");
    if constexpr (N == 1) {
        asm("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %1, 0;\n\t@p add.rn.f32 %0, %0, %2;\n\t}"
            : "+f"(*a[0]) : "r"(b), "f"(w[0]));
    } else if constexpr (N == 2) {
        asm("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %2, 0;\n\t@p add.rn.f32 %0, %0, %3;\n\t@p add.rn.f32 %1, %1, %4;\n\t}"
            : "+f"(*a[0]), "+f"(*a[1]) : "r"(b), "f"(w[0]), "f"(w[1]));
    } else if constexpr (N == 3) {
        asm("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %3, 0;\n\t"
            "@p add.rn.f32 %0, %0, %4;\n\t@p add.rn.f32 %1, %1, %5;\n\t@p add.rn.f32 %2, %2, %6;\n\t}"
            : "+f"(*a[0]), "+f"(*a[1]), "+f"(*a[2]) : "r"(b), "f"(w[0]), "f"(w[1]), "f"(w[2]));
    } else if constexpr (N == 4) {
        asm("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
            "@p add.rn.f32 %0, %0, %5;\n\t@p add.rn.f32 %1, %1, %6;\n\t@p add.rn.f32 %2, %2, %7;\n\t"
            "@p add.rn.f32 %3, %3, %8;\n\t}"
            : "+f"(*a[0]), "+f"(*a[1]), "+f"(*a[2]), "+f"(*a[3])
            : "r"(b), "f"(w[0]), "f"(w[1]), "f"(w[2]), "f"(w[3]));
    } else if constexpr (N == 5) {
        asm("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %5, 0;\n\t"
            "@p add.rn.f32 %0, %0, %6;\n\t@p add.rn.f32 %1, %1, %7;\n\t@p add.rn.f32 %2, %2, %8;\n\t"
            "@p add.rn.f32 %3, %3, %9;\n\t@p add.rn.f32 %4, %4, %10;\n\t}"
            : "+f"(*a[0]), "+f"(*a[1]), "+f"(*a[2]), "+f"(*a[3]), "+f"(*a[4])
            : "r"(b), "f"(w[0]), "f"(w[1]), "f"(w[2]), "f"(w[3]), "f"(w[4]));
    } else {
        static_assert(N == 9, "");
        asm("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %9, 0;\n\t"
            "@p add.rn.f32 %0, %0, %10;\n\t@p add.rn.f32 %1, %1, %11;\n\t@p add.rn.f32 %2, %2, %12;\n\t"
            "@p add.rn.f32 %3, %3, %13;\n\t@p add.rn.f32 %4, %4, %14;\n\t@p add.rn.f32 %5, %5, %15;\n\t"
            "@p add.rn.f32 %6, %6, %16;\n\t@p add.rn.f32 %7, %7, %17;\n\t@p add.rn.f32 %8, %8, %18;\n\t}"
            : "+f"(*a[0]), "+f"(*a[1]), "+f"(*a[2]), "+f"(*a[3]), "+f"(*a[4]), "+f"(*a[5]), "+f"(*a[6]), "+f"(*a[7]),
              "+f"(*a[8])
            : "r"(b), "f"(w[0]), "f"(w[1]), "f"(w[2]), "f"(w[3]), "f"(w[4]), "f"(w[5]), "f"(w[6]), "f"(w[7]),
              "f"(w[8]));
    }
}
template <int N>
__device__ __forceinline__ void add_if(uint32_t b, double* const (&a)[N], const double* w) {
    const double m = __hiloint2double(b ? 0x3ff00000 : 0, 0);
#pragma unroll
    for (int k = 0; k < N; ++k) *a[k] = __fma_rn(w[k], m, *a[k]);
}

// ---- the packed tap table -----------------------------------------------------
// components in the order Ix Iy Ixx Iyy Ixy Iz Izz Ixz Iyz (2-D: the first five)
enum { C_X, C_Y, C_XX, C_YY, C_XY, C_Z, C_ZZ, C_XZ, C_YZ };

// The sums a tap feeds depend on which of its Gaussian factors are zero: the
// inner taps of a row (NV sums) and the two edge taps at each end (NE sums),
// whose x factor is zero.  ZY: zero y factor (row), ZZ: zero z factor (plane).
template <bool IS3D, bool ZY, bool ZZ> struct RowComps;
#define GPK_ROW(IS3D, ZY, ZZ, NV_, NE_, ...)                      \
    template <> struct RowComps<IS3D, ZY, ZZ> {                   \
        static constexpr int NV = NV_, NE = NE_;                 \
        __host__ __device__ static constexpr int comp(int k) {   \
            constexpr int c[NV_ + NE_ + 1] = {__VA_ARGS__};      \
            return c[k];                                         \
        }                                                        \
    };
GPK_ROW(true, false, false, 9, 4, C_X, C_XX, C_XY, C_XZ, C_Y, C_YY, C_YZ, C_Z, C_ZZ, C_X, C_XX, C_XY, C_XZ, 0)
GPK_ROW(true, true, false, 4, 1, C_Y, C_YY, C_XY, C_YZ, C_XY, 0)
GPK_ROW(true, false, true, 4, 1, C_Z, C_ZZ, C_XZ, C_YZ, C_XZ, 0)
GPK_ROW(true, true, true, 1, 0, C_YZ, 0)
GPK_ROW(false, false, false, 5, 3, C_X, C_XX, C_XY, C_Y, C_YY, C_X, C_XX, C_XY, 0)
GPK_ROW(false, true, false, 3, 1, C_Y, C_YY, C_XY, C_XY, 0)
#undef GPK_ROW

__host__ __device__ constexpr int round_up(int v, int m) { return (v + m - 1) / m * m; }

// A row's table: NP pairs of inner taps of PS reals each (2 NV values), then
// the two edge taps of each end, ES reals per end (2 NE values); everything
// in whole 16-byte units.
template <typename real, int R, int NV, int NE>
struct RowLayout {
    static constexpr int W = 2 * R + 1, U = 16 / (int)sizeof(real);
    static constexpr int NIN = W - 4, NP = (NIN + 1) / 2;
    static constexpr int PS = round_up(2 * NV, U), ES = NE ? round_up(2 * NE, U) : 0;
    static constexpr int STRIDE = NP * PS + 2 * ES;
};

// The planes in order, a plane's W rows in order.  Shared memory holds the
// planes [S0, S1): all of them where they fit (FP32 to R = 9), else as many of
// the middle ones as do; the others, which feed the fewest sums and hold the
// smallest products, are read from global memory.
static constexpr int GEO_SMEM_MAX = 218 * 1024;
template <typename real, int R, bool IS3D>
struct GeoTable {
    static constexpr int W = 2 * R + 1, NPLANE = IS3D ? W : 1;
    template <bool ZY, bool ZZ> using Comps = RowComps<IS3D, ZY, ZZ>;
    template <bool ZY, bool ZZ> using Row = RowLayout<real, R, Comps<ZY, ZZ>::NV, Comps<ZY, ZZ>::NE>;
    template <bool ZZ> __host__ __device__ static constexpr int plane() {
        return (W - 4) * Row<false, ZZ>::STRIDE + 4 * Row<true, ZZ>::STRIDE;
    }
    __host__ __device__ static constexpr bool zz(int p) { return IS3D && (p <= 1 || p >= W - 2); }
    __host__ __device__ static constexpr bool zy(int r) { return r <= 1 || r >= W - 2; }
    // reals before plane p
    __host__ __device__ static constexpr int offset(int p) {
        if constexpr (IS3D)
            return (p < 2 ? p : 2) * plane<true>() + (p < 2 ? 0 : (p < W - 2 ? p - 2 : W - 4)) * plane<false>() +
                   (p < W - 2 ? 0 : p - (W - 2)) * plane<true>();
        else return p * plane<false>();
    }
    static constexpr int skip() {  // planes left out at each end
        int k = 0;
        while ((size_t)(offset(NPLANE - k) - offset(k)) * sizeof(real) > (size_t)GEO_SMEM_MAX) ++k;
        return k;
    }
    static constexpr int S0 = skip(), S1 = NPLANE - skip();
    static constexpr bool ALL = S0 == 0;
    static constexpr size_t smem() { return (size_t)(offset(S1) - offset(S0)) * sizeof(real); }
};

// host: packs the table from the per-tap products (12 per tap, see
// gpk_build_tables)
template <typename real, int R, bool IS3D>
static void pack_table(const std::vector<real>& taps, std::vector<real>& out) {
    typedef GeoTable<real, R, IS3D> T;
    constexpr int W = T::W;
    static const int slot[9] = {0, 4, 1, 5, 2, 8, 9, 3, 7};  // component -> its place among a tap's 12 products
    size_t at = 0;
    out.assign(T::offset(T::NPLANE), (real)0);
    for (int p = 0; p < T::NPLANE; ++p)
        for (int r = 0; r < W; ++r) {
            auto row = [&](auto comps, auto lay) {
                typedef decltype(comps) K;
                typedef decltype(lay) L;
                auto put = [&](size_t o, int j, int first, int n) {
                    for (int k = 0; k < n; ++k)
                        out[o + k] = taps[(((size_t)p * W + r) * W + j) * 12 + slot[K::comp(first + k)]];
                };
                for (int i = 0; i < L::NIN; ++i) put(at + (i / 2) * L::PS + (i % 2) * K::NV, 2 + i, 0, K::NV);
                for (int e = 0; e < 4; ++e)
                    put(at + L::NP * L::PS + (e / 2) * L::ES + (e % 2) * K::NE, e < 2 ? e : W - 4 + e, K::NV, K::NE);
                at += L::STRIDE;
            };
            auto kind = [&](auto zy, auto zz) {
                row(RowComps<IS3D, decltype(zy)::value, decltype(zz)::value>(),
                    typename T::template Row<decltype(zy)::value, decltype(zz)::value>());
            };
            typedef std::integral_constant<bool, true> Y;
            typedef std::integral_constant<bool, false> N;
            if constexpr (IS3D) {
                if (T::zz(p)) {
                    if (T::zy(r)) kind(Y(), Y()); else kind(N(), Y());
                    continue;
                }
            }
            if (T::zy(r)) kind(Y(), N()); else kind(N(), N());
        }
}

// ---- prepare: items and bitmaps -------------------------------------------------
template <int R, bool IS3D, int TD>
struct ItemTile {
    static constexpr int W = 2 * R + 1;
    static constexpr int TX = 32 - 2 * R;  // a halo row = 32 cells = one bitmap word
    static constexpr int TY = IS3D ? 16 : 32 / TD;
    static constexpr int TZ = IS3D ? 8 : 1;
    static constexpr int HY = TY + 2 * R, HZ = IS3D ? TZ + 2 * R : 1;
    static constexpr int NROW = HZ * HY;
    static constexpr int NROWP = NROW | 1;  // odd pitch in shared memory: one row's words hit distinct banks
    static constexpr int NCELL = TX * TY * TZ;
    static constexpr int CX = TX + 2, CY = TY + 2, CZ = IS3D ? TZ + 2 : 1;  // labels with a halo of one cell
    static constexpr int NCORE = CX * CY * CZ;
    static constexpr int NLB = 8;   // labels staged at a time
    static constexpr int HN = NCELL <= 1024 ? 2048 : (NCELL <= 2048 ? 4096 : 8192);  // label hash slots
    // one region: label hash (keys, indices), then sort bins, then staged words
    static constexpr int A1 = HN * 6, A2 = (NCELL + 8) * 4, A3 = NLB * NROWP * 4;
    static constexpr int REGION = round_up(A1 > A2 ? (A1 > A3 ? A1 : A3) : (A2 > A3 ? A2 : A3), 16);
    static constexpr size_t SMEM = REGION + (size_t)NCORE * 4 + NCELL * 4 + NCELL * 2 * 3 + (HY + HZ) * 4;
    static_assert(NCELL <= 4096 && HN >= NCELL, "tile shape");
};

struct GeoItems {
    int32_t* word;       // per item cell: index of its first bitmap word, or -1 (no bitmap: the pool was full)
    int32_t* cell;       // its flat cell index, or -1 (padding of the last item of a tile)
    uint32_t* support;   // per face 5 bits: like labels around the cell, 31 where the face has the cell's own label
    uint32_t* words;     // bitmap pool
    unsigned pool;       // words in the pool
    ItemCounters* counters;  // (the geometry's mask launch clears them)
};

struct PoolCounter {
    unsigned long long* p;
    __device__ __forceinline__ unsigned long long load() { return *(volatile unsigned long long*)p; }
    __device__ __forceinline__ unsigned long long add(unsigned v) { return atomicAdd(p, (unsigned long long)v); }
};

template <int R, bool IS3D, int TD>
__global__ void __launch_bounds__(256) k_geo_prepare(Dims D, const int32_t* __restrict__ phi,
                                                     const uint8_t* __restrict__ mask, int ntx, int nty, GeoItems it) {
    typedef ItemTile<R, IS3D, TD> S;
    extern __shared__ __align__(16) unsigned char smem[];
    int32_t* hkey = reinterpret_cast<int32_t*>(smem);
    uint16_t* hidx = reinterpret_cast<uint16_t*>(smem + S::HN * 4);
    int32_t* bins = reinterpret_cast<int32_t*>(smem);
    uint32_t* bm = reinterpret_cast<uint32_t*>(smem);
    int32_t* core = reinterpret_cast<int32_t*>(smem + S::REGION);
    int32_t* dl = core + S::NCORE;  // distinct labels of the interface cells
    int32_t* yoff = dl + S::NCELL;
    int32_t* zoff = yoff + S::HY;
    uint16_t* cells = reinterpret_cast<uint16_t*>(zoff + S::HZ);
    uint16_t* lidx = cells + S::NCELL;   // per cell: hash slot, then label index
    uint16_t* order = lidx + S::NCELL;   // sort key, then sorted position -> cell number
    __shared__ int s_count, s_nl;
    __shared__ unsigned s_item, s_word;
    __shared__ int s_ok;
    typedef cub::BlockScan<int, 256> BS;
    __shared__ typename BS::TempStorage scan;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int t = blockIdx.x;
    const int x0 = (t % ntx) * S::TX, y0 = (t / ntx) % nty * S::TY, z0 = t / (ntx * nty) * S::TZ;

    if (tid == 0) { s_count = 0; s_nl = 0; }
    for (int e = tid; e < S::HY; e += 256) yoff[e] = wrap_any(y0 - R + e, D.Ny) * D.Nx;
    for (int e = tid; e < S::HZ; e += 256) zoff[e] = IS3D ? wrap_any(z0 - R + e, D.Nz) * (D.Nx * D.Ny) : 0;
    for (int e = tid; e < S::HN; e += 256) hkey[e] = -1;
    __syncthreads();
    // 1. interface cells: a thread's flags load together, one slot request per warp
    {
        constexpr int PER = (S::NCELL + 255) / 256;
        bool f[PER];
#pragma unroll
        for (int q = 0; q < PER; ++q) {
            const int c = (q * 8 + warp) * 32 + lane;
            const int lx = c % S::TX, ly = (c / S::TX) % S::TY, lz = c / (S::TX * S::TY);
            const int x = x0 + lx, y = y0 + ly, z = z0 + lz;
            f[q] = c < S::NCELL && x < D.Nx && y < D.Ny && z < D.Nz && mask[D.idx(z, y, x)];
        }
        unsigned b[PER];
        int sum = 0;
#pragma unroll
        for (int q = 0; q < PER; ++q) {
            b[q] = __ballot_sync(0xffffffffu, f[q]);
            sum += __popc(b[q]);
        }
        int at = 0;
        if (lane == 0 && sum) at = atomicAdd(&s_count, sum);
        at = __shfl_sync(0xffffffffu, at, 0);
#pragma unroll
        for (int q = 0; q < PER; ++q) {
            if (f[q]) cells[at + __popc(b[q] & ((1u << lane) - 1u))] = (uint16_t)((q * 8 + warp) * 32 + lane);
            at += __popc(b[q]);
        }
    }
    __syncthreads();
    const int ncell = s_count;
    if (ncell == 0) return;
    // labels of the tile with a periodic halo of one cell
#pragma unroll 4
    for (int e = tid; e < S::NCORE; e += 256) {
        const int cx = e % S::CX, cy = (e / S::CX) % S::CY, cz = e / (S::CX * S::CY);
        const int xw = wrap1(x0 + cx - 1 >= D.Nx + 1 ? 0 : x0 + cx - 1, D.Nx);
        core[e] = phi[zoff[IS3D ? cz + R - 1 : 0] + yoff[cy + R - 1] + xw];
    }
    __syncthreads();
    auto core_of = [&](int c) {
        const int lx = c % S::TX, ly = (c / S::TX) % S::TY, lz = c / (S::TX * S::TY);
        return ((IS3D ? lz + 1 : 0) * S::CY + ly + 1) * S::CX + lx + 1;
    };
    // 2. distinct labels: one insertion per label and warp into a hash table
    for (int k0 = 0; k0 < ncell; k0 += 256) {
        const int k = k0 + tid;
        const bool v = k < ncell;
        const unsigned am = __ballot_sync(0xffffffffu, v);
        if (!v) continue;
        const int32_t lab = core[core_of(cells[k])];
        const unsigned grp = __match_any_sync(am, lab);
        const int lead = __ffs(grp) - 1;
        int h = 0;
        if (lane == lead) {
            h = (int)(((uint32_t)lab * 2654435761u) >> 16) & (S::HN - 1);
            for (;;) {
                const int32_t old = atomicCAS(&hkey[h], -1, lab);
                if (old == -1) {
                    const int n = atomicAdd(&s_nl, 1);
                    dl[n] = lab;
                    hidx[h] = (uint16_t)n;
                }
                if (old == -1 || old == lab) break;
                h = (h + 1) & (S::HN - 1);
            }
        }
        lidx[k] = (uint16_t)__shfl_sync(grp, h, lead);
    }
    __syncthreads();
    const int nl = s_nl;
    for (int k = tid; k < ncell; k += 256) lidx[k] = hidx[lidx[k]];
    __syncthreads();
    // 3. sort by label and, with few labels, by the octant of the direction in
    //    which the cell's own label lies (order within a bin does not matter)
    const bool oct = nl * 8 <= 256;
    const int nbin = oct ? nl * 8 : nl;
    for (int e = tid; e <= nbin; e += 256) bins[e] = 0;
    __syncthreads();
    for (int k = tid; k < ncell; k += 256) {
        int key = lidx[k];
        if (oct) {
            const int c = core_of(cells[k]);
            const int32_t own = core[c];
            int sx = 0, sy = 0, sz = 0;
#pragma unroll
            for (int dz = IS3D ? -1 : 0; dz <= (IS3D ? 1 : 0); ++dz)
#pragma unroll
                for (int dy = -1; dy <= 1; ++dy)
#pragma unroll
                    for (int dx = -1; dx <= 1; ++dx) {
                        const int m = core[c + (dz * S::CY + dy) * S::CX + dx] == own;
                        sx += m * dx;
                        sy += m * dy;
                        sz += m * dz;
                    }
            // neighbouring octants in the order share a sign of two components
            const int o = (sz > 0 ? 4 : 0) | ((sy > 0) != (sz > 0) ? 2 : 0) | ((sx > 0) != (sy > 0) ? 1 : 0);
            key = key * 8 + o;
        }
        order[k] = (uint16_t)key;
        atomicAdd(&bins[key], 1);
    }
    __syncthreads();
    {
        int carry = 0;
        for (int b0 = 0; b0 < nbin; b0 += 256) {
            const int v = b0 + tid < nbin ? bins[b0 + tid] : 0;
            int ex, total;
            BS(scan).ExclusiveSum(v, ex, total);
            __syncthreads();
            if (b0 + tid < nbin) bins[b0 + tid] = carry + ex;
            carry += total;
        }
    }
    __syncthreads();
    // place: a cell's position in its own registers, then the list
    int pos[(S::NCELL + 255) / 256];
#pragma unroll
    for (int q = 0; q < (S::NCELL + 255) / 256; ++q) {
        const int k = q * 256 + tid;
        pos[q] = k < ncell ? atomicAdd(&bins[order[k]], 1) : -1;
    }
    __syncthreads();
#pragma unroll
    for (int q = 0; q < (S::NCELL + 255) / 256; ++q)
        if (pos[q] >= 0) order[pos[q]] = (uint16_t)(q * 256 + tid);
    // 4. room for the items and the words
    const int nitem = (ncell + 63) / 64;
    if (tid == 0) {
        s_item = atomicAdd(&it.counters->items, (unsigned)nitem);
        PoolCounter taken{&it.counters->words};
        s_ok = pool_take(taken, (unsigned)nl * S::NROW, it.pool, s_word);
        if (!s_ok) atomicAdd(&it.counters->no_bitmap, 1u);
    }
    __syncthreads();
    const bool okw = s_ok != 0;
    const unsigned wbase = s_word;
    for (int q = tid; q < nitem * 64; q += 256) {
        const size_t o = (size_t)s_item * 64 + q;
        if (q >= ncell) {
            it.cell[o] = -1;
            it.word[o] = 0;
            continue;
        }
        const int k = order[q], c = cells[k];
        const int lx = c % S::TX, ly = (c / S::TX) % S::TY, lz = c / (S::TX * S::TY);
        it.cell[o] = D.idx(z0 + lz, y0 + ly, x0 + lx);
        // bitmap word of halo row (lz + dz + R, ly + dy + R): this one + (dz+R)*HY + (dy+R)
        it.word[o] = okw ? (int)(wbase + (unsigned)lidx[k] * S::NROW + (unsigned)((IS3D ? lz : 0) * S::HY + ly)) : -1;
        // support of each unlike face neighbour's label around the cell (src/gpk_geometry.cpp:154-182)
        const int cc = core_of(c);
        constexpr int NB = IS3D ? 27 : 9;
        int32_t nb[NB];
#pragma unroll
        for (int e = 0; e < NB; ++e)
            nb[e] = core[cc + ((IS3D ? e / 9 - 1 : 0) * S::CY + (e / 3) % 3 - 1) * S::CX + e % 3 - 1];
        constexpr int MID = NB / 2;
        constexpr int face[6] = {MID - 1, MID + 1, MID - 3, MID + 3, IS3D ? MID - 9 : MID, IS3D ? MID + 9 : MID};
        uint32_t sup = 0;
#pragma unroll
        for (int f = 0; f < 6; ++f) {
            uint32_t n = 0;
#pragma unroll
            for (int e = 0; e < NB; ++e) n += e != MID && nb[e] == nb[face[f]];
            sup |= (nb[face[f]] == nb[MID] ? 31u : n) << (5 * f);
        }
        it.support[o] = sup;
    }
    if (!okw) return;
    // 5. the words: a warp takes eight halo rows at a time, their labels loaded together
    const int xw = wrap_any(x0 - R + lane, D.Nx);
    for (int lb0 = 0; lb0 < nl; lb0 += S::NLB) {
        const int nb = nl - lb0 < S::NLB ? nl - lb0 : S::NLB;
        __syncthreads();  // the region is free
        for (int r0 = warp; r0 < S::NROW; r0 += 64) {
            int32_t gv[8];
#pragma unroll
            for (int u = 0; u < 8; ++u) {
                const int r = r0 + 8 * u;
                gv[u] = r < S::NROW ? phi[zoff[r / S::HY] + yoff[r % S::HY] + xw] : -1;
            }
            uint32_t mine[8] = {};
            for (int L = 0; L < nb; ++L) {
                const int32_t lab = dl[lb0 + L];
#pragma unroll
                for (int u = 0; u < 8; ++u) {
                    const uint32_t bits = __ballot_sync(0xffffffffu, gv[u] == lab);
                    if (lane == L) mine[u] = bits;
                }
            }
            if (lane < nb)
#pragma unroll
                for (int u = 0; u < 8; ++u)
                    if (r0 + 8 * u < S::NROW) bm[lane * S::NROWP + r0 + 8 * u] = mine[u];
        }
        __syncthreads();
        uint32_t* dst = it.words + wbase + (size_t)lb0 * S::NROW;
        for (int e = tid; e < nb * S::NROW; e += 256) dst[e] = bm[(e / S::NROW) * S::NROWP + e % S::NROW];
    }
}

// ---- the sums ---------------------------------------------------------------------
template <typename real, bool IS3D> constexpr int geo_warps() { return !IS3D ? 8 : (sizeof(real) == 4 ? 24 : 16); }
static constexpr int GEO_SLOTS = 2;  // cells of an item per lane

template <typename real>
struct SumArgs {
    Dims D;
    const int32_t* phi;
    GeoItems it;
    const real* table;   // packed
    int TX;
    real inv_dx, inv_dx2, dx, kappa_limit;
    real *nx, *ny, *nz, *kappa;
    int32_t* phi_comp;
};

template <typename real, int N>
__device__ __forceinline__ void load_units(const real* __restrict__ p, real (&v)[N]) {
    static_assert(N * sizeof(real) % 16 == 0, "");
    if constexpr (sizeof(real) == 4) {
#pragma unroll
        for (int k = 0; k < N; k += 4) {
            const float4 q = *reinterpret_cast<const float4*>(p + k);
            v[k] = q.x; v[k + 1] = q.y; v[k + 2] = q.z; v[k + 3] = q.w;
        }
    } else {
#pragma unroll
        for (int k = 0; k < N; k += 2) {
            const double2 q = *reinterpret_cast<const double2*>(p + k);
            v[k] = q.x; v[k + 1] = q.y;
        }
    }
}

// The nine sums as three groups (x: Ix Ixx Ixy Ixz, y: Iy Iyy Iyz, z: Iz Izz)
// that separate warps can take.  Comps of a row kind's entries
// [FIRST, FIRST + N) that belong to group GRP (GRP < 0: all).
__host__ __device__ constexpr int comp_group(int c) {
    return c == C_X || c == C_XX || c == C_XY || c == C_XZ ? 0 : (c == C_Z || c == C_ZZ ? 2 : 1);
}
template <typename K, int GRP, int FIRST, int N>
struct Pick {
    __host__ __device__ static constexpr int count() {
        int n = 0;
        for (int k = 0; k < N; ++k) n += GRP < 0 || comp_group(K::comp(FIRST + k)) == GRP;
        return n;
    }
    __host__ __device__ static constexpr int at(int i) {  // the i-th one's place among the N
        int n = 0;
        for (int k = 0; k < N; ++k)
            if (GRP < 0 || comp_group(K::comp(FIRST + k)) == GRP)
                if (n++ == i) return k;
        return 0;
    }
    static constexpr int C = count();
};

// the additions of one tap; w: its N values
template <typename real, typename K, int GRP, int FIRST, int N>
__device__ __forceinline__ void tap_adds(uint32_t b, real (&acc)[9], const real* w) {
    typedef Pick<K, GRP, FIRST, N> P;
    if constexpr (P::C > 0) {
        real* a[P::C];
        real v[P::C];
#pragma unroll
        for (int k = 0; k < P::C; ++k) {
            a[k] = &acc[K::comp(FIRST + P::at(k))];
            v[k] = w[P::at(k)];
        }
        add_if<P::C>(b, a, v);
    }
}

// One row of taps (fixed dz, dy): w[s] holds bit j set when tap x-offset j - R
// of slot s matches, u[s] the OR of w[s] over the warp.
template <typename real, int R, bool IS3D, bool ZY, bool ZZ, int GRP, int SL>
__device__ __forceinline__ void sum_row(const real* __restrict__ row, const uint32_t (&w)[SL],
                                        const uint32_t (&u)[SL], real (&acc)[SL][9]) {
    typedef RowComps<IS3D, ZY, ZZ> K;
    typedef RowLayout<real, R, K::NV, K::NE> L;
    constexpr int W = 2 * R + 1;
    uint32_t both = 0;
#pragma unroll
    for (int s = 0; s < SL; ++s) both |= u[s];
    auto edge = [&](int j0, const real* p) {
        if constexpr (Pick<K, GRP, K::NV, K::NE>::C > 0) {
            if ((both & (3u << j0)) == 0u) return;
            real v[L::ES];
            load_units<real, L::ES>(p, v);
#pragma unroll
            for (int s = 0; s < SL; ++s) {
                tap_adds<real, K, GRP, K::NV, K::NE>(w[s] & (1u << j0), acc[s], v);
                tap_adds<real, K, GRP, K::NV, K::NE>(w[s] & (2u << j0), acc[s], v + K::NE);
            }
        }
    };
    edge(0, row + L::NP * L::PS);
    if constexpr (Pick<K, GRP, 0, K::NV>::C > 0) {
        // pairs per chunk: one where a tap feeds nine (2-D: five) sums
        constexpr int PC = K::NV > 4 ? 1 : 2;
#pragma unroll
        for (int q0 = 0; q0 < L::NP; q0 += PC) {
            const int q1 = q0 + PC < L::NP ? q0 + PC : L::NP;
            const int nt = 2 * q1 < L::NIN ? 2 * (q1 - q0) : L::NIN - 2 * q0;
            const uint32_t m = ((1u << nt) - 1u) << (2 + 2 * q0);
            if ((both & m) == 0u) continue;
            real v[PC][L::PS];
            if (GRP < 0) {
#pragma unroll
                for (int q = q0; q < q1; ++q) load_units<real, L::PS>(row + q * L::PS, v[q - q0]);
            } else {
#pragma unroll
                for (int q = q0; q < q1; ++q)
#pragma unroll
                    for (int k = 0; k < 2 * K::NV; ++k)
                        if (comp_group(K::comp(k % K::NV)) == GRP) v[q - q0][k] = row[q * L::PS + k];
            }
#pragma unroll
            for (int s = 0; s < SL; ++s) {
                if (SL > 1 && K::NV > 4 && (u[s] & m) == 0u) continue;
#pragma unroll
                for (int q = q0; q < q1; ++q) {
                    tap_adds<real, K, GRP, 0, K::NV>(w[s] & (1u << (2 + 2 * q)), acc[s], v[q - q0]);
                    if (2 * q + 1 < L::NIN)
                        tap_adds<real, K, GRP, 0, K::NV>(w[s] & (2u << (2 + 2 * q)), acc[s], v[q - q0] + K::NV);
                }
            }
        }
    }
    edge(W - 2, row + L::NP * L::PS + L::ES);
}

template <typename real, int R, bool IS3D, int HY, int GRP, int SL>
__device__ __forceinline__ void sum_item(const SumArgs<real>& a, const real* __restrict__ tab,
                                         const int (&word)[SL], const int (&cell)[SL],
                                         const int (&lx)[SL], bool slow, real (&acc)[SL][9]) {
    typedef GeoTable<real, R, IS3D> T;
    constexpr int W = 2 * R + 1;
#pragma unroll
    for (int s = 0; s < SL; ++s)
#pragma unroll
        for (int k = 0; k < 9; ++k) acc[s][k] = (real)0;
    // the next row's words load while a row is summed
    uint32_t next[SL];
    auto fetch = [&](int p, int dy) {
#pragma unroll
        for (int s = 0; s < SL; ++s) {
            if (!slow) {
                next[s] = __ldg(a.it.words + ((unsigned)word[s] + (unsigned)(p * HY + dy)));
                continue;
            }
            // no bitmap: the row's labels compared one by one
            uint32_t b = 0;
            if (cell[s] >= 0) {
                int z, y, x;
                a.D.decode(cell[s], z, y, x);
                const int32_t own = a.phi[cell[s]];
                const int zz = IS3D ? wrap_any(z + p - R, a.D.Nz) : 0, yy = wrap_any(y + dy - R, a.D.Ny);
                const int32_t* row = a.phi + (size_t)(zz * a.D.Ny + yy) * a.D.Nx;
                for (int j = 0; j < W; ++j) b |= (uint32_t)(row[wrap_any(x + j - R, a.D.Nx)] == own) << j;
            }
            next[s] = b << lx[s];
        }
    };
    constexpr uint32_t WM = (1u << W) - 1u;
    fetch(0, 0);
    // rows of planes in shared memory, and of the others (two pointers, so that
    // each load's address space is known to the compiler)
    const real* srow = tab;
    const real* grow = a.table;
    for (int p = 0; p < T::NPLANE; ++p) {
        const bool zz = T::zz(p), in = T::ALL || (p >= T::S0 && p < T::S1);
        if (!T::ALL && p == T::S1) grow = a.table + T::offset(T::S1);
#pragma unroll 1
        for (int dy = 0; dy < W; ++dy) {
            uint32_t w[SL], u[SL], any = 0;
#pragma unroll
            for (int s = 0; s < SL; ++s) {
                w[s] = cell[s] >= 0 ? (next[s] >> lx[s]) & WM : 0u;
                u[s] = __reduce_or_sync(0xffffffffu, w[s]);
                any |= u[s];
            }
            const bool wrap = dy + 1 == W;
            if (!(wrap && p + 1 == T::NPLANE)) fetch(wrap ? p + 1 : p, wrap ? 0 : dy + 1);
            const bool zy = T::zy(dy);
            auto take = [&](auto zyc, auto zzc) {
                constexpr bool ZY = decltype(zyc)::value, ZZ = decltype(zzc)::value;
                constexpr int stride = T::template Row<ZY, ZZ>::STRIDE;
                // at radius 8 and below every plane with a nonzero z factor is in shared memory
                constexpr bool MAYBE_G = !T::ALL && (ZZ || T::S0 > 2), MAYBE_S = T::ALL || !ZZ || T::S0 < 2;
                if (MAYBE_S && (in || !MAYBE_G)) {
                    if (any) sum_row<real, R, IS3D, ZY, ZZ, GRP>(srow, w, u, acc);
                    srow += stride;
                } else if constexpr (MAYBE_G) {
                    if (any) sum_row<real, R, IS3D, ZY, ZZ, GRP>(grow, w, u, acc);
                    grow += stride;
                }
            };
            typedef std::integral_constant<bool, true> Y;
            typedef std::integral_constant<bool, false> N;
            if (IS3D && zz) {
                if constexpr (IS3D) {
                    if (zy) take(Y(), Y());
                    else take(N(), Y());
                }
            } else if (zy) take(Y(), N());
            else take(N(), N());
        }
    }
}

// normals, curvature (src/gpk_geometry.cpp:135-152) and the competitor's choice (:154-182) of a cell;
// sum[] in component order
template <typename real>
__device__ __forceinline__ void finish_cell(const SumArgs<real>& a, int i, const real (&sum)[9], uint32_t support) {
    const real Ix = sum[C_X] * a.inv_dx, Iy = sum[C_Y] * a.inv_dx, Iz = sum[C_Z] * a.inv_dx;
    const real Ixx = sum[C_XX] * a.inv_dx2, Iyy = sum[C_YY] * a.inv_dx2, Izz = sum[C_ZZ] * a.inv_dx2;
    const real Ixy = sum[C_XY] * a.inv_dx2, Ixz = sum[C_XZ] * a.inv_dx2, Iyz = sum[C_YZ] * a.inv_dx2;
    const real dx = a.dx;
    const real grad_sq = Ix * Ix + Iy * Iy + Iz * Iz;
    real nxv = 0, nyv = 0, nzv = 0;
    if (grad_sq * dx * dx > (real)1e-8) {
        const real grad = sqrt(grad_sq);
        nxv = -Ix / grad;
        nyv = -Iy / grad;
        nzv = -Iz / grad;
        const real trace_H = Ixx + Iyy + Izz;
        const real gHg = Ix * Ix * Ixx + Iy * Iy * Iyy + Iz * Iz * Izz + (real)2 * (Ix * Iy * Ixy + Ix * Iz * Ixz + Iy * Iz * Iyz);
        real curvature = (gHg - grad_sq * trace_H) / (grad_sq * grad);
        if (fabs(curvature * dx) < (real)1e-6) curvature = (real)0;
        a.nx[i] = nxv; a.ny[i] = nyv; a.nz[i] = nzv;
        a.kappa[i] = dclamp(curvature, -a.kappa_limit, a.kappa_limit);
    }
    const real score[6] = {-nxv, nxv, -nyv, nyv, -nzv, nzv};
    int best = -1, best_support = -1;
    real best_score = (real)-2;
#pragma unroll
    for (int k = 0; k < 6; ++k) {
        const int s = (int)((support >> (5 * k)) & 31u);
        if (s == 31) continue;
        if (s > best_support || (s == best_support && score[k] > best_score)) {
            best = k; best_support = s; best_score = score[k];
        }
    }
    int src = i;
    if (best >= 0) {
        int nb[6];
        a.D.faces(i, nb);
#pragma unroll
        for (int k = 0; k < 6; ++k) src = best == k ? nb[k] : src;
    }
    a.phi_comp[i] = a.phi[src];
}

// copies a table into shared memory (all threads)
__device__ __forceinline__ void copy_table(void* dst, const void* src, int bytes) {
    const uint4* s = reinterpret_cast<const uint4*>(src);
    uint4* d = reinterpret_cast<uint4*>(dst);
    for (int k = threadIdx.x; k < bytes / 16; k += blockDim.x) d[k] = __ldg(s + k);
}

template <typename real>
__device__ __forceinline__ void load_slot(const SumArgs<real>& a, size_t o, int& cell, int& word, int& lx) {
    cell = a.it.cell[o];
    word = a.it.word[o];
    lx = cell < 0 ? 0 : (cell % a.D.Nx) % a.TX;
}

// Few items: half an item per three warps, each with one group of the sums.
// A lone warp with all nine sums of 64 cells takes 265 us (FP64, R = 8)
// because nothing hides its latencies, and so small a count leaves the SMs'
// other warps free: 151 us for the 10^4 interface cells of a solid sphere.
template <typename real, int R, bool IS3D, int HY>
__device__ __forceinline__ void sum_thin(const SumArgs<real>& a, real* tab, int n) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, G = gridDim.x;
    constexpr int NT = geo_warps<real, IS3D>() / 3;
    const int h = (warp / 3) * G + blockIdx.x, grp = warp % 3;
    const bool mine = warp < 3 * NT && h < 2 * n;
    int cell[1] = {-1}, word[1], lx[1];
    real acc[1][9];
    if (mine) {
        load_slot(a, (size_t)h * 32 + lane, cell[0], word[0], lx[0]);
        const bool slow = __any_sync(0xffffffffu, word[0] < 0) != 0;
        if (grp == 0) sum_item<real, R, IS3D, HY, 0>(a, tab, word, cell, lx, slow, acc);
        else if (grp == 1) sum_item<real, R, IS3D, HY, 1>(a, tab, word, cell, lx, slow, acc);
        else sum_item<real, R, IS3D, HY, 2>(a, tab, word, cell, lx, slow, acc);
    }
    __syncthreads();  // the table has been read: its memory takes the sums
    real* mysum = tab + (size_t)(warp / 3) * 9 * 32 + lane;
    if (mine) {
#pragma unroll
        for (int k = 0; k < 9; ++k)
            if (comp_group(k) == grp) mysum[k * 32] = acc[0][k];
    }
    __syncthreads();
    if (mine && grp == 0 && cell[0] >= 0) {
        real sum[9];
#pragma unroll
        for (int k = 0; k < 9; ++k) sum[k] = mysum[k * 32];
        finish_cell<real>(a, cell[0], sum, a.it.support[(size_t)h * 32 + lane]);
    }
}

// At most one half item per warp: twice the warps of whole items.
template <typename real, int R, bool IS3D, int HY>
__device__ __forceinline__ void sum_half(const SumArgs<real>& a, real* tab, int n) {
    const int lane = threadIdx.x & 31, h = (threadIdx.x >> 5) * gridDim.x + blockIdx.x;
    if (h >= 2 * n) return;
    int cell[1], word[1], lx[1];
    load_slot(a, (size_t)h * 32 + lane, cell[0], word[0], lx[0]);
    const bool slow = __any_sync(0xffffffffu, word[0] < 0) != 0;
    real acc[1][9];
    sum_item<real, R, IS3D, HY, -1>(a, tab, word, cell, lx, slow, acc);
    if (cell[0] >= 0) finish_cell<real>(a, cell[0], acc[0], a.it.support[(size_t)h * 32 + lane]);
}

// (out of line: inlined, their registers spill in the main loop's FP32 form)
template <typename real, int R, bool IS3D, int HY>
__device__ __noinline__ void sum_few(const SumArgs<real>& a, real* tab, int n) {
    if (IS3D && 2 * n <= geo_warps<real, IS3D>() / 3 * (int)gridDim.x) sum_thin<real, R, IS3D, HY>(a, tab, n);
    else sum_half<real, R, IS3D, HY>(a, tab, n);
}

template <typename real, int R, bool IS3D, int HY>
__global__ void __launch_bounds__(geo_warps<real, IS3D>() * 32, IS3D ? 1 : 3) k_geo_sum(const __grid_constant__ SumArgs<real> a) {
    extern __shared__ __align__(16) unsigned char smem[];
    typedef GeoTable<real, R, IS3D> T;
    real* tab = reinterpret_cast<real*>(smem);
    const int n = (int)a.it.counters->items;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, G = gridDim.x;
    if ((int)blockIdx.x >= 2 * n) return;  // (a CTA may take half an item)
    copy_table(tab, a.table + T::offset(T::S0), (int)T::smem());
    __syncthreads();
    constexpr int SL = GEO_SLOTS, NW = geo_warps<real, IS3D>();
    if (2 * n <= NW * G) {
        sum_few<real, R, IS3D, HY>(a, tab, n);
        return;
    }
    // the first items go round the CTAs, the rest as warps come free
    for (int item = warp * G + blockIdx.x; item < n;) {
        int cell[SL], word[SL], lx[SL];
        bool slow = false;
#pragma unroll
        for (int s = 0; s < SL; ++s) {
            load_slot(a, (size_t)item * 64 + 32 * s + lane, cell[s], word[s], lx[s]);
            slow |= word[s] < 0;
        }
        slow = __any_sync(0xffffffffu, slow) != 0;
        real acc[SL][9];
        sum_item<real, R, IS3D, HY, -1>(a, tab, word, cell, lx, slow, acc);
#pragma unroll
        for (int s = 0; s < SL; ++s)
            if (cell[s] >= 0)
                finish_cell<real>(a, cell[s], acc[s], a.it.support[(size_t)item * 64 + 32 * s + lane]);
        int nx = 0;
        if (lane == 0) nx = (int)atomicAdd(&a.it.counters->next, 1u) + G * NW;
        item = __shfl_sync(0xffffffffu, nx, 0);
    }
}

template <typename real, int R, bool IS3D, int TD>
static int launch_items(gpk_grid* G, const SumArgs<real>& a0) {
    typedef ItemTile<R, IS3D, TD> S;
    SumArgs<real> a = a0;
    const int ntx = (G->d.Nx + S::TX - 1) / S::TX, nty = (G->d.Ny + S::TY - 1) / S::TY,
              ntz = (G->d.Nz + S::TZ - 1) / S::TZ;
    a.TX = S::TX;
    a.table = (const real*)G->d_geom_packed;
    constexpr size_t smem = GeoTable<real, R, IS3D>::smem();
    // set once per process (thread-safe initialisation of a function-local static)
    static const cudaError_t rc1 = cudaFuncSetAttribute(k_geo_prepare<R, IS3D, TD>,
                                                        cudaFuncAttributeMaxDynamicSharedMemorySize, (int)S::SMEM);
    static const cudaError_t rc2 = cudaFuncSetAttribute(k_geo_sum<real, R, IS3D, S::HY>,
                                                        cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    GPK_CUDA_TRY(rc1);
    GPK_CUDA_TRY(rc2);
    const int ntiles = ntx * nty * ntz;
    k_geo_prepare<R, IS3D, TD><<<ntiles, 256, S::SMEM, G->stream>>>(G->d, G->phi, G->mask, ntx, nty, a.it);
    // the CTAs that are resident together, and no more than the largest number of items
    const long long most = ((long long)G->d.N + 63) / 64 + ntiles;
    const int grid = (int)std::min<long long>(IS3D ? G->num_sms : 3 * G->num_sms, most);
    k_geo_sum<real, R, IS3D, S::HY><<<grid, geo_warps<real, IS3D>() * 32, smem, G->stream>>>(a);
    G->launches += 2;
    GPK_CUDA_TRY(cudaGetLastError());
    return GPK_OK;
}

}  // namespace gpk_dev

using namespace gpk_dev;

// calls f(std::integral_constant<int, R>) for the kernel radii 4..10; false for others
template <typename F>
static bool for_radius(int R, F f) {
    switch (R) {
    case 4: f(std::integral_constant<int, 4>()); return true;
    case 5: f(std::integral_constant<int, 5>()); return true;
    case 6: f(std::integral_constant<int, 6>()); return true;
    case 7: f(std::integral_constant<int, 7>()); return true;
    case 8: f(std::integral_constant<int, 8>()); return true;
    case 9: f(std::integral_constant<int, 9>()); return true;
    case 10: f(std::integral_constant<int, 10>()); return true;
    default: return false;
    }
}

// item slots of a grid: its cells, and for every tile the padding of its last item
static size_t item_slots(const Dims& D, int R) {
    long long ntiles = 0;
    for_radius(R, [&](auto r) {
        constexpr int RR = decltype(r)::value;
        auto tiles = [&](int tx, int ty, int tz) {
            ntiles = (long long)((D.Nx + tx - 1) / tx) * ((D.Ny + ty - 1) / ty) * ((D.Nz + tz - 1) / tz);
        };
        // (the lowest 2-D tile: the most tiles)
        if (D.is3d()) tiles(ItemTile<RR, true, 1>::TX, ItemTile<RR, true, 1>::TY, ItemTile<RR, true, 1>::TZ);
        else tiles(ItemTile<RR, false, 4>::TX, ItemTile<RR, false, 4>::TY, 1);
    });
    return ((size_t)D.N + 64 * (size_t)ntiles + 3) & ~(size_t)3;
}

// Scratch that a grid's items and bitmaps need at the least (the padding of an
// item reads the pool's first words)
size_t gpk_geometry_items_scratch(const gpk_grid* G, int R) { return 12 * item_slots(G->d, R) + 4 * 4096; }

// The packed tap table and the counters of a grid (kernel radii 4..10), and
// where in its scratch the items and the bitmap pool lie: made with the grid,
// so that no step allocates.  The scratch holds the crossing and remap records,
// which nothing reads while the geometry runs.  (As an allocation of their own,
// 28 bytes a cell and more, the items cost a grid's first step 1 to 120 ms,
// and the 48 instances of a sweep 20 to 700.)
template <typename real>
int gpk_geometry_items_init(gpk_grid* G) {
    const HostKernels<real>* hk = (const HostKernels<real>*)G->host_kernels;
    const std::vector<real>& taps = hk->geom_table;
    std::vector<real> packed;
    const Dims D = G->d;
    if (!for_radius(hk->geom_radius, [&](auto r) {
            constexpr int RR = decltype(r)::value;
            if (D.is3d()) pack_table<real, RR, true>(taps, packed);
            else pack_table<real, RR, false>(taps, packed);
        }))
        return GPK_OK;
    const size_t slots = item_slots(D, hk->geom_radius);
    const size_t table = sizeof(real) * packed.size();
    unsigned char* base = nullptr;
    constexpr size_t head = sizeof(ItemCounters);
    static_assert(head % 16 == 0, "the table is copied in 16-byte units");
    GPK_TRY(gpk_alloc(G, (void**)&base, head + table));
    GPK_CUDA_TRY(cudaMemset(base, 0, head));
    GPK_CUDA_TRY(cudaMemcpy(base + head, packed.data(), table, cudaMemcpyHostToDevice));
    G->d_geom_packed = base + head;
    G->item_word = (int32_t*)G->scratch;
    G->item_cell = G->item_word + slots;
    G->item_support = (uint32_t*)(G->item_cell + slots);
    G->item_words = G->item_support + slots;
    // words: what is left, 25 a cell (FP64: 29): 66 labels in every tile at R = 8,
    // 50 at R = 9 and 38 at R = 10 (0.38, 0.49 and 0.66 words a cell and label;
    // tiles of a polycrystal with grains of 1500 cells meet 9 to 11 on average).
    // Tiles that find the pool full compare labels instead, and are counted
    const size_t words = (G->scratch_bytes - 12 * slots) / 4;
    G->item_pool = (unsigned)std::min(words, (size_t)1 << 31);
    G->item_counters = (ItemCounters*)base;
    return GPK_OK;
}
template int gpk_geometry_items_init<float>(gpk_grid*);
template int gpk_geometry_items_init<double>(gpk_grid*);

// The direct geometry for kernel radii 4..10 (Gaussian radius 2..8); returns
// -1 for other radii (the caller then uses the per-cell kernel).
template <typename real>
int gpk_geometry_items(gpk_grid* G, int R, real inv_dx, real inv_dx2, real dx, real kappa_limit) {
    if (!G->item_counters) return -1;
    SumArgs<real> a{};
    a.D = G->d;
    a.phi = G->phi;
    // kind 2 gives no tile a bitmap: every row is compared label by label
    a.it = GeoItems{G->item_word, G->item_cell, G->item_support, G->item_words,
                    G->geometry_kernel == 2 ? 0u : G->item_pool, G->item_counters};
    a.inv_dx = inv_dx; a.inv_dx2 = inv_dx2; a.dx = dx; a.kappa_limit = kappa_limit;
    a.nx = (real*)G->f[GPK_FIELD_NX]; a.ny = (real*)G->f[GPK_FIELD_NY]; a.nz = (real*)G->f[GPK_FIELD_NZ];
    a.kappa = (real*)G->f[GPK_FIELD_KAPPA];
    a.phi_comp = G->phi_comp;
    int rc = -1;
    for_radius(R, [&](auto r) {
        constexpr int RR = decltype(r)::value;
        if (G->d.is3d()) rc = launch_items<real, RR, true, 1>(G, a);
        else if (RR == 8 && G->tile_rows_div == 4) rc = launch_items<real, RR, false, RR == 8 ? 4 : 1>(G, a);
        else if (RR == 8 && G->tile_rows_div == 2) rc = launch_items<real, RR, false, RR == 8 ? 2 : 1>(G, a);
        else rc = launch_items<real, RR, false, 1>(G, a);
    });
    return rc;
}
template int gpk_geometry_items<float>(gpk_grid*, int, float, float, float, float);
template int gpk_geometry_items<double>(gpk_grid*, int, double, double, double, double);
