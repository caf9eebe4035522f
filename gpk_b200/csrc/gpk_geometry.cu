// gpk_geometry.cu — separable tiles: the FP64 throughput geometry, sm_100a.
#include <cuda_runtime.h>

#include <cub/cub.cuh>

#include "gpk_grid.h"

namespace gpk_dev {

// Tile of TX x TY x TZ cells with TX = 32 - 2R, so that a halo row is exactly
// 32 cells and, for one label, one 32-bit word.
template <int R, bool IS3D>
struct GeoShape {
    static constexpr int TX = 32 - 2 * R;
    static constexpr int TY = IS3D ? 8 : 1024 / TX;
    static constexpr int TZ = IS3D ? 1024 / (TX * 8) : 1;
    static constexpr int HY = TY + 2 * R, HZ = IS3D ? TZ + 2 * R : 1;
    static constexpr int NROW = HZ * HY;
    static constexpr int NROWP = NROW | 1;  // odd pitch: one row's words for several labels hit distinct banks
    static constexpr int NCELL = TX * TY * TZ;
    static constexpr int CX = TX + 2, CY = TY + 2, CZ = IS3D ? TZ + 2 : 1;  // tile labels with a 1-cell halo
    static constexpr int NCORE = CX * CY * CZ;
    static_assert(NCELL <= 1024, "tile shape");
};

// competitor choice (src/gpk_geometry.cpp:154-182) from the staged labels
template <typename real>
__device__ __forceinline__ void geo_competitor(int32_t* __restrict__ phi_comp, int i, real nxv, real nyv, real nzv,
                                               const int32_t* __restrict__ lab, int cbase, int pitch, int rows,
                                               bool is3d) {
    const int32_t pi = lab[cbase];
    const int plane = rows * pitch;
    const int fo[6] = {-1, +1, -pitch, +pitch, -plane, +plane};
    const real score[6] = {-nxv, nxv, -nyv, nyv, -nzv, nzv};
    const int nf = is3d ? 6 : 4;
    int best = -1, best_support = -1;
    real best_score = (real)-2;
    for (int k = 0; k < nf; ++k) {
        const int32_t q = lab[cbase + fo[k]];
        if (q == pi) continue;
        int support = 0;
        for (int dz = (is3d ? -1 : 0); dz <= (is3d ? 1 : 0); ++dz)
            for (int dy = -1; dy <= 1; ++dy)
                for (int dxs = -1; dxs <= 1; ++dxs) {
                    if (!dxs && !dy && !dz) continue;
                    support += lab[cbase + dz * plane + dy * pitch + dxs] == q;
                }
        if (support > best_support || (support == best_support && score[k] > best_score)) {
            best = k; best_support = support; best_score = score[k];
        }
    }
    phi_comp[i] = (best >= 0) ? lab[cbase + fo[best]] : pi;
}

// ---------------------------------------------------------------------------
// Separable tiles (FP64 throughput mode)
// ---------------------------------------------------------------------------
// The reference's separable geometry (src/gpk_geometry.cpp:185-347: Gaussian
// smoothing of one label's indicator, then fourth-order differences at that
// label's interface cells) evaluated per tile instead of per label over the
// whole grid.  The direct stencil's tap products are exactly these filters
// composed (w1 = d1 * G, w2 = d2 * G), so both give the same fields up to
// rounding; in FP64 the two agree far below 1e-10.  Per tile and label:
//   x: a 2K+1-tap window of a halo row is 2K+1 bits of its bitmap word; its
//      smoothed value is two or three table lookups (7-bit chunks);
//   y: each thread owns a column (x, y) of the smoothed region and sums the
//      2K+1 x-values above and below it for every halo plane, in registers;
//   z: the same column's planes give the smoothed indicator S on the tile
//      plus two cells each side, stored in shared memory;
//   then the differences at the label's interface cells.
struct SepArgs {
    Dims D;
    const int32_t* phi;
    const uint8_t* mask;
    int ntx, nty;
    double g[17];  // Gaussian taps (radius K = R - 2 <= 8)
    double dx, idx12, idx12_sq, idx144_sq, kappa_limit;
    double *nx, *ny, *nz, *kappa;
    int32_t* phi_comp;
};

template <int R, bool IS3D>
struct SepShape {
    typedef GeoShape<R, IS3D> G;
    static constexpr int K = R - 2, NT = 2 * K + 1, NCH = (NT + 6) / 7;
    static constexpr int SX = G::TX + 4, SY = G::TY + 4, SZ = IS3D ? G::TZ + 4 : 1;
    static constexpr int NS = SX * SY * SZ;
    static constexpr int NY = IS3D ? SX * SY * G::HZ : 0;  // y-smoothed values of every halo plane
    static constexpr int NLB = 4;                            // labels per bitmap batch
    // the bitmaps' words first hold up to one label candidate per interface cell
    static constexpr int BM_WORDS = NLB * G::NROWP > G::NCELL ? NLB * G::NROWP : G::NCELL;
};

template <int R, bool IS3D>
constexpr size_t sep_smem_bytes() {
    typedef GeoShape<R, IS3D> S;
    typedef SepShape<R, IS3D> P;
    // smoothed indicator | y-smoothed planes | chunk tables | bitmaps | core labels | distinct labels |
    // cells | cell label index
    return (size_t)(P::NS + P::NY) * 8 + (size_t)P::NCH * 128 * 8 + (size_t)P::BM_WORDS * 4 +
           (size_t)S::NCORE * 4 + (size_t)S::NCELL * 4 + (size_t)S::NCELL * 2 * 2;
}

template <int R, bool IS3D>
__global__ void __launch_bounds__(256) k_geometry_sep_tiles(SepArgs a) {
    typedef GeoShape<R, IS3D> S;
    typedef SepShape<R, IS3D> P;
    extern __shared__ __align__(128) unsigned char smem[];
    double* Sm = reinterpret_cast<double*>(smem);  // P::NS
    double* Ym = Sm + P::NS;                        // P::NY
    double* lut = Ym + P::NY;                       // P::NCH x 128
    uint32_t* bm = reinterpret_cast<uint32_t*>(lut + P::NCH * 128);
    int32_t* core = reinterpret_cast<int32_t*>(bm + P::BM_WORDS);
    int32_t* dl = core + S::NCORE;
    int16_t* cells = reinterpret_cast<int16_t*>(dl + S::NCELL);
    uint16_t* cli = reinterpret_cast<uint16_t*>(cells + S::NCELL);
    int32_t* cand = reinterpret_cast<int32_t*>(bm);  // label candidates, before the first bitmap
    __shared__ int s_count, s_ncand, s_nl;
    __shared__ int sbox[6 * P::NLB];  // per label of the batch: min x, y, z, max x, y, z of its cells
    typedef cub::BlockScan<int, 256> BS;
    __shared__ typename BS::TempStorage scan;
    constexpr int PER = (S::NCELL + 255) / 256;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const Dims D = a.D;
    const int t = blockIdx.x;
    const int tx = t % a.ntx, ty = (t / a.ntx) % a.nty, tz = t / (a.ntx * a.nty);
    const int x0 = tx * S::TX, y0 = ty * S::TY, z0 = tz * S::TZ;

    // interface cells of the tile, in flat order
    {
        int flags[PER];
        int cnt = 0;
#pragma unroll
        for (int k = 0; k < PER; ++k) {
            const int c = tid * PER + k;
            int f = 0;
            if (c < S::NCELL) {
                const int lx = c % S::TX, ly = (c / S::TX) % S::TY, lz = c / (S::TX * S::TY);
                const int x = x0 + lx, y = y0 + ly, z = z0 + lz;
                if (x < D.Nx && y < D.Ny && z < D.Nz) f = a.mask[D.idx(z, y, x)];
            }
            flags[k] = f;
            cnt += f;
        }
        int ex, total;
        BS(scan).ExclusiveSum(cnt, ex, total);
#pragma unroll
        for (int k = 0; k < PER; ++k)
            if (flags[k]) cells[ex++] = (int16_t)(tid * PER + k);
        if (tid == 0) { s_count = total; s_ncand = 0; s_nl = 0; }
    }
    __syncthreads();
    const int ncell = s_count;
    if (ncell == 0) return;
    // tile labels with a one-cell periodic halo (competitor choice); chunk tables
    for (int e = tid; e < S::NCORE; e += 256) {
        const int cx = e % S::CX, cy = (e / S::CX) % S::CY, cz = e / (S::CX * S::CY);
        const int x = wrap_any(x0 + cx - 1, D.Nx), y = wrap_any(y0 + cy - 1, D.Ny);
        const int z = IS3D ? wrap_any(z0 + cz - 1, D.Nz) : 0;
        core[e] = a.phi[D.idx(z, y, x)];
    }
    for (int e = tid; e < P::NCH * 128; e += 256) {
        const int ch = e >> 7, pat = e & 127;
        double v = 0.0;
        for (int j = 0; j < 7; ++j)
            if ((pat >> j) & 1) {
                const int tap = 7 * ch + j;
                if (tap < P::NT) v += a.g[tap];
            }
        lut[e] = v;
    }
    __syncthreads();
    // distinct labels of the interface cells
    auto core_of = [&](int c) {
        const int lx = c % S::TX, ly = (c / S::TX) % S::TY, lz = c / (S::TX * S::TY);
        return ((IS3D ? lz + 1 : 0) * S::CY + ly + 1) * S::CX + lx + 1;
    };
    for (int k0 = 0; k0 < ncell; k0 += 256) {
        const int k = k0 + tid;
        const bool v = k < ncell;
        const unsigned am = __ballot_sync(0xffffffffu, v);
        if (v) {
            const int32_t lab = core[core_of(cells[k])];
            const unsigned grp = __match_any_sync(am, lab);
            if (lane == __ffs(grp) - 1) cand[atomicAdd(&s_ncand, 1)] = lab;
        }
    }
    __syncthreads();
    const int ncand = s_ncand;
    for (int e = tid; e < ncand; e += 256) {
        const int32_t lab = cand[e];
        bool first = true;
        for (int j = 0; j < e && first; ++j) first = cand[j] != lab;
        if (first) dl[atomicAdd(&s_nl, 1)] = lab;
    }
    __syncthreads();
    const int nl = s_nl;
    for (int k = tid; k < ncell; k += 256) {
        const int32_t lab = core[core_of(cells[k])];
        int li = 0;
        while (li < nl - 1 && dl[li] != lab) ++li;
        cli[k] = (uint16_t)li;
    }
    const double dx = a.dx;
    for (int lb0 = 0; lb0 < nl; lb0 += P::NLB) {
        const int nb = nl - lb0 < P::NLB ? nl - lb0 : P::NLB;
        __syncthreads();  // the previous batch's bitmaps and smoothed values are free
        // a warp takes four halo rows at a time, their label loads issued together
        const int xw = wrap_any(x0 - R + lane, D.Nx);
        for (int r0 = warp; r0 < S::NROW; r0 += 32) {
            int32_t gv[4];
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                const int r = r0 + 8 * u;
                const int hz = r / S::HY, hy = r % S::HY;
                const int y = wrap_any(y0 + hy - R, D.Ny);
                const int z = IS3D ? wrap_any(z0 + hz - R, D.Nz) : 0;
                gv[u] = r < S::NROW ? a.phi[D.idx(z, y, xw)] : -1;
            }
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                const int r = r0 + 8 * u;
                if (r >= S::NROW) break;
                for (int L = 0; L < nb; ++L) {
                    const uint32_t bits = __ballot_sync(0xffffffffu, gv[u] == dl[lb0 + L]);
                    if (lane == 0) bm[L * S::NROWP + r] = bits;
                }
            }
        }
        // each label's interface cells span a box of the tile; its smoothed
        // values are needed there plus two cells each side (the differences)
        if (tid < 6 * P::NLB) sbox[tid] = (tid % 6) < 3 ? 1 << 20 : -1;
        __syncthreads();
        for (int k = tid; k < ncell; k += 256) {
            const int L = (int)cli[k] - lb0;
            if (L < 0 || L >= nb) continue;
            const int c = cells[k];
            atomicMin(&sbox[6 * L + 0], c % S::TX);
            atomicMin(&sbox[6 * L + 1], (c / S::TX) % S::TY);
            atomicMin(&sbox[6 * L + 2], c / (S::TX * S::TY));
            atomicMax(&sbox[6 * L + 3], c % S::TX);
            atomicMax(&sbox[6 * L + 4], (c / S::TX) % S::TY);
            atomicMax(&sbox[6 * L + 5], c / (S::TX * S::TY));
        }
        for (int L = 0; L < nb; ++L) {
            __syncthreads();  // bitmaps and boxes written / the previous label's S read
            const uint32_t* bml = bm + L * S::NROWP;
            // the label's box in smoothed-value coordinates: x in [bx, bx + nsx)
            const int bx = sbox[6 * L + 0], by = sbox[6 * L + 1], bz = IS3D ? sbox[6 * L + 2] : 0;
            const int nsx = sbox[6 * L + 3] - bx + 5, nsy = sbox[6 * L + 4] - by + 5;
            const int nhz = IS3D ? sbox[6 * L + 5] - bz + 5 + 2 * P::K : 1;
            // smoothed x value of the window starting at bit xs of halo row `row`
            auto xval = [&](int row, int xs) -> double {
                const uint32_t w = bml[row] >> xs;
                double v = lut[w & 0x7Fu];
                if (P::NCH > 1) v += lut[128 + ((w >> 7) & 0x7Fu)];
                if (P::NCH > 2) v += lut[256 + ((w >> 14) & 0x7Fu)];
                return v;
            };
            if (IS3D) {
                // a strip (x, halo plane): its x values down all halo rows, then
                // the y sums of the tile's rows plus two each side
                // (the strips and columns outside the label's box are skipped;
                // their stale values are never read)
                for (int st = tid; st < nsx * nhz; st += 256) {
                    const int xs = bx + st % nsx, hz = bz + st / nsx;
                    double X[S::HY];
#pragma unroll
                    for (int r = 0; r < S::HY; ++r) X[r] = xval(hz * S::HY + r, xs);
#pragma unroll
                    for (int ys = 0; ys < P::SY; ++ys) {
                        double acc = 0.0;
#pragma unroll
                        for (int j = 0; j < P::NT; ++j) acc = __fma_rn(a.g[j], X[ys + j], acc);
                        Ym[(hz * P::SY + ys) * P::SX + xs] = acc;
                    }
                }
                __syncthreads();
                // a column (x, y): the z sums from its y-smoothed planes
                for (int cc = tid; cc < nsx * nsy; cc += 256) {
                    const int col = (by + cc / nsx) * P::SX + bx + cc % nsx;
                    double Y[S::HZ];
#pragma unroll
                    for (int hz = 0; hz < S::HZ; ++hz) Y[hz] = Ym[hz * P::SX * P::SY + col];
#pragma unroll
                    for (int zs = 0; zs < P::SZ; ++zs) {
                        double acc = 0.0;
#pragma unroll
                        for (int j = 0; j < P::NT; ++j) acc = __fma_rn(a.g[j], Y[zs + j], acc);
                        Sm[zs * P::SX * P::SY + col] = acc;
                    }
                }
            } else {
                for (int pt = tid; pt < nsx * nsy; pt += 256) {
                    const int xs = bx + pt % nsx, ys = by + pt / nsx;
                    double acc = 0.0;
#pragma unroll
                    for (int j = 0; j < P::NT; ++j) acc = __fma_rn(a.g[j], xval(ys + j, xs), acc);
                    Sm[ys * P::SX + xs] = acc;
                }
            }
            __syncthreads();
            // fourth-order differences at this label's interface cells
            for (int k = tid; k < ncell; k += 256) {
                if ((int)cli[k] != lb0 + L) continue;
                const int c = cells[k];
                const int lx = c % S::TX, ly = (c / S::TX) % S::TY, lz = c / (S::TX * S::TY);
                const int PY = P::SX, PZ = P::SX * P::SY;
                const int c0 = ((IS3D ? lz + 2 : 0) * P::SY + ly + 2) * P::SX + lx + 2;
                const double I0 = Sm[c0];
                const double Ix = (Sm[c0 - 2] - 8.0 * Sm[c0 - 1] + 8.0 * Sm[c0 + 1] - Sm[c0 + 2]) * a.idx12;
                const double Iy = (Sm[c0 - 2 * PY] - 8.0 * Sm[c0 - PY] + 8.0 * Sm[c0 + PY] - Sm[c0 + 2 * PY]) * a.idx12;
                const double Iz = IS3D ? (Sm[c0 - 2 * PZ] - 8.0 * Sm[c0 - PZ] + 8.0 * Sm[c0 + PZ] - Sm[c0 + 2 * PZ]) *
                                             a.idx12
                                       : 0.0;
                const double Ixx =
                    (-Sm[c0 + 2] + 16.0 * Sm[c0 + 1] - 30.0 * I0 + 16.0 * Sm[c0 - 1] - Sm[c0 - 2]) * a.idx12_sq;
                const double Iyy = (-Sm[c0 + 2 * PY] + 16.0 * Sm[c0 + PY] - 30.0 * I0 + 16.0 * Sm[c0 - PY] -
                                    Sm[c0 - 2 * PY]) *
                                   a.idx12_sq;
                const double Izz = IS3D ? (-Sm[c0 + 2 * PZ] + 16.0 * Sm[c0 + PZ] - 30.0 * I0 + 16.0 * Sm[c0 - PZ] -
                                           Sm[c0 - 2 * PZ]) *
                                              a.idx12_sq
                                        : 0.0;
                const int off[4] = {-2, -1, 1, 2};
                const double dc[4] = {1.0, -8.0, 8.0, -1.0};
                double sxy = 0.0, sxz = 0.0, syz = 0.0;
#pragma unroll
                for (int p = 0; p < 4; ++p)
#pragma unroll
                    for (int q = 0; q < 4; ++q) {
                        const double w = dc[p] * dc[q];
                        sxy += w * Sm[c0 + off[q] * PY + off[p]];
                        if (IS3D) {
                            sxz += w * Sm[c0 + off[q] * PZ + off[p]];
                            syz += w * Sm[c0 + off[q] * PZ + off[p] * PY];
                        }
                    }
                const double Ixy = sxy * a.idx144_sq, Ixz = IS3D ? sxz * a.idx144_sq : 0.0;
                const double Iyz = IS3D ? syz * a.idx144_sq : 0.0;
                const double grad_sq = Ix * Ix + Iy * Iy + Iz * Iz;
                double nxv = 0.0, nyv = 0.0, nzv = 0.0;
                const int i = D.idx(z0 + lz, y0 + ly, x0 + lx);
                if (grad_sq * dx * dx > 1e-8) {
                    const double inv_grad = 1.0 / sqrt(grad_sq);
                    nxv = -Ix * inv_grad;
                    nyv = -Iy * inv_grad;
                    nzv = -Iz * inv_grad;
                    const double trace_H = Ixx + Iyy + Izz;
                    const double gHg =
                        Ix * Ix * Ixx + Iy * Iy * Iyy + Iz * Iz * Izz + 2.0 * (Ix * Iy * Ixy + Ix * Iz * Ixz + Iy * Iz * Iyz);
                    double kap = (gHg - grad_sq * trace_H) / (grad_sq * sqrt(grad_sq));
                    if (fabs(kap * dx) < 1e-6) kap = 0.0;
                    a.nx[i] = nxv; a.ny[i] = nyv; a.nz[i] = nzv;
                    a.kappa[i] = dclamp(kap, -a.kappa_limit, a.kappa_limit);
                }
                geo_competitor<double>(a.phi_comp, i, nxv, nyv, nzv, core, core_of(c), S::CX, S::CY, IS3D);
            }
        }
    }
}

template <int R, bool IS3D>
static int launch_sep_tiles(gpk_grid* G, SepArgs a) {
    typedef GeoShape<R, IS3D> S;
    a.ntx = (G->d.Nx + S::TX - 1) / S::TX;
    a.nty = (G->d.Ny + S::TY - 1) / S::TY;
    const int ntz = (G->d.Nz + S::TZ - 1) / S::TZ;
    const size_t smem = sep_smem_bytes<R, IS3D>();
    // set once per process (thread-safe initialisation of a function-local static)
    static const cudaError_t attr_rc =
        cudaFuncSetAttribute(k_geometry_sep_tiles<R, IS3D>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    GPK_CUDA_TRY(attr_rc);
    k_geometry_sep_tiles<R, IS3D><<<a.ntx * a.nty * ntz, 256, smem, G->stream>>>(a);
    G->launches++;
    GPK_CUDA_TRY(cudaGetLastError());
    return GPK_OK;
}

}  // namespace gpk_dev

using namespace gpk_dev;

// Separable tiles (FP64 grids, kernel radii 4..10); -1 when they do not apply.
int gpk_geometry_sep_tiles(gpk_grid* G, int R, const double* gauss, int gauss_radius, double dx,
                           double kappa_limit) {
    if (G->precision != GPK_PREC_F64 || gauss_radius != R - 2 || R < 4 || R > 10) return -1;
    SepArgs a{};
    a.D = G->d;
    a.phi = G->phi;
    a.mask = G->mask;
    for (int j = 0; j < 2 * gauss_radius + 1; ++j) a.g[j] = gauss[j];
    a.dx = dx;
    a.idx12 = 1.0 / (12.0 * dx);
    const double idx_sq = 1.0 / (dx * dx);
    a.idx12_sq = idx_sq / 12.0;
    a.idx144_sq = idx_sq / 144.0;
    a.kappa_limit = kappa_limit;
    a.nx = (double*)G->f[GPK_FIELD_NX]; a.ny = (double*)G->f[GPK_FIELD_NY]; a.nz = (double*)G->f[GPK_FIELD_NZ];
    a.kappa = (double*)G->f[GPK_FIELD_KAPPA];
    a.phi_comp = G->phi_comp;
    if (G->d.is3d()) {
        switch (R) {
        case 4: return launch_sep_tiles<4, true>(G, a);
        case 5: return launch_sep_tiles<5, true>(G, a);
        case 6: return launch_sep_tiles<6, true>(G, a);
        case 7: return launch_sep_tiles<7, true>(G, a);
        case 8: return launch_sep_tiles<8, true>(G, a);
        case 9: return launch_sep_tiles<9, true>(G, a);
        default: return launch_sep_tiles<10, true>(G, a);
        }
    }
    switch (R) {
    case 4: return launch_sep_tiles<4, false>(G, a);
    case 5: return launch_sep_tiles<5, false>(G, a);
    case 6: return launch_sep_tiles<6, false>(G, a);
    case 7: return launch_sep_tiles<7, false>(G, a);
    case 8: return launch_sep_tiles<8, false>(G, a);
    case 9: return launch_sep_tiles<9, false>(G, a);
    default: return launch_sep_tiles<10, false>(G, a);
    }
}
