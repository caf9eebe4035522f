// gpk_separable.cu — the separable geometry of broad 3-D kernels, sm_100a.
//
// The reference smooths the indicator of every interface label over the whole
// grid (src/gpk_gaussian.cpp:9-72: per axis acc = 0; acc += w[k] * in[q+k-R]
// for k = 0..2R), then takes fourth-order differences at that label's
// interface cells (src/gpk_geometry.cpp:185-390).  The smoothed values are
// read only within two cells of those interface cells, so each label's passes
// here cover the periodic box of its interface cells plus two cells (and the
// kernel's radius more along the axes still to be smoothed), and all labels'
// boxes run in one launch per pass.  Every value that is formed has the
// reference's operations in its order.
//
//   x  the window of a row is 2R+1 bits of the label's row; a run of ones has
//      one of (2R+1)(2R+2)/2 sums, tabulated on the host in tap order, and
//      other patterns add their set taps (adding w * 0 = +0 changes nothing);
//   y, z  a thread forms eight outputs of a line from a register ring: one
//      value load and one tap load per tap and eight outputs; bound by the
//      unfused multiplies and adds (74 per output at radius 18).
// The whole-grid passes, one label after another (four launches each), took
// 7.0 ms plus 2.9 ms of evaluation and gaps for eight steps of 128^3 with 24
// grains at sigma 5.
#include <cuda_runtime.h>

#include <algorithm>
#include <cstring>
#include <vector>

#include "gpk_grid.h"

namespace gpk_dev {

struct SepRegion {
    int32_t label;
    int ox, oy, oz;           // first smoothed cell (in the grid)
    int nx, ny, nz;           // smoothed cells per axis
    int sy, ey, sz, ez;       // rows and planes that the y and z sums read: start, count (at most a period)
    long long t1, t2, s;      // offsets of the x-smoothed, y-smoothed and smoothed values
};

static constexpr int SEP_MAX_R = 31;  // a window of 63 bits

// marks the coordinates of each label's interface cells, per axis
__global__ void k_sep_marks(Dims D, const int32_t* __restrict__ active, const unsigned* __restrict__ n_active,
                            const int32_t* __restrict__ phi, uint8_t* __restrict__ marks) {
    const int na = (int)*n_active, S = D.Nx + D.Ny + D.Nz;
    for (int a = blockIdx.x * blockDim.x + threadIdx.x; a < na; a += gridDim.x * blockDim.x) {
        const int i = active[a];
        int z, y, x;
        D.decode(i, z, y, x);
        uint8_t* m = marks + (size_t)phi[i] * S;
        m[x] = 1;
        m[D.Nx + y] = 1;
        m[D.Nx + D.Ny + z] = 1;
    }
}

// x sums: a warp per row of a region, blockIdx.y = region (whose label's index it
// writes, for the evaluation)
template <typename real>
__global__ void __launch_bounds__(256) k_sep_box_x(Dims D, const int32_t* __restrict__ phi,
                                                   const SepRegion* __restrict__ regions, int R, int words,
                                                   const real* __restrict__ w, const real* __restrict__ runs,
                                                   real* __restrict__ out, int32_t* __restrict__ index) {
    extern __shared__ uint32_t sep_words[];
    const SepRegion g = regions[blockIdx.y];
    if (blockIdx.x == 0 && threadIdx.x == 0) index[g.label] = blockIdx.y;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, K = 2 * R + 1;
    uint32_t* row_bits = sep_words + warp * (words + 2);
    const int rows = g.ey * g.ez, nbit = g.nx + 2 * R;
    const int x0 = wrap_any(g.ox - R + lane, D.Nx);
    for (int r = blockIdx.x * 8 + warp; r < rows; r += gridDim.x * 8) {
        int y = g.sy + r % g.ey, z = g.sz + r / g.ey;
        if (y >= D.Ny) y -= D.Ny;
        if (z >= D.Nz) z -= D.Nz;
        const int32_t* row = phi + (size_t)(z * D.Ny + y) * D.Nx;
        __syncwarp();
        int x = x0;
        for (int b = 0; b < nbit; b += 128) {
            int32_t v[4];
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                v[u] = row[x];
                x += 32;
                while (x >= D.Nx) x -= D.Nx;
            }
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                const uint32_t bits = __ballot_sync(0xffffffffu, v[u] == g.label);
                if (lane == 0 && b + 32 * u < nbit) row_bits[(b >> 5) + u] = bits;
            }
        }
        if (lane < 2) row_bits[((nbit + 31) >> 5) + lane] = 0u;
        __syncwarp();
        real* o = out + g.t1 + (long long)r * g.nx;
        for (int e = lane; e < g.nx; e += 32) {
            const int q = e >> 5, sh = e & 31;
            const uint32_t lo = __funnelshift_r(row_bits[q], row_bits[q + 1], sh);
            const uint32_t hi = __funnelshift_r(row_bits[q + 1], row_bits[q + 2], sh);
            uint64_t p = (((uint64_t)hi << 32) | lo) & ((1ull << K) - 1ull);
            real v = (real)0;
            if (p) {
                const int first = __ffsll((long long)p) - 1;
                const uint64_t t = p >> first;
                if ((t & (t + 1ull)) == 0ull) {
                    v = runs[first * (K + 1) + __popcll(t)];
                } else {
                    while (p) {
                        v += w[__ffsll((long long)p) - 1];
                        p &= p - 1ull;
                    }
                }
            }
            o[e] = v;
        }
    }
}

// y sums (AXIS 1: ey rows -> ny) and z sums (AXIS 2: ez planes -> nz)
template <typename real, int AXIS>
__global__ void __launch_bounds__(256) k_sep_box_line(Dims D, const SepRegion* __restrict__ regions, int R,
                                                      const real* __restrict__ w, const real* __restrict__ in,
                                                      real* __restrict__ out) {
    constexpr int M = 8;
    __shared__ real tap[2 * SEP_MAX_R + 1];
    const SepRegion g = regions[blockIdx.y];
    const int K = 2 * R + 1;
    for (int k = threadIdx.x; k < K; k += 256) tap[k] = w[k];
    __syncthreads();
    const int n = AXIS == 1 ? g.ny : g.nz, e = AXIS == 1 ? g.ey : g.ez;
    const int period = AXIS == 1 ? D.Ny : D.Nz;
    const int nb = (n + M - 1) / M;
    // lines: (x, z) for y, (x, y) for z; threads run along x
    const int plane = AXIS == 1 ? g.nx : g.nx * g.ny;  // in and out: step along the line
    const int others = AXIS == 1 ? g.ez : 1;
    const int inner = AXIS == 1 ? g.nx : g.nx * g.ny;
    const long long total = (long long)inner * nb * others;
    for (long long t = blockIdx.x * 256LL + threadIdx.x; t < total; t += gridDim.x * 256LL) {
        const int l = (int)(t % inner), b = (int)(t / inner % nb), o = (int)(t / inner / nb);
        const real* src = in + (AXIS == 1 ? g.t1 + (long long)o * g.ey * g.nx : g.t2) + l;
        real* dst = out + (AXIS == 1 ? g.t2 + (long long)o * g.ny * g.nx : g.s) + l;
        // position of the window's first value; past the last one a period
        // starts again, or (values that no stored output reads) the last stays
        int j = b * M;
        if (e == period) j %= period;
        auto next = [&]() {
            const real v = src[(long long)j * plane];
            if (++j >= e) j = e == period ? 0 : e - 1;
            return v;
        };
        real v[M], acc[M];
#pragma unroll
        for (int m = 0; m < M; ++m) {
            v[m] = next();
            acc[m] = (real)0;
        }
        int k = 0;
        for (; k + M <= K; k += M) {
#pragma unroll
            for (int q = 0; q < M; ++q) {
                const real wk = tap[k + q];
#pragma unroll
                for (int m = 0; m < M; ++m) acc[m] += wk * v[(m + q) % M];
                v[q] = next();
            }
        }
#pragma unroll
        for (int q = 0; q < M - 1; ++q) {
            if (k + q >= K) break;
            const real wk = tap[k + q];
#pragma unroll
            for (int m = 0; m < M; ++m) acc[m] += wk * v[(m + q) % M];
            v[q] = next();
        }
#pragma unroll
        for (int m = 0; m < M; ++m)
            if (b * M + m < n) dst[(long long)(b * M + m) * plane] = acc[m];
    }
}

// fourth-order differences at the interface cells of the labels in `index`
// (label -> region, -1: another batch's)
template <typename real>
__global__ void k_sep_box_eval(Dims D, const int32_t* __restrict__ active, const unsigned* __restrict__ n_active,
                               const int32_t* __restrict__ phi, const int32_t* __restrict__ index,
                               const SepRegion* __restrict__ regions, const real* __restrict__ Sv, real dx,
                               real kappa_limit, real* __restrict__ nxo, real* __restrict__ nyo,
                               real* __restrict__ nzo, real* __restrict__ ko) {
    const real idx12 = (real)1 / ((real)12 * dx);
    const real idx_sq = (real)1 / (dx * dx);
    const real idx12_sq = idx_sq / (real)12;
    const real idx144_sq = idx_sq / (real)144;
    const int na = (int)*n_active;
    for (int a = blockIdx.x * blockDim.x + threadIdx.x; a < na; a += gridDim.x * blockDim.x) {
        const int i = active[a];
        const int r = index[phi[i]];
        if (r < 0) continue;
        const SepRegion g = regions[r];
        int z, y, x;
        D.decode(i, z, y, x);
        // the cell in its region, and the two cells to each side (a region
        // that is a whole period wraps)
        int xo[5], yo[5], zo[5];
#pragma unroll
        for (int d = 0; d < 5; ++d) {
            xo[d] = wrap_any(x - g.ox + d - 2, D.Nx);
            yo[d] = wrap_any(y - g.oy + d - 2, D.Ny) * g.nx;
            zo[d] = wrap_any(z - g.oz + d - 2, D.Nz) * (g.nx * g.ny);
        }
        const real* S = Sv + g.s;
        auto at = [&](int c, int b, int e) { return S[zo[c] + yo[b] + xo[e]]; };
        const real I0 = at(2, 2, 2);
        const real Ix = (at(2, 2, 0) - (real)8 * at(2, 2, 1) + (real)8 * at(2, 2, 3) - at(2, 2, 4)) * idx12;
        const real Iy = (at(2, 0, 2) - (real)8 * at(2, 1, 2) + (real)8 * at(2, 3, 2) - at(2, 4, 2)) * idx12;
        const real Iz = (at(0, 2, 2) - (real)8 * at(1, 2, 2) + (real)8 * at(3, 2, 2) - at(4, 2, 2)) * idx12;
        const real Ixx = (-at(2, 2, 4) + (real)16 * at(2, 2, 3) - (real)30 * I0 + (real)16 * at(2, 2, 1) - at(2, 2, 0)) * idx12_sq;
        const real Iyy = (-at(2, 4, 2) + (real)16 * at(2, 3, 2) - (real)30 * I0 + (real)16 * at(2, 1, 2) - at(2, 0, 2)) * idx12_sq;
        const real Izz = (-at(4, 2, 2) + (real)16 * at(3, 2, 2) - (real)30 * I0 + (real)16 * at(1, 2, 2) - at(0, 2, 2)) * idx12_sq;
        constexpr int off[4] = {0, 1, 3, 4};
        const real dc[4] = {(real)1, (real)-8, (real)8, (real)-1};
        real Ixy_sum = 0, Ixz_sum = 0, Iyz_sum = 0;
#pragma unroll
        for (int aa = 0; aa < 4; ++aa)
#pragma unroll
            for (int b = 0; b < 4; ++b) {
                const real wt = dc[aa] * dc[b];
                Ixy_sum += wt * at(2, off[b], off[aa]);
                Ixz_sum += wt * at(off[b], 2, off[aa]);
                Iyz_sum += wt * at(off[b], off[aa], 2);
            }
        const real Ixy = Ixy_sum * idx144_sq, Ixz = Ixz_sum * idx144_sq, Iyz = Iyz_sum * idx144_sq;
        const real grad_sq = Ix * Ix + Iy * Iy + Iz * Iz;
        if (grad_sq * dx * dx > (real)1e-8) {
            const real inv_grad = (real)1 / sqrt(grad_sq);
            nxo[i] = -Ix * inv_grad;
            nyo[i] = -Iy * inv_grad;
            nzo[i] = -Iz * inv_grad;
            const real trace_H = Ixx + Iyy + Izz;
            const real gHg = Ix * Ix * Ixx + Iy * Iy * Iyy + Iz * Iz * Izz + (real)2 * (Ix * Iy * Ixy + Ix * Iz * Ixz + Iy * Iz * Iyz);
            real k = (gHg - grad_sq * trace_H) / (grad_sq * sqrt(grad_sq));
            if (fabs(k * dx) < (real)1e-6) k = (real)0;
            ko[i] = dclamp(k, -kappa_limit, kappa_limit);
        }
    }
}

// the shortest periodic run of coordinates that holds every marked one of m[0, n): a
// warp reads 32 marks at a time and walks the runs of marked coordinates
__device__ __forceinline__ void arc_of(const uint8_t* __restrict__ m, int n, int lane, int& start, int& len) {
    int first = -1, last = -1, best = -1, at = 0;
    unsigned carry = 0;  // the coordinate before this word is marked
    for (int b = 0; b < n; b += 32) {
        const unsigned w = __ballot_sync(0xffffffffu, b + lane < n && m[b + lane]);
        for (unsigned s = w & ~((w << 1) | carry); s; s &= s - 1u) {  // first coordinates of the runs
            const int q = __ffs(s) - 1;
            const unsigned below = w & ((1u << q) - 1u);
            if (below) last = b + 31 - __clz(below);
            if (first < 0) first = b + q;
            else if (b + q - last - 1 > best) {
                best = b + q - last - 1;
                at = b + q;
            }
        }
        if (w) last = b + 31 - __clz(w);
        carry = w >> 31;
    }
    if (first + n - last - 1 > best) {
        best = first + n - last - 1;
        at = first;
    }
    start = at;  // the marked coordinate after the longest gap
    len = n - best;
}

struct SepArc {
    int32_t label;
    int start[3], len[3];  // x, y, z
};

// The arcs of every label with marks, in any order.  On the host this took a
// copy of the marks and a walk over all labels a grid has had, up to 8 bytes a
// cell: 3 ms of 4.6 for 128^3 with 24 grains and ids up to 40 000.
__global__ void __launch_bounds__(256) k_sep_arcs(Dims D, int label_cap, const uint8_t* __restrict__ marks,
                                                  unsigned* __restrict__ count, SepArc* __restrict__ arcs) {
    const int lane = threadIdx.x & 31, S = D.Nx + D.Ny + D.Nz;
    for (int p = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; p < label_cap; p += (gridDim.x * blockDim.x) >> 5) {
        const uint8_t* m = marks + (size_t)p * S;
        unsigned any = 0;
        for (int b = 0; b < D.Nx && !any; b += 32) any = __ballot_sync(0xffffffffu, b + lane < D.Nx && m[b + lane]);
        if (!any) continue;
        SepArc r;
        r.label = p;
        arc_of(m, D.Nx, lane, r.start[0], r.len[0]);
        arc_of(m + D.Nx, D.Ny, lane, r.start[1], r.len[1]);
        arc_of(m + D.Nx + D.Ny, D.Nz, lane, r.start[2], r.len[2]);
        if (lane == 0) arcs[atomicAdd(count, 1u)] = r;
    }
}

}  // namespace gpk_dev

using namespace gpk_dev;

// The sums of the runs of taps (radii to 31), made with the grid: the first step
// allocates nothing.
template <typename real>
int gpk_geometry_separable_init(gpk_grid* G) {
    const HostKernels<real>* hk = (const HostKernels<real>*)G->host_kernels;
    const int R = hk->gauss_radius, K = 2 * R + 1;
    if (!hk->global_separable || R > SEP_MAX_R) return GPK_OK;
    std::vector<real> runs((size_t)K * (K + 1), (real)0);
    for (int s = 0; s < K; ++s) {
        real acc = (real)0;
        for (int l = 1; s + l <= K; ++l) {
            acc += hk->gauss_w[s + l - 1];
            runs[(size_t)s * (K + 1) + l] = acc;
        }
    }
    GPK_TRY(gpk_alloc(G, &G->d_sep_runs, sizeof(real) * runs.size()));
    GPK_CUDA_TRY(cudaMemcpy(G->d_sep_runs, runs.data(), sizeof(real) * runs.size(), cudaMemcpyHostToDevice));
    return GPK_OK;
}
template int gpk_geometry_separable_init<float>(gpk_grid*);
template int gpk_geometry_separable_init<double>(gpk_grid*);

// Smoothing and differences of every interface label into nx, ny, nz, kappa
// (zero on entry); -1 where this form does not apply (the caller then smooths
// label by label over the whole grid).
template <typename real>
int gpk_geometry_separable(gpk_grid* G, real dx, real kappa_limit) {
    HostKernels<real>* hk = (HostKernels<real>*)G->host_kernels;
    const Dims D = G->d;
    const int R = hk->gauss_radius, span = D.Nx + D.Ny + D.Nz;
    // in the scratch for now: marks, then the number of arcs and the arcs
    const size_t mark_bytes = (size_t)G->label_cap * span, at = (mark_bytes + 15) & ~(size_t)15;
    if (!G->d_sep_runs || !D.is3d() || D.Nx < 2 || D.Ny < 2 || mark_bytes > 8 * (size_t)D.N ||
        at + 16 + sizeof(SepArc) * (size_t)G->label_cap > G->scratch_bytes)
        return -1;
    unsigned char* counted = G->scratch + at;
    GPK_CUDA_TRY(cudaMemsetAsync(G->scratch, 0, at + 16, G->stream));
    k_sep_marks<<<G->num_sms * 8, 256, 0, G->stream>>>(D, G->active, &G->scal->n_active, G->phi, G->scratch);
    k_sep_arcs<<<std::min(G->num_sms * 8, (G->label_cap + 7) / 8), 256, 0, G->stream>>>(
        D, G->label_cap, G->scratch, (unsigned*)counted, (SepArc*)(counted + 16));
    G->launches += 2;
    GPK_CUDA_TRY(cudaGetLastError());
    // (one copy where there are at most FIRST labels)
    constexpr int FIRST = 1024;
    std::vector<unsigned char> got(16 + sizeof(SepArc) * (size_t)std::min(FIRST, G->label_cap));
    GPK_CUDA_TRY(cudaMemcpyAsync(got.data(), counted, got.size(), cudaMemcpyDeviceToHost, G->stream));
    GPK_CUDA_TRY(cudaStreamSynchronize(G->stream));
    unsigned n_arcs;
    std::memcpy(&n_arcs, got.data(), sizeof(n_arcs));
    const size_t have = got.size(), need = 16 + sizeof(SepArc) * (size_t)n_arcs;
    got.resize(std::max(have, need));
    if (need > have) {
        GPK_CUDA_TRY(cudaMemcpyAsync(got.data() + have, counted + have, need - have, cudaMemcpyDeviceToHost, G->stream));
        GPK_CUDA_TRY(cudaStreamSynchronize(G->stream));
    }
    std::vector<SepArc> arcs(n_arcs);
    if (n_arcs) std::memcpy(arcs.data(), got.data() + 16, sizeof(SepArc) * n_arcs);
    std::sort(arcs.begin(), arcs.end(), [](const SepArc& a, const SepArc& b) { return a.label < b.label; });
    std::vector<SepRegion> regions;
    regions.reserve(n_arcs);
    for (const SepArc& a : arcs) {
        SepRegion g{};
        g.label = a.label;
        auto box = [&](int axis, int n, int& o, int& c) {
            c = a.len[axis] + 4;
            o = a.start[axis] - 2 < 0 ? a.start[axis] - 2 + n : a.start[axis] - 2;
            if (c >= n) { o = 0; c = n; }
        };
        auto ext = [&](int o, int c, int n, int& s, int& e) {
            e = c + 2 * R < n ? c + 2 * R : n;
            s = wrap_any(o - R, n);
        };
        box(0, D.Nx, g.ox, g.nx);
        box(1, D.Ny, g.oy, g.ny);
        box(2, D.Nz, g.oz, g.nz);
        ext(g.oy, g.ny, D.Ny, g.sy, g.ey);
        ext(g.oz, g.nz, D.Nz, g.sz, g.ez);
        regions.push_back(g);
    }
    if (regions.empty()) return GPK_OK;
    // in the scratch (the marks have been read): label index and regions, then
    // the values of the three passes
    const size_t head = ((sizeof(int32_t) * (size_t)G->label_cap + 15) & ~(size_t)15);
    const size_t table = head + sizeof(SepRegion) * regions.size();
    const size_t values = (table + 255) & ~(size_t)255;
    if (values + 3 * sizeof(real) * (size_t)D.N > G->scratch_bytes) return -1;
    const size_t room = (G->scratch_bytes - values) / sizeof(real);
    // (a region needs at most N values of each pass; the x-smoothed box is the largest, by its halo)
    const size_t cap1 = (size_t)D.N + (room - 3 * (size_t)D.N) / 2;
    const size_t cap2 = (size_t)D.N + (room - 3 * (size_t)D.N) / 4, cap3 = cap2;
    real* t1 = (real*)(G->scratch + values);
    real* t2 = t1 + cap1;
    real* s = t2 + cap2;
    const real* runs = (const real*)G->d_sep_runs;
    for (size_t r0 = 0; r0 < regions.size();) {
        size_t n = 0, u1 = 0, u2 = 0, u3 = 0;
        int max_rows = 0, max_y = 0, max_z = 0, max_x = 0;
        for (; r0 + n < regions.size(); ++n) {
            SepRegion& g = regions[r0 + n];
            const size_t a = (size_t)g.nx * g.ey * g.ez, b = (size_t)g.nx * g.ny * g.ez, c = (size_t)g.nx * g.ny * g.nz;
            if (n > 0 && (u1 + a > cap1 || u2 + b > cap2 || u3 + c > cap3 || n == 65535)) break;
            g.t1 = (long long)u1; g.t2 = (long long)u2; g.s = (long long)u3;
            u1 += a; u2 += b; u3 += c;
            max_rows = std::max(max_rows, g.ey * g.ez);
            max_y = std::max(max_y, (int)std::min<long long>((long long)g.nx * ((g.ny + 7) / 8) * g.ez, 1 << 30));
            max_z = std::max(max_z, (int)std::min<long long>((long long)g.nx * ((g.nz + 7) / 8) * g.ny, 1 << 30));
            max_x = std::max(max_x, g.nx);
        }
        // (pageable memory: staged when the call returns)
        GPK_CUDA_TRY(cudaMemsetAsync(G->scratch, 0xff, sizeof(int32_t) * (size_t)G->label_cap, G->stream));
        GPK_CUDA_TRY(cudaMemcpyAsync(G->scratch + head, &regions[r0], sizeof(SepRegion) * n, cudaMemcpyHostToDevice,
                                     G->stream));
        const SepRegion* dr = (const SepRegion*)(G->scratch + head);
        const int words = (max_x + 2 * R + 31) / 32 + 1;
        auto blocks = [&](long long work) { return (unsigned)std::max(1LL, std::min(work, 4096LL)); };
        const size_t smem = sizeof(uint32_t) * 8 * (size_t)(words + 2);
        if (smem > 48 * 1024) return -1;  // (rows of 48 000 cells)
        k_sep_box_x<real><<<dim3(blocks((max_rows + 7) / 8), (unsigned)n), 256, smem, G->stream>>>(
            D, G->phi, dr, R, words, (const real*)G->d_gauss, runs, t1, (int32_t*)G->scratch);
        k_sep_box_line<real, 1><<<dim3(blocks((max_y + 255) / 256), (unsigned)n), 256, 0, G->stream>>>(
            D, dr, R, (const real*)G->d_gauss, t1, t2);
        k_sep_box_line<real, 2><<<dim3(blocks((max_z + 255) / 256), (unsigned)n), 256, 0, G->stream>>>(
            D, dr, R, (const real*)G->d_gauss, t2, s);
        k_sep_box_eval<real><<<G->num_sms * 8, 256, 0, G->stream>>>(
            D, G->active, &G->scal->n_active, G->phi, (const int32_t*)G->scratch, dr, s, dx, kappa_limit,
            (real*)G->f[GPK_FIELD_NX], (real*)G->f[GPK_FIELD_NY], (real*)G->f[GPK_FIELD_NZ],
            (real*)G->f[GPK_FIELD_KAPPA]);
        G->launches += 4;
        GPK_CUDA_TRY(cudaGetLastError());
        r0 += n;
    }
    return GPK_OK;
}
template int gpk_geometry_separable<float>(gpk_grid*, float, float);
template int gpk_geometry_separable<double>(gpk_grid*, double, double);
