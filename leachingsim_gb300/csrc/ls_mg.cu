// ls_mg.cu - geometric multigrid preconditioner of the inner pressure PCG.
//
// Every level holds its operator in "excess + graph Laplacian" form,
//     (M x)_i = e_i x_i + sum_{links ij} c_ij (x_i - x_j),   e_i >= 0, c_ij >= 0,
// so M is symmetric positive (semi)definite for any rounding of e and c: the FP32 copy of
// the finest operator cannot turn indefinite, and the Galerkin coarse operators are sums of
// positive terms (no cancellation). The finest level is the inner system itself (excess =
// links of a Pore row to rows that are not inner unknowns).
//
// The Pore network is masked by Dirichlet voxels everywhere and its links span ~13 orders
// of magnitude, so plain 2x2x2 aggregation would hand coarse corrections to Pore clusters
// that merely share a block with the main network while being joined to it by no strong
// link; such a cluster's near-null mode then keeps the correction (its residual is ~1e-13
// of the error). The hierarchy therefore works per strong component:
//   * components: connected pieces of the unknowns over links with
//     c_ij / sqrt(d_i d_j) > kStrong (union-find on the device);
//   * aggregation: each 2x2x2 block becomes one coarse cell owned by the component with
//     most members in the block; only its members are restricted to / prolongated from it
//     (piecewise-constant interpolation); links from members to non-members become excess;
//   * V-cycle: two damped-Jacobi sweeps before and after the coarse correction, a fixed
//     number of Jacobi sweeps by one CTA on the coarsest level, so the cycle is a symmetric
//     operator usable inside CG.
#include <algorithm>
#include <functional>
#include <type_traits>
#include <cstdio>

#include "ls_internal.cuh"

namespace ls {

constexpr double kStrong = 1e-3;   // scaled link weight below which a link joins no components
constexpr double kOmega = 2.0 / 3.0;
constexpr int kCoarsestCells = 512;
constexpr int kCoarseSweeps = 48;
constexpr double kProlongScale = 1.8;
constexpr int kKLevels = 3;   // levels 1..kKLevels take a K-cycle coarse correction
constexpr int kKSlot0 = 32;   // device scalar slots of the K-cycle FCG (5 per level)
// Levels up to these sizes run fused (k_mg_fused). FP32: one block with a cell per thread; a level of two
// cells per thread, or one on the cluster, takes longer than its kernels do. With the largest fused
// level just left out and taken in, ms: 80x80x80 (1,000 cells) 6.14 and 6.04; 61x83x101, implicit
// saturation (1,144) 124.7 and 126.1; 101x77x95 (1,560) 7.8 and 8.1; 200x160x240 (1,950) 17.8 and
// 19.5; 160x256x256 (2,560) 18.2 and 19.8; 64x64x64 with acid (4,096) 58.9 and 61.0; a fractured
// step of 224x320x320 (5,600) 284 and 300; without any fused level 8.4, 165, 10.7, 21.4, 21.3, 69 and 303.
// FP64 (48x64x64, 3,072 cells): 26.3 and 26.0.
constexpr long long kFuseCells32 = 1024;
constexpr long long kFuseCells64 = 8192;
// FP64 with at most this many cells on the coarsest level keeps the level kernels: its 48 sweeps cost 48
// cluster barriers, and one SM does them faster. Cold solves, fused and not: 40x40x40 (125 cells)
// 10.3 and 8.1 ms, 128x160x120 (80) 41.4 and 33.1, 61x83x101 (168) 21.6 and 20.1, 48x48x48 (216) 10.2
// and 10.0, 48x52x48 (252) 9.6 and 9.9, 64x48x48 (288) 12.3 and 13.5, 64x64x64 (512) 13.3 and 19.3.
constexpr long long kFuseCoarsest64 = 232;
constexpr int kUnionSpin = 1 << 20;  // bound on the union-find retry loop
// learned coarse solver (LS_PRESS_LEARNED): the network solves level kLearnedLevel in place of
// the V-cycle below the K-cycle levels
constexpr int kLearnedLevel = kKLevels + 1;  // the level below the K-cycle levels
constexpr float kLpcOutScale = 64.f;  // network output x this x max|D^-1/2 b| = D^1/2 x
constexpr int kLpcSlot = 60;          // device scalar: max |D^-1/2 b| over the level's members

}  // namespace ls

#include "ls_mg_fused.cuh"

namespace ls {

__device__ __forceinline__ long long lidx(const Grid& g, int i, int j, int k) {
    return (long long)k + (long long)g.K * ((long long)j + (long long)g.J * i);
}

// (M x)_r in difference form (links on the six faces; f0/f1/f2 hold the + faces)
template <typename T>
__device__ __forceinline__ T m_apply(const Grid& g, long long r, int i, int j, int k, const T* __restrict__ e,
                                     const T* __restrict__ f0, const T* __restrict__ f1,
                                     const T* __restrict__ f2, const T* __restrict__ x) {
    const T xr = x[r];
    T acc = e[r] * xr;
    if (i > 0) acc += f0[r - g.JK] * (xr - x[r - g.JK]);
    if (j > 0) acc += f1[r - g.K] * (xr - x[r - g.K]);
    if (k > 0) acc += f2[r - 1] * (xr - x[r - 1]);
    if (k + 1 < g.K) acc += f2[r] * (xr - x[r + 1]);
    if (j + 1 < g.J) acc += f1[r] * (xr - x[r + g.K]);
    if (i + 1 < g.I) acc += f0[r] * (xr - x[r + g.JK]);
    return acc;
}

// Resident blocks per SM of the passes that hold more than 32 registers and sum nothing, whose
// grid is that many blocks per SM: with grid_for's 8 a second, partly filled wave followed (the
// finest sweep with the correction at 338x338x283: 186 us, now 165). 4, 5 or 6 blocks: a step with
// acid there differs by 0.4 %. The passes that leave partial sums keep grid_for's
// grid, which is part of the order of their sums.
constexpr int kPassBlocks = 5;
static int pass_grid(const ls_ctx* c, long long n) { return std::min(grid_for(c, n), c->num_sms * kPassBlocks); }

constexpr uint8_t kCellMember = 1, kCellLive = 2;

static size_t level_pad(const Grid& g) { return ((size_t)g.JK + 31) / 32 * 32; }

// 1 / (e + sum of the six links) of live cells, 1 elsewhere
template <typename T>
__global__ void k_level_invd(Grid g, const int* __restrict__ comp, const int8_t* __restrict__ kind,
                             const T* __restrict__ e, const T* __restrict__ f0, const T* __restrict__ f1,
                             const T* __restrict__ f2, T* __restrict__ invd) {
    for (long long r = blockIdx.x * (long long)blockDim.x + threadIdx.x; r < g.N;
         r += (long long)gridDim.x * blockDim.x) {
        T out = (T)1;
        bool live = comp ? comp[r] >= 0 : kind[r] == 2;
        if (live) {
            int i, j, k;
            decode(g, r, i, j, k);
            T d = e[r];
            if (i > 0) d += f0[r - g.JK];
            if (j > 0) d += f1[r - g.K];
            if (k > 0) d += f2[r - 1];
            if (k + 1 < g.K) d += f2[r];
            if (j + 1 < g.J) d += f1[r];
            if (i + 1 < g.I) d += f0[r];
            out = (d > (T)0) ? (T)1 / d : (T)1;
        }
        invd[r] = out;
    }
}

// ---------------------------------------------------------------------------
// strong components (union-find with path halving; ids are voxel indices, the root is the
// smallest voxel of the component)

// find with path halving (hooking). Each store points a non-root at one of its ancestors,
// and a parent value read from a stale L1 line (L1 is not coherent across SMs) is a former
// ancestor, so still an ancestor. A stale line can however show a root that another SM has
// hooked since; the CAS then fails, and the retry reads with FRESH loads that bypass L1.
template <bool FRESH>
__device__ __forceinline__ int cc_find(int* parent, int x) {
    int p = FRESH ? __ldcg(parent + x) : parent[x];
    int guard = 0;
    while (p != x && guard++ < kUnionSpin) {
        int gp = FRESH ? __ldcg(parent + p) : parent[p];
        parent[x] = gp;
        x = p;
        p = gp;
    }
    return x;
}

// read-only find (compression): a path-halving store from a stale parent value could
// otherwise overwrite a cell's final root with an intermediate ancestor
__device__ __forceinline__ int cc_find_ro(const int* parent, int x) {
    int p = parent[x];
    int guard = 0;
    while (p != x && guard++ < kUnionSpin) {
        x = p;
        p = parent[x];
    }
    return x;
}

// is the link c between cells r and nb strong? c / sqrt(d_r d_nb) > kStrong, squared: no square
// root on the FP64 pipe (c > 0 only between two unknowns)
template <typename T>
__device__ __forceinline__ bool cc_strong(T c, T ir, T inb) {
    const T w2 = c * c * ir * inb;
    return c > (T)0 && w2 > (T)(kStrong * kStrong);
}

// Every unknown points at the first cell of its strong run along k within the warp's 32 cells
// (itself where it is not linked to the cell before): the hooks below start from trees of whole
// runs, not of single cells.
template <typename T>
__global__ void __launch_bounds__(kBlock) k_cc_init(Grid g, const int8_t* __restrict__ kind, const T* __restrict__ f2,
                                                    const T* __restrict__ invd, int* __restrict__ parent) {
    const int lane = (int)(threadIdx.x & 31u);
    for (long long r0 = (long long)blockIdx.x * blockDim.x + (threadIdx.x & ~31u); r0 < g.N;
         r0 += (long long)gridDim.x * blockDim.x) {
        const long long r = r0 + lane;
        bool next = false;
        if (r + 1 < g.N) next = cc_strong(f2[r], invd[r], invd[r + 1]);
        const unsigned int linked = __ballot_sync(0xffffffffu, next) << 1;  // bit l: to the cell before
        if (r < g.N) {
            const int start = 31 - __clz(~linked & (0xffffffffu >> (31 - lane)));
            parent[r] = (kind[r] == 2) ? (int)(r0 + start) : -1;
        }
    }
}

template <typename T>
__device__ __forceinline__ void cc_hook(int* parent, int a, int b, int* __restrict__ err) {
    int spins = 0;
    while (true) {
        int ra = spins ? cc_find<true>(parent, a) : cc_find<false>(parent, a);
        int rb = spins ? cc_find<true>(parent, b) : cc_find<false>(parent, b);
        if (ra == rb) break;
        int lo = ra < rb ? ra : rb, hi = ra < rb ? rb : ra;
        if (atomicCAS(&parent[hi], hi, lo) == hi) break;
        if (++spins > kUnionSpin) { atomicExch(err, 1); break; }
    }
}

// Joins the runs over the strong i and j links, and along k from one warp's cells to the next.
// Two runs that face each other need one hook: a cell leaves it to the cell before when that one
// is in the same run, has a strong link in the same direction, and their neighbours are linked
// too. The finds are chains of dependent loads, so their number is what counts: 0.81 ms
// at 338x338x283 (8 M unknowns) and 0.14 at 64x64x64, against 5.0 and 0.73 with every cell its own
// tree and a hook per strong link.
template <typename T>
__global__ void __launch_bounds__(kBlock) k_cc_hook(Grid g, const T* __restrict__ f0, const T* __restrict__ f1,
                                                    const T* __restrict__ f2, const T* __restrict__ invd, int* parent,
                                                    int* __restrict__ err) {
    const int lane = (int)(threadIdx.x & 31u);
    for (long long r0 = (long long)blockIdx.x * blockDim.x + (threadIdx.x & ~31u); r0 < g.N;
         r0 += (long long)gridDim.x * blockDim.x) {
        const long long r = r0 + lane;
        const bool in = r < g.N;
        const T ir = in ? invd[r] : (T)0;
        const bool next = in && r + 1 < g.N && cc_strong(f2[r], ir, invd[r + 1]);
        const bool before = __shfl_up_sync(0xffffffffu, next, 1) && lane > 0;  // linked to the cell before
        if (next && lane == 31) cc_hook<T>(parent, (int)r, (int)(r + 1), err);
#pragma unroll
        for (int d = 0; d < 2; ++d) {
            const long long nb = r + (d ? (long long)g.K : g.JK);
            const T c = in ? (d ? f1 : f0)[r] : (T)0;
            bool s = false, nb_next = false;
            if (c > (T)0) {
                const T in0 = invd[nb];
                s = cc_strong(c, ir, in0);
                if (s && nb + 1 < g.N) nb_next = cc_strong(f2[nb], in0, invd[nb + 1]);
            }
            const bool prev = __shfl_up_sync(0xffffffffu, s && nb_next, 1) && before;
            if (s && !prev) cc_hook<T>(parent, (int)r, (int)nb, err);
        }
    }
}

__global__ void k_cc_compress(Grid g, int* parent) {
    for (long long r = blockIdx.x * (long long)blockDim.x + threadIdx.x; r < g.N;
         r += (long long)gridDim.x * blockDim.x) {
        if (parent[r] < 0) continue;
        parent[r] = cc_find_ro(parent, (int)r);
    }
}

// ---------------------------------------------------------------------------
// hierarchy construction

// dominant component of each 2x2x2 block (most members; ties: smallest id)
__global__ void k_mg_dom(Grid f, Grid cg, const int* __restrict__ fcomp, int* __restrict__ ccomp) {
    for (long long R = blockIdx.x * (long long)blockDim.x + threadIdx.x; R < cg.N;
         R += (long long)gridDim.x * blockDim.x) {
        int I, J, K;
        decode(cg, R, I, J, K);
        int ids[8];
        int n = 0;
        for (int a = 0; a < 2; ++a)
            for (int b = 0; b < 2; ++b)
                for (int c = 0; c < 2; ++c) {
                    int i = 2 * I + a, j = 2 * J + b, k = 2 * K + c;
                    if (i >= f.I || j >= f.J || k >= f.K) continue;
                    int id = fcomp[lidx(f, i, j, k)];
                    if (id >= 0) ids[n++] = id;
                }
        int best = -1, bestc = 0;
        for (int q = 0; q < n; ++q) {
            int cnt = 0;
            for (int s = 0; s < n; ++s) cnt += (ids[s] == ids[q]);
            if (cnt > bestc || (cnt == bestc && ids[q] < best)) { best = ids[q]; bestc = cnt; }
        }
        ccomp[R] = best;
    }
}

__global__ void k_mg_flags(Grid f, Grid cg, const int* __restrict__ fcomp, const int* __restrict__ ccomp,
                           uint8_t* __restrict__ flags) {
    for (long long r = blockIdx.x * (long long)blockDim.x + threadIdx.x; r < f.N; r += (long long)gridDim.x * blockDim.x) {
        const int id = fcomp[r];
        int out = 0;
        if (id >= 0) {
            int i, j, k;
            decode(f, r, i, j, k);
            out = kCellLive | (ccomp[lidx(cg, i >> 1, j >> 1, k >> 1)] == id ? kCellMember : 0);
        }
        flags[r] = (uint8_t)out;
    }
}

// is fine cell (i,j,k) a member of its own block's owner?
__device__ __forceinline__ bool is_member(const Grid& f, const Grid& cg, const int* fcomp, const int* ccomp,
                                          int i, int j, int k) {
    int id = fcomp[lidx(f, i, j, k)];
    return id >= 0 && ccomp[lidx(cg, i >> 1, j >> 1, k >> 1)] == id;
}

// Galerkin coarse operator P^T M P for piecewise-constant P restricted to the members of
// each block's owner: coarse excess = member excess + member links to non-members;
// coarse + face link = member-to-member links crossing the block's + face.
template <typename T>
__global__ void k_mg_coarse_op(Grid f, Grid cg, const int* __restrict__ fcomp, const int* __restrict__ ccomp,
                               const T* __restrict__ fe, const T* __restrict__ f0, const T* __restrict__ f1,
                               const T* __restrict__ f2, T* __restrict__ ce, T* __restrict__ c0,
                               T* __restrict__ c1, T* __restrict__ c2) {
    for (long long R = blockIdx.x * (long long)blockDim.x + threadIdx.x; R < cg.N;
         R += (long long)gridDim.x * blockDim.x) {
        int I, J, K;
        decode(cg, R, I, J, K);
        const int own = ccomp[R];
        double ex = 0.0, e0 = 0.0, e1 = 0.0, e2 = 0.0;
        if (own >= 0) {
            for (int a = 0; a < 2; ++a)
                for (int b = 0; b < 2; ++b)
                    for (int c = 0; c < 2; ++c) {
                        int i = 2 * I + a, j = 2 * J + b, k = 2 * K + c;
                        if (i >= f.I || j >= f.J || k >= f.K) continue;
                        long long fr = lidx(f, i, j, k);
                        if (fcomp[fr] != own) continue;
                        ex += (double)fe[fr];
                        // the six links of this member
                        const int di[6] = {1, -1, 0, 0, 0, 0}, dj[6] = {0, 0, 1, -1, 0, 0},
                                  dk[6] = {0, 0, 0, 0, 1, -1};
                        for (int d = 0; d < 6; ++d) {
                            int ni = i + di[d], nj = j + dj[d], nk = k + dk[d];
                            if (ni < 0 || nj < 0 || nk < 0 || ni >= f.I || nj >= f.J || nk >= f.K) continue;
                            long long nr = lidx(f, ni, nj, nk);
                            double cl;
                            switch (d) {
                            case 0: cl = (double)f0[fr]; break;
                            case 1: cl = (double)f0[nr]; break;
                            case 2: cl = (double)f1[fr]; break;
                            case 3: cl = (double)f1[nr]; break;
                            case 4: cl = (double)f2[fr]; break;
                            default: cl = (double)f2[nr]; break;
                            }
                            if (cl == 0.0) continue;
                            bool nmem = is_member(f, cg, fcomp, ccomp, ni, nj, nk);
                            bool same_block = (ni >> 1) == I && (nj >> 1) == J && (nk >> 1) == K;
                            if (!nmem) { ex += cl; continue; }  // P = 0 on the other end
                            if (same_block) continue;           // internal link
                            // member of another block: a coarse link (stored on + faces)
                            if (d == 0) e0 += cl;
                            else if (d == 2) e1 += cl;
                            else if (d == 4) e2 += cl;
                        }
                    }
        }
        ce[R] = (T)(own >= 0 ? ex : 1.0);
        c0[R] = (T)e0;
        c1[R] = (T)e1;
        c2[R] = (T)e2;
    }
}

// ---------------------------------------------------------------------------
// V-cycle kernels

// x_out = x + omega invd (b - M x), a damped-Jacobi sweep. With dotv, the per-block partial of
// (dotv, x_out) is stored (the (r, z) of the PCG).
// Cells that are not unknowns keep 0 in every level vector: the buffers are cleared when
// allocated and nothing writes them there, so the smoother skips them.
template <typename T>
__global__ void __launch_bounds__(kBlock) k_mg_smooth(int N, int JK, int K, const uint8_t* __restrict__ flags,
                                                      const T* __restrict__ e, const T* __restrict__ f0,
                                                      const T* __restrict__ f1, const T* __restrict__ f2,
                                                      const T* __restrict__ invd, const T* __restrict__ b,
                                                      const T* __restrict__ x, T* __restrict__ xo,
                                                      const T* __restrict__ dotv, const T* __restrict__ dotv2,
                                                      double* __restrict__ partials) {
    pdl_enter();
    T acc = (T)0, acc2 = (T)0;
    for (int r = blockIdx.x * blockDim.x + threadIdx.x; r < N; r += gridDim.x * blockDim.x) {
        if (!flags[r]) continue;
        const T xr = x[r], bv = b[r], iv = invd[r];
        const T res = bv - m_cell(r, JK, K, e, f0, f1, f2, xr, [=](int q) { return x[q]; });
        const T out = xr + (T)kOmega * iv * res;
        xo[r] = out;
        if (dotv) acc += dotv[r] * out;
        if (dotv2) acc2 += dotv2[r] * out;
    }
    if (dotv) {
        double a[2] = {widen(acc), widen(acc2)};
        block_sum_store<2>(a, partials);
    }
}

// The finest-level smoother on pairs of cells (FP32, K even, padded arrays; see
// m0_apply_pair): the same sweep as k_mg_smooth for kind-2 cells.
__global__ void __launch_bounds__(kBlock) k_mg_smooth0_pair(int N2, int JK2, int K2,
                                                            const int8_t* __restrict__ kind,
                                                            const float* __restrict__ e, const float* __restrict__ f0,
                                                            const float* __restrict__ f1, const float* __restrict__ f2,
                                                            const float* __restrict__ invd, const float* __restrict__ b,
                                                            const float* __restrict__ x, float* __restrict__ xo,
                                                            const float* __restrict__ dotv,
                                                            const float* __restrict__ dotv2,
                                                            double* __restrict__ partials) {
    pdl_enter();
    float acc = 0.f, acc2 = 0.f;
    for (int t = blockIdx.x * blockDim.x + threadIdx.x; t < N2; t += gridDim.x * blockDim.x) {
        const char2 kd = reinterpret_cast<const char2*>(kind)[t];
        const bool l0 = kd.x == 2, l1 = kd.y == 2;
        if (!l0 && !l1) continue;
        const float2 m = m0_apply_pair(t, JK2, K2, e, f0, f1, f2, x);
        const float2 xv = reinterpret_cast<const float2*>(x)[t];
        const float2 bv = reinterpret_cast<const float2*>(b)[t];
        const float2 iv = reinterpret_cast<const float2*>(invd)[t];
        const float o0 = xv.x + (float)kOmega * iv.x * (bv.x - m.x);
        const float o1 = xv.y + (float)kOmega * iv.y * (bv.y - m.y);
        if (l0) xo[2 * t] = o0;
        if (l1) xo[2 * t + 1] = o1;
        if (dotv) {
            if (l0) acc += dotv[2 * t] * o0;
            if (l1) acc += dotv[2 * t + 1] * o1;
        }
        if (dotv2) {
            if (l0) acc2 += dotv2[2 * t] * o0;
            if (l1) acc2 += dotv2[2 * t + 1] * o1;
        }
    }
    if (dotv) {
        double a[2] = {widen(acc), widen(acc2)};
        block_sum_store<2>(a, partials);
    }
}

// The two sweeps from zero that begin a cycle, in one pass: t = omega invd b is formed again at
// the neighbours instead of stored by a pass of its own (cells without an unknown hold b = 0).
// Finest level of 160x256x256: 45 us instead of 2 x 39.
template <typename T>
__global__ void __launch_bounds__(kBlock) k_mg_smooth_two(int N, int JK, int K, const uint8_t* __restrict__ flags,
                                                          const T* __restrict__ e, const T* __restrict__ f0,
                                                          const T* __restrict__ f1, const T* __restrict__ f2,
                                                          const T* __restrict__ invd, const T* __restrict__ b,
                                                          T* __restrict__ xo) {
    pdl_enter();
    for (int r = blockIdx.x * blockDim.x + threadIdx.x; r < N; r += gridDim.x * blockDim.x) {
        if (!flags[r]) continue;
        const T bv = b[r], iv = invd[r], xr = (T)kOmega * iv * bv;
        const T acc = m_cell(r, JK, K, e, f0, f1, f2, xr, [=](int q) { return (T)kOmega * invd[q] * b[q]; });
        xo[r] = xr + (T)kOmega * iv * (bv - acc);
    }
}

// In FP64 the values formed again cost more than the pass that they save (FP64 issue bounds these
// passes: cold FP64 solve of 338x338x283 219 ms, 188 with the three passes below and k_cg_dir), so
// there the first sweep, the correction and the second direction are passes of their own.
template <typename T>
constexpr bool form_again() { return sizeof(T) == 4; }

// t = omega invd b, the first sweep from zero
template <typename T>
__global__ void k_mg_first(int N, const uint8_t* __restrict__ flags, const T* __restrict__ invd,
                           const T* __restrict__ b, T* __restrict__ t) {
    pdl_enter();
    for (int r = blockIdx.x * blockDim.x + threadIdx.x; r < N; r += gridDim.x * blockDim.x)
        if (flags[r]) t[r] = (T)kOmega * invd[r] * b[r];
}

// x += scale * x_c(block) of the members
template <typename T>
__global__ void k_mg_correct(Grid g, Grid cg, const uint8_t* __restrict__ flags, const T* __restrict__ cx,
                             T* __restrict__ x, T scale) {
    pdl_enter();
    for (int r = blockIdx.x * blockDim.x + threadIdx.x; r < (int)g.N; r += gridDim.x * blockDim.x) {
        if (!(flags[r] & kCellMember)) continue;
        int i, j, k;
        decode(g, r, i, j, k);
        x[r] += scale * cx[(k >> 1) + cg.K * ((j >> 1) + cg.J * (i >> 1))];
    }
}

// pd1 = z - ((z, q0) / (pd0, q0)) pd0
template <typename T>
__global__ void k_kc_dir(int N, const uint8_t* __restrict__ flags, const double* __restrict__ s,
                         const T* __restrict__ z, const T* __restrict__ pd0, T* __restrict__ pd1) {
    pdl_enter();
    const T b = block_scalar<T>([=] { return (T)((s[0] > 0.0) ? -s[2] / s[0] : 0.0); });
    for (int r = blockIdx.x * blockDim.x + threadIdx.x; r < N; r += gridDim.x * blockDim.x)
        if (flags[r]) pd1[r] = z[r] + b * pd0[r];
}

// ... on pairs of cells of the finest level (FP32, K even, padded arrays)
__global__ void __launch_bounds__(kBlock) k_mg_smooth0_two_pair(int N2, int JK2, int K2,
                                                                const int8_t* __restrict__ kind,
                                                                const float* __restrict__ e,
                                                                const float* __restrict__ f0,
                                                                const float* __restrict__ f1,
                                                                const float* __restrict__ f2,
                                                                const float* __restrict__ invd,
                                                                const float* __restrict__ b, float* __restrict__ xo) {
    pdl_enter();
    const float om = (float)kOmega;
    auto two = [&](int t) {
        const float2 iv = reinterpret_cast<const float2*>(invd)[t], bv = reinterpret_cast<const float2*>(b)[t];
        return make_float2(om * iv.x * bv.x, om * iv.y * bv.y);
    };
    for (int t = blockIdx.x * blockDim.x + threadIdx.x; t < N2; t += gridDim.x * blockDim.x) {
        const char2 kd = reinterpret_cast<const char2*>(kind)[t];
        const bool l0 = kd.x == 2, l1 = kd.y == 2;
        if (!l0 && !l1) continue;
        const int r = 2 * t;
        const float2 iv = reinterpret_cast<const float2*>(invd)[t], bv = reinterpret_cast<const float2*>(b)[t];
        const float2 xc = make_float2(om * iv.x * bv.x, om * iv.y * bv.y);
        const float2 m = m0_pair(t, JK2, K2, e, f0, f1, f2, xc, two(t - JK2), two(t + JK2), two(t - K2), two(t + K2),
                                 om * invd[r - 1] * b[r - 1], om * invd[r + 2] * b[r + 2]);
        if (l0) xo[r] = xc.x + om * iv.x * (bv.x - m.x);
        if (l1) xo[r + 1] = xc.y + om * iv.y * (bv.y - m.y);
    }
}

// The prolongation and the sweep after it in one pass: x + scale * x_c(block) of the members is
// formed again at the neighbours instead of stored by a pass of its own.
// Piecewise-constant prolongation undershoots smooth error; scaling the coarse correction
// (over-correction) below the K-cycle levels roughly halves the PCG iterations on these
// pore-space operators (33 instead of 71 on a 96^3 porosity-0.25 field).
// All of its neighbours' flags and corrections are L1 hits: on the finest level of 160x256x256 57
// us instead of 25 + 39. A link out of the box reads a flag and a correction from the zero pads.
template <typename T>
__global__ void __launch_bounds__(kBlock, kPassBlocks) k_mg_smooth_corr(Grid g, Grid cg, const uint8_t* __restrict__ flags,
                                                           const T* __restrict__ e, const T* __restrict__ f0,
                                                           const T* __restrict__ f1, const T* __restrict__ f2,
                                                           const T* __restrict__ invd, const T* __restrict__ b,
                                                           const T* __restrict__ x, const T* __restrict__ cx, T scale,
                                                           T* __restrict__ xo) {
    pdl_enter();
    const int JK = (int)g.JK, K = g.K, CJK = (int)cg.JK, CK = cg.K;
    for (int r = blockIdx.x * blockDim.x + threadIdx.x; r < (int)g.N; r += gridDim.x * blockDim.x) {
        if (!flags[r]) continue;
        int i, j, k;
        decode(g, r, i, j, k);
        const int R = (k >> 1) + CK * ((j >> 1) + cg.J * (i >> 1));
        auto at = [=](int q, int Q) {
            const T v = x[q], w = v + scale * cx[Q];
            return flags[q] & kCellMember ? w : v;
        };
        const T xr = at(r, R), bv = b[r], iv = invd[r];
        const T er = e[r], l0m = f0[r - JK], l1m = f1[r - K], l2m = f2[r - 1], l2 = f2[r], l1 = f1[r], l0 = f0[r];
        const T xim = at(r - JK, i & 1 ? R : R - CJK), xip = at(r + JK, i & 1 ? R + CJK : R);
        const T xjm = at(r - K, j & 1 ? R : R - CK), xjp = at(r + K, j & 1 ? R + CK : R);
        const T xkm = at(r - 1, k & 1 ? R : R - 1), xkp = at(r + 1, k & 1 ? R + 1 : R);
        T acc = er * xr;
        acc += l0m * (xr - xim);
        acc += l1m * (xr - xjm);
        acc += l2m * (xr - xkm);
        acc += l2 * (xr - xkp);
        acc += l1 * (xr - xjp);
        acc += l0 * (xr - xip);
        xo[r] = xr + (T)kOmega * iv * (bv - acc);
    }
}

// ... on pairs of cells of the finest level (FP32, K even, padded arrays): the two cells of a pair
// and the pairs beside it over i and j each lie in one block.
__global__ void __launch_bounds__(kBlock, kPassBlocks) k_mg_smooth0_corr_pair(Grid g, Grid cg, FastDiv div_k2,
                                                                 const int8_t* __restrict__ kind,
                                                                 const uint8_t* __restrict__ flags,
                                                                 const float* __restrict__ e,
                                                                 const float* __restrict__ f0,
                                                                 const float* __restrict__ f1,
                                                                 const float* __restrict__ f2,
                                                                 const float* __restrict__ invd,
                                                                 const float* __restrict__ b,
                                                                 const float* __restrict__ x,
                                                                 const float* __restrict__ cx, float scale,
                                                                 float* __restrict__ xo) {
    pdl_enter();
    const int N2 = (int)(g.N / 2), K2 = g.K / 2, JK2 = (int)(g.JK / 2), CK = cg.K, CJK = (int)cg.JK;
    for (int t = blockIdx.x * blockDim.x + threadIdx.x; t < N2; t += gridDim.x * blockDim.x) {
        const char2 kd = reinterpret_cast<const char2*>(kind)[t];
        const bool l0 = kd.x == 2, l1 = kd.y == 2;
        if (!l0 && !l1) continue;
        const int r = 2 * t;
        const int row = (int)fdiv(div_k2, (unsigned int)t), kk = t - row * K2;
        const int i = (int)fdiv(g.div_jk, (unsigned int)r), j = row - i * g.J;
        const int R = kk + CK * ((j >> 1) + cg.J * (i >> 1));
        auto two = [=](int q, int Q) {
            const float2 v = reinterpret_cast<const float2*>(x)[q];
            const uchar2 m = reinterpret_cast<const uchar2*>(flags)[q];
            const float c = scale * cx[Q];
            return make_float2(m.x & kCellMember ? v.x + c : v.x, m.y & kCellMember ? v.y + c : v.y);
        };
        auto one = [=](int q, int Q) {
            const float v = x[q], c = scale * cx[Q];
            return flags[q] & kCellMember ? v + c : v;
        };
        const float2 xc = two(t, R);
        const float2 m = m0_pair(t, JK2, K2, e, f0, f1, f2, xc, two(t - JK2, i & 1 ? R : R - CJK),
                                 two(t + JK2, i & 1 ? R + CJK : R), two(t - K2, j & 1 ? R : R - CK),
                                 two(t + K2, j & 1 ? R + CK : R), one(r - 1, R - 1), one(r + 2, R + 1));
        const float2 iv = reinterpret_cast<const float2*>(invd)[t], bv = reinterpret_cast<const float2*>(b)[t];
        if (l0) xo[r] = xc.x + (float)kOmega * iv.x * (bv.x - m.x);
        if (l1) xo[r + 1] = xc.y + (float)kOmega * iv.y * (bv.y - m.y);
    }
}

// Coarse right-hand side of the finest level on pairs (FP32, K even, padded arrays): a thread
// forms the residuals of its block's four pairs and sums the members' in the child order of
// k_mg_restrict. The residuals stay in registers: 41 us instead of 38 for a
// residual pass and 28 for a gather at 160x256x256.
__global__ void __launch_bounds__(kBlock, kPassBlocks) k_mg_restrict0_pair(Grid g, Grid cg, const uint8_t* __restrict__ flags,
                                                              const float* __restrict__ e,
                                                              const float* __restrict__ f0,
                                                              const float* __restrict__ f1,
                                                              const float* __restrict__ f2,
                                                              const float* __restrict__ b,
                                                              const float* __restrict__ x, float* __restrict__ cb) {
    pdl_enter();
    const int K2 = g.K / 2, JK2 = (int)(g.JK / 2);
    for (int R = blockIdx.x * blockDim.x + threadIdx.x; R < (int)cg.N; R += gridDim.x * blockDim.x) {
        int I, J, K;
        decode(cg, R, I, J, K);
        float acc = 0.f;
#pragma unroll
        for (int a = 0; a < 2; ++a)
#pragma unroll
            for (int c = 0; c < 2; ++c) {
                const int i = 2 * I + a, j = 2 * J + c;
                if (i >= g.I || j >= g.J) continue;
                const int t = K + K2 * (j + g.J * i);
                const uchar2 fl = reinterpret_cast<const uchar2*>(flags)[t];
                const bool m0 = fl.x & kCellMember, m1 = fl.y & kCellMember;
                if (!m0 && !m1) continue;
                const float2 ax = m0_apply_pair(t, JK2, K2, e, f0, f1, f2, x);
                const float2 bv = reinterpret_cast<const float2*>(b)[t];
                if (m0) acc += bv.x - ax.x;
                if (m1) acc += bv.y - ax.y;
            }
        cb[R] = acc;
    }
}

// Coarse right-hand side: b_c(R) = sum over the owned members of (b - M x), the children in the
// order of their indices. Two threads per coarse cell, one for each k of its children, so that a
// warp reads its rows without gaps; the even one adds up both's residuals.
template <typename T>
__global__ void __launch_bounds__(kBlock, kPassBlocks) k_mg_restrict(Grid f, Grid cg, const uint8_t* __restrict__ flags,
                                                        const T* __restrict__ e, const T* __restrict__ f0,
                                                        const T* __restrict__ f1, const T* __restrict__ f2,
                                                        const T* __restrict__ fb, const T* __restrict__ fx,
                                                        T* __restrict__ cb) {
    pdl_enter();
    const int JK = (int)f.JK, K = f.K, n = 2 * (int)cg.N;
    for (int u = blockIdx.x * blockDim.x + threadIdx.x; u < (n + 31) / 32 * 32; u += gridDim.x * blockDim.x) {
        int I, J, KC;
        decode(cg, min(u, n - 1) >> 1, I, J, KC);
        const int k = 2 * KC + (u & 1);
        int at[4], m[4];
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            const int i = 2 * I + (q >> 1), j = 2 * J + (q & 1);
            const bool in = i < f.I && j < f.J && k < K;
            at[q] = (in ? k : 2 * KC) + K * ((in ? j : 2 * J) + f.J * (in ? i : 2 * I));
            m[q] = flags[at[q]] & (in ? kCellMember : 0);
        }
        T v[4] = {(T)0, (T)0, (T)0, (T)0};
        if (m[0] | m[1] | m[2] | m[3]) {
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                const T xr = fx[at[q]], bv = fb[at[q]];
                v[q] = bv - m_cell(at[q], JK, K, e, f0, f1, f2, xr, [=](int s) { return fx[s]; });
            }
        }
        T acc = (T)0;
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            const T w = __shfl_xor_sync(0xffffffffu, v[q], 1);
            const int mw = __shfl_xor_sync(0xffffffffu, m[q], 1);
            if (m[q]) acc += v[q];
            if (mw) acc += w;
        }
        if (!(u & 1) && u < n) cb[u >> 1] = acc;
    }
}

// ---------------------------------------------------------------------------
// K-cycle (Notay-Vassilevski): on the levels 1..kKLevels the coarse correction is two
// flexible-CG iterations on that level, preconditioned by the cycle from that level down,
// instead of one cycle. The scalars of each level's FCG live on the device (slots kKSlot0 +
// 5 (level - 1) + {pq0, prr0, zq0, pq1, prr1}), so no host synchronisation is needed.

// q = M pd and the partial dots (pd, q), (pd, rr). SECOND: the second direction,
// pd1 = z - ((z, q0) / (pd0, q0)) pd0, is formed here, and again at the neighbours, instead of by a
// pass of its own.
template <typename T, bool SECOND>
__global__ void __launch_bounds__(kBlock) k_kc_apply(int N, int JK, int K, const uint8_t* __restrict__ flags,
                                                     const double* __restrict__ s, const T* __restrict__ e,
                                                     const T* __restrict__ f0, const T* __restrict__ f1,
                                                     const T* __restrict__ f2, const T* __restrict__ z,
                                                     const T* __restrict__ pd0, const T* __restrict__ rr,
                                                     T* __restrict__ pd1, T* __restrict__ q,
                                                     double* __restrict__ partials) {
    pdl_enter();
    T b = (T)0;
    if (SECOND) b = block_scalar<T>([=] { return (T)((s[0] > 0.0) ? -s[2] / s[0] : 0.0); });
    auto dir = [=](int v) { return SECOND ? z[v] + b * pd0[v] : pd0[v]; };
    T a0 = (T)0, a1 = (T)0;
    for (int r = blockIdx.x * blockDim.x + threadIdx.x; r < N; r += gridDim.x * blockDim.x) {
        if (!flags[r]) continue;
        const T p = dir(r), rv = rr[r];
        const T qv = m_cell(r, JK, K, e, f0, f1, f2, p, dir);
        if (SECOND) pd1[r] = p;
        q[r] = qv;
        a0 += p * qv;
        a1 += p * rv;
    }
    double a[2] = {widen(a0), widen(a1)};
    block_sum_store<2>(a, partials);
}

// first iteration: e = alpha pd, rr -= alpha q with alpha = (pd, rr) / (pd, q)
template <typename T>
__global__ void k_kc_first(int N, const uint8_t* __restrict__ flags, const double* __restrict__ s,
                           const T* __restrict__ pd, const T* __restrict__ q, T* __restrict__ e,
                           T* __restrict__ rr) {
    pdl_enter();
    const T a = block_scalar<T>([=] { return (T)((s[0] > 0.0) ? s[1] / s[0] : 0.0); });
    for (int r = blockIdx.x * blockDim.x + threadIdx.x; r < N; r += gridDim.x * blockDim.x) {
        if (!flags[r]) continue;
        e[r] = a * pd[r];
        rr[r] -= a * q[r];
    }
}

// second iteration: e += alpha1 pd1, alpha1 = (pd1, rr) / (pd1, q1)
template <typename T>
__global__ void k_kc_second(int N, const uint8_t* __restrict__ flags, const double* __restrict__ s,
                            const T* __restrict__ pd1, T* __restrict__ e) {
    pdl_enter();
    const T a = block_scalar<T>([=] { return (T)((s[3] > 0.0) ? s[4] / s[3] : 0.0); });
    for (int r = blockIdx.x * blockDim.x + threadIdx.x; r < N; r += gridDim.x * blockDim.x)
        if (flags[r]) e[r] += a * pd1[r];
}

// coarsest level: a fixed number of damped Jacobi sweeps from zero by one CTA
template <typename T>
__device__ __forceinline__ void coarsest_block(const Grid& g, const int* __restrict__ comp, const T* __restrict__ e,
                                               const T* __restrict__ f0, const T* __restrict__ f1,
                                               const T* __restrict__ f2, const T* __restrict__ invd,
                                               const T* __restrict__ b, T* x, T* t, int sweeps) {
    for (long long r = threadIdx.x; r < g.N; r += blockDim.x)
        x[r] = (comp[r] >= 0) ? (T)kOmega * invd[r] * b[r] : (T)0;
    __syncthreads();
    for (int s = 1; s < sweeps; ++s) {
        for (long long r = threadIdx.x; r < g.N; r += blockDim.x) {
            T out = (T)0;
            if (comp[r] >= 0) {
                int i, j, k;
                decode(g, r, i, j, k);
                T res = b[r] - m_apply(g, r, i, j, k, e, f0, f1, f2, x);
                out = x[r] + (T)kOmega * invd[r] * res;
            }
            t[r] = out;
        }
        __syncthreads();
        for (long long r = threadIdx.x; r < g.N; r += blockDim.x) x[r] = t[r];
        __syncthreads();
    }
}

template <typename T>
__global__ void k_mg_coarsest(Grid g, const int* __restrict__ comp, const T* __restrict__ e,
                              const T* __restrict__ f0, const T* __restrict__ f1, const T* __restrict__ f2,
                              const T* __restrict__ invd, const T* __restrict__ b, T* x, T* t, int sweeps) {
    pdl_enter();
    coarsest_block(g, comp, e, f0, f1, f2, invd, b, x, t, sweeps);
}

// ---------------------------------------------------------------------------
// learned coarse solver: the network maps (member mask, anchoring fraction e/d, D^-1/2 b / s)
// on a D x H x W grid holding the level at its origin to D^1/2 x / (s kLpcOutScale), the
// Jacobi-scaled correction, s = max |D^-1/2 b| over the members. The unit-diagonal scaling
// makes the inputs and outputs independent of the level's coefficient magnitudes.

__device__ __forceinline__ bool lpc_cell(const Grid& g, int W, int H, long long v, long long& r) {
    const long long hw = (long long)W * H;
    const int z = (int)(v / hw);
    const long long rem = v - (long long)z * hw;
    const int y = (int)(rem / W), x = (int)(rem - (long long)y * W);
    if (z >= g.I || y >= g.J || x >= g.K) return false;
    r = lidx(g, z, y, x);
    return true;
}

// Components the network serves: those with a cell on the level whose excess is above
// kLpcAnchor of its diagonal (coupled to fixed values). Elsewhere the level is singular or
// nearly so; a correction there would excite near-null modes that only smoothing removes,
// so those cells keep the zero correction. anchored is indexed by component id (N bytes).
constexpr float kLpcAnchor = 1e-3f;

template <typename T>
__global__ void k_lpc_anchor(Grid g, const int* __restrict__ comp, const T* __restrict__ e,
                             const T* __restrict__ invd, uint8_t* __restrict__ anchored) {
    for (long long r = blockIdx.x * (long long)blockDim.x + threadIdx.x; r < g.N; r += (long long)gridDim.x * blockDim.x) {
        const int id = comp[r];
        if (id >= 0 && (float)e[r] * (float)invd[r] > kLpcAnchor) anchored[id] = 1;
    }
}

// the fixed inputs of a hierarchy: mask, anchoring fraction e/d (the share of the diagonal
// that couples to fixed values) and 1/sqrt(d) of the cells of anchored components (0 marks
// the cells the network does not serve)
template <typename T>
__global__ void k_lpc_setup(Grid g, int D, int H, int W, const int* __restrict__ comp, const T* __restrict__ e,
                            const T* __restrict__ invd, const uint8_t* __restrict__ anchored,
                            float* __restrict__ c0, float* __restrict__ c1, float* __restrict__ isd) {
    const long long n = (long long)D * H * W;
    for (long long v = blockIdx.x * (long long)blockDim.x + threadIdx.x; v < n; v += (long long)gridDim.x * blockDim.x) {
        long long r = 0;
        float m = 0.f, a = 0.f;
        if (lpc_cell(g, W, H, v, r)) {
            float q = 0.f;
            if (comp[r] >= 0 && anchored[comp[r]]) {
                m = 1.f;
                a = (float)e[r] * (float)invd[r];
                q = sqrtf((float)invd[r]);
            }
            isd[r] = q;
        }
        c0[v] = m;
        c1[v] = a;
    }
}

// s = max |b| / sqrt(d) over the served cells (one block; NaN entries are passed over here and
// reach the network through k_lpc_pack, whose output then carries them to the caller)
__global__ void __launch_bounds__(1024) k_lpc_scale(Grid g, const int* __restrict__ comp, const float* __restrict__ b,
                                                    const float* __restrict__ isd, double* __restrict__ out) {
    float m = 0.f;
    for (long long r = threadIdx.x; r < g.N; r += blockDim.x)
        if (comp[r] >= 0) m = fmaxf(m, fabsf(b[r] * isd[r]));
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, o));
    __shared__ float sh[32];
    if ((threadIdx.x & 31) == 0) sh[threadIdx.x >> 5] = m;
    __syncthreads();
    if (threadIdx.x < 32) {
        m = (threadIdx.x < (blockDim.x >> 5)) ? sh[threadIdx.x] : 0.f;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, o));
        if (threadIdx.x == 0) *out = (double)m;
    }
}

__global__ void k_lpc_pack(Grid g, int D, int H, int W, const int* __restrict__ comp, const float* __restrict__ b,
                           const float* __restrict__ isd, const double* __restrict__ s, float* __restrict__ c2) {
    const float inv = (*s > 0.0) ? (float)(1.0 / *s) : 0.f;
    const long long n = (long long)D * H * W;
    for (long long v = blockIdx.x * (long long)blockDim.x + threadIdx.x; v < n; v += (long long)gridDim.x * blockDim.x) {
        long long r = 0;
        float val = 0.f;
        if (lpc_cell(g, W, H, v, r) && comp[r] >= 0) val = b[r] * isd[r] * inv;  // isd 0: not served
        c2[v] = val;
    }
}

// x = s kLpcOutScale D^-1/2 y on the served cells, 0 on the other members (non-members keep
// their 0)
__global__ void k_lpc_unpack(Grid g, int H, int W, const int* __restrict__ comp, const float* __restrict__ y,
                             const float* __restrict__ isd, const double* __restrict__ s, float* __restrict__ x) {
    const float sc = (float)(*s) * kLpcOutScale;
    for (long long r = blockIdx.x * (long long)blockDim.x + threadIdx.x; r < g.N; r += (long long)gridDim.x * blockDim.x) {
        if (comp[r] < 0) continue;
        if (isd[r] == 0.f) {
            x[r] = 0.f;
            continue;
        }
        const int i = (int)(r / g.JK);
        const long long rem = r - (long long)i * g.JK;
        const int j = (int)(rem / g.K), k = (int)(rem - (long long)j * g.K);
        x[r] = sc * isd[r] * y[((long long)i * H + j) * W + k];
    }
}

ls_status lpnet_forward_on(ls_lpnet* n, cudaStream_t s, const float* c0, const float* c1, const float* c2,
                           float* out, std::string* err);

static int round8(int v) { return ((v + 7) / 8) * 8; }

void mg_graphs_clear(ls_ctx* c);

// Build (or reuse) the network for the learned level of the current hierarchy and its fixed
// inputs. Without weights the learned solver is an argument error; a hierarchy too shallow
// to have the level leaves the plain cycle in use.
static ls_status lpc_prepare(ls_ctx* c) {
    c->lpc_ready = 0;
    if (c->p.press_solver != LS_PRESS_LEARNED) return LS_OK;
    if (c->lpc_params.empty())
        return set_error(c, LS_BAD_ARG, "learned pressure solver: no weights (ls_pressure_set_precond_weights)");
    if (c->mg.size() < (size_t)kLearnedLevel) return LS_OK;
    const auto& lv = c->mg[kLearnedLevel - 1];
    const Grid lg = lv.g;
    const int dims[3] = {round8(lg.I), round8(lg.J), round8(lg.K)};
    if (!c->lpc || dims[0] != c->lpc_dims[0] || dims[1] != c->lpc_dims[1] || dims[2] != c->lpc_dims[2]) {
        mg_graphs_clear(c);  // captured cycles name the old network's buffers
        if (c->lpc) {
            ls_lpnet_destroy(c->lpc);
            c->lpc = nullptr;
        }
        const size_t old_nn = (size_t)c->lpc_dims[0] * c->lpc_dims[1] * c->lpc_dims[2];
        dfree_t(c, &c->lpc_c0, old_nn);
        dfree_t(c, &c->lpc_c1, old_nn);
        dfree_t(c, &c->lpc_c2, old_nn);
        dfree_t(c, &c->lpc_out, old_nn);
        dfree_t(c, &c->lpc_isd, (size_t)c->lpc_isd_n);
        ls_lpnet* n = nullptr;
        ls_status st = ls_lpnet_create(dims[0], dims[1], dims[2], 0, &n);
        if (st != LS_OK) return set_error(c, st, "learned pressure solver: network creation failed");
        c->lpc = n;
        if (ls_lpnet_param_count(n) != (long long)c->lpc_params.size())
            return set_error(c, LS_BAD_ARG, "learned pressure solver: weight count does not match the network");
        st = ls_lpnet_set_params(n, c->lpc_params.data(), (long long)c->lpc_params.size());
        if (st != LS_OK) return set_error(c, st, "learned pressure solver: loading the weights failed");
        const size_t nn = (size_t)dims[0] * dims[1] * dims[2];
        LS_TRY(dalloc_t(c, &c->lpc_c0, nn));
        LS_TRY(dalloc_t(c, &c->lpc_c1, nn));
        LS_TRY(dalloc_t(c, &c->lpc_c2, nn));
        LS_TRY(dalloc_t(c, &c->lpc_out, nn));
        LS_TRY(dalloc_t(c, &c->lpc_isd, (size_t)lg.N));
        c->lpc_isd_n = lg.N;
        for (int q = 0; q < 3; ++q) c->lpc_dims[q] = dims[q];
    }
    if (!c->lpc_anchor) LS_TRY(dalloc_t(c, &c->lpc_anchor, (size_t)c->g.N));
    LS_CUDA(c, cudaMemsetAsync(c->lpc_anchor, 0, (size_t)c->g.N, c->stream));
    LS_LAUNCH(c, k_lpc_anchor<float>, grid_for(c, lg.N), kBlock, 0, lg, (const int*)lv.comp, (const float*)lv.e,
              (const float*)lv.invd, c->lpc_anchor);
    const long long nn = (long long)dims[0] * dims[1] * dims[2];
    LS_LAUNCH(c, k_lpc_setup<float>, grid_for(c, nn), kBlock, 0, lg, dims[0], dims[1], dims[2],
              (const int*)lv.comp, (const float*)lv.e, (const float*)lv.invd, (const uint8_t*)c->lpc_anchor,
              c->lpc_c0, c->lpc_c1, c->lpc_isd);
    c->lpc_ready = 1;
    return LS_OK;
}

// x = the network's approximation of M_l^-1 b on the learned level
static ls_status lpc_solve(ls_ctx* c, const Grid& lg, const int* comp, const float* b, float* x) {
    const int* d = c->lpc_dims;
    const long long nn = (long long)d[0] * d[1] * d[2];
    LS_LAUNCH(c, k_lpc_scale, 1, 1024, 0, lg, comp, b, (const float*)c->lpc_isd, c->scal + kLpcSlot);
    LS_LAUNCH(c, k_lpc_pack, grid_for(c, nn), kBlock, 0, lg, d[0], d[1], d[2], comp, b, (const float*)c->lpc_isd,
              (const double*)(c->scal + kLpcSlot), c->lpc_c2);
    std::string err;
    const ls_status st = lpnet_forward_on(c->lpc, c->stream, c->lpc_c0, c->lpc_c1, c->lpc_c2, c->lpc_out, &err);
    if (st != LS_OK) return set_error(c, st, "learned coarse solve: " + err);
    c->launches += 16;  // the network's own launches: input pack, 8 convolutions, 3 poolings, 3 upsamplings, output
    LS_LAUNCH(c, k_lpc_unpack, grid_for(c, lg.N), kBlock, 0, lg, d[1], d[2], comp, (const float*)c->lpc_out,
              (const float*)c->lpc_isd, (const double*)(c->scal + kLpcSlot), x);
    return LS_OK;
}

// ---------------------------------------------------------------------------

static Grid coarse_of(const Grid& f) {
    Grid c;
    c.I = (f.I + 1) / 2;
    c.J = (f.J + 1) / 2;
    c.K = (f.K + 1) / 2;
    c.JK = (long long)c.J * c.K;
    c.N = (long long)c.I * c.JK;
    c.NP = c.N;
    grid_init_div(c);
    return c;
}

void mg_graphs_clear(ls_ctx* c) {
    for (auto& gr : c->mg_graphs)
        if (gr.exec) cudaGraphExecDestroy(gr.exec);
    c->mg_graphs.clear();
}

static ls_status level_alloc(ls_ctx* c, const Grid& g, size_t esize, void** out) {
    const size_t pad = level_pad(g), bytes = esize * ((size_t)g.N + 2 * pad);
    void* base = nullptr;
    LS_TRY(walloc(c, &base, bytes));
    *out = (char*)base + esize * pad;
    LS_CUDA(c, cudaMemsetAsync(base, 0, bytes, c->stream));
    return LS_OK;
}

static void level_free(ls_ctx* c, const Grid& g, size_t esize, void** p) {
    if (!*p) return;
    const size_t pad = level_pad(g);
    void* base = (char*)*p - esize * pad;
    dfree(c, &base, esize * ((size_t)g.N + 2 * pad));
    *p = nullptr;
}

void mg_free(ls_ctx* c) {
    mg_graphs_clear(c);
    for (size_t m = 0; m < c->mg.size(); ++m) {
        auto& lv = c->mg[m];
        dfree_t(c, &lv.comp, (size_t)lv.g.N);
        level_free(c, lv.g, 1, (void**)&lv.flags);
        void** lp[] = {&lv.e, &lv.face[0], &lv.face[1], &lv.face[2], &lv.invd, &lv.x, &lv.b, &lv.t};
        for (void** q : lp) level_free(c, lv.g, (size_t)lv.esize, q);
        for (void*& q : lv.kv) level_free(c, lv.g, (size_t)lv.esize, &q);
    }
    c->mg.clear();
    level_free(c, c->g, 1, (void**)&c->mg0_flags);
    l0_free(c, 10, &c->mg0_p);
    l0_free(c, 11, &c->mg0_t);
    c->mg_is64 = -1;
}

// Coarse levels of at most this many cells are run by k_mg_fused (LS_MG_TAIL_CELLS overrides it,
// 0: a kernel per step).
template <typename T>
static long long fuse_cells(const ls_ctx* c) {
    const long long cap = (long long)c->num_sms * 8 * kBlock;  // one cell per thread of a level kernel
    const long long want = c->mg_tail_cells >= 0 ? c->mg_tail_cells : sizeof(T) == 4 ? kFuseCells32 : kFuseCells64;
    return std::min(want, cap);
}

constexpr size_t kFuseSmem = 227 * 1024;

// Slabs and shared memory of the levels in fa; false when a slab would be thinner than a plane
// (its halo would reach past the neighbouring slabs) or the levels do not fit.
template <typename T>
static bool fuse_plan(FuseArgs<T>& fa, int blocks, size_t* smem) {
    const bool f64 = sizeof(T) == 8;
    size_t at = 0;
    fa.nc = 0;
    for (int q = 0; q < fa.n; ++q)
        if (f64 || fa.lv[q].g.N > kBlockCells) fa.nc = q + 1;
    for (int q = 0; q < fa.n; ++q) {
        FLevel<T>& L = fa.lv[q];
        const long long N = L.g.N, JK = L.g.JK;
        L.blk = q >= fa.nc;
        const long long share = L.blk ? N : (N + blocks - 1) / blocks;
        L.per = (int)((share + 255) / 256 * 256);
        L.div_per = make_fastdiv((unsigned int)L.per);
        auto take = [&](long long n) {
            const int o = (int)at;
            at += (size_t)n;
            return o;
        };
        L.oM = (int)(at * sizeof(T));
        if (q > 0) take((L.per + (long long)sizeof(T) - 1) / (long long)sizeof(T));
        if (!(f64 && q + 1 == fa.n)) {  // (the coarsest FP64 iterate has its own place)
            if (!L.blk && JK > L.per) return false;
            L.oE = take(L.per);
            L.oW = take(L.per);
            L.oF0 = take(L.per + JK);
            L.oF1 = take(L.per + L.g.K);
            L.oF2 = take(L.per + 1);
            L.oX = take(L.per + 2 * JK);
            L.oT = take(L.per + 2 * JK);
            L.oB = take(L.per);
            if (q < fa.nk) {
                L.oZ = take(L.per);
                L.oQ = take(L.per);
                L.oV = take(L.per);
            }
        }
        if (at * sizeof(T) > kFuseSmem) return false;
    }
    int widest = 0;
    for (int q = 0; q < fa.nk; ++q) widest = std::max(widest, fa.lv[q].per);
    fa.oP = (int)at;
    at += (size_t)widest;
    *smem = fuse_fixed<T>() + sizeof(T) * at;
    return *smem <= kFuseSmem;
}

static void fuse_config(cudaLaunchConfig_t& cfg, cudaLaunchAttribute (&at)[2], int blocks, size_t smem, int pdl) {
    cfg.gridDim = dim3(blocks);
    cfg.blockDim = dim3(kFuseThreads);
    cfg.dynamicSmemBytes = smem;
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim = {(unsigned)blocks, 1, 1};
    at[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[1].val.programmaticStreamSerializationAllowed = pdl ? 1 : 0;
    cfg.attrs = at;
    cfg.numAttrs = 2;
}

template <typename T>
static ls_status fuse_launch(ls_ctx* c, const FuseArgs<T>& fa, size_t smem) {
    cudaLaunchConfig_t cfg = {};
    cudaLaunchAttribute at[2];
    fuse_config(cfg, at, fa.nc > 0 ? c->mg_cluster : 1, smem, c->pdl);
    cfg.stream = c->stream;
    cudaError_t e = cudaLaunchKernelEx(&cfg, k_mg_fused<T>, fa);
    c->launches++;
    if (e == cudaSuccess) e = cudaGetLastError();
    return e == cudaSuccess ? LS_OK : check_cuda(c, e, "k_mg_fused");
}

// The cluster of k_mg_fused: 16 blocks where the device can hold such a cluster (and max_blocks
// allows it), else 8, else none (0: the level kernels).
template <typename T>
static int fuse_cluster(int max_blocks) {
    if (cudaFuncSetAttribute(k_mg_fused<T>, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) != cudaSuccess ||
        cudaFuncSetAttribute(k_mg_fused<T>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kFuseSmem) != cudaSuccess) {
        cudaGetLastError();
        return 0;
    }
    for (int blocks = 16; blocks >= 8; blocks /= 2) {
        if (blocks > max_blocks) continue;
        cudaLaunchConfig_t cfg = {};
        cudaLaunchAttribute at[2];
        fuse_config(cfg, at, blocks, kFuseSmem, 0);
        int n = 0;
        if (cudaOccupancyMaxActiveClusters(&n, k_mg_fused<T>, &cfg) == cudaSuccess && n > 0) return blocks;
        cudaGetLastError();
    }
    return 0;
}

template <typename T>
static ls_status mg_alloc(ls_ctx* c) {
    const int is64 = sizeof(T) == 8;
    if (c->mg_is64 == is64) return LS_OK;
    mg_free(c);
    c->mg_cluster = fuse_cluster<T>(c->mg_cluster_max);
    if (!c->comp) LS_TRY(walloc_t(c, &c->comp, (size_t)c->g.N));
    if (!c->cc_flag) LS_TRY(dalloc_t(c, &c->cc_flag, (size_t)4));
    LS_TRY(level_alloc(c, c->g, 1, (void**)&c->mg0_flags));
    if (form_again<T>()) LS_TRY(l0_alloc(c, 10, sizeof(T), &c->mg0_p));
    LS_TRY(l0_alloc(c, 11, sizeof(T), &c->mg0_t));
    Grid g = c->g;
    g.NP = g.N;
    while ((c->mg.empty() || g.N > kCoarsestCells) && (g.I > 1 || g.J > 1 || g.K > 1)) {
        Grid cg = coarse_of(g);
        c->mg.push_back({});
        ls_ctx::MGLevel& lv = c->mg.back();
        lv.g = cg;
        lv.esize = (int)sizeof(T);
        LS_TRY(walloc_t(c, &lv.comp, (size_t)cg.N));
        LS_TRY(level_alloc(c, cg, 1, (void**)&lv.flags));
        void** arrs[] = {&lv.e, &lv.face[0], &lv.face[1], &lv.face[2], &lv.invd, &lv.x, &lv.b, &lv.t};
        for (void** q : arrs) LS_TRY(level_alloc(c, cg, sizeof(T), q));
        g = cg;
    }
    // K-cycle vectors on the levels 1..kKLevels that have a coarser level below them
    for (size_t m = 1; m <= (size_t)kKLevels && m < c->mg.size(); ++m) {
        auto& lv = c->mg[m - 1];
        for (void*& q : lv.kv) LS_TRY(level_alloc(c, lv.g, sizeof(T), &q));
    }
    c->mg_is64 = is64;
    return LS_OK;
}

// 1/diagonal of the finest inner operator (rows of kind 2 live)
template <typename T>
ls_status inner_invd(ls_ctx* c) {
    LS_LAUNCH(c, k_level_invd<T>, grid_for(c, c->g.N), kBlock, 0, c->g, (const int*)nullptr,
              (const int8_t*)c->pkind, (const T*)c->ie, (const T*)c->iface[0], (const T*)c->iface[1],
              (const T*)c->iface[2], (T*)c->iinvd);
    return LS_OK;
}

// Components and coarse operators for the current fine inner operator (c->ie, c->iface,
// c->iinvd, precision T).
template <typename T>
ls_status mg_setup(ls_ctx* c) {
    LS_TRY(mg_alloc<T>(c));
    const Grid g = c->g;
    const int grid = grid_for(c, g.N);
    LS_CUDA(c, cudaMemsetAsync(c->cc_flag, 0, sizeof(int), c->stream));
    LS_LAUNCH(c, k_cc_init<T>, grid, kBlock, 0, g, (const int8_t*)c->pkind, (const T*)c->iface[2],
              (const T*)c->iinvd, c->comp);
    LS_LAUNCH(c, k_cc_hook<T>, grid, kBlock, 0, g, (const T*)c->iface[0], (const T*)c->iface[1],
              (const T*)c->iface[2], (const T*)c->iinvd, c->comp, c->cc_flag);
    LS_LAUNCH(c, k_cc_compress, grid, kBlock, 0, g, c->comp);
    Grid fg = g;
    const int* fcomp = c->comp;
    const T* fe = (const T*)c->ie;
    const T* ff[3] = {(const T*)c->iface[0], (const T*)c->iface[1], (const T*)c->iface[2]};
    for (size_t l = 0; l < c->mg.size(); ++l) {
        auto& cl = c->mg[l];
        const int cgd = grid_for(c, cl.g.N);
        LS_LAUNCH(c, k_mg_dom, cgd, kBlock, 0, fg, cl.g, fcomp, cl.comp);
        LS_LAUNCH(c, k_mg_flags, grid_for(c, fg.N), kBlock, 0, fg, cl.g, fcomp, (const int*)cl.comp,
                  l == 0 ? c->mg0_flags : c->mg[l - 1].flags);
        LS_LAUNCH(c, k_mg_coarse_op<T>, cgd, kBlock, 0, fg, cl.g, fcomp, (const int*)cl.comp, fe, ff[0], ff[1],
                  ff[2], (T*)cl.e, (T*)cl.face[0], (T*)cl.face[1], (T*)cl.face[2]);
        LS_LAUNCH(c, k_level_invd<T>, cgd, kBlock, 0, cl.g, (const int*)cl.comp, (const int8_t*)nullptr,
                  (const T*)cl.e, (const T*)cl.face[0], (const T*)cl.face[1], (const T*)cl.face[2],
                  (T*)cl.invd);
        fg = cl.g;
        fcomp = cl.comp;
        fe = (const T*)cl.e;
        ff[0] = (const T*)cl.face[0];
        ff[1] = (const T*)cl.face[1];
        ff[2] = (const T*)cl.face[2];
    }
    int flag = 0;
    LS_CUDA(c, cudaMemcpyAsync(&flag, c->cc_flag, sizeof(int), cudaMemcpyDeviceToHost, c->stream));
    LS_CUDA(c, cudaStreamSynchronize(c->stream));
    if (flag) return set_error(c, LS_TIMEOUT, "multigrid: component labelling gave up");
    if (std::is_same<T, float>::value) return lpc_prepare(c);
    c->lpc_ready = 0;
    return LS_OK;
}

// Zero every level vector (the smoother and the PCG skip non-member cells, which must hold 0).
template <typename T>
ls_status mg_clear(ls_ctx* c) {
    if (c->mg0_p) LS_CUDA(c, cudaMemsetAsync(c->mg0_p, 0, sizeof(T) * (size_t)c->g.N, c->stream));
    LS_CUDA(c, cudaMemsetAsync(c->mg0_t, 0, sizeof(T) * (size_t)c->g.N, c->stream));
    for (auto& lv : c->mg) {
        const size_t b = sizeof(T) * (size_t)lv.g.N;
        LS_CUDA(c, cudaMemsetAsync(lv.x, 0, b, c->stream));
        LS_CUDA(c, cudaMemsetAsync(lv.b, 0, b, c->stream));
        LS_CUDA(c, cudaMemsetAsync(lv.t, 0, b, c->stream));
        for (void* q : lv.kv)
            if (q) LS_CUDA(c, cudaMemsetAsync(q, 0, b, c->stream));
    }
    return LS_OK;
}

// z = B r: one K-cycle (levels 1..kKLevels take the two-iteration FCG coarse correction,
// deeper levels a plain V-cycle). The per-block partials of (r, z) and (dotv2, z) are left in
// c->partials (two values per block, dotv2 may be null) and their count in *nblocks_out.
template <typename T>
ls_status mg_apply(ls_ctx* c, const T* r, T* z, const T* dotv2, int* nblocks_out) {
    const size_t L = c->mg.size();  // coarse levels
    if (L == 0) return set_error(c, LS_BAD_ARG, "multigrid hierarchy missing");
    struct Lv {
        Grid g;
        const int* comp;
        const uint8_t* flags;
        const T *e, *f0, *f1, *f2, *invd;
        T *x, *b, *t;
        T* kv[6];
    };
    std::vector<Lv> lv(L + 1);
    lv[0] = {c->g, c->comp, c->mg0_flags, (const T*)c->ie, (const T*)c->iface[0], (const T*)c->iface[1], (const T*)c->iface[2],
             (const T*)c->iinvd, z, nullptr, (T*)c->mg0_t, {}};
    for (size_t l = 0; l < L; ++l) {
        auto& m = c->mg[l];
        lv[l + 1] = {m.g, m.comp, m.flags, (const T*)m.e, (const T*)m.face[0], (const T*)m.face[1], (const T*)m.face[2],
                     (const T*)m.invd, (T*)m.x, (T*)m.b, (T*)m.t, {}};
        for (int q = 0; q < 6; ++q) lv[l + 1].kv[q] = (T*)m.kv[q];
    }
    // one damped-Jacobi sweep on level l (paired finest-level kernel for FP32 and even K)
    const bool pair0 = std::is_same<T, float>::value && (c->g.K % 2 == 0);
    const bool learned = std::is_same<T, float>::value && c->lpc_active && c->lpc_ready && L >= (size_t)kLearnedLevel;
    auto smooth = [&](size_t l, const T* b, const T* x, T* xo, const T* dv, const T* dv2, int* nb) -> ls_status {
        Lv& a = lv[l];
        double* partials = dv ? c->partials : (double*)nullptr;
        if (l == 0 && pair0) {
            const int N2 = (int)(a.g.N / 2);
            const int gd = grid_for(c, N2);
            LS_LAUNCH_PDL(c, k_mg_smooth0_pair, gd, kBlock, 0, N2, (int)(a.g.JK / 2), a.g.K / 2,
                      (const int8_t*)c->pkind, (const float*)a.e, (const float*)a.f0, (const float*)a.f1,
                      (const float*)a.f2, (const float*)a.invd, (const float*)b, (const float*)x, (float*)xo,
                      (const float*)dv, (const float*)dv2, partials);
            if (nb) *nb = gd;
            return LS_OK;
        }
        const int gd = grid_for(c, a.g.N);
        LS_LAUNCH_PDL(c, k_mg_smooth<T>, gd, kBlock, 0, (int)a.g.N, (int)a.g.JK, a.g.K, a.flags, a.e, a.f0, a.f1, a.f2,
                  a.invd, b, x, xo, dv, dv2, partials);
        if (nb) *nb = gd;
        return LS_OK;
    };
    // cycle(l, b, out): out = B_l b; with dv non-null the final sweep leaves the partial dots
    // (dv, out), (dv2, out) and their block count in *nb. Level l's x and t are its scratch.
    std::function<ls_status(size_t, const T*, T*, const T*, const T*, int*)> cycle;
    // kfcg(m): two FCG iterations on level m for M_m e = b_m (m's b, left as the residual of the
    // first), result in kv[5]
    auto kfcg = [&](size_t m) -> ls_status {
        Lv& a = lv[m];
        T *rr = a.b, *za = a.kv[0], *zb = a.kv[1], *pd = a.kv[2], *q0 = a.kv[3], *q1 = a.kv[4], *e = a.kv[5];
        const int slot = kKSlot0 + 5 * ((int)m - 1);
        const double* s = c->scal + slot;
        const int gd = grid_for(c, a.g.N), N = (int)a.g.N, JK = (int)a.g.JK, K = a.g.K;
        LS_TRY(cycle(m, (const T*)rr, za, nullptr, nullptr, nullptr));
        LS_LAUNCH_PDL(c, (k_kc_apply<T, false>), gd, kBlock, 0, N, JK, K, a.flags, s, a.e, a.f0, a.f1, a.f2,
                  (const T*)nullptr, (const T*)za, (const T*)rr, (T*)nullptr, q0, c->partials);
        LS_TRY(finalize_sum(c, gd, 2, slot));  // (za, q0), (za, rr)
        LS_LAUNCH_PDL(c, k_kc_first<T>, gd, kBlock, 0, N, a.flags, s, (const T*)za, (const T*)q0, e, rr);
        int nb = 0;
        LS_TRY(cycle(m, (const T*)rr, zb, (const T*)q0, nullptr, &nb));
        LS_TRY(finalize_sum(c, nb, 2, slot + 2));  // (zb, q0)
        if (form_again<T>()) {
            LS_LAUNCH_PDL(c, (k_kc_apply<T, true>), gd, kBlock, 0, N, JK, K, a.flags, s, a.e, a.f0, a.f1, a.f2,
                      (const T*)zb, (const T*)za, (const T*)rr, pd, q1, c->partials);
        } else {
            LS_LAUNCH_PDL(c, k_kc_dir<T>, gd, kBlock, 0, N, a.flags, s, (const T*)zb, (const T*)za, pd);
            LS_LAUNCH_PDL(c, (k_kc_apply<T, false>), gd, kBlock, 0, N, JK, K, a.flags, s, a.e, a.f0, a.f1, a.f2,
                      (const T*)nullptr, (const T*)pd, (const T*)rr, (T*)nullptr, q1, c->partials);
        }
        LS_TRY(finalize_sum(c, gd, 2, slot + 3));  // (pd, q1), (pd, rr)
        LS_LAUNCH_PDL(c, k_kc_second<T>, gd, kBlock, 0, N, a.flags, s, (const T*)pd, e);
        return LS_OK;
    };
    // the levels from `fuse` down run as one launch each time they are visited (k_mg_fused)
    size_t fuse = L + 1, fuse_smem = 0;
    FuseArgs<T> fa = {};
    const bool small64 = sizeof(T) == 8 && c->mg_tail_cells < 0 && lv[L].g.N <= kFuseCoarsest64;
    if (!learned && !small64 && c->mg_cluster > 0) {
        for (size_t l = L >= (size_t)kMaxFuse ? L + 1 - kMaxFuse : 1; l <= L && fuse > L; ++l) {
            if (lv[l].g.N > fuse_cells<T>(c)) continue;
            fa = {};
            fa.n = (int)(L - l + 1);
            fa.sweeps = kCoarseSweeps;
            fa.scale = (T)kProlongScale;
            fa.partials = c->partials;
            for (int q = 0; q < fa.n; ++q) {
                const Lv& a = lv[l + q];
                FLevel<T>& f = fa.lv[q];
                f.g = a.g;
                f.comp = a.comp;
                f.e = a.e;
                f.f0 = a.f0;
                f.f1 = a.f1;
                f.f2 = a.f2;
                f.invd = a.invd;
                f.x = a.x;
                f.b = a.b;
                f.ev = a.kv[5];
                if (l + q <= (size_t)kKLevels && l + q < L) fa.nk = q + 1;
            }
            if (fuse_plan(fa, c->mg_cluster, &fuse_smem)) fuse = l;
        }
    }
    cycle = [&](size_t l, const T* b, T* out, const T* dv, const T* dv2, int* nb) -> ls_status {
        Lv& a = lv[l];
        if (l == L) {
            LS_LAUNCH_PDL(c, k_mg_coarsest<T>, 1, 1024, 0, a.g, a.comp, a.e, a.f0, a.f1, a.f2, a.invd, b, out, a.t,
                      kCoarseSweeps);
            return LS_OK;
        }
        Lv& cl = lv[l + 1];
        const int gd = grid_for(c, a.g.N);
        const int N2 = (int)(a.g.N / 2), JK2 = (int)(a.g.JK / 2), K2 = a.g.K / 2;
        if (l == 0 && pair0) {
            LS_LAUNCH_PDL(c, k_mg_smooth0_two_pair, grid_for(c, N2), kBlock, 0, N2, JK2, K2,
                      (const int8_t*)c->pkind, (const float*)a.e,
                      (const float*)a.f0, (const float*)a.f1, (const float*)a.f2, (const float*)a.invd,
                      (const float*)b, (float*)a.x);
            LS_LAUNCH_PDL(c, k_mg_restrict0_pair, pass_grid(c, cl.g.N), kBlock, 0, a.g, cl.g, a.flags, (const float*)a.e,
                      (const float*)a.f0, (const float*)a.f1, (const float*)a.f2, (const float*)b, (const float*)a.x,
                      (float*)cl.b);
        } else {
            if (form_again<T>()) {
                LS_LAUNCH_PDL(c, k_mg_smooth_two<T>, gd, kBlock, 0, (int)a.g.N, (int)a.g.JK, a.g.K, a.flags, a.e, a.f0,
                          a.f1, a.f2, a.invd, b, a.x);
            } else {
                LS_LAUNCH_PDL(c, k_mg_first<T>, gd, kBlock, 0, (int)a.g.N, a.flags, a.invd, b, a.t);
                LS_TRY(smooth(l, b, (const T*)a.t, a.x, nullptr, nullptr, nullptr));
            }
            LS_LAUNCH_PDL(c, k_mg_restrict<T>, pass_grid(c, 2 * cl.g.N), kBlock, 0, a.g, cl.g, a.flags, a.e, a.f0, a.f1,
                      a.f2, b, (const T*)a.x, cl.b);
        }
        const T* corr;
        T scale;
        if (l + 1 >= fuse) {
            LS_TRY(fuse_launch<T>(c, fa, fuse_smem));
            const bool kc = l + 1 <= (size_t)kKLevels && l + 1 < L;
            corr = kc ? cl.kv[5] : cl.x;
            scale = kc ? (T)1 : (T)kProlongScale;
        } else if (l + 1 <= (size_t)kKLevels && l + 1 < L) {
            LS_TRY(kfcg(l + 1));
            corr = cl.kv[5];
            scale = (T)1;  // the FCG steps carry the optimal scaling
        } else if (learned && l + 1 == (size_t)kLearnedLevel) {
            LS_TRY(lpc_solve(c, cl.g, cl.comp, (const float*)cl.b, (float*)cl.x));
            corr = cl.x;
            scale = (T)1;
        } else {
            LS_TRY(cycle(l + 1, (const T*)cl.b, cl.x, nullptr, nullptr, nullptr));
            corr = cl.x;
            scale = (T)kProlongScale;
        }
        if (l == 0 && pair0)
            LS_LAUNCH_PDL(c, k_mg_smooth0_corr_pair, pass_grid(c, N2), kBlock, 0, a.g, cl.g, make_fastdiv((unsigned)K2),
                      (const int8_t*)c->pkind, a.flags, (const float*)a.e, (const float*)a.f0, (const float*)a.f1, (const float*)a.f2,
                      (const float*)a.invd, (const float*)b, (const float*)a.x, (const float*)corr, (float)scale,
                      (float*)a.t);
        else if (form_again<T>())
            LS_LAUNCH_PDL(c, k_mg_smooth_corr<T>, pass_grid(c, a.g.N), kBlock, 0, a.g, cl.g, a.flags, a.e, a.f0, a.f1, a.f2, a.invd, b,
                      (const T*)a.x, corr, scale, a.t);
        else {
            LS_LAUNCH_PDL(c, k_mg_correct<T>, gd, kBlock, 0, a.g, cl.g, a.flags, corr, a.x, scale);
            LS_TRY(smooth(l, b, (const T*)a.x, a.t, nullptr, nullptr, nullptr));
        }
        return smooth(l, b, (const T*)a.t, out, dv, dv2, nb);
    };
    return cycle(0, r, z, r, dotv2, nblocks_out);
}

// z = B r and the partials of (r, z), (dotv2, z) finalized into slot, slot + 1. The cycle's
// ~150 launches (most on coarse levels, a few microseconds each) are captured into a CUDA graph
// on first use and replayed from then on: one launch per application.
template <typename T>
ls_status mg_precondition(ls_ctx* c, const T* r, T* z, const T* dotv2, int slot) {
    const int learned = (std::is_same<T, float>::value && c->lpc_active && c->lpc_ready) ? 1 : 0;
    const int is64 = sizeof(T) == 8;
    if (c->mg_graphs_off) {
        int nb = 0;
        LS_TRY(mg_apply<T>(c, r, z, dotv2, &nb));
        return finalize_sum(c, nb, 2, slot);
    }
    for (const auto& gr : c->mg_graphs)
        if (gr.r == r && gr.z == z && gr.dv2 == dotv2 && gr.slot == slot && gr.learned == learned &&
            gr.is64 == is64) {
            LS_CUDA(c, cudaGraphLaunch(gr.exec, c->stream));
            c->launches += gr.launches;
            return LS_OK;
        }
    const long long l0 = c->launches;
    LS_CUDA(c, cudaStreamBeginCapture(c->stream, cudaStreamCaptureModeThreadLocal));
    int nb = 0;
    ls_status st = mg_apply<T>(c, r, z, dotv2, &nb);
    if (st == LS_OK) st = finalize_sum(c, nb, 2, slot);
    cudaGraph_t graph = nullptr;
    const cudaError_t ec = cudaStreamEndCapture(c->stream, &graph);
    const long long n = c->launches - l0;
    c->launches = l0;
    if (st != LS_OK || ec != cudaSuccess) {
        if (graph) cudaGraphDestroy(graph);
        cudaGetLastError();
        return st != LS_OK ? st : set_error(c, LS_CUDA_ERROR, std::string("multigrid graph capture: ") +
                                                                  cudaGetErrorString(ec));
    }
    cudaGraphExec_t exec = nullptr;
    const cudaError_t ei = cudaGraphInstantiate(&exec, graph, 0);
    cudaGraphDestroy(graph);
    if (ei != cudaSuccess)
        return set_error(c, LS_CUDA_ERROR, std::string("multigrid graph instantiation: ") + cudaGetErrorString(ei));
    c->mg_graphs.push_back(MGGraph{r, z, dotv2, slot, learned, is64, exec, n});
    LS_CUDA(c, cudaGraphLaunch(exec, c->stream));
    c->launches += n;
    return LS_OK;
}

template ls_status mg_precondition<float>(ls_ctx*, const float*, float*, const float*, int);
template ls_status mg_precondition<double>(ls_ctx*, const double*, double*, const double*, int);
template ls_status inner_invd<float>(ls_ctx*);
template ls_status inner_invd<double>(ls_ctx*);
template ls_status mg_setup<float>(ls_ctx*);
template ls_status mg_setup<double>(ls_ctx*);
template ls_status mg_clear<float>(ls_ctx*);
template ls_status mg_clear<double>(ls_ctx*);
template ls_status mg_apply<float>(ls_ctx*, const float*, float*, const float*, int*);
template ls_status mg_apply<double>(ls_ctx*, const double*, double*, const double*, int*);

}  // namespace ls
