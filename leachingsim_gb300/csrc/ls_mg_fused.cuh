// ls_mg_fused.cuh - the coarse levels of the pressure multigrid in one launch (included by
// ls_mg.cu).
//
// A K-cycle visits level 3 eight times and the levels below it as often, and a kernel there
// runs for 3-9 us however few cells it has: launch, two memory round trips, drain. Here one
// launch runs the whole correction from some level down: the K-cycle FCG of that level, the
// levels below it and the coarsest solve. FP32 takes levels of up to a cell per thread, in one block; FP64
// and LS_MG_TAIL_CELLS above 2,048 take a thread-block cluster. Each of its blocks owns a slab of consecutive cells
// of every level and holds its coefficients and vectors in shared memory; a new value of an
// iterate also goes to the halos of the slabs on either side (distributed shared memory), so a
// sweep reads local shared memory only, and a cluster barrier (about 1 us) ends it. Small levels
// (kBlockCells) are held whole by the cluster's first block, which runs them alone with block
// barriers; the coarsest level's sweeps keep the coefficients in registers. In FP64 the coarsest
// cells are spread over the cluster instead (its 48 sweeps would wait for one SM's FP64 pipe),
// every block holding the whole iterate.
//
// Every cell value is formed by the same operations in the same order as by the level kernels of
// ls_mg.cu, and the dot products by the same tree (a warp's shuffle sum, eight warps, then
// k_finalize's tree over the 256-cell partials), so the results are the same. (A link that
// leaves the domain is a zero coefficient here and a skipped term there: only the sign of a
// zero could differ.) The trees agree for levels that the level kernels cover with one cell per
// thread, which bounds the levels taken here.
//
// What bounds it: a step's issue and shared-memory reads on one SM (a sweep over 1,144 cells 1.1
// us), the cluster barrier (0.7-1 us), the coarsest sweeps' dependent chain (0.18 us each, 48 of
// them). A visit from a level of 320 cells down takes 17 us (160x256x256), from 700 down with its
// K-cycle 29 (224x320x320). Against level kernels alone: 160x256x256 21.3 and 18.2 ms, 32x40x40
// (ten steps) 12.2 and 11.0, 48x64x64 with the FP64 solver 30.1 and 26.0; which levels gain is at
// kFuseCells32 in ls_mg.cu.
#pragma once

#include <cooperative_groups.h>

namespace ls {

constexpr int kFuseThreads = 1024;
constexpr int kMaxFuse = 10;
constexpr int kBlockCells = 2048;

template <typename T>
struct FLevel {
    Grid g;
    const int* comp;
    const T *e, *f0, *f1, *f2, *invd;
    T *x, *b, *ev;                        // results and right-hand side in global memory
    FastDiv div_per;
    int per;                              // cells of a slab, a multiple of 256 (a block level: all)
    int blk;                              // 1: held and run by the first block alone
    // shared-memory offsets, in elements of T: excess (negative: the cell is not a member of its
    // block's owner), omega invd (negative: no unknown), lower faces, two iterates with halos,
    // right-hand side, FCG vectors (levels with a K-cycle); oM: the children that are members of
    // the cell, a bit each, in bytes
    int oE, oW, oF0, oF1, oF2, oX, oT, oB, oZ, oQ, oV, oM;
};

template <typename T>
struct FuseArgs {
    FLevel<T> lv[kMaxFuse];
    int n;            // levels; lv[n - 1] is the coarsest
    int nk;           // the first nk of them are corrected by two FCG iterations
    int nc;           // the first nc of them run on the whole cluster, the rest in its first block
    int sweeps;       // of the coarsest level
    int oP;           // shared-memory offset of a slab of products, for the dots
    T scale;          // over-correction below the K-cycle levels
    double* partials; // per-256-cell partial dots
};

// shared memory: this, the FP64 coarsest iterate (2 kCoarsestCells), the levels' arrays
struct FuseRed {
    double tree[2][kFinalizeThreads];
    double part[2 * kBlockCells / 256];  // a block level's partial dots
    double s[3];
    double coef;
};
extern __shared__ double fuse_smem[];
template <typename T>
__device__ __forceinline__ FuseRed& fuse_red() {
    return *reinterpret_cast<FuseRed*>(fuse_smem);
}
template <typename T>
__host__ __device__ constexpr size_t fuse_fixed() {
    return sizeof(FuseRed) + (sizeof(T) == 8 ? 2 * kCoarsestCells * sizeof(T) : 0);
}

// The threads that share a step: CL, all of the cluster; else one block of it. A level's cells
// base .. base + count are this block's.
template <typename T, bool CL>
struct Fuse {
    const FuseArgs<T>& A;
    int rank, blocks;

    // (from the shared array itself, so that the accesses are shared-memory instructions)
    static __device__ __forceinline__ T* shm(int o) {
        return reinterpret_cast<T*>(reinterpret_cast<char*>(fuse_smem) + fuse_fixed<T>()) + o;
    }
    static __device__ __forceinline__ T* xs() {
        return reinterpret_cast<T*>(reinterpret_cast<char*>(fuse_smem) + sizeof(FuseRed));
    }

    __device__ __forceinline__ void sync() const {
        if (CL) {
            asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
            asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
        } else {
            __syncthreads();
        }
    }
    __device__ __forceinline__ int base(const FLevel<T>& L) const { return CL ? rank * L.per : 0; }
    __device__ __forceinline__ int count(const FLevel<T>& L) const {
        const int n = (int)L.g.N - base(L);
        return n < 0 ? 0 : n < L.per ? n : L.per;
    }
    template <typename P>
    __device__ __forceinline__ P* at(P* p, int r) const {
        return cooperative_groups::this_cluster().map_shared_rank(p, r);
    }
    // element r of a level's iterate at offset o, wherever it is held
    __device__ __forceinline__ const T* place(const FLevel<T>& L, int o, int r) const {
        const int own = L.blk ? 0 : (int)fdiv(L.div_per, (unsigned int)r);
        const T* p = shm(0) + o + (int)L.g.JK + (r - own * L.per);
        return CL ? at(p, own) : p;
    }
    // value of own cell lc into the vector at offset o and into the neighbouring slabs' halos
    __device__ __forceinline__ void put(const FLevel<T>& L, int o, int lc, T v) const {
        const int JK = (int)L.g.JK;
        T* y = shm(0) + o + JK + lc;
        *y = v;
        if (CL) {
            if (lc < JK && rank > 0) *at(y + L.per, rank - 1) = v;
            if (lc >= L.per - JK && rank + 1 < blocks) *at(y - L.per, rank + 1) = v;
        }
    }
    // (M y)_r of own cell lc, y at offset o, the terms in m_apply's order
    __device__ __forceinline__ T apply(const FLevel<T>& L, int o, int lc, T yr) const {
        const int JK = (int)L.g.JK, K = L.g.K;
        const T* y = shm(0) + o + JK + lc;
        const T *F0 = shm(0) + L.oF0 + lc, *F1 = shm(0) + L.oF1 + lc, *F2 = shm(0) + L.oF2 + lc;
        T acc = fabs(shm(0)[L.oE + lc]) * yr;
        acc += F0[0] * (yr - y[-JK]);
        acc += F1[0] * (yr - y[-K]);
        acc += F2[0] * (yr - y[-1]);
        acc += F2[1] * (yr - y[1]);
        acc += F1[K] * (yr - y[K]);
        acc += F0[JK] * (yr - y[JK]);
        return acc;
    }
    // the own slab of level q; the lower faces' arrays start one neighbour before it
    __device__ void load(int q) const {
        const FLevel<T>& L = A.lv[q];
        const int b0 = base(L), N = (int)L.g.N, JK = (int)L.g.JK, K = L.g.K, t = (int)threadIdx.x;
        const bool parent = q + 1 < A.n;
        for (int c = t; c < L.per; c += kFuseThreads) {
            const int r = b0 + c;
            const int id = r < N ? __ldg(L.comp + r) : -1;
            T e = r < N ? __ldg(L.e + r) : (T)0;
            if (id >= 0 && parent) {
                int i, j, k;
                decode(L.g, r, i, j, k);
                const FLevel<T>& C = A.lv[q + 1];
                if (__ldg(C.comp + (k >> 1) + C.g.K * ((j >> 1) + C.g.J * (i >> 1))) != id) e = copysign(e, (T)-1);
            }
            shm(0)[L.oE + c] = e;
            shm(0)[L.oW + c] = id >= 0 ? (T)kOmega * __ldg(L.invd + r) : (T)-1;
            shm(0)[L.oB + c] = (T)0;
        }
        auto faces = [&](int o, const T* f, int lead) {
            for (int c = t; c < L.per + lead; c += kFuseThreads) {
                const int r = b0 - lead + c;
                shm(0)[o + c] = r >= 0 && r < N ? __ldg(f + r) : (T)0;
            }
        };
        faces(L.oF0, L.f0, JK);
        faces(L.oF1, L.f1, K);
        faces(L.oF2, L.f2, 1);
        for (int c = t; c < L.per + 2 * JK; c += kFuseThreads) shm(0)[L.oX + c] = shm(0)[L.oT + c] = (T)0;
        load_members(q);
    }
    // per own cell of level q > 0: which of its children are members of it
    __device__ void load_members(int q) const {
        if (q == 0) return;
        const FLevel<T>& L = A.lv[q];
        const FLevel<T>& F = A.lv[q - 1];
        uint8_t* m = reinterpret_cast<uint8_t*>(shm(0)) + L.oM;
        for (int c = threadIdx.x; c < L.per; c += kFuseThreads) {
            const int R = base(L) + c;
            unsigned int bits = 0;
            const int own = R < (int)L.g.N ? __ldg(L.comp + R) : -1;
            if (own >= 0) {
                int I, J, K;
                decode(L.g, R, I, J, K);
#pragma unroll
                for (int z = 0; z < 8; ++z) {
                    const int i = 2 * I + (z >> 2), j = 2 * J + ((z >> 1) & 1), k = 2 * K + (z & 1);
                    if (i < F.g.I && j < F.g.J && k < F.g.K &&
                        __ldg(F.comp + k + F.g.K * (j + F.g.J * i)) == own)
                        bits |= 1u << z;
                }
            }
            m[c] = (uint8_t)bits;
        }
    }

    // Partial sums of the products in p0 and, when given, p1 (zeros where there is no unknown) over
    // the 256-cell groups, as the level kernels form them: per 32 cells the shuffle tree (lane l +
    // lane l + 16, + 8, ...), then the eight in order. FP64 additions bound this (a warp's takes 64
    // clocks of its quarter of the SM), so a warp takes 128 cells and at the first two steps the
    // lanes that would compute values nobody reads take over other cells' halves: six additions
    // for four trees. (a + b is b + a bit for bit.)
    __device__ __noinline__ void partial(const FLevel<T>& L, const T* p0, const T* p1) const {
        __syncthreads();
        const int lane = (int)threadIdx.x & 31, warp = (int)threadIdx.x >> 5;
        double* const unit = &fuse_red<T>().tree[0][0];  // sums of 32 cells, two per index
        const int chunks = (L.per >> 7) * (p1 ? 2 : 1);
        for (int q = warp; q < chunks; q += kFuseThreads / 32) {
            const int v = p1 ? q & 1 : 0, c0 = (p1 ? q >> 1 : q) << 7;
            const T* p = (v ? p1 : p0) + c0 + 2 * (lane & 16) + (lane & 15);
            const double a = widen(p[0]) + widen(p[16]), b = widen(p[64]) + widen(p[80]);
            const bool up = lane & 8;
            double x = (up ? b : a) + __shfl_xor_sync(0xffffffffu, up ? a : b, 8);
#pragma unroll
            for (int o = 4; o > 0; o >>= 1) x = x + __shfl_xor_sync(0xffffffffu, x, o);
            // lanes 0, 16: cells 0-31, 32-63 of the chunk; lanes 8, 24: 64-95, 96-127
            if ((lane & 7) == 0) unit[2 * ((c0 >> 5) + ((lane >> 4) & 1) + ((lane >> 2) & 2)) + v] = x;
        }
        __syncthreads();
        const int g = (int)threadIdx.x >> 1, v = (int)threadIdx.x & 1;
        if (256 * g < count(L) && (v == 0 || p1)) {
            double s = 0.0;
#pragma unroll
            for (int w = 0; w < 8; ++w) s += unit[2 * (8 * g + w) + v];
            (CL ? A.partials : fuse_red<T>().part)[2 * (((base(L)) >> 8) + g) + v] = s;
        }
    }
    // k_finalize's tree over the partials of N cells, then the step's scalar in every block, by one
    // thread (a thousand FP64 divisions would hold the pipe for 5 us): MODE 0 (za, q0), (za, r):
    // their quotient, (za, q0) in s0; 1 (q0, zb): -(q0, zb) / s0; 2 (pd, q1), (pd, r): their quotient
    template <int MODE>
    __device__ __noinline__ T finalize(int N, double& s0) const {
        sync();
        const int nb = (N + 255) >> 8, t = (int)threadIdx.x & 255, v = (int)threadIdx.x >> 8;
        const int wide = nb > 32;  // else the upper steps of the tree add zeros
        if (v < 2 && (wide || t < 32)) {
            double acc = 0.0;
            for (int b = t; b < nb; b += kFinalizeThreads) acc = acc + (CL ? __ldcg(A.partials + 2 * b + v) : fuse_red<T>().part[2 * b + v]);
            fuse_red<T>().tree[v][t] = acc;
        }
        for (int w = wide ? kFinalizeThreads / 2 : 0; w >= 32; w >>= 1) {
            __syncthreads();
            if (v < 2 && t < w) fuse_red<T>().tree[v][t] = fuse_red<T>().tree[v][t] + fuse_red<T>().tree[v][t + w];
        }
        if (v < 2 && t < 32) {  // the last additions within the warp that made its inputs
            __syncwarp();
            double x = fuse_red<T>().tree[v][t];
            for (int w = 16; w > 0; w >>= 1) x = x + __shfl_down_sync(0xffffffffu, x, w);
            if (t == 0) fuse_red<T>().s[v] = x;
        }
        __syncthreads();
        if (threadIdx.x == 0) {
            FuseRed& red = fuse_red<T>();
            const double den = MODE == 1 ? s0 : red.s[0], num = MODE == 1 ? -red.s[0] : red.s[1];
            red.coef = dpos(den) ? num / den : 0.0;
        }
        __syncthreads();
        if (MODE == 0) s0 = fuse_red<T>().s[0];
        return (T)fuse_red<T>().coef;
    }

    // y = x + omega invd (b - M x), x at offset ox, y into offset oy; keep: y into the vector at
    // that offset too; gout: and into global memory; dotv: the partial dots (vector at dotv, y)
    __device__ __noinline__ void smooth(const FLevel<T>& L, int ox, int oy, int keep, T* gout, int dotv) const {
        const int cnt = count(L), JK = (int)L.g.JK;
        const T *W = shm(L.oW), *B = shm(L.oB), *X = shm(ox + JK);
        const int top = dotv >= 0 ? L.per : cnt;
        // two cells at a time, computed whether they hold an unknown or not, so that the second
        // one's loads do not wait for the first
        for (int l0 = threadIdx.x; l0 < top; l0 += 2 * kFuseThreads) {
            const int l1 = l0 + kFuseThreads < top ? l0 + kFuseThreads : l0;
            const T w0 = W[l0], w1 = W[l1], x0 = X[l0], x1 = X[l1];
            const T y0 = x0 + w0 * (B[l0] - apply(L, ox, l0, x0)), y1 = x1 + w1 * (B[l1] - apply(L, ox, l1, x1));
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const int lc = h ? l1 : l0;
                const T out = h ? y1 : y0;
                if (h && l1 == l0) break;
                const bool live = (h ? w1 : w0) > (T)0;
                if (live) {
                    put(L, oy, lc, out);
                    if (keep >= 0) shm(keep)[lc] = out;
                    if (gout) gout[base(L) + lc] = out;
                }
                if (dotv >= 0) shm(A.oP)[lc] = live ? shm(dotv)[lc] * out : (T)0;
            }
        }
        if (dotv >= 0) partial(L, shm(0) + A.oP, nullptr);  // finalize synchronises
        else sync();
    }

    // t = omega invd b, the first sweep from zero
    __device__ __forceinline__ void first(const FLevel<T>& L) const {
        const int cnt = count(L);
        for (int lc = threadIdx.x; lc < cnt; lc += kFuseThreads) {
            const T w = shm(0)[L.oW + lc];
            if (w > (T)0) put(L, L.oT, lc, w * shm(0)[L.oB + lc]);
        }
        sync();
    }

    // way down from level q (its first sweep is in t): second sweep, residual (left in t), coarse
    // right-hand side: the members' residuals in k_mg_restrict's child order. A block level's is
    // formed by the first block, a cluster level's by its owners, the FP64 coarsest level's in
    // global memory.
    __device__ __noinline__ void down(int q) const {
        const FLevel<T>& L = A.lv[q];
        const FLevel<T>& C = A.lv[q + 1];
        smooth(L, L.oT, L.oX, -1, nullptr, -1);
        const int cnt = count(L), JK = (int)L.g.JK;
        for (int lc = threadIdx.x; lc < cnt; lc += kFuseThreads)
            if (shm(0)[L.oW + lc] > (T)0)
                shm(0)[L.oT + JK + lc] = shm(0)[L.oB + lc] - apply(L, L.oX, lc, shm(0)[L.oX + JK + lc]);
        sync();
        const bool spread = CL && !C.blk, own_place = !(sizeof(T) == 8 && CL && q + 2 == A.n);
        const int c0 = spread ? rank * C.per : 0;
        int ccnt = min(C.per, (int)C.g.N - c0);
        if (CL && C.blk && rank != 0) ccnt = 0;
        const uint8_t* mem = reinterpret_cast<const uint8_t*>(shm(0)) + C.oM;
        for (int lc = threadIdx.x; lc < ccnt; lc += kFuseThreads) {
            int I, J, K;
            decode(C.g, c0 + lc, I, J, K);
            const unsigned int bits = mem[lc];
            const int f0 = 2 * K + L.g.K * (2 * J + L.g.J * 2 * I);
            T v[8];
#pragma unroll
            for (int z = 0; z < 8; ++z) {
                const int fr = f0 + (z & 1) + ((z >> 1) & 1) * L.g.K + (z >> 2) * JK;
                v[z] = *place(L, L.oT, bits >> z & 1 ? fr : f0);  // no branch: the eight loads go out together
            }
            T acc = (T)0;
#pragma unroll
            for (int z = 0; z < 8; ++z)
                if (bits >> z & 1) acc += v[z];
            if (own_place) shm(0)[C.oB + lc] = acc;
            else C.b[c0 + lc] = acc;
        }
        // the owner of a coarse cell goes on with it; the barriers of the next steps cover the rest
    }

    // way up on level q: the correction of level q + 1 (its X), two sweeps; the result in X
    __device__ __noinline__ void up(int q, T scale, int keep, T* gout, int dotv) const {
        const FLevel<T>& L = A.lv[q];
        const FLevel<T>& C = A.lv[q + 1];
        const int b0 = base(L), cnt = count(L), JK = (int)L.g.JK;
        const bool local = sizeof(T) == 8 && CL && q + 2 == A.n;  // every block holds the coarsest iterate
        for (int lc = threadIdx.x; lc < cnt; lc += kFuseThreads) {
            if (!(shm(0)[L.oW + lc] > (T)0)) continue;
            T xv = shm(0)[L.oX + JK + lc];
            if (!signbit(shm(0)[L.oE + lc])) {
                int i, j, k;
                decode(L.g, b0 + lc, i, j, k);
                const int R = (k >> 1) + C.g.K * ((j >> 1) + C.g.J * (i >> 1));
                xv += scale * (local ? xs()[R] : *place(C, C.oX, R));
            }
            put(L, L.oX, lc, xv);
        }
        sync();
        smooth(L, L.oX, L.oT, -1, nullptr, -1);
        smooth(L, L.oT, L.oX, keep, gout, dotv);
    }

    // the coarsest level (at most kCoarsestCells cells): damped Jacobi sweeps from zero, one cell
    // per thread, the iterate in X (one block) or in xs() of every block (FP64 on the cluster)
    __device__ __noinline__ void coarsest(int q, bool top) const {
        const FLevel<T>& L = A.lv[q];
        const int N = (int)L.g.N, JK = (int)L.g.JK, K = L.g.K;
        const int per = CL ? (N + blocks - 1) / blocks : N;
        int r = (int)threadIdx.x;
        const bool mine = r < per && (CL ? rank * per : 0) + r < N;
        const int team = (N + 31) & ~31;  // one block: the warps that hold cells
        if (CL) r += rank * per;
        if (CL) sync();  // the right-hand side comes from the whole cluster
        if (CL || r < team) {
            // no branch in the sweeps: a cell without an unknown has zero coefficients and stays 0
            T e = (T)0, c[6], w = (T)0, bv = (T)0;
            int nb[6];
#pragma unroll
            for (int d = 0; d < 6; ++d) {
                c[d] = (T)0;
                nb[d] = r < N ? r : 0;
            }
            if (mine && __ldg(L.comp + r) >= 0) {
                int i, j, k;
                decode(L.g, r, i, j, k);
                const bool h[6] = {i > 0, j > 0, k > 0, k + 1 < K, j + 1 < L.g.J, i + 1 < L.g.I};
                const int off[6] = {-JK, -K, -1, 1, K, JK};
                const T* const f[6] = {L.f0, L.f1, L.f2, L.f2, L.f1, L.f0};
#pragma unroll
                for (int d = 0; d < 6; ++d)
                    if (h[d]) {
                        nb[d] = r + off[d];
                        c[d] = __ldg(f[d] + (d < 3 ? nb[d] : r));
                    }
                e = __ldg(L.e + r);
                w = (T)kOmega * __ldg(L.invd + r);
                bv = CL ? __ldcg(L.b + r) : shm(0)[L.oB + r];
            }
            const int p0 = L.oX + JK, p1 = L.oT + JK;
            T x = w * bv;
            auto store = [&](int side) {
                if (CL) {
                    if (mine) {
                        T* const p = xs() + side * kCoarsestCells + r;
                        for (int z = 0; z < blocks; ++z) *at(p, z) = x;
                    }
                } else {
                    shm(0)[(side ? p1 : p0) + r] = x;  // (the array goes on past the last cell: zeros)
                }
                if (CL) sync();
                else asm volatile("bar.sync 1, %0;" ::"r"(team) : "memory");
            };
            auto sweep = [&](int side) {  // reads this side
                const T* in = CL ? xs() + side * kCoarsestCells : shm(side ? p1 : p0);
                if (!CL || mine) {  // (the cluster's blocks hold a warp's worth of cells each)
                    T acc = e * x;
#pragma unroll
                    for (int d = 0; d < 6; ++d) acc += c[d] * (x - in[nb[d]]);
                    x = x + w * (bv - acc);
                }
                store(side ^ 1);
            };
            // pairs of sweeps, so that the sides are known to the compiler; the result on side 0
            store(0);
            if ((A.sweeps & 1) == 0) {
                sweep(0);
                for (int s = 2; s < A.sweeps; s += 2) {
                    sweep(1);
                    sweep(0);
                }
                store(0);
            } else {
                for (int s = 1; s < A.sweeps; s += 2) {
                    sweep(0);
                    sweep(1);
                }
            }
            if (top && mine) L.x[r] = x;
        }
        if (!CL) __syncthreads();
    }

    // x = B b on level q by one V-cycle from there down; gout: its result's place in global memory
    __device__ __noinline__ void vcycle(int q, T* gout) const {
        int l = q;
        const int stop = CL ? min(A.nc, A.n - 1) : A.n - 1;
        for (; l < stop; ++l) {
            first(A.lv[l]);
            down(l);
        }
        if (CL && l >= A.nc) alone<0>(l);
        else coarsest(l, l == q && gout);
        for (--l; l >= q; --l) up(l, A.scale, -1, l == q ? gout : (T*)nullptr, -1);
    }

    // levels from q on in the first block alone
    template <int D>
    __device__ __forceinline__ void alone(int q) const {
        if constexpr (CL) {
            if (rank == 0) {
                const Fuse<T, false> f{A, rank, blocks};
                f.sync();  // the right-hand side, formed by this block's threads
                f.template solve<D>(q, nullptr);
            }
            sync();
        }
    }

    // the correction of level q: K-cycle FCG (at most D K-cycle levels remain) or V-cycle
    template <int D>
    __device__ __forceinline__ void solve(int q, T* gout) const {
        if (CL && q >= A.nc) {
            alone<D>(q);
            return;
        }
        if constexpr (D > 0) {
            if (q < A.nk) {
                kfcg<D - 1>(q, gout);
                return;
            }
        }
        vcycle(q, gout);
    }

    // two flexible-CG iterations on level q for M e = b (k_kc_*), the residual in B; the result in
    // X and gout
    template <int D>
    __device__ __noinline__ void kfcg(int q, T* gout) const {
        const FLevel<T>& L = A.lv[q];
        const int N = (int)L.g.N, cnt = count(L), JK = (int)L.g.JK;
        T *const W = shm(0) + L.oW, *const B = shm(0) + L.oB, *const Z = shm(0) + L.oZ, *const Q = shm(0) + L.oQ, *const V = shm(0) + L.oV,
                 *const X = shm(0) + L.oX + JK;
        // q = M pd (pd in X) with the partials of (pd, q), (pd, B); t's own cells hold the second
        // products meanwhile (0 where there is no unknown)
        auto dots = [&](bool store) {
            for (int lc = threadIdx.x; lc < L.per; lc += kFuseThreads) {
                T a0 = (T)0, a1 = (T)0;
                if (W[lc] > (T)0) {
                    const T pr = X[lc];
                    const T v = apply(L, L.oX, lc, pr);
                    if (store) Q[lc] = v;
                    a0 += pr * v;
                    a1 += pr * B[lc];
                }
                shm(0)[A.oP + lc] = a0;
                shm(0)[L.oT + JK + lc] = a1;
            }
            partial(L, shm(0) + A.oP, shm(0) + L.oT + JK);
        };
        const bool kc = q + 1 < A.nk;
        const T scale = kc ? (T)1 : A.scale;  // the FCG steps carry the optimal scaling
        first(L);
        down(q);
        solve<D>(q + 1, nullptr);
        up(q, scale, L.oZ, nullptr, -1);
        dots(true);
        double s0 = 0.0;
        {
            const T a = finalize<0>(N, s0);
            for (int lc = threadIdx.x; lc < cnt; lc += kFuseThreads) {
                const T w = W[lc];
                if (!(w > (T)0)) continue;
                V[lc] = a * Z[lc];
                const T rv = B[lc] - a * Q[lc];
                B[lc] = rv;
                put(L, L.oT, lc, w * rv);  // first sweep of the second cycle
            }
            sync();
        }
        down(q);
        solve<D>(q + 1, nullptr);
        up(q, scale, -1, nullptr, L.oQ);  // zb in X
        {
            const T b = finalize<1>(N, s0);
            for (int lc = threadIdx.x; lc < cnt; lc += kFuseThreads)
                if (W[lc] > (T)0) put(L, L.oX, lc, X[lc] + b * Z[lc]);
            sync();
        }
        dots(false);
        const T a = finalize<2>(N, s0);
        for (int lc = threadIdx.x; lc < cnt; lc += kFuseThreads)
            if (W[lc] > (T)0) {
                const T ev = V[lc] + a * X[lc];
                X[lc] = ev;
                if (gout) gout[base(L) + lc] = ev;
            }
        sync();
    }
};

// The correction of level 0 of `A`: its K-cycle FCG (result in ev) when nk > 0, else its cycle
// (result in x). One cluster; nc = 0 runs everything in one block.
template <typename T>
__global__ void __launch_bounds__(kFuseThreads) k_mg_fused(const __grid_constant__ FuseArgs<T> A) {
    pdl_enter();
    T* const out = A.nk > 0 ? A.lv[0].ev : A.lv[0].x;
    auto cl = cooperative_groups::this_cluster();
    const int rank = A.nc > 0 ? (int)cl.block_rank() : 0, blocks = A.nc > 0 ? (int)cl.num_blocks() : 1;
    {
        const Fuse<T, true> f{A, rank, blocks};
        for (int q = 0; q < A.nc; ++q) {
            if (sizeof(T) == 8 && q + 1 == A.n) f.load_members(q);  // its iterate has its own place
            else f.load(q);
        }
    }
    if (rank == 0) {
        const Fuse<T, false> f{A, rank, blocks};
        for (int q = A.nc; q < A.n; ++q) f.load(q);
    }
    // the right-hand side of the first level, each value by the thread that goes on with it
    const bool spread0 = A.nc > 0;
    const int per0 = A.lv[0].per, b0 = spread0 ? rank * per0 : 0;
    const bool coarsest0 = sizeof(T) == 8 && A.n == 1 && spread0;  // reads it from global memory
    __syncthreads();
    if (!coarsest0)
        for (int lc = threadIdx.x; lc < per0 && b0 + lc < (int)A.lv[0].g.N; lc += kFuseThreads)
            Fuse<T, false>::shm(A.lv[0].oB)[lc] = A.lv[0].b[b0 + lc];
    if (A.nc > 0) {
        const Fuse<T, true> f{A, rank, blocks};
        f.sync();  // every block runs and has cleared its halos
        f.template solve<kKLevels>(0, out);
        f.sync();  // no block leaves while another may still read its shared memory
    } else {
        __syncthreads();
        Fuse<T, false>{A, rank, blocks}.template solve<kKLevels>(0, out);
    }
}

}  // namespace ls
