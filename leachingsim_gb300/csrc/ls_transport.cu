// ls_transport.cu - advection-diffusion-reaction transport of
// Simulation::setupConcentrationEqns + solveConc / solveAcid (src/Simulation.cpp:966-1295,
// 2167-2224) and the implicit saturation system of setupSaturationEqns + solveSaturation
// (src/Simulation.cpp:1858-2053), matrix-free.
//
// Transport rows (active code, src/Simulation.cpp:1129-1232):
//   Precipitate: c = c_old (identity); its flux is zeroed
//   Rock: (1/dt + alpha*n_pore) c - alpha * sum_{Pore nb} c_nb = c_old/dt; flux zeroed
//   others (Air, Pore, Sulphide, any other label): 1/dt diagonal plus, per neighbour:
//     Rock nb -> alpha exchange only; else theta-weighted diffusion (D*Dpore_fac to a Pore
//     nb, D otherwise) and upwind advection of q_face = +q_self on + faces, -q_nb on -
//     faces (zero next to Precipitate/Sulphide); explicit (1-theta) part on the RHS.
//   Links to neighbours outside the domain are skipped.
// conc and acid share the matrix (labels and flux are the same for both solves) and are
// solved together, two right-hand sides per pass.
//
// Solver (GB300 has little FP64 throughput, so FP64 divisions and FP64 Krylov sweeps are
// kept out of the iteration): the FP64 row coefficients and right-hand sides are computed
// once per solve, exactly as the reference assembles them; an FP64 refinement loop forms
// the true residual r = b - A x and its Jacobi-scaled norm ||D^-1 r|| / ||D^-1 b|| (the
// test PETSc applies to left-Jacobi GMRES); each correction comes from an FP32 BiCGStab on
// the red-black reduced form of the unit-diagonal system (D^-1 A) d = D^-1 r with FP32 scaled
// off-diagonals.
#include <algorithm>
#include <cmath>
#include <cstdio>
#include <cstring>

#include "ls_internal.cuh"

namespace ls {

struct TransConst {
    double inv_dt, theta, alpha, D, Dpore, dx2, dx;
    double dc_pore, dc_other;  // -D_eff / dx^2 for a Pore neighbour / any other neighbour
    DxDiv dd;
    int inlet;                 // flow-through model: plane i = 0 holds the inflow values
    double in_val[2];          // inflow value of right-hand side 0 / 1
};

// Inflow row of the flow-through model (LS_BC_FLOW_I, no counterpart in the reference): the
// Pore and Air voxels of plane i = 0 hold the inflow value, like the inlet_bc rows of the
// reference's disabled block (src/Simulation.cpp:997-1004).
__device__ __forceinline__ bool inflow_row(const TransConst& tc, int t, int i) {
    return tc.inlet && i == 0 && (t == kPore || t == kAir);
}

// Coefficients of one transport row: diag, off[6] (+i,-i,+j,-j,+k,-k) and the explicit
// right-hand-side part for field f (f may be null). kind: 1 identity holding its old value,
// 2 coupled, 3 identity holding the inflow value.
// EXPL = false is the fully implicit case theta = 1: the theta factors are 1 and the
// explicit part (1 - theta) * (...) adds zero to the right-hand side (for finite fields), so
// both are left out, which takes most of the FP64 work out of the row.
template <typename L, bool EXPL = true>
__device__ __forceinline__ int trans_row(const Grid& g, const TransConst& tc,
                                         const L* __restrict__ label,
                                         const double* __restrict__ fx,
                                         const double* __restrict__ fy,
                                         const double* __restrict__ fz, long long r, int i, int j,
                                         int k, double& diag, double off[6],
                                         const double* f0, const double* f1, double rhs[2]) {
    const int t = (int)label[r];
#pragma unroll
    for (int d = 0; d < 6; ++d) off[d] = 0.0;
    if (inflow_row(tc, t, i)) {
        diag = 1.0;
        if (f0) rhs[0] = 0.0 + tc.in_val[0];
        if (f1) rhs[1] = 0.0 + tc.in_val[1];
        return 3;
    }
    if (t == kPrecipitate) {
        diag = 1.0;
        if (f0) rhs[0] = 0.0 + f0[r];
        if (f1) rhs[1] = 0.0 + f1[r];
        return 1;
    }
    const long long nbs[6] = {r + g.JK, r - g.JK, r + g.K, r - g.K, r + 1, r - 1};
    const bool val[6] = {i + 1 < g.I, i > 0, j + 1 < g.J, j > 0, k + 1 < g.K, k > 0};
    if (t == kRock) {
        double dg = tc.inv_dt;
        if (f0) rhs[0] = 0.0 + f0[r] * tc.inv_dt;
        if (f1) rhs[1] = 0.0 + f1[r] * tc.inv_dt;
#pragma unroll
        for (int d = 0; d < 6; ++d) {
            if (val[d] && (int)label[nbs[d]] == kPore) {
                dg += tc.alpha;
                off[d] = -tc.alpha;
            }
        }
        diag = dg;
        return 2;
    }
    double dg = tc.inv_dt;
    double fr0 = 0.0, fr1 = 0.0;
    if (f0) { fr0 = f0[r]; rhs[0] = 0.0 + fr0 * tc.inv_dt; }
    if (f1) { fr1 = f1[r]; rhs[1] = 0.0 + fr1 * tc.inv_dt; }
#pragma unroll
    for (int d = 0; d < 6; ++d) {
        if (!val[d]) continue;
        const long long nb = nbs[d];
        const int nt = (int)label[nb];
        if (nt == kRock) {
            dg += tc.alpha;
            off[d] = -tc.alpha;
            continue;
        }
        double q_face;
        switch (d) {
        case 0: q_face = fx[r]; break;
        case 1: q_face = -fx[nb]; break;
        case 2: q_face = fy[r]; break;
        case 3: q_face = -fy[nb]; break;
        case 4: q_face = fz[r]; break;
        default: q_face = -fz[nb]; break;
        }
        double actual_q_face = (nt == kPrecipitate || nt == kSulphide) ? 0.0 : q_face;
        // -D_eff / dx^2 takes one of two values, evaluated once on the host
        double diffusion_coeff = (nt == kPore) ? tc.dc_pore : tc.dc_other;
        double coeff_neighbor = diffusion_coeff;
        double coeff_self = -diffusion_coeff;
        double adv_coeff = tc.dd.div(actual_q_face);
        if (dpos(adv_coeff)) coeff_self += adv_coeff;
        else coeff_neighbor -= adv_coeff;
        if (EXPL) {
            off[d] = tc.theta * coeff_neighbor;
            dg += tc.theta * coeff_self;
            if (f0) rhs[0] += (1.0 - tc.theta) * (-(coeff_self * fr0 + coeff_neighbor * f0[nb]));
            if (f1) rhs[1] += (1.0 - tc.theta) * (-(coeff_self * fr1 + coeff_neighbor * f1[nb]));
        } else {
            off[d] = coeff_neighbor;
            dg += coeff_self;
        }
    }
    diag = dg;
    return 2;
}

struct SatConst {
    double phi_dt, dx, evap;
    DxDiv dd;
};

// Coefficients of one implicit-saturation row (src/Simulation.cpp:1877-1958), from the
// saturation before the solve (s).
template <typename L>
__device__ __forceinline__ int sat_row(const Grid& g, const SatConst& sc,
                                       const L* __restrict__ label,
                                       const double* __restrict__ fx,
                                       const double* __restrict__ fy,
                                       const double* __restrict__ fz,
                                       const double* __restrict__ s, long long r, int i, int j,
                                       int k, double& diag, double off[6], double* rhs) {
    const int t = (int)label[r];
#pragma unroll
    for (int d = 0; d < 6; ++d) off[d] = 0.0;
    if (t == kAir || t == kRock || t == kSulphide || t == kPrecipitate) {
        diag = 1.0;
        if (rhs) *rhs = 0.0 + s[r];
        return 1;
    }
    const long long nbs[6] = {r + g.JK, r - g.JK, r + g.K, r - g.K, r + 1, r - 1};
    const bool val[6] = {i + 1 < g.I, i > 0, j + 1 < g.J, j > 0, k + 1 < g.K, k > 0};
    int air_faces = 0;
#pragma unroll
    for (int d = 0; d < 6; ++d)
        if (val[d] && (int)label[nbs[d]] == kAir) air_faces++;
    double evap_sink = sc.dd.div(air_faces * sc.evap);
    const double sr = s[r];
    double coeff_self = sc.phi_dt;
    if (rhs) *rhs = 0.0 + ((sc.phi_dt * sr) - evap_sink);
    const double* fl[3] = {fx, fy, fz};
#pragma unroll
    for (int d = 0; d < 6; ++d) {
        if (!val[d]) continue;
        const double* f = fl[d >> 1];
        double q = (f[r] + f[nbs[d]]) / 2.0;
        double q_face_outward = (d & 1) ? -q : q;
        if (q_face_outward > 0) {
            double v_eff = q_face_outward / smax(sr, 1e-6);
            coeff_self += sc.dd.div(v_eff);
        } else {
            double v_eff = q_face_outward / smax(s[nbs[d]], 1e-6);
            off[d] = sc.dd.div(v_eff);
        }
    }
    diag = coeff_self;
    return 2;
}


// ---------------------------------------------------------------------------
// setup: FP64 coefficients, right-hand sides, FP32 scaled off-diagonals

template <typename L>
struct Rows {
    int mode;  // 0 transport, 1 implicit saturation
    Grid g;
    TransConst tc;
    SatConst sc;
    const L* label;
    const double *fx, *fy, *fz, *s;
};

// Red-black layout of the inner FP32 system. The seven-point stencil couples a voxel only to
// voxels of the other parity of i + j + k, so the voxels of each colour (0 black, 1 red) sit in
// an array of their own, H = I J K2p elements: voxel (i, j, k) at (k >> 1) + K2p (j + J i),
// K2p = ceil(K / 2) rounded up to 4 (16-byte chunks of a row never straddle rows; the elements
// past a row's end are virtual: zero links, zero values). The neighbours of an element at h are
// the other colour's elements at h -+ J K2p (i), h -+ K2p (j), and along k at h ("near") and at
// h + 1 (odd k) or h - 1 (even k) ("far").
// I, J, K are the layout's extents and i, j, k its coordinates: those of the grid (axis 2), or,
// where rows along k are so short that the rounding makes the arrays larger, the grid's (i, k, j)
// (axis 1) or (j, k, i) (axis 0).
struct RBGrid {
    int I, J, K, K2p, JK2;
    int axis;        // of the grid, along which the layout's rows run
    int si, sj, sk;  // strides of i, j and k in the voxel arrays
    int pair;        // from the place of the grid's voxel (i, j, k), k even, to that of (i, j, k + 1)
    long long H;
    FastDiv div4, div2, div_j;  // by K2p / 4, K2p / 2 and J
};

// of the grid's voxel (i, j, k)
__host__ __device__ __forceinline__ int rb_index(const RBGrid& g, int i, int j, int k, int& colour) {
    colour = (i + j + k) & 1;
    const int li = g.axis == 0 ? j : i, lj = g.axis == 2 ? j : k, lk = g.axis == 2 ? k : g.axis == 1 ? j : i;
    return (lk >> 1) + g.K2p * (lj + g.J * li);
}

static RBGrid make_rb_axis(const Grid& g, int axis) {
    const int n[3] = {g.I, g.J, g.K}, stride[3] = {(int)g.JK, g.K, 1};
    const int ai = axis == 0 ? 1 : 0, aj = axis == 2 ? 1 : 2;
    RBGrid r;
    r.axis = axis;
    r.I = n[ai];
    r.J = n[aj];
    r.K = n[axis];
    r.si = stride[ai];
    r.sj = stride[aj];
    r.sk = stride[axis];
    r.K2p = (((r.K + 1) / 2 + 3) / 4) * 4;
    r.JK2 = r.J * r.K2p;
    r.pair = axis == 2 ? 0 : r.K2p;
    r.H = (long long)r.I * r.JK2;
    r.div4 = make_fastdiv((unsigned int)(r.K2p / 4));
    r.div2 = make_fastdiv((unsigned int)(r.K2p / 2));
    r.div_j = make_fastdiv((unsigned int)r.J);
    return r;
}

// Rows along k, whose chunks are neighbours in the voxel arrays too, unless the virtual elements
// make more than 3/8 of the real ones (K of 2-5, 9-11, 17): the links, residuals and vectors of the
// solve, 64 bytes a voxel with none, would take more than the 88 that a layout of whole rows takes.
// Then the axis whose vectors, with the plane of zeros at either end, are the smallest. Two
// species to 1e-10, rows along k against rows along j: 2000x2000x2 6.9 and 3.2 ms, 2000x2000x5 8.8
// and 8.0, 1700x1700x9 12.2 and 10.4, 1500x1500x11 10.3 and 9.9, 1200x1200x17 9.96 and 9.76 (whole
// rows: 7.5, 16.5, 21.0, 20.1, 19.9).
static RBGrid make_rb(const Grid& g) {
    RBGrid best = make_rb_axis(g, 2);
    if (16 * best.H <= 11 * g.N) return best;
    for (int axis = 1; axis >= 0; --axis) {
        const RBGrid r = make_rb_axis(g, axis);
        if (r.H + 2 * r.JK2 < best.H + 2 * best.JK2) best = r;
    }
    return best;
}

struct TBuf {
    double* c[7];
    double* b[2];
    float* o[6];  // FP32 scaled links, black then red (H each): -i, -j, near, far, +j, +i of the layout
    double* inv;
    int8_t* kind;  // trans_row's, kHardRow added on hard rows
    RBGrid rb;
};

// A hard row: its links outweigh its diagonal by more than kHardSum (much more inflow than outflow; a
// flow without sources has at most as much). Systems with one keep their first solution and turn
// to the whole system when the reduced one fails (mixed_solve).
constexpr int kHardRow = 4;
constexpr float kHardSum = 16.f;
__device__ __forceinline__ int row_kind(int k) { return k & (kHardRow - 1); }

// the FP32 links of row (i, j, k) from its FP64 off-diagonals (+i,-i,+j,-j,+k,-k); whether they
// make a hard row
__device__ __forceinline__ bool store_links(const TBuf& tb, int i, int j, int k, const double off[6], float inv32) {
    int colour;
    const int h = rb_index(tb.rb, i, j, k, colour);
    const long long at = colour * tb.rb.H + h;
    float o[6], sum = 0.f;
#pragma unroll
    for (int d = 0; d < 6; ++d) {
        o[d] = d2f_rz(off[d]) * inv32;
        sum += fabsf(o[d]);
    }
    auto put = [&](float ip, float im, float jp, float jm, float kp, float km, int lk) {
        const bool odd = lk & 1;
        tb.o[0][at] = im;
        tb.o[1][at] = jm;
        tb.o[2][at] = odd ? km : kp;
        tb.o[3][at] = odd ? kp : km;
        tb.o[4][at] = jp;
        tb.o[5][at] = ip;
    };
    if (tb.rb.axis == 2) put(o[0], o[1], o[2], o[3], o[4], o[5], k);
    else if (tb.rb.axis == 1) put(o[0], o[1], o[4], o[5], o[2], o[3], j);
    else put(o[2], o[3], o[4], o[5], o[0], o[1], i);
    return sum > kHardSum;
}

template <typename L, bool EXPL>
__global__ void __launch_bounds__(kBlock) k_t_setup(Rows<L> op, TBuf tb, int nrhs, const double* f0,
                                                    const double* f1, int* __restrict__ hard,
                                                    double* __restrict__ partials) {
    double acc[2] = {0.0, 0.0};
    const Grid& g = op.g;
    for (long long r = blockIdx.x * (long long)blockDim.x + threadIdx.x; r < g.N;
         r += (long long)gridDim.x * blockDim.x) {
        int i, j, k;
        decode(g, r, i, j, k);
        double dg, off[6], rhs[2] = {0.0, 0.0};
        int kind;
        if (op.mode == 0)
            kind = trans_row<L, EXPL>(g, op.tc, op.label, op.fx, op.fy, op.fz, r, i, j, k, dg, off, f0, f1, rhs);
        else
            kind = sat_row(g, op.sc, op.label, op.fx, op.fy, op.fz, op.s, r, i, j, k, dg, off, rhs);
        // the row scaling (not a reference value): reciprocal without an FP64 division
        const double inv = drcp_nr(dg);
        const float inv32 = d2f_rz(inv);
        tb.c[0][r] = dg;
        tb.inv[r] = inv;
#pragma unroll
        for (int d = 0; d < 6; ++d) tb.c[1 + d][r] = off[d];
        const bool hr = store_links(tb, i, j, k, off, inv32);
        if (hr) atomicAdd(hard, 1);
        tb.kind[r] = (int8_t)(kind + (hr ? kHardRow : 0));
        for (int q = 0; q < nrhs; ++q) {
            tb.b[q][r] = rhs[q];
            double bt = rhs[q] * inv;
            acc[q] += bt * bt;
        }
    }
    block_sum_store<2>(acc, partials);
}

// Change test of the transport-row inputs (pass 1 of the fully implicit setup): the dirty
// bit of voxel r is set when its label or own face fluxes differ bitwise from their values at
// the last setup.
template <typename L>
__global__ void __launch_bounds__(kBlock) k_t_dirty(Grid g, const L* __restrict__ label,
                                                    const double* __restrict__ fx,
                                                    const double* __restrict__ fy,
                                                    const double* __restrict__ fz,
                                                    L* __restrict__ sl, double* __restrict__ sx,
                                                    double* __restrict__ sy, double* __restrict__ sz,
                                                    unsigned int* __restrict__ bits, int force) {
    for (long long r0 = (long long)blockIdx.x * blockDim.x + (threadIdx.x & ~31u); r0 < g.N;
         r0 += (long long)gridDim.x * blockDim.x) {
        const long long r = r0 + (threadIdx.x & 31u);
        bool d = false;
        if (r < g.N) {
            const L lab = label[r];
            const long long xb = __double_as_longlong(fx[r]), yb = __double_as_longlong(fy[r]),
                            zb = __double_as_longlong(fz[r]);
            d = force || lab != sl[r] || xb != __double_as_longlong(sx[r]) || yb != __double_as_longlong(sy[r]) ||
                zb != __double_as_longlong(sz[r]);
            if (d) {
                sl[r] = lab;
                sx[r] = __longlong_as_double(xb);
                sy[r] = __longlong_as_double(yb);
                sz[r] = __longlong_as_double(zb);
            }
        }
        const unsigned int w = __ballot_sync(0xffffffffu, d);
        if ((threadIdx.x & 31u) == 0u) bits[r0 >> 5] = w;
    }
}

// Fully implicit (theta = 1) transport setup. A row is a pure function of its own and its
// six neighbours' labels and of its own and its lower neighbours' face fluxes; pass 2 lists
// the rows with a dirty voxel among those, pass 3 recomputes their coefficients, pass 4
// forms the right-hand sides of every row (old value over dt, or the old value on identity
// rows) and the partial norms in a fixed order.
__global__ void __launch_bounds__(kBlock) k_t_scan(Grid g, const unsigned int* __restrict__ bits, long long nw,
                                                   int per, int* __restrict__ list,
                                                   unsigned int* __restrict__ count) {
    const int lane = (int)(threadIdx.x & 31u);
    scan_blocks(g.N, per, [=](long long v0) {
        const long long s = v0 + 32 * lane;
        unsigned int need = 0u;
        if (lane < per && s < g.N) need = stencil_word<true>(g, bits, nw, s, bits[s >> 5]);
        append_words(need, v0, per, list, count);
    });
}

template <typename L>
__global__ void __launch_bounds__(kBlock) k_t_rows(Rows<L> op, TBuf tb, int force, const int* __restrict__ list,
                                                   const unsigned int* __restrict__ count, int* __restrict__ hard) {
    const Grid& g = op.g;
    const int n = (int)*count;
    for (int q = blockIdx.x * blockDim.x + threadIdx.x; q < n; q += gridDim.x * blockDim.x) {
        const int r = list[q];
        int i, j, k;
        decode(g, r, i, j, k);
        double dg, off[6], unused[2];
        const int kind = trans_row<L, false>(g, op.tc, op.label, op.fx, op.fy, op.fz, r, i, j, k, dg, off,
                                             nullptr, nullptr, unused);
        const double inv = drcp_nr(dg);
        const float inv32 = d2f_rz(inv);
        tb.c[0][r] = dg;
        tb.inv[r] = inv;
#pragma unroll
        for (int d = 0; d < 6; ++d) tb.c[1 + d][r] = off[d];
        // the number of hard rows follows the marks (force: it starts from 0, the old marks mean nothing)
        const bool hr = store_links(tb, i, j, k, off, inv32), was = !force && (tb.kind[r] & kHardRow);
        if (hr != was) atomicAdd(hard, hr ? 1 : -1);
        tb.kind[r] = (int8_t)(kind + (hr ? kHardRow : 0));
    }
}

// Also counts, per right-hand side, the rows where b or the solution after k_t_xid (b on
// identity rows) is nonzero: a system with none has the exact solution x = 0 already.
// 0.0 + v on the integer pipe: v, with -0.0 as +0.0
__device__ __forceinline__ double plus_zero(double v) {
    return __double_as_longlong(v) == (long long)0x8000000000000000ull ? 0.0 : v;
}

__global__ void __launch_bounds__(kBlock) k_t_rhs(Grid g, double inv_dt, double in0, double in1, TBuf tb,
                                                  int nrhs, const double* f0, const double* f1,
                                                  const double* __restrict__ x0, const double* __restrict__ x1,
                                                  const int* __restrict__ hard, double* __restrict__ hard_out,
                                                  double* __restrict__ partials) {
    double acc[4] = {0.0, 0.0, 0.0, 0.0};
    unsigned int nz[2] = {0u, 0u};
    for (int r = blockIdx.x * blockDim.x + threadIdx.x; r < (int)g.N; r += gridDim.x * blockDim.x) {
        const int kind = row_kind(tb.kind[r]);
        const double inv = tb.inv[r];
        for (int q = 0; q < nrhs; ++q) {
            const double fv = (q ? f1 : f0)[r];
            // trans_row's right-hand side at theta = 1: 0.0 + c_old on Precipitate rows,
            // the inflow value on inflow rows, 0.0 + c_old * (1/dt) on every other row
            const double rhs = plus_zero(kind == 1 ? fv : kind == 3 ? (q ? in1 : in0) : fv * inv_dt);
            tb.b[q][r] = rhs;
            const double xv = (kind == 1 || kind == 3) ? rhs : (q ? x1 : x0)[r];
            const long long m = 0x7fffffffffffffffll;
            const bool nzb = (__double_as_longlong(rhs) & m) != 0;
            if (nzb) {  // a zero adds nothing to the norm
                const double bt = rhs * inv;
                acc[q] = __fma_rn(bt, bt, acc[q]);
            }
            if (nzb || (__double_as_longlong(xv) & m) != 0) nz[q]++;
        }
    }
    acc[2] = (double)nz[0];
    acc[3] = (double)nz[1];
    if (blockIdx.x == 0 && threadIdx.x == 0) *hard_out = (double)*hard;  // read with the sums
    block_sum_store<4>(acc, partials);
}

// after k_t_setup, which counts no nonzero rows
__global__ void k_t_counts(const int* __restrict__ hard, double* __restrict__ v) {
    v[0] = v[1] = 1.0;
    v[2] = (double)*hard;
}

// identity rows take their value
__global__ void k_t_xid(Grid g, TBuf tb, double* x0, double* x1, int nrhs) {
    for (long long r = blockIdx.x * (long long)blockDim.x + threadIdx.x; r < g.N;
         r += (long long)gridDim.x * blockDim.x) {
        const int kind = row_kind(tb.kind[r]);
        if (kind != 1 && kind != 3) continue;
        x0[r] = tb.b[0][r];
        if (nrhs > 1) x1[r] = tb.b[1][r];
    }
}

// Outer residual: rhs32 = D^-1 (b - A x) in FP32 (red-black layout); partials sum (D^-1 r)^2
// and NaN count. MASK: the right-hand sides it runs for. HBM bounds it (84 bytes a row, 98 with
// the neighbours' second reads) and FP64 issue comes close (nine operations a row, b - A x being
// fused multiply-subtracts from b: 0.5 ms for 32.3 M rows). The coefficients of links that leave
// the domain are zero, so their neighbour index is clamped to the row and nothing branches; with
// an even row length (V = 2) a thread takes two neighbouring rows with 16-byte loads. One
// right-hand side at 338x338x283: 0.58 ms at 5.4 TB/s (0.97 a row at a time with a branch per
// link); two: 0.99 ms (1.50).
struct alignas(16) D2 {
    double v[2];
};
template <int V>
__device__ __forceinline__ void ld_rows(const double* __restrict__ p, int r, double (&o)[V]) {
    if (V == 2) {
        const D2 q = *reinterpret_cast<const D2*>(p + r);
        o[0] = q.v[0];
        o[V - 1] = q.v[1];
    } else {
        o[0] = p[r];
    }
}

template <int MASK, int V>
__global__ void __launch_bounds__(kBlock) k_t_resid(Grid g, TBuf tb, const double* x0, const double* x1,
                                                    float* __restrict__ r0, float* __restrict__ r1,
                                                    double* __restrict__ partials) {
    double acc[4] = {0.0, 0.0, 0.0, 0.0};
    const int n = (int)(g.N / V), JK = (int)g.JK, K = g.K;
    int nan[2] = {0, 0};
    for (int t = blockIdx.x * blockDim.x + threadIdx.x; t < n; t += gridDim.x * blockDim.x) {
        const int r = t * V;
        int i, j, k;
        decode(g, r, i, j, k);
        const int im = i > 0 ? r - JK : r, ip = i + 1 < g.I ? r + JK : r;
        const int jm = j > 0 ? r - K : r, jp = j + 1 < g.J ? r + K : r;
        const int km = k > 0 ? r - 1 : r, kp = k + V < K ? r + V : r;
        double c[7][V], inv[V];
#pragma unroll
        for (int d = 0; d < 7; ++d) ld_rows<V>(tb.c[d], r, c[d]);
        ld_rows<V>(tb.inv, r, inv);
        int colour;
        const int h = rb_index(tb.rb, i, j, k, colour);
#pragma unroll
        for (int q = 0; q < 2; ++q) {
            if (!(MASK >> q & 1)) continue;
            const double* __restrict__ x = q ? x1 : x0;
            double b[V], xc[V], xim[V], xip[V], xjm[V], xjp[V];
            ld_rows<V>(tb.b[q], r, b);
            ld_rows<V>(x, r, xc);
            const double xkm = x[km], xkp = x[kp];
            ld_rows<V>(x, jm, xjm);
            ld_rows<V>(x, jp, xjp);
            ld_rows<V>(x, im, xim);
            ld_rows<V>(x, ip, xip);
#pragma unroll
            for (int e = 0; e < V; ++e) {
                // the diagonal between the lower and the upper links, which have the other sign: taken
                // first it doubles the partial sums, and their rounding kept the norm above 1.55e-16
                // where it now reaches 1.25e-16 (long time steps, 32x40x40)
                double a = __fma_rn(-c[6][e], e == 0 ? xkm : xc[0], b[e]);
                a = __fma_rn(-c[4][e], xjm[e], a);
                a = __fma_rn(-c[2][e], xim[e], a);
                a = __fma_rn(-c[0][e], xc[e], a);
                a = __fma_rn(-c[5][e], e == V - 1 ? xkp : xc[V - 1], a);
                a = __fma_rn(-c[3][e], xjp[e], a);
                a = __fma_rn(-c[1][e], xip[e], a);
                const double rv = a * inv[e];
                // the inner right-hand side in FP32 rounded toward zero on the integer pipe (its
                // rounding is the inner solve's business)
                const long long at = (e ? colour ^ 1 : colour) * tb.rb.H + h + (e ? tb.rb.pair : 0);
                (q ? r1 : r0)[at] = d2f_rz(rv);
                acc[q] = __fma_rn(rv, rv, acc[q]);
                nan[q] += disnan(rv) ? 1 : 0;
            }
        }
    }
    acc[2] = (double)nan[0];
    acc[3] = (double)nan[1];
    block_sum_store<4>(acc, partials);
}

// ---------------------------------------------------------------------------
// Inner FP32 BiCGStab. With the unit diagonal the system is, per colour (b black, r red; O: FP32
// off-diagonals scaled by the row diagonal),
//     x_b + O_b x_r = f_b,     x_r + O_r x_b = f_r,
// and eliminating the red half (Hageman and Young's reduced system) leaves
//     S x_b = f_b - O_b f_r,   S = I - O_b O_r,     x_r = f_r - O_r x_b.
// S is applied by two half sweeps, z = O_r p then v = p - O_b z, which read every link once,
// as one application of the whole matrix does, while the Krylov vectors are half as long, and
// it takes about half the iterations (33 -> 16 to a residual of 1e-13 at 32x28x30): the
// eigenvalues of I + O at 1 -+ mu fold onto 1 - mu^2. The residual of the whole system is the
// reduced one (its red half is zero by construction), so the stopping test is unchanged: ||r||
// against ||f||. An iteration moves 94 bytes per voxel for one right-hand side (whole matrix:
// 112). Two species to 1e-12 with all rows new: 1.46 ms at 97x128x121 (4.43 with BiCGStab on the
// whole matrix), 18.7 at 338x338x283 (46.5); with unchanged rows 1.38 (4.67) and 16.8 (47.1).
// Rows whose links outweigh their diagonal by far can defeat it: mixed_solve.
//
// NQ right-hand sides go together; with NQ = 2 they share the link loads and each vector
// element is a float2 with one lane per right-hand side. Every vector has `pad` zero elements
// before and after its H elements, so the stencil needs no bounds tests (a link that leaves
// the domain has a zero coefficient, and 0 * 0 adds nothing). Each thread takes 16-byte chunks.
//
// Iteration n, with the per-lane scalars a (alpha), w (omega), b (beta) on the device:
//   XP (n > 0): r = s - w t;  d += a p + w s;  p = r + b (p - w v)
//   Z, V      : z = O_r p, v = p - O_b z (n = 0: p = r);        dots (rh, v)
//   ZS, T     : s = r - a v, z = O_r s, t = s - O_b z;          dots (t,s) (t,t) (rh,s) (rh,t) (s,s)
// ZS recomputes s at the six neighbours from r and v, so s is stored once, by T. The
// next rho = (rh, r) = (rh,s) - w (rh,t) and ||r||^2 = (s,s) - 2w (t,s) + w^2 (t,t) come from
// the T dots, so one iteration takes two reductions. Each reduction's one-block finalize updates
// the scalars on the device; kernels return at once when no lane is active, so the host
// launches iterations in batches and reads the state once per batch. The update a p + w s
// still pending after the last iteration goes into d before the red half is formed.

enum {
    TI_BASE = 64,    // lane l: TI_BASE + TI_STRIDE * l + TI_*
    TI_STRIDE = 16,
    TI_RHO = 0,
    TI_ALPHA,
    TI_OMEGA,
    TI_BETA,
    TI_R2,           // ||r||^2 after the last iteration
    TI_RR0,          // ||r0||^2
    TI_TOL2,         // (relative tolerance)^2
    TI_ACT,          // 1 while the lane iterates
    TI_ITS,
    TI_REASON,       // 1 converged, -1 breakdown, -4 NaN/Inf
    TI_F32,          // three slots: alpha, omega and beta as FP32 (k_ti_fin rounds them once;
                     // a conversion per thread would cost the passes 1-3 us of the FP64 pipe)
    TI_ANY = 100     // 1 while some lane iterates
};
__host__ __device__ __forceinline__ int tslot(int l, int v) { return TI_BASE + TI_STRIDE * l + v; }
static_assert((int)TI_ANY < (int)S_COUNT, "transport scalars exceed the scalar block");

enum { PH_INIT = 0, PH_V = 1, PH_ST = 2 };

// inner vectors: pointers to element 0 in the active layout (float or float2 elements)
struct TIVec {
    float *r, *rh, *p, *v, *s, *t, *d, *z;
    const float* rhs[2];  // FP32 D^-1 (b - A x) per lane: black then red, H each, zero-padded
    const float* o[6];    // links, black then red
};

// A thread's 16-byte chunk: 4 / NQ elements of NQ lanes (value m: element m / NQ, lane m % NQ).
template <int NQ>
struct Chunk {
    static constexpr int W = 4 / NQ;
    float v[4];
};

template <int NQ>
__device__ __forceinline__ Chunk<NQ> ld_chunk(const float* __restrict__ x, int h) {
    const float4 q = *reinterpret_cast<const float4*>(x + (long long)NQ * h);
    return {{q.x, q.y, q.z, q.w}};
}
template <int NQ>
__device__ __forceinline__ void st_chunk(float* __restrict__ x, int h, const Chunk<NQ>& c) {
    *reinterpret_cast<float4*>(x + (long long)NQ * h) = make_float4(c.v[0], c.v[1], c.v[2], c.v[3]);
}
// links of the W elements at h
template <int NQ>
__device__ __forceinline__ void ld_link(const float* __restrict__ o, int h, float (&l)[4 / NQ]) {
    if (NQ == 1) {
        const float4 q = __ldg(reinterpret_cast<const float4*>(o + h));
        l[0] = q.x;
        l[1 % (4 / NQ)] = q.y;
        l[2 % (4 / NQ)] = q.z;
        l[3 % (4 / NQ)] = q.w;
    } else {
        const float2 q = __ldg(reinterpret_cast<const float2*>(o + h));
        l[0] = q.x;
        l[1 % (4 / NQ)] = q.y;
    }
}

// sources of the neighbour values: a vector, s = r - a v of two vectors, or the right-hand sides
template <int NQ>
struct SrcVec {
    const float* x;
    __device__ __forceinline__ Chunk<NQ> chunk(int h) const { return ld_chunk<NQ>(x, h); }
    __device__ __forceinline__ void one(int h, float (&e)[NQ]) const {
#pragma unroll
        for (int l = 0; l < NQ; ++l) e[l] = x[(long long)NQ * h + l];
    }
};
template <int NQ>
struct SrcS {
    const float *r, *v;
    float na[NQ];  // -alpha per lane
    __device__ __forceinline__ Chunk<NQ> chunk(int h) const {
        Chunk<NQ> a = ld_chunk<NQ>(r, h);
        const Chunk<NQ> b = ld_chunk<NQ>(v, h);
#pragma unroll
        for (int m = 0; m < 4; ++m) a.v[m] = __fmaf_rn(na[m % NQ], b.v[m], a.v[m]);
        return a;
    }
    __device__ __forceinline__ void one(int h, float (&e)[NQ]) const {
#pragma unroll
        for (int l = 0; l < NQ; ++l)
            e[l] = __fmaf_rn(na[l], v[(long long)NQ * h + l], r[(long long)NQ * h + l]);
    }
};
template <int NQ>
struct SrcRhs {
    const float *f0, *f1;
    __device__ __forceinline__ Chunk<NQ> chunk(int h) const {
        if (NQ == 1) return ld_chunk<NQ>(f0, h);
        const float2 a = *reinterpret_cast<const float2*>(f0 + h), b = *reinterpret_cast<const float2*>(f1 + h);
        return {{a.x, b.x, a.y, b.y}};
    }
    __device__ __forceinline__ void one(int h, float (&e)[NQ]) const {
        e[0] = f0[h];
        if (NQ > 1) e[NQ - 1] = f1[h];
    }
};

// sum over the six links of the elements of a colour in chunk ch, times the other colour's
// values; near = the other colour's chunk at the same place
template <int NQ, typename SRC>
__device__ __forceinline__ Chunk<NQ> rb_links(const RBGrid& g, const TIVec& iv, int colour, int ch, const SRC& src,
                                              Chunk<NQ>& near) {
    constexpr int W = 4 / NQ;
    const int h = ch * W;
    const int row = (int)fdiv(NQ == 1 ? g.div4 : g.div2, (unsigned int)ch);
    const int i = (int)fdiv(g.div_j, (unsigned int)row);
    const bool odd = ((row - i * g.J + i) & 1) != colour;  // odd k: the far neighbour is at h + 1
    const long long base = colour * g.H;
    float l[6][W];
#pragma unroll
    for (int d = 0; d < 6; ++d) ld_link<NQ>(iv.o[d] + base, h, l[d]);
    const Chunk<NQ> im = src.chunk(h - g.JK2), jm = src.chunk(h - g.K2p);
    near = src.chunk(h);
    const Chunk<NQ> jp = src.chunk(h + g.K2p), ip = src.chunk(h + g.JK2);
    float e[NQ];
    src.one(odd ? h + W : h - 1, e);
    Chunk<NQ> far;
#pragma unroll
    for (int m = 0; m < 4; ++m) {
        const float up = m + NQ < 4 ? near.v[(m + NQ) % 4] : e[m % NQ];
        const float dn = m >= NQ ? near.v[(m + 4 - NQ) % 4] : e[m % NQ];
        far.v[m] = odd ? up : dn;
    }
    Chunk<NQ> acc;
#pragma unroll
    for (int m = 0; m < 4; ++m) {
        float a = l[0][m / NQ] * im.v[m];
        a = __fmaf_rn(l[1][m / NQ], jm.v[m], a);
        a = __fmaf_rn(l[2][m / NQ], near.v[m], a);
        a = __fmaf_rn(l[3][m / NQ], far.v[m], a);
        a = __fmaf_rn(l[4][m / NQ], jp.v[m], a);
        a = __fmaf_rn(l[5][m / NQ], ip.v[m], a);
        acc.v[m] = a;
    }
    return acc;
}

// block sums of the per-thread FP32 partials, value v of block b at partials[v gridDim + b]
template <int NV>
__device__ __forceinline__ void ti_block_sum(const float (&acc)[NV], double* __restrict__ partials) {
    double v[NV];
#pragma unroll
    for (int q = 0; q < NV; ++q) v[q] = widen(acc[q]);
    block_sums<NV>(v, partials, (int)gridDim.x, 1);
}

// v: TI_ALPHA, TI_OMEGA or TI_BETA
template <int NQ>
__device__ __forceinline__ void ti_scal(const double* __restrict__ scal, int v, float (&out)[NQ]) {
#pragma unroll
    for (int l = 0; l < NQ; ++l)
        out[l] = *reinterpret_cast<const float*>(scal + tslot(l, TI_F32 + v - TI_ALPHA));
}

// r = rh = f_b - O_b f_r, d = 0, zero halos of the vectors; dots (r, r) and (f, f) per lane
template <int NQ>
__global__ void __launch_bounds__(kBlock) k_rb_init(RBGrid g, int pad, TIVec iv, double* __restrict__ partials) {
    float acc[2 * NQ];
#pragma unroll
    for (int q = 0; q < 2 * NQ; ++q) acc[q] = 0.f;
    const int n = (int)(g.H / (4 / NQ)), stride = gridDim.x * blockDim.x;
    const int t0 = blockIdx.x * blockDim.x + threadIdx.x;
    const SrcRhs<NQ> black{iv.rhs[0], iv.rhs[1]}, red{iv.rhs[0] + g.H, iv.rhs[1] + g.H};
    for (int ch = t0; ch < n; ch += stride) {
        const int h = ch * (4 / NQ);
        const Chunk<NQ> fb = black.chunk(h);
        Chunk<NQ> fr;
        const Chunk<NQ> y = rb_links<NQ>(g, iv, 0, ch, red, fr);
        Chunk<NQ> r;
#pragma unroll
        for (int m = 0; m < 4; ++m) {
            r.v[m] = fb.v[m] - y.v[m];
            acc[m % NQ] = __fmaf_rn(r.v[m], r.v[m], acc[m % NQ]);
            float f2 = __fmaf_rn(fb.v[m], fb.v[m], acc[NQ + m % NQ]);
            acc[NQ + m % NQ] = __fmaf_rn(fr.v[m], fr.v[m], f2);
        }
        st_chunk<NQ>(iv.r, h, r);
        st_chunk<NQ>(iv.rh, h, r);
        st_chunk<NQ>(iv.d, h, Chunk<NQ>{{0.f, 0.f, 0.f, 0.f}});
    }
    float* const vecs[5] = {iv.r, iv.p, iv.v, iv.d, iv.z};
    const long long end = (long long)NQ * g.H;
    for (int q = t0; q < NQ * pad; q += stride)
#pragma unroll
        for (int v = 0; v < 5; ++v) {
            vecs[v][-1 - q] = 0.f;
            vecs[v][end + q] = 0.f;
        }
    ti_block_sum<2 * NQ>(acc, partials);
}

// z = O_r x (x: p, or r on the first iteration)
template <int NQ>
__global__ void __launch_bounds__(kBlock) k_rb_z(RBGrid g, TIVec iv, const float* __restrict__ x,
                                                 const double* __restrict__ scal) {
    pdl_enter();
    if (scal[TI_ANY] == 0.0) return;
    const int n = (int)(g.H / (4 / NQ));
    const SrcVec<NQ> src{x};
    for (int ch = blockIdx.x * blockDim.x + threadIdx.x; ch < n; ch += gridDim.x * blockDim.x) {
        Chunk<NQ> near;
        st_chunk<NQ>(iv.z, ch * (4 / NQ), rb_links<NQ>(g, iv, 1, ch, src, near));
    }
}

// v = p - O_b z (FIRST: p = r, stored); dots (rh, v)
template <int NQ, bool FIRST>
__global__ void __launch_bounds__(kBlock) k_rb_v(RBGrid g, TIVec iv, const double* __restrict__ scal,
                                                 double* __restrict__ partials) {
    pdl_enter();
    if (scal[TI_ANY] == 0.0) return;
    float acc[NQ];
#pragma unroll
    for (int q = 0; q < NQ; ++q) acc[q] = 0.f;
    const int n = (int)(g.H / (4 / NQ));
    const SrcVec<NQ> src{iv.z};
    for (int ch = blockIdx.x * blockDim.x + threadIdx.x; ch < n; ch += gridDim.x * blockDim.x) {
        const int h = ch * (4 / NQ);
        const Chunk<NQ> p = ld_chunk<NQ>(FIRST ? iv.r : iv.p, h), rh = ld_chunk<NQ>(iv.rh, h);
        Chunk<NQ> near;
        Chunk<NQ> y = rb_links<NQ>(g, iv, 0, ch, src, near);
#pragma unroll
        for (int m = 0; m < 4; ++m) {
            y.v[m] = p.v[m] - y.v[m];
            acc[m % NQ] = __fmaf_rn(rh.v[m], y.v[m], acc[m % NQ]);
        }
        st_chunk<NQ>(iv.v, h, y);
        if (FIRST) st_chunk<NQ>(iv.p, h, p);
    }
    ti_block_sum<NQ>(acc, partials);
}

// z = O_r s, s = r - a v formed at the neighbours
template <int NQ>
__global__ void __launch_bounds__(kBlock) k_rb_zs(RBGrid g, TIVec iv, const double* __restrict__ scal) {
    pdl_enter();
    if (scal[TI_ANY] == 0.0) return;
    const int n = (int)(g.H / (4 / NQ));
    SrcS<NQ> src{iv.r, iv.v, {}};
    ti_scal<NQ>(scal, TI_ALPHA, src.na);
#pragma unroll
    for (int l = 0; l < NQ; ++l) src.na[l] = -src.na[l];
    for (int ch = blockIdx.x * blockDim.x + threadIdx.x; ch < n; ch += gridDim.x * blockDim.x) {
        Chunk<NQ> near;
        st_chunk<NQ>(iv.z, ch * (4 / NQ), rb_links<NQ>(g, iv, 1, ch, src, near));
    }
}

// s = r - a v, t = s - O_b z; dots (t,s) (t,t) (rh,s) (rh,t) (s,s) per lane
template <int NQ>
__global__ void __launch_bounds__(kBlock) k_rb_t(RBGrid g, TIVec iv, const double* __restrict__ scal,
                                                 double* __restrict__ partials) {
    pdl_enter();
    if (scal[TI_ANY] == 0.0) return;
    float na[NQ];
    ti_scal<NQ>(scal, TI_ALPHA, na);
    float acc[5 * NQ];
#pragma unroll
    for (int q = 0; q < 5 * NQ; ++q) acc[q] = 0.f;
    const int n = (int)(g.H / (4 / NQ));
    const SrcVec<NQ> src{iv.z};
    for (int ch = blockIdx.x * blockDim.x + threadIdx.x; ch < n; ch += gridDim.x * blockDim.x) {
        const int h = ch * (4 / NQ);
        const Chunk<NQ> r = ld_chunk<NQ>(iv.r, h), v = ld_chunk<NQ>(iv.v, h), rh = ld_chunk<NQ>(iv.rh, h);
        Chunk<NQ> near;
        Chunk<NQ> t = rb_links<NQ>(g, iv, 0, ch, src, near);
        Chunk<NQ> s;
#pragma unroll
        for (int m = 0; m < 4; ++m) {
            const int q = 5 * (m % NQ);
            s.v[m] = __fmaf_rn(-na[m % NQ], v.v[m], r.v[m]);
            t.v[m] = s.v[m] - t.v[m];
            acc[q + 0] = __fmaf_rn(t.v[m], s.v[m], acc[q + 0]);
            acc[q + 1] = __fmaf_rn(t.v[m], t.v[m], acc[q + 1]);
            acc[q + 2] = __fmaf_rn(rh.v[m], s.v[m], acc[q + 2]);
            acc[q + 3] = __fmaf_rn(rh.v[m], t.v[m], acc[q + 3]);
            acc[q + 4] = __fmaf_rn(s.v[m], s.v[m], acc[q + 4]);
        }
        st_chunk<NQ>(iv.s, h, s);
        st_chunk<NQ>(iv.t, h, t);
    }
    ti_block_sum<5 * NQ>(acc, partials);
}

// r = s - w t; d += a p + w s; p = r + b (p - w v)
template <int NQ>
__global__ void __launch_bounds__(kBlock) k_rb_xp(RBGrid g, TIVec iv, const double* __restrict__ scal) {
    pdl_enter();
    if (scal[TI_ANY] == 0.0) return;
    float a[NQ], w[NQ], b[NQ];
    ti_scal<NQ>(scal, TI_ALPHA, a);
    ti_scal<NQ>(scal, TI_OMEGA, w);
    ti_scal<NQ>(scal, TI_BETA, b);
    const int n = (int)(g.H / (4 / NQ));
    for (int ch = blockIdx.x * blockDim.x + threadIdx.x; ch < n; ch += gridDim.x * blockDim.x) {
        const int h = ch * (4 / NQ);
        const Chunk<NQ> s = ld_chunk<NQ>(iv.s, h), t = ld_chunk<NQ>(iv.t, h), v = ld_chunk<NQ>(iv.v, h);
        Chunk<NQ> p = ld_chunk<NQ>(iv.p, h), d = ld_chunk<NQ>(iv.d, h), r;
#pragma unroll
        for (int m = 0; m < 4; ++m) {
            const int l = m % NQ;
            r.v[m] = __fmaf_rn(-w[l], t.v[m], s.v[m]);
            d.v[m] = __fmaf_rn(a[l], p.v[m], __fmaf_rn(w[l], s.v[m], d.v[m]));
            p.v[m] = __fmaf_rn(b[l], __fmaf_rn(-w[l], v.v[m], p.v[m]), r.v[m]);
        }
        st_chunk<NQ>(iv.d, h, d);
        st_chunk<NQ>(iv.r, h, r);
        st_chunk<NQ>(iv.p, h, p);
    }
}

// d += a p + w s: the pending update of the last iteration
template <int NQ>
__global__ void __launch_bounds__(kBlock) k_rb_pending(RBGrid g, TIVec iv, const double* __restrict__ scal) {
    pdl_enter();
    float a[NQ], w[NQ];
    ti_scal<NQ>(scal, TI_ALPHA, a);
    ti_scal<NQ>(scal, TI_OMEGA, w);
    const int n = (int)(g.H / (4 / NQ));
    for (int ch = blockIdx.x * blockDim.x + threadIdx.x; ch < n; ch += gridDim.x * blockDim.x) {
        const int h = ch * (4 / NQ);
        const Chunk<NQ> s = ld_chunk<NQ>(iv.s, h), p = ld_chunk<NQ>(iv.p, h);
        Chunk<NQ> d = ld_chunk<NQ>(iv.d, h);
#pragma unroll
        for (int m = 0; m < 4; ++m) {
            if (w[m % NQ] != 0.f) d.v[m] = __fmaf_rn(w[m % NQ], s.v[m], d.v[m]);
            if (a[m % NQ] != 0.f) d.v[m] = __fmaf_rn(a[m % NQ], p.v[m], d.v[m]);
        }
        st_chunk<NQ>(iv.d, h, d);
    }
}

// both halves of the correction into the FP64 solution: x_b += d, x_r += f_r - O_r d (EVEN: rows
// along k whose pairs of voxels are 16-byte aligned). A lane whose system FP32 does not hold (a norm that
// overflowed before the first update, or one that underflowed to 0) keeps its solution.
template <int NQ, bool EVEN>
__global__ void __launch_bounds__(kBlock) k_rb_accum(RBGrid g, TIVec iv, const double* __restrict__ scal,
                                                     double* __restrict__ x0, double* __restrict__ x1) {
    pdl_enter();
    bool add[NQ];
#pragma unroll
    for (int l = 0; l < NQ; ++l) {
        const long long reason = __double_as_longlong(scal[tslot(l, TI_REASON)]);
        const bool started = __double_as_longlong(scal[tslot(l, TI_ITS)]) != 0;
        add[l] = (started || reason != __double_as_longlong(-4.0)) && dpos(scal[tslot(l, TI_RR0)]);
    }
    const int n = (int)(g.H / (4 / NQ));
    const SrcVec<NQ> src{iv.d};
    const SrcRhs<NQ> red{iv.rhs[0] + g.H, iv.rhs[1] + g.H};
    for (int ch = blockIdx.x * blockDim.x + threadIdx.x; ch < n; ch += gridDim.x * blockDim.x) {
        const int h = ch * (4 / NQ);
        Chunk<NQ> d;
        const Chunk<NQ> y = rb_links<NQ>(g, iv, 1, ch, src, d);
        const Chunk<NQ> f = red.chunk(h);
        const int row = (int)fdiv(NQ == 1 ? g.div4 : g.div2, (unsigned int)ch), i = (int)fdiv(g.div_j, (unsigned int)row);
        const int k2 = h - row * g.K2p, j = row - i * g.J;
        const int par = (i + j) & 1;  // black at k = 2 k2 + par, red at 2 k2 + 1 - par
        const long long base = (long long)i * g.si + (long long)j * g.sj;
#pragma unroll
        for (int m = 0; m < 4; ++m) {
            double* x = (m % NQ) ? x1 : x0;
            const int k0 = 2 * (k2 + m / NQ);
            const float dr = f.v[m] - y.v[m];
            const double e0 = widen(par ? dr : d.v[m]), e1 = widen(par ? d.v[m] : dr);  // at k0, k0 + 1
            if (!add[m % NQ]) continue;
            if (EVEN) {
                if (k0 < g.K) {
                    D2* q = reinterpret_cast<D2*>(x + base + k0);
                    D2 w = *q;
                    w.v[0] += e0;
                    w.v[1] += e1;
                    *q = w;
                }
            } else {
                if (k0 < g.K) x[base + k0 * g.sk] += e0;
                if (k0 + 1 < g.K) x[base + (k0 + 1) * g.sk] += e1;
            }
        }
    }
}

// The whole system (one right-hand side): the same iteration on vectors of both colours, black
// from element 0 and red from element cs, with v = p + O p and t = s + O s, both colours' links in
// one pass, twice the iterations. Where rows' links outweigh their diagonal (sum |O| > 1) the two
// forms differ: with many such rows the reduced one holds longer (33x35x37, sums up to 50: 28
// iterations, this one diverges); with a few extreme ones among ordinary rows (2e6 in four of 84) it
// fails, its right-hand side and products taking up FP32's rounding times the sums, and this one
// takes 39.
__global__ void __launch_bounds__(kBlock) k_rw_init(RBGrid g, int cs, int pad, TIVec iv, double* __restrict__ partials) {
    float acc[2] = {0.f, 0.f};
    const int n = (int)(g.H / 4), stride = gridDim.x * blockDim.x;
    const int t0 = blockIdx.x * blockDim.x + threadIdx.x;
    for (int c = t0; c < 2 * n; c += stride) {
        const int colour = c >= n, h = 4 * (c - colour * n), at = h + colour * cs;
        const Chunk<1> f = ld_chunk<1>(iv.rhs[0] + colour * g.H, h);
#pragma unroll
        for (int m = 0; m < 4; ++m) acc[0] = __fmaf_rn(f.v[m], f.v[m], acc[0]);
        st_chunk<1>(iv.r, at, f);
        st_chunk<1>(iv.rh, at, f);
        st_chunk<1>(iv.d, at, Chunk<1>{{0.f, 0.f, 0.f, 0.f}});
    }
    // zeros before, between and after the colours
    float* const vecs[7] = {iv.r, iv.rh, iv.p, iv.v, iv.s, iv.t, iv.d};
    for (int q = t0; q < pad; q += stride)
#pragma unroll
        for (int v = 0; v < 7; ++v) {
            vecs[v][-1 - q] = 0.f;
            vecs[v][g.H + q] = 0.f;
            vecs[v][cs + g.H + q] = 0.f;
        }
    acc[1] = acc[0];
    ti_block_sum<2>(acc, partials);
}

template <bool FIRST>
__global__ void __launch_bounds__(kBlock) k_rw_v(RBGrid g, int cs, TIVec iv, const double* __restrict__ scal,
                                                 double* __restrict__ partials) {
    pdl_enter();
    if (scal[TI_ANY] == 0.0) return;
    float acc[1] = {0.f};
    const int n = (int)(g.H / 4);
    const float* const x = FIRST ? iv.r : iv.p;
    for (int c = blockIdx.x * blockDim.x + threadIdx.x; c < 2 * n; c += gridDim.x * blockDim.x) {
        const int colour = c >= n, ch = c - colour * n, at = 4 * ch + colour * cs;
        const Chunk<1> p = ld_chunk<1>(x, at), rh = ld_chunk<1>(iv.rh, at);
        Chunk<1> near;
        Chunk<1> y = rb_links<1>(g, iv, colour, ch, SrcVec<1>{x + (colour ? 0 : cs)}, near);
#pragma unroll
        for (int m = 0; m < 4; ++m) {
            y.v[m] = p.v[m] + y.v[m];
            acc[0] = __fmaf_rn(rh.v[m], y.v[m], acc[0]);
        }
        st_chunk<1>(iv.v, at, y);
        if (FIRST) st_chunk<1>(iv.p, at, p);
    }
    ti_block_sum<1>(acc, partials);
}

__global__ void __launch_bounds__(kBlock) k_rw_t(RBGrid g, int cs, TIVec iv, const double* __restrict__ scal,
                                                 double* __restrict__ partials) {
    pdl_enter();
    if (scal[TI_ANY] == 0.0) return;
    float a[1], acc[5] = {0.f, 0.f, 0.f, 0.f, 0.f};
    ti_scal<1>(scal, TI_ALPHA, a);
    const int n = (int)(g.H / 4);
    for (int c = blockIdx.x * blockDim.x + threadIdx.x; c < 2 * n; c += gridDim.x * blockDim.x) {
        const int colour = c >= n, ch = c - colour * n, at = 4 * ch + colour * cs, other = colour ? 0 : cs;
        const Chunk<1> rh = ld_chunk<1>(iv.rh, at), s = SrcS<1>{iv.r, iv.v, {-a[0]}}.chunk(at);
        Chunk<1> near;
        Chunk<1> t = rb_links<1>(g, iv, colour, ch, SrcS<1>{iv.r + other, iv.v + other, {-a[0]}}, near);
#pragma unroll
        for (int m = 0; m < 4; ++m) {
            t.v[m] = s.v[m] + t.v[m];
            acc[0] = __fmaf_rn(t.v[m], s.v[m], acc[0]);
            acc[1] = __fmaf_rn(t.v[m], t.v[m], acc[1]);
            acc[2] = __fmaf_rn(rh.v[m], s.v[m], acc[2]);
            acc[3] = __fmaf_rn(rh.v[m], t.v[m], acc[3]);
            acc[4] = __fmaf_rn(s.v[m], s.v[m], acc[4]);
        }
        st_chunk<1>(iv.s, at, s);
        st_chunk<1>(iv.t, at, t);
    }
    ti_block_sum<5>(acc, partials);
}

// x += d
__global__ void __launch_bounds__(kBlock) k_rw_accum(RBGrid g, int cs, TIVec iv, double* __restrict__ x) {
    pdl_enter();
    const int n = (int)(g.H / 4);
    for (int c = blockIdx.x * blockDim.x + threadIdx.x; c < 2 * n; c += gridDim.x * blockDim.x) {
        const int colour = c >= n, ch = c - colour * n, h = 4 * ch;
        const Chunk<1> d = ld_chunk<1>(iv.d, h + colour * cs);
        const int row = (int)fdiv(g.div4, (unsigned int)ch), i = (int)fdiv(g.div_j, (unsigned int)row);
        const int j = row - i * g.J, k0 = 2 * (h - row * g.K2p) + ((i + j + colour) & 1);
        const long long base = (long long)i * g.si + (long long)j * g.sj;
#pragma unroll
        for (int m = 0; m < 4; ++m)
            if (k0 + 2 * m < g.K) x[base + (k0 + 2 * m) * g.sk] += widen(d.v[m]);
    }
}

__global__ void k_t_copy(long long n, const double* __restrict__ from, double* __restrict__ to) {
    for (long long r = blockIdx.x * (long long)blockDim.x + threadIdx.x; r < n; r += (long long)gridDim.x * blockDim.x)
        to[r] = from[r];
}

__device__ __forceinline__ bool finite_d(double v) { return v == v && fabs(v) < INFINITY; }

// scalar update of lane l after a reduction (a thread per lane); whether the lane goes on
template <int PH, int NQ>
__device__ bool ti_phase(double* scal, const double* red, double tol2_0, double tol2_1, int l) {
    double* s = scal + tslot(l, 0);
    {
        if (PH == PH_INIT) {
            const double rr = red[l], ff = red[NQ + l];  // the reduced and the whole right-hand side
            s[TI_RR0] = ff;
            s[TI_RHO] = rr;
            s[TI_R2] = rr;
            s[TI_TOL2] = l ? tol2_1 : tol2_0;
            s[TI_ALPHA] = s[TI_OMEGA] = s[TI_BETA] = 0.0;
            s[TI_ITS] = 0.0;
            const bool fin = finite_d(rr) && finite_d(ff);
            const bool ok = fin && rr > s[TI_TOL2] * ff;
            s[TI_ACT] = ok ? 1.0 : 0.0;
            s[TI_REASON] = ok ? 0.0 : (fin ? 1.0 : -4.0);
        } else if (PH == PH_V) {
            if (s[TI_ACT] != 0.0) {
                const double rv = red[l];
                if (rv != 0.0 && finite_d(rv)) {
                    s[TI_ALPHA] = s[TI_RHO] / rv;
                } else {
                    s[TI_ACT] = 0.0;
                    s[TI_REASON] = finite_d(rv) ? -1.0 : -4.0;
                    s[TI_ALPHA] = s[TI_OMEGA] = s[TI_BETA] = 0.0;
                }
            } else {
                s[TI_ALPHA] = s[TI_OMEGA] = s[TI_BETA] = 0.0;
            }
        } else {  // PH_ST
            if (s[TI_ACT] != 0.0) {
                const double ts = red[5 * l + 0], tt = red[5 * l + 1], hs = red[5 * l + 2],
                             ht = red[5 * l + 3], ss = red[5 * l + 4];
                const double w = (tt > 0.0) ? ts / tt : 0.0;
                const double rho = hs - w * ht;
                const double r2 = fmax(ss - 2.0 * w * ts + w * w * tt, 0.0);
                s[TI_ITS] += 1.0;
                s[TI_OMEGA] = w;
                s[TI_R2] = r2;
                if (!(finite_d(w) && finite_d(rho) && finite_d(r2) && finite_d(s[TI_ALPHA]))) {
                    s[TI_ACT] = 0.0;
                    s[TI_REASON] = -4.0;
                    s[TI_ALPHA] = s[TI_OMEGA] = s[TI_BETA] = 0.0;
                } else if (r2 <= s[TI_TOL2] * s[TI_RR0]) {
                    s[TI_ACT] = 0.0;
                    s[TI_REASON] = 1.0;
                    s[TI_BETA] = 0.0;
                } else if (w == 0.0 || rho == 0.0) {
                    s[TI_ACT] = 0.0;
                    s[TI_REASON] = -1.0;
                    s[TI_BETA] = 0.0;
                } else {
                    s[TI_BETA] = (rho / s[TI_RHO]) * (s[TI_ALPHA] / w);
                    s[TI_RHO] = rho;
                }
            } else {
                s[TI_ALPHA] = s[TI_OMEGA] = s[TI_BETA] = 0.0;
            }
        }
    }
#pragma unroll
    for (int v = 0; v < 3; ++v) *reinterpret_cast<float*>(s + TI_F32 + v) = (float)s[TI_ALPHA + v];
    return s[TI_ACT] != 0.0;
}

__host__ __device__ constexpr int ti_values(int ph, int nq) { return ph == PH_ST ? 5 * nq : ph == PH_INIT ? 2 * nq : nq; }
// up to four warps per value
__host__ __device__ constexpr int ti_fin_threads(int nv) { return 32 * nv * (4 * nv <= 32 ? 4 : 32 / nv); }

// Fixed-order reduction of the per-block partials by one block, up to four warps per value, and
// the scalar update of phase PH by one thread per lane. The block is bound by its SM's FP64 pipe
// (two additions a clock over up to ten values of 608 partials) and by the update's chain: 7-8 us
// under a profiler, against 9-11 with a block per value, or with one warp per value and 1,216
// partials.
template <int PH, int NQ>
__global__ void __launch_bounds__(ti_fin_threads(ti_values(PH, NQ)))
    k_ti_fin(const double* __restrict__ partials, int nblocks, double* scal, double tol2_0, double tol2_1) {
    pdl_enter();
    if (PH != PH_INIT && scal[TI_ANY] == 0.0) return;
    constexpr int NV = ti_values(PH, NQ);
    constexpr int WPV = ti_fin_threads(NV) / 32 / NV;  // warps per value
    __shared__ double part[NV][4];
    __shared__ double red[NV];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int v = warp / WPV, w = warp - v * WPV;
    if (v < NV) {
        const double* __restrict__ mine = partials + (size_t)v * nblocks;
        double a[2] = {0.0, 0.0};
        for (int b = 32 * w + lane; b < nblocks; b += 64 * WPV) {
            a[0] += mine[b];
            if (b + 32 * WPV < nblocks) a[1] += mine[b + 32 * WPV];
        }
        double x[1] = {a[0] + a[1]};
        warp_sums<1, 16>(x);
        if (lane == 0) part[v][w] = x[0];
    }
    __syncthreads();
    if (threadIdx.x < NV) {
        double x = part[threadIdx.x][0];
        for (int q = 1; q < WPV; ++q) x += part[threadIdx.x][q];
        red[threadIdx.x] = x;
    }
    __syncthreads();
    if (threadIdx.x < 32) {
        const bool on = threadIdx.x < NQ && ti_phase<PH, NQ>(scal, red, tol2_0, tol2_1, (int)threadIdx.x);
        const bool any = __any_sync(0xffffffffu, on);
        if (threadIdx.x == 0) scal[TI_ANY] = any ? 1.0 : 0.0;
    }
}

// min / max of x over the rows
__global__ void __launch_bounds__(kBlock) k_minmax(Grid g, const double* __restrict__ x,
                                                   double* __restrict__ partials) {
    long long k0 = kKeyNegInf, k1 = kKeyNegInf;  // maxima of x and -x (NaN skipped), as integer keys
    for (long long r = blockIdx.x * (long long)blockDim.x + threadIdx.x; r < g.N;
         r += (long long)gridDim.x * blockDim.x) {
        const double v = x[r];
        if (disnan(v)) continue;
        k0 = max(k0, dkey(v));
        k1 = max(k1, dkey_neg(v));
    }
    double m[2] = {dunkey(k0), dunkey(k1)};
    block_max_store<2>(m, partials);
}

// The Rock and Precipitate voxels at the end of a transport solve, one bit each: the voxels
// whose flux the reference zeroes then (src/Simulation.cpp:1134-1149; no transport row uses
// the flux of such a voxel). Labels change after the solve (precipitation makes Pore voxels
// Precipitate), so the deferred zeroing works from these bits, not from the labels it finds.
template <typename L>
__global__ void k_solid_bits(Grid g, const L* __restrict__ label, unsigned int* __restrict__ bits) {
    for (long long r0 = (long long)blockIdx.x * blockDim.x + (threadIdx.x & ~31u); r0 < g.N;
         r0 += (long long)gridDim.x * blockDim.x) {
        const long long r = r0 + (threadIdx.x & 31u);
        bool s = false;
        if (r < g.N) {
            const int t = (int)label[r];
            s = t == kRock || t == kPrecipitate;
        }
        const unsigned int w = __ballot_sync(0xffffffffu, s);
        if ((threadIdx.x & 31u) == 0u) bits[r0 >> 5] = w;
    }
}

__global__ void k_zero_solid_flux(Grid g, const unsigned int* __restrict__ bits, double* __restrict__ fx,
                                  double* __restrict__ fy, double* __restrict__ fz) {
    for (long long r = blockIdx.x * (long long)blockDim.x + threadIdx.x; r < g.N;
         r += (long long)gridDim.x * blockDim.x) {
        if ((bits[r >> 5] >> (r & 31)) & 1u) { fx[r] = 0.0; fy[r] = 0.0; fz[r] = 0.0; }
    }
}

static ls_status t_alloc(ls_ctx* c) {
    const size_t n = (size_t)c->g.N;
    const RBGrid rb = make_rb(c->g);
    LS_TRY(lean_phase(c, kPhaseTransport));  // lean: the transport arrays take the pressure solve's memory
    c->ti_half = rb.H;
    // a plane and a chunk around each vector
    c->ti_pad = ((rb.JK2 + 4 + 31) / 32) * 32;
    // largest first (lean: an arena sized for the other phase then wastes the least)
    if (!c->ti) {
        // inner vectors of up to H float2 each, with `pad` elements on both sides
        c->ti_stride = ((2 * (rb.H + 2 * c->ti_pad) + 63) / 64) * 64;
        LS_TRY(walloc_t(c, &c->ti, (size_t)c->ti_stride * kTiVecs));
        LS_CUDA(c, cudaMemsetAsync(c->ti, 0, sizeof(float) * (size_t)c->ti_stride * kTiVecs, c->stream));
    }
    for (int q = 0; q < 7; ++q)
        if (!c->tc[q]) LS_TRY(walloc_t(c, &c->tc[q], n));
    for (int q = 0; q < 2; ++q)
        if (!c->tb[q]) LS_TRY(walloc_t(c, &c->tb[q], n));
    if (!c->tinv) LS_TRY(walloc_t(c, &c->tinv, n));
    // the virtual elements of the links and right-hand sides hold zeros, and nothing writes them
    for (int q = 0; q < 6; ++q)
        if (!c->to[q]) {
            LS_TRY(walloc_t(c, &c->to[q], 2 * (size_t)rb.H));
            LS_CUDA(c, cudaMemsetAsync(c->to[q], 0, sizeof(float) * 2 * (size_t)rb.H, c->stream));
        }
    for (int q = 0; q < 2; ++q)
        if (!c->trhs[q]) {
            const size_t m = 2 * (size_t)rb.H + 2 * (size_t)c->ti_pad;
            LS_TRY(walloc_t(c, &c->trhs[q], m));
            LS_CUDA(c, cudaMemsetAsync(c->trhs[q], 0, sizeof(float) * m, c->stream));
        }
    if (!c->tkind) LS_TRY(walloc_t(c, &c->tkind, n));
    if (!c->t_hard) LS_TRY(dalloc_t(c, &c->t_hard, 1));
    return LS_OK;
}

static TBuf make_tbuf(ls_ctx* c) {
    TBuf tb;
    for (int q = 0; q < 7; ++q) tb.c[q] = c->tc[q];
    for (int q = 0; q < 2; ++q) tb.b[q] = c->tb[q];
    for (int q = 0; q < 6; ++q) tb.o[q] = c->to[q];
    tb.inv = c->tinv;
    tb.kind = c->tkind;
    tb.rb = make_rb(c->g);
    return tb;
}

// Inner solve of the right-hand sides lane_q[0..NQ-1] (indices into trhs / x), each to its
// relative tolerance tol[l]; the correction is added to x[lane_q[l]]. Returns the
// iterations of each lane. WHOLE (one right-hand side): the whole system instead of the reduced one.
template <int NQ, bool WHOLE>
static ls_status inner_solve(ls_ctx* c, const TBuf& tb, const int lane_q[NQ], const double tol[NQ],
                             int max_it, double* const x[2], int its[NQ]) {
    static_assert(!WHOLE || NQ == 1, "the vectors hold both colours of one right-hand side");
    const Grid g = c->g;
    const RBGrid rb = tb.rb;
    const int pad = (int)c->ti_pad, cs = (int)rb.H + pad;  // WHOLE: red follows black and a pad
    const int grid = grid_for(c, WHOLE ? rb.H / 2 : rb.H / (4 / NQ));
    // the kernels with dots: four blocks per SM are resident together (up to 56 registers a
    // thread), and more would only add partial sums
    const int dgrid = std::min(grid, 4 * c->num_sms);
    TIVec iv;
    float** vecs[kTiVecs] = {&iv.r, &iv.rh, &iv.p, &iv.v, &iv.s, &iv.t, &iv.d, &iv.z};
    if (WHOLE) {  // seven vectors of 2 H + 3 pad elements in the room of eight of 2 (H + 2 pad)
        for (int v = 0; v < kTiVecs - 1; ++v) *vecs[v] = c->ti + (size_t)v * (2 * (size_t)rb.H + 3 * pad) + pad;
        iv.z = nullptr;
    } else {
        for (int v = 0; v < kTiVecs; ++v) *vecs[v] = c->ti + (size_t)v * c->ti_stride + 2 * pad;
    }
    iv.rhs[0] = c->trhs[lane_q[0]] + pad;
    iv.rhs[1] = c->trhs[NQ > 1 ? lane_q[1] : lane_q[0]] + pad;
    for (int d = 0; d < 6; ++d) iv.o[d] = tb.o[d];
    RBGrid el = rb;  // what the element-wise passes run over
    if (WHOLE) el.H = cs + rb.H;
    const double t0 = tol[0] * tol[0], t1 = NQ > 1 ? tol[1] * tol[1] : 0.0;
    const double* const scal = c->scal;
    if constexpr (WHOLE) LS_LAUNCH(c, k_rw_init, dgrid, kBlock, 0, rb, cs, pad, iv, c->partials);
    else LS_LAUNCH(c, k_rb_init<NQ>, dgrid, kBlock, 0, rb, pad, iv, c->partials);
    LS_LAUNCH_PDL(c, (k_ti_fin<PH_INIT, NQ>), 1, ti_fin_threads(ti_values(PH_INIT, NQ)), 0, (const double*)c->partials, dgrid,
                  c->scal, t0, t1);
    auto apply_v = [&](bool first) -> ls_status {  // v of p (first: of r, which p takes)
        Timed tm(c, LS_T_KRY_APPLY);
        if constexpr (WHOLE) {
            if (first) LS_LAUNCH_PDL(c, k_rw_v<true>, dgrid, kBlock, 0, rb, cs, iv, scal, c->partials);
            else LS_LAUNCH_PDL(c, k_rw_v<false>, dgrid, kBlock, 0, rb, cs, iv, scal, c->partials);
        } else {
            LS_LAUNCH_PDL(c, k_rb_z<NQ>, grid, kBlock, 0, rb, iv, (const float*)(first ? iv.r : iv.p), scal);
            if (first) LS_LAUNCH_PDL(c, (k_rb_v<NQ, true>), dgrid, kBlock, 0, rb, iv, scal, c->partials);
            else LS_LAUNCH_PDL(c, (k_rb_v<NQ, false>), dgrid, kBlock, 0, rb, iv, scal, c->partials);
        }
        return LS_OK;
    };
    auto apply_t = [&]() -> ls_status {  // s and t
        Timed tm(c, LS_T_KRY_APPLY);
        if constexpr (WHOLE) {
            LS_LAUNCH_PDL(c, k_rw_t, dgrid, kBlock, 0, rb, cs, iv, scal, c->partials);
        } else {
            LS_LAUNCH_PDL(c, k_rb_zs<NQ>, grid, kBlock, 0, rb, iv, scal);
            LS_LAUNCH_PDL(c, k_rb_t<NQ>, dgrid, kBlock, 0, rb, iv, scal, c->partials);
        }
        return LS_OK;
    };
    // algorithmic bytes of the two operator applications: FP32 off-diagonals (24 per row) plus per
    // lane 2 bytes for each half-length vector (WHOLE: 4 for each vector) read or written once
    const double v_bytes = (double)g.N * (24.0 + 12.0 * NQ);
    const double st_bytes = (double)g.N * (24.0 + (WHOLE ? 20.0 : 18.0 * NQ));
    int it = 0, batch = 4;
    double sc[TI_STRIDE * 2 + 8];
    while (it < max_it) {
        const int nb = std::min(batch, max_it - it);
        for (int b = 0; b < nb; ++b, ++it) {
            if (it > 0) LS_LAUNCH_PDL(c, k_rb_xp<NQ>, grid, kBlock, 0, el, iv, scal);
            LS_TRY(apply_v(it == 0));
            LS_LAUNCH_PDL(c, (k_ti_fin<PH_V, NQ>), 1, ti_fin_threads(ti_values(PH_V, NQ)), 0, (const double*)c->partials, dgrid,
                          c->scal, 0.0, 0.0);
            LS_TRY(apply_t());
            LS_LAUNCH_PDL(c, (k_ti_fin<PH_ST, NQ>), 1, ti_fin_threads(ti_values(PH_ST, NQ)), 0, (const double*)c->partials, dgrid,
                          c->scal, 0.0, 0.0);
        }
        LS_TRY(read_scalars(c, TI_BASE, TI_ANY - TI_BASE + 1, sc));
        if (sc[TI_ANY - TI_BASE] == 0.0) break;
        // next batch: the iterations the observed convergence rate still needs (at least 1)
        batch = 1;
        for (int l = 0; l < NQ; ++l) {
            const double* s = sc + TI_STRIDE * l;
            if (s[TI_ACT] == 0.0 || !(s[TI_R2] > 0.0) || !(s[TI_RR0] > 0.0) || s[TI_ITS] < 1.0) continue;
            const double red = s[TI_R2] / s[TI_RR0];
            const double per_it = log(red) / s[TI_ITS];
            if (per_it < 0.0) {
                const double need = log(s[TI_TOL2]) / per_it - s[TI_ITS];
                batch = std::max(batch, (int)std::min(16.0, std::max(1.0, ceil(need))));
            }
        }
    }
    LS_LAUNCH_PDL(c, k_rb_pending<NQ>, grid, kBlock, 0, el, iv, scal);
    double* const xl[2] = {x[lane_q[0]], NQ > 1 ? x[lane_q[1]] : (double*)nullptr};
    if constexpr (WHOLE) LS_LAUNCH_PDL(c, k_rw_accum, grid, kBlock, 0, rb, cs, iv, xl[0]);
    else if (rb.axis == 2 && g.K % 2 == 0) LS_LAUNCH_PDL(c, (k_rb_accum<NQ, true>), grid, kBlock, 0, rb, iv, scal, xl[0], xl[1]);
    else LS_LAUNCH_PDL(c, (k_rb_accum<NQ, false>), grid, kBlock, 0, rb, iv, scal, xl[0], xl[1]);
    for (int l = 0; l < NQ; ++l) its[l] = (int)sc[TI_STRIDE * l + TI_ITS];
    // the launches of a batch beyond the last iteration return at once and move nothing
    if (c->timing) {
        const int live = NQ > 1 ? std::max(its[0], its[NQ - 1]) : its[0];
        c->timer_bytes[LS_T_KRY_APPLY] += live * (v_bytes + st_bytes) + (live > 0 ? (WHOLE ? 4.0 : 2.0) * NQ * g.N : 0.0);
    }
    return LS_OK;
}

// Mixed-precision solve of the rows in `rows` for nrhs right-hand sides (x warm-started in
// place), fields f0/f1 supplying the right-hand sides.
template <typename L>
static ls_status mixed_solve(ls_ctx* c, const Rows<L>& rows, int nrhs, const double* f0, const double* f1,
                             double* x0, double* x1, double rtol, int max_it, ls_solve_info* info[2],
                             int* zero_lanes = nullptr) {
    LS_TRY(t_alloc(c));
    const Grid g = c->g;
    const int grid = grid_for(c, g.N);
    TBuf tb = make_tbuf(c);
    if (rows.mode == 0 && rows.tc.theta == 1.0 && !c->lean) {
        // fully implicit transport rows: recompute only the rows whose inputs changed
        const TransConst& tc = rows.tc;
        // the inflow values enter the right-hand sides only (k_t_rhs), not the rows
        const double consts[9] = {tc.inv_dt, tc.alpha, tc.D, tc.Dpore, tc.dx, tc.dc_pore, tc.dc_other,
                                  (double)tc.dd.pow2, (double)tc.inlet};
        if (!c->sht_fx) {
            const size_t n = (size_t)g.N;
            LS_TRY(dalloc(c, &c->sht_label, n * c->label_bytes));
            LS_TRY(dalloc_t(c, &c->sht_fx, n));
            LS_TRY(dalloc_t(c, &c->sht_fy, n));
            LS_TRY(dalloc_t(c, &c->sht_fz, n));
            c->t_valid = 0;
        }
        const int force = (!c->t_valid || memcmp(consts, c->t_consts, sizeof(consts)) != 0) ? 1 : 0;
        if (force) LS_CUDA(c, cudaMemsetAsync(c->t_hard, 0, sizeof(int), c->stream));
        c->t_valid = 0;  // until the rows, their marks and the count belong together again
        LS_TRY(wlist_reset(c));
        LS_LAUNCH(c, k_t_dirty<L>, grid, kBlock, 0, g, rows.label, rows.fx, rows.fy, rows.fz,
                  (L*)c->sht_label, c->sht_fx, c->sht_fy, c->sht_fz, c->dbits, force);
        const int per = scan_words(c->num_sms, g.N);
        LS_LAUNCH(c, k_t_scan, scan_grid(c->num_sms, g.N, per), kBlock, 0, g, (const unsigned int*)c->dbits, c->dwords,
                  per, c->wlist, c->wcount);
        LS_LAUNCH(c, k_t_rows<L>, grid, kBlock, 0, rows, tb, force, (const int*)c->wlist, (const unsigned int*)c->wcount,
                  c->t_hard);
        LS_LAUNCH(c, k_t_rhs, grid, kBlock, 0, g, rows.tc.inv_dt, rows.tc.in_val[0], rows.tc.in_val[1], tb, nrhs,
                  f0, f1, (const double*)x0, (const double*)x1, (const int*)c->t_hard, c->scal + S_RED0 + 8, c->partials);
        LS_TRY(finalize_sum(c, grid, 4, S_RED0 + 4));
        memcpy(c->t_consts, consts, sizeof(consts));
        c->t_valid = 1;
    } else {
        LS_CUDA(c, cudaMemsetAsync(c->t_hard, 0, sizeof(int), c->stream));
        if (rows.mode == 0)
            LS_LAUNCH(c, (k_t_setup<L, true>), grid, kBlock, 0, rows, tb, nrhs, f0, f1, c->t_hard, c->partials);
        else
            LS_LAUNCH(c, (k_t_setup<L, false>), grid, kBlock, 0, rows, tb, nrhs, f0, f1, c->t_hard, c->partials);
        LS_TRY(finalize_sum(c, grid, 2, S_RED0 + 4));
        LS_LAUNCH(c, k_t_counts, 1, 1, 0, (const int*)c->t_hard, c->scal + S_RED0 + 6);
        c->t_valid = 0;  // the row buffers now hold other rows
    }
    LS_LAUNCH(c, k_t_xid, grid, kBlock, 0, g, tb, x0, x1, nrhs);
    double den[5];
    LS_TRY(read_scalars(c, S_RED0 + 4, 5, den));
    int mask = nrhs > 1 ? 3 : 1;
    int its[2] = {0, 0}, sweeps[2] = {0, 0}, reason[2] = {0, 0};
    // a system with b = 0 and x = 0 on every row is solved exactly: no residual pass
    for (int q = 0; q < nrhs; ++q)
        if (den[2 + q] == 0.0) { reason[q] = 2; mask &= ~(1 << q); }
    if (zero_lanes) {
        *zero_lanes = 0;
        for (int q = 0; q < nrhs; ++q)
            if (den[2 + q] == 0.0) *zero_lanes |= 1 << q;
    }
    double rel[2] = {0.0, 0.0}, prev[2] = {INFINITY, INFINITY};
    int stagnant[2] = {0, 0}, floored[2] = {0, 0};
    // Hard rows: the first solution is kept (without memory for it the reduced solve is all there is),
    // and a lane whose reduced solve ends without convergence starts again from it on the whole
    // system, with all of max_it.
    bool whole[2] = {false, false}, kept[2] = {false, false};
    double* const xs[2] = {x0, x1};
    if (den[4] > 0.0)
        for (int q = 0; q < nrhs; ++q) {
            if (!((mask >> q) & 1)) continue;
            if (!c->t_keep[q]) dalloc_t(c, &c->t_keep[q], (size_t)g.N);
            kept[q] = c->t_keep[q] != nullptr;
            if (kept[q]) LS_LAUNCH(c, k_t_copy, grid, kBlock, 0, g.N, (const double*)xs[q], c->t_keep[q]);
        }
    auto restart = [&](int q) {
        if (!kept[q] || whole[q]) return false;
        whole[q] = true;
        its[q] = sweeps[q] = stagnant[q] = floored[q] = 0;
        prev[q] = INFINITY;
        return true;
    };
    const int max_sweeps = 40;
    const double inner_floor = 1e-6;
    while (mask) {
        {
            float *t0 = c->trhs[0] + c->ti_pad, *t1 = c->trhs[1] + c->ti_pad;
            const bool two = g.K % 2 == 0;  // pairs of rows stay within a row of voxels, 16-byte aligned
            const double *y0 = x0, *y1 = x1;
            if (mask == 3 && two) LS_LAUNCH(c, (k_t_resid<3, 2>), grid, kBlock, 0, g, tb, y0, y1, t0, t1, c->partials);
            else if (mask == 3) LS_LAUNCH(c, (k_t_resid<3, 1>), grid, kBlock, 0, g, tb, y0, y1, t0, t1, c->partials);
            else if (mask == 1 && two) LS_LAUNCH(c, (k_t_resid<1, 2>), grid, kBlock, 0, g, tb, y0, y1, t0, t1, c->partials);
            else if (mask == 1) LS_LAUNCH(c, (k_t_resid<1, 1>), grid, kBlock, 0, g, tb, y0, y1, t0, t1, c->partials);
            else if (two) LS_LAUNCH(c, (k_t_resid<2, 2>), grid, kBlock, 0, g, tb, y0, y1, t0, t1, c->partials);
            else LS_LAUNCH(c, (k_t_resid<2, 1>), grid, kBlock, 0, g, tb, y0, y1, t0, t1, c->partials);
        }
        LS_TRY(finalize_sum(c, grid, 4, S_RED0));
        double h[4];
        LS_TRY(read_scalars(c, S_RED0, 4, h));
        int solve_mask = 0;
        bool again = false;
        double tol[2] = {0.5, 0.5};
        for (int q = 0; q < nrhs; ++q) {
            if (!((mask >> q) & 1)) continue;
            const bool bad = h[2 + q] > 0.0 || h[q] != h[q];
            rel[q] = bad ? NAN : den[q] > 0.0 ? sqrt(h[q] / den[q]) : sqrt(h[q]);
            // A sweep aims at 0.2 rtol. One that the floor of the inner tolerance stopped above
            // that is followed by another (an iteration or two) while the residual still falls,
            // so that the margin holds at tight tolerances too.
            const bool refine = floored[q] && rel[q] > 0.3 * rtol && rel[q] <= 0.5 * prev[q] && its[q] < max_it &&
                                sweeps[q] < max_sweeps;
            if (!bad && ((rel[q] <= rtol && !refine) || h[q] == 0.0)) { reason[q] = 2; mask &= ~(1 << q); continue; }
            const bool still = rel[q] > 0.5 * prev[q];
            if (bad || its[q] >= max_it || sweeps[q] >= max_sweeps || (still && stagnant[q] >= 5)) {
                if (sweeps[q] > 0 && restart(q)) {
                    LS_LAUNCH(c, k_t_copy, grid, kBlock, 0, g.N, (const double*)c->t_keep[q], xs[q]);
                    again = true;
                } else {
                    reason[q] = bad ? -4 : -3;
                    mask &= ~(1 << q);
                }
                continue;
            }
            stagnant[q] = still ? stagnant[q] + 1 : 0;
            prev[q] = rel[q];
            // inner tolerance: what reaches rtol from here (with a margin), floored at what
            // the FP32 inner system still resolves (a relative 1e-6 is ~17 FP32 ulps)
            const double want = 0.2 * rtol / std::max(rel[q], 1e-300);
            floored[q] = want < inner_floor;
            tol[q] = std::min(0.5, std::max(inner_floor, want));
            solve_mask |= 1 << q;
        }
        if (!solve_mask && !again) break;
        const int budget = std::max(1, max_it - std::max(its[0], its[1]));
        int lane_q[2] = {0, 0}, nq = 0, lits[2] = {0, 0};
        for (int q = 0; q < 2; ++q) {
            if (!((solve_mask >> q) & 1)) continue;
            sweeps[q]++;
            if (!whole[q]) {
                lane_q[nq++] = q;
                continue;
            }
            LS_TRY((inner_solve<1, true>(c, tb, &q, &tol[q], budget, xs, lits)));
            its[q] += lits[0];
        }
        const double ltol[2] = {tol[lane_q[0]], tol[lane_q[nq > 1 ? 1 : 0]]};
        if (nq == 2) LS_TRY((inner_solve<2, false>(c, tb, lane_q, ltol, budget, xs, lits)));
        else if (nq == 1) LS_TRY((inner_solve<1, false>(c, tb, lane_q, ltol, budget, xs, lits)));
        for (int l = 0; l < nq; ++l) its[lane_q[l]] += lits[l];
    }
    ls_status st = LS_OK;
    for (int q = 0; q < nrhs; ++q) {
        double mm[2] = {0.0, -0.0};  // max x, max -x
        if (den[2 + q] != 0.0) {  // otherwise x = 0 on every row
            LS_LAUNCH(c, k_minmax, grid, kBlock, 0, g, (const double*)xs[q], c->partials);
            LS_TRY(finalize_max(c, grid, 2, S_RED0 + 2));
            LS_TRY(read_scalars(c, S_RED0 + 2, 2, mm));
        }
        if (info[q]) {
            info[q]->iterations = its[q];
            info[q]->outer_iterations = sweeps[q];
            info[q]->converged = reason[q] > 0;
            info[q]->reason = reason[q];
            info[q]->rel_residual = rel[q];
            info[q]->max_value = mm[0];
            info[q]->min_value = -mm[1];
        }
        if (reason[q] == -4) st = set_error(c, LS_NONFINITE, "Krylov solve met NaN/Inf");
        else if (reason[q] <= 0 && st == LS_OK) {
            char buf[160];
            snprintf(buf, sizeof(buf), "Krylov solve not converged (rel %.3e after %d its, %d sweeps)",
                     rel[q], its[q], sweeps[q]);
            st = set_error(c, LS_NOT_CONVERGED, buf);
        }
    }
    return st;
}

static TransConst trans_const(const ls_ctx* c, double dt) {
    TransConst tc;
    tc.inv_dt = 1.0 / dt;
    tc.theta = c->p.theta;
    tc.alpha = c->p.alpha_transfer;
    tc.D = c->p.D;
    tc.Dpore = c->p.D * c->p.Dpore_fac;
    tc.dx = c->p.dx;
    tc.dx2 = c->p.dx * c->p.dx;
    tc.dc_pore = -tc.Dpore / tc.dx2;
    tc.dc_other = -tc.D / tc.dx2;
    tc.dd = make_dxdiv(c->p.dx);
    tc.inlet = (c->p.bc_mode == LS_BC_FLOW_I) ? 1 : 0;
    tc.in_val[0] = tc.in_val[1] = 0.0;
    return tc;
}

template <typename L>
static Rows<L> trans_rows(ls_ctx* c, double dt) {
    Rows<L> rows;
    rows.mode = 0;
    rows.g = c->g;
    rows.tc = trans_const(c, dt);
    rows.sc = SatConst{0.0, 1.0, 0.0, make_dxdiv(1.0)};
    rows.label = (const L*)c->label;
    rows.fx = c->fx; rows.fy = c->fy; rows.fz = c->fz; rows.s = nullptr;
    return rows;
}

template <typename L>
static ls_status transport_t(ls_ctx* c, double dt, int which, ls_solve_info* ci, ls_solve_info* ai) {
    Rows<L> rows = trans_rows<L>(c, dt);
    const long long sh = c->p.compat_shift ? c->g.JK : 0;
    double* fields[2] = {c->conc, c->acid};
    double* f[2] = {nullptr, nullptr};
    ls_solve_info* inf[2] = {nullptr, nullptr};
    // An acid field that is identically 0 (the last solve found b = 0 and x = 0 on every row,
    // and nothing has written the field since) gives b = 0 and x = 0 again: the solve would
    // leave it as it is, so it is skipped with the info such a solve reports. (A nonzero
    // inflow of acid gives b != 0 on the inflow rows, so no skip then.)
    const bool acid_inflow = rows.tc.inlet && c->p.acid_inlet != 0.0;
    if ((which & 2) && c->acid_zero && !acid_inflow) {
        which &= ~2;
        if (ai) {
            memset(ai, 0, sizeof(*ai));
            ai->converged = 1;
            ai->reason = 2;
        }
    }
    int n = 0, acid_lane = -1;
    if (which & 1) { f[n] = fields[0]; inf[n] = ci; rows.tc.in_val[n] = c->p.conc_inlet; n++; }
    if (which & 2) { f[n] = fields[1]; inf[n] = ai; rows.tc.in_val[n] = c->p.acid_inlet; acid_lane = n; n++; }
    ls_status st = LS_OK;
    if (n > 0) {
        int zero_lanes = 0;
        st = mixed_solve<L>(c, rows, n, f[0], f[1], f[0] + sh, n > 1 ? f[1] + sh : nullptr, c->p.conc_rtol,
                            c->p.conc_max_it, inf, &zero_lanes);
        if (acid_lane >= 0) c->acid_zero = (st == LS_OK && ((zero_lanes >> acid_lane) & 1)) ? 1 : 0;
    }
    if (st != LS_OK && st != LS_NOT_CONVERGED && st != LS_NONFINITE) return st;
    // the Rock / Precipitate fluxes are zeroed when next looked at: record which they are
    if (!c->solid_bits) {
        const size_t words = (size_t)((c->g.N + 31) / 32);
        LS_TRY(dalloc_t(c, &c->solid_bits, words));
        LS_TRY(dalloc_t(c, &c->solid_bits_b, words));
    }
    LS_LAUNCH(c, k_solid_bits<L>, grid_for(c, c->g.N), kBlock, 0, c->g, (const L*)c->label, c->solid_bits);
    c->flux_zero_pending = 1;
    return st;
}

// The reference zeroes the flux of Rock and Precipitate voxels after the transport solve
// (src/Simulation.cpp:1134-1149). Nothing in a time step reads those fluxes again before the
// next step's flux evaluation overwrites them, so the zeroing waits until something looks:
// the field transfers, counts and asynchronous downloads and the saturation updates call
// this first. It zeroes the voxels recorded at the solve (k_solid_bits), whatever their
// labels have become since; a snapshot keeps the pending state and those bits with the
// fields it copies. Until then the fluxes keep equal to the change-tracking shadows, and the
// next flux evaluation need not restore them.
ls_status flux_zero_now(ls_ctx* c) {
    if (!c->flux_zero_pending) return LS_OK;
    snap_fence(c, kSnapFlux);
    LS_LAUNCH(c, k_zero_solid_flux, grid_for(c, c->g.N), kBlock, 0, c->g, (const unsigned int*)c->solid_bits, c->fx,
              c->fy, c->fz);
    c->flux_zero_pending = 0;
    c->fx_is_shadow = 0;
    return LS_OK;
}

ls_status transport_run(ls_ctx* c, double dt, int which, ls_solve_info* ci, ls_solve_info* ai) {
    snap_fence(c, kSnapRest);  // conc, acid
    if (c->label_bytes == 1) return transport_t<uint8_t>(c, dt, which, ci, ai);
    return transport_t<uint16_t>(c, dt, which, ci, ai);
}

// test hook: y = A x (unscaled, separate multiply and add like an assembled matrix)
template <typename L>
__global__ void k_trans_apply_full(Rows<L> op, const double* __restrict__ x, double* __restrict__ y) {
    const Grid& g = op.g;
    for (long long r = blockIdx.x * (long long)blockDim.x + threadIdx.x; r < g.N;
         r += (long long)gridDim.x * blockDim.x) {
        int i, j, k;
        decode(g, r, i, j, k);
        double dg, off[6];
        trans_row(g, op.tc, op.label, op.fx, op.fy, op.fz, r, i, j, k, dg, off, nullptr, nullptr, nullptr);
        double acc = 0.0;
        if (i > 0) acc += off[1] * x[r - g.JK];
        if (j > 0) acc += off[3] * x[r - g.K];
        if (k > 0) acc += off[5] * x[r - 1];
        acc += dg * x[r];
        if (k + 1 < g.K) acc += off[4] * x[r + 1];
        if (j + 1 < g.J) acc += off[2] * x[r + g.K];
        if (i + 1 < g.I) acc += off[0] * x[r + g.JK];
        y[r] = acc;
    }
}

template <typename L>
static ls_status transport_apply_t(ls_ctx* c, double dt, const double* xh, double* yh) {
    LS_TRY(t_alloc(c));
    c->t_valid = 0;  // tc[0] and tc[1] serve as scratch below
    Rows<L> rows = trans_rows<L>(c, dt);
    const size_t bytes = sizeof(double) * (size_t)c->g.N;
    LS_CUDA(c, cudaMemcpyAsync(c->tc[0], xh, bytes, cudaMemcpyHostToDevice, c->stream));
    LS_LAUNCH(c, k_trans_apply_full<L>, grid_for(c, c->g.N), kBlock, 0, rows, (const double*)c->tc[0],
              c->tc[1]);
    LS_CUDA(c, cudaMemcpyAsync(yh, c->tc[1], bytes, cudaMemcpyDeviceToHost, c->stream));
    LS_CUDA(c, cudaStreamSynchronize(c->stream));
    return LS_OK;
}

ls_status transport_apply_run(ls_ctx* c, double dt, const double* x, double* y) {
    if (c->label_bytes == 1) return transport_apply_t<uint8_t>(c, dt, x, y);
    return transport_apply_t<uint16_t>(c, dt, x, y);
}

// ---------------------------------------------------------------------------
// implicit saturation: the coefficients are taken from the saturation before the solve
// (the setup kernel reads every slot before any solution slot is written)

__global__ void k_clamp_sat(Grid g, double* __restrict__ s) {
    for (long long r = blockIdx.x * (long long)blockDim.x + threadIdx.x; r < g.N;
         r += (long long)gridDim.x * blockDim.x)
        s[r] = smax(0.0, smin(1.0, s[r]));
}

template <typename L>
static ls_status sat_implicit_t(ls_ctx* c, double dt, ls_solve_info* info) {
    Rows<L> rows;
    rows.mode = 1;
    rows.g = c->g;
    rows.tc = trans_const(c, 1.0);
    rows.sc.phi_dt = c->p.porosity * (1.0 / dt);
    rows.sc.dx = c->p.dx;
    rows.sc.evap = c->p.evaporative_flux;
    rows.sc.dd = make_dxdiv(c->p.dx);
    rows.label = (const L*)c->label;
    rows.fx = c->fx; rows.fy = c->fy; rows.fz = c->fz; rows.s = c->sat;
    const long long sh = c->p.compat_shift ? c->g.JK : 0;
    ls_solve_info loc;
    ls_solve_info* inf[2] = {&loc, nullptr};
    ls_status st = mixed_solve<L>(c, rows, 1, nullptr, nullptr, c->sat + sh, nullptr, c->p.sat_rtol,
                                  c->p.sat_max_it, inf);
    if (info) *info = loc;
    if (st != LS_OK && st != LS_NOT_CONVERGED) return st;
    // physics check and clamp over the voxel slots (src/Simulation.cpp:2007-2047)
    bool valid = !(loc.max_value > 1.05 || loc.min_value < -0.05);
    if (valid) LS_LAUNCH(c, k_clamp_sat, grid_for(c, c->g.N), kBlock, 0, c->g, c->sat);
    if (st == LS_NOT_CONVERGED) return st;
    if (!valid) return set_error(c, LS_UNPHYSICAL, "implicit saturation outside [-0.05, 1.05]");
    return LS_OK;
}

ls_status saturation_implicit_run(ls_ctx* c, double dt, ls_solve_info* info) {
    LS_TRY(flux_zero_now(c));  // after a transport without a flux evaluation since
    snap_fence(c, kSnapSat);
    if (c->label_bytes == 1) return sat_implicit_t<uint8_t>(c, dt, info);
    return sat_implicit_t<uint16_t>(c, dt, info);
}

}  // namespace ls
