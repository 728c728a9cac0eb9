// kernels.cuh -- the residual-and-update kernels.
//
// One residual evaluation (solverCalcR, solver.c:685) is three passes over HBM:
//   k_grad   per cell:  gathers neighbour primitives (ghost states of boundary neighbours are evaluated on
//                       the fly from the cell's own state: a ghost is only ever its owner's neighbour),
//                       least-squares gradient + Venkatakrishnan limiter          (solver.c:451-548)
//   k_flux   per face:  MUSCL states, rotation, Riemann flux * |dS| for interior faces, first-order
//                       boundary fluxes for boundary faces; one launch, block-uniform split (inter 550-644,
//                       boundary.c:143-443)
//   k_rk / k_impl per cell: gathers the signed face fluxes in the reference's order (inter 646-667, then
//                       boundary faces, then the axisymmetric source) and fuses the state update that follows
//                       (solverRK, or the implicit diagonal and DPLUR blocks), the next stage's primitives
//                       with their clamps, local time steps and residual-norm partial sums.
// Nothing is scattered, so no atomics are needed on the state; the only atomics are order-free min/max of
// scalars. Kernels exit immediately once the solve's device status says "done" or "error", so whole
// iteration sequences can be captured in one CUDA graph.
#pragma once
#include "engine.cuh"
#include "launch_rules.h"

namespace csu {

__device__ __forceinline__ bool halted(const Scalars* sc)
{
    return (sc->status | sc->done) != 0;
}

// The halt test of the kernels that, in DPLUR, may run beside the previous iteration's k_finalize (limiter
// bounds, gradients, face fluxes): the flags k_finalize is writing are not read; `frozen` (the flags one
// k_finalize behind) is. A solve halted by iteration i's k_finalize therefore still gets iteration i + 1's
// gradients and face fluxes, of the state it stopped at, and nothing after them: its later iterations
// either skip these kernels or recompute the same values, whichever flag value they read.
__device__ __forceinline__ bool halted_behind(const Prm& p, const Scalars* sc)
{
    return p.defer_fin ? sc->frozen != 0 : halted(sc);
}

// Solve of a cell block (in a pack every block holds cells of one solve) and of a cell; cells of the
// solve are [p.cell0, p.cell0 + p.nc), the rest of its last block is padding.
__device__ __forceinline__ int block_solve(const State& s)
{
    return s.bsolve ? s.bsolve[blockIdx.x] : 0;
}

__device__ __forceinline__ int cell_solve(const State& s, int c)
{
    return s.csolve ? s.csolve[c] : 0;
}

__device__ __forceinline__ bool cell_in(const Prm& p, int c)
{
    return (unsigned)(c - p.cell0) < (unsigned)p.nc;
}

// ------------------------------------------------------------------------------------------------
// k_prim: W = primitives of clamp(U), U := clamp(U) (solverCalcPrimitive cell loop). With dt: the local
// step of the unclamped state first (solverCalcDt precedes solverCalcR, solver.c:1868-1869).
// ------------------------------------------------------------------------------------------------
template <int MODEL>
__global__ void __launch_bounds__(BLOCK) k_prim(const Prm* __restrict__ P, const __grid_constant__ Mesh m,
                                                const __grid_constant__ State s, int with_dt, int only_fresh)
{
    constexpr int NV = Model<MODEL>::NV, NP = Model<MODEL>::NP;
    const int sid = block_solve(s);
    const Prm& p = P[sid];
    Scalars* const sc = s.sc + sid;
    // prologue of a pack: solves carried over from another pack keep their primitives and step
    if (only_fresh && !sc->fresh) return;
    int c = blockIdx.x * BLOCK + threadIdx.x;
    double lmin = __longlong_as_double(0x7ff0000000000000LL);
    if (cell_in(p, c)) {
        double U[NV], P[NP];
        loadU<MODEL>(s, m.nc, c, U);
        if (with_dt) {
            double l = local_step<MODEL>(p, U, m.sxh[c], m.syh[c], m.omega[c]);
            s.dtl[c] = cfl_at(p, sc->iter) * l;
            lmin = l;
        }
        clamp_prim<MODEL>(p, U, P);
        storeU<MODEL>(s, m.nc, c, U);
        storeP<MODEL>(s, m.nc, c, P);
    }
    if (with_dt) {
        double v = block_min(lmin);
        if (threadIdx.x == 0 && !(v > bitsd(0x7fefffffffffffffULL))) atomicMin(&sc->dtmin_bits, dbits(v));
    }
}

// ------------------------------------------------------------------------------------------------
// k_grad: solverUpdateGrad + the limiter loop of inter (solver.c:451-548), one thread per cell and variable (and T in
// viscous models); a block holds GRAD_CELLS cells.
// DBG also records ghost primitives (boundaryCalcPrimitive) in reference order.
// LSQ selects the least-squares arithmetic (Prm::lsq_exact): 0 precomputed FP64 weights, 1 the integer x87
// model (ext80.cuh) for every component, 2 the FP64 x87 emulation and certified double-double solve of
// lsqdd.cuh, with the integer model only for the rare components those cannot decide.
//
// Bound by latency: a thread's chain of dependent FP64 operations and L2 loads. So a thread has one variable (four
// lanes share a cell's double4 records), the certified solve keeps every x87 rounding in its bound instead of in the
// arithmetic (lsq_decide), the two branches of the limiter are one, and the components left undecided (1-3 % of a
// smooth field's, half of a one-directional one's) are finished together, one variable per thread of the block.
// Against one thread per cell with the x87 sums emulated in every component, the rare ones in a kernel behind it:
// 3,049 mixed cells 36.7 -> 14.7 us, 30,000 laminar 37.9 -> 20.8, 160,000 triangles 68 -> 50, 500,000 170 -> 122, the
// 209,825-quad SA plate 109 -> 94 (events, launch gap included; at 160,000 triangles 15 % of the measured copy
// bandwidth for the 50 MB it must move). Measured and dropped, against an earlier 59 us at 160,000 and 147 at 500,000:
// the undecided components where they arise (67 us; a warp has one nearly every time), in a kernel of their own (137 us
// at 500,000, but 28 us at 3,049), on a warp of their own beside the next group's (109 us).
// ------------------------------------------------------------------------------------------------
constexpr int GRAD_CELLS = 32;

// k_lim3: the cell-size factor of limiterCalc's epsilon^2, type 0 (limiter.c:98-119), which no iteration changes.
__global__ void __launch_bounds__(BLOCK) k_lim3(const Prm* __restrict__ P, const __grid_constant__ Mesh m,
                                                const __grid_constant__ State s, double* lim3)
{
    const Prm& p = P[block_solve(s)];
    const int c = blockIdx.x * BLOCK + threadIdx.x;
    if (!cell_in(p, c)) return;
    double aux = p.lim_k * sqrt(m.omega[c] / p.vol_max);
    lim3[c] = aux * aux * aux;
}

// limiterCalc epsilon^2 of slot kk (limiter.c:98-119); aux = (K sqrt(omega / omega_max))^3 for type 0
__device__ __forceinline__ double limiter_eps2(const Prm& p, const Scalars* sc, int kk, double aux)
{
    if (p.limiter_type == 0) return p.pref20[kk] * aux;
    // type 1 (limiter.c:61-94): ((max - min) K)^2 over the solve's cells, from k_minmax
    double a2 = (ordbits_inv(sc->qmax_bits[kk]) - ordbits_inv(sc->qmin_bits[kk])) * p.lim_k;
    return a2 * a2;
}

// The integer x87 model's constants of cell c: a, b, c (exact as double-doubles), det = a c - b b as the host's long
// double rounds it (solver.c:1063-1073), and the reciprocal of its significand.
struct LsqX87 {
    X80 a, b, c, det;
    unsigned long long rv;
};

__device__ __forceinline__ LsqX87 lsq_x87_consts(const Mesh& m, int c)
{
    const double2 qa = m.lq[c], qb = m.lq[m.nc + c], qc = m.lq[2 * m.nc + c];
    LsqX87 K;
    K.a = x80_add(x80_from_double(qa.x), x80_from_double(qa.y));
    K.b = x80_add(x80_from_double(qb.x), x80_from_double(qb.y));
    K.c = x80_add(x80_from_double(qc.x), x80_from_double(qc.y));
    K.det = x80_add(x80_mul(K.a, K.c), x80_neg(x80_mul(K.b, K.b)));
    K.rv = K.det.m ? x80_recip(K.det.m) : 0;
    return K;
}

// Both gradient components of cell c from the differences du(j) of a variable to its neighbours, every operation with
// the integer x87 model: the rare variables nothing else can decide, and every variable with CSU_LSQ=x87. Bound by
// integer issue: the components share the sums, a cell's variables (k_grad with LSQ 1) the constants.
template <typename DU>
__device__ __forceinline__ double2 lsq_x87(const Mesh& m, const LsqX87& K, int c, int np, DU du)
{
    X80 A = x80_zero(0), B = x80_zero(0);
#pragma unroll 1
    for (int j = 0; j < np; j++) {
        const double2 d = m.ld[j * m.nc + c];
        const double v = du(j);
        A = x80_add(A, x80_from_double(d.x * v));
        B = x80_add(B, x80_from_double(d.y * v));
    }
    const X80 nx = x80_add(x80_mul(K.c, A), x80_neg(x80_mul(K.b, B)));
    const X80 ny = x80_add(x80_mul(x80_neg(K.b), A), x80_mul(K.a, B));
    return make_double2(x80_to_double(x80_div_pre(nx, K.det, K.rv)), x80_to_double(x80_div_pre(ny, K.det, K.rv)));
}

// the same from differences in shared memory, out of line: k_grad's undecided variables
static __device__ __noinline__ double2 lsq_x87_left(const Mesh& m, int c, int np, const double* du)
{
    return lsq_x87(m, lsq_x87_consts(m, c), c, np, [=](int j) { return du[j * GRAD_CELLS]; });
}

// ------------------------------------------------------------------------------------------------
// k_minmax: limiterUpdate type 1 (limiter.c:61-94): the minimum and maximum over the solve's cells of each
// limited primitive (slot 4 reads P[5], limiter.c:66-70), as order-preserving bits (exact, order-free).
// k_minmax_init resets them, one block per solve.
// ------------------------------------------------------------------------------------------------
__global__ void k_minmax_init(State s)
{
    Scalars* sc = s.sc + blockIdx.x;
    pdl_wait();
    if (threadIdx.x < 6) {
        sc->qmin_bits[threadIdx.x] = ~0ULL;
        sc->qmax_bits[threadIdx.x] = 0ULL;
    }
}

template <int MODEL>
__global__ void __launch_bounds__(BLOCK) k_minmax(const Prm* __restrict__ P, const __grid_constant__ Mesh m,
                                                  const __grid_constant__ State s)
{
    constexpr int NV = Model<MODEL>::NV, NP = Model<MODEL>::NP;
    const int sid = block_solve(s);
    const Prm& p = P[sid];
    Scalars* const sc = s.sc + sid;
    pdl_wait();
    if (halted_behind(p, sc)) return;
    const int c = blockIdx.x * BLOCK + threadIdx.x;
    const bool ok = cell_in(p, c);
    double W[NP];
    if (ok) loadP<MODEL>(s, m.nc, c, W);
#pragma unroll
    for (int kk = 0; kk < NV; kk++) {
        double v = ok ? W[kk == 4 ? 5 : kk] : 0.0;
        const bool use = ok && !isnan(v); // fmin / fmax skip NaN operands (limiter.c:84-85)
        unsigned long long lo = use ? ordbits(v) : ~0ULL, hi = use ? ordbits(v) : 0ULL;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            lo = min(lo, __shfl_xor_sync(0xffffffffu, lo, o));
            hi = max(hi, __shfl_xor_sync(0xffffffffu, hi, o));
        }
        if ((threadIdx.x & 31) == 0) {
            atomicMin(&sc->qmin_bits[kk], lo);
            atomicMax(&sc->qmax_bits[kk], hi);
        }
    }
}

// The limiter of variable kk of cell c from its final gradient (limiterCalc, limiter.c:98-119), and their stores;
// kk == NV: the temperature gradient. d1min, d1max: the variable's largest decrease and increase to a neighbour.
template <int MODEL>
__device__ __forceinline__ void grad_finish(const Prm& p, const Mesh& m, const State& s, const Scalars* sc, int c,
                                            int kk, int np, double gx, double gy, double d1min, double d1max)
{
    constexpr int NV = Model<MODEL>::NV;
    const int nc = m.nc;
    if (kk == NV) {
        s.GTx[c] = gx;
        s.GTy[c] = gy;
        return;
    }
    double phi = 1.0;
    if (p.order == 2) {
        const double ee = limiter_eps2(p, sc, kk, m.lim3[c]);
#pragma unroll
        for (int j = 0; j < 4; j++) {
            if (j < 3 || np > 3) {
                const double2 e = m.em[j * nc + c];
                const double d2 = (gx * e.x + gy * e.y);
                const double phi0 = p.lim_func == 1 ? limiterBJ(d1min, d1max, d2) : limiterV2(d1min, d1max, d2, ee);
                phi = j == 0 ? phi0 : fmin(phi, phi0);
            }
        }
    }
    if (kk < 4) {
        reinterpret_cast<double*>(s.G4x + c)[kk] = gx;
        reinterpret_cast<double*>(s.G4y + c)[kk] = gy;
        reinterpret_cast<double*>(s.PH4 + c)[kk] = phi;
    } else {
        const size_t o = (size_t)(kk - 4) * nc + c;
        s.Gxx[o] = gx;
        s.Gxy[o] = gy;
        s.PHx[o] = phi;
    }
}

// Blocks per SM of k_grad's register budget (64 registers; SST 72): with fewer the loads' latency shows (160,000
// triangles, Euler: 4 blocks 68 us, 5 61, 6 59), with more the undecided components' code spills into the rest (8: 71).
// SMALL: small meshes' undecided components without spills (grad_small). LSQ 1: 80 registers (200,000 cells, RK5 with
// CSU_LSQ=x87: 922 us an iteration; two blocks of 96 registers 1,025).
template <int MODEL, int LSQ, bool SMALL>
constexpr int grad_blocks()
{
    if (LSQ == 1) return 800 / (GRAD_CELLS * (Model<MODEL>::NV + 1));
    return SMALL ? 2 : MODEL == 0 ? 6 : (MODEL == 1 ? 5 : 4);
}

template <int MODEL, bool DBG, int LSQ, bool SMALL = false>
__global__ void __launch_bounds__(GRAD_CELLS * (Model<MODEL>::NV + 1), grad_blocks<MODEL, LSQ, SMALL>())
    k_grad(const Prm* __restrict__ P, const __grid_constant__ Mesh m, const __grid_constant__ State s)
{
    constexpr int NV = Model<MODEL>::NV, NP = Model<MODEL>::NP;
    static_assert(GRAD_CELLS == 32 && BLOCK % GRAD_CELLS == 0, "blocks tile the cell blocks");
    // undecided variables: differences, range, components; list of lane (cell of the block) | variable << 5 | mask << 8
    __shared__ double sdu[LSQ == 2 ? NV + 1 : 1][8][GRAD_CELLS];
    __shared__ unsigned short list[LSQ == 2 ? (NV + 1) * GRAD_CELLS : 1];
    __shared__ unsigned nlist;
    __shared__ LsqX87 sk[LSQ == 1 ? GRAD_CELLS : 1];
    const int sid = s.bsolve ? s.bsolve[blockIdx.x / (BLOCK / GRAD_CELLS)] : 0;
    const Prm& p = P[sid];
    const Scalars* const sc = s.sc + sid;
    // four lanes per cell for r u v p, whose records are double4; a warp each for the scalars and T
    const int kk = threadIdx.x < 4 * GRAD_CELLS ? threadIdx.x & 3 : threadIdx.x >> 5; // variable slot; NV: T
    const int lane = threadIdx.x < 4 * GRAD_CELLS ? threadIdx.x >> 2 : threadIdx.x & 31;
    const int vi = kk < NV ? slot2p(kk) : 4;
    const int c = blockIdx.x * GRAD_CELLS + lane;
    const int nc = m.nc; // 4 nc < 2^31
    if (LSQ == 2 && threadIdx.x == 0) nlist = 0;
    if (LSQ == 2) __syncthreads();
    // the mesh rows before the wait for the previous kernel (padding rows are in bounds and hold zeros)
    const double* const W = kk < 4 ? reinterpret_cast<const double*>(s.W4) + kk
                                   : vi == 4 ? s.WT : s.Wx + (size_t)(vi - 5) * nc;
    const int ws = kk < 4 ? 4 : 1;
    const int cr = min(c, nc - 1), np = m.npts[cr];
    int nj[4];
    double2 d[4];
#pragma unroll
    for (int j = 0; j < 4; j++) {
        nj[j] = cr;
        if (j < 3 || np > 3) {
            nj[j] = m.nei[j * nc + cr];
            d[j] = (LSQ == 0 ? m.lw : m.ld)[j * nc + cr];
        }
    }
    if (LSQ == 1) {
        // padding rows hold zeros, whose constants nothing reads
        if (threadIdx.x < GRAD_CELLS)
            sk[threadIdx.x] = lsq_x87_consts(m, min(blockIdx.x * GRAD_CELLS + threadIdx.x, nc - 1));
        __syncthreads();
    }
    pdl_wait();
    const bool stop = halted_behind(p, sc);
    const double u0 = W[(size_t)cr * ws];
    double un[4];
    unsigned ghosts = 0;
#pragma unroll
    for (int j = 0; j < 4; j++) {
        un[j] = W[(size_t)(nj[j] < nc ? nj[j] : cr) * ws];
        if (nj[j] >= nc) ghosts |= 1u << j;
    }
    if (cell_in(p, c) && !stop) {
        if (ghosts) {
            double P0[NP], Pn[NP];
            loadP<MODEL>(s, nc, c, P0);
            const double dw = m.wall_d ? m.wall_d[c] : 0.0;
#pragma unroll 1
            while (ghosts) {
                const int j = __ffs(ghosts) - 1;
                ghosts &= ghosts - 1;
                const int b = (j == 0 ? nj[0] : j == 1 ? nj[1] : j == 2 ? nj[2] : nj[3]) - nc;
                double2 dSv = m.bn[b];
                ghost_state<MODEL>(p, m.bflag[b], dSv.x, dSv.y, m.bds[b], P0, dw, Pn);
                if (DBG && kk == 0) {
                    int bo = m.bold[b];
                    for (int k = 0; k < NP; k++) s.dbg_ghost[(size_t)bo * NP + k] = Pn[k];
                }
                double v = Pn[0];
#pragma unroll
                for (int k = 1; k < NP; k++)
                    if (k == vi) v = Pn[k];
#pragma unroll
                for (int q = 0; q < 4; q++)
                    if (q == j) un[q] = v;
            }
        }
        double gx = 0.0, gy = 0.0, qmin = u0, qmax = u0, du[4];
#pragma unroll
        for (int j = 0; j < 4; j++) {
            qmax = un[j] > qmax ? un[j] : qmax;
            qmin = un[j] < qmin ? un[j] : qmin;
            du[j] = un[j] - u0;
        }
        const double d1max = qmax - u0, d1min = qmin - u0;
        unsigned need = 0; // bits 0 (x) and 1 (y) set where the certified solve cannot decide
        if (LSQ == 0) {
#pragma unroll
            for (int j = 0; j < 4; j++) {
                if (j < 3 || np > 3) {
                    gx += d[j].x * du[j];
                    gy += d[j].y * du[j];
                }
            }
        } else if (LSQ == 1) {
            const double2 g = lsq_x87(m, sk[lane], c, np, [&](int j) {
                return j == 0 ? du[0] : j == 1 ? du[1] : j == 2 ? du[2] : du[3];
            });
            gx = g.x;
            gy = g.y;
        } else {
            // solverCalcGrad3 (solver.c:1063-1073): double products summed in long double, then
            // dUx = (c A - b B) / (a c - b b), dUy = (-b A + a B) / (a c - b b) in long double
            LsqSum X = lsq_sum2(d[0].x * du[0], d[1].x * du[1]), Y = lsq_sum2(d[0].y * du[0], d[1].y * du[1]);
            lsq_sum_add(X, d[2].x * du[2]);
            lsq_sum_add(Y, d[2].y * du[2]);
            if (np > 3) {
                lsq_sum_add(X, d[3].x * du[3]);
                lsq_sum_add(Y, d[3].y * du[3]);
            }
            const double2 qa = m.lk[c], qb = m.lk[nc + c], qc = m.lk[2 * nc + c];
            const DD ka = {qa.x, qa.y}, kb = {qb.x, qb.y}, kc = {qc.x, qc.y};
            need = lsq_decide(kc, kb, X, Y, &gx) ? 0u : 1u;
            if (!lsq_decide(ka, kb, Y, X, &gy)) need |= 2u;
            if (need) {
                list[atomicAdd(&nlist, 1u)] = (unsigned short)(lane | kk << 5 | need << 8);
#pragma unroll
                for (int j = 0; j < 4; j++) sdu[kk][j][lane] = du[j];
                sdu[kk][4][lane] = d1min;
                sdu[kk][5][lane] = d1max;
                sdu[kk][6][lane] = gx;
                sdu[kk][7][lane] = gy;
            }
        }
        if (!need) grad_finish<MODEL>(p, m, s, sc, c, kk, np, gx, gy, d1min, d1max);
    }
    if (LSQ == 2) {
        // The undecided variables of the whole block, one per thread: the x87 sums and the numerator exactly, and the
        // integer model for what that cannot decide either. Done where they arise they would cost nearly every
        // warp a pass through this code for one or two lanes.
        __syncthreads();
        const unsigned n = nlist;
#pragma unroll 1
        for (unsigned e = threadIdx.x; e < n; e += blockDim.x) {
            const unsigned w = list[e];
            const int l = w & 31u, q = (w >> 5) & 7u, c2 = blockIdx.x * GRAD_CELLS + l, np = m.npts[c2];
            bool ok = true;
            const double2 d0 = m.ld[c2], d1 = m.ld[nc + c2];
            const double v0 = sdu[q][0][l], v1 = sdu[q][1][l];
            DD X = x87_sum2(d0.x * v0, d1.x * v1, ok), Y = x87_sum2(d0.y * v0, d1.y * v1, ok);
#pragma unroll 1
            for (int j = 2; j < np; j++) {
                const double2 dj = m.ld[j * nc + c2];
                const double v = sdu[q][j][l];
                X = x87_sum_add(X, dj.x * v, ok);
                Y = x87_sum_add(Y, dj.y * v, ok);
            }
            const double2 qb = m.lq[nc + c2], qr = m.lq[3 * nc + c2];
            const DD kb = {qb.x, qb.y}, R = {qr.x, qr.y};
            double gx = sdu[q][6][l], gy = sdu[q][7][l];
            bool left = false; // either component left to the integer model: the variable counts once
#pragma unroll 1
            for (unsigned nd = w >> 8; nd; nd &= nd - 1) {
                const bool y = (nd & 1u) == 0;
                const double2 qk = m.lq[(y ? 0 : 2) * nc + c2];
                const DD k1 = {qk.x, qk.y};
                double g = 0.0;
                if (!ok || !lsq_exact_numerator(k1, kb, R, y ? Y : X, y ? X : Y, &g)) {
                    const double2 g2 = lsq_x87_left(m, c2, np, &sdu[q][0][l]);
                    g = y ? g2.y : g2.x;
                    left = true;
                }
                if (y) gy = g;
                else gx = g;
            }
            if (left) atomicAdd(s.lsq_x87, 1ULL);
            grad_finish<MODEL>(p, m, s, sc, c2, q, np, gx, gy, sdu[q][4][l], sdu[q][5][l]);
        }
    }
}

// The owner's gradients a boundary face's viscous flux uses: u, v, T, then nt (SA) or k (SST), then the rho
// gradient (SA: saCC's density terms) or omega (SST).
template <int MODEL>
__device__ __forceinline__ void owner_visc_gradients(const State& s, int nc, int c, double* gvx, double* gvy)
{
    double4 a = ld4(s.G4x + c), bb = ld4(s.G4y + c);
    gvx[0] = a.y; gvx[1] = a.z; gvx[2] = s.GTx[c];
    gvy[0] = bb.y; gvy[1] = bb.z; gvy[2] = s.GTy[c];
    gvx[3] = MODEL >= 1 ? s.Gxx[c] : 0.0;
    gvy[3] = MODEL >= 1 ? s.Gxy[c] : 0.0;
    gvx[4] = MODEL == 2 ? s.Gxx[(size_t)nc + c] : (MODEL == 1 ? a.x : 0.0);
    gvy[4] = MODEL == 2 ? s.Gxy[(size_t)nc + c] : (MODEL == 1 ? bb.x : 0.0);
}

// Viscous flux of boundary face b (device order; fi its slot in the face arrays) from its owner c's
// primitives E0 and gradients: boundaryFaceViscFlux (laminar.c:128-346), saBoundaryFaceViscFlux (sa.c:370-692)
// or its saCC variant, sstBoundaryFaceViscFlux (sst.c:202-547); stored in FV (and FV5) at fi.
template <int MODEL>
__device__ __forceinline__ void bface_visc(const Prm& p, const Mesh& m, const State& s, int b, int fi, int c,
                                           int flag, double dSx, double dSy, const double* E0, const double* gvx,
                                           const double* gvy, double2 bdv, double bLv)
{
    if constexpr (MODEL == 2) {
        double2 un = m.bun[b];
        double fv[5];
        sst_boundary_flux(p.gas, p.sst_k, p.pr, p.pr_t, p.t_wall, p.pin, flag, gvx, gvy, E0, m.wall_d[c], dSx, dSy,
                          bdv.x, bdv.y, bLv, un.x, un.y, m.bds2[b], fv);
        st4(s.FV + fi, make_double4(fv[0], fv[1], fv[2], fv[3]));
        s.FV5[fi] = fv[4];
    } else if constexpr (MODEL == 1) {
        double2 un = m.bun[b];
        double fv[4];
        if (p.sa_cc)
            sacc_boundary_flux(p.gas, p.pr, p.pr_t, p.t_wall, p.pin, flag, gvx, gvy, E0, dSx, dSy, bdv.x, bdv.y,
                               bLv, un.x, un.y, m.bds2[b], fv);
        else
            sa_boundary_flux(p.gas, p.pr, p.pr_t, p.t_wall, p.pin, flag, gvx, gvy, E0, dSx, dSy, bdv.x, bdv.y, bLv,
                             un.x, un.y, m.bds2[b], fv);
        st4(s.FV + fi, make_double4(fv[0], fv[1], fv[2], fv[3]));
    } else {
        if (p.laminar == 1) {
            double2 un = m.bun[b];
            double fv[3];
            laminar_boundary(p.gas, p.pr, p.t_wall, p.pin, flag, gvx, gvy, E0, dSx, dSy, bdv.x, bdv.y, bLv, un.x,
                             un.y, m.bds2[b], fv);
            st4(s.FV + fi, make_double4(fv[0], fv[1], fv[2], 0.0));
        }
    }
}

// ------------------------------------------------------------------------------------------------
// k_wall_data: what the reference's surface writers read after its last iteration (solverWriteSolution2
// recomputes the cell and ghost primitives of the final state, solver.c:2038, while the gradients stay
// those of the last residual evaluation): per boundary face, the ghost primitives of the current cell
// primitives (into dbg_ghost, reference order) and the boundary viscous flux of the current primitives and
// gradients (into FV).
// ------------------------------------------------------------------------------------------------
template <int MODEL>
__global__ void __launch_bounds__(BLOCK) k_wall_data(const Prm* __restrict__ P, const __grid_constant__ Mesh m,
                                                     const __grid_constant__ State s)
{
    constexpr int NP = Model<MODEL>::NP;
    const int b = blockIdx.x * BLOCK + threadIdx.x;
    if (b >= m.nb) return;
    const int nc = m.nc, c = m.bown[b];
    const Prm& p = P[cell_solve(s, c)];
    const int flag = m.bflag[b];
    const double2 dSv = m.bn[b];
    const double dSx = dSv.x, dSy = dSv.y, dS = m.bds[b];
    double E0[NP], G[NP];
    loadP<MODEL>(s, nc, c, E0);
    ghost_state<MODEL>(p, flag, dSx, dSy, dS, E0, m.wall_d ? m.wall_d[c] : 0.0, G);
    const int bo = m.bold[b];
#pragma unroll
    for (int k = 0; k < NP; k++) s.dbg_ghost[(size_t)bo * NP + k] = G[k];
    if (p.visc) {
        double gvx[5], gvy[5];
        owner_visc_gradients<MODEL>(s, nc, c, gvx, gvy);
        bface_visc<MODEL>(p, m, s, b, m.nf + b, c, flag, dSx, dSy, E0, gvx, gvy, m.bd[b], m.bL[b]);
    }
}

// One interior face of k_flux (inter, solver.c:550-644, and the viscous face terms): MUSCL reconstruction,
// rotation, Riemann flux times |dS|, and the face's viscous flux and eddy viscosity. The two cells'
// primitives r u v p T, gradients and limiters of r u v p come in as values (read from global memory, or
// from a shared-memory window of cells); everything else is read here.
template <int MODEL>
__device__ __forceinline__ void interior_face(const Prm& p, const Mesh& m, const State& s, int f, int2 e,
                                              double4 w0, double t0, double4 gx0, double4 gy0, double4 ph0,
                                              double4 w1, double t1, double4 gx1, double4 gy1, double4 ph1)
{
    constexpr int NV = Model<MODEL>::NV, NP = Model<MODEL>::NP;
    const int nc = m.nc;
    double2 dSv = m.fn[f];
    double dSx = dSv.x, dSy = dSv.y, dS = m.fds[f];
    double PL[6] = {0.0, 0.0, 0.0, 0.0, 0.0, 0.0};
    double PR[6] = {0.0, 0.0, 0.0, 0.0, 0.0, 0.0};
    double A[NP], B[NP];
    A[0] = w0.x; A[1] = w0.y; A[2] = w0.z; A[3] = w0.w; A[4] = t0;
    B[0] = w1.x; B[1] = w1.y; B[2] = w1.z; B[3] = w1.w; B[4] = t1;
#pragma unroll
    for (int k = 5; k < NP; k++) {
        A[k] = s.Wx[(size_t)(k - 5) * nc + e.x];
        B[k] = s.Wx[(size_t)(k - 5) * nc + e.y];
    }
    if (p.order == 2) {
        double2 r0 = m.r0[f], r1 = m.r1[f];
        double g0x[4] = {gx0.x, gx0.y, gx0.z, gx0.w}, g0y[4] = {gy0.x, gy0.y, gy0.z, gy0.w};
        double g1x[4] = {gx1.x, gx1.y, gx1.z, gx1.w}, g1y[4] = {gy1.x, gy1.y, gy1.z, gy1.w};
        double f0[4] = {ph0.x, ph0.y, ph0.z, ph0.w}, f1[4] = {ph1.x, ph1.y, ph1.z, ph1.w};
#pragma unroll
        for (int kk = 0; kk < 4; kk++) {
            PL[kk] = A[kk] + (g0x[kk] * r0.x + g0y[kk] * r0.y) * f0[kk];
            PR[kk] = B[kk] + (g1x[kk] * r1.x + g1y[kk] * r1.y) * f1[kk];
        }
#pragma unroll
        for (int kk = 4; kk < NV; kk++) {
            if (p.turb1order) {
                PL[kk] = A[kk + 1];
                PR[kk] = B[kk + 1];
            } else {
                size_t o = (size_t)(kk - 4) * nc;
                PL[kk] = A[kk + 1] + (s.Gxx[o + e.x] * r0.x + s.Gxy[o + e.x] * r0.y) * s.PHx[o + e.x];
                PR[kk] = B[kk + 1] + (s.Gxx[o + e.y] * r1.x + s.Gxy[o + e.y] * r1.y) * s.PHx[o + e.y];
            }
        }
    } else {
#pragma unroll
        for (int kk = 0; kk < NV; kk++) {
            PL[kk] = A[slot2p(kk)];
            PR[kk] = B[slot2p(kk)];
        }
    }
    if constexpr (MODEL == 2) {
        const double4 a = gx0, b = gy0, cc = gx1, d = gy1;
        double g0x[5] = {a.y, a.z, s.GTx[e.x], s.Gxx[e.x], s.Gxx[(size_t)nc + e.x]};
        double g0y[5] = {b.y, b.z, s.GTy[e.x], s.Gxy[e.x], s.Gxy[(size_t)nc + e.x]};
        double g1x[5] = {cc.y, cc.z, s.GTx[e.y], s.Gxx[e.y], s.Gxx[(size_t)nc + e.y]};
        double g1y[5] = {d.y, d.z, s.GTy[e.y], s.Gxy[e.y], s.Gxy[(size_t)nc + e.y]};
        double2 dd = m.fd[f];
        double fv[5], mit;
        sst_face_flux(p.gas, p.sst_k, p.pr, p.pr_t, g0x, g0y, g1x, g1y, A, B, m.wall_d[e.x], m.wall_d[e.y], dd.x,
                      dd.y, m.fL[f], dSx, dSy, fv, &mit);
        st4(s.FV + f, make_double4(fv[0], fv[1], fv[2], fv[3]));
        s.FV5[f] = fv[4];
        s.MIT[f] = mit;
    } else if constexpr (MODEL == 1) {
        const double4 a = gx0, b = gy0, cc = gx1, d = gy1;
        double g0x[5] = {a.y, a.z, s.GTx[e.x], s.Gxx[e.x], a.x}, g0y[5] = {b.y, b.z, s.GTy[e.x], s.Gxy[e.x], b.x};
        double g1x[5] = {cc.y, cc.z, s.GTx[e.y], s.Gxx[e.y], cc.x}, g1y[5] = {d.y, d.z, s.GTy[e.y], s.Gxy[e.y], d.x};
        double2 dd = m.fd[f];
        double fv[4], mit;
        if (p.sa_cc)
            sacc_face_flux(p.gas, p.pr, p.pr_t, g0x, g0y, g1x, g1y, A, B, dSx, dSy, fv, &mit);
        else
            sa_face_flux(p.gas, p.pr, p.pr_t, p.visc_blazek, g0x, g0y, g1x, g1y, A, B, dd.x, dd.y, m.fL[f], dSx,
                         dSy, fv, &mit);
        st4(s.FV + f, make_double4(fv[0], fv[1], fv[2], fv[3]));
        if (!p.mit_early) s.MIT[f] = mit;
    } else if (p.laminar == 1) {
        const double4 a = gx0, b = gy0, cc = gx1, d = gy1;
        double g0x[3] = {a.y, a.z, s.GTx[e.x]}, g0y[3] = {b.y, b.z, s.GTy[e.x]};
        double g1x[3] = {cc.y, cc.z, s.GTx[e.y]}, g1y[3] = {d.y, d.z, s.GTy[e.y]};
        double2 dd = m.fd[f];
        double fv[3];
        laminar_face(p.gas, p.pr, g0x, g0y, g1x, g1y, A, B, dd.x, dd.y, m.fL[f], dSx, dSy, fv);
        st4(s.FV + f, make_double4(fv[0], fv[1], fv[2], 0.0));
    }
    rotation(PL, dSx, dSy, dS);
    rotation(PR, dSx, dSy, dS);
    double fl[NV];
    riemann<MODEL>(p.scheme, p.gas, p.e_fix, p.mach_inf, PL, PR, fl);
    rotation(fl, dSx, -dSy, dS);
    st4(s.F4 + f, make_double4(fl[0] * dS, fl[1] * dS, fl[2] * dS, fl[3] * dS));
#pragma unroll
    for (int kk = 4; kk < NV; kk++) s.Fx[(size_t)(kk - 4) * (m.nf + m.nb) + f] = fl[kk] * dS;
}

// One boundary face b of k_flux (device order): the boundary flux of boundary.c:143-464 from the owner's
// first-order state and the ghost, the face's viscous flux, and the wall pressure and friction terms of
// solverCalcCoeff3 when `coef`.
template <int MODEL>
__device__ __forceinline__ void boundary_face(const Prm* __restrict__ P, const Mesh& m, const State& s, int b,
                                              const int* wall_rank, int coef)
{
    constexpr int NV = Model<MODEL>::NV, NP = Model<MODEL>::NP;
    const int nc = m.nc;
    int c = m.bown[b];
    const int sid = cell_solve(s, c);
    const Prm& p = P[sid];
    if (halted_behind(p, s.sc + sid)) return;
    int flag = m.bflag[b];
    double2 dSv = m.bn[b];
    double dSx = dSv.x, dSy = dSv.y, dS = m.bds[b];
    double E0[NP];
    loadP<MODEL>(s, nc, c, E0);
    double fl[NV];
    boundary_flux<MODEL>(p, flag, dSx, dSy, dS, E0, fl);
    int fi = m.nf + b;
    double sc = dS > 0 ? dS : 0.0;
    st4(s.F4 + fi, dS > 0 ? make_double4(fl[0] * dS, fl[1] * dS, fl[2] * dS, fl[3] * dS)
                          : make_double4(0.0, 0.0, 0.0, 0.0));
#pragma unroll
    for (int kk = 4; kk < NV; kk++) s.Fx[(size_t)(kk - 4) * (m.nf + m.nb) + fi] = dS > 0 ? fl[kk] * sc : 0.0;
    double gvx[5], gvy[5];
    double2 bdv = make_double2(0.0, 0.0);
    double bLv = 0.0;
    if (p.visc) {
        owner_visc_gradients<MODEL>(s, nc, c, gvx, gvy);
        bdv = m.bd[b];
        bLv = m.bL[b];
        bface_visc<MODEL>(p, m, s, b, fi, c, flag, dSx, dSy, E0, gvx, gvy, bdv, bLv);
    }
    if (coef && (flag == 3 || flag == 4)) {
        double* const bc = coef == 2 ? s.bcoef2 : s.bcoef;
        double G[NP];
        ghost_state<MODEL>(p, flag, dSx, dSy, dS, E0, m.wall_d ? m.wall_d[c] : 0.0, G);
        double cp = (G[3] - p.p_inf) / p.q_inf;
        int r = wall_rank[b];
        bc[(size_t)r * 4 + 0] = cp * dSx;
        bc[(size_t)r * 4 + 1] = cp * dSy;
        double fx = 0.0, fy = 0.0;
        if (p.visc) friction_wall(gvx, gvy, E0, dSx, dSy, bdv.x, bdv.y, bLv, &fx, &fy);
        bc[(size_t)r * 4 + 2] = p.visc ? fx / p.q_inf : 0.0;
        bc[(size_t)r * 4 + 3] = p.visc ? fy / p.q_inf : 0.0;
    }
}

// ------------------------------------------------------------------------------------------------
// k_flux: interior faces (blocks [0, nbi)) and boundary faces (blocks [nbi, ...)).
// coef: also record the wall pressure-coefficient terms of solverCalcCoeff3 (solver.c:1360-1385).
// ------------------------------------------------------------------------------------------------
template <int MODEL, int FB>
__global__ void __launch_bounds__(FB) k_flux(const Prm* __restrict__ P, const __grid_constant__ Mesh m,
                                             const __grid_constant__ State s, int nbi, const int* wall_rank,
                                             int coef)
{
    if ((int)blockIdx.x < nbi) {
        int f = blockIdx.x * FB + threadIdx.x;
        if (f >= m.nf) return;
        int2 e = m.fe[f];
        const int sid = cell_solve(s, e.x);
        const Prm& p = P[sid];
        const bool o2 = p.order == 2, grad = o2 || p.visc;
        prefetch_l1(m.fn + f);
        prefetch_l1(m.fds + f);
        if (o2) {
            prefetch_l1(m.r0 + f);
            prefetch_l1(m.r1 + f);
        }
        pdl_wait();
        if (halted_behind(p, s.sc + sid)) return;
        const double4 z4 = make_double4(0.0, 0.0, 0.0, 0.0);
        interior_face<MODEL>(p, m, s, f, e, ld4(s.W4 + e.x), s.WT[e.x], grad ? ld4(s.G4x + e.x) : z4,
                             grad ? ld4(s.G4y + e.x) : z4, o2 ? ld4(s.PH4 + e.x) : z4, ld4(s.W4 + e.y), s.WT[e.y],
                             grad ? ld4(s.G4x + e.y) : z4, grad ? ld4(s.G4y + e.y) : z4, o2 ? ld4(s.PH4 + e.y) : z4);
    } else {
        int b = (blockIdx.x - nbi) * FB + threadIdx.x;
        if (b >= m.nb) return;
        pdl_wait();
        boundary_face<MODEL>(P, m, s, b, wall_rank, coef);
    }
}

// ------------------------------------------------------------------------------------------------
// k_flux_st: k_flux with the interior faces' cell data staged in shared memory. Faces are sorted by their
// lower cell, so a block of FB faces starts at its first face's lower cell and most of its cells, both
// sides, lie in the next WIN cells (94 % of the faces on the 160,000-cell ramp for FB 128, WIN 256). The
// block loads that window's primitives r u v p T (and, when the faces need them, gradients and limiters of
// r u v p) with coalesced loads, then each face reads its cells from the window, or from global memory when
// a cell lies outside it. Same arithmetic, same bits as k_flux; the boundary faces are k_flux's.
// ------------------------------------------------------------------------------------------------
template <int MODEL, int FB, int WIN>
__global__ void __launch_bounds__(FB) k_flux_st(const Prm* __restrict__ P, const __grid_constant__ Mesh m,
                                                const __grid_constant__ State s, int nbi, const int* wall_rank,
                                                int coef)
{
    pdl_wait();
    if ((int)blockIdx.x >= nbi) {
        const int b = (blockIdx.x - nbi) * FB + threadIdx.x;
        if (b < m.nb) boundary_face<MODEL>(P, m, s, b, wall_rank, coef);
        return;
    }
    __shared__ double4 sw[WIN], sgx[WIN], sgy[WIN], sph[WIN];
    __shared__ double st[WIN];
    const int nc = m.nc;
    const int f0 = blockIdx.x * FB;
    const int f = f0 + threadIdx.x;
    const int2 e0 = m.fe[f0];
    const int base = min(e0.x, e0.y);
    // order and viscosity are shared by every solve of a pack
    const bool o2 = P[0].order == 2, grad = o2 || P[0].visc;
    for (int i = threadIdx.x; i < WIN; i += FB) {
        const int c = base + i;
        if (c < nc) {
            sw[i] = ld4(s.W4 + c);
            st[i] = s.WT[c];
            if (grad) {
                sgx[i] = ld4(s.G4x + c);
                sgy[i] = ld4(s.G4y + c);
            }
            if (o2) sph[i] = ld4(s.PH4 + c);
        }
    }
    __syncthreads();
    if (f >= m.nf) return;
    const int2 e = m.fe[f];
    const int sid = cell_solve(s, e.x);
    const Prm& p = P[sid];
    if (halted_behind(p, s.sc + sid)) return;
    const double4 z4 = make_double4(0.0, 0.0, 0.0, 0.0);
    const unsigned i0 = (unsigned)(e.x - base), i1 = (unsigned)(e.y - base);
    const bool in0 = i0 < (unsigned)WIN, in1 = i1 < (unsigned)WIN;
    const double4 w0 = in0 ? sw[i0] : ld4(s.W4 + e.x), w1 = in1 ? sw[i1] : ld4(s.W4 + e.y);
    const double t0 = in0 ? st[i0] : s.WT[e.x], t1 = in1 ? st[i1] : s.WT[e.y];
    double4 gx0 = z4, gy0 = z4, gx1 = z4, gy1 = z4, ph0 = z4, ph1 = z4;
    if (grad) {
        gx0 = in0 ? sgx[i0] : ld4(s.G4x + e.x);
        gy0 = in0 ? sgy[i0] : ld4(s.G4y + e.x);
        gx1 = in1 ? sgx[i1] : ld4(s.G4x + e.y);
        gy1 = in1 ? sgy[i1] : ld4(s.G4y + e.y);
    }
    if (o2) {
        ph0 = in0 ? sph[i0] : ld4(s.PH4 + e.x);
        ph1 = in1 ? sph[i1] : ld4(s.PH4 + e.y);
    }
    interior_face<MODEL>(p, m, s, f, e, w0, t0, gx0, gy0, ph0, w1, t1, gx1, gy1, ph1);
}

// Sum of the signed face fluxes of one cell in the reference's order (inter, then boundary, then the
// axisymmetric pressure source interAxisPressure, solver.c:646-683).
template <int MODEL>
__device__ __forceinline__ void gather_residual(const Prm& p, const Mesh& m, const State& s, int c, const double* P,
                                                double* R)
{
    constexpr int NV = Model<MODEL>::NV;
    const int nc = m.nc, nft = m.nf + m.nb;
#pragma unroll
    for (int k = 0; k < NV; k++) R[k] = 0.0;
    const int ns = m.nslot[c];
#pragma unroll
    for (int j = 0; j < 4; j++) {
        if (j < ns) {
            int sf = m.fslot[(size_t)j * nc + c];
            int fi = sf > 0 ? sf - 1 : -sf - 1;
            double4 F = ld4(s.F4 + fi);
            double fv[NV];
            fv[0] = F.x; fv[1] = F.y; fv[2] = F.z; fv[3] = F.w;
#pragma unroll
            for (int k = 4; k < NV; k++) fv[k] = s.Fx[(size_t)(k - 4) * nft + fi];
            if (sf > 0) {
#pragma unroll
                for (int k = 0; k < NV; k++) R[k] += fv[k];
            } else {
#pragma unroll
                for (int k = 0; k < NV; k++) R[k] -= fv[k];
            }
        }
    }
    if (p.axi == 1) {
        double dS = m.dslat[c];
        R[2] -= P[3] * dS;
        if constexpr (MODEL == 2) R[2] -= (2. / 3.) * P[0] * P[5] * dS;
    }
    if (p.laminar == 1 || MODEL >= 1) {
        // laminarInter / saInter face gather (laminar.c:77-98, sa.c:197-220), the SA source (sa.c:224-256),
        // then laminarBoundary / saBoundary (laminar.c:101-125, sa.c:351-368, 695-701)
        const int ni = m.nint[c];
#pragma unroll
        for (int j = 0; j < 4; j++) {
            if (j < ni) {
                int sf = m.fslot[(size_t)j * nc + c];
                int fi = sf > 0 ? sf - 1 : -sf - 1;
                double4 V = ld4(s.FV + fi);
                if (sf > 0) {
                    R[1] -= V.x;
                    R[2] -= V.y;
                    R[3] -= V.z;
                    if constexpr (MODEL >= 1) R[4] -= V.w;
                    if constexpr (MODEL == 2) R[5] -= s.FV5[fi];
                } else {
                    R[1] += V.x;
                    R[2] += V.y;
                    R[3] += V.z;
                    if constexpr (MODEL >= 1) R[4] += V.w;
                    if constexpr (MODEL == 2) R[5] += s.FV5[fi];
                }
            }
        }
        if constexpr (MODEL == 1) {
            double4 gx = ld4(s.G4x + c), gy = ld4(s.G4y + c);
            double rho = P[0], T = P[4], n = P[5];
            double d = m.wall_d[c];
            double mi_L = sutherland(T);
            double n_L = mi_L / rho;
            double S = fabs(gy.y - gx.z);
            double Qt = p.sa_cc ? sacc_source(n, n_L, S, d, rho, gx.x, gy.x, s.Gxx[c], s.Gxy[c])
                                : sa_source(n, n_L, S, d, rho, gx.x, gy.x, s.Gxx[c], s.Gxy[c]);
            R[4] -= Qt * m.omega[c];
        }
        if constexpr (MODEL == 2) {
            double4 gx = ld4(s.G4x + c), gy = ld4(s.G4y + c);
            double sgx[4] = {gx.y, gx.z, s.Gxx[c], s.Gxx[(size_t)nc + c]};
            double sgy[4] = {gy.y, gy.z, s.Gxy[c], s.Gxy[(size_t)nc + c]};
            double Qtk, Qto;
            sst_cell_source(p.sst_k, sgx, sgy, P, m.wall_d[c], &Qtk, &Qto);
            if (P[6] != 0.0) {
                R[4] -= Qtk * m.omega[c];
                R[5] -= Qto * m.omega[c];
            }
        }
#pragma unroll
        for (int j = 0; j < 4; j++) {
            if (j >= ni && j < ns) {
                int fi = m.fslot[(size_t)j * nc + c] - 1;
                double4 V = ld4(s.FV + fi);
                R[1] -= V.x;
                R[2] -= V.y;
                R[3] -= V.z;
                if constexpr (MODEL >= 1) R[4] -= V.w;
                if constexpr (MODEL == 2) R[5] -= s.FV5[fi];
            }
        }
    }
}

template <int MODEL>
__device__ __forceinline__ void storeR(const State& s, int nc, int c, const double* R)
{
    st4(s.R4 + c, make_double4(R[0], R[1], R[2], R[3]));
#pragma unroll
    for (int k = 4; k < Model<MODEL>::NV; k++) s.Rx[(size_t)(k - 4) * nc + c] = R[k];
}

// the block's sum of R^2 per variable into s.part[blockIdx.x]: one row per cell block of NT cells (k_finalize
// is told how many rows a BLOCK-cell block has)
template <int MODEL, int NT = BLOCK>
__device__ __forceinline__ void partial_norms(const State& s, bool valid, const double* R)
{
    constexpr int NV = Model<MODEL>::NV;
    __shared__ double sh[NV][NT / 32];
    double v[NV];
#pragma unroll
    for (int k = 0; k < NV; k++) v[k] = valid ? R[k] * R[k] : 0.0;
    block_sum<NV, NT>(v, sh);
    if (threadIdx.x == 0)
        for (int k = 0; k < NV; k++) s.part[(size_t)blockIdx.x * NV + k] = v[k];
}

// The same partial sums one row per warp (32 cells, row = cell / 32), whatever the block size of the
// kernel: the rows, and so the norms summed from them, do not depend on the launch shape.
template <int MODEL>
__device__ __forceinline__ void partial_norms_warp(const State& s, bool valid, const double* R, int c)
{
    constexpr int NV = Model<MODEL>::NV;
    const int lane = threadIdx.x & 31;
#pragma unroll
    for (int k = 0; k < NV; k++) {
        const double x = warp_sum(valid ? R[k] * R[k] : 0.0);
        if (lane == 0) s.part[(size_t)(c >> 5) * NV + k] = x;
    }
}

// ------------------------------------------------------------------------------------------------
// k_resid: R only (csu_residual).
// ------------------------------------------------------------------------------------------------
template <int MODEL>
__global__ void __launch_bounds__(BLOCK) k_resid(const Prm* __restrict__ P, const __grid_constant__ Mesh m,
                                                 const __grid_constant__ State s)
{
    constexpr int NV = Model<MODEL>::NV, NP = Model<MODEL>::NP;
    const Prm& p = P[block_solve(s)];
    int c = blockIdx.x * BLOCK + threadIdx.x;
    bool valid = cell_in(p, c);
    double R[NV];
    if (valid) {
        double W[NP];
        loadP<MODEL>(s, m.nc, c, W);
        gather_residual<MODEL>(p, m, s, c, W, R);
        storeR<MODEL>(s, m.nc, c, R);
    }
    partial_norms<MODEL>(s, valid, R);
}

// ------------------------------------------------------------------------------------------------
// k_rk: one RK stage update (solverRK, solver.c:741-766) fused with the next residual's primitives.
// LAST: the stage that ends the iteration -- stores the state, the next local steps (solverCalcDt on the
// new, unclamped state) and the residual-norm partial sums of this stage's R (solverCalcRes).
// ------------------------------------------------------------------------------------------------
template <int MODEL, bool LAST>
__global__ void __launch_bounds__(BLOCK) k_rk(const Prm* __restrict__ P, const __grid_constant__ Mesh m,
                                              const __grid_constant__ State s, double a)
{
    constexpr int NV = Model<MODEL>::NV, NP = Model<MODEL>::NP;
    const int sid = block_solve(s);
    const Prm& p = P[sid];
    Scalars* const sc = s.sc + sid;
    int c = blockIdx.x * BLOCK + threadIdx.x;
    bool valid = cell_in(p, c);
    if (valid) {
        // mesh rows before the wait for the previous kernel
        prefetch_l1(m.nslot + c);
        prefetch_l1(m.omega + c);
        if (p.visc) prefetch_l1(m.nint + c);
#pragma unroll
        for (int j = 0; j < 4; j++) prefetch_l1(m.fslot + j * m.nc + c);
    }
    pdl_wait();
    if (halted(sc)) return;
    double R[NV];
    double lmin = bitsd(0x7ff0000000000000ULL);
    if (valid) {
        double P[NP], U[NV];
        loadP<MODEL>(s, m.nc, c, P);
        gather_residual<MODEL>(p, m, s, c, P, R);
        loadU<MODEL>(s, m.nc, c, U);
        double om = m.omega[c];
        double dt = sc->dt_local == 1 ? s.dtl[c] : sc->dt;
#pragma unroll
        for (int k = 0; k < NV; k++) U[k] = U[k] - dt * p.sigma * a * R[k] / om;
        if (LAST) {
            double l = local_step<MODEL>(p, U, m.sxh[c], m.syh[c], om);
            s.dtl[c] = cfl_at(p, sc->iter + 1) * l;
            lmin = l;
            clamp_prim<MODEL>(p, U, P);
            storeU<MODEL>(s, m.nc, c, U);
            storeR<MODEL>(s, m.nc, c, R);
        } else {
            clamp_prim<MODEL>(p, U, P);
        }
        storeP<MODEL>(s, m.nc, c, P);
    }
    if (LAST) {
        double v = block_min(lmin);
        if (threadIdx.x == 0 && !(v > bitsd(0x7fefffffffffffffULL))) atomicMin(&sc->dtmin_bits, dbits(v));
        partial_norms<MODEL>(s, valid, R);
    }
}

// implicitAuxCalcFlux2 (implicit.c:183-191) and its _sa/_sst forms
template <int NV>
__device__ __forceinline__ void aux_flux(const double* U, double pr, double nx, double ny, double* F)
{
    double V = (nx * U[1] + ny * U[2]) / U[0];
    F[0] = U[0] * V;
    F[1] = U[1] * V + nx * pr;
    F[2] = U[2] * V + ny * pr;
    F[3] = (U[3] + pr) * V;
#pragma unroll
    for (int k = 4; k < NV; k++) F[k] = U[k] * V;
}

// Convective spectral radius of interior face f times |dS|, and the viscous one (0 inviscid) times |dS|, from the face
// means of the two cells (implicitCalcD, implicit.c:19-181).
template <int MODEL>
__device__ __forceinline__ void face_radii(const Prm& p, const Mesh& m, const State& s, int f, double* Lc, double* Lv)
{
    const int2 e = m.fe[f];
    const double4 w0 = ld4(s.W4 + e.x), w1 = ld4(s.W4 + e.y);
    const double T0 = s.WT[e.x], T1 = s.WT[e.y];
    const double2 un = m.fun[f];
    const double dS = m.fds[f];
    double u = (w0.y + w1.y) * 0.5;
    double v = (w0.z + w1.z) * 0.5;
    double T = (T0 + T1) * 0.5;
    double cc = T2c(p.gas, T);
    *Lc = (fabs(un.x * u + un.y * v) + cc) * dS;
    *Lv = 0.0;
    if constexpr (MODEL >= 1) {
        double r = (w0.x + w1.x) * 0.5;
        double mi = sutherland(T);
        *Lv = fmax(4 / (3 * r), T2gamma(p.gas, T) / r) * (mi / p.pr + s.MIT[f] / p.pr_t) * dS;
    } else if (p.laminar) {
        double r = (w0.x + w1.x) * 0.5;
        *Lv = visc_radius(p.gas, p.pr, r, T) * dS;
    }
}

// ------------------------------------------------------------------------------------------------
// k_impl: R (WITH_R) and the implicit diagonal (implicitCalcD, implicit.c:19-181) of each cell. The
// diagonal, the local steps and their minimum need only the iteration's start state, so DPLUR computes them
// beside the gradient and flux kernels and gathers R in its first sweep.
// ------------------------------------------------------------------------------------------------
template <int MODEL, bool WITH_R>
__global__ void __launch_bounds__(BLOCK) k_impl(const Prm* __restrict__ P, const __grid_constant__ Mesh m,
                                                const __grid_constant__ State s)
{
    constexpr int NV = Model<MODEL>::NV, NP = Model<MODEL>::NP;
    const int sid = block_solve(s);
    const Prm& p = P[sid];
    Scalars* const sc = s.sc + sid;
    int c = blockIdx.x * BLOCK + threadIdx.x;
    bool valid = cell_in(p, c);
    pdl_wait();
    if (halted(sc)) return;
    double R[NV];
    double lmin = bitsd(0x7ff0000000000000ULL);
    if (valid) {
        const int nc = m.nc;
        double P[NP];
        loadP<MODEL>(s, nc, c, P);
        if (WITH_R) {
            gather_residual<MODEL>(p, m, s, c, P, R);
            storeR<MODEL>(s, nc, c, R);
        }
        {
            if constexpr (MODEL == 1) {
                // extension (saImplicitSource): the SA source's derivative in rho nt by a forward difference
                // in nt (the gradients held), its negative (destruction-dominated) part taken implicitly:
                // dQ = -Omega min(dQt/d(rho nt), 0) >= 0 joins the diagonal of the nt row
                if (p.sa_isrc) {
                    double4 gx = ld4(s.G4x + c), gy = ld4(s.G4y + c);
                    double rho = P[0], T = P[4], n = P[5];
                    double d = m.wall_d[c];
                    double mi_L = sutherland(T);
                    double n_L = mi_L / rho;
                    double S = fabs(gy.y - gx.z);
                    double hn = 1e-6 * fmax(fabs(n), n_L);
                    double q0 = p.sa_cc ? sacc_source(n, n_L, S, d, rho, gx.x, gy.x, s.Gxx[c], s.Gxy[c])
                                        : sa_source(n, n_L, S, d, rho, gx.x, gy.x, s.Gxx[c], s.Gxy[c]);
                    double q1 = p.sa_cc ? sacc_source(n + hn, n_L, S, d, rho, gx.x, gy.x, s.Gxx[c], s.Gxy[c])
                                        : sa_source(n + hn, n_L, S, d, rho, gx.x, gy.x, s.Gxx[c], s.Gxy[c]);
                    double dq = (q1 - q0) / hn / rho;
                    s.dQ[c] = isfinite(dq) ? -m.omega[c] * fmin(dq, 0.0) : 0.0;
                }
            }
            if constexpr (MODEL == 2) {
                // the SST source Jacobians of the implicit diagonal (sstInterSource, sst.c:643-680): LU-SGS
                // as the reference, DPLUR as the extension's k-omega diagonal block
                if (s.dQ) {
                    double4 gx = ld4(s.G4x + c), gy = ld4(s.G4y + c);
                    double sgx[4] = {gx.y, gx.z, s.Gxx[c], s.Gxx[(size_t)nc + c]};
                    double sgy[4] = {gy.y, gy.z, s.Gxy[c], s.Gxy[(size_t)nc + c]};
                    double J[6];
                    sst_source_jacobians(p.sst_k, sgx, sgy, P, m.wall_d[c], m.omega[c], J);
#pragma unroll
                    for (int q = 0; q < 6; q++) s.dQ[(size_t)q * nc + c] = J[q];
                }
            }
        }
        const int ni = m.nint[c], ns = m.nslot[c];
        double Lc = 0, Lv = 0;
        if constexpr (WITH_R) {
            for (int j = 0; j < ni; j++) {
                int sf = m.fslot[(size_t)j * nc + c];
                double Lcf, Lvf;
                face_radii<MODEL>(p, m, s, sf > 0 ? sf - 1 : -sf - 1, &Lcf, &Lvf);
                Lc += Lcf;
                Lv += Lvf * m.fds[sf > 0 ? sf - 1 : -sf - 1];
            }
        } else {
            // DPLUR: k_side's, one gather per face
            double2 fr[4];
#pragma unroll
            for (int j = 0; j < 4; j++) {
                if (j < ni) {
                    const int sf = m.fslot[j * nc + c];
                    fr[j] = s.FR[(sf > 0 ? sf : -sf) - 1];
                }
            }
#pragma unroll
            for (int j = 0; j < 4; j++) {
                if (j < ni) {
                    Lc += fr[j].x;
                    Lv += fr[j].y;
                }
            }
        }
        double D = 0.5 * p.w_imp * Lc;
        if (p.visc) D += Lv / m.omega[c];
        for (int j = ni; j < ns; j++) {
            int b = m.fslot[(size_t)j * nc + c] - 1 - m.nf;
            double2 dSv = m.bn[b];
            double dS = m.bds[b];
            double cc = T2c(p.gas, P[4]);
            double nx, ny;
            if (dS > 0) {
                nx = dSv.x / dS;
                ny = dSv.y / dS;
            } else {
                nx = 0.0;
                ny = 1.0;
            }
            double Lb = (fabs(nx * P[1] + ny * P[2]) + cc) * dS;
            Lc += Lb;
            D += 0.5 * p.w_imp * Lb;
            if (p.visc) {
                double Lvb = visc_radius(p.gas, p.pr, P[0], P[4]) * dS * dS;
                D += Lvb / m.omega[c];
            }
        }
        double om = m.omega[c];
        double l = om / Lc;
        s.dtl[c] = l;
        s.dpart[c] = D;
        lmin = l;
    }
    double v = block_min(lmin);
    if (threadIdx.x == 0 && !(v > bitsd(0x7fefffffffffffffULL))) atomicMin(&sc->dtmin_bits, dbits(v));
    if (WITH_R) partial_norms<MODEL>(s, valid, R);
}

// Step of the blocks' finite difference in variable mm (implicit.c:692). SST: rho omega reaches 1e10 beside a wall,
// where a step of 1e-6 is below its last bit; its column (a flux linear in rho omega) and rho k's take a step relative
// to the value.
constexpr double BLOCK_H = 1.0e-6;

template <int MODEL>
__device__ __forceinline__ double pert_step(int mm, const double* U)
{
    return MODEL == 2 && mm >= 4 ? BLOCK_H * fmax(1.0, fabs(U[mm])) : BLOCK_H;
}

// a / BLOCK_H, correctly rounded, by the divisor's reciprocal as a double-double: q = RN(a zh + RN(a zl)) (Brisebarre,
// Muller & Raina, "Accelerating correctly rounded floating-point division when the divisor is known in advance", IEEE
// Trans. Computers 53, 2004) is within 2^-105 of the quotient, and no quotient of a double by this divisor whose
// rounding that could change does change (tests/test_block_step.py checks every one). Zeros keep their sign; outside
// the exponents where the products are exact enough, the division itself, out of line.
static __host__ __device__ __noinline__ double over_h_any(double a)
{
    return a / BLOCK_H;
}

__host__ __device__ __forceinline__ double over_h(double a)
{
    const double zh = 0x1.e848p+19, zl = 0x1.8e0a318p-35;
    const double m = fabs(a);
    if (m == 0.0 || (m >= 0x1p-900 && m <= 0x1p+900)) return fma(a, zh, a * zl);
    return over_h_any(a);
}

// ------------------------------------------------------------------------------------------------
// k_side: what the DPLUR blocks and diagonal need once per cell or face, before them on the side stream. The first gc
// blocks: the pressures of a cell's states with one conserved variable stepped (implicitUpdateA, implicit.c:692-788),
// 14 divisions per cell instead of per block. The others: a face's spectral radii, which both cells' diagonals and both
// its blocks use, and for SA the face eddy viscosity mu_t = fv1 rho nt of the face means of the two cells' primitives
// (saBoundaryVisc's interior part, sa.c: the same expressions as sa_face_flux / sacc_face_flux, whose value it equals
// bit for bit): it needs no gradient, so the blocks and the diagonal can run beside k_grad and k_flux.
// ------------------------------------------------------------------------------------------------
template <int MODEL>
__global__ void __launch_bounds__(BLOCK) k_side(const Prm* __restrict__ P, const __grid_constant__ Mesh m,
                                                const __grid_constant__ State s, int gc)
{
    constexpr int NV = Model<MODEL>::NV, NM = MODEL == 2 ? 5 : 4;
    if ((int)blockIdx.x >= gc) {
        const int f = (blockIdx.x - gc) * BLOCK + threadIdx.x;
        if (f >= m.nf) return;
        const int2 e = m.fe[f];
        const int sid = cell_solve(s, e.x);
        const Prm& p = P[sid];
        if (halted(s.sc + sid)) return;
        if constexpr (MODEL == 1) {
            const double r = (ld4(s.W4 + e.y).x + ld4(s.W4 + e.x).x) * 0.5;
            const double T = (s.WT[e.y] + s.WT[e.x]) * 0.5;
            const double n = (s.Wx[e.y] + s.Wx[e.x]) * 0.5;
            const double mi_L = sutherland(T);
            const double n_L = mi_L / r;
            double fv1, tx, ty;
            sa_face(n, n_L, r, 0.0, 0.0, &fv1, &tx, &ty);
            s.MIT[f] = fv1 * r * n;
        }
        double Lc, Lv;
        face_radii<MODEL>(p, m, s, f, &Lc, &Lv);
        s.FR[f] = make_double2(Lc, Lv * m.fds[f]);
        if (s.FB) s.FB[f] = Lv / m.fL[f];
        return;
    }
    const int sid = block_solve(s);
    const Prm& p = P[sid];
    const int c = blockIdx.x * BLOCK + threadIdx.x;
    if (!cell_in(p, c) || halted(s.sc + sid)) return;
    double U[NV], Uq[NV], pr[NM];
    loadU<MODEL>(s, m.nc, c, U);
    const double T0 = s.WT[c];
    double rho = U[0];
    double uu = U[1] / rho;
    double vv = U[2] / rho;
    double E = U[3] / rho;
    double ee0 = E - 0.5 * (uu * uu + vv * vv);
    // SST (an extension: the reference's SST DPLUR multiplies 4x4 blocks into six variables, implicit.c:
    // 990-1000 with 938-972): the energy holds the turbulent kinetic energy, as in its SST delta flux
    // (implicitCalcDeltaFlux_sst, implicit.c:1048-1118)
    if constexpr (MODEL == 2) ee0 = ee0 - U[4] / rho;
#pragma unroll
    for (int mm = 0; mm < NM; mm++) {
        const double hm = pert_step<MODEL>(mm, U);
#pragma unroll
        for (int nn = 0; nn < NV; nn++) Uq[nn] = mm == nn ? U[nn] + hm : U[nn];
        double r2 = Uq[0];
        double u2 = Uq[1] / r2;
        double v2 = Uq[2] / r2;
        double E2 = Uq[3] / r2;
        double ee1 = E2 - 0.5 * (u2 * u2 + v2 * v2);
        if constexpr (MODEL == 2) ee1 = ee1 - Uq[4] / r2;
        double T = e2Taprox(p.gas, ee0, T0, ee1);
        pr[mm] = p.gas.R * r2 * T;
    }
    st4(s.PR4 + c, make_double4(pr[0], pr[1], pr[2], pr[3]));
    if constexpr (MODEL == 2) s.PRx[c] = pr[4];
}

// ------------------------------------------------------------------------------------------------
// k_blocks: the DPLUR off-diagonal blocks of implicitUpdateA (implicit.c:689-813; implicitUpdateA_sa
// 860-935), one thread per interior face slot j of a cell: the finite-difference Jacobian (h = 1e-6) of the
// neighbour's face flux, minus half the face's spectral radius on the diagonal. A block needs only the state at the
// start of the iteration and k_side's quantities, so the engine runs this kernel beside the gradient and flux kernels.
// Blocks [j gb, (j + 1) gb) of the grid hold slot j of the cells of cell blocks [0, gb).
//
// Bound by FP64 issue and the latency of its gathers; most of it was divisions that k_side now does once per cell or
// face (pressures, unit normals, spectral radii) or that over_h replaces. With k_side: SA plate 143 -> 84 us (its
// diagonal 35 -> 15), 100,000-cell SA FP64 77 -> 52, 160,000 triangles 43 -> 42 (19 -> 12.5), 500,000 125 -> 123
// (43 -> 23). Registers for three blocks per SM (SST two; four: SA the same, 500,000 triangles 133).
// ------------------------------------------------------------------------------------------------
template <int MODEL>
__global__ void __launch_bounds__(BLOCK, MODEL == 2 ? 2 : 3)
    k_blocks(const Prm* __restrict__ P, const __grid_constant__ Mesh m, const __grid_constant__ State s, int gb,
             int slots)
{
    constexpr int NV = Model<MODEL>::NV, NP = Model<MODEL>::NP;
    const int j = blockIdx.x / gb, cb = blockIdx.x - j * gb;
    const int sid = s.bsolve ? s.bsolve[cb] : 0;
    const Prm& p = P[sid];
    const Scalars* const sc = s.sc + sid;
    if (halted(sc)) return;
    const int c = cb * BLOCK + threadIdx.x;
    if (!cell_in(p, c)) return;
    const int nc = m.nc;
    const int sf = m.fslot[j * nc + c], nb = m.fnb[j * nc + c];
    if (j >= m.nint[c]) return;
    const int f = sf > 0 ? sf - 1 : -sf - 1;
    const double2 un = m.fun[f];
    const double nx = sf > 0 ? un.x : -un.x, ny = sf > 0 ? un.y : -un.y;
    const double dS = m.fds[f];
    double Un[NV], Pn[NP], pr[NV];
    loadU<MODEL>(s, nc, nb, Un);
    loadP<MODEL>(s, nc, nb, Pn);
    {
        const double4 t = ld4(s.PR4 + nb);
        pr[0] = t.x; pr[1] = t.y; pr[2] = t.z; pr[3] = t.w;
        if constexpr (MODEL == 2) pr[4] = s.PRx[nb];
        // the last variable (nt, omega) is in no energy: e2Taprox returns the temperature itself
        if constexpr (MODEL >= 1) pr[NV - 1] = p.gas.R * Un[0] * Pn[4];
    }
    double F0[NV], F[NV], Uq[NV];
    aux_flux<NV>(Un, Pn[3], nx, ny, F0);
    double A[NV * NV];
#pragma unroll
    for (int mm = 0; mm < NV; mm++) {
        const double hm = pert_step<MODEL>(mm, Un);
#pragma unroll
        for (int nn = 0; nn < NV; nn++) Uq[nn] = mm == nn ? Un[nn] + hm : Un[nn];
        aux_flux<NV>(Uq, pr[mm], nx, ny, F);
#pragma unroll
        for (int nn = 0; nn < NV; nn++) {
            if (!block_nz(nn, mm)) continue;
            const double d = 0.5 * (F[nn] - F0[nn]) * dS;
            A[nn * NV + mm] = MODEL == 2 && mm >= 4 ? d / hm : over_h(d);
        }
    }
    double cc = T2c(p.gas, Pn[4]);
    double ra = p.w_imp * (fabs(nx * Pn[1] + ny * Pn[2]) + cc) * dS;
    // implicitUpdateA_sa (implicit.c:920-928): with the face eddy viscosity (SST: the same radius with its own)
    if (MODEL >= 1 || p.laminar) ra += s.FB[f];
#pragma unroll
    for (int nn = 0; nn < NV; nn++) A[nn * NV + nn] -= 0.5 * ra;
    const size_t base = block_at<MODEL>(c, j, slots);
#pragma unroll
    for (int q = 0; q < NV * NV; q++) {
        if (!block_nz(q / NV, q % NV)) continue;
        const size_t o = base + 32 * block_entry<MODEL>(q / NV, q % NV);
        if (p.blk32) s.blocks32[o] = (float)A[q];
        else s.blocks[o] = A[q];
    }
}

// y += A x, terms in the reference's order (implicitMultA), the entries that are always zero left out
template <int MODEL, typename T>
__device__ __forceinline__ void block_times(const T* A, const double* x, double* y)
{
    constexpr int NV = Model<MODEL>::NV;
#pragma unroll
    for (int r = 0; r < NV; r++)
#pragma unroll
        for (int c = 0; c < NV; c++)
            if (block_nz(r, c)) y[r] += (double)A[block_entry<MODEL>(r, c)] * x[c];
}

// the relaxed update of one cell from y = D x + sum_j A_j x_j (SST: the sum alone); D4: the SA variable's diagonal
template <int MODEL>
__device__ __forceinline__ void jacobi_update(const State& s, int nc, int c, double D, double D4, const double* R,
                                              const double* y, const double* xo, double* xn)
{
    constexpr int NV = Model<MODEL>::NV;
    const double w = 2. / 3.;
    if constexpr (MODEL == 2) {
        // SST (extension): D on the mean flow; on k and omega, D minus the non-positive (destruction) part of the
        // source Jacobians' diagonal, with their coupling to rho (the LU-SGS diagonal block, implicit.c:323-345,
        // without its production part and k-omega cross terms, which made the iteration diverge at CFL 2 on
        // wall-resolved meshes): x* = Dblock^-1 (-R - sum_j A_j x_j), then x += w (x* - x)
        double z[NV], xs[NV];
#pragma unroll
        for (int k = 0; k < NV; k++) z[k] = -R[k] - y[k];
#pragma unroll
        for (int k = 0; k < 4; k++) xs[k] = z[k] / D;
        const double a = D - fmin(s.dQ[(size_t)nc + c], 0.0);
        const double dq = D - fmin(s.dQ[(size_t)5 * nc + c], 0.0);
        xs[4] = (z[4] + s.dQ[c] * xs[0]) / a;
        xs[5] = (z[5] + s.dQ[(size_t)3 * nc + c] * xs[0]) / dq;
#pragma unroll
        for (int k = 0; k < NV; k++) xn[k] = xo[k] + w * (xs[k] - xo[k]);
    } else {
#pragma unroll
        for (int k = 0; k < NV; k++) xn[k] = w * (-R[k] - y[k]) / (k == 4 ? D4 : D) + xo[k];
    }
}

// ------------------------------------------------------------------------------------------------
// k_sweep: one relaxed Jacobi sweep of implicitCalcDPLUR (implicit.c:1006-1033, implicitMultA 938-972):
//   x_new = w (-R - (D x + sum_j A_j x_j)) / D + x,  w = 2/3,  D += Omega/dt with dt = CFL min(Omega/Lc).
// The early exit of the reference (max |dx_0| < 1e-14 after a sweep) is taken on the device: a sweep that
// finds the previous one converged copies x forward. LAST adds the increment to the state
// (solverUpdateUImplicit, solver.c:1945-1955) and computes the next iteration's primitives. FIRST gathers
// the cell's residual R from the face fluxes (as k_impl does), stores it for the later sweeps and writes
// the block's partial norms.
// ------------------------------------------------------------------------------------------------
//
// Bound by HBM (or L2, when the blocks stay there) and the latency of the gathers. The blocks are stored without their
// zeros in 32-cell tiles, each warp's a contiguous run (block_at): steady middle sweep of 160,000 triangles FP64
// 16.5 -> 13.4 us, of 500,000 58 -> 47 us (244 MB, 5.2 TB/s, 79 % of the measured copy bandwidth), of the SA plate
// (209,825 quads, FP32) 38.7 -> 23.8 us, SST airfoil pack 22 % faster per pass. SA's register budget is 96 (640
// threads per SM in blocks of 64 and 128 cells; 128 in blocks of 256): at the compiler's own 64 the plate's sweep
// takes 28.6 us, at 80 23.0 but the SA pack 5 % more; Euler and SST are fastest at the compiler's choice (Euler held
// to 48: 16.7 us, SST held to 96 or 128: 2-5 % slower).
//
// On small meshes a sweep is one chain of loads: EARLY issues the gathers before the halt and early-exit flags arrive,
// for registers that cost more than the chain once several waves hide it (sweep_early: where the line lies).
//
// WIDE holds Euler and laminar, 88 registers by themselves, to 56 in blocks of 64 and 128 cells and to 64 in blocks of
// 256 (sweep_wide: on which meshes).
// Blocks per SM of a sweep's register budget: WIDE 1,152 threads, SA 640, the others the compiler's choice.
template <int MODEL, int SB, int MODE>
constexpr int sweep_blocks()
{
    return MODE == SWEEP_WIDE ? 1152 / SB : MODEL == 1 && MODE == SWEEP_PLAIN ? 640 / SB : 1;
}

template <int MODEL, bool LAST, bool FIRST, int SB, bool F32, int MODE = SWEEP_PLAIN>
__global__ void __launch_bounds__(SB, sweep_blocks<MODEL, SB, MODE>())
    k_sweep(const Prm* __restrict__ P, const __grid_constant__ Mesh m, const __grid_constant__ State s, int sweep,
            int cur, int slots)
{
    constexpr int NV = Model<MODEL>::NV, NP = Model<MODEL>::NP;
    constexpr bool EARLY = MODE == SWEEP_EARLY;
    static_assert(BLOCK % SB == 0, "sweep blocks tile the cell blocks");
    // SB-thread blocks: BLOCK / SB of them cover one cell block of the solve map
    const int sid = s.bsolve ? s.bsolve[blockIdx.x / (BLOCK / SB)] : 0;
    const Prm& p = P[sid];
    Scalars* const sc = s.sc + sid;
    int c = blockIdx.x * SB + threadIdx.x;
    const int nc = m.nc;
    const bool valid = cell_in(p, c);
    // Slots 0-2 are gathered unconditionally (a slot without a face reads the cell itself and some block, both in
    // bounds, and is not summed), so their index and neighbour loads issue together instead of one dependent chain
    // per face; slot 3 only exists in quadrilaterals. The indices are read before the wait for the previous sweep.
    int ni = 0, nbj[4] = {c, c, c, c};
    if (valid) {
        ni = m.nint[c];
#pragma unroll
        for (int j = 0; j < 3; j++) {
            int q = m.fnb[j * nc + c];
            nbj[j] = q >= 0 ? q : c;
        }
        if (ni > 3) nbj[3] = m.fnb[3 * nc + c];
    }
    pdl_wait();
    const double4* const xo4 = s.X4[cur];
    const double* const xox = s.Xx[cur];
    // EARLY: the increments are under way before the flags that may make them needless are known
    double4 x4c = make_double4(0.0, 0.0, 0.0, 0.0), x4n[EARLY ? 3 : 1];
    if (EARLY && valid) {
        x4c = ld4(xo4 + c);
#pragma unroll
        for (int j = 0; j < (EARLY ? 3 : 1); j++) x4n[j] = ld4(xo4 + nbj[j]);
    }
    if (halted(sc)) return;
    bool conv = !FIRST && sweep > 0 && bitsd(sc->sweep_max[sweep - 1]) < 1e-14;
    double dmax = 0.0;
    double R[NV];
    if (valid) {
        double4* xn4 = s.X4[cur ^ 1];
        double* xnx = s.Xx[cur ^ 1];
        double xo[NV], xn[NV];
        {
            double4 t = EARLY ? x4c : ld4(xo4 + c);
            xo[0] = t.x; xo[1] = t.y; xo[2] = t.z; xo[3] = t.w;
#pragma unroll
            for (int k = 4; k < NV; k++) xo[k] = xox[(size_t)(k - 4) * nc + c];
        }
        if constexpr (FIRST) {
            double Pc[NP];
            loadP<MODEL>(s, nc, c, Pc);
            gather_residual<MODEL>(p, m, s, c, Pc, R);
            storeR<MODEL>(s, nc, c, R);
        } else {
            double4 t = ld4(s.R4 + c);
            R[0] = t.x; R[1] = t.y; R[2] = t.z; R[3] = t.w;
#pragma unroll
            for (int k = 4; k < NV; k++) R[k] = s.Rx[(size_t)(k - 4) * nc + c];
        }
        if (conv) {
#pragma unroll
            for (int k = 0; k < NV; k++) xn[k] = xo[k];
        } else {
            // the first sweep leaves the diagonal (implicitCalcD) for the others
            double D;
            if constexpr (FIRST) {
                double cfl = cfl_at(p, sc->iter);
                double dt = p.implicit_local_dt ? s.dtl[c] * cfl : bitsd(sc->dtmin_bits) * cfl;
                D = s.dpart[c] + m.omega[c] / dt;
                s.diag[c] = D;
            } else {
                D = s.diag[c];
            }
            // y = D x + sum_j A_j x_j; SST keeps the off-diagonal sum alone (its diagonal is a block)
            double y[NV];
#pragma unroll
            for (int k = 0; k < NV; k++) y[k] = MODEL == 2 ? 0.0 : D * xo[k];
            // SA with saImplicitSource: the nt row's diagonal also holds the implicit source part
            double D4 = D;
            if constexpr (MODEL == 1) {
                if (p.sa_isrc) {
                    D4 = D + s.dQ[c];
                    y[4] = D4 * xo[4];
                }
            }
#pragma unroll
            for (int j = 0; j < 4; j++) {
                if (j == 3 && ni <= 3) break;
                const int nb = nbj[j];
                double xb[NV];
                double4 t = EARLY && j < 3 ? x4n[EARLY && j < 3 ? j : 0] : ld4(xo4 + nb);
                xb[0] = t.x; xb[1] = t.y; xb[2] = t.z; xb[3] = t.w;
#pragma unroll
                for (int k = 4; k < NV; k++) xb[k] = xox[(size_t)(k - 4) * nc + nb];
                const size_t base = block_at<MODEL>(c, j, slots);
                const bool use = j < ni;
                double A[BLOCK_NE<MODEL>];
#pragma unroll
                for (int q = 0; q < BLOCK_NE<MODEL>; q++)
                    A[q] = F32 ? (double)s.blocks32[base + 32 * q] : s.blocks[base + 32 * q];
                if (use) block_times<MODEL>(A, xb, y);
            }
            jacobi_update<MODEL>(s, nc, c, D, D4, R, y, xo, xn);
            dmax = fabs(xn[0] - xo[0]);
        }
        st4(xn4 + c, make_double4(xn[0], xn[1], xn[2], xn[3]));
#pragma unroll
        for (int k = 4; k < NV; k++) xnx[(size_t)(k - 4) * nc + c] = xn[k];
        if (LAST) {
            double U[NV], P[NP];
            loadU<MODEL>(s, nc, c, U);
#pragma unroll
            for (int k = 0; k < NV; k++) U[k] += xn[k];
            clamp_prim<MODEL>(p, U, P);
            storeU<MODEL>(s, nc, c, U);
            storeP<MODEL>(s, nc, c, P);
        }
    }
    if (!conv) {
        double v = block_max<SB>(dmax);
        if (threadIdx.x == 0) atomicMax(&sc->sweep_max[sweep], dbits(v));
    }
    if (FIRST) partial_norms_warp<MODEL>(s, valid, R, c);
}

// implicitCalcDeltaFlux (implicit.c:194-231) and implicitCalcDeltaFlux_sa (495-552): F(U + d) - F(U) on the
// face normal, from the neighbour's primitives P and increment d.
template <int MODEL>
__device__ __forceinline__ void delta_flux(const Prm& p, const double* P, const double* d, double nx, double ny,
                                           double* dF)
{
    constexpr int NV = Model<MODEL>::NV;
    double rho = P[0], u = P[1], v = P[2], pr = P[3];
    double U[NV], F0[NV], F1[NV];
    double T = pr / (p.gas.R * rho);
    double e0 = T2e(p.gas, T);
    double E = e0 + (u * u + v * v) / 2;
    if constexpr (MODEL == 2) E = E + P[5]; // implicitCalcDeltaFlux_sst (implicit.c:1048-1118): + k
    U[0] = rho;
    U[1] = rho * u;
    U[2] = rho * v;
    U[3] = rho * E;
    if constexpr (MODEL >= 1) U[4] = rho * P[5];
    if constexpr (MODEL == 2) U[5] = rho * P[6];
    aux_flux<NV>(U, pr, nx, ny, F0);
#pragma unroll
    for (int k = 0; k < NV; k++) U[k] = U[k] + d[k];
    if constexpr (MODEL == 0) {
        rho = U[0];
        u = U[1] / rho;
        v = U[2] / rho;
        E = U[3] / rho;
        double e1 = E - 0.5 * (u * u + v * v);
        T = e2Taprox(p.gas, e0, T, e1);
        pr = p.gas.R * T * rho;
    } else if constexpr (MODEL == 2) {
        rho = U[0];
        rho = fmax(rho, p.r_lim);
        U[0] = rho;
        u = U[1] / rho;
        v = U[2] / rho;
        double k = U[4] / rho;
        if (k < 1e-14) {
            k = 1e-14;
            U[4] = rho * k;
        }
        double om = U[5] / rho;
        if (om < 0.0) { // omLim = 0 (solver.c:1155)
            om = 0.0;
            U[5] = rho * om;
        }
        E = U[3] / rho;
        double e1 = E - (u * u + v * v) * 0.5 - k;
        e1 = fmax(e1, 7.176325e+02);
        T = e2Taprox(p.gas, e0, T, e1);
        if (T < 1) {
            T = 1;
            e1 = T2e(p.gas, T);
            E = e1 + (u * u + v * v) * 0.5 + k;
            U[3] = rho * E;
        }
        pr = p.gas.R * T * rho;
    } else {
        rho = U[0];
        rho = fmax(rho, p.r_lim);
        U[0] = rho;
        u = U[1] / rho;
        v = U[2] / rho;
        E = U[3] / rho;
        double e1 = E - (u * u + v * v) * 0.5;
        e1 = fmax(e1, 7.176325e+02);
        T = e2Taprox(p.gas, e0, T, e1);
        if (T < 1) {
            T = 1;
            e1 = T2e(p.gas, T);
            E = e1 + (u * u + v * v) * 0.5;
            U[3] = rho * E;
        }
        pr = p.gas.R * T * rho;
        double n = U[4] / rho;
        n = fmax(n, 0);
        U[4] = rho * n;
    }
    aux_flux<NV>(U, pr, nx, ny, F1);
#pragma unroll
    for (int k = 0; k < NV; k++) dF[k] = F1[k] - F0[k];
}

// ------------------------------------------------------------------------------------------------
// k_lusgs: one colour of the LU-SGS sweeps (implicitLUSGS_L / _U, implicit.c:274-482) as a multicolour
// Gauss-Seidel: the reference sweeps cells in index order using the already-updated lower (upper) index
// neighbours; here the cells of one colour update together using the neighbours of lower (higher) colours.
// Same operator, another ordering: the converged solution is the same, the path to it is not.
//   FWD: x0_i = (-R_i - sum_{lower} 0.5 (dF(x0_j) dS - ra_j x0_j)) / D_i
//   BWD: x1_i = (D_i x0_i - sum_{higher} 0.5 (dF(x1_j) dS - ra_j x1_j)) / D_i
// A colour holds a quarter of the cells and depends on the one before, so a launch is one thread's latency, not
// throughput: four lanes share a cell, one per face slot, and every lane then subtracts the faces' terms in slot order.
// A launch between events, one lane -> four, meshes of 6,000, 100,000, 300,000 and 1,000,000 cells: Euler 15.8 -> 8.3
// us, 17.6 -> 10.9, 22.1 -> 16.1, 55.8 -> 43.6; SST 19.1 -> 10.1, 22.3 -> 15.5, 31.5 -> 28.3, 78.2 -> 82.1 (its
// diagonal block's x87 quotients one to a lane; repeated by every lane 87.3). 5,928-cell wedge: the iteration 100 -> 57
// us in its graph.
// ------------------------------------------------------------------------------------------------
constexpr int LUSGS_THREADS = 128;

template <int MODEL, bool FWD>
__global__ void __launch_bounds__(LUSGS_THREADS) k_lusgs(const Prm* __restrict__ P, const __grid_constant__ Mesh m,
                                                         const __grid_constant__ State s, const int* color,
                                                         const int* cells, int mycolor, int start, int count)
{
    constexpr int NV = Model<MODEL>::NV, NP = Model<MODEL>::NP;
    const int t = (blockIdx.x * LUSGS_THREADS + threadIdx.x) >> 2, j = threadIdx.x & 3;
    const int nc = m.nc;
    // lanes past the last cell repeat it without storing: the shuffles below need whole warps
    const int c = cells[start + min(t, count - 1)];
    const int sid = cell_solve(s, c);
    const Prm& p = P[sid];
    Scalars* const sc = s.sc + sid;
    const int sf = m.fslot[j * nc + c];
    const int nb = max(m.fnb[j * nc + c], 0);
    const bool use = j < m.nint[c];
    const int cn = color[nb];
    pdl_wait();
    const bool store = t < count && !halted(sc);
    const double4* src4 = FWD ? s.X4[0] : s.X4[1];
    const double* srcx = FWD ? s.Xx[0] : s.Xx[1];
    const double cfl = cfl_at(p, sc->iter);
    const double dt = p.implicit_local_dt ? s.dtl[c] * cfl : bitsd(sc->dtmin_bits) * cfl;
    const double D = s.dpart[c] + m.omega[c] / dt;
    double x[NV];
    if (FWD) {
        double4 t4 = ld4(s.R4 + c);
        x[0] = -t4.x; x[1] = -t4.y; x[2] = -t4.z; x[3] = -t4.w;
#pragma unroll
        for (int k = 4; k < NV; k++) x[k] = -s.Rx[(size_t)(k - 4) * nc + c];
    } else {
        double4 t4 = ld4(s.X4[0] + c);
        x[0] = D * t4.x; x[1] = D * t4.y; x[2] = D * t4.z; x[3] = D * t4.w;
#pragma unroll
        for (int k = 4; k < NV; k++) x[k] = D * s.Xx[0][(size_t)(k - 4) * nc + c];
        if constexpr (MODEL == 2) {
            // implicitLUSGS_U (implicit.c:372-390): the k, omega rows multiply by the SST diagonal block
            const double x0 = t4.x, x4 = s.Xx[0][c], x5 = s.Xx[0][(size_t)nc + c];
            const double a = D - s.dQ[(size_t)nc + c], b = -s.dQ[(size_t)2 * nc + c];
            const double cq = -s.dQ[(size_t)4 * nc + c], dq = D - s.dQ[(size_t)5 * nc + c];
            const double det = a * dq - b * cq;
            if (!(fabs(det) < 1e-14)) {
                x[4] = a * x4 + b * x5 - s.dQ[c] * x0;
                x[5] = cq * x4 + dq * x5 - s.dQ[(size_t)3 * nc + c] * x0;
            }
        }
    }
    // this lane's face
    const bool mine = use && (FWD ? cn < mycolor : cn > mycolor);
    double term[NV];
#pragma unroll
    for (int k = 0; k < NV; k++) term[k] = 0.0;
    if (mine && store) {
        const int f = sf > 0 ? sf - 1 : -sf - 1;
        double2 un = m.fun[f];
        double nx = sf > 0 ? un.x : -un.x, ny = sf > 0 ? un.y : -un.y;
        double dS = m.fds[f];
        double Pn[NP], dn[NV], dF[NV];
        loadP<MODEL>(s, nc, nb, Pn);
        {
            double4 t4 = ld4(src4 + nb);
            dn[0] = t4.x; dn[1] = t4.y; dn[2] = t4.z; dn[3] = t4.w;
#pragma unroll
            for (int k = 4; k < NV; k++) dn[k] = srcx[(size_t)(k - 4) * nc + nb];
        }
        delta_flux<MODEL>(p, Pn, dn, nx, ny, dF);
        double cc = T2c(p.gas, Pn[4]);
        double ra = p.w_imp * (fabs(nx * Pn[1] + ny * Pn[2]) + cc) * dS;
        if constexpr (MODEL >= 1) {
            // implicitFunc_sa / implicitFunc_sst (implicit.c:560-567, 1140-1150): the face eddy viscosity
            double r = Pn[0], T = Pn[4];
            double mi = sutherland(T);
            ra += fmax(4 / (3 * r), T2gamma(p.gas, T) / r) * (mi / p.pr + s.MIT[f] / p.pr_t) * dS / m.fL[f];
        } else if (p.laminar) {
            ra += visc_radius(p.gas, p.pr, Pn[0], Pn[4]) * dS / m.fL[f];
        }
#pragma unroll
        for (int k = 0; k < NV; k++) term[k] = 0.5 * (dF[k] * dS - ra * dn[k]);
    }
    const unsigned who = __ballot_sync(0xffffffffu, mine) >> (threadIdx.x & 28);
#pragma unroll
    for (int q = 0; q < 4; q++)
#pragma unroll
        for (int k = 0; k < NV; k++) {
            const double v = __shfl_sync(0xffffffffu, term[k], q, 4);
            if (who >> q & 1u) x[k] -= v;
        }
    // lane j finishes component j, lanes 0 and 1 a scalar each
    double v = (j == 0 ? x[0] : j == 1 ? x[1] : j == 2 ? x[2] : x[3]) / D, vx = 0.0;
    if constexpr (MODEL == 1) vx = x[4] / D;
    if constexpr (MODEL == 2) {
        // the SST diagonal (implicit.c:323-345, 444-465): D on the mean flow, a 2x2 block with the source
        // Jacobians on k (lane 0) and omega (lane 1), its determinant in double and the quotients in long double
        const double x0 = __shfl_sync(0xffffffffu, v, 0, 4);
        const bool om = j & 1;
        const double A = x[4] + s.dQ[c] * x0;
        const double B = x[5] + s.dQ[(size_t)3 * nc + c] * x0;
        const double a = D - s.dQ[(size_t)nc + c], b = -s.dQ[(size_t)2 * nc + c];
        const double cq = -s.dQ[(size_t)4 * nc + c], dq = D - s.dQ[(size_t)5 * nc + c];
        const double det = a * dq - b * cq;
        if (fabs(det) < 1e-14) {
            vx = (om ? x[5] : x[4]) / D;
        } else {
            const double n = om ? -A * cq + B * a : A * dq - B * b;
            bool ok = true;
            vx = x87_div_d(n, det, ok);
            if (!ok) vx = x80_to_double(x80_div(x80_from_double(n), x80_from_double(det)));
        }
    }
    if (!store) return;
    reinterpret_cast<double*>((FWD ? s.X4[0] : s.X4[1]) + c)[j] = v;
    if (j < NV - 4) (FWD ? s.Xx[0] : s.Xx[1])[(size_t)j * nc + c] = vx;
}

// U += dW1 (solverUpdateUImplicit), then the next iteration's primitives and clamps
template <int MODEL>
__global__ void __launch_bounds__(BLOCK) k_update(const Prm* __restrict__ P, const __grid_constant__ Mesh m,
                                                  const __grid_constant__ State s)
{
    constexpr int NV = Model<MODEL>::NV, NP = Model<MODEL>::NP;
    const Prm& p = P[block_solve(s)];
    pdl_wait();
    if (halted(s.sc + block_solve(s))) return;
    int c = blockIdx.x * BLOCK + threadIdx.x;
    if (!cell_in(p, c)) return;
    const int nc = m.nc;
    double U[NV], W[NP];
    loadU<MODEL>(s, nc, c, U);
    double4 t4 = ld4(s.X4[1] + c);
    U[0] += t4.x; U[1] += t4.y; U[2] += t4.z; U[3] += t4.w;
#pragma unroll
    for (int k = 4; k < NV; k++) U[k] += s.Xx[1][(size_t)(k - 4) * nc + c];
    clamp_prim<MODEL>(p, U, W);
    storeU<MODEL>(s, nc, c, U);
    storeP<MODEL>(s, nc, c, W);
}

// ------------------------------------------------------------------------------------------------
// k_finalize: one block closing an iteration (solverCalcRes, solverCalcCoeff3, history row, flags) and
// preparing the next step size. mode: 0 RK iteration, 1 implicit iteration, 2 prologue (step size only),
// 3 residual only (norms). bsel: the face-coefficient buffer k_flux wrote (0 bcoef, 1 bcoef2). In mode 1
// it records the halt flags it found on entry in `frozen` (halted_behind).
// ------------------------------------------------------------------------------------------------
template <int MODEL>
__global__ void __launch_bounds__(BLOCK) k_finalize(const Prm* __restrict__ P, const __grid_constant__ Mesh m,
                                                    const __grid_constant__ State s, int mode, int ppb, int bsel)
{
    constexpr int NV = Model<MODEL>::NV;
    __shared__ double sh[NV + 4][BLOCK / 32];
    const int sid = blockIdx.x; // one block per solve
    const Prm& p = P[sid];
    Scalars* const sc = s.sc + sid;
    // ppb rows of partial norms per cell block (the DPLUR first sweep writes one per 128 cells)
    const int npart = p.nblk * ppb, nwall = p.nwall;
    const double* part = s.part + (size_t)p.blk0 * ppb * NV;
    const double* bcoef = (bsel ? s.bcoef2 : s.bcoef) + (size_t)p.wall0 * 4;
    // Everything the block reads is requested before the halted test, so the loads overlap: a chain of
    // dependent round trips to the L2 would be most of a one-block kernel's time. Thread 0 keeps a copy of
    // the solve's scalars and writes back only what changes.
    pdl_wait();
    const bool stop = mode != 2 && mode != 3 && halted(sc);
    double v[NV + 4];
#pragma unroll
    for (int k = 0; k < NV + 4; k++) v[k] = 0.0;
    if (mode != 2) {
        // rows strided over the threads (consecutive threads read consecutive rows), four rows per thread in
        // flight before any is added, then a fixed tree: deterministic
        constexpr int U = 4;
        for (int i0 = threadIdx.x; i0 < npart; i0 += U * BLOCK) {
            double t[U][NV];
#pragma unroll
            for (int u = 0; u < U; u++) {
                const int i = i0 + u * BLOCK;
#pragma unroll
                for (int k = 0; k < NV; k++) t[u][k] = i < npart ? part[(size_t)i * NV + k] : 0.0;
            }
#pragma unroll
            for (int u = 0; u < U; u++)
#pragma unroll
                for (int k = 0; k < NV; k++) v[k] += t[u][k];
        }
        for (int i0 = threadIdx.x; i0 < nwall; i0 += U * BLOCK) {
            double t[U][4];
#pragma unroll
            for (int u = 0; u < U; u++) {
                const int i = i0 + u * BLOCK;
#pragma unroll
                for (int k = 0; k < 4; k++) t[u][k] = i < nwall ? bcoef[(size_t)i * 4 + k] : 0.0;
            }
#pragma unroll
            for (int u = 0; u < U; u++)
#pragma unroll
                for (int k = 0; k < 4; k++) v[NV + k] += t[u][k];
        }
    }
    Scalars S;
    if (threadIdx.x == 0) {
        S = *sc;
        if (mode == 1) sc->frozen = stop;
    }
    if (stop) return;
    block_sum<NV + 4>(v, sh);
    if (threadIdx.x != 0) return;
    if (mode != 2) {
        bool bad = false;
        double res[NV];
        for (int k = 0; k < NV; k++) {
            res[k] = sqrt(v[k] / p.nc);
            sc->res[k] = res[k];
            if (!isfinite(res[k])) bad = true;
        }
        // Cx_v -= fx/q per wall face (solver.c:1376-1380): the negated sum
        double cxp = v[NV] / p.sref, cyp = v[NV + 1] / p.sref;
        double cxv = (0.0 - v[NV + 2]) / p.sref, cyv = (0.0 - v[NV + 3]) / p.sref;
        if (p.axi) {
            cxp *= 2 * M_PI;
            cxv *= 2 * M_PI;
        }
        sc->coef[0] = cxp; sc->coef[1] = cxv; sc->coef[2] = cyp; sc->coef[3] = cyv;
        if (mode == 3) return;
        if (S.hist && S.hist_row < S.hist_cap) {
            double* row = S.hist + (size_t)S.hist_row * (NV + 4);
            for (int k = 0; k < NV; k++) row[k] = res[k];
            row[NV] = cxp; row[NV + 1] = cxv; row[NV + 2] = cyp; row[NV + 3] = cyv;
        }
        sc->hist_row = S.hist_row + 1;
        // the residual-drop stop measures from the largest residual so far (a free-stream start has a first
        // density residual of round-off size; the start-up transient then raises it)
        double r00 = S.res0[0];
        if (!S.have_res0) {
            for (int k = 0; k < NV; k++) sc->res0[k] = res[k];
            sc->have_res0 = 1;
            r00 = res[0];
        } else {
            for (int k = 0; k < NV; k++)
                if (res[k] > S.res0[k]) sc->res0[k] = res[k];
            r00 = fmax(r00, res[0]);
        }
        sc->steps = S.steps + 1;
        if (S.iter == p.dt_local_n) sc->dt_local = 0;
        S.iter++;
        sc->iter = S.iter;
        if (bad) sc->status = 4; // CSU_ERR_NONFINITE
        if (p.tube) {
            S.t += S.dt * p.stages / 2.0;
            sc->t = S.t;
            if (S.stop_after) sc->done = 1;
        }
        if (p.conv_tol > 0 && res[0] <= p.conv_tol * r00) sc->done = 1;
        else if (p.iter_cap > 0 && S.iter >= p.iter_cap) sc->done = 2;
        for (int k = 0; k < MAX_SWEEPS; k++) sc->sweep_max[k] = 0ULL;
    }
    if (mode == 2 && !S.fresh) {
        sc->dtmin_bits = 0x7ff0000000000000ULL;
        return;
    }
    if (mode == 2) sc->fresh = 0;
    if (mode == 0 || mode == 2) {
        // solverCalcDt (solver.c:925-950) for the next iteration, from the minimum gathered above
        double dt = bitsd(S.dtmin_bits);
        dt *= cfl_at(p, S.iter);
        if (p.tube && S.t + dt > p.tmax) {
            dt = (p.tmax - S.t);
            sc->stop_after = 1;
        }
        sc->dt = dt;
    }
    sc->dtmin_bits = 0x7ff0000000000000ULL;
}

} // namespace csu
