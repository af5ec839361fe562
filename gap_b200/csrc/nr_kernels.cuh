// Device kernels of the Newton-Raphson loop.
//
// Layout: scenarios sharing one plan are packed in groups of SW ("lanes"); every per-bus,
// per-node and per-slot quantity is stored [group][item][lane], so the SW threads that
// handle the same item for the SW scenarios of a group touch one contiguous run of memory
// (SW*16 B for a complex FP64 value, SW*16 B for an FP32 2x2 block).  Index lists (CSR of
// Y, factor schedule) are shared by all lanes and read once per warp.
//
// Reference semantics restated (src/solver/powerflow/cpu/cpu_newton_raphson.cpp):
//   mismatch   :243-337  S = V conj(Y V), Delta = S - S_spec, P rows for non-slack buses, Q
//                        rows for PQ buses, converged when max |Delta| < tol (:115-157)
//   Jacobian   :546-727  polar partial derivatives; |V| < 1e-6 replaced by 1 (:578)
//   update     :438-504  damped (0.9) and clamped polar update (policy REFERENCE)
#pragma once
#include <cooperative_groups.h>
#include <cuda_runtime.h>

#include <cstddef>

#include "blocks.cuh"

namespace gapk {

enum { BUS_PQ = 0, BUS_PV = 1, BUS_SLACK = 2 };
enum { SC_CONVERGED = 0, SC_MAXITER = 1, SC_SINGULAR = 2, SC_NONFINITE = 3 };

struct PlanDev {
    int n_bus, nb, nnz_y, n_slots, nnz_l, n_levels, n_a;
    int jac_mode;  // 0: reference (last duplicate, |x| <= 1e-12 dropped), 1: exact
    int ns, n_tail, n_schur;  // sparse nodes, dense-tail nodes, Schur targets (= n_tail^2)
    const int4* schur;        // (slot, pair_begin, pair_end, position r*n_tail+c | hasval<<30)
    const int* a_slots;       // slots holding Jacobian values (the only ones the fill writes)
    const int4* a_rec;        // per Jacobian block: slot, row bus, column bus, Y entry (jac_block)
    const int* acol_ptr;      // A blocks by block column: (a index, row node)
    const int2* acol;
    const int* y_row_ptr;
    const int* y_col;
    const int* bus_type;
    const int* node_of_bus;
    const int4* slot_info;
    const int* slot_src;
    const int* level_ptr;
    const int4* levels;       // k_nr_small's level records and packed schedule (null when the
    const unsigned* words;    // grid is too large for it)
    const uint2* ell;
    const int* fa_ptr;
    const int4* targets;
    const int2* pairs;
    const int* fb_ptr;
    const int2* scale;
    const int* lptr;
    const int* lidx;
    const int* rptr;
    const int2* rlist;
    const int* arow_ptr;
    const int2* arow;
};

// Per-batch device state.  q = group*SW + lane indexes per-scenario arrays.
struct BatchDev {
    int n_scen, n_groups, sw, y_shared;
    double2* V;       // [G][n_bus][SW]
    double2* Sspec;   // [G][n_bus][SW]
    double2* Scalc;   // [G][n_bus][SW]
    double2* Y;       // [nnz] (shared) or [G][nnz][SW]
    void* F;          // factor blocks [G][n_slots][SW]
    double* A64;      // FP64 Jacobian blocks [G][n_a][SW][4] (iterative refinement) or null
    double2* rhs;     // -Delta per node [G][nb][SW]
    double2* dx;      // Newton correction per node [G][nb][SW]
    double2* res;     // refinement residual [G][nb][SW]
    void* X;          // triangular-solve work vector [G][nb][SW] (T2)
    void* Dt;         // dense tail per scenario [G*SW][2*n_tail][dense_ld] (T), row-major
    unsigned long long* mis_bits;  // [G*SW] max |Delta| bits of the current iteration
    int* state;       // [G*SW] 0 iterating, 1 done
    int* solving;     // [G*SW] correction + update this iteration
    int* singular;    // [G*SW]
    int* iters;       // [G*SW]
    int* status;      // [G*SW]
    double* final_mis;  // [G*SW]
    int* gsolve;      // [G]
    int* giter;       // [G]
    int* ctrl;        // [0] iteration, [1] max_iter, [2] any iterating, [3] policy, [4] loops,
                      // [5] tensor-core LU wait ran out, [6] wait test (skip the MMAs)
    double* tol;      // [0] tolerance, [1] refine below, [2] reuse the factors below this mismatch
                      //     (0: never); the allocation-free path has [0] only
    int* grefine;     // [G] refinement pass runs for the group this iteration (null: always)
    int* gfactor;     // [G] the group refactorises this iteration (null: always); else the
                      //     previous factors precondition the refined solve
    unsigned long long* lvl_ts;  // level trace (null: off): %globaltimer stamps
                                 // [3 kernels: factor, forward, backward][G][n_levels + 2]
    unsigned long long* dlu_ts;  // dense-tail panel trace of k_dense_lu (null: off)
                                 // [G*SW][1 + 3 * panels]: start, then per panel the ends of
                                 // the diagonal block, the L21/U12 solves, the trailing update
};

// nanosecond clock of the level trace (PTX special register %globaltimer)
__device__ __forceinline__ unsigned long long gtimer() {
    unsigned long long t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}
// stamp j of kernel `which` for group g: 0 = start, 1 + h = level h done (in execution order),
// n_levels + 1 = end; one thread per group, after a barrier
__device__ __forceinline__ void lvl_stamp(BatchDev const& B, int n_levels, int which, int g, int j,
                                          int rank) {
    if (threadIdx.x == 0 && rank == 0)
        B.lvl_ts[((size_t)which * B.n_groups + g) * (n_levels + 2) + j] = gtimer();
}

// ---------------------------------------------------------------------------------------
// load: interleave inputs, flat start, reset state
// ---------------------------------------------------------------------------------------
// Loop options of one solve, kernel arguments of k_load (no host copies, so that a graph can hold
// several batches' solves); set = 0 leaves the control words and tolerances to the caller.
struct SolveOpts {
    int set, max_iter, policy;
    double tol, refine_below, reuse_below;
};

template <int SW>
__global__ void k_load(PlanDev P, BatchDev B, const double2* __restrict__ y_in,
                       const double2* __restrict__ s_in, const double2* __restrict__ v_in,
                       const double* __restrict__ u_pu, int v_shared, SolveOpts opt) {
    const int g = blockIdx.y;
    const int n = P.n_bus;
    const long tid = (long)blockIdx.x * blockDim.x + threadIdx.x;
    const int i = (int)(tid / SW), lane = (int)(tid % SW);
    int q = g * SW + lane;
    if (opt.set && g == 0 && tid == 0) {
        B.ctrl[0] = 0;
        B.ctrl[1] = opt.max_iter;
        B.ctrl[2] = 1;
        B.ctrl[3] = opt.policy;
        B.ctrl[4] = 0;
        B.ctrl[5] = 0;  // set by a tensor-core LU whose bounded wait ran out during the solve
        B.tol[0] = opt.tol;
        B.tol[1] = opt.refine_below;
        B.tol[2] = opt.reuse_below;
    }
    int src = q < B.n_scen ? q : g * SW;  // padding lanes mirror the group's first scenario
    if (i < n) {
        size_t o = ((size_t)g * n + i) * SW + lane;
        B.Sspec[o] = s_in[(size_t)src * n + i];
        double2 v;
        if (v_in) {
            v = v_in[(size_t)(v_shared ? 0 : src) * n + i];
        } else {
            // flat start (cpu_newton_raphson.cpp:77-88): SLACK/PV at u_pu, PQ at 0.98, angle 0
            int t = P.bus_type[i];
            double m = (t == BUS_PQ) ? 0.98 : (u_pu ? u_pu[i] : 1.0);
            v = make_double2(m, 0.0);
        }
        B.V[o] = v;
    }
    if (i < n) {
        if (!B.y_shared) {
            for (int p = i; p < P.nnz_y; p += n)
                B.Y[((size_t)g * P.nnz_y + p) * SW + lane] = y_in[(size_t)src * P.nnz_y + p];
        } else if (g == 0 && lane == 0) {
            for (int p = i; p < P.nnz_y; p += n) B.Y[p] = y_in[p];
        }
    }
    if (i == 0) {
        B.mis_bits[q] = 0ull;
        B.state[q] = q < B.n_scen ? 0 : 1;
        B.solving[q] = q < B.n_scen ? 1 : 0;
        B.singular[q] = 0;
        B.iters[q] = 0;
        B.status[q] = SC_MAXITER;
        B.final_mis[q] = 0.0;
        if (lane == 0) {
            B.gsolve[g] = 1;
            B.giter[g] = 1;
            if (B.grefine) B.grefine[g] = 1;  // the stage API refines unless k_check says not
            if (B.gfactor) B.gfactor[g] = 1;
        }
    }
}

// ---------------------------------------------------------------------------------------
// in-graph control: the retry of unconverged lanes
// ---------------------------------------------------------------------------------------
// Retry after the loop (one CTA): every scenario that ended at max_iterations or with a
// non-finite mismatch starts again with the step policy `policy` (its other scenarios stay
// done); the groups holding one iterate again, refactorising and refining.  With use_cond, sets
// the retry loop's condition to whether any scenario retries.
template <int SW>
__global__ void k_retry_flags(BatchDev B, int policy, int use_cond, cudaGraphConditionalHandle handle) {
    __shared__ int any;
    if (threadIdx.x == 0) any = 0;
    __syncthreads();
    const int total = B.n_groups * SW;
    for (int q = threadIdx.x; q < total; q += blockDim.x) {
        const bool again = q < B.n_scen && (B.status[q] == SC_MAXITER || B.status[q] == SC_NONFINITE);
        if (again) {
            B.state[q] = 0;
            B.solving[q] = 1;
            B.singular[q] = 0;
            B.iters[q] = 0;
            B.status[q] = SC_MAXITER;
            B.mis_bits[q] = 0ull;
            B.final_mis[q] = 0.0;
            any = 1;  // benign race: every writer stores 1
        }
    }
    __syncthreads();
    for (int g = threadIdx.x; g < B.n_groups; g += blockDim.x) {
        int iv = 0;
        for (int l = 0; l < SW; ++l) {
            const int q = g * SW + l;
            iv |= q < B.n_scen && B.state[q] == 0;
        }
        B.gsolve[g] = iv;
        B.giter[g] = iv;
        if (B.grefine) B.grefine[g] = 1;
        if (B.gfactor) B.gfactor[g] = 1;
    }
    if (threadIdx.x == 0) {
        B.ctrl[0] = 0;
        B.ctrl[2] = any;
        B.ctrl[3] = policy;
        if (any) B.ctrl[4] = 0;  // the retry's loop counts anew
        if (use_cond) cudaGraphSetConditional(handle, any ? 1u : 0u);
    }
}

// The retried scenarios' voltages back at their start (as k_load sets them).
template <int SW>
__global__ void k_retry_v(PlanDev P, BatchDev B, const double2* __restrict__ v_in,
                          const double* __restrict__ u_pu, int v_shared) {
    const int g = blockIdx.y;
    const long tid = (long)blockIdx.x * blockDim.x + threadIdx.x;
    const int i = (int)(tid / SW), lane = (int)(tid % SW);
    const int q = g * SW + lane;
    if (i >= P.n_bus || q >= B.n_scen || B.state[q] != 0) return;
    double2 v;
    if (v_in) {
        v = v_in[(size_t)(v_shared ? 0 : q) * P.n_bus + i];
    } else {
        const int t = P.bus_type[i];
        v = make_double2((t == BUS_PQ) ? 0.98 : (u_pu ? u_pu[i] : 1.0), 0.0);
    }
    B.V[((size_t)g * P.n_bus + i) * SW + lane] = v;
}

// ---------------------------------------------------------------------------------------
// mismatch: fused Y*V SpMV, S = V conj(I), Delta, rhs, per-scenario max |Delta|
// ---------------------------------------------------------------------------------------
// Each CTA covers MM_TILES consecutive tiles of 256 / SW buses (x SW lanes); the per-scenario
// maxima are reduced within the CTA (shuffles, then shared memory) before one atomicMax per
// lane, so a group's scenarios see n / (MM_TILES * 256 / SW) atomics instead of one per warp
// (same-address atomics serialise in L2).
constexpr int MM_TILES = 4;

template <int SW>
__global__ void __launch_bounds__(256, 8) k_mismatch(PlanDev P, BatchDev B) {
    const int g = blockIdx.y;
    if (!B.giter[g]) return;
    const int n = P.n_bus;
    const int lane = threadIdx.x % SW;
    const double2* Vg = B.V + (size_t)g * n * SW;
    const double2* Yg = B.y_shared ? B.Y : B.Y + (size_t)g * P.nnz_y * SW;
    const int ys = B.y_shared ? 0 : 1;  // Y value of entry p at Yg[p * (ys ? SW : 1) + ys * lane]
    double m = 0.0;
    // S = V conj(Y V) and the mismatch of bus i from its accumulated current (vi, sp, t, node:
    // the bus's own voltage, specified power, type and block node).  Loading these before the
    // gathers needs more than the 32 registers of 8 CTAs per SM and measured slower.
    auto finish = [&](int i, double ir, double ii, double2 vi, double2 sp, int t, int node) {
        const size_t o = ((size_t)g * n + i) * SW + lane;
        const double2 s = make_double2(fma(vi.x, ir, vi.y * ii), fma(vi.y, ir, -vi.x * ii));
        B.Scalc[o] = s;
        if (t != BUS_SLACK) {
            const double dp = s.x - sp.x;
            const double dq = (t == BUS_PQ) ? s.y - sp.y : 0.0;
            B.rhs[((size_t)g * P.nb + node) * SW + lane] = make_double2(-dp, -dq);
            m = nmax(m, nmax(fabs(dp), fabs(dq)));
        }
    };
    // two tiles at a time: the rows of buses i0 and i1 = i0 + 256 / SW are walked together, so
    // that each thread keeps two independent column -> V gather chains in flight
#pragma unroll 1
    for (int tile = 0; tile < MM_TILES; tile += 2) {
        const int i0 = ((blockIdx.x * MM_TILES + tile) * blockDim.x + threadIdx.x) / SW;
        const int i1 = i0 + (int)blockDim.x / SW;
        if (i0 >= n) break;
        const bool a1 = i1 < n;
        int p0 = P.y_row_ptr[i0], p1 = a1 ? P.y_row_ptr[i1] : 0;
        const int e0 = P.y_row_ptr[i0 + 1], e1 = a1 ? P.y_row_ptr[i1 + 1] : 0;
        double r0 = 0.0, q0 = 0.0, r1 = 0.0, q1 = 0.0;
        while (p0 < e0 || p1 < e1) {
            if (p0 < e0) {
                const double2 y = ys ? Yg[(size_t)p0 * SW + lane] : Yg[p0];
                const double2 v = Vg[(size_t)P.y_col[p0] * SW + lane];
                r0 = fma(y.x, v.x, r0);
                r0 = fma(-y.y, v.y, r0);
                q0 = fma(y.x, v.y, q0);
                q0 = fma(y.y, v.x, q0);
                ++p0;
            }
            if (p1 < e1) {
                const double2 y = ys ? Yg[(size_t)p1 * SW + lane] : Yg[p1];
                const double2 v = Vg[(size_t)P.y_col[p1] * SW + lane];
                r1 = fma(y.x, v.x, r1);
                r1 = fma(-y.y, v.y, r1);
                q1 = fma(y.x, v.y, q1);
                q1 = fma(y.y, v.x, q1);
                ++p1;
            }
        }
        finish(i0, r0, q0, Vg[(size_t)i0 * SW + lane], B.Sspec[((size_t)g * n + i0) * SW + lane],
               P.bus_type[i0], P.node_of_bus[i0]);
        if (a1)
            finish(i1, r1, q1, Vg[(size_t)i1 * SW + lane], B.Sspec[((size_t)g * n + i1) * SW + lane],
                   P.bus_type[i1], P.node_of_bus[i1]);
    }
#pragma unroll
    for (int off = SW; off < 32; off <<= 1) m = nmax(m, __shfl_xor_sync(0xffffffffu, m, off));
    __shared__ double red[8][8];  // [warp][lane] (blockDim 256, SW <= 8)
    const int w = threadIdx.x >> 5;
    if ((threadIdx.x & 31) < SW) red[w][lane] = m;
    __syncthreads();
    if (threadIdx.x < SW) {
        double r = red[0][threadIdx.x];
        for (int k = 1; k < (int)(blockDim.x >> 5); ++k) r = nmax(r, red[k][threadIdx.x]);
        if (r != 0.0)
            atomicMax(&B.mis_bits[g * SW + threadIdx.x], (unsigned long long)__double_as_longlong(r));
    }
}

// Grid of k_mismatch for G lane groups.
template <int SW>
inline dim3 mismatch_grid(PlanDev const& P, int G) {
    const long per = (long)MM_TILES * 256;
    return dim3((unsigned)(((long)P.n_bus * SW + per - 1) / per), (unsigned)G);
}

// ---------------------------------------------------------------------------------------
// convergence test and loop control (one CTA)
// ---------------------------------------------------------------------------------------
template <int SW>
__global__ void k_check(BatchDev B, int use_cond, cudaGraphConditionalHandle handle) {
    __shared__ int any_iter;
    if (threadIdx.x == 0) any_iter = 0;
    __syncthreads();
    const int it = B.ctrl[0];
    const int max_iter = B.ctrl[1];
    const double tol = B.tol[0];
    const int total = B.n_groups * SW;
    for (int q = threadIdx.x; q < total; q += blockDim.x) {
        if (q >= B.n_scen || B.state[q] != 0) {
            B.solving[q] = 0;
            continue;
        }
        const double m = __longlong_as_double((long long)B.mis_bits[q]);
        B.mis_bits[q] = 0ull;
        B.final_mis[q] = m;
        if (!isfinite(m)) {
            B.state[q] = 1;
            B.status[q] = SC_NONFINITE;
            B.iters[q] = it + 1;
            B.solving[q] = 0;
        } else if (m < tol) {
            B.state[q] = 1;
            B.status[q] = SC_CONVERGED;
            B.iters[q] = it + 1;
            B.solving[q] = 0;
        } else {
            B.solving[q] = 1;
            if (it + 1 >= max_iter) {
                B.state[q] = 1;
                B.status[q] = SC_MAXITER;
                B.iters[q] = max_iter;
            }
        }
    }
    __syncthreads();
    for (int g = threadIdx.x; g < B.n_groups; g += blockDim.x) {
        int sv = 0, iv = 0;
        for (int l = 0; l < SW; ++l) {
            const int q = g * SW + l;
            if (q < B.n_scen) {
                sv |= B.solving[q];
                iv |= (B.state[q] == 0);
            }
        }
        B.gsolve[g] = sv;
        B.giter[g] = iv;
        if (B.grefine) {
            // refinement only once some iterating lane of the group is close to convergence
            const double rb = B.tol[1];
            int rv = rb <= 0.0;
            for (int l = 0; l < SW && !rv; ++l) {
                const int q = g * SW + l;
                if (q < B.n_scen && B.solving[q] && B.final_mis[q] < rb) rv = 1;
            }
            // the factors are reused once every iterating lane of the group is below [2];
            // the solve is then refined against the current FP64 Jacobian.  Only factors of this
            // solve: before its first iteration the batch holds none, or another state's
            const double rf = B.tol[2];
            int fv = 1;
            if (B.gfactor && rf > 0.0 && sv && it > 0) {
                fv = 0;
                for (int l = 0; l < SW; ++l) {
                    const int q = g * SW + l;
                    if (q < B.n_scen && B.solving[q] && !(B.final_mis[q] < rf)) fv = 1;
                }
            }
            if (B.gfactor) B.gfactor[g] = fv;
            B.grefine[g] = rv || !fv;
        }
        if (iv) atomicOr(&any_iter, 1);
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        B.ctrl[0] = it + 1;
        B.ctrl[2] = any_iter;
        B.ctrl[4] = it + 1;
        if (use_cond) cudaGraphSetConditional(handle, any_iter ? 1u : 0u);
    }
}

// ---------------------------------------------------------------------------------------
// Jacobian value fill on the fixed factor pattern (fill-in slots are zeroed)
// ---------------------------------------------------------------------------------------
__device__ __forceinline__ void polar_parts(double2 v, double& vmr, double& c, double& s) {
    const double vm = hypot(v.x, v.y);
    if (vm > 0.0) {
        const double inv = 1.0 / vm;  // one division for both direction cosines
        c = v.x * inv;
        s = v.y * inv;
    } else {
        c = 1.0;
        s = 0.0;
    }
    vmr = vm < 1e-6 ? 1.0 : vm;
}

// The Jacobian block of bus i's own entry (G + jB its diagonal admittance, S its power).
__device__ __forceinline__ Blk<double> jac_diag(double G, double Bv, double2 v, double2 S, bool pq) {
    double n = v.x * v.x + v.y * v.y, ivm = rsqrt(n), vm = n * ivm;
    if (n < 1.1e-12) {  // |V| below 1e-6 counts as 1
        double c, s;
        polar_parts(v, vm, c, s);
        n = vm * vm;
        ivm = 1.0 / vm;
    }
    if (!pq) return {-S.y - Bv * n, 0.0, 0.0, 1.0};
    return {-S.y - Bv * n, S.x * ivm + G * vm, S.x - G * n, S.y * ivm - Bv * vm};
}
// The block of buses i (row) and j (column) joined by the admittance G + jB: with the products
// |V_i||V_j| cos / sin(theta_i - theta_j) = Re / Im(V_i conj(V_j)) it needs one reciprocal root
// and no polar form (two hypot and two divisions made the fill FP64-issue bound).
__device__ __forceinline__ Blk<double> jac_off(double G, double Bv, double2 vi, double2 vj, bool pqi,
                                               bool pqj) {
    const double ni = vi.x * vi.x + vi.y * vi.y, nj = vj.x * vj.x + vj.y * vj.y;
    double pr = vi.x * vj.x + vi.y * vj.y, pi = vi.y * vj.x - vi.x * vj.y, rj = rsqrt(nj);
    if (ni < 1.1e-12 || nj < 1.1e-12) {  // |V| below 1e-6 counts as 1, along its direction
        double vmi, ci, sni, vmj, cj, snj;
        polar_parts(vi, vmi, ci, sni);
        polar_parts(vj, vmj, cj, snj);
        pr = vmi * vmj * (ci * cj + sni * snj);
        pi = vmi * vmj * (sni * cj - ci * snj);
        rj = 1.0 / vmj;
    }
    const double t = G * pr + Bv * pi, u = G * pi - Bv * pr;
    Blk<double> J = {u, t * rj, -t, u * rj};
    if (!pqi) {
        J.c = 0.0;
        J.d = 0.0;
    }
    if (!pqj) {
        J.b = 0.0;
        J.d = 0.0;
    }
    return J;
}
// Reference mode: convert_to_sparse_matrix drops |x| <= 1e-12 (cpu_newton_raphson.cpp:754).
__device__ __forceinline__ void jac_drop(Blk<double>& J, bool diag) {
    if (fabs(J.a) <= 1e-12) J.a = 0.0;
    if (fabs(J.b) <= 1e-12) J.b = 0.0;
    if (fabs(J.c) <= 1e-12) J.c = 0.0;
    if (fabs(J.d) <= 1e-12 && !(diag && J.d == 1.0)) J.d = 0.0;
}

// One record per Jacobian block (P.a_rec): its slot, its row and column bus (bit 30: a PQ bus)
// and the Y entry it is made of, or -1 where the sources are listed (none, or several) -- one
// load where slot, slot_info, slot_src and the bus types were a chain of four.
constexpr int REC_PQ = 1 << 30, REC_BUS = REC_PQ - 1;

// Block a of the Jacobian at voltages v(bus), powers s(bus) and admittances y(entry).
template <typename FV, typename FS, typename FY>
__device__ __forceinline__ Blk<double> jac_block(PlanDev const& P, int4 rec, FV v, FS s, FY y) {
    const int i = rec.y & REC_BUS, j = rec.z & REC_BUS;
    const bool diag = i == j, pqi = rec.y & REC_PQ, pqj = rec.z & REC_PQ;
    const double2 vi = v(i), vj = v(j);
    double G = 0.0, Bv = 0.0;
    if (rec.w >= 0) {
        const double2 a = y(rec.w);
        G = a.x;
        Bv = a.y;
    } else {
        const int4 si = P.slot_info[rec.x];
        if (!diag && si.z >= si.w) return {0.0, 0.0, 0.0, 0.0};
        for (int e = si.z; e < si.w; ++e) {
            const double2 a = y(P.slot_src[e]);
            G += a.x;
            Bv += a.y;
        }
    }
    Blk<double> J = diag ? jac_diag(G, Bv, vi, s(i), pqi) : jac_off(G, Bv, vi, vj, pqi, pqj);
    if (P.jac_mode == 0) jac_drop(J, diag);
    return J;
}

template <typename T, int SW>
__global__ void __launch_bounds__(256) k_jfill(PlanDev P, BatchDev B) {
    const int g = blockIdx.y;
    if (!B.gsolve[g]) return;
    const int tid = blockIdx.x * blockDim.x + threadIdx.x;
    const int a_idx = tid / SW, lane = tid % SW;
    if (a_idx >= P.n_a) return;
    const int4 rec = P.a_rec[a_idx];
    const int slot = rec.x, n = P.n_bus;
    const Blk<double> J = jac_block(
        P, rec, [&](int i) { return B.V[((size_t)g * n + i) * SW + lane]; },
        [&](int i) { return B.Scalc[((size_t)g * n + i) * SW + lane]; },
        [&](int p) { return B.y_shared ? B.Y[p] : B.Y[((size_t)g * P.nnz_y + p) * SW + lane]; });
    if (!B.gfactor || B.gfactor[g]) {  // a group that reuses its factors keeps them
        Blk<T>* F = reinterpret_cast<Blk<T>*>(B.F) + ((size_t)g * P.n_slots + slot) * SW + lane;
        stb(F, Blk<T>{(T)J.a, (T)J.b, (T)J.c, (T)J.d});
    }
    // the FP64 copy feeds only the refinement residual: skipped for groups that do not
    // refine this iteration
    if (B.A64 && (!B.grefine || B.grefine[g])) {
        Blk<double>* A = reinterpret_cast<Blk<double>*>(B.A64) +
                         ((size_t)g * P.n_a + a_idx) * SW + lane;
        stb(A, J);
    }
}

// ---------------------------------------------------------------------------------------
// The level-scheduled kernels (k_factor, k_solve_fwd, k_solve_bwd) give a lane group one CTA, or
// a cluster of up to 8 CTAs when the batch has too few groups to fill the GPU (level_ctas): its
// wide levels are spread over the cluster's threads, with a cluster barrier (release / acquire,
// so that the other CTAs' global writes are seen) where one CTA has __syncthreads.  How sums are
// split over threads does not depend on the cluster: the solves split by the CTA size, the
// factorisation by split_slots, the slots that the batch has when it runs alone (0: no splits).
// Both are bound by the latency of dependent gathers, level after level.  30,000 buses x 8
// scenarios (one group, FP32): factor 1,480 -> 374 us, forward 351 -> 124, backward 369 -> 152;
// 10,000 buses x 256 in FP64 (32 groups, 256 -> 1024 threads a CTA): 2,249 -> 541, 948 -> 191,
// 954 -> 212 us, of which the CTA size alone 1,041, 335 and 348; x 1024 in FP32 (128 groups of one
// CTA): 843 -> 822, 315 -> 297, 330 -> 314.  In the narrow levels warps without rows go straight to
// the barrier, and a split row's entries are loaded ROW_BATCH at a time (left to the compiler:
// backward 222 us at 30,000 buses, 152 so).
// ---------------------------------------------------------------------------------------
struct LevelCta {
    int nc, rank, g;
    __device__ __forceinline__ LevelCta() {
        asm("mov.u32 %0, %%cluster_nctaid.x;" : "=r"(nc));
        asm("mov.u32 %0, %%cluster_ctarank;" : "=r"(rank));
        g = blockIdx.x / nc;
    }
    __device__ __forceinline__ LevelCta(int nc, int rank) : nc(nc), rank(rank), g(blockIdx.x / nc) {}
    __device__ __forceinline__ void sync() const {
        if (nc == 1) {
            __syncthreads();
        } else {
            asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
            asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
        }
    }
    // after a level that only rank 0 works on, before another one: the other ranks run ahead
    __device__ __forceinline__ void sync_solo() const {
        if (rank == 0) __syncthreads();
    }
};
// Level bounds in shared memory (read once per level by every thread of every CTA).
constexpr int LV_MAX = 256;
__device__ __forceinline__ const int* level_bounds(const int* ptr, int n_levels, int* buf) {
    if (n_levels > LV_MAX) return ptr;
    for (int i = threadIdx.x; i <= n_levels; i += blockDim.x) buf[i] = ptr[i];
    return buf;
}

// Levels with few nodes split every row over s sub-slots (s a power of two, up to 32): the
// sub-slots of one warp reduce with shuffles, the warps of one row through shared memory.
// split_log: the largest l <= 5 with c << l <= ne (at least 0; c >= 1), s = 1 << l.
__device__ __forceinline__ int split_log(int c, int ne) {
    int l = __clz(c) - __clz(ne);
    if (l > 0 && c << l > ne) --l;
    return max(0, min(l, 5));
}

// Sum `acc` over the s = 1 << ls sub-slots of each row (slot e0 = row * s + sub); the result is
// valid in sub-slot 0.  Every thread of the block calls this (uniform s) unless s <= 32 / SW, where
// whole warps may stay away.
template <typename T, int SW>
__device__ __forceinline__ Vec2<T> split_reduce(Vec2<T> acc, int s, int sub, int row, int lane,
                                                Vec2<T>* red) {
    constexpr int S = 32 / SW;  // slots per warp
    const int sw = s < S ? s : S;
    for (int d = 1; d < sw; d *= 2) {
        acc.x += __shfl_xor_sync(0xffffffffu, acc.x, d * SW);
        acc.y += __shfl_xor_sync(0xffffffffu, acc.y, d * SW);
    }
    if (s > S) {
        const int parts = s / S;
        if (sub % S == 0) red[(row * parts + sub / S) * SW + lane] = acc;
        __syncthreads();
        if (sub == 0) {
            acc = red[(row * parts) * SW + lane];
            for (int w = 1; w < parts; ++w) {
                const Vec2<T> v = red[(row * parts + w) * SW + lane];
                acc.x += v.x;
                acc.y += v.y;
            }
        }
    }
    return acc;
}

// ---------------------------------------------------------------------------------------
// numeric block LU (left-looking Crout), level by level
// ---------------------------------------------------------------------------------------
// Entries of a split row or target that a thread loads together (as many as 64 registers hold).
template <typename T>
constexpr int ROW_BATCH = sizeof(T) == 4 ? 4 : 2;

// acc -= sum of the block products of pairs p, p + step, ... < pe, U pairs' blocks loaded together:
// left to the compiler the loop keeps one or two in flight.
template <typename T, int SW, int U>
__device__ __forceinline__ void pair_sum(Blk<T>& acc, const Blk<T>* F, const int2* pairs, int lane, int p,
                                         int pe, int step) {
    for (; p + (U - 1) * step < pe; p += U * step) {
        int2 r[U];
        Blk<T> a[U], b[U];
#pragma unroll
        for (int u = 0; u < U; ++u) r[u] = pairs[p + u * step];
#pragma unroll
        for (int u = 0; u < U; ++u) {
            a[u] = ldb(F + (size_t)r[u].x * SW + lane);
            b[u] = ldb(F + (size_t)r[u].y * SW + lane);
        }
#pragma unroll
        for (int u = 0; u < U; ++u) msub(acc, a[u], b[u]);
    }
    for (; p < pe; p += step) {
        const int2 r = pairs[p];
        msub(acc, ldb(F + (size_t)r.x * SW + lane), ldb(F + (size_t)r.y * SW + lane));
    }
}

// SPLIT: narrow levels split their targets over split_slots.  Without it the kernel has registers to
// spare for its two targets in flight: one scenario of 100 / 300 / 1,000 buses in FP64 57 / 68 / 72 us,
// 62 / 72 / 73 with the split code in it and not taken.
template <typename T, int SW, bool SPLIT>
__global__ void __launch_bounds__(1024) k_factor(PlanDev P, BatchDev B, int split_slots) {
    // read again where they are used, which frees two registers; the sweeps, with registers to spare,
    // are faster with the values kept (10,000 buses x 1024: 0.32 against 0.35 ms)
    const LevelCta cta(__clusterSizeInBlocks(), __clusterRelativeBlockRank());
    const int g = cta.g;
    if (!B.gsolve[g] || (B.gfactor && !B.gfactor[g])) return;
    __shared__ int fa_buf[LV_MAX + 1], fb_buf[LV_MAX + 1];
    const int* fa = level_bounds(P.fa_ptr, P.n_levels, fa_buf);
    const int* fb = level_bounds(P.fb_ptr, P.n_levels, fb_buf);
    Blk<T>* F = reinterpret_cast<Blk<T>*>(B.F) + (size_t)g * P.n_slots * SW;
    const int lane = threadIdx.x % SW;
    const int e0 = (cta.rank * blockDim.x + threadIdx.x) / SW, ne = cta.nc * blockDim.x / SW;
    constexpr int SW_LOG = SW == 8 ? 3 : SW == 4 ? 2 : SW == 2 ? 1 : 0;
    bool bad = false;
    if (B.lvl_ts) lvl_stamp(B, P.n_levels, 0, g, 0, cta.rank);
    __syncthreads();
    for (int h = 0; h < P.n_levels; ++h) {
        const int ta = fa[h], tb = fa[h + 1];
        const int ls = SPLIT && tb > ta ? min(split_log(tb - ta, split_slots), 5 - SW_LOG) : 0, s = 1 << ls;
        if (SPLIT && s > 1) {
            // narrow levels: s neighbouring threads share a target's pairs (the longest lists, 20
            // to 40 pairs, set the level's latency)
            const int sub = e0 & (s - 1), wl = e0 % (32 / SW);
            for (int e = e0; e - wl < (tb - ta) << ls; e += ne) {
                const bool on = e < (tb - ta) << ls;
                const int4 tg = on ? P.targets[ta + (e >> ls)] : make_int4(0, 0, 0, 0);
                Blk<T> acc = on && sub == 0 && (tg.w & 2) ? ldb(F + (size_t)tg.x * SW + lane) : Blk<T>{0, 0, 0, 0};
                pair_sum<T, SW, ROW_BATCH<T>>(acc, F, P.pairs, lane, tg.y + sub, tg.z, s);
                for (int d = SW; d < s * SW; d <<= 1) {
                    acc.a += __shfl_xor_sync(0xffffffffu, acc.a, d);
                    acc.b += __shfl_xor_sync(0xffffffffu, acc.b, d);
                    acc.c += __shfl_xor_sync(0xffffffffu, acc.c, d);
                    acc.d += __shfl_xor_sync(0xffffffffu, acc.d, d);
                }
                if (on && sub == 0) {
                    if (tg.w & 1) {
                        bool ok;
                        acc = inv2(acc, ok);
                        bad |= !ok;
                    }
                    stb(F + (size_t)tg.x * SW + lane, acc);
                }
            }
        }
        // two targets per worker at a time (targets of one level are independent), so that
        // their gathers overlap in memory
        for (int t = SPLIT && s > 1 ? tb : ta + e0; t < tb; t += 2 * ne) {
            const bool two = t + ne < tb;
            const int4 tg = P.targets[t];
            const int4 tg2 = two ? P.targets[t + ne] : make_int4(0, 0, 0, 0);
            Blk<T> acc = (tg.w & 2) ? ldb(F + (size_t)tg.x * SW + lane) : Blk<T>{0, 0, 0, 0};
            Blk<T> acc2 = (tg2.w & 2) ? ldb(F + (size_t)tg2.x * SW + lane) : Blk<T>{0, 0, 0, 0};
            const int nb = min(tg.z - tg.y, tg2.z - tg2.y);
#pragma unroll 2
            for (int i = 0; i < nb; ++i) {
                const int2 pr = P.pairs[tg.y + i];
                const int2 pr2 = P.pairs[tg2.y + i];
                msub(acc, ldb(F + (size_t)pr.x * SW + lane), ldb(F + (size_t)pr.y * SW + lane));
                msub(acc2, ldb(F + (size_t)pr2.x * SW + lane), ldb(F + (size_t)pr2.y * SW + lane));
            }
#pragma unroll 4
            for (int p = tg.y + nb; p < tg.z; ++p) {
                const int2 pr = P.pairs[p];
                msub(acc, ldb(F + (size_t)pr.x * SW + lane), ldb(F + (size_t)pr.y * SW + lane));
            }
#pragma unroll 4
            for (int p = tg2.y + nb; p < tg2.z; ++p) {
                const int2 pr = P.pairs[p];
                msub(acc2, ldb(F + (size_t)pr.x * SW + lane), ldb(F + (size_t)pr.y * SW + lane));
            }
            if (tg.w & 1) {
                bool ok;
                acc = inv2(acc, ok);
                bad |= !ok;
            }
            stb(F + (size_t)tg.x * SW + lane, acc);
            if (two) {
                if (tg2.w & 1) {
                    bool ok;
                    acc2 = inv2(acc2, ok);
                    bad |= !ok;
                }
                stb(F + (size_t)tg2.x * SW + lane, acc2);
            }
        }
        cta.sync();
        const int sa = fb[h], sb = fb[h + 1];
        if (sb > sa) {
            for (int t = sa + e0; t < sb; t += ne) {
                const int2 sc = P.scale[t];
                Blk<T>* Lp = F + (size_t)sc.x * SW + lane;
                stb(Lp, mul(ldb(Lp), ldb(F + (size_t)sc.y * SW + lane)));
            }
            cta.sync();
        }
        if (B.lvl_ts) lvl_stamp(B, P.n_levels, 0, g, h + 1, cta.rank);
    }
    if (B.lvl_ts) lvl_stamp(B, P.n_levels, 0, g, P.n_levels + 1, cta.rank);
    if (bad) B.singular[g * SW + lane] = 1;
}

// ---------------------------------------------------------------------------------------
// dense tail: Schur-complement gather from the sparse part, blocked dense LU, dense solves
// ---------------------------------------------------------------------------------------
// Row stride of the dense tail: N rounded up to 8, so that every 8-column group that starts
// on a multiple of 8 stays inside its (padded) row.
__host__ __device__ __forceinline__ int dense_ld(int N) { return (N + 7) & ~7; }

template <typename T>
struct V4 {
    T v[4];
};
__device__ __forceinline__ V4<float> ld4(const float* p) {
    const float4 a = *reinterpret_cast<const float4*>(p);
    return {{a.x, a.y, a.z, a.w}};
}
__device__ __forceinline__ V4<double> ld4(const double* p) {
    const double2 a = reinterpret_cast<const double2*>(p)[0];
    const double2 b = reinterpret_cast<const double2*>(p)[1];
    return {{a.x, a.y, b.x, b.y}};
}
__device__ __forceinline__ void st4(float* p, V4<float> const& a) {
    *reinterpret_cast<float4*>(p) = make_float4(a.v[0], a.v[1], a.v[2], a.v[3]);
}
__device__ __forceinline__ void st4(double* p, V4<double> const& a) {
    reinterpret_cast<double2*>(p)[0] = make_double2(a.v[0], a.v[1]);
    reinterpret_cast<double2*>(p)[1] = make_double2(a.v[2], a.v[3]);
}

// Two pairs' blocks in flight per thread, and the CTAs per SM that this leaves registers for: one
// pair more costs resident warps.  10,000 buses: 1024 scenarios in FP32 1,250 -> 1,140 us (1 / 3 / 4
// pairs: 1,335 / 1,398 / 1,464), 256 in FP64 608 -> 591 us (8 CTAs: 837).
template <typename T, int SW>
__global__ void __launch_bounds__(256, sizeof(T) == 4 ? 8 : 6) k_schur(PlanDev P, BatchDev B) {
    const int g = blockIdx.y;
    if (!B.gsolve[g] || (B.gfactor && !B.gfactor[g])) return;
    const int tid = blockIdx.x * blockDim.x + threadIdx.x;
    const int t = tid / SW, lane = tid % SW;
    if (t >= P.n_schur) return;
    const int q = g * SW + lane;
    const Blk<T>* F = reinterpret_cast<const Blk<T>*>(B.F) + (size_t)g * P.n_slots * SW;
    const int4 tg = P.schur[t];
    Blk<T> acc = (tg.w >> 30) ? ldb(F + (size_t)tg.x * SW + lane) : Blk<T>{0, 0, 0, 0};
    pair_sum<T, SW, 2>(acc, F, P.pairs, lane, tg.y, tg.z, 1);
    const int N = 2 * P.n_tail, ld = dense_ld(N);
    const int pos = tg.w & ((1 << 30) - 1);
    const int r = 2 * (pos / P.n_tail), c = 2 * (pos % P.n_tail);
    T* D = reinterpret_cast<T*>(B.Dt) + (size_t)q * N * ld;
    D[(size_t)r * ld + c] = acc.a;
    D[(size_t)r * ld + c + 1] = acc.b;
    D[(size_t)(r + 1) * ld + c] = acc.c;
    D[(size_t)(r + 1) * ld + c + 1] = acc.d;
}

// Asynchronous global -> shared copies (cp.async): the copies of one thread are all in flight
// together, so a staging loop costs one memory latency instead of one per element.
template <int BYTES>
__device__ __forceinline__ void cp_async(void* smem, const void* gmem) {
    const unsigned s = (unsigned)__cvta_generic_to_shared(smem);
    if constexpr (BYTES == 16)
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(s), "l"(gmem) : "memory");
    else
        asm volatile("cp.async.ca.shared.global [%0], [%1], %2;\n" ::"r"(s), "l"(gmem), "n"(BYTES)
                     : "memory");
}
__device__ __forceinline__ void cp_async_wait_all() { asm volatile("cp.async.wait_all;\n" ::: "memory"); }
// Hint: bring the line holding p into L2 (no register result, nothing to wait for).
__device__ __forceinline__ void prefetch_l2(const void* p) {
    asm volatile("prefetch.global.L2 [%0];" ::"l"(p));
}

// Right-looking blocked LU without pivoting of one scenario's N x N tail (row-major, row
// stride dense_ld(N), in place), panels of W columns (W = 8, 16 or 32; compile time):
//   A. warp 0 factors the W x W diagonal block in registers (lane r holds row r; the pivot
//      row is broadcast with shuffles) and publishes U11 (transposed, in the panel buffer),
//      L11 (row-major) and 1/diag(U11) in shared memory;
//   B. every thread then solves whole rows of L21 (x U11 = a) and whole columns of U12
//      (L11 y = a), register resident and independent of each other -- two barriers per panel
//      in all; the L21 rows also go to the transposed panel buffer PT[c][r] for the trailing
//      update;
//   C. the trailing update streams U12 through a double-buffered shared-memory chunk of DCW
//      columns (cp.async prefetch of chunk i+1 during chunk i, one barrier per chunk); each
//      thread owns 8x8 register tiles and per k reads 8 rows of L21 and 8 columns of U12 (four
//      vector loads) for 64 FMAs.  The trailing matrix is read and written once per panel.
// Rows and columns past the last partial panel are padded with the identity, which leaves the
// factors unchanged.  A pivot below 1e-14 in magnitude (the reference LU's tolerance) marks the
// scenario singular.  Shared memory: dense_lu_elems(N, W) elements.  The register-resident
// steps A and B are separate (non-inlined) functions: each then gets the full register budget
// for its unrolled W-element row, instead of sharing it with the trailing-update tiles.
constexpr int DCW = 128;

__host__ __device__ __forceinline__ size_t dense_lu_elems(int N, int W) {
    return (size_t)W * dense_ld(N) + 2 * (size_t)W * DCW + (size_t)W * (W + 4) + (size_t)W;
}

// A: factor the diagonal block A[k0.., k0..] (w <= W rows and columns) in the lanes of one warp.
// Returns 1 if a pivot is below the tolerance.
template <typename T, int W>
__device__ __noinline__ int dense_diag_block(T* A, int ld, int k0, int w, T* PT, int pld, T* SL,
                                             T* SD) {
    const int r = threadIdx.x & 31;
    T a[W];
    if (r < w) {
        const T* row = A + (size_t)(k0 + r) * ld + k0;
#pragma unroll
        for (int c4 = 0; c4 < W; c4 += 4) {
            // columns up to ld - 1 lie inside the padded row
            const V4<T> v = k0 + c4 < ld ? ld4(row + c4) : V4<T>{{T(0), T(0), T(0), T(0)}};
#pragma unroll
            for (int t = 0; t < 4; ++t) a[c4 + t] = c4 + t < w ? v.v[t] : T(0);
        }
    } else {
#pragma unroll
        for (int c = 0; c < W; ++c) a[c] = c == r ? T(1) : T(0);
    }
    int badl = 0;
#pragma unroll
    for (int kk = 0; kk < W; ++kk) {
        const T piv = __shfl_sync(0xffffffffu, a[kk], kk);
        if (kk < w && !(fabs(piv) >= T(1e-14))) badl = 1;
        const T inv = T(1) / piv;
        if (r == 0) SD[kk] = inv;
        const bool below = r > kk;
        const T l = a[kk] * inv;
        if (below) a[kk] = l;
#pragma unroll
        for (int c = kk + 1; c < W; ++c) {
            const T u = __shfl_sync(0xffffffffu, a[c], kk);
            if (below) a[c] = fma(-l, u, a[c]);
        }
    }
    if (r < W) {
#pragma unroll
        for (int c = 0; c < W; ++c) PT[c * pld + r] = a[c];  // U11 read as PT[c][k], k <= c
    }
    if (r < w) {
        T* row = A + (size_t)(k0 + r) * ld + k0;
        if (w == W) {
#pragma unroll
            for (int c4 = 0; c4 < W; c4 += 4) st4(row + c4, V4<T>{{a[c4], a[c4 + 1], a[c4 + 2], a[c4 + 3]}});
        } else {
#pragma unroll
            for (int c = 0; c < W; ++c)
                if (c < w) row[c] = a[c];
        }
    }
    if (r < W) {
#pragma unroll
        for (int c = 0; c < W; ++c) SL[r * (W + 4) + c] = a[c];  // L11 row-major, stride W + 4
    }
    return badl;
}

// B, one row of L21: x U11 = a for the row at `row` (W values; U11 transposed in PT with row
// stride pld), written back and, when PTr is given, to PTr[c * pld].
template <typename T, int W>
__device__ __noinline__ void dense_l21_row(T* row, const T* PT, int pld, const T* SD, T* PTr) {
    T x[W];
#pragma unroll
    for (int c4 = 0; c4 < W; c4 += 4) {
        const V4<T> v = ld4(row + c4);
#pragma unroll
        for (int t = 0; t < 4; ++t) x[c4 + t] = v.v[t];
    }
#pragma unroll
    for (int c = 0; c < W; ++c) {
        T s0 = x[c], s1 = T(0);
#pragma unroll
        for (int k4 = 0; k4 < c; k4 += 4) {
            const V4<T> u = ld4(PT + c * pld + k4);
#pragma unroll
            for (int t = 0; t < 4; ++t)
                if (k4 + t < c) {
                    if (t & 1) s1 = fma(-x[k4 + t], u.v[t], s1);
                    else s0 = fma(-x[k4 + t], u.v[t], s0);
                }
        }
        x[c] = (s0 + s1) * SD[c];
    }
    if (PTr) {
#pragma unroll
        for (int c = 0; c < W; ++c) PTr[c * pld] = x[c];
    }
#pragma unroll
    for (int c4 = 0; c4 < W; c4 += 4) st4(row + c4, V4<T>{{x[c4], x[c4 + 1], x[c4 + 2], x[c4 + 3]}});
}

// B, one column of U12: L11 y = a (unit lower) for the column at `col` (W values, stride ld),
// in place; L11 row-major in SL with row stride W + 4.
template <typename T, int W>
__device__ __noinline__ void dense_u12_col(T* col, const T* SL, int ld) {
    T y[W];
#pragma unroll
    for (int i = 0; i < W; ++i) y[i] = col[(size_t)i * ld];
#pragma unroll
    for (int i = 1; i < W; ++i) {
        T s0 = y[i], s1 = T(0);
#pragma unroll
        for (int k4 = 0; k4 < i; k4 += 4) {
            const V4<T> l = ld4(SL + i * (W + 4) + k4);
#pragma unroll
            for (int t = 0; t < 4; ++t)
                if (k4 + t < i) {
                    if (t & 1) s1 = fma(-l.v[t], y[k4 + t], s1);
                    else s0 = fma(-l.v[t], y[k4 + t], s0);
                }
        }
        y[i] = s0 + s1;
    }
#pragma unroll
    for (int i = 0; i < W; ++i) col[(size_t)i * ld] = y[i];
}

template <typename T, int W>
__global__ void __launch_bounds__(256, sizeof(T) == 4 ? 2 : 1) k_dense_lu(BatchDev B, int N) {
    static_assert(W == 8 || W == 16 || W == 32, "panel width");
    const int q = blockIdx.x;
    if (q >= B.n_scen || !B.solving[q] || (B.gfactor && !B.gfactor[q / B.sw])) return;
    const int ld = dense_ld(N);
    T* A = reinterpret_cast<T*>(B.Dt) + (size_t)q * N * ld;
    extern __shared__ __align__(16) unsigned char smraw[];
    T* PT = reinterpret_cast<T*>(smraw);        // [W][ld]: PT[c*ld + r] = panel (r, c)
    T* Ub0 = PT + (size_t)W * ld;               // [W][DCW] U12 chunk, two buffers
    T* Ub1 = Ub0 + W * DCW;
    T* SL = Ub1 + W * DCW;                      // [W][W + 4] L11 row-major
    T* SD = SL + W * (W + 4);                         // [W] 1 / U11 diagonal
    __shared__ int bad;
    const int tid = threadIdx.x, nt = blockDim.x;
    constexpr int VE = 16 / sizeof(T);
    if (tid == 0) bad = 0;
    // panel trace stamp j of this scenario (the address is rebuilt from the kernel
    // parameters at each stamp, so that the trace holds no registers across the loop)
    auto stamp = [&](int j, bool copy_prev) {
        if (B.dlu_ts && tid == 0) {
            unsigned long long* t = B.dlu_ts + (size_t)q * (1 + 3 * ((N + W - 1) / W)) + j;
            *t = copy_prev ? t[-1] : gtimer();
        }
    };
    stamp(0, false);
    for (int k0 = 0; k0 < N; k0 += W) {
        const int w = min(W, N - k0);
        const int m = N - k0;
        const int n2 = m - w;  // > 0 only for full panels
        // ---- A: diagonal block, warp 0
        if (tid < 32) {
            if (dense_diag_block<T, W>(A, ld, k0, w, PT, ld, SL, SD)) bad = 1;
        }
        __syncthreads();
        stamp(1 + 3 * (k0 / W), false);
        if (n2 > 0) {
            // ---- B: rows of L21 and columns of U12, one per thread at a time
            for (int it = tid; it < 2 * n2; it += nt) {
                if (it < n2) {
                    const int r = W + it;
                    dense_l21_row<T, W>(A + (size_t)(k0 + r) * ld + k0, PT, ld, SD, PT + r);
                } else {
                    dense_u12_col<T, W>(A + (size_t)k0 * ld + k0 + W + (it - n2), SL, ld);
                }
            }
            __syncthreads();
            stamp(2 + 3 * (k0 / W), false);
            // ---- C: trailing update, U12 in double-buffered chunks
            const int nch = (n2 + DCW - 1) / DCW;
            auto stage = [&](int ch, T* buf) {
                const int c0 = ch * DCW;
                const int cwp = (min(DCW, n2 - c0) + 7) & ~7;
                const int vpr = cwp / VE;
                // the columns past N are row padding and only ever feed padding columns
                for (int e2 = tid; e2 < W * vpr; e2 += nt) {
                    const int r = e2 / vpr, c = (e2 % vpr) * VE;
                    cp_async<16>(buf + r * DCW + c, A + (size_t)(k0 + r) * ld + k0 + W + c0 + c);
                }
            };
            stage(0, Ub0);
            cp_async_wait_all();
            __syncthreads();
            for (int ch = 0; ch < nch; ++ch) {
                T* cur = (ch & 1) ? Ub1 : Ub0;
                if (ch + 1 < nch) stage(ch + 1, (ch & 1) ? Ub0 : Ub1);
                const int c0 = ch * DCW;
                const int tcn = ((min(DCW, n2 - c0) + 7) & ~7) / 8;
                const int tr8 = (n2 + 7) / 8;
                const int ntile = tr8 * tcn;
                for (int tix = tid; tix < ntile; tix += nt) {
                    const int i0 = W + (tix / tcn) * 8, cc0 = (tix % tcn) * 8;
                    if (tix + nt < ntile) {
                        // the thread's next tile goes to L2 while this one computes
                        const int j0 = W + ((tix + nt) / tcn) * 8, dc0 = ((tix + nt) % tcn) * 8;
                        const T* pf = A + (size_t)(k0 + j0) * ld + k0 + W + c0 + dc0;
#pragma unroll
                        for (int ii = 0; ii < 8; ++ii)
                            if (j0 + ii < m) prefetch_l2(pf + (size_t)ii * ld);
                    }
                    T acc[8][8];
#pragma unroll
                    for (int ii = 0; ii < 8; ++ii) {
                        if (i0 + ii < m) {
                            const T* row = A + (size_t)(k0 + i0 + ii) * ld + k0 + W + c0 + cc0;
                            const V4<T> a = ld4(row), b = ld4(row + 4);
#pragma unroll
                            for (int c = 0; c < 4; ++c) { acc[ii][c] = a.v[c]; acc[ii][c + 4] = b.v[c]; }
                        } else {
#pragma unroll
                            for (int c = 0; c < 8; ++c) acc[ii][c] = T(0);
                        }
                    }
#pragma unroll 2
                    for (int r = 0; r < W; ++r) {
                        const V4<T> l0 = ld4(PT + r * ld + i0), l1 = ld4(PT + r * ld + i0 + 4);
                        const V4<T> u0 = ld4(cur + r * DCW + cc0), u1 = ld4(cur + r * DCW + cc0 + 4);
#pragma unroll
                        for (int ii = 0; ii < 4; ++ii)
#pragma unroll
                            for (int c = 0; c < 4; ++c) {
                                acc[ii][c] = fma(-l0.v[ii], u0.v[c], acc[ii][c]);
                                acc[ii][c + 4] = fma(-l0.v[ii], u1.v[c], acc[ii][c + 4]);
                                acc[ii + 4][c] = fma(-l1.v[ii], u0.v[c], acc[ii + 4][c]);
                                acc[ii + 4][c + 4] = fma(-l1.v[ii], u1.v[c], acc[ii + 4][c + 4]);
                            }
                    }
#pragma unroll
                    for (int ii = 0; ii < 8; ++ii) {
                        if (i0 + ii < m) {
                            T* row = A + (size_t)(k0 + i0 + ii) * ld + k0 + W + c0 + cc0;
                            st4(row, V4<T>{{acc[ii][0], acc[ii][1], acc[ii][2], acc[ii][3]}});
                            st4(row + 4, V4<T>{{acc[ii][4], acc[ii][5], acc[ii][6], acc[ii][7]}});
                        }
                    }
                }
                cp_async_wait_all();
                __syncthreads();
            }
        } else {
            stamp(2 + 3 * (k0 / W), true);
        }
        stamp(3 + 3 * (k0 / W), false);
    }
    if (tid == 0 && bad) B.singular[q] = 1;
}

constexpr int DLU_W = 32, DLU_TILE = 64, DLU_ROWS = 128;

// The next diagonal block (k1, k1) by warp 0, its trailing block just updated by this CTA.
// `buf`: shared memory of dlu_diag_elems elements.
constexpr int DLU_DIAG_ELEMS = 2 * DLU_W * (DLU_W + 4) + DLU_W;
template <typename T>
__device__ __forceinline__ void dlu_next_diag(BatchDev const& B, int q, T* A, int ld, int N, int k1, T* buf) {
    if (threadIdx.x < 32) {
        if (dense_diag_block<T, DLU_W>(A, ld, k1, min(DLU_W, N - k1), buf, DLU_W + 4,
                                       buf + DLU_W * (DLU_W + 4), buf + 2 * DLU_W * (DLU_W + 4)))
            B.singular[q] = 1;
    }
}

}  // namespace gapk

#include "dense_lu_tc.cuh"

namespace gapk {

// Host side: opt in to the kernel's shared memory and launch it for panel width W.  With `tc`
// (FP32, W = 32) the tail is factorised by k_dense_lu_tc instead, the trailing update on the
// tensor cores; its shared memory does not depend on N.  k_dense_lu opts in to all that a block may
// have: the attribute is the kernel's, and a batch with a smaller tail must not lower it.
constexpr size_t DENSE_LU_SMEM_MAX = 232448 - 1024;  // opt-in shared memory per block, less static
template <typename T>
cudaError_t dense_lu_attributes(int W, bool tc) {
    auto set = [&](auto fn, size_t bytes) {
        cudaError_t e = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
        if (e == cudaSuccess) e = cudaFuncSetAttribute(fn, cudaFuncAttributePreferredSharedMemoryCarveout, 100);
        return e;
    };
    if constexpr (sizeof(T) == 4) {
        if (tc) return W == 32 ? set(k_dense_lu_tc, dense_lu_tc_smem()) : cudaErrorInvalidValue;
    }
    switch (W) {
        case 32: return set(k_dense_lu<T, 32>, DENSE_LU_SMEM_MAX);
        case 16: return set(k_dense_lu<T, 16>, DENSE_LU_SMEM_MAX);
        case 8: return set(k_dense_lu<T, 8>, DENSE_LU_SMEM_MAX);
    }
    return cudaErrorInvalidValue;
}

template <typename T>
void launch_dense_lu(int W, int grid, size_t smem, cudaStream_t st, BatchDev const& B, int N, bool tc) {
    if constexpr (sizeof(T) == 4) {
        if (tc) {
            k_dense_lu_tc<<<grid, 256, dense_lu_tc_smem(), st>>>(B, N);
            return;
        }
    }
    switch (W) {
        case 32: k_dense_lu<T, 32><<<grid, 256, smem, st>>>(B, N); break;
        case 16: k_dense_lu<T, 16><<<grid, 256, smem, st>>>(B, N); break;
        case 8: k_dense_lu<T, 8><<<grid, 256, smem, st>>>(B, N); break;
    }
}

// Split dense LU (the batch path): the same right-looking factorisation as k_dense_lu, one
// panel of W = 32 columns at a time, as two launches per panel so that the panel's solves and
// the rank-W trailing update of every scenario are spread over many small CTAs:
//   k_dlu_solves one CTA per (scenario, 128 rows of L21 or columns of U12): a thread per row or
//                column, the factored diagonal block staged in shared memory;
//   k_dlu_update one CTA per (scenario, 64 x 64 tile of the trailing matrix): C -= L21 U12 in
//                place; the CTA of tile (0, 0) then factors the next panel's diagonal block (one
//                warp, dense_diag_block), which its tile alone holds, so that no launch waits for
//                that serial step by itself.
// No dynamic shared memory, so the tail size is limited only by device memory.
// With the diagonal block and all its solves in one CTA per scenario, the panels of a tail of
// order 506 took 396 us for one FP64 scenario and 612 us for 256; the solves now take 112 and 458
// us, the diagonal blocks are part of the updates (165 us for one scenario, 173 without them).
// Bound by the solves' and the diagonal block's dependent steps for few scenarios, by the
// re-reading of the trailing matrix for many.
// The first diagonal block.
template <typename T>
__global__ void __launch_bounds__(32) k_dlu_diag(BatchDev B, int N) {
    const int q = blockIdx.x;
    if (q >= B.n_scen || !B.solving[q] || (B.gfactor && !B.gfactor[q / B.sw])) return;
    __shared__ __align__(16) T buf[DLU_DIAG_ELEMS];
    const int ld = dense_ld(N);
    dlu_next_diag<T>(B, q, reinterpret_cast<T*>(B.Dt) + (size_t)q * N * ld, ld, N, 0, buf);
}

template <typename T>
__global__ void __launch_bounds__(DLU_ROWS) k_dlu_solves(BatchDev B, int N, int k0) {
    constexpr int W = DLU_W;
    const int q = blockIdx.y;
    if (q >= B.n_scen || !B.solving[q] || (B.gfactor && !B.gfactor[q / B.sw])) return;
    const int ld = dense_ld(N);
    T* A = reinterpret_cast<T*>(B.Dt) + (size_t)q * N * ld;
    __shared__ __align__(16) T U11[W * (W + 4)];  // transposed: U11[c][k], stride W + 4
    __shared__ __align__(16) T SL[W * (W + 4)];   // L11 row-major, stride W + 4
    __shared__ __align__(16) T SD[W];
    const int tid = threadIdx.x;
    V4<T> blk[2];  // all of a thread's loads in flight together
#pragma unroll
    for (int i = 0; i < 2; ++i) {
        const int e = tid + i * DLU_ROWS;
        blk[i] = ld4(A + (size_t)(k0 + e / (W / 4)) * ld + k0 + (e % (W / 4)) * 4);
    }
#pragma unroll
    for (int i = 0; i < 2; ++i) {
        const int e = tid + i * DLU_ROWS, r = e / (W / 4), c = (e % (W / 4)) * 4;
        st4(SL + r * (W + 4) + c, blk[i]);
#pragma unroll
        for (int t = 0; t < 4; ++t) {
            U11[(c + t) * (W + 4) + r] = blk[i].v[t];
            if (r == c + t) SD[r] = T(1) / blk[i].v[t];
        }
    }
    static_assert(W * W == 2 * 4 * DLU_ROWS);
    __syncthreads();
    const int n2 = N - k0 - W, it = blockIdx.x * DLU_ROWS + tid;
    if (it < n2)
        dense_l21_row<T, W>(A + (size_t)(k0 + W + it) * ld + k0, U11, W + 4, SD, nullptr);
    else if (it < 2 * n2)
        dense_u12_col<T, W>(A + (size_t)k0 * ld + k0 + W + (it - n2), SL, ld);
}

// FP32, CUDA cores: 64 threads, 8 x 8 values each.
__global__ void __launch_bounds__(64, 8) k_dlu_update(BatchDev B, int N, int k0, int tiles_j) {
    using T = float;
    constexpr int W = DLU_W, TS = DLU_TILE;
    const int q = blockIdx.y;
    if (q >= B.n_scen || !B.solving[q] || (B.gfactor && !B.gfactor[q / B.sw])) return;
    const int ld = dense_ld(N);
    T* A = reinterpret_cast<T*>(B.Dt) + (size_t)q * N * ld;
    const int n2 = N - k0 - W;
    const int i0 = (blockIdx.x / tiles_j) * TS, j0 = (blockIdx.x % tiles_j) * TS;
    __shared__ __align__(16) T LT[W][TS];  // LT[c][r] = L21(i0 + r, c)
    __shared__ __align__(16) T UT[W][TS];  // UT[r][c] = U12(r, j0 + c)
    __shared__ __align__(16) T diag[DLU_DIAG_ELEMS];
    const int tid = threadIdx.x;
    T* base = A + (size_t)(k0 + W) * ld + k0 + W;  // trailing matrix origin
    {
        // one L21 row per thread (TS rows, TS threads); rows past the matrix are zero
        const int r = tid;
        if (i0 + r < n2) {
            const T* row = A + (size_t)(k0 + W + i0 + r) * ld + k0;
#pragma unroll
            for (int c4 = 0; c4 < W; c4 += 4) {
                const V4<T> v = ld4(row + c4);
#pragma unroll
                for (int t = 0; t < 4; ++t) LT[c4 + t][r] = v.v[t];
            }
        } else {
#pragma unroll
            for (int c = 0; c < W; ++c) LT[c][r] = T(0);
        }
        // U12 rows 0..W-1, columns j0..j0+TS-1 in groups of 4; a group that starts inside the
        // matrix ends inside the padded row (k0 + W and ld are multiples of 8)
        for (int e = tid; e < W * (TS / 4); e += TS) {
            const int r2 = e / (TS / 4), c = (e % (TS / 4)) * 4;
            const V4<T> v = j0 + c < n2 ? ld4(A + (size_t)(k0 + r2) * ld + k0 + W + j0 + c)
                                        : V4<T>{{T(0), T(0), T(0), T(0)}};
            st4(&UT[r2][c], v);
        }
    }
    __syncthreads();
    const int r0 = (tid / 8) * 8, c0 = (tid % 8) * 8;
    if (i0 + r0 < n2 && j0 + c0 < n2) {
        T acc[8][8];
#pragma unroll
        for (int ii = 0; ii < 8; ++ii) {
            if (i0 + r0 + ii < n2) {
                const T* row = base + (size_t)(i0 + r0 + ii) * ld + j0 + c0;
                const V4<T> a = ld4(row), b = ld4(row + 4);
#pragma unroll
                for (int c = 0; c < 4; ++c) {
                    acc[ii][c] = a.v[c];
                    acc[ii][c + 4] = b.v[c];
                }
            } else {
#pragma unroll
                for (int c = 0; c < 8; ++c) acc[ii][c] = T(0);
            }
        }
#pragma unroll 2
        for (int r = 0; r < W; ++r) {
            const V4<T> l0 = ld4(&LT[r][r0]), l1 = ld4(&LT[r][r0 + 4]);
            const V4<T> u0 = ld4(&UT[r][c0]), u1 = ld4(&UT[r][c0 + 4]);
#pragma unroll
            for (int ii = 0; ii < 4; ++ii)
#pragma unroll
                for (int c = 0; c < 4; ++c) {
                    acc[ii][c] = fma(-l0.v[ii], u0.v[c], acc[ii][c]);
                    acc[ii][c + 4] = fma(-l0.v[ii], u1.v[c], acc[ii][c + 4]);
                    acc[ii + 4][c] = fma(-l1.v[ii], u0.v[c], acc[ii + 4][c]);
                    acc[ii + 4][c + 4] = fma(-l1.v[ii], u1.v[c], acc[ii + 4][c + 4]);
                }
        }
#pragma unroll
        for (int ii = 0; ii < 8; ++ii) {
            if (i0 + r0 + ii < n2) {
                T* row = base + (size_t)(i0 + r0 + ii) * ld + j0 + c0;
                st4(row, V4<T>{{acc[ii][0], acc[ii][1], acc[ii][2], acc[ii][3]}});
                st4(row + 4, V4<T>{{acc[ii][4], acc[ii][5], acc[ii][6], acc[ii][7]}});
            }
        }
    }
    if (blockIdx.x == 0) {
        __syncthreads();
        dlu_next_diag<T>(B, q, A, ld, N, k0 + W, diag);
    }
}

// FP64: 128 threads, 8 rows x 2 column pairs each; a warp's loads and stores of C cover 256
// adjacent bytes of a row, L21 stays row-major in shared memory (a row's value is one broadcast
// read).  256 tails of order 506: 2,858 -> 1,480 us (64 threads with 8 x 8 values each before, rows
// of L21 staged a thread per row).
__global__ void __launch_bounds__(128, 4) k_dlu_update64(BatchDev B, int N, int k0, int tiles_j) {
    using T = double;
    constexpr int W = DLU_W, TS = DLU_TILE;
    const int q = blockIdx.y;
    if (q >= B.n_scen || !B.solving[q] || (B.gfactor && !B.gfactor[q / B.sw])) return;
    const int ld = dense_ld(N);
    T* A = reinterpret_cast<T*>(B.Dt) + (size_t)q * N * ld;
    const int n2 = N - k0 - W;
    const int i0 = (blockIdx.x / tiles_j) * TS, j0 = (blockIdx.x % tiles_j) * TS;
    struct Smem {
        T Ls[TS][W + 2];  // L21(i0 + r, c)
        T Us[W][TS];      // U12(r, j0 + c)
    };
    __shared__ __align__(16) Smem sm;
    auto& Ls = sm.Ls;
    auto& Us = sm.Us;
    const int tid = threadIdx.x;
    T* base = A + (size_t)(k0 + W) * ld + k0 + W;  // trailing matrix origin
    // rows and columns past the matrix are left as they are: they feed values that are not stored
    for (int e = tid; e < TS * (W / 2); e += 128) {
        const int r = e / (W / 2), c = (e % (W / 2)) * 2;
        if (i0 + r < n2) cp_async<16>(&Ls[r][c], A + (size_t)(k0 + W + i0 + r) * ld + k0 + c);
    }
    for (int e = tid; e < W * (TS / 2); e += 128) {
        const int r = e / (TS / 2), c = (e % (TS / 2)) * 2;
        // a pair that starts inside the matrix ends inside the padded row
        if (j0 + c < n2) cp_async<16>(&Us[r][c], A + (size_t)(k0 + r) * ld + k0 + W + j0 + c);
    }
    // rows r0 .. r0 + 7, columns c0 + 32 j and the next, j = 0, 1
    const int r0 = (tid / 16) * 8, c0 = (tid % 16) * 2;
    double2 acc[8][2];
#pragma unroll
    for (int ii = 0; ii < 8; ++ii)
#pragma unroll
        for (int j = 0; j < 2; ++j)
            acc[ii][j] = i0 + r0 + ii < n2 && j0 + c0 + 32 * j < n2
                             ? *reinterpret_cast<const double2*>(base + (size_t)(i0 + r0 + ii) * ld + j0 + c0 + 32 * j)
                             : make_double2(0.0, 0.0);
    cp_async_wait_all();
    __syncthreads();
#pragma unroll 4
    for (int k = 0; k < W; ++k) {
        double2 u[2];
        double l[8];
#pragma unroll
        for (int j = 0; j < 2; ++j) u[j] = *reinterpret_cast<const double2*>(&Us[k][c0 + 32 * j]);
#pragma unroll
        for (int ii = 0; ii < 8; ++ii) l[ii] = Ls[r0 + ii][k];
#pragma unroll
        for (int ii = 0; ii < 8; ++ii)
#pragma unroll
            for (int j = 0; j < 2; ++j) {
                acc[ii][j].x = fma(-l[ii], u[j].x, acc[ii][j].x);
                acc[ii][j].y = fma(-l[ii], u[j].y, acc[ii][j].y);
            }
    }
#pragma unroll
    for (int ii = 0; ii < 8; ++ii)
#pragma unroll
        for (int j = 0; j < 2; ++j)
            if (i0 + r0 + ii < n2 && j0 + c0 + 32 * j < n2)
                *reinterpret_cast<double2*>(base + (size_t)(i0 + r0 + ii) * ld + j0 + c0 + 32 * j) = acc[ii][j];
    if (blockIdx.x == 0) {
        __syncthreads();
        static_assert(offsetof(Smem, Us) == sizeof(Smem::Ls) && sizeof(Smem) >= DLU_DIAG_ELEMS * sizeof(T));
        dlu_next_diag<T>(B, q, A, ld, N, k0 + W, &sm.Ls[0][0]);
    }
}

// Host side: the split factorisation of every scenario's N x N tail (grid = padded scenarios).
// With `tc` (FP32) the trailing updates of at least one full 128 x 128 tile run on the tensor
// cores (k_dlu_update_tc; its shared memory opted in by split_lu_attributes); smaller trailing
// blocks, mostly empty as tensor-core tiles, keep the 64 x 64 CUDA-core tiles.
template <typename T>
void launch_dense_lu_split(int grid, cudaStream_t st, BatchDev const& B, int N, bool tc) {
    k_dlu_diag<T><<<grid, 32, 0, st>>>(B, N);
    for (int k0 = 0; k0 + DLU_W < N; k0 += DLU_W) {
        const int n2 = N - k0 - DLU_W;
        k_dlu_solves<T><<<dim3((2 * n2 + DLU_ROWS - 1) / DLU_ROWS, grid), DLU_ROWS, 0, st>>>(B, N, k0);
        const int tj = (n2 + DLU_TILE - 1) / DLU_TILE;
        if constexpr (sizeof(T) == 8) {
            k_dlu_update64<<<dim3(tj * tj, grid), 128, 0, st>>>(B, N, k0, tj);
        } else if (tc && n2 >= TC_N) {
            const int tt = (n2 + TC_N - 1) / TC_N;
            k_dlu_update_tc<<<dim3(tt * tt, grid), 256, TC_OPER_BYTES, st>>>(B, N, k0, tt);
        } else {
            k_dlu_update<<<dim3(tj * tj, grid), DLU_TILE, 0, st>>>(B, N, k0, tj);
        }
    }
}
inline cudaError_t split_lu_attributes() {
    return cudaFuncSetAttribute(k_dlu_update_tc, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                TC_OPER_BYTES);
}

// Forward (unit L) then backward (U) substitution on one scenario's tail vector, blocked by
// 32 rows.  Per block, the dot products of its rows with the solved part stream the factor:
// warp w takes rows w, w + 8, w + 16, w + 24 of the block together, each lane reading one
// 4-element vector per row per step (128 columns per warp-wide load), so every thread keeps
// four vector loads in flight; the block's 32 x 32 triangle is staged in shared memory by the
// whole CTA (one vector per thread) at the same time, and warp 0 then solves it with shuffles.
// At <= 36 registers, seven CTAs fit on an SM, so a 1024-scenario batch runs in one wave.  y
// lives in shared memory, ld = dense_ld(N) entries, zero beyond N (the factor's padding
// columns hold no values and are masked).
template <typename T>
__device__ __forceinline__ void dense_dot4(const T* __restrict__ A, int ld, int r0, int wid,
                                           int ln, int cb, int ce, int N, const T* y, T acc[4]) {
#pragma unroll
    for (int i = 0; i < 4; ++i) acc[i] = T(0);
#pragma unroll 1
    for (int c = cb + 4 * ln; c < ce; c += 128) {
        const V4<T> yv = ld4(y + c);
        V4<T> a[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const int row = r0 + wid + 8 * i;
            a[i] = row < N ? ld4(A + (size_t)row * ld + c) : V4<T>{{T(0), T(0), T(0), T(0)}};
        }
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
            for (int t = 0; t < 4; ++t) acc[i] = fma(c + t < N ? a[i].v[t] : T(0), yv.v[t], acc[i]);
    }
}

// The 32 x 32 diagonal block at (r0, r0) into tri[32][33], one 4-vector per thread of the
// first 256 (a vector that starts inside the padded row ends inside it, ld % 8 == 0).
template <typename T>
__device__ __forceinline__ void dense_stage_tri(const T* __restrict__ A, int ld, int r0, int N,
                                                T (*tri)[33]) {
    const int t = threadIdx.x;
    if (t < 256) {
        const int r = t >> 3, c = (t & 7) * 4;
        const V4<T> v = r0 + r < N && r0 + c < ld ? ld4(A + (size_t)(r0 + r) * ld + r0 + c)
                                                 : V4<T>{{T(0), T(0), T(0), T(0)}};
#pragma unroll
        for (int k = 0; k < 4; ++k) tri[r][c + k] = v.v[k];
    }
}

template <typename T, int SW>
__global__ void __launch_bounds__(256, sizeof(T) == 4 ? 7 : 4) k_dense_solve(PlanDev P, BatchDev B, double2* out,
                                                        int accumulate) {
    const int q = blockIdx.x;
    if (q >= B.n_scen || !B.solving[q]) return;
    const int g = q / SW, lane = q % SW;
    if (accumulate && B.grefine && !B.grefine[g]) return;
    const int N = 2 * P.n_tail, ld = dense_ld(N);
    const T* A = reinterpret_cast<const T*>(B.Dt) + (size_t)q * N * ld;
    Vec2<T>* X = reinterpret_cast<Vec2<T>*>(B.X) + (size_t)g * P.nb * SW;
    extern __shared__ __align__(16) unsigned char smraw[];
    T* y = reinterpret_cast<T*>(smraw);
    __shared__ T tri[32][33];
    const int tid = threadIdx.x, wid = tid >> 5, ln = tid & 31;
    for (int i = tid; i < ld / 2; i += blockDim.x) {
        const Vec2<T> v = i < P.n_tail ? ldv(X + (size_t)(P.ns + i) * SW + lane) : Vec2<T>{T(0), T(0)};
        y[2 * i] = v.x;
        y[2 * i + 1] = v.y;
    }
    __syncthreads();
    // L y = b, unit lower
    for (int r0 = 0; r0 < N; r0 += 32) {
        dense_stage_tri<T>(A, ld, r0, N, tri);
        if (r0 > 0) {
            T acc[4];
            // blockDim is 256: 8 warps x 4 rows = the 32 rows of the block
            dense_dot4<T>(A, ld, r0, wid, ln, 0, r0, N, y, acc);
#pragma unroll
            for (int i = 0; i < 4; ++i) {
#pragma unroll
                for (int off = 16; off; off >>= 1) acc[i] += __shfl_xor_sync(0xffffffffu, acc[i], off);
            }
            if (ln == 0) {
#pragma unroll
                for (int i = 0; i < 4; ++i)
                    if (r0 + wid + 8 * i < N) y[r0 + wid + 8 * i] -= acc[i];
            }
        }
        __syncthreads();
        if (wid == 0) {
            const int row = r0 + ln;
            T v = row < N ? y[row] : T(0);
            for (int j = 0; j < 32; ++j) {
                const T vj = __shfl_sync(0xffffffffu, v, j);
                if (ln > j && row < N && r0 + j < N) v = fma(-tri[ln][j], vj, v);
            }
            if (row < N) y[row] = v;
        }
        __syncthreads();
    }
    // U x = y
    const int last = ((N - 1) / 32) * 32;
    for (int r0 = last; r0 >= 0; r0 -= 32) {
        const int r1 = min(r0 + 32, N);
        dense_stage_tri<T>(A, ld, r0, N, tri);
        if (r1 < N) {
            T acc[4];
            dense_dot4<T>(A, ld, r0, wid, ln, r1, ld, N, y, acc);
#pragma unroll
            for (int i = 0; i < 4; ++i) {
#pragma unroll
                for (int off = 16; off; off >>= 1) acc[i] += __shfl_xor_sync(0xffffffffu, acc[i], off);
            }
            if (ln == 0) {
#pragma unroll
                for (int i = 0; i < 4; ++i)
                    if (r0 + wid + 8 * i < N) y[r0 + wid + 8 * i] -= acc[i];
            }
        }
        __syncthreads();
        if (wid == 0) {
            const int row = r0 + ln;
            T v = row < N ? y[row] : T(0);
            for (int j = 31; j >= 0; --j) {
                if (r0 + j < N) {
                    if (ln == j) v = v / tri[j][j];
                    const T vj = __shfl_sync(0xffffffffu, v, j);
                    if (ln < j && row < N) v = fma(-tri[ln][j], vj, v);
                }
            }
            if (row < N) y[row] = v;
        }
        __syncthreads();
    }
    double2* O = out + (size_t)g * P.nb * SW;
    for (int i = tid; i < P.n_tail; i += blockDim.x) {
        const int k = P.ns + i;
        stv(X + (size_t)k * SW + lane, Vec2<T>{y[2 * i], y[2 * i + 1]});
        double2* o = O + (size_t)k * SW + lane;
        if (accumulate) {
            const double2 old = *o;
            *o = make_double2(old.x + (double)y[2 * i], old.y + (double)y[2 * i + 1]);
        } else {
            *o = make_double2((double)y[2 * i], (double)y[2 * i + 1]);
        }
    }
}

// Dynamic shared memory of the dense solves: the tail vector, padded to whole blocks of 32.
__host__ __forceinline__ size_t dense_solve_smem(int n_tail, size_t esz) {
    return (size_t)((2 * n_tail + 31) / 32 * 32) * esz;
}

// The same two substitutions with a cluster of CTAs per scenario, for batches of few scenarios
// (one CTA streams the factor at 10 to 100 GB/s: every block of 32 waits for its dot products),
// and the transposed ones of the adjoint.  Right-looking by blocks of 32:
// block b belongs to CTA b % nc, which solves its triangle (one warp, reciprocals of the diagonal
// taken beforehand) and sends the 32 values to every CTA; after a cluster barrier each CTA takes
// them out of the rows of its own blocks, whose factor entries it has already loaded.  Every
// value's sum is formed block by block in four parts, whatever the cluster's size.
// TR: U^T w = y and L^T x = w, a thread per column instead of four threads per row.
// Bound by the chain of blocks, 2 to 2.4 us each (triangle, cluster barrier, update).  One FP64
// tail of order 506: 158 -> 79 us with 8 CTAs; 8 FP32 tails of order 1,424: 659 -> 176 us; the
// transposed solves of 256 FP64 tails, column by column before: 991 -> 242 us.
constexpr int DS_THREADS = 256;

template <typename T, int SW, bool TR>
__global__ void __launch_bounds__(DS_THREADS) k_dense_solve_cl(PlanDev P, BatchDev B, double2* out,
                                                               int accumulate) {
    namespace cg = cooperative_groups;
    const LevelCta cta;
    const int q = cta.g, nc = cta.nc, rank = cta.rank;
    if (q >= B.n_scen || !B.solving[q]) return;
    const int g = q / SW, lane = q % SW;
    if (accumulate && B.grefine && !B.grefine[g]) return;
    const int N = 2 * P.n_tail, ld = dense_ld(N), nblk = (N + 31) / 32;
    const T* A = reinterpret_cast<const T*>(B.Dt) + (size_t)q * N * ld;
    Vec2<T>* X = reinterpret_cast<Vec2<T>*>(B.X) + (size_t)g * P.nb * SW;
    extern __shared__ __align__(16) unsigned char smraw[];
    T* y = reinterpret_cast<T*>(smraw);  // [32 * nblk], kept up to date for this CTA's blocks
    __shared__ T tri[2][32][33], rdiag[2][32], sol[2][32], red[4][64];
    const int tid = threadIdx.x, wid = tid >> 5, ln = tid & 31;
    for (int i = tid; i < 16 * nblk; i += DS_THREADS) {
        const Vec2<T> v = i < P.n_tail ? ldv(X + (size_t)(P.ns + i) * SW + lane) : Vec2<T>{T(0), T(0)};
        y[2 * i] = v.x;
        y[2 * i + 1] = v.y;
    }
    // block b's triangle (transposed for TR; the identity past the matrix) and its diagonal, by
    // the threads from t0 on (all loads before the first store)
    auto stage = [&](int b, bool unit, T (*tri)[33], T* rdiag, int t0) {
        T a[5];
#pragma unroll
        for (int k = 0; k < 5; ++k) {
            const int e = tid - t0 + k * (DS_THREADS - t0), i = 32 * b + (e >> 5), j = 32 * b + (e & 31);
            a[k] = (e >> 5) == (e & 31) ? T(1) : T(0);
            if (e < 32 * 32 && i < N && j < N) a[k] = A[(size_t)i * ld + j];
        }
#pragma unroll
        for (int k = 0; k < 5; ++k) {
            const int e = tid - t0 + k * (DS_THREADS - t0), r = e >> 5, c = e & 31;
            if (e >= 32 * 32) break;
            if (TR) tri[c][r] = a[k];
            else tri[r][c] = a[k];
            if (r == c) rdiag[r] = unit ? T(1) : T(1) / a[k];
        }
    };
    static_assert(5 * (DS_THREADS - 32) >= 32 * 32);
    for (int sweep = 0; sweep < 2; ++sweep) {  // the lower triangle ascending, the upper descending
        const bool up = sweep == 1, unit = up == TR;
        const int top = rank + (nblk - 1 - rank) / nc * nc;  // this CTA's last block
        int buf = 0;  // this CTA's next triangle is in tri[buf]
        if (rank < nblk) stage(up ? top : rank, unit, tri[0], rdiag[0], 0);
        // a CTA of the cluster must have started before another one writes into its `sol`
        if (up) __syncthreads();
        else cta.sync();
        for (int step = 0; step < nblk; ++step) {
            const int b = up ? nblk - 1 - step : step;
            const bool own = b % nc == rank;
            // this CTA's remaining blocks: first, first + nc, ..., count of them
            const int first = up ? rank : b + 1 + ((rank - b - 1) % nc + nc) % nc;
            const int count = up ? (b - rank + nc - 1) / nc : (nblk - first + nc - 1) / nc;
            // the 8 entries of this thread's part of a row or column, NP of them ahead of the
            // barrier: nothing here depends on the solution (masked only where they are used, so
            // that no thread waits for them before)
            constexpr int NP = 4;
            T pre[NP][8];
            auto fetch = [&](int item, T (&a)[8]) {
                const int blk = first + nc * (item >> 5);
#pragma unroll
                for (int t = 0; t < 8; ++t) a[t] = T(0);
                if ((item >> 5) >= count) return;
                if (TR) {
                    const int col = 32 * blk + (item & 31), r = 32 * b + 8 * (tid >> 6);
#pragma unroll
                    for (int t = 0; t < 8; ++t)
                        if (r + t < N && col < N) a[t] = A[(size_t)(r + t) * ld + col];
                } else {
                    const int row = 32 * blk + (item & 31), c = 32 * b + 8 * (tid & 3);
                    if (row < N && c < ld) {
                        const V4<T> u = ld4(A + (size_t)row * ld + c), w = ld4(A + (size_t)row * ld + c + 4);
#pragma unroll
                        for (int t = 0; t < 4; ++t) {
                            a[t] = u.v[t];
                            a[t + 4] = w.v[t];
                        }
                    }
                }
            };
            const int item0 = TR ? tid & 63 : tid >> 2;
#pragma unroll
            for (int p = 0; p < NP; ++p) fetch(item0 + 64 * p, pre[p]);
            if (own && wid == 0) {
                T v = y[32 * b + ln], m[32];
                const T rd = rdiag[buf][ln];
                if (up) {
#pragma unroll
                    for (int j = 31; j >= 0; --j) m[j] = ln < j ? -tri[buf][ln][j] : T(0);
#pragma unroll
                    for (int j = 31; j >= 0; --j) {
                        if (ln == j) v *= rd;
                        v = fma(m[j], __shfl_sync(0xffffffffu, v, j), v);
                    }
                } else {
#pragma unroll
                    for (int j = 0; j < 32; ++j) m[j] = ln > j ? -tri[buf][ln][j] : T(0);
#pragma unroll
                    for (int j = 0; j < 32; ++j) {
                        if (ln == j) v *= rd;
                        v = fma(m[j], __shfl_sync(0xffffffffu, v, j), v);
                    }
                }
                y[32 * b + ln] = v;
                if (nc == 1) sol[step & 1][ln] = v;
                else
                    for (int r = 0; r < nc; ++r) *cg::this_cluster().map_shared_rank(&sol[step & 1][ln], r) = v;
            }
            if (own) {
                // meanwhile the other warps fetch this CTA's next triangle
                const int next = up ? b - nc : b + nc;
                if (wid > 0 && next >= 0 && next < nblk) stage(next, unit, tri[buf ^ 1], rdiag[buf ^ 1], 32);
                buf ^= 1;
            }
            cta.sync();
            const T* s = sol[step & 1] + 8 * (TR ? tid >> 6 : tid & 3);
            const int left = TR ? 8 : N - 32 * b - 8 * (tid & 3);  // columns of this part in the matrix
            auto take = [&](int item, T const (&a)[8]) {
                T acc = T(0);
#pragma unroll
                for (int t = 0; t < 8; ++t) acc = fma(t < left ? a[t] : T(0), s[t], acc);
                const int i = 32 * (first + nc * (item >> 5)) + (item & 31);
                if (TR) {
                    red[tid >> 6][tid & 63] = acc;
                    __syncthreads();
                    if (tid < 64 && (item >> 5) < count)
                        y[i] -= (red[0][tid] + red[1][tid]) + (red[2][tid] + red[3][tid]);
                    __syncthreads();
                } else {
                    acc += __shfl_xor_sync(0xffffffffu, acc, 1);
                    acc += __shfl_xor_sync(0xffffffffu, acc, 2);
                    if ((tid & 3) == 0 && (item >> 5) < count) y[i] -= acc;
                }
            };
#pragma unroll
            for (int p = 0; p < NP; ++p)
                if (64 * p < 32 * count) take(item0 + 64 * p, pre[p]);
            for (int base = 64 * NP; base < 32 * count; base += 64) {
                fetch(item0 + base, pre[0]);
                take(item0 + base, pre[0]);
            }
            __syncthreads();
        }
    }
    double2* O = out + (size_t)g * P.nb * SW;
    for (int i = tid; i < P.n_tail; i += DS_THREADS) {
        if ((i >> 4) % nc != rank) continue;
        const int k = P.ns + i;
        stv(X + (size_t)k * SW + lane, Vec2<T>{y[2 * i], y[2 * i + 1]});
        double2* o = O + (size_t)k * SW + lane;
        const double2 old = accumulate ? *o : make_double2(0.0, 0.0);
        *o = make_double2(old.x + (double)y[2 * i], old.y + (double)y[2 * i + 1]);
    }
}

// ---------------------------------------------------------------------------------------
// sparse triangular solves: L y = b (unit lower) over the sparse levels, then every tail
// node gathers its sparse contributions; U x = y over the sparse levels (descending) once
// the dense tail is solved.  x is written as FP64 (optionally added to `out`).
// ---------------------------------------------------------------------------------------
// Forward: L y = b, or with TR (the adjoint) U^T y = b, over the sparse levels, then every tail
// node gathers its sparse contributions.
template <typename T, int SW, bool TR>
__global__ void __launch_bounds__(1024) k_solve_fwd(PlanDev P, BatchDev B, const double2* __restrict__ rhs,
                            int refine_pass) {
    const LevelCta cta;
    const int g = cta.g;
    if (!B.gsolve[g] || (refine_pass && B.grefine && !B.grefine[g])) return;
    __shared__ Vec2<T> red[256];  // (blockDim / (32 / SW)) partial sums, <= 256 for SW <= 8
    __shared__ int lv_buf[LV_MAX + 1];
    const int* lv = level_bounds(P.level_ptr, P.n_levels, lv_buf);
    const Blk<T>* F = reinterpret_cast<const Blk<T>*>(B.F) + (size_t)g * P.n_slots * SW;
    const Blk<T>* E = F + (TR ? (size_t)P.nnz_l * SW : 0);  // U(k, j) sits nnz_l past L(j, k)
    Vec2<T>* X = reinterpret_cast<Vec2<T>*>(B.X) + (size_t)g * P.nb * SW;
    const double2* R = rhs + (size_t)g * P.nb * SW;
    const int lane = threadIdx.x % SW, n1 = blockDim.x / SW;  // slots of one CTA
    const int e1 = threadIdx.x / SW;
    const int e0 = cta.rank * n1 + e1, ne = cta.nc * n1;
    auto entry = [&](Vec2<T>& acc, int2 r) {
        const Blk<T> m = ldb(E + (size_t)r.x * SW + lane);
        const Vec2<T> x = ldv(X + (size_t)r.y * SW + lane);
        if (TR) msubtv(acc, m, x);
        else msubv(acc, m, x);
    };
    auto finish = [&](int k, Vec2<T> acc) {
        if (TR) acc = multv(ldb(F + (size_t)k * SW + lane), acc);
        stv(X + (size_t)k * SW + lane, acc);
    };
    if (B.lvl_ts) lvl_stamp(B, P.n_levels, 1, g, 0, cta.rank);
    __syncthreads();
    for (int h = 0; h < P.n_levels; ++h) {
        const int lb = lv[h], c = lv[h + 1] - lb;
        const int ls = split_log(c, n1), s = 1 << ls;
        if (s == 1) {
            // two nodes per worker at a time (nodes of one level are independent)
            for (int k = lb + e0; k < lb + c; k += 2 * ne) {
                const bool two = k + ne < lb + c;
                const int k2 = two ? k + ne : k;
                const double2 b = R[(size_t)k * SW + lane];
                const double2 b2 = R[(size_t)k2 * SW + lane];
                Vec2<T> acc = {(T)b.x, (T)b.y}, acc2 = {(T)b2.x, (T)b2.y};
                const int qa = P.rptr[k], qe = P.rptr[k + 1];
                const int qa2 = two ? P.rptr[k2] : 0, qe2 = two ? P.rptr[k2 + 1] : 0;
                const int nb = min(qe - qa, qe2 - qa2);
#pragma unroll 2
                for (int i = 0; i < nb; ++i) {
                    const int2 r = P.rlist[qa + i], r2 = P.rlist[qa2 + i];
                    entry(acc, r);
                    entry(acc2, r2);
                }
#pragma unroll 4
                for (int q = qa + nb; q < qe; ++q) entry(acc, P.rlist[q]);
#pragma unroll 4
                for (int q = qa2 + nb; q < qe2; ++q) entry(acc2, P.rlist[q]);
                finish(k, acc);
                if (two) finish(k2, acc2);
            }
        } else if (cta.rank == 0 && (threadIdx.x & ~31) / SW >= c << ls) {
            if (s > 32 / SW) __syncthreads();  // a warp without rows: split_reduce's barrier
        } else if (cta.rank == 0) {
            const int j = e1 >> ls, sub = e1 & (s - 1);
            const int k = lb + min(j, c - 1);
            Vec2<T> acc = {T(0), T(0)};
            if (j < c) {
                int q = P.rptr[k] + sub;
                const int qe = P.rptr[k + 1];
                for (; q + (ROW_BATCH<T> - 1) * s < qe; q += ROW_BATCH<T> * s) {
                    int2 r[ROW_BATCH<T>];
                    Blk<T> m[ROW_BATCH<T>];
                    Vec2<T> x[ROW_BATCH<T>];
#pragma unroll
                    for (int u = 0; u < ROW_BATCH<T>; ++u) r[u] = P.rlist[q + u * s];
#pragma unroll
                    for (int u = 0; u < ROW_BATCH<T>; ++u) {
                        m[u] = ldb(E + (size_t)r[u].x * SW + lane);
                        x[u] = ldv(X + (size_t)r[u].y * SW + lane);
                    }
#pragma unroll
                    for (int u = 0; u < ROW_BATCH<T>; ++u) {
                        if (TR) msubtv(acc, m[u], x[u]);
                        else msubv(acc, m[u], x[u]);
                    }
                }
                for (; q < qe; q += s) entry(acc, P.rlist[q]);
            }
            acc = split_reduce<T, SW>(acc, s, sub, j, lane, red);
            if (j < c && sub == 0) {
                const double2 b = R[(size_t)k * SW + lane];
                finish(k, Vec2<T>{(T)b.x + acc.x, (T)b.y + acc.y});
            }
        }
        // a level split over sub-slots fits one CTA: between two of them the others run ahead
        if (s > 1 && h + 1 < P.n_levels && split_log(lv[h + 2] - lv[h + 1], n1) > 0) cta.sync_solo();
        else cta.sync();
        if (B.lvl_ts) lvl_stamp(B, P.n_levels, 1, g, h + 1, cta.rank);
    }
    {
        // tail rows gather long sparse rows: 4 sub-slots per row (a shuffle reduction within
        // the warp, 4 <= 32 / SW), rounds uniform across the block
        constexpr int TS = 4;
        const int sub = e0 % TS, per = ne / TS;
        for (int base = P.ns; base < P.nb; base += per) {
            const int k = base + e0 / TS;
            Vec2<T> acc = {T(0), T(0)};
            if (k < P.nb) {
#pragma unroll 4
                for (int q = P.rptr[k] + sub; q < P.rptr[k + 1]; q += TS) entry(acc, P.rlist[q]);
            }
            acc = split_reduce<T, SW>(acc, TS, sub, 0, lane, red);
            if (k < P.nb && sub == 0) {
                const double2 b = R[(size_t)k * SW + lane];
                stv(X + (size_t)k * SW + lane, Vec2<T>{(T)b.x + acc.x, (T)b.y + acc.y});
            }
        }
    }
    if (B.lvl_ts) {
        __syncthreads();
        lvl_stamp(B, P.n_levels, 1, g, P.n_levels + 1, cta.rank);
    }
}

// Backward: U x = y, or with TR L^T x = y, over the sparse levels (descending) once the dense tail
// is solved; x written as FP64 (optionally added to `out`).
template <typename T, int SW, bool TR>
__global__ void __launch_bounds__(1024) k_solve_bwd(PlanDev P, BatchDev B, double2* out, int accumulate) {
    const LevelCta cta;
    const int g = cta.g;
    if (!B.gsolve[g] || (accumulate && B.grefine && !B.grefine[g])) return;
    __shared__ Vec2<T> red[256];
    __shared__ int lv_buf[LV_MAX + 1];
    const int* lv = level_bounds(P.level_ptr, P.n_levels, lv_buf);
    const Blk<T>* F = reinterpret_cast<const Blk<T>*>(B.F) + (size_t)g * P.n_slots * SW;
    const Blk<T>* E = F + ((size_t)P.nb + (TR ? 0 : P.nnz_l)) * SW;
    Vec2<T>* X = reinterpret_cast<Vec2<T>*>(B.X) + (size_t)g * P.nb * SW;
    double2* O = out + (size_t)g * P.nb * SW;
    const int lane = threadIdx.x % SW, n1 = blockDim.x / SW;
    const int e1 = threadIdx.x / SW;
    const int e0 = cta.rank * n1 + e1, ne = cta.nc * n1;
    auto entry = [&](Vec2<T>& acc, int p) {
        const Blk<T> m = ldb(E + (size_t)p * SW + lane);
        const Vec2<T> x = ldv(X + (size_t)P.lidx[p] * SW + lane);
        if (TR) msubtv(acc, m, x);
        else msubv(acc, m, x);
    };
    auto finish = [&](int k, Vec2<T> acc) {
        const Vec2<T> x = TR ? acc : mulv(ldb(F + (size_t)k * SW + lane), acc);
        stv(X + (size_t)k * SW + lane, x);
        double2* o = O + (size_t)k * SW + lane;
        if (accumulate) {
            const double2 old = *o;
            *o = make_double2(old.x + (double)x.x, old.y + (double)x.y);
        } else {
            *o = make_double2((double)x.x, (double)x.y);
        }
    };
    if (B.lvl_ts) lvl_stamp(B, P.n_levels, 2, g, 0, cta.rank);
    __syncthreads();
    for (int h = P.n_levels - 1; h >= 0; --h) {
        const int lb = lv[h], c = lv[h + 1] - lb;
        const int ls = split_log(c, n1), s = 1 << ls;
        if (s == 1) {
            // two nodes per worker at a time (nodes of one level are independent)
            for (int k = lb + e0; k < lb + c; k += 2 * ne) {
                const bool two = k + ne < lb + c;
                const int k2 = two ? k + ne : k;
                Vec2<T> acc = ldv(X + (size_t)k * SW + lane);
                Vec2<T> acc2 = ldv(X + (size_t)k2 * SW + lane);
                const int pa = P.lptr[k], pe = P.lptr[k + 1];
                const int pa2 = two ? P.lptr[k2] : 0, pe2 = two ? P.lptr[k2 + 1] : 0;
                const int nb = min(pe - pa, pe2 - pa2);
#pragma unroll 2
                for (int i = 0; i < nb; ++i) {
                    entry(acc, pa + i);
                    entry(acc2, pa2 + i);
                }
#pragma unroll 4
                for (int p = pa + nb; p < pe; ++p) entry(acc, p);
#pragma unroll 4
                for (int p = pa2 + nb; p < pe2; ++p) entry(acc2, p);
                finish(k, acc);
                if (two) finish(k2, acc2);
            }
        } else if (cta.rank == 0 && (threadIdx.x & ~31) / SW >= c << ls) {
            if (s > 32 / SW) __syncthreads();  // a warp without rows: split_reduce's barrier
        } else if (cta.rank == 0) {
            const int j = e1 >> ls, sub = e1 & (s - 1);
            const int k = lb + min(j, c - 1);
            Vec2<T> acc = {T(0), T(0)};
            if (j < c) {
                int p = P.lptr[k] + sub;
                const int pe = P.lptr[k + 1];
                for (; p + (ROW_BATCH<T> - 1) * s < pe; p += ROW_BATCH<T> * s) {
                    int i[ROW_BATCH<T>];
                    Blk<T> m[ROW_BATCH<T>];
                    Vec2<T> x[ROW_BATCH<T>];
#pragma unroll
                    for (int u = 0; u < ROW_BATCH<T>; ++u) i[u] = P.lidx[p + u * s];
#pragma unroll
                    for (int u = 0; u < ROW_BATCH<T>; ++u) {
                        m[u] = ldb(E + (size_t)(p + u * s) * SW + lane);
                        x[u] = ldv(X + (size_t)i[u] * SW + lane);
                    }
#pragma unroll
                    for (int u = 0; u < ROW_BATCH<T>; ++u) {
                        if (TR) msubtv(acc, m[u], x[u]);
                        else msubv(acc, m[u], x[u]);
                    }
                }
                for (; p < pe; p += s) entry(acc, p);
            }
            acc = split_reduce<T, SW>(acc, s, sub, j, lane, red);
            if (j < c && sub == 0) {
                const Vec2<T> xk = ldv(X + (size_t)k * SW + lane);
                finish(k, Vec2<T>{xk.x + acc.x, xk.y + acc.y});
            }
        }
        if (s > 1 && h > 0 && split_log(lv[h] - lv[h - 1], n1) > 0) cta.sync_solo();
        else cta.sync();
        if (B.lvl_ts) lvl_stamp(B, P.n_levels, 2, g, P.n_levels - h, cta.rank);
    }
    if (B.lvl_ts) lvl_stamp(B, P.n_levels, 2, g, P.n_levels + 1, cta.rank);
}

// refinement residual: res = rhs - J dx with the FP64 Jacobian blocks
template <int SW>
__global__ void __launch_bounds__(256, 8) k_residual(PlanDev P, BatchDev B) {
    const int g = blockIdx.y;
    if (!B.gsolve[g] || (B.grefine && !B.grefine[g])) return;
    const int tid = blockIdx.x * blockDim.x + threadIdx.x;
    const int k = tid / SW, lane = tid % SW;
    if (k >= P.nb) return;
    const size_t base = (size_t)g * P.nb * SW;
    const double2 b = B.rhs[base + (size_t)k * SW + lane];
    Vec2<double> acc = {b.x, b.y};
    const Blk<double>* A = reinterpret_cast<const Blk<double>*>(B.A64) + (size_t)g * P.n_a * SW;
#pragma unroll 4
    for (int e = P.arow_ptr[k]; e < P.arow_ptr[k + 1]; ++e) {
        const int2 ac = P.arow[e];
        const double2 x = B.dx[base + (size_t)ac.y * SW + lane];
        msubv(acc, ldb(A + (size_t)ac.x * SW + lane), Vec2<double>{x.x, x.y});
    }
    B.res[base + (size_t)k * SW + lane] = make_double2(acc.x, acc.y);
}

// ---------------------------------------------------------------------------------------
// voltage update
// ---------------------------------------------------------------------------------------
// One bus's voltage after the Newton correction d = (dtheta, d|V|), by step policy.
__device__ __forceinline__ double2 newton_step(double2 v, double2 d, bool pq, int policy) {
    if (policy != 1) {
        // reference policy (cpu_newton_raphson.cpp:457-503): damping 0.9 and the clamps;
        // clamped policy: the same clamps and order with the full step
        const double damp = policy == 0 ? 0.9 : 1.0;
        const double vm = hypot(v.x, v.y);
        double a = damp * d.x;
        if (fabs(a) > 0.15) a = 0.15 * (a > 0 ? 1.0 : -1.0);
        double sn, cs;
        sincos(atan2(v.y, v.x) + a, &sn, &cs);
        v = make_double2(vm * cs, vm * sn);
        if (pq) {
            const double vm0 = hypot(v.x, v.y);
            double c = damp * d.y;
            if (fabs(c) > 0.08) c = 0.08 * (c > 0 ? 1.0 : -1.0);
            double vmn = vm0 + c;
            vmn = (vmn < 0.5) ? 0.5 : vmn;
            vmn = (1.5 < vmn) ? 1.5 : vmn;
            sincos(atan2(v.y, v.x), &sn, &cs);
            v = make_double2(vmn * cs, vmn * sn);
        }
    } else {
        // Newton step in polar form, |V| e^{j theta} -> (|V| + d|V|) e^{j (theta + dtheta)}:
        // V rotated by dtheta and scaled by (|V| + d|V|) / |V|, one sincos of the (small)
        // correction instead of atan2 and a sincos of the full angle
        const double vm = hypot(v.x, v.y);
        double sn, cs;
        sincos(d.x, &sn, &cs);
        if (vm > 0.0) {
            const double sc = pq ? (vm + d.y) / vm : 1.0;
            v = make_double2(sc * fma(v.x, cs, -v.y * sn), sc * fma(v.x, sn, v.y * cs));
        } else {
            const double m = pq ? d.y : 0.0;  // from V = 0 the angle is the correction's
            v = make_double2(m * cs, m * sn);
        }
    }
    return v;
}

template <int SW>
__global__ void __launch_bounds__(256, 8) k_update(PlanDev P, BatchDev B) {
    const int g = blockIdx.y;
    if (!B.gsolve[g]) return;
    const int n = P.n_bus;
    const int tid = blockIdx.x * blockDim.x + threadIdx.x;
    const int i = tid / SW, lane = tid % SW;
    if (i >= n) return;
    const int q = g * SW + lane;
    // the loads that do not depend on the flags below go first (padding lanes have storage),
    // so that one memory latency covers them and the flags
    const int node = P.node_of_bus[i];
    const size_t o = ((size_t)g * n + i) * SW + lane;
    double2 v = B.V[o];
    const bool pq = P.bus_type[i] == BUS_PQ;
    const double2 d = node >= 0 ? B.dx[((size_t)g * P.nb + node) * SW + lane] : make_double2(0.0, 0.0);
    if (q >= B.n_scen) return;  // padding lanes are never updated
    {
        if (B.singular[q]) {
            // the reference keeps V unchanged when factorize() fails and runs to max_iter
            if (i == 0 && B.solving[q]) {
                B.state[q] = 1;
                B.status[q] = SC_SINGULAR;
                B.iters[q] = B.ctrl[1];
                B.solving[q] = 0;
            }
            return;
        }
        if (!B.solving[q]) return;
    }
    if (node < 0) return;
    B.V[o] = newton_step(v, d, pq, B.ctrl[3]);
}

// ---------------------------------------------------------------------------------------
// results out (scenario-major) and reference-order views of the stage vectors
// ---------------------------------------------------------------------------------------
template <int SW>
__global__ void k_store(PlanDev P, BatchDev B, double2* v_out, int* it_out, int* st_out,
                        double* fm_out) {
    const int n = P.n_bus;
    const long tid = (long)blockIdx.x * blockDim.x + threadIdx.x;
    const long total = (long)B.n_scen * n;
    if (tid < total) {
        const int s = (int)(tid / n), i = (int)(tid % n);
        const int g = s / SW, lane = s % SW;
        if (v_out) v_out[tid] = B.V[((size_t)g * n + i) * SW + lane];
        if (i == 0) {
            if (it_out) it_out[s] = B.iters[s];
            if (st_out) st_out[s] = B.status[s];
            if (fm_out) fm_out[s] = B.final_mis[s];
        }
    }
}

// current state per scenario in bus order: V, I = Y V and S = V conj(I), per unit
// (IterationState of powerflow_interface.h:28-35, filled as cpu_newton_raphson.cpp:125-149)
template <int SW>
__global__ void k_state(PlanDev P, BatchDev B, double2* v_out, double2* i_out,
                        double2* s_out) {
    const int n = P.n_bus;
    const long tid = (long)blockIdx.x * blockDim.x + threadIdx.x;
    if (tid >= (long)B.n_scen * n) return;
    const int s = (int)(tid / n), i = (int)(tid % n);
    const int g = s / SW, lane = s % SW;
    const double2* Vg = B.V + (size_t)g * n * SW;
    const double2* Yg = B.y_shared ? B.Y : B.Y + (size_t)g * P.nnz_y * SW;
    const size_t ys = B.y_shared ? 1 : SW;
    const size_t yl = B.y_shared ? 0 : lane;
    double ir = 0.0, ii = 0.0;
    for (int p = P.y_row_ptr[i]; p < P.y_row_ptr[i + 1]; ++p) {
        const double2 y = Yg[(size_t)p * ys + yl];
        const double2 v = Vg[(size_t)P.y_col[p] * SW + lane];
        ir = fma(y.x, v.x, ir);
        ir = fma(-y.y, v.y, ir);
        ii = fma(y.x, v.y, ii);
        ii = fma(y.y, v.x, ii);
    }
    const double2 vi = Vg[(size_t)i * SW + lane];
    if (v_out) v_out[tid] = vi;
    if (i_out) i_out[tid] = make_double2(ir, ii);
    if (s_out) s_out[tid] = make_double2(fma(vi.x, ir, vi.y * ii), fma(vi.y, ir, -vi.x * ii));
}

// node vector [G][nb][SW] -> reference order [n_scen][n_vars]; map[node*2+c] gives the
// reference index (or -1); sign multiplies the value
template <int SW>
__global__ void k_node_to_ref(const double2* __restrict__ src, int nb, int n_scen, int n_vars,
                              const int* __restrict__ map, double sign, double* dst) {
    const long tid = (long)blockIdx.x * blockDim.x + threadIdx.x;
    if (tid >= (long)n_scen * nb) return;
    const int s = (int)(tid / nb), k = (int)(tid % nb);
    const int g = s / SW, lane = s % SW;
    const double2 v = src[((size_t)g * nb + k) * SW + lane];
    const int a = map[2 * k], b = map[2 * k + 1];
    if (a >= 0) dst[(size_t)s * n_vars + a] = sign * v.x;
    if (b >= 0) dst[(size_t)s * n_vars + b] = sign * v.y;
}

// ---------------------------------------------------------------------------------------
// adjoint: J^T lambda = dL/dx with the factors of J = L U
//   U^T z = g   : sparse forward sweep with U slots transposed (D^-T on sparse nodes), the
//                 tail gathers its sparse contributions, then a dense U_tt^T solve
//   L^T lam = z : dense L_tt^T solve, then a sparse backward sweep with L slots transposed
// ---------------------------------------------------------------------------------------
template <int SW>
__global__ void k_adj_prep(BatchDev B) {
    const int q = blockIdx.x * blockDim.x + threadIdx.x;
    if (q >= B.n_groups * SW) return;
    B.solving[q] = q < B.n_scen ? 1 : 0;
    B.singular[q] = 0;
    if (q % SW == 0) {
        B.gsolve[q / SW] = 1;
        B.giter[q / SW] = 1;
        // refactorised and refined, whatever the last solve's thresholds left here
        if (B.grefine) B.grefine[q / SW] = 1;
        if (B.gfactor) B.gfactor[q / SW] = 1;
    }
}

// g per node: (dL/dtheta, dL/d|V| for PQ buses); inputs scenario-major [n_scen][n_bus]
template <int SW>
__global__ void k_adj_rhs(PlanDev P, BatchDev B, const double* __restrict__ dvm,
                          const double* __restrict__ dva) {
    const int g = blockIdx.y;
    const int tid = blockIdx.x * blockDim.x + threadIdx.x;
    const int i = tid / SW, lane = tid % SW;
    if (i >= P.n_bus) return;
    const int node = P.node_of_bus[i];
    if (node < 0) return;
    const int q = g * SW + lane;
    const int src = q < B.n_scen ? q : g * SW;
    const double gt = dva[(size_t)src * P.n_bus + i];
    const double gv = P.bus_type[i] == BUS_PQ ? dvm[(size_t)src * P.n_bus + i] : 0.0;
    B.rhs[((size_t)g * P.nb + node) * SW + lane] = make_double2(gt, gv);
}

// res = g - J^T lam with the FP64 Jacobian blocks, by block column
template <int SW>
__global__ void __launch_bounds__(256) k_residual_t(PlanDev P, BatchDev B) {
    const int g = blockIdx.y;
    if (!B.gsolve[g]) return;
    const int tid = blockIdx.x * blockDim.x + threadIdx.x;
    const int c = tid / SW, lane = tid % SW;
    if (c >= P.nb) return;
    const size_t base = (size_t)g * P.nb * SW;
    const double2 b = B.rhs[base + (size_t)c * SW + lane];
    Vec2<double> acc = {b.x, b.y};
    const Blk<double>* A = reinterpret_cast<const Blk<double>*>(B.A64) + (size_t)g * P.n_a * SW;
#pragma unroll 4
    for (int e = P.acol_ptr[c]; e < P.acol_ptr[c + 1]; ++e) {
        const int2 ar = P.acol[e];
        const double2 x = B.dx[base + (size_t)ar.y * SW + lane];
        msubtv(acc, ldb(A + (size_t)ar.x * SW + lane), Vec2<double>{x.x, x.y});
    }
    B.res[base + (size_t)c * SW + lane] = make_double2(acc.x, acc.y);
}

// dL/dP_spec = lambda_P, dL/dQ_spec = lambda_Q (PQ buses), per bus, scenario-major
template <int SW>
__global__ void k_adj_out(PlanDev P, BatchDev B, double* dp, double* dq) {
    const long tid = (long)blockIdx.x * blockDim.x + threadIdx.x;
    if (tid >= (long)B.n_scen * P.n_bus) return;
    const int s = (int)(tid / P.n_bus), i = (int)(tid % P.n_bus);
    const int g = s / SW, lane = s % SW;
    const int node = P.node_of_bus[i];
    double a = 0.0, b = 0.0;
    if (node >= 0) {
        const double2 l = B.dx[((size_t)g * P.nb + node) * SW + lane];
        a = l.x;
        b = P.bus_type[i] == BUS_PQ ? l.y : 0.0;
    }
    if (dp) dp[tid] = a;
    if (dq) dq[tid] = b;
}

// dL/dr, dL/dx per branch (per unit): -lambda^T dF/dp through the branch's pi stamps with
// y = 1/(r + jx), dy/dr = -y^2, dy/dx = -j y^2; brp = (r, x, g, b, k, theta) per unit
template <int SW>
__global__ void k_adj_branch(PlanDev P, BatchDev B, int m, const int* __restrict__ from,
                             const int* __restrict__ to, const double* __restrict__ brp,
                             double* dr, double* dxo) {
    const long tid = (long)blockIdx.x * blockDim.x + threadIdx.x;
    if (tid >= (long)B.n_scen * m) return;
    const int s = (int)(tid / m), b = (int)(tid % m);
    const int g = s / SW, lane = s % SW;
    const int f = from[b], t = to[b];
    double gr = 0.0, gx = 0.0;
    const double* q = brp + (size_t)b * 6;
    const double r = q[0], x = q[1], k = q[4], th = q[5];
    const double z2 = r * r + x * x;
    if (f >= 0 && t >= 0 && z2 > 0.0) {
        const double yr = r / z2, yi = -x / z2;
        const double y2r = yr * yr - yi * yi, y2i = 2.0 * yr * yi;  // y^2
        double sn, cs;
        sincos(th, &sn, &cs);
        const double tr = k * cs, ti = k * sn, k2 = k * k;
        const double2 vf = B.V[((size_t)g * P.n_bus + f) * SW + lane];
        const double2 vt = B.V[((size_t)g * P.n_bus + t) * SW + lane];
        const int nf = P.node_of_bus[f], nt = P.node_of_bus[t];
        const double2 lf = nf >= 0 ? B.dx[((size_t)g * P.nb + nf) * SW + lane] : make_double2(0, 0);
        const double2 lt = nt >= 0 ? B.dx[((size_t)g * P.nb + nt) * SW + lane] : make_double2(0, 0);
        const double lqf = P.bus_type[f] == BUS_PQ ? lf.y : 0.0;
        const double lqt = P.bus_type[t] == BUS_PQ ? lt.y : 0.0;
        for (int which = 0; which < 2; ++which) {
            // dy: -y^2 (r) or -j y^2 (x)
            const double dyr = which == 0 ? -y2r : y2i, dyi = which == 0 ? -y2i : -y2r;
            // dYff = dy/k^2, dYtt = dy, dYft = -dy*t/k^2, dYtf = -dy*conj(t)/k^2
            const double ffr = dyr / k2, ffi = dyi / k2;
            const double ftr = -(dyr * tr - dyi * ti) / k2, fti = -(dyr * ti + dyi * tr) / k2;
            const double tfr = -(dyr * tr + dyi * ti) / k2, tfi = -(dyi * tr - dyr * ti) / k2;
            // dI_f = dYff vf + dYft vt ; dI_t = dYtf vf + dYtt vt
            const double ifr = ffr * vf.x - ffi * vf.y + ftr * vt.x - fti * vt.y;
            const double ifi = ffr * vf.y + ffi * vf.x + ftr * vt.y + fti * vt.x;
            const double itr = tfr * vf.x - tfi * vf.y + dyr * vt.x - dyi * vt.y;
            const double iti = tfr * vf.y + tfi * vf.x + dyr * vt.y + dyi * vt.x;
            // dS = V conj(dI)
            const double sfr = vf.x * ifr + vf.y * ifi, sfi = vf.y * ifr - vf.x * ifi;
            const double str = vt.x * itr + vt.y * iti, sti = vt.y * itr - vt.x * iti;
            const double adj = lf.x * sfr + lqf * sfi + lt.x * str + lqt * sti;
            if (which == 0)
                gr = -adj;
            else
                gx = -adj;
        }
    }
    dr[tid] = gr;
    dxo[tid] = gx;
}

}  // namespace gapk
