// The whole Newton loop of a small grid in one kernel.
//
// A grid whose factor fits in shared memory needs no launches between its phases: one CTA takes
// CL scenarios of a lane group through every iteration -- mismatch, convergence test, Jacobian,
// block LU, dense tail, triangular solves, refinement, voltage update -- with the factor blocks,
// the solve vectors, the voltages and the dense tail in shared memory and a block barrier where
// the separate kernels have a launch.  The arithmetic is theirs, block by block.
//
// What bounds it is the latency of the level schedule: a 200-bus feeder has 25 levels, each a
// dependent step of the factorisation and of both triangular solves.  So a step is kept to a
// shared-memory gather, the block arithmetic and a barrier, in as few instructions as possible:
// the schedule is stored level by level as equally long lists of packed 16-bit index pairs (short
// rows padded with a zero block), so that a thread's next index is one load at a known address,
// taken (from L1) before this level's barrier; the right-hand side is already in the solve
// vector; and long rows are split over 2 or 4 threads (by the plan alone, so that results do not
// depend on the launch shape).  A step still takes 0.4 us, mostly dependent instructions.
// 200-bus feeder, FP64, 10 iterations: 1,340 -> 450 us for one scenario, 1,590 -> 745 us for
// 1024; a 500-bus grid, one scenario: 754 -> 358 us.
//
// Lanes per CTA: lanes are independent unless per-group refinement or reuse thresholds make a
// group's lanes decide together; then the group's CTAs form a cluster and exchange their flags.
// The host picks the CL and the CTA size (small_choice).
#pragma once

#include <cooperative_groups.h>

namespace gapk {

// Shared memory of one CTA: byte offsets of the factor blocks (and a zero block), voltages, solve
// vector (and a zero entry), FP64 correction (FP32 factors only), dense tail and level records;
// total size.
struct SmallLayout {
    size_t f, v, x, dx, d, lv, total;
};
__host__ __device__ __forceinline__ int small_ld(int N) { return N | 1; }  // odd: no conflicts
__host__ __device__ inline SmallLayout small_layout(int n_bus, int nb, int n_slots, int n_tail,
                                                    int n_levels, int cl, size_t esz) {
    SmallLayout s;
    const size_t N = 2 * (size_t)n_tail;
    auto up = [](size_t b) { return (b + 15) & ~size_t(15); };
    s.f = 0;
    s.v = s.f + ((size_t)n_slots + 1) * cl * 4 * esz;
    s.x = s.v + (size_t)n_bus * cl * 16;
    s.dx = s.x + up(((size_t)nb + 1) * cl * 2 * esz);
    s.d = s.dx + (esz == 4 ? (size_t)nb * cl * 16 : 0);
    s.lv = s.d + up((N * small_ld((int)N) + N) * cl * esz);
    s.total = s.lv + ((size_t)n_levels + 1) * 48;
    return s;
}

// Largest tail order: a warp keeps the tail vector in registers, SMALL_YR values per thread.
constexpr int SMALL_YR = 4, SMALL_MAX_TAIL = 32 * SMALL_YR / 2;
constexpr int SMALL_THREADS = 256;
constexpr size_t SMALL_SMEM_MAX = 232448 - 2048;  // opt-in shared memory per block, less static
constexpr long SMALL_SM_SMEM = 233472;            // shared memory of an SM

// The packed schedule (built by the plan): 32-bit words of two 16-bit indices, single ones for
// targets and scalings (P.words) and two entries together for pairs and rows (P.ell), so that a
// thread keeps two entries in flight.  Level record h, three int4:
//   (first node, nodes, first target word, targets)
//   (first pair entry, entries per slot | split << 16, first scale word, scale words)
//   (first forward entry, entries per slot | split << 16, the same two of the backward sweep)
// A target or row takes 1 << split neighbouring slots; entry m of slot e sits at
// first + m * (rows << split) + e.  The last record is the tail's forward rows.
constexpr unsigned SMALL_DIAG = 1u << 16, SMALL_VALUE = 1u << 17;  // of a target word

template <typename T, int CL>
struct SmallCta {
    PlanDev const& P;
    BatchDev const& B;
    int of_v, of_x, of_dx, of_d, of_lv;  // byte offsets in shared memory
    int lane, e0, ne;
    size_t gl;      // lane of the group's storage
    int g, SW;

    static __device__ __forceinline__ unsigned char* sm() {
        extern __shared__ __align__(16) unsigned char smraw[];
        return smraw;
    }
    // [n_slots + 1][CL], [nb + 1][CL] (the right-hand side, then the solution), [n_bus][CL],
    // [nb][CL] FP64 correction (FP32 factors; FP64 ones leave it in x)
    __device__ __forceinline__ Blk<T>* f(int slot) const {
        return reinterpret_cast<Blk<T>*>(sm()) + slot * CL + lane;
    }
    __device__ __forceinline__ Vec2<T>* x(int k) const {
        return reinterpret_cast<Vec2<T>*>(sm() + of_x) + k * CL + lane;
    }
    __device__ __forceinline__ double2& v(int i) const {
        return reinterpret_cast<double2*>(sm() + of_v)[i * CL + lane];
    }
    __device__ __forceinline__ double2& dx(int k) const {
        return reinterpret_cast<double2*>(sm() + of_dx)[k * CL + lane];
    }
    // dense tail [N][ld][CL] (L unscaled until the factorisation ends), then 1 / pivot [N][CL]
    __device__ __forceinline__ T* d(int i) const { return reinterpret_cast<T*>(sm() + of_d) + i * CL; }
    __device__ __forceinline__ int4 rec(int h, int w) const {
        return reinterpret_cast<const int4*>(sm() + of_lv)[3 * h + w];
    }

    __device__ __forceinline__ size_t at(int items, int i) const {
        return ((size_t)g * items + i) * SW + gl;
    }
    __device__ __forceinline__ double2 y_value(int p) const {
        return B.y_shared ? B.Y[p] : B.Y[at(P.nnz_y, p)];
    }

    // S = V conj(Y V) and -Delta of every bus; returns this thread's max |Delta|
    __device__ __forceinline__ double mismatch() const {
        double m = 0.0;
        for (int i = e0; i < P.n_bus; i += ne) {
            double ir = 0.0, ii = 0.0;
            const int p1 = P.y_row_ptr[i + 1], t = P.bus_type[i], node = P.node_of_bus[i];
            const double2 sp = B.Sspec[at(P.n_bus, i)], vi = v(i);
#pragma unroll 4
            for (int p = P.y_row_ptr[i]; p < p1; ++p) {
                const double2 y = y_value(p), u = v(P.y_col[p]);
                ir = fma(y.x, u.x, ir);
                ir = fma(-y.y, u.y, ir);
                ii = fma(y.x, u.y, ii);
                ii = fma(y.y, u.x, ii);
            }
            const double2 s = make_double2(fma(vi.x, ir, vi.y * ii), fma(vi.y, ir, -vi.x * ii));
            B.Scalc[at(P.n_bus, i)] = s;
            if (t != BUS_SLACK) {
                const double dp = s.x - sp.x, dq = (t == BUS_PQ) ? s.y - sp.y : 0.0;
                B.rhs[at(P.nb, node)] = make_double2(-dp, -dq);
                stv(x(node), Vec2<T>{(T)-dp, (T)-dq});
                m = nmax(m, nmax(fabs(dp), fabs(dq)));
            }
        }
        return m;
    }

    __device__ __forceinline__ void jacobian(bool to_f, bool to_a64) const {
        for (int a = e0; a < P.n_a; a += ne) {
            const int4 rec = P.a_rec[a];
            const Blk<double> J = jac_block(
                P, rec, [&](int i) { return v(i); },
                [&](int i) { return B.Scalc[at(P.n_bus, i)]; }, [&](int p) { return y_value(p); });
            if (to_f) stb(f(rec.x), Blk<T>{(T)J.a, (T)J.b, (T)J.c, (T)J.d});
            if (to_a64) stb(reinterpret_cast<Blk<double>*>(B.A64) + at(P.n_a, a), J);
        }
    }

    // sum over the 1 << ls (1, 2 or 4) sub-slots of a row, neighbouring slots of one warp; the
    // values' shuffles overlap
    template <int NV>
    __device__ __forceinline__ void row_sum(T (&v)[NV], int ls) const {
        if (ls > 0) {
#pragma unroll
            for (int i = 0; i < NV; ++i) v[i] += __shfl_xor_sync(0xffffffffu, v[i], CL);
        }
        if (ls > 1) {
#pragma unroll
            for (int i = 0; i < NV; ++i) v[i] += __shfl_xor_sync(0xffffffffu, v[i], 2 * CL);
        }
    }

    // block LU level by level, then the tail's Schur complement and its dense LU; false when a
    // pivot of this thread's fails
    __device__ __forceinline__ bool factor() const {
        bool ok_all = true;
        const int wl = e0 & (32 / CL - 1);  // slot within the warp
        unsigned tw = 0, sw = 0;
        uint2 pw = make_uint2(0, 0);
        auto fetch = [&](int h) {  // this thread's first target, pair and scale of level h
            const int4 ra = rec(h, 0), rb = rec(h, 1);
            const int ls = rb.y >> 16;
            if (e0 < ra.w << ls) {
                tw = P.words[ra.z + (e0 >> ls)];
                if (rb.y & 0xffff) pw = P.ell[rb.x + e0];
            }
            if (e0 < rb.w) sw = P.words[rb.z + e0];
        };
        if (P.n_levels > 0) fetch(0);
        for (int h = 0; h < P.n_levels; ++h) {
            const int4 ra = rec(h, 0), rb = rec(h, 1);
            const int ls = rb.y >> 16, M = rb.y & 0xffff, W = ra.w << ls;
            unsigned t = tw, s = sw;
            uint2 p = pw;
            if (h + 1 < P.n_levels) fetch(h + 1);
            for (int e = e0; e - wl < W; e += ne) {
                const bool on = e < W, own = on && (e & ((1 << ls) - 1)) == 0;
                if (e != e0 && on) {
                    t = P.words[ra.z + (e >> ls)];
                    if (M) p = P.ell[rb.x + e];
                }
                Blk<T> acc = own && (t & SMALL_VALUE) ? ldb(f(t & 0xffff)) : Blk<T>{0, 0, 0, 0};
                if (on) {
                    const uint2* next = P.ell + rb.x + e;
                    for (int m = 1; m <= M; ++m) {
                        const uint2 c = p;
                        if (m < M) p = *(next += W);
                        Blk<T> odd = {0, 0, 0, 0};
                        msub(acc, ldb(f(c.x & 0xffff)), ldb(f(c.x >> 16)));
                        msub(odd, ldb(f(c.y & 0xffff)), ldb(f(c.y >> 16)));
                        acc = {acc.a + odd.a, acc.b + odd.b, acc.c + odd.c, acc.d + odd.d};
                    }
                }
                T v[4] = {acc.a, acc.b, acc.c, acc.d};
                row_sum(v, ls);
                acc = {v[0], v[1], v[2], v[3]};
                if (own) {
                    if (t & SMALL_DIAG) {
                        bool ok;
                        acc = inv2(acc, ok);
                        ok_all &= ok;
                    }
                    stb(f(t & 0xffff), acc);
                }
            }
            __syncthreads();
            if (rb.w > 0) {
                for (int e = e0; e < rb.w; e += ne) {
                    if (e != e0) s = P.words[rb.z + e];
                    Blk<T>* l = f(s & 0xffff);
                    stb(l, mul(ldb(l), ldb(f(s >> 16))));
                }
                __syncthreads();
            }
        }
        if (P.n_tail > 0) {
            const int N = 2 * P.n_tail, ld = small_ld(N);
            for (int t = e0; t < P.n_schur; t += ne) {
                const int4 q = P.schur[t];
                Blk<T> acc = (q.w >> 30) ? ldb(f(q.x)) : Blk<T>{0, 0, 0, 0};
#pragma unroll 4
                for (int p = q.y; p < q.z; ++p) {
                    const int2 c = P.pairs[p];
                    msub(acc, ldb(f(c.x)), ldb(f(c.y)));
                }
                const int pos = q.w & ((1 << 30) - 1);
                const int r = 2 * (pos / P.n_tail) * ld + 2 * (pos % P.n_tail);
                d(r)[lane] = acc.a;
                d(r + 1)[lane] = acc.b;
                d(r + ld)[lane] = acc.c;
                d(r + ld + 1)[lane] = acc.d;
            }
            __syncthreads();
            ok_all &= dense_lu(N, ld);
        }
        return ok_all;
    }
    // Right-looking, one barrier per column: column k of L stays unscaled while the updates read
    // it (every thread forms l = a / pivot itself) and all of L is scaled at the end.
    __device__ __forceinline__ bool dense_lu(int N, int ld) const {
        constexpr int TJ = 16;
        const int tj = e0 % TJ, ti = e0 / TJ, ni = ne / TJ;
        bool ok = true;
        for (int k = 0; k + 1 < N; ++k) {
            const T piv = d(k * ld + k)[lane];
            ok &= fabs(piv) >= T(1e-14);
            const T inv = T(1) / piv;
            if (e0 == 0) d(N * ld + k)[lane] = inv;
            for (int i = k + 1 + ti; i < N; i += ni) {
                const T l = d(i * ld + k)[lane] * inv;
                for (int j = k + 1 + tj; j < N; j += TJ) {
                    T* c = d(i * ld + j) + lane;
                    *c = fma(-l, d(k * ld + j)[lane], *c);
                }
            }
            __syncthreads();
        }
        ok &= fabs(d((N - 1) * ld + N - 1)[lane]) >= T(1e-14);
        for (int i = 1 + ti; i < N; i += ni)
            for (int j = tj; j < i; j += TJ) d(i * ld + j)[lane] *= d(N * ld + j)[lane];
        __syncthreads();
        return ok;
    }

    // One sweep over a level's rows: x(k) takes the sum of row k's entries (factor slot, node) and,
    // in the backward sweep, its pivot block.  `w`: this thread's first entry, fetched a level
    // ahead; the row's own values are read before its entries, off the chain of the sums.
    template <bool BWD>
    __device__ __forceinline__ void level_rows(int lb, int rows, int base, int ml, uint2 w, bool accumulate) const {
        const int ls = ml >> 16, M = ml & 0xffff, W = rows << ls, wl = e0 & (32 / CL - 1);
        for (int e = e0; e - wl < W; e += ne) {
            const bool on = e < W, own = on && (e & ((1 << ls) - 1)) == 0;
            const int k = lb + (e >> ls);
            Vec2<T> b = {T(0), T(0)};
            Blk<T> pivot = {T(0), T(0), T(0), T(0)};
            if (own) {
                b = ldv(x(k));
                if (BWD) pivot = ldb(f(k));
            }
            Vec2<T> acc = {T(0), T(0)};
            if (on) {
                const uint2* next = P.ell + base + e;
                if (e != e0 && M) w = *next;
                for (int m = 1; m <= M; ++m) {
                    const uint2 c = w;
                    if (m < M) w = *(next += W);
                    Vec2<T> odd = {T(0), T(0)};
                    msubv(acc, ldb(f(c.x & 0xffff)), ldv(x(c.x >> 16)));
                    msubv(odd, ldb(f(c.y & 0xffff)), ldv(x(c.y >> 16)));
                    acc = {acc.x + odd.x, acc.y + odd.y};
                }
            }
            T v[2] = {acc.x, acc.y};
            row_sum(v, ls);
            if (own) {
                Vec2<T> r = {b.x + v[0], b.y + v[1]};
                if (BWD) r = mulv(pivot, r);
                stv(x(k), r);
                if (BWD) out(k, r, accumulate);
            }
        }
        __syncthreads();
    }
    // x: right-hand side -> solution (L y = b, then U x = y); the FP64 correction = or += x
    __device__ __forceinline__ void solve(bool accumulate) const {
        const int n_fwd = P.n_levels + (P.n_tail > 0 ? 1 : 0);
        uint2 w1 = make_uint2(0, 0);
        auto first = [&](int rows, int base, int ml) {
            if (e0 < rows << (ml >> 16) && (ml & 0xffff)) w1 = P.ell[base + e0];
        };
        if (n_fwd > 0) first(rec(0, 0).y, rec(0, 2).x, rec(0, 2).y);
        for (int h = 0; h < n_fwd; ++h) {
            const int4 ra = rec(h, 0), rc = rec(h, 2);
            const uint2 w = w1;
            if (h + 1 < n_fwd) first(rec(h + 1, 0).y, rec(h + 1, 2).x, rec(h + 1, 2).y);
            level_rows<false>(ra.x, ra.y, rc.x, rc.y, w, false);
        }
        if (P.n_tail > 0) {
            dense_solve(2 * P.n_tail);
            __syncthreads();
            for (int k = P.ns + e0; k < P.nb; k += ne) out(k, ldv(x(k)), accumulate);
        }
        const int hl = P.n_levels - 1;
        if (hl >= 0) first(rec(hl, 0).y, rec(hl, 2).z, rec(hl, 2).w);
        for (int h = hl; h >= 0; --h) {
            const int4 ra = rec(h, 0), rc = rec(h, 2);
            const uint2 w = w1;
            if (h > 0) first(rec(h - 1, 0).y, rec(h - 1, 2).z, rec(h - 1, 2).w);
            level_rows<true>(ra.x, ra.y, rc.z, rc.w, w, accumulate);
        }
    }
    __device__ __forceinline__ void out(int k, Vec2<T> r, bool accumulate) const {
        double2 c = make_double2((double)r.x, (double)r.y);
        if constexpr (sizeof(T) == 4) {
            if (accumulate) c = make_double2(dx(k).x + c.x, dx(k).y + c.y);
            dx(k) = c;
        }
        B.dx[at(P.nb, k)] = c;
    }
    __device__ __forceinline__ double2 correction(int k) const {
        if constexpr (sizeof(T) == 4) return dx(k);
        const Vec2<T> r = ldv(x(k));
        return make_double2((double)r.x, (double)r.y);
    }
    // One warp per lane, the tail vector in its registers (entry 32 r + thread), column by column
    __device__ __forceinline__ void dense_solve(int N) const {
        const int ln = threadIdx.x & 31, ld = small_ld(N), nw = blockDim.x >> 5;
        T* xt = reinterpret_cast<T*>(sm() + of_x);
        for (int w = threadIdx.x >> 5; w < CL; w += nw) {
            auto xi = [&](int i) { return ((P.ns + (i >> 1)) * CL + w) * 2 + (i & 1); };
            T y[SMALL_YR];
#pragma unroll
            for (int r = 0; r < SMALL_YR; ++r) y[r] = 32 * r + ln < N ? xt[xi(32 * r + ln)] : T(0);
#pragma unroll
            for (int rk = 0; rk < SMALL_YR; ++rk) {
                for (int kk = 0; kk < 32 && 32 * rk + kk < N; ++kk) {
                    const int k = 32 * rk + kk;
                    const T yk = __shfl_sync(0xffffffffu, y[rk], kk);
#pragma unroll
                    for (int r = rk; r < SMALL_YR; ++r) {
                        const int i = 32 * r + ln;
                        if (i > k && i < N) y[r] = fma(-d(i * ld + k)[w], yk, y[r]);
                    }
                }
            }
#pragma unroll
            for (int rk = SMALL_YR - 1; rk >= 0; --rk) {
                for (int kk = min(31, N - 1 - 32 * rk); kk >= 0; --kk) {
                    const int k = 32 * rk + kk;
                    if (ln == kk) y[rk] = y[rk] / d(k * ld + k)[w];
                    const T yk = __shfl_sync(0xffffffffu, y[rk], kk);
#pragma unroll
                    for (int r = 0; r <= rk; ++r) {
                        const int i = 32 * r + ln;
                        if (i < k) y[r] = fma(-d(i * ld + k)[w], yk, y[r]);
                    }
                }
            }
#pragma unroll
            for (int r = 0; r < SMALL_YR; ++r)
                if (32 * r + ln < N) xt[xi(32 * r + ln)] = y[r];
        }
    }
    // x = rhs - J dx with the FP64 Jacobian
    __device__ __forceinline__ void residual() const {
        const Blk<double>* A = reinterpret_cast<const Blk<double>*>(B.A64);
        for (int k = e0; k < P.nb; k += ne) {
            const double2 b = B.rhs[at(P.nb, k)];
            Vec2<double> acc = {b.x, b.y};
#pragma unroll 4
            for (int e = P.arow_ptr[k]; e < P.arow_ptr[k + 1]; ++e) {
                const int2 ac = P.arow[e];
                const double2 u = correction(ac.y);
                msubv(acc, ldb(A + at(P.n_a, ac.x)), Vec2<double>{u.x, u.y});
            }
            stv(x(k), Vec2<T>{(T)acc.x, (T)acc.y});
        }
    }
};

// One CTA per (lane group, CL of its lanes), from iteration it0 for `passes` iterations (0: until
// the lanes are done).  State and group words, voltages, rhs, dx and, on exit, the factors are the
// ones the separate kernels keep, so every other call on the batch finds them (a CTA that factorised
// nothing leaves the stored factors as they are).  With `together` the group's CTAs are one cluster.
// A group's giter and gsolve are written by several CTAs: none of them reads these words.
template <typename T, int CL>
__global__ void __launch_bounds__(SMALL_THREADS, 4)
    k_nr_small(PlanDev P, BatchDev B, int refine, int together, int passes) {
    namespace cg = cooperative_groups;
    __shared__ double red[SMALL_THREADS / 32][CL];
    __shared__ double mis[CL];
    __shared__ int state[CL], solving[CL], singular[CL];
    __shared__ int any_solving, any_iter, do_factor, do_refine, factorised, word[2];
    const SmallLayout L = small_layout(P.n_bus, P.nb, P.n_slots, P.n_tail, P.n_levels, CL, sizeof(T));
    const int parts = B.sw / CL, g = blockIdx.x / parts, tid = threadIdx.x;
    bool iterates = false;  // any lane that decides with this CTA's (padding lanes are done)
    for (int l = 0; l < (together ? B.sw : CL); ++l)
        iterates |= B.state[g * B.sw + (together ? 0 : blockIdx.x % parts * CL) + l] == 0;
    if (!iterates) return;
    const int lane = tid % CL, gl = (blockIdx.x % parts) * CL + lane, q = g * B.sw + gl;
    const int N = 2 * P.n_tail;
    const SmallCta<T, CL> c{P, B, (int)L.v, (int)L.x, (int)L.dx, (int)L.d, (int)L.lv, lane, tid / CL,
                            (int)blockDim.x / CL, (size_t)gl, g, B.sw};
    int4* lv = reinterpret_cast<int4*>(c.sm() + L.lv);
    for (int i = tid; i < 3 * (P.n_levels + 1); i += blockDim.x) lv[i] = P.levels[i];
    for (int i = c.e0; i < P.n_bus; i += c.ne) c.v(i) = B.V[c.at(P.n_bus, i)];
    if (tid < CL) {
        stb(c.f(P.n_slots), Blk<T>{0, 0, 0, 0});
        stv(c.x(P.nb), Vec2<T>{0, 0});
    }
    if (tid == 0) factorised = 0;
    if (tid < CL) {
        state[tid] = B.state[q];
        solving[tid] = B.solving[q];
        singular[tid] = B.singular[q];
    }
    if (passes) {
        // a later step: the factors may be reused
        const Blk<T>* Fg = reinterpret_cast<const Blk<T>*>(B.F);
        for (int s = c.e0; s < P.n_slots; s += c.ne) stb(c.f(s), ldb(Fg + c.at(P.n_slots, s)));
        if (N > 0) {
            const T* Dg = reinterpret_cast<const T*>(B.Dt) + (size_t)q * N * dense_ld(N);
            for (int i = c.e0; i < N; i += c.ne)
                for (int j = 0; j < N; ++j)
                    c.d(i * small_ld(N) + j)[lane] = Dg[(size_t)i * dense_ld(N) + j];
        }
    }
    const int max_iter = B.ctrl[1], policy = B.ctrl[3], it0 = passes ? B.ctrl[0] : 0;
    const double tol = B.tol[0];
    const double below_refine = B.A64 ? B.tol[1] : 0.0, below_reuse = B.A64 ? B.tol[2] : 0.0;
    __syncthreads();
    int it = it0;
    for (;; ++it) {
        double m = c.mismatch();
#pragma unroll
        for (int off = CL; off < 32; off <<= 1) m = nmax(m, __shfl_xor_sync(0xffffffffu, m, off));
        if ((tid & 31) < CL) red[tid >> 5][tid & 31] = m;
        __syncthreads();
        if (tid < CL) {
            // k_check's test of this lane
            double r = red[0][tid];
            for (int k = 1; k < (int)(blockDim.x >> 5); ++k) r = nmax(r, red[k][tid]);
            solving[tid] = 0;
            if (q < B.n_scen && state[tid] == 0) {
                mis[tid] = r;
                B.final_mis[q] = r;
                if (!isfinite(r) || r < tol) {
                    state[tid] = 1;
                    B.status[q] = isfinite(r) ? SC_CONVERGED : SC_NONFINITE;
                    B.iters[q] = it + 1;
                } else {
                    solving[tid] = 1;
                    if (it + 1 >= max_iter) {
                        state[tid] = 1;
                        B.status[q] = SC_MAXITER;
                        B.iters[q] = max_iter;
                    }
                }
            }
            __syncwarp((1u << CL) - 1);
            if (tid == 0) {
                // bits: a lane solves, a lane iterates, one below the refinement threshold, one
                // not below the reuse threshold
                int w = 0;
                for (int l = 0; l < CL; ++l) {
                    if (q + l < B.n_scen && state[l] == 0) w |= 2;
                    if (solving[l]) w |= 1 | (mis[l] < below_refine ? 4 : 0) | (mis[l] < below_reuse ? 0 : 8);
                }
                word[it & 1] = w;
            }
        }
        if (together) cg::this_cluster().sync();
        else __syncthreads();
        if (tid == 0) {
            int w = word[it & 1];
            any_solving = w & 1;
            if (together)
                for (int r = 0; r < parts; ++r) w |= *cg::this_cluster().map_shared_rank(&word[it & 1], r);
            any_iter = w & 2;
            // (only factors of this solve are reused)
            do_factor = it == 0 || !(below_reuse > 0.0 && (w & 1) && !(w & 8));
            if (any_solving && do_factor) factorised = 1;  // by this CTA
            do_refine = below_refine <= 0.0 || (w & 4) || !do_factor;
        }
        __syncthreads();
        if (any_solving) {
            c.jacobian(do_factor, refine > 0 && do_refine);
            __syncthreads();
            if (do_factor && !c.factor()) singular[lane] = 1;
            c.solve(false);
            if (do_refine) {
                for (int r = 0; r < refine; ++r) {
                    __syncthreads();
                    c.residual();
                    __syncthreads();
                    c.solve(true);
                }
            }
            __syncthreads();
            if (q < B.n_scen && solving[lane] && !singular[lane]) {
                for (int i = c.e0; i < P.n_bus; i += c.ne) {
                    const int node = P.node_of_bus[i];
                    if (node >= 0)
                        c.v(i) = newton_step(c.v(i), c.correction(node), P.bus_type[i] == BUS_PQ, policy);
                }
            }
            __syncthreads();
            if (tid < CL && q < B.n_scen && solving[tid] && singular[tid]) {
                // the reference keeps V unchanged when factorize() fails and runs to max_iter
                state[tid] = 1;
                solving[tid] = 0;
                B.status[q] = SC_SINGULAR;
                B.iters[q] = max_iter;
            }
        }
        if (!any_iter || it + 1 - it0 == passes) break;
        __syncthreads();  // the flags are read before the next test writes them
    }
    __syncthreads();
    for (int i = c.e0; i < P.n_bus; i += c.ne) B.V[c.at(P.n_bus, i)] = c.v(i);
    if (factorised) {
        Blk<T>* Fg = reinterpret_cast<Blk<T>*>(B.F);
        for (int s = c.e0; s < P.n_slots; s += c.ne) stb(Fg + c.at(P.n_slots, s), ldb(c.f(s)));
    }
    if (factorised && N > 0) {
        T* Dg = reinterpret_cast<T*>(B.Dt) + (size_t)q * N * dense_ld(N);
        for (int i = c.e0; i < N; i += c.ne)
            for (int j = 0; j < N; ++j)
                Dg[(size_t)i * dense_ld(N) + j] = c.d(i * small_ld(N) + j)[lane];
    }
    if (tid < CL) {
        B.state[q] = state[tid];
        B.solving[q] = solving[tid];
        B.singular[q] = singular[tid];
    }
    if (tid == 0) {
        // the words of the last k_check; gsolve is 0 before a stepped pass and 1 before a whole
        // solve, whose CTAs collect theirs in bit 1
        if (any_solving) atomicOr(&B.gsolve[g], 2);
        if (!passes) {
            atomicAnd(&B.gsolve[g], ~1);
            B.giter[g] = 0;
        }
        if (B.grefine) B.grefine[g] = do_refine;
        if (B.gfactor) B.gfactor[g] = do_factor;
        if (passes) {
            if (any_iter) atomicOr(&B.ctrl[2], 1);  // k_small_step advances the other words
        } else {
            atomicMax(&B.ctrl[0], it + 1);
            atomicMax(&B.ctrl[4], it + 1);
            B.ctrl[2] = 0;
        }
    }
    if (together) cg::this_cluster().sync();  // a neighbour may still read this CTA's word
}

// Around one stepped pass: before it ([2] any iterating and each group's gsolve = 0), after it (the
// iteration count and which groups still iterate).
__global__ void k_small_step(BatchDev B, int after) {
    if (!after) {
        if (threadIdx.x == 0) B.ctrl[2] = 0;
        for (int g = threadIdx.x; g < B.n_groups; g += blockDim.x) B.gsolve[g] = 0;
        return;
    }
    for (int g = threadIdx.x; g < B.n_groups; g += blockDim.x) {
        int iv = 0;
        for (int l = 0; l < B.sw; ++l) iv |= g * B.sw + l < B.n_scen && B.state[g * B.sw + l] == 0;
        B.giter[g] = iv;
    }
    if (threadIdx.x == 0) {
        B.ctrl[0] += 1;
        B.ctrl[4] = B.ctrl[0];
    }
}

}  // namespace gapk
