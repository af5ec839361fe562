// Host side of the Newton-Raphson engine: plan upload, batch state, the device-resident
// iteration loop (CUDA graph with a conditional while node), and the gapk_nr_* C ABI.
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdio>
#include <cstring>
#include <memory>
#include <mutex>
#include <string>
#include <type_traits>
#include <vector>

#include <nvtx3/nvToolsExt.h>

#include "../../include/gapk.h"
#include "internal.h"
#include "nr_kernels.cuh"
#include "nr_small.cuh"

namespace gapk {

namespace {
thread_local std::string g_err = "no error";
}
void set_error(std::string const& msg) { g_err = msg; }

#define GAPK_CUDA_TRY(expr)                                                         \
    do {                                                                            \
        cudaError_t e__ = (expr);                                                   \
        if (e__ != cudaSuccess) {                                                   \
            set_error(std::string(#expr) + ": " + cudaGetErrorString(e__));         \
            return e__ == cudaErrorMemoryAllocation ? GAPK_ENOMEM : GAPK_ECUDA;     \
        }                                                                           \
    } while (0)

// ---- device buffers -------------------------------------------------------------------
struct DevBuf {
    void* p = nullptr;
    size_t bytes = 0;
    DevBuf() = default;
    DevBuf(DevBuf const&) = delete;
    DevBuf& operator=(DevBuf const&) = delete;
    ~DevBuf() {
        if (p) cudaFree(p);
    }
    int alloc(size_t n) {
        if (p) cudaFree(p);
        p = nullptr;
        bytes = n;
        if (n == 0) return GAPK_OK;
        GAPK_CUDA_TRY(cudaMalloc(&p, n));
        return GAPK_OK;
    }
    template <typename V>
    int upload(std::vector<V> const& v) {
        int rc = alloc(v.size() * sizeof(V));
        if (rc) return rc;
        if (!v.empty()) GAPK_CUDA_TRY(cudaMemcpy(p, v.data(), bytes, cudaMemcpyHostToDevice));
        return GAPK_OK;
    }
    template <typename P>
    P* as() const {
        return reinterpret_cast<P*>(p);
    }
};

}  // namespace gapk

using namespace gapk;

struct gapk_nr_plan_s {
    NRPlanHost h;
    std::vector<int> y_row_ptr, y_col;
    bool general = false;  // the plan of a general LU, not of a Newton solve
    std::vector<int> a_rec;  // a_records(), made with the plan
    // device copy (current device at first upload): all lists in one allocation
    bool uploaded = false;
    int device = -1;
    DevBuf d_lists;
    PlanDev dev{};
    const int *var_of_comp = nullptr, *eq_of_comp = nullptr;

    // the Jacobian fill's records (jac_block), four ints per block
    std::vector<int> a_records() const {
        std::vector<int> r(4 * (size_t)h.n_a);
        auto bus = [&](int i) { return i | (h.bus_type[i] == BUS_PQ ? REC_PQ : 0); };
        for (int a = 0; a < h.n_a; ++a) {
            const int slot = h.a_slots[a];
            const int* si = &h.slot_info[4 * (size_t)slot];
            r[4 * (size_t)a] = slot;
            r[4 * (size_t)a + 1] = bus(si[0]);
            r[4 * (size_t)a + 2] = bus(si[1]);
            r[4 * (size_t)a + 3] = si[3] - si[2] == 1 ? h.slot_src[si[2]] : -1;
        }
        return r;
    }

    // k_nr_small's packed schedule (SmallCta): false when not even one FP32 scenario fits its shared
    // memory, its 16-bit indices or its tail, and for a general matrix.  Threads per target or row
    // (1, 2 or 4): a pass over two entries costs about 70 cycles of latency, adding up two threads'
    // parts about 45, so the longest row decides where the level leaves threads idle; a wide level
    // keeps a thread per row.
    bool small_schedule(std::vector<int>& rec, std::vector<unsigned>& words,
                        std::vector<unsigned>& ell) const {
        if (general || h.n_slots > 0xffff || h.nb > 0xffff || h.n_tail > SMALL_MAX_TAIL ||
            small_layout(h.n_bus, h.nb, h.n_slots, h.n_tail, h.n_levels, 1, 4).total > SMALL_SMEM_MAX)
            return false;
        // rows [0, rows) of count(r) words word(r, i), two words to an entry, padded to the
        // longest part with `pad`; returns (first entry, entries of the longest part | split << 16)
        auto lists = [&](int rows, auto count, auto word, unsigned pad, int* out) {
            int most = 0;
            for (int r = 0; r < rows; ++r) most = std::max(most, count(r));
            const int ls = rows <= 64 && most > 4 ? 2 : rows <= 128 && most > 2 ? 1 : 0;
            const int s = 1 << ls, longest = (most + 2 * s - 1) / (2 * s);
            const size_t at = ell.size();
            out[0] = (int)(at / 2);
            out[1] = longest | ls << 16;
            ell.resize(at + 2 * (size_t)longest * rows * s, pad);
            // word i = (2 m + o) s + sub of a row: half o of entry m of its part `sub`
            for (int r = 0; r < rows; ++r)
                for (int i = 0, n = count(r); i < n; ++i) {
                    const int sub = i % s, k = i / s;
                    ell[at + 2 * (((size_t)(k / 2) * rows + r) * s + sub) + k % 2] = word(r, i);
                }
        };
        auto pack = [](int lo, int hi) { return (unsigned)lo | (unsigned)hi << 16; };
        const unsigned none = pack(h.n_slots, h.n_slots), no_row = pack(h.n_slots, h.nb);
        rec.assign(12 * ((size_t)h.n_levels + 1), 0);
        for (int l = 0; l <= h.n_levels; ++l) {
            const bool tail = l == h.n_levels;
            int* q = &rec[12 * (size_t)l];
            const int lb = tail ? h.ns : h.level_ptr[l], c = tail ? h.n_tail : h.level_ptr[l + 1] - lb;
            q[0] = lb;
            q[1] = c;
            if (!tail) {
                const int t0 = h.fa_ptr[l], nt = h.fa_ptr[l + 1] - t0;
                const int* tg = &h.targets[4 * (size_t)t0];
                q[2] = (int)words.size();
                q[3] = nt;
                for (int t = 0; t < nt; ++t)
                    words.push_back((unsigned)tg[4 * t] | (tg[4 * t + 3] & 1 ? SMALL_DIAG : 0) |
                                  (tg[4 * t + 3] & 2 ? SMALL_VALUE : 0));
                lists(nt, [&](int t) { return tg[4 * t + 2] - tg[4 * t + 1]; },
                      [&](int t, int i) {
                          const int* p = &h.pairs[2 * (size_t)(tg[4 * t + 1] + i)];
                          return pack(p[0], p[1]);
                      }, none, q + 4);
                q[6] = (int)words.size();
                q[7] = h.fb_ptr[l + 1] - h.fb_ptr[l];
                for (int t = h.fb_ptr[l]; t < h.fb_ptr[l + 1]; ++t)
                    words.push_back(pack(h.scale[2 * (size_t)t], h.scale[2 * (size_t)t + 1]));
                lists(c, [&](int r) { return h.lptr[lb + r + 1] - h.lptr[lb + r]; },
                      [&](int r, int i) {
                          const int p = h.lptr[lb + r] + i;
                          return pack(h.nb + h.nnz_l + p, h.lidx[p]);
                      }, no_row, q + 10);
            }
            lists(c, [&](int r) { return h.rptr[lb + r + 1] - h.rptr[lb + r]; },
                  [&](int r, int i) {
                      const int* p = &h.rlist[2 * (size_t)(h.rptr[lb + r] + i)];
                      return pack(p[0], p[1]);
                  }, no_row, q + 8);
        }
        return true;
    }

    // One allocation for all lists, one copy for those of at most 64 KB (a 200-bus plan and its
    // one-scenario FP64 batch made and destroyed: 735 us with an allocation and a copy for each list,
    // 440 so).  Larger lists are copied from where they are: collecting them too costs more than their
    // copies' calls.
    int upload() {
        if (uploaded) return GAPK_OK;
        std::vector<int> rec;
        std::vector<unsigned> words, ell;
        std::vector<unsigned char> host;  // the small lists, the allocation's front
        auto lists = [&](auto f) {
            f(dev.y_row_ptr, y_row_ptr);
            f(dev.y_col, y_col);
            f(dev.bus_type, h.bus_type);
            f(dev.node_of_bus, h.node_of_bus);
            f(dev.slot_info, h.slot_info);
            f(dev.slot_src, h.slot_src);
            f(dev.level_ptr, h.level_ptr);
            f(dev.fa_ptr, h.fa_ptr);
            f(dev.targets, h.targets);
            f(dev.pairs, h.pairs);
            f(dev.fb_ptr, h.fb_ptr);
            f(dev.scale, h.scale);
            f(dev.lptr, h.lptr);
            f(dev.lidx, h.lidx);
            f(dev.rptr, h.rptr);
            f(dev.rlist, h.rlist);
            f(dev.arow_ptr, h.arow_ptr);
            f(dev.arow, h.arow);
            f(dev.acol_ptr, h.acol_ptr);
            f(dev.acol, h.acol);
            f(dev.schur, h.schur);
            f(dev.a_slots, h.a_slots);
            f(dev.a_rec, a_rec);
            f(var_of_comp, h.var_of_comp);
            f(eq_of_comp, h.eq_of_comp);
            f(dev.levels, rec);
            f(dev.words, words);
            f(dev.ell, ell);
        };
        // f(pointer, list, offset, small)
        size_t front = 0, total = 0;
        auto each = [&](auto f) {
            size_t at[2] = {front, 0};  // of the next large, small list
            lists([&](auto& p, auto const& v) {
                const size_t bytes = v.size() * 4;
                const bool small = bytes <= 64 * 1024;
                f(p, v, at[small], small);
                at[small] += (bytes + 255) & ~size_t(255);
            });
            total = at[0];
            return at[1];
        };
        try {
            if (!small_schedule(rec, words, ell)) {
                rec.clear();
                words.clear();
                ell.clear();
            }
            front = each([](auto&, auto const&, size_t, bool) {});
            host.resize(front);
        } catch (std::bad_alloc const&) {
            set_error("plan upload: host allocation failed");
            return GAPK_ENOMEM;
        }
        each([&](auto&, auto const& v, size_t at, bool small) {
            if (small && !v.empty()) std::memcpy(host.data() + at, v.data(), v.size() * 4);
        });
        int rc = d_lists.alloc(total);
        if (rc) return rc;
        cudaError_t e = cudaMemcpy(d_lists.p, host.data(), front, cudaMemcpyHostToDevice);
        each([&](auto& p, auto const& v, size_t at, bool small) {
            using P = std::remove_reference_t<decltype(p)>;
            unsigned char* d = d_lists.as<unsigned char>() + at;
            p = v.empty() ? nullptr : reinterpret_cast<P>(d);
            if (!small && e == cudaSuccess) e = cudaMemcpy(d, v.data(), v.size() * 4, cudaMemcpyHostToDevice);
        });
        GAPK_CUDA_TRY(e);
        cudaGetDevice(&device);
        dev.n_bus = h.n_bus;
        dev.nb = h.nb;
        dev.nnz_y = h.nnz_y;
        dev.n_slots = h.n_slots;
        dev.nnz_l = h.nnz_l;
        dev.n_levels = h.n_levels;
        dev.n_a = h.n_a;
        dev.jac_mode = h.jac_mode;
        dev.ns = h.ns;
        dev.n_tail = h.n_tail;
        dev.n_schur = static_cast<int>(h.schur.size() / 4);
        uploaded = true;
        return GAPK_OK;
    }
};

struct SmallRun {
    int cl = 0, threads = 0, together = 0, carveout = 100;
};

struct gapk_nr_batch_s {
    gapk_nr_plan plan = nullptr;
    int n_scen = 0, sw = 8, G = 0, precision = 0, y_shared = 1, threads = 256, use_graph = 1;
    int dense_fused = 0;
    int level_ctas = 1;  // CTAs per lane group of the level-scheduled kernels
    int split_slots = 0; // k_factor's split_slots
    int dense_ctas = 1;  // CTAs per scenario of the dense tail's solves
    DevBuf V, Sspec, Scalc, Y, F, A64, rhs, dx, res, X, Dt, mis, state, solving, singular,
        iters, status, fmis, gsolve, giter, grefine, gfactor, ctrl, tol;
    int dense_w = 0;          // panel width of the one-CTA-per-scenario dense LU (0: not used)
    size_t dense_smem = 0;    // its dynamic shared memory
    bool dense_split = false; // factorise the tail with the split kernels
    bool dense_tc = false;    // FP32 tail: trailing updates on the tensor cores (either LU path)
    BatchDev dev{};
    // graph cache
    cudaGraph_t graph = nullptr;
    cudaGraphExec_t exec = nullptr;
    int graph_refine = -1;
    int cur_refine = 0;
    SmallRun cur_small;  // how the last inputs' solve runs
    int wait_test = 0;   // the tensor-core LU's wait test is on
    ~gapk_nr_batch_s() {
        if (exec) cudaGraphExecDestroy(exec);
        if (graph) cudaGraphDestroy(graph);
    }
};

namespace {

inline unsigned blocks_for(long items, int threads) {
    return static_cast<unsigned>((items + threads - 1) / threads);
}

// `units` clusters of nc CTAs (plain CTAs for nc = 1).
template <typename K, typename... A>
void launch_clusters(int units, int nc, int threads, size_t smem, cudaStream_t st, K kernel, A... args) {
    cudaLaunchConfig_t cfg{};
    cudaLaunchAttribute cluster{};
    cluster.id = cudaLaunchAttributeClusterDimension;
    cluster.val.clusterDim.x = nc;
    cluster.val.clusterDim.y = cluster.val.clusterDim.z = 1;
    cfg.gridDim = dim3(units * nc);
    cfg.blockDim = dim3(threads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cfg.attrs = &cluster;
    cfg.numAttrs = nc > 1 ? 1 : 0;
    cudaLaunchKernelEx(&cfg, kernel, args...);
}
// A level-scheduled kernel, b->level_ctas CTAs per lane group.
template <typename K, typename... A>
void launch_levels(gapk_nr_batch b, cudaStream_t st, K kernel, A... args) {
    launch_clusters(b->G, b->level_ctas, b->threads, 0, st, kernel, args...);
}
template <typename T, int SW>
void launch_sparse_factor(gapk_nr_batch b, cudaStream_t st) {
    launch_levels(b, st, b->split_slots ? k_factor<T, SW, true> : k_factor<T, SW, false>, b->plan->dev,
                  b->dev, b->split_slots);
}
// The tail's two substitutions; k_dense_solve streams best when its CTAs fill the GPU, for tails that
// fit the 48 KB that any launch gets (order 5,088 in FP64).
template <typename T, int SW, bool TR>
void launch_dense_solve(gapk_nr_batch b, cudaStream_t st, double2* out, int acc) {
    PlanDev const& P = b->plan->dev;
    if (P.n_tail == 0) return;
    const size_t smem = dense_solve_smem(P.n_tail, sizeof(T));
    if (TR || b->dense_ctas > 1 || smem + 32 * 33 * sizeof(T) > 48 * 1024)
        launch_clusters(b->G * SW, b->dense_ctas, DS_THREADS, smem, st, k_dense_solve_cl<T, SW, TR>, P, b->dev, out, acc);
    else
        k_dense_solve<T, SW><<<b->G * SW, 256, smem, st>>>(P, b->dev, out, acc);
}

template <typename T, int SW>
void launch_solve(gapk_nr_batch b, cudaStream_t st, const double2* rhs, double2* out, int acc) {
    PlanDev const& P = b->plan->dev;
    BatchDev const& B = b->dev;
    launch_levels(b, st, k_solve_fwd<T, SW, false>, P, B, rhs, acc);
    launch_dense_solve<T, SW, false>(b, st, out, acc);
    launch_levels(b, st, k_solve_bwd<T, SW, false>, P, B, out, acc);
}

template <typename T, int SW>
void launch_factor(gapk_nr_batch b, cudaStream_t st) {
    PlanDev const& P = b->plan->dev;
    BatchDev const& B = b->dev;
    launch_sparse_factor<T, SW>(b, st);
    if (P.n_tail > 0) {
        dim3 gs(blocks_for((long)P.n_schur * SW, 256), b->G);
        k_schur<T, SW><<<gs, 256, 0, st>>>(P, B);
        if (b->dense_split)
            launch_dense_lu_split<T>(b->G * SW, st, B, 2 * P.n_tail, b->dense_tc);
        else
            launch_dense_lu<T>(b->dense_w, b->G * SW, b->dense_smem, st, B, 2 * P.n_tail, b->dense_tc);
    }
}

template <typename T, int SW>
void launch_body(gapk_nr_batch b, cudaStream_t st, int use_cond, cudaGraphConditionalHandle h) {
    PlanDev const& P = b->plan->dev;
    BatchDev const& B = b->dev;
    const int G = b->G;
    k_mismatch<SW><<<mismatch_grid<SW>(P, G), 256, 0, st>>>(P, B);
    k_check<SW><<<1, 1024, 0, st>>>(B, use_cond, h);
    dim3 gj(blocks_for((long)P.n_a * SW, 256), G);
    k_jfill<T, SW><<<gj, 256, 0, st>>>(P, B);
    launch_factor<T, SW>(b, st);
    launch_solve<T, SW>(b, st, B.rhs, B.dx, 0);
    for (int r = 0; r < b->cur_refine; ++r) {
        dim3 gr(blocks_for((long)P.nb * SW, 256), G);
        k_residual<SW><<<gr, 256, 0, st>>>(P, B);
        launch_solve<T, SW>(b, st, B.res, B.dx, 1);
    }
    dim3 gu(blocks_for((long)P.n_bus * SW, 256), G);
    k_update<SW><<<gu, 256, 0, st>>>(P, B);
}

template <int SW>
void launch_load(gapk_nr_batch b, const gapk_nr_inputs* in, cudaStream_t st) {
    PlanDev const& P = b->plan->dev;
    dim3 g(blocks_for((long)P.n_bus * SW, 256), b->G);
    k_load<SW><<<g, 256, 0, st>>>(P, b->dev, reinterpret_cast<const double2*>(in->d_y),
                                  reinterpret_cast<const double2*>(in->d_s_spec),
                                  reinterpret_cast<const double2*>(in->d_v_init), in->d_u_pu,
                                  in->v_init_shared,
                                  SolveOpts{1, in->max_iterations, in->policy, in->tolerance,
                                            in->refine_below, in->reuse_below});
}

template <int SW>
void launch_store(gapk_nr_batch b, const gapk_nr_outputs* out, cudaStream_t st) {
    PlanDev const& P = b->plan->dev;
    long total = (long)b->n_scen * P.n_bus;
    k_store<SW><<<blocks_for(total, 256), 256, 0, st>>>(
        P, b->dev, reinterpret_cast<double2*>(out->d_v), out->d_iterations, out->d_status,
        out->d_final_mismatch);
}

// dispatch on (precision, lanes)
template <template <typename, int> class F, typename... A>
int dispatch_tsw(int precision, int sw, A&&... a) {
#define GAPK_CASE(T, S) F<T, S>::run(std::forward<A>(a)...)
    if (precision == GAPK_PREC_FP64) {
        switch (sw) {
            case 1: GAPK_CASE(double, 1); return 0;
            case 2: GAPK_CASE(double, 2); return 0;
            case 4: GAPK_CASE(double, 4); return 0;
            case 8: GAPK_CASE(double, 8); return 0;
        }
    } else {
        switch (sw) {
            case 1: GAPK_CASE(float, 1); return 0;
            case 2: GAPK_CASE(float, 2); return 0;
            case 4: GAPK_CASE(float, 4); return 0;
            case 8: GAPK_CASE(float, 8); return 0;
        }
    }
#undef GAPK_CASE
    return -1;
}

template <typename T, int SW>
struct BodyOp {
    static void run(gapk_nr_batch b, cudaStream_t st, int uc, cudaGraphConditionalHandle h) {
        launch_body<T, SW>(b, st, uc, h);
    }
};
template <typename T, int SW>
struct LoadOp {
    static void run(gapk_nr_batch b, const gapk_nr_inputs* in, cudaStream_t st) {
        launch_load<SW>(b, in, st);
    }
};
template <typename T, int SW>
struct StoreOp {
    static void run(gapk_nr_batch b, const gapk_nr_outputs* out, cudaStream_t st) {
        launch_store<SW>(b, out, st);
    }
};
template <typename T, int SW>
struct StageOp {
    static void run(gapk_nr_batch b, int which, cudaStream_t st) {
        PlanDev const& P = b->plan->dev;
        BatchDev const& B = b->dev;
        const int G = b->G;
        switch (which) {
            case 0:
                k_mismatch<SW><<<mismatch_grid<SW>(P, G), 256, 0, st>>>(P, B);
                break;
            case 1: {
                dim3 gj(blocks_for((long)P.n_a * SW, 256), G);
                k_jfill<T, SW><<<gj, 256, 0, st>>>(P, B);
                break;
            }
            case 2:
                launch_factor<T, SW>(b, st);
                break;
            case 3:
                launch_solve<T, SW>(b, st, B.rhs, B.dx, 0);
                for (int r = 0; r < b->cur_refine; ++r) {
                    dim3 gr(blocks_for((long)P.nb * SW, 256), G);
                    k_residual<SW><<<gr, 256, 0, st>>>(P, B);
                    launch_solve<T, SW>(b, st, B.res, B.dx, 1);
                }
                break;
            case 4: {
                dim3 gu(blocks_for((long)P.n_bus * SW, 256), G);
                k_update<SW><<<gu, 256, 0, st>>>(P, B);
                break;
            }
        }
    }
};
template <typename T, int SW>
struct KernelOp {
    static void run(gapk_nr_batch b, int which, cudaStream_t st) {
        PlanDev const& P = b->plan->dev;
        BatchDev const& B = b->dev;
        const int G = b->G;
        switch (which) {
            case 0: k_mismatch<SW><<<mismatch_grid<SW>(P, G), 256, 0, st>>>(P, B); break;
            case 1: k_jfill<T, SW><<<dim3(blocks_for((long)P.n_a * SW, 256), G), 256, 0, st>>>(P, B); break;
            case 2: launch_sparse_factor<T, SW>(b, st); break;
            case 3:
                if (P.n_tail > 0)
                    k_schur<T, SW><<<dim3(blocks_for((long)P.n_schur * SW, 256), G), 256, 0, st>>>(P, B);
                break;
            case 4:
                if (P.n_tail > 0)
                    if (b->dense_split)
                        launch_dense_lu_split<T>(G * SW, st, B, 2 * P.n_tail, b->dense_tc);
                    else
                        launch_dense_lu<T>(b->dense_w, G * SW, b->dense_smem, st, B, 2 * P.n_tail, b->dense_tc);
                break;
            case 5: launch_levels(b, st, k_solve_fwd<T, SW, false>, P, B, (const double2*)B.rhs, 0); break;
            case 6:
                launch_dense_solve<T, SW, false>(b, st, B.dx, 0);
                break;
            case 7: launch_levels(b, st, k_solve_bwd<T, SW, false>, P, B, B.dx, 0); break;
            case 8: k_update<SW><<<dim3(blocks_for((long)P.n_bus * SW, 256), G), 256, 0, st>>>(P, B); break;
            case 9:
                if (B.A64) k_residual<SW><<<dim3(blocks_for((long)P.nb * SW, 256), G), 256, 0, st>>>(P, B);
                break;
        }
    }
};
template <typename T, int SW>
void launch_solve_t(gapk_nr_batch b, cudaStream_t st, const double2* rhs, double2* out, int acc) {
    PlanDev const& P = b->plan->dev;
    BatchDev const& B = b->dev;
    launch_levels(b, st, k_solve_fwd<T, SW, true>, P, B, rhs, 0);
    launch_dense_solve<T, SW, true>(b, st, out, acc);
    launch_levels(b, st, k_solve_bwd<T, SW, true>, P, B, out, acc);
}

template <typename T, int SW>
struct AdjointOp {
    static void run(gapk_nr_batch b, const double* dvm, const double* dva, double* dp, double* dq,
                    cudaStream_t st) {
        PlanDev const& P = b->plan->dev;
        BatchDev const& B = b->dev;
        const int G = b->G;
        k_adj_prep<SW><<<blocks_for((long)G * SW, 256), 256, 0, st>>>(B);
        k_mismatch<SW><<<mismatch_grid<SW>(P, G), 256, 0, st>>>(P, B);
        k_jfill<T, SW><<<dim3(blocks_for((long)P.n_a * SW, 256), G), 256, 0, st>>>(P, B);
        launch_factor<T, SW>(b, st);
        k_adj_rhs<SW><<<dim3(blocks_for((long)P.n_bus * SW, 256), G), 256, 0, st>>>(P, B, dvm, dva);
        launch_solve_t<T, SW>(b, st, B.rhs, B.dx, 0);
        if (B.A64) {
            k_residual_t<SW><<<dim3(blocks_for((long)P.nb * SW, 256), G), 256, 0, st>>>(P, B);
            launch_solve_t<T, SW>(b, st, B.res, B.dx, 1);
        }
        k_adj_out<SW><<<blocks_for((long)b->n_scen * P.n_bus, 256), 256, 0, st>>>(P, B, dp, dq);
    }
};
template <typename T, int SW>
struct AdjBranchOp {
    static void run(gapk_nr_batch b, int m, const int* f, const int* t, const double* brp, double* dr,
                    double* dx, cudaStream_t st) {
        k_adj_branch<SW><<<blocks_for((long)b->n_scen * m, 256), 256, 0, st>>>(
            b->plan->dev, b->dev, m, f, t, brp, dr, dx);
    }
};

template <typename T, int SW>
struct ToRefOp {
    static void run(gapk_nr_batch b, const double2* src, const int* map, int n_out, double sign,
                    double* dst, cudaStream_t st) {
        PlanDev const& P = b->plan->dev;
        long total = (long)b->n_scen * P.nb;
        if (total == 0) return;
        k_node_to_ref<SW><<<blocks_for(total, 256), 256, 0, st>>>(src, P.nb, b->n_scen, n_out,
                                                                   map, sign, dst);
    }
};

template <typename T, int SW>
struct StateOp {
    static void run(gapk_nr_batch b, double2* v, double2* i, double2* s, cudaStream_t st) {
        long total = (long)b->n_scen * b->plan->dev.n_bus;
        if (total == 0) return;
        k_state<SW><<<blocks_for(total, 256), 256, 0, st>>>(b->plan->dev, b->dev, v, i, s);
    }
};

// CTA size of the level-scheduled kernels where the caller leaves it open: a thread for every
// eighth (node, lane), which takes all but the widest levels in one round, while the 1,024 threads
// that their registers allow on an SM still hold all groups at once.  Whole solves with 256 / 512 /
// 1024 threads, 8 lanes: 3,001 buses, 42 groups 8.0 / - / 4.6 ms; 2,000 buses in FP32, 148 groups
// 5.74 / 4.59 / 4.06, 149 groups 5.95 / 4.81 / 5.77, 296 groups 7.82 / 6.73 / 7.81, 297 groups 7.97 /
// 9.02 / 9.44, 592 groups 12.2 / 13.1 / 15.2 ms; the same lines at 1,000 to 10,000 buses and in FP64.
// Past 592 groups the CTAs shrink by the same rule: 500 buses in FP32 with 64 / 96 / 128 / 160 / 192 /
// 256 threads, 740 groups 5.05 / 4.37 / 3.99 / 3.80 / 3.76 / 4.99 ms, 888 groups 5.39 / 4.72 / 4.36 /
// 4.17 / 4.43 / 5.34, 2,368 groups 9.4 / 10.8 / 10.0 / 11.2 / 11.4 / 11.9; where not even 64 threads
// hold them, 128 (3,000 groups: 13.9 / 12.8 / 13.4 / 13.1 / 14.5 / 16.2; in FP64 14.3 / 14.5 / 13.4 /
// 14.2 / 15.1 / 15.4).  From 1,600 buses on 64 threads are too few for a level (2,000 buses, 1,481
// groups: 32.5 / 31.8 / 32.8 / 30.8 / 30.9 / 30.9).
int default_threads(int nb, int lanes, long groups) {
    int thr = 256;
    while (thr < 1024 && 8L * thr < (long)nb * lanes && groups * 2 * thr <= 148 * 1024) thr *= 2;
    if (groups * 256 <= 148 * 1024) return thr;
    for (int t : {192, 160, 128, 96})
        if (groups <= 148 * (1024 / t)) return t;
    if (nb >= 1600) return 160;
    return groups * 64 <= 148 * 1024 ? 64 : 128;
}
// CTAs per lane group of the level-scheduled kernels, one cluster: 8 or 4 where that makes at most
// 128 CTAs (16 clusters of 8 sit on the GPCs side by side; 18 groups of a 2,000-bus grid took 2.2 ms
// with one CTA each, 2.7 ms with clusters of 8 in two waves), else 2 up to 148.  Small grids lack
// the wide levels that pay for the cluster's barriers: one scenario of 600 buses takes 757 us with
// 8 CTAs and 831 with one, 300 buses 616 and 602; two CTAs gain from 2,000 buses on (38 groups:
// 2,837 / 3,004 us; at 1,200 buses 1,820 / 1,774).  A batch that shares the GPU with concurrent ones
// (dense_fused, four of them in the benchmark's pipeline) takes two where four such batches fit:
// four parts of 16 groups each took 26.5, 26.0, 28.6 and 37.2 ms with 1, 2, 4 and 8, four of 32
// groups 42.2 and 44.6 ms with 1 and 2.
int level_ctas(int groups, int nb, int dense_fused) {
    if (dense_fused) groups *= 4;
    else if (nb >= 600)
        for (int nc : {8, 4})
            if (groups * nc <= 128) return nc;
    return nb >= 1600 && groups * 2 <= 148 ? 2 : 1;
}

int check_launch() {
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) {
        set_error(std::string("kernel launch: ") + cudaGetErrorString(e));
        return GAPK_ECUDA;
    }
    return GAPK_OK;
}

int build_graph(gapk_nr_batch b, cudaStream_t st) {
    if (b->exec && b->graph_refine == b->cur_refine) return GAPK_OK;
    if (b->exec) {
        cudaGraphExecDestroy(b->exec);
        b->exec = nullptr;
    }
    if (b->graph) {
        cudaGraphDestroy(b->graph);
        b->graph = nullptr;
    }
    GAPK_CUDA_TRY(cudaGraphCreate(&b->graph, 0));
    cudaGraphConditionalHandle h;
    GAPK_CUDA_TRY(cudaGraphConditionalHandleCreate(&h, b->graph, 1, cudaGraphCondAssignDefault));
    cudaGraphNodeParams np{};
    np.type = cudaGraphNodeTypeConditional;
    np.conditional.handle = h;
    np.conditional.type = cudaGraphCondTypeWhile;
    np.conditional.size = 1;
    cudaGraphNode_t node;
    GAPK_CUDA_TRY(cudaGraphAddNode(&node, b->graph, nullptr, 0, &np));
    cudaGraph_t body = np.conditional.phGraph_out[0];
    // capture the iteration body into the while node's graph
    cudaStream_t cs;
    GAPK_CUDA_TRY(cudaStreamCreateWithFlags(&cs, cudaStreamNonBlocking));
    cudaError_t e = cudaStreamBeginCaptureToGraph(cs, body, nullptr, nullptr, 0,
                                                  cudaStreamCaptureModeThreadLocal);
    if (e != cudaSuccess) {
        cudaStreamDestroy(cs);
        set_error(std::string("cudaStreamBeginCaptureToGraph: ") + cudaGetErrorString(e));
        return GAPK_ECUDA;
    }
    dispatch_tsw<BodyOp>(b->precision, b->sw, b, cs, 1, h);
    cudaGraph_t captured = nullptr;
    e = cudaStreamEndCapture(cs, &captured);
    cudaStreamDestroy(cs);
    if (e != cudaSuccess) {
        set_error(std::string("cudaStreamEndCapture: ") + cudaGetErrorString(e));
        return GAPK_ECUDA;
    }
    GAPK_CUDA_TRY(cudaGraphInstantiate(&b->exec, b->graph, 0));
    b->graph_refine = b->cur_refine;
    (void)st;
    return GAPK_OK;
}

int validate_inputs(gapk_nr_batch b, const gapk_nr_inputs* in) {
    if (!in || !in->d_y || !in->d_s_spec) {
        set_error("inputs: d_y and d_s_spec are required");
        return GAPK_EINVAL;
    }
    if (in->max_iterations < 0 || in->refine < 0 || in->refine > 8 ||
        (in->policy < GAPK_POLICY_REFERENCE || in->policy > GAPK_POLICY_CLAMPED)) {
        set_error("inputs: bad max_iterations / refine / policy");
        return GAPK_EINVAL;
    }
    if (in->refine > 0 && !b->A64.p) {
        set_error("inputs: refine > 0 needs a batch created with precision FP32");
        return GAPK_EINVAL;
    }
    if (!(in->refine_below >= 0.0) || !(in->reuse_below >= 0.0)) {
        set_error("inputs: refine_below and reuse_below must be >= 0");
        return GAPK_EINVAL;
    }
    if (in->reuse_below > 0.0 && in->refine < 1) {
        set_error("inputs: reuse_below > 0 needs refine >= 1");
        return GAPK_EINVAL;
    }
    return GAPK_OK;
}

// How the one-kernel loop (k_nr_small) runs this batch, with or without per-group refinement or
// reuse thresholds: lanes per CTA (0: the separate kernels are used), CTA size, whether a group's
// lanes decide together, and the shared memory share of the SM.  Shapes are ranked by waves of CTAs, then by fewer lanes per CTA (a
// lane more in a CTA lengthens every step of the level schedule), then by 256 threads over 128.
// Against the separate kernels on transmission grids of 120 to 1,200 buses it takes 1/1.6 to 1/3
// of their time while one wave holds the scenarios and 1/1.1 to 1/1.6 with two.  With three it
// still wins where an SM holds several FP32 CTAs (500 buses x 1024: 1,564 us against 1,610) or one
// FP64 CTA (900 x 300: 1,507 / 1,583), and loses with several FP64 ones (300 x 1024: 982 / 856) or
// one FP32 CTA, whose groups wait for each other across SMs (900 x 300: 1,481 / 1,365).
SmallRun small_choice(gapk_nr_batch b, bool thresholds) {
    auto const& h = b->plan->h;
    SmallRun r;
    // dense_fused asks for the separate kernels' one-CTA dense LU
    if (b->dev.lvl_ts || b->wait_test || b->dense_fused || !b->plan->dev.levels) return r;
    const size_t esz = b->precision == GAPK_PREC_FP64 ? 8 : 4;
    r.together = thresholds;
    long best_cost = 0;
    for (int cl = 1; cl <= b->sw; cl *= 2) {
        const size_t bytes = small_layout(h.n_bus, h.nb, h.n_slots, h.n_tail, h.n_levels, cl, esz).total;
        if (bytes > SMALL_SMEM_MAX) break;
        for (int thr : {256, 128}) {
            const long per_cta = (long)bytes + 2048;  // with its static and reserved shared memory
            const long per_sm = std::min<long>(1024 / thr, SMALL_SM_SMEM / per_cta);
            const long ctas = ((long)b->n_scen + cl - 1) / cl;
            const long waves = (ctas + 148 * per_sm - 1) / (148 * per_sm);
            const long cost = waves * (4 + cl);
            if (waves > ((esz == 4) == (per_sm > 1) ? 3 : 2) || (r.cl && cost >= best_cost)) continue;
            r.cl = cl;
            r.threads = thr;
            r.carveout = (int)std::min<long>(
                100, (100 * std::min(per_sm, (ctas + 147) / 148) * per_cta + SMALL_SM_SMEM - 1) / SMALL_SM_SMEM);
            best_cost = cost;
        }
    }
    r.together &= r.cl < b->sw;  // one CTA holds the whole group otherwise
    return r;
}
SmallRun small_choice(gapk_nr_batch b, const gapk_nr_inputs* in) {
    return small_choice(b, in->refine > 0 && (in->refine_below > 0.0 || in->reuse_below > 0.0));
}

template <typename T, int CL>
struct SmallOp {
    static void run(gapk_nr_batch b, SmallRun r, int refine, int passes, cudaStream_t st) {
        auto const& h = b->plan->h;
        cudaLaunchConfig_t cfg{};
        // what shared memory the launch does not need is left to L1, which holds the lists
        cudaLaunchAttribute attr[2]{};
        attr[0].id = cudaLaunchAttributePreferredSharedMemoryCarveout;
        attr[0].val.sharedMemCarveout = r.carveout;
        attr[1].id = cudaLaunchAttributeClusterDimension;
        attr[1].val.clusterDim.x = b->sw / CL;
        attr[1].val.clusterDim.y = attr[1].val.clusterDim.z = 1;
        cfg.gridDim = dim3(b->G * (b->sw / CL));
        cfg.blockDim = dim3(r.threads);
        cfg.dynamicSmemBytes =
            small_layout(h.n_bus, h.nb, h.n_slots, h.n_tail, h.n_levels, CL, sizeof(T)).total;
        cfg.stream = st;
        cfg.attrs = attr;
        cfg.numAttrs = r.together ? 2 : 1;
        cudaLaunchKernelEx(&cfg, k_nr_small<T, CL>, b->plan->dev, b->dev, refine, r.together, passes);
    }
};
// Large tails need more shared memory for their vector than a launch gets without opting in (one
// limit for every batch: the attribute is the kernel's, not the batch's).
constexpr size_t DENSE_SOLVE_SMEM_MAX = 200 * 1024;
template <typename T, int SW>
struct DenseSolveAttributesOp {
    static void run(cudaError_t* e) {
        auto set = [](auto fn) {
            return cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)DENSE_SOLVE_SMEM_MAX);
        };
        *e = set(k_dense_solve_cl<T, SW, false>);
        if (*e == cudaSuccess) *e = set(k_dense_solve_cl<T, SW, true>);
    }
};
template <typename T, int CL>
struct SmallAttributesOp {
    static void run(cudaError_t* e) {
        *e = cudaFuncSetAttribute(k_nr_small<T, CL>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                  (int)SMALL_SMEM_MAX);
    }
};

int load_inputs(gapk_nr_batch b, const gapk_nr_inputs* in, cudaStream_t st) {
    int rc = validate_inputs(b, in);
    if (rc) return rc;
    b->cur_refine = in->refine;
    b->cur_small = small_choice(b, in);
    dispatch_tsw<LoadOp>(b->precision, b->sw, b, in, st);
    return check_launch();
}

}  // namespace

extern "C" {

const char* gapk_last_error(void) { return g_err.c_str(); }
int gapk_version(void) { return 100; }
int gapk_device_count(void) {
    int n = 0;
    if (cudaGetDeviceCount(&n) != cudaSuccess) {
        cudaGetLastError();
        return 0;
    }
    return n;
}

int gapk_nr_plan_create(int n_bus, int nnz_y, const int* h_y_row_ptr, const int* h_y_col_idx,
                        const int* h_bus_type, const gapk_nr_plan_options* opt,
                        gapk_nr_plan* out) {
    TraceRange tr("gapk_nr_plan_create: ordering and symbolic analysis");
    if (!out || n_bus < 0 || nnz_y < 0 || !h_y_row_ptr || (nnz_y && !h_y_col_idx) ||
        (n_bus && !h_bus_type)) {
        set_error("gapk_nr_plan_create: bad arguments");
        return GAPK_EINVAL;
    }
    int jac = opt ? opt->jacobian_mode : GAPK_JAC_REFERENCE;
    int ord = opt ? opt->ordering : GAPK_ORDER_MINDEG;
    int dmin = opt ? opt->dense_min : 0;
    if (dmin == 0) dmin = 16;
    if ((jac != 0 && jac != 1) || (ord != 0 && ord != 1)) {
        set_error("gapk_nr_plan_create: bad options");
        return GAPK_EINVAL;
    }
    auto p = std::make_unique<gapk_nr_plan_s>();
    try {
        if (!analyze_nr(n_bus, nnz_y, h_y_row_ptr, h_y_col_idx, h_bus_type, jac, ord, dmin, p->h))
            return GAPK_EINVAL;
        p->y_row_ptr.assign(h_y_row_ptr, h_y_row_ptr + n_bus + 1);
        p->y_col.assign(h_y_col_idx, h_y_col_idx + nnz_y);
        p->a_rec = p->a_records();
    } catch (std::bad_alloc const&) {
        set_error("gapk_nr_plan_create: host allocation failed");
        return GAPK_ENOMEM;
    }
    *out = p.release();
    return GAPK_OK;
}

int gapk_nr_plan_destroy(gapk_nr_plan p) {
    delete p;
    return GAPK_OK;
}

int gapk_nr_plan_get_info(gapk_nr_plan p, gapk_nr_plan_info* info) {
    if (!p || !info) {
        set_error("gapk_nr_plan_get_info: null argument");
        return GAPK_EINVAL;
    }
    auto const& h = p->h;
    info->n_bus = h.n_bus;
    info->n_block = h.nb;
    info->n_pq = h.n_pq;
    info->n_pv = h.n_pv;
    info->n_slack = h.n_slack;
    info->n_vars = h.n_vars;
    info->nnz_y = h.nnz_y;
    info->nnz_l_blocks = h.nnz_l;
    info->n_slots = h.n_slots;
    info->n_a_blocks = h.n_a;
    info->n_levels = h.n_levels;
    info->n_pairs = h.n_pairs;
    info->n_rows_pairs = h.nnz_l;
    info->max_level_width = h.max_level_width;
    info->n_tail = h.n_tail;
    int64_t sp = 0;
    for (size_t t = 0; t + 3 < h.schur.size(); t += 4) sp += h.schur[t + 2] - h.schur[t + 1];
    info->n_schur_pairs = sp;
    return GAPK_OK;
}

int64_t gapk_nr_plan_export(gapk_nr_plan p, int what, int* h_buf) {
    if (!p) return GAPK_EINVAL;
    auto const& h = p->h;
    std::vector<int> const* v = nullptr;
    switch (what) {
        case 0: v = &h.bus_of_node; break;
        case 1: v = &h.node_pq; break;
        case 2: v = &h.lptr; break;
        case 3: v = &h.lidx; break;
        case 4: v = &h.level_ptr; break;
        case 5: v = &h.level_nodes; break;
        case 6: v = &h.slot_info; break;
        case 7: {
            // slot_src_ptr derived from slot_info
            int64_t n = h.n_slots + 1;
            if (h_buf) {
                for (int s = 0; s < h.n_slots; ++s) h_buf[s] = h.slot_info[4 * s + 2];
                h_buf[h.n_slots] = static_cast<int>(h.slot_src.size());
            }
            return n;
        }
        case 8: v = &h.slot_src; break;
        case 9: v = &h.fa_ptr; break;
        case 10: v = &h.targets; break;
        case 11: v = &h.pairs; break;
        case 12: v = &h.fb_ptr; break;
        case 13: v = &h.scale; break;
        case 14: v = &h.rptr; break;
        case 15: v = &h.rlist; break;
        case 16: v = &h.var_of_comp; break;
        case 17: v = &h.eq_of_comp; break;
        case 18: v = &h.slot_a; break;
        case 19: v = &h.arow_ptr; break;
        case 20: v = &h.arow; break;
        case 21: v = &h.schur; break;
        default:
            set_error("gapk_nr_plan_export: unknown selector");
            return GAPK_EINVAL;
    }
    if (h_buf && !v->empty()) std::memcpy(h_buf, v->data(), v->size() * sizeof(int));
    return static_cast<int64_t>(v->size());
}

int gapk_nr_batch_create(gapk_nr_plan p, int n_scen, const gapk_nr_batch_options* opt,
                         gapk_nr_batch* out) {
    TraceRange tr("gapk_nr_batch_create");
    if (!p || !out || n_scen <= 0) {
        set_error("gapk_nr_batch_create: bad arguments");
        return GAPK_EINVAL;
    }
    auto b = std::make_unique<gapk_nr_batch_s>();
    b->plan = p;
    b->n_scen = n_scen;
    b->precision = opt ? opt->precision : GAPK_PREC_FP64;
    b->y_shared = opt ? (opt->y_shared ? 1 : 0) : 1;
    int lanes = opt ? opt->lanes : 0;
    if (lanes == 0) lanes = n_scen >= 8 ? 8 : (n_scen >= 4 ? 4 : (n_scen >= 2 ? 2 : 1));
    if (lanes != 1 && lanes != 2 && lanes != 4 && lanes != 8) {
        set_error("gapk_nr_batch_create: lanes must be 1, 2, 4 or 8");
        return GAPK_EINVAL;
    }
    if (b->precision != GAPK_PREC_FP64 && b->precision != GAPK_PREC_FP32) {
        set_error("gapk_nr_batch_create: bad precision");
        return GAPK_EINVAL;
    }
    b->sw = lanes;
    int thr = opt ? opt->threads : 0;
    if (thr == 0) thr = default_threads(p->h.nb, lanes, (n_scen + lanes - 1) / lanes);
    if (thr < 32 || thr > 1024 || thr % 32) {
        set_error("gapk_nr_batch_create: threads must be a multiple of 32 in [32, 1024]");
        return GAPK_EINVAL;
    }
    b->threads = thr;
    b->use_graph = opt ? opt->use_graph : 1;
    b->dense_fused = opt ? opt->dense_fused : 0;
    int rc = p->upload();
    if (rc) return rc;
    auto const& h = p->h;
    const size_t G = (n_scen + lanes - 1) / lanes;
    b->G = static_cast<int>(G);
    b->level_ctas = level_ctas(b->G, h.nb, b->dense_fused);
    // the dense tail's solves: clusters of small CTAs, no more of them than blocks of 32 rows
    for (int nc = 8; nc > 1 && b->dense_ctas == 1; nc /= 2)
        if (!b->dense_fused && (long)G * lanes * nc <= 148 && 32 * nc <= 2 * h.n_tail + 31) b->dense_ctas = nc;
    b->split_slots = b->level_ctas >= 4 ? b->level_ctas * b->threads / lanes : 0;
    const size_t L = G * lanes;
    const size_t esz = b->precision == GAPK_PREC_FP64 ? 8 : 4;
    const size_t n = h.n_bus, nb = h.nb;
    auto A = [&](DevBuf& d, size_t bytes) {
        if (!rc) rc = d.alloc(bytes < 16 ? 16 : bytes);
    };
    A(b->V, L * n * 16);
    A(b->Sspec, L * n * 16);
    A(b->Scalc, L * n * 16);
    A(b->Y, (b->y_shared ? (size_t)h.nnz_y : L * h.nnz_y) * 16);
    A(b->F, L * (size_t)h.n_slots * 4 * esz);
    if (b->precision == GAPK_PREC_FP32) A(b->A64, L * (size_t)h.n_a * 32);
    A(b->rhs, L * nb * 16);
    A(b->dx, L * nb * 16);
    A(b->res, L * nb * 16);
    A(b->X, L * nb * 2 * esz);
    if (h.n_tail > 0) {
        // Dense-tail LU: one CTA per scenario (k_dense_lu, the panel in shared memory) when
        // there are enough scenarios to fill the GPU (or the caller says that concurrent
        // batches will, dense_fused) and the panel fits; otherwise the split kernels, which
        // spread each scenario's trailing update over many CTAs and have no shared-memory
        // limit on the tail size.
        const size_t N = 2 * (size_t)h.n_tail;
        b->dense_w = 0;
        for (int w : {32, 16, 8}) {
            size_t bytes = dense_lu_elems((int)N, w) * esz;
            if (bytes <= DENSE_LU_SMEM_MAX && (w < 32 || esz == 4 || N <= 200)) {
                b->dense_w = w;
                b->dense_smem = bytes;
                break;
            }
        }
        int dev = 0, n_sm = 148;
        if (cudaGetDevice(&dev) == cudaSuccess)
            cudaDeviceGetAttribute(&n_sm, cudaDevAttrMultiProcessorCount, dev);
        b->dense_split = b->dense_w == 0 || (L < 2 * (size_t)n_sm && !b->dense_fused);
        // FP32 tails have their trailing updates on the tensor cores unless the caller asks for
        // CUDA-core FMA: k_dense_lu_tc one CTA per scenario (panel width 32), k_dlu_update_tc
        // on the split path
        b->dense_tc = !(opt && opt->dense_fma) && b->precision == GAPK_PREC_FP32 &&
                      (b->dense_split || b->dense_w == 32);
        A(b->Dt, L * N * dense_ld((int)N) * esz);
        cudaError_t e = cudaSuccess;
        if (!b->dense_split)
            e = b->precision == GAPK_PREC_FP64
                    ? dense_lu_attributes<double>(b->dense_w, false)
                    : dense_lu_attributes<float>(b->dense_w, b->dense_tc);
        else if (b->dense_tc)
            e = split_lu_attributes();
        // dynamic + k_dense_solve_cl's 19 KB of static shared memory past the 48 KB of any launch
        const size_t vec = dense_solve_smem(h.n_tail, esz);
        if (e == cudaSuccess && vec > 28 * 1024)
            dispatch_tsw<DenseSolveAttributesOp>(b->precision, lanes, &e);
        if (e != cudaSuccess) {
            set_error(std::string("cudaFuncSetAttribute: ") + cudaGetErrorString(e));
            return GAPK_ECUDA;
        }
    }
    // (the lanes per CTA do not depend on a solve's inputs)
    if (const SmallRun r = small_choice(b.get(), false); r.cl) {
        cudaError_t e = cudaSuccess;
        dispatch_tsw<SmallAttributesOp>(b->precision, r.cl, &e);
        if (e != cudaSuccess) {
            set_error(std::string("cudaFuncSetAttribute: ") + cudaGetErrorString(e));
            return GAPK_ECUDA;
        }
    }
    A(b->mis, L * 8);
    A(b->state, L * 4);
    A(b->solving, L * 4);
    A(b->singular, L * 4);
    A(b->iters, L * 4);
    A(b->status, L * 4);
    A(b->fmis, L * 8);
    A(b->gsolve, G * 4);
    A(b->giter, G * 4);
    A(b->ctrl, 8 * 4);
    A(b->grefine, G * 4);
    A(b->gfactor, G * 4);
    A(b->tol, 24);
    if (rc) return rc;
    // per-group flags start true (any non-zero byte pattern): callers that factorise without
    // a load (the general LU) refine and refactorise as before
    GAPK_CUDA_TRY(cudaMemset(b->grefine.p, 1, b->grefine.bytes));
    GAPK_CUDA_TRY(cudaMemset(b->gfactor.p, 1, b->gfactor.bytes));
    // control words: [5] the tensor-core LU's wait error, [6] its wait test (both off)
    GAPK_CUDA_TRY(cudaMemset(b->ctrl.p, 0, b->ctrl.bytes));
    BatchDev& d = b->dev;
    d.n_scen = n_scen;
    d.n_groups = b->G;
    d.sw = lanes;
    d.y_shared = b->y_shared;
    d.V = b->V.as<double2>();
    d.Sspec = b->Sspec.as<double2>();
    d.Scalc = b->Scalc.as<double2>();
    d.Y = b->Y.as<double2>();
    d.F = b->F.p;
    d.A64 = b->A64.as<double>();
    d.rhs = b->rhs.as<double2>();
    d.dx = b->dx.as<double2>();
    d.res = b->res.as<double2>();
    d.X = b->X.p;
    d.Dt = b->Dt.p;
    d.mis_bits = b->mis.as<unsigned long long>();
    d.state = b->state.as<int>();
    d.solving = b->solving.as<int>();
    d.singular = b->singular.as<int>();
    d.iters = b->iters.as<int>();
    d.status = b->status.as<int>();
    d.final_mis = b->fmis.as<double>();
    d.gsolve = b->gsolve.as<int>();
    d.giter = b->giter.as<int>();
    d.ctrl = b->ctrl.as<int>();
    d.tol = b->tol.as<double>();
    d.grefine = b->grefine.as<int>();
    d.gfactor = b->gfactor.as<int>();
    *out = b.release();
    return GAPK_OK;
}

int gapk_nr_batch_destroy(gapk_nr_batch b) {
    delete b;
    return GAPK_OK;
}

int gapk_nr_batch_lanes(gapk_nr_batch b) { return b ? b->sw : 0; }

int64_t gapk_nr_batch_device_bytes(gapk_nr_batch b) {
    if (!b) return 0;
    int64_t s = 0;
    for (DevBuf* d : {&b->V, &b->Sspec, &b->Scalc, &b->Y, &b->F, &b->A64, &b->rhs, &b->dx,
                      &b->res, &b->X, &b->Dt, &b->mis, &b->state, &b->solving, &b->singular, &b->iters,
                      &b->status, &b->fmis, &b->gsolve, &b->giter, &b->grefine, &b->gfactor, &b->ctrl, &b->tol})
        s += static_cast<int64_t>(d->bytes);
    return s;
}

int gapk_nr_solve(gapk_nr_batch b, const gapk_nr_inputs* in, const gapk_nr_outputs* out,
                  void* stream) {
    TraceRange tr("gapk_nr_solve");
    if (!b) {
        set_error("gapk_nr_solve: null batch");
        return GAPK_EINVAL;
    }
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    int rc = load_inputs(b, in, st);
    if (rc) return rc;
    if (in->max_iterations > 0) {
        if (const SmallRun r = b->cur_small; r.cl) {
            dispatch_tsw<SmallOp>(b->precision, r.cl, b, r, in->refine, 0, st);
            rc = check_launch();
            if (rc) return rc;
        } else if (b->use_graph) {
            rc = build_graph(b, st);
            if (rc) return rc;
            GAPK_CUDA_TRY(cudaGraphLaunch(b->exec, st));
        } else {
            // host-driven loop: one synchronisation per iteration
            for (int it = 0; it < in->max_iterations; ++it) {
                dispatch_tsw<BodyOp>(b->precision, b->sw, b, st, 0,
                                     cudaGraphConditionalHandle{});
                rc = check_launch();
                if (rc) return rc;
                int any = 0;
                GAPK_CUDA_TRY(cudaMemcpyAsync(&any, b->dev.ctrl + 2, sizeof(int),
                                              cudaMemcpyDeviceToHost, st));
                GAPK_CUDA_TRY(cudaStreamSynchronize(st));
                if (!any) break;
            }
        }
    }
    if (out) {
        dispatch_tsw<StoreOp>(b->precision, b->sw, b, out, st);
        rc = check_launch();
        if (rc) return rc;
    }
    return GAPK_OK;
}

int gapk_nr_last_loop_count(gapk_nr_batch b, void* stream, int* h_loops) {
    if (!b || !h_loops) return GAPK_EINVAL;
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    GAPK_CUDA_TRY(cudaMemcpyAsync(h_loops, b->dev.ctrl + 4, sizeof(int), cudaMemcpyDeviceToHost,
                                  st));
    GAPK_CUDA_TRY(cudaStreamSynchronize(st));
    return GAPK_OK;
}

int gapk_nr_stage_load(gapk_nr_batch b, const gapk_nr_inputs* in, void* stream) {
    if (!b) return GAPK_EINVAL;
    return load_inputs(b, in, static_cast<cudaStream_t>(stream));
}

static int stage(gapk_nr_batch b, int which, void* stream) {
    if (!b) {
        set_error("stage: null batch");
        return GAPK_EINVAL;
    }
    static const char* names[] = {"gapk stage: mismatch", "gapk stage: jacobian",
                                  "gapk stage: factor", "gapk stage: solve", "gapk stage: update"};
    TraceRange tr(which >= 0 && which < 5 ? names[which] : "gapk stage");
    dispatch_tsw<StageOp>(b->precision, b->sw, b, which, static_cast<cudaStream_t>(stream));
    return check_launch();
}
int gapk_nr_stage_mismatch(gapk_nr_batch b, void* s) { return stage(b, 0, s); }
int gapk_nr_stage_jacobian(gapk_nr_batch b, void* s) { return stage(b, 1, s); }
int gapk_nr_stage_factor(gapk_nr_batch b, void* s) { return stage(b, 2, s); }
int gapk_nr_stage_solve(gapk_nr_batch b, void* s) { return stage(b, 3, s); }

int gapk_nr_stage_kernel(gapk_nr_batch b, int kernel, void* stream) {
    if (!b || kernel < 0 || kernel > 9) {
        set_error("gapk_nr_stage_kernel: bad arguments");
        return GAPK_EINVAL;
    }
    dispatch_tsw<KernelOp>(b->precision, b->sw, b, kernel, static_cast<cudaStream_t>(stream));
    return check_launch();
}

int gapk_nr_adjoint(gapk_nr_batch b, const double* d_dl_dvm, const double* d_dl_dva,
                    double* d_dl_dp, double* d_dl_dq, void* stream) {
    if (!b || !d_dl_dvm || !d_dl_dva) {
        set_error("gapk_nr_adjoint: bad arguments");
        return GAPK_EINVAL;
    }
    dispatch_tsw<AdjointOp>(b->precision, b->sw, b, d_dl_dvm, d_dl_dva, d_dl_dp, d_dl_dq,
                            static_cast<cudaStream_t>(stream));
    return check_launch();
}

int gapk_nr_adjoint_branch(gapk_nr_batch b, int n_branch, const int* d_from, const int* d_to,
                           const double* d_branch_pu, double* d_dl_dr, double* d_dl_dx,
                           void* stream) {
    if (!b || n_branch < 0 || (n_branch > 0 && (!d_from || !d_to || !d_branch_pu || !d_dl_dr ||
                                                !d_dl_dx))) {
        set_error("gapk_nr_adjoint_branch: bad arguments");
        return GAPK_EINVAL;
    }
    if (n_branch == 0) return GAPK_OK;
    dispatch_tsw<AdjBranchOp>(b->precision, b->sw, b, n_branch, d_from, d_to, d_branch_pu,
                              d_dl_dr, d_dl_dx, static_cast<cudaStream_t>(stream));
    return check_launch();
}

int gapk_nr_stage_get_correction(gapk_nr_batch b, double* d_dx, void* stream) {
    if (!b || !d_dx) return GAPK_EINVAL;
    dispatch_tsw<ToRefOp>(b->precision, b->sw, b, b->dev.dx, b->plan->var_of_comp,
                          b->plan->h.n_vars, 1.0, d_dx, static_cast<cudaStream_t>(stream));
    return check_launch();
}

int gapk_nr_stage_get_mismatch(gapk_nr_batch b, double* d_f, void* stream) {
    if (!b || !d_f) return GAPK_EINVAL;
    dispatch_tsw<ToRefOp>(b->precision, b->sw, b, b->dev.rhs, b->plan->eq_of_comp,
                          b->plan->h.n_vars, -1.0, d_f, static_cast<cudaStream_t>(stream));
    return check_launch();
}

int gapk_nr_step(gapk_nr_batch b, int* h_active, void* stream) {
    TraceRange tr("gapk_nr_step: one Newton iteration");
    if (!b || !h_active) {
        set_error("gapk_nr_step: bad arguments");
        return GAPK_EINVAL;
    }
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    if (const SmallRun r = b->cur_small; r.cl) {
        k_small_step<<<1, 256, 0, st>>>(b->dev, 0);
        dispatch_tsw<SmallOp>(b->precision, r.cl, b, r, b->cur_refine, 1, st);
        k_small_step<<<1, 256, 0, st>>>(b->dev, 1);
    } else {
        dispatch_tsw<BodyOp>(b->precision, b->sw, b, st, 0, cudaGraphConditionalHandle{});
    }
    int rc = check_launch();
    if (rc) return rc;
    GAPK_CUDA_TRY(cudaMemcpyAsync(h_active, b->dev.ctrl + 2, sizeof(int),
                                  cudaMemcpyDeviceToHost, st));
    GAPK_CUDA_TRY(cudaStreamSynchronize(st));
    return GAPK_OK;
}

int gapk_nr_get_state(gapk_nr_batch b, double* d_v, double* d_i, double* d_s, void* stream) {
    if (!b) {
        set_error("gapk_nr_get_state: null batch");
        return GAPK_EINVAL;
    }
    dispatch_tsw<StateOp>(b->precision, b->sw, b, reinterpret_cast<double2*>(d_v),
                          reinterpret_cast<double2*>(d_i), reinterpret_cast<double2*>(d_s),
                          static_cast<cudaStream_t>(stream));
    return check_launch();
}

static int64_t sparse_trace_size(gapk_nr_batch b) {
    return 3 * static_cast<int64_t>(b->G) * (b->plan->h.n_levels + 2);
}
// the panel trace exists when the one-CTA-per-scenario dense LU factorises the tail
static int64_t dense_trace_size(gapk_nr_batch b) {
    const int N = 2 * b->plan->h.n_tail;
    if (N == 0 || b->dense_split || b->dense_w <= 0) return 0;
    return static_cast<int64_t>(b->G) * b->sw * (1 + 3 * ((N + b->dense_w - 1) / b->dense_w));
}

int64_t gapk_nr_level_trace_size(gapk_nr_batch b) {
    if (!b) return 0;
    return sparse_trace_size(b) + dense_trace_size(b);
}

int gapk_nr_batch_device_error(gapk_nr_batch b) {
    if (!b || !b->ctrl.p) return 0;
    int w = 0;
    if (cudaMemcpy(&w, b->ctrl.as<int>() + 5, sizeof(int), cudaMemcpyDeviceToHost) != cudaSuccess) {
        set_error("gapk_nr_batch_device_error: cudaMemcpy failed");
        return GAPK_ECUDA;
    }
    return w ? 1 : 0;
}

int gapk_nr_batch_set_wait_test(gapk_nr_batch b, int skip) {
    if (!b || !b->ctrl.p) {
        set_error("gapk_nr_batch_set_wait_test: null batch");
        return GAPK_EINVAL;
    }
    const int v = skip ? 1 : 0;
    b->wait_test = v;
    GAPK_CUDA_TRY(cudaMemcpy(b->ctrl.as<int>() + 6, &v, sizeof(int), cudaMemcpyHostToDevice));
    return GAPK_OK;
}

int gapk_nr_dense_trace_panels(gapk_nr_batch b) {
    if (!b || dense_trace_size(b) == 0) return 0;
    const int N = 2 * b->plan->h.n_tail;
    return (N + b->dense_w - 1) / b->dense_w;
}

int gapk_nr_set_level_trace(gapk_nr_batch b, unsigned long long* d_stamps, int64_t n_stamps) {
    if (!b || (d_stamps && n_stamps < gapk_nr_level_trace_size(b))) {
        set_error("gapk_nr_set_level_trace: null batch or stamp buffer too small");
        return GAPK_EINVAL;
    }
    b->dev.lvl_ts = d_stamps;
    b->dev.dlu_ts = d_stamps && dense_trace_size(b) ? d_stamps + sparse_trace_size(b) : nullptr;
    // the solve graph holds the previous setting: rebuild it on the next gapk_nr_solve
    if (b->exec) {
        cudaGraphExecDestroy(b->exec);
        b->exec = nullptr;
    }
    if (b->graph) {
        cudaGraphDestroy(b->graph);
        b->graph = nullptr;
    }
    return GAPK_OK;
}

int gapk_nr_get_outputs(gapk_nr_batch b, const gapk_nr_outputs* out, void* stream) {
    if (!b || !out) {
        set_error("gapk_nr_get_outputs: bad arguments");
        return GAPK_EINVAL;
    }
    dispatch_tsw<StoreOp>(b->precision, b->sw, b, out, static_cast<cudaStream_t>(stream));
    return check_launch();
}

}  // extern "C"

// ===========================================================================================
// Heterogeneous batches in one graph launch: every batch's whole solve (options, load, the
// Newton loop in a device-side while node, optionally a retry loop for the scenarios that
// did not converge, results out) is one branch of a single CUDA graph; the branches share no
// edges, so the device runs them concurrently and one cudaGraphLaunch solves them all.
// ===========================================================================================
namespace gapk {
namespace {

template <typename T, int SW>
struct RetryOp {
    static void run(gapk_nr_batch b, const gapk_nr_inputs* in, int policy, int use_cond,
                    cudaGraphConditionalHandle h, cudaStream_t st) {
        PlanDev const& P = b->plan->dev;
        k_retry_flags<SW><<<1, 1024, 0, st>>>(b->dev, policy, use_cond, h);
        dim3 g(blocks_for((long)P.n_bus * SW, 256), b->G);
        k_retry_v<SW><<<g, 256, 0, st>>>(P, b->dev, reinterpret_cast<const double2*>(in->d_v_init),
                                         in->d_u_pu, in->v_init_shared);
    }
};

// Adds a while node after the capture's current dependencies on `cs` and captures the batch's
// loop body into it on `body_stream`; the capture on `cs` then continues after the node.
int add_loop(gapk_nr_batch b, cudaStream_t cs, cudaStream_t body_stream, unsigned dflt,
             cudaGraphConditionalHandle* h_out) {
    cudaStreamCaptureStatus stat;
    cudaGraph_t g = nullptr;
    const cudaGraphNode_t* deps = nullptr;
    size_t nd = 0;
    GAPK_CUDA_TRY(cudaStreamGetCaptureInfo(cs, &stat, nullptr, &g, &deps, &nd));
    if (stat != cudaStreamCaptureStatusActive) {
        set_error("mix graph: capture not active");
        return GAPK_ECUDA;
    }
    cudaGraphConditionalHandle h;
    GAPK_CUDA_TRY(cudaGraphConditionalHandleCreate(&h, g, dflt, cudaGraphCondAssignDefault));
    cudaGraphNodeParams np{};
    np.type = cudaGraphNodeTypeConditional;
    np.conditional.handle = h;
    np.conditional.type = cudaGraphCondTypeWhile;
    np.conditional.size = 1;
    std::vector<cudaGraphNode_t> dv(nd);
    for (size_t k = 0; k < nd; ++k) dv[k] = deps[k];
    cudaGraphNode_t node;
    GAPK_CUDA_TRY(cudaGraphAddNode(&node, g, dv.data(), dv.size(), &np));
    GAPK_CUDA_TRY(cudaStreamUpdateCaptureDependencies(cs, &node, 1, cudaStreamSetCaptureDependencies));
    cudaGraph_t body = np.conditional.phGraph_out[0];
    cudaError_t e = cudaStreamBeginCaptureToGraph(body_stream, body, nullptr, nullptr, 0,
                                                  cudaStreamCaptureModeThreadLocal);
    if (e != cudaSuccess) {
        set_error(std::string("mix graph body capture: ") + cudaGetErrorString(e));
        return GAPK_ECUDA;
    }
    dispatch_tsw<BodyOp>(b->precision, b->sw, b, body_stream, 1, h);
    cudaGraph_t captured = nullptr;
    GAPK_CUDA_TRY(cudaStreamEndCapture(body_stream, &captured));
    *h_out = h;
    return GAPK_OK;
}

}  // namespace
}  // namespace gapk

struct gapk_nr_mix_s {
    std::vector<gapk_nr_batch> batches;
    // the inputs / outputs the graph was built for, as bytes (the C structs are unnamed)
    std::vector<unsigned char> in_bytes, out_bytes;
    int retry = -2;
    cudaGraph_t graph = nullptr;
    cudaGraphExec_t exec = nullptr;
    cudaStream_t cs = nullptr, body = nullptr;
    ~gapk_nr_mix_s() {
        if (exec) cudaGraphExecDestroy(exec);
        if (graph) cudaGraphDestroy(graph);
        if (cs) cudaStreamDestroy(cs);
        if (body) cudaStreamDestroy(body);
    }
    int build(const gapk_nr_inputs* ins, const gapk_nr_outputs* outs, int retry_policy) {
        if (exec) cudaGraphExecDestroy(exec);
        if (graph) cudaGraphDestroy(graph);
        exec = nullptr;
        graph = nullptr;
        if (!cs) GAPK_CUDA_TRY(cudaStreamCreateWithFlags(&cs, cudaStreamNonBlocking));
        if (!body) GAPK_CUDA_TRY(cudaStreamCreateWithFlags(&body, cudaStreamNonBlocking));
        GAPK_CUDA_TRY(cudaGraphCreate(&graph, 0));
        // the branches run side by side: their groups share the SMs (ten studies of 48 groups:
        // 5.3 ms with the clusters each would have alone, 4.5 ms with two CTAs)
        int groups = 0;
        for (gapk_nr_batch b : batches) groups += b->G;
        for (size_t i = 0; i < batches.size(); ++i) {
            gapk_nr_batch b = batches[i];
            struct Shared {
                gapk_nr_batch b;
                int alone;
                ~Shared() { b->level_ctas = alone; }
            } shared{b, b->level_ctas};
            b->level_ctas = std::min(b->level_ctas, level_ctas(groups, b->plan->h.nb, 0));
            b->cur_refine = ins[i].refine;
            cudaError_t e = cudaStreamBeginCaptureToGraph(cs, graph, nullptr, nullptr, 0,
                                                          cudaStreamCaptureModeThreadLocal);
            if (e != cudaSuccess) {
                set_error(std::string("mix graph capture: ") + cudaGetErrorString(e));
                return GAPK_ECUDA;
            }
            int rc = GAPK_OK;
            dispatch_tsw<LoadOp>(b->precision, b->sw, b, &ins[i], cs);
            cudaGraphConditionalHandle h{};
            const SmallRun sm = ins[i].max_iterations > 0 ? small_choice(b, &ins[i]) : SmallRun{};
            if (sm.cl) {
                // the retry is the same kernel again: groups without a retried scenario return
                dispatch_tsw<SmallOp>(b->precision, sm.cl, b, sm, ins[i].refine, 0, cs);
                if (retry_policy >= 0) {
                    dispatch_tsw<RetryOp>(b->precision, b->sw, b, &ins[i], retry_policy, 0, h, cs);
                    dispatch_tsw<SmallOp>(b->precision, sm.cl, b, sm, ins[i].refine, 0, cs);
                }
            } else if (ins[i].max_iterations > 0) {
                rc = add_loop(b, cs, body, 1, &h);
            }
            if (!rc && !sm.cl && retry_policy >= 0 && ins[i].max_iterations > 0) {
                cudaGraphConditionalHandle r{};
                // the retry loop's condition starts false; k_retry_flags sets it
                rc = add_loop_after(b, &ins[i], retry_policy, &r);
            }
            if (!rc) dispatch_tsw<StoreOp>(b->precision, b->sw, b, &outs[i], cs);
            cudaGraph_t captured = nullptr;
            cudaError_t e2 = cudaStreamEndCapture(cs, &captured);
            if (rc) return rc;
            if (e2 != cudaSuccess) {
                set_error(std::string("mix graph capture end: ") + cudaGetErrorString(e2));
                return GAPK_ECUDA;
            }
        }
        GAPK_CUDA_TRY(cudaGraphInstantiate(&exec, graph, 0));
        in_bytes.resize(batches.size() * sizeof(gapk_nr_inputs));
        out_bytes.resize(batches.size() * sizeof(gapk_nr_outputs));
        std::memcpy(in_bytes.data(), ins, in_bytes.size());
        std::memcpy(out_bytes.data(), outs, out_bytes.size());
        retry = retry_policy;
        return GAPK_OK;
    }
    // retry: flags + start voltages (handle r, default 0), then a second loop on handle r
    int add_loop_after(gapk_nr_batch b, const gapk_nr_inputs* in, int policy,
                       cudaGraphConditionalHandle* r_out) {
        cudaStreamCaptureStatus stat;
        cudaGraph_t g = nullptr;
        GAPK_CUDA_TRY(cudaStreamGetCaptureInfo(cs, &stat, nullptr, &g, nullptr, nullptr));
        cudaGraphConditionalHandle r;
        GAPK_CUDA_TRY(cudaGraphConditionalHandleCreate(&r, g, 0, cudaGraphCondAssignDefault));
        dispatch_tsw<RetryOp>(b->precision, b->sw, b, in, policy, 1, r, cs);
        // the while node reads the condition k_retry_flags set
        cudaStreamCaptureStatus stat2;
        const cudaGraphNode_t* deps = nullptr;
        size_t nd = 0;
        GAPK_CUDA_TRY(cudaStreamGetCaptureInfo(cs, &stat2, nullptr, &g, &deps, &nd));
        cudaGraphNodeParams np{};
        np.type = cudaGraphNodeTypeConditional;
        np.conditional.handle = r;
        np.conditional.type = cudaGraphCondTypeWhile;
        np.conditional.size = 1;
        std::vector<cudaGraphNode_t> dv(nd);
    for (size_t k = 0; k < nd; ++k) dv[k] = deps[k];
        cudaGraphNode_t node;
        GAPK_CUDA_TRY(cudaGraphAddNode(&node, g, dv.data(), dv.size(), &np));
        GAPK_CUDA_TRY(cudaStreamUpdateCaptureDependencies(cs, &node, 1, cudaStreamSetCaptureDependencies));
        cudaGraph_t bg = np.conditional.phGraph_out[0];
        cudaError_t e = cudaStreamBeginCaptureToGraph(body, bg, nullptr, nullptr, 0,
                                                      cudaStreamCaptureModeThreadLocal);
        if (e != cudaSuccess) {
            set_error(std::string("mix graph retry body capture: ") + cudaGetErrorString(e));
            return GAPK_ECUDA;
        }
        dispatch_tsw<BodyOp>(b->precision, b->sw, b, body, 1, r);
        cudaGraph_t captured = nullptr;
        GAPK_CUDA_TRY(cudaStreamEndCapture(body, &captured));
        *r_out = r;
        return GAPK_OK;
    }
};

extern "C" {

int gapk_nr_mix_create(int n, const gapk_nr_batch* batches, gapk_nr_mix* out) {
    if (!out || n <= 0 || !batches) {
        set_error("gapk_nr_mix_create: bad arguments");
        return GAPK_EINVAL;
    }
    auto m = std::make_unique<gapk_nr_mix_s>();
    for (int i = 0; i < n; ++i) {
        if (!batches[i]) {
            set_error("gapk_nr_mix_create: null batch");
            return GAPK_EINVAL;
        }
        for (int j = 0; j < i; ++j)
            if (batches[j] == batches[i]) {
                set_error("gapk_nr_mix_create: a batch appears twice");
                return GAPK_EINVAL;
            }
        m->batches.push_back(batches[i]);
    }
    *out = m.release();
    return GAPK_OK;
}

int gapk_nr_mix_destroy(gapk_nr_mix m) {
    delete m;
    return GAPK_OK;
}

int gapk_nr_mix_solve(gapk_nr_mix m, const gapk_nr_inputs* in, const gapk_nr_outputs* out,
                      int retry_policy, void* stream) {
    TraceRange tr("gapk_nr_mix_solve");
    if (!m || !in || !out ||
        (retry_policy != -1 &&
         (retry_policy < GAPK_POLICY_REFERENCE || retry_policy > GAPK_POLICY_CLAMPED))) {
        set_error("gapk_nr_mix_solve: bad arguments");
        return GAPK_EINVAL;
    }
    const size_t n = m->batches.size();
    for (size_t i = 0; i < n; ++i) {
        int rc = validate_inputs(m->batches[i], &in[i]);
        if (rc) return rc;
    }
    const bool same = m->exec && m->retry == retry_policy &&
                      m->in_bytes.size() == n * sizeof(gapk_nr_inputs) &&
                      std::memcmp(m->in_bytes.data(), in, m->in_bytes.size()) == 0 &&
                      std::memcmp(m->out_bytes.data(), out, m->out_bytes.size()) == 0;
    if (!same) {
        int rc = m->build(in, out, retry_policy);
        if (rc) return rc;
    }
    GAPK_CUDA_TRY(cudaGraphLaunch(m->exec, static_cast<cudaStream_t>(stream)));
    return GAPK_OK;
}

}  // extern "C"

// ===========================================================================================
// General sparse LU (ILUSolver): complex a + jb handled as the 2x2 real block [a -b; b a], so
// the Newton engine's analysis, level-scheduled factor, dense tail and solves are reused.
// ===========================================================================================
namespace gapk {

__global__ void k_cfill(PlanDev P, BatchDev B, const double2* __restrict__ vals,
                        const int* __restrict__ val_map) {
    const int a_idx = blockIdx.x * blockDim.x + threadIdx.x;
    if (a_idx >= P.n_a) return;
    const int slot = P.a_slots[a_idx];
    const int4 si = P.slot_info[slot];
    double re = 0.0, im = 0.0;
    for (int e = si.z; e < si.w; ++e) {
        const double2 v = vals[val_map[P.slot_src[e]]];
        re += v.x;
        im += v.y;
    }
    stb(reinterpret_cast<Blk<double>*>(B.F) + slot, Blk<double>{re, -im, im, re});
}

__global__ void k_crhs(int nb, const int* __restrict__ bus_of_node, const int* __restrict__ rp,
                       const double2* __restrict__ b, double2* rhs) {
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k < nb) rhs[k] = b[rp[bus_of_node[k]]];
}

__global__ void k_csol(int nb, const int* __restrict__ bus_of_node, const double2* __restrict__ x,
                       double2* out) {
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k < nb) out[bus_of_node[k]] = x[k];
}

}  // namespace gapk

struct gapk_splu_s {
    gapk_nr_plan_s plan;
    std::vector<int> rp, val_map;
    gapk_nr_batch batch = nullptr;
    DevBuf d_valmap, d_rp, d_bon;
    bool factorized = false;
    ~gapk_splu_s() {
        if (batch) gapk_nr_batch_destroy(batch);
    }
    int ready() {
        if (batch) return GAPK_OK;
        gapk_nr_batch_options o{GAPK_PREC_FP64, 1, 1, 512, 0};
        int rc = gapk_nr_batch_create(&plan, 1, &o, &batch);
        if (rc) return rc;
        rc = d_valmap.upload(val_map);
        if (!rc) rc = d_rp.upload(rp);
        if (!rc) rc = d_bon.upload(plan.h.bus_of_node);
        return rc;
    }
};

extern "C" {

int gapk_splu_create(int n, int nnz, const int* h_row_ptr, const int* h_col_idx,
                     gapk_splu* out) {
    if (!out || !h_row_ptr || (nnz > 0 && !h_col_idx)) {
        set_error("gapk_splu_create: bad arguments");
        return GAPK_EINVAL;
    }
    auto s = std::make_unique<gapk_splu_s>();
    s->plan.general = true;
    try {
        if (!analyze_general(n, nnz, h_row_ptr, h_col_idx, 16, s->plan.h, s->rp, s->val_map))
            return GAPK_EINVAL;
    } catch (std::bad_alloc const&) {
        set_error("gapk_splu_create: host allocation failed");
        return GAPK_ENOMEM;
    }
    // the plan's "Y" pattern is the row-permuted matrix
    s->plan.y_row_ptr.assign(n + 1, 0);
    s->plan.y_col.clear();
    for (int i = 0; i < n; ++i) {
        const int r = s->rp[i];
        for (int p = h_row_ptr[r]; p < h_row_ptr[r + 1]; ++p) s->plan.y_col.push_back(h_col_idx[p]);
        s->plan.y_row_ptr[i + 1] = static_cast<int>(s->plan.y_col.size());
    }
    *out = s.release();
    return GAPK_OK;
}

int gapk_splu_destroy(gapk_splu s) {
    delete s;
    return GAPK_OK;
}

int gapk_splu_factorize(gapk_splu s, const double* d_values, void* stream) {
    if (!s || !d_values) {
        set_error("gapk_splu_factorize: bad arguments");
        return GAPK_EINVAL;
    }
    s->factorized = false;
    int rc = s->ready();
    if (rc) return rc;
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    gapk_nr_batch b = s->batch;
    const int one[2] = {1, 0};
    GAPK_CUDA_TRY(cudaMemcpyAsync(b->dev.gsolve, one, sizeof(int), cudaMemcpyHostToDevice, st));
    GAPK_CUDA_TRY(cudaMemcpyAsync(b->dev.solving, one, sizeof(int), cudaMemcpyHostToDevice, st));
    GAPK_CUDA_TRY(cudaMemcpyAsync(b->dev.singular, one + 1, sizeof(int), cudaMemcpyHostToDevice, st));
    PlanDev const& P = s->plan.dev;
    k_cfill<<<blocks_for((long)P.n_a, 256), 256, 0, st>>>(
        P, b->dev, reinterpret_cast<const double2*>(d_values), s->d_valmap.as<int>());
    launch_factor<double, 1>(b, st);
    rc = check_launch();
    if (rc) return rc;
    int sing = 0;
    GAPK_CUDA_TRY(cudaMemcpyAsync(&sing, b->dev.singular, sizeof(int), cudaMemcpyDeviceToHost, st));
    GAPK_CUDA_TRY(cudaStreamSynchronize(st));
    if (sing) {
        set_error("gapk_splu_factorize: pivot below 1e-14 (numerically singular under static "
                  "pivoting)");
        return GAPK_ESINGULAR;
    }
    s->factorized = true;
    return GAPK_OK;
}

int gapk_splu_solve(gapk_splu s, const double* d_rhs, double* d_x, void* stream) {
    if (!s || !d_rhs || !d_x) {
        set_error("gapk_splu_solve: bad arguments");
        return GAPK_EINVAL;
    }
    if (!s->factorized) {
        set_error("gapk_splu_solve: matrix not factorized");
        return GAPK_ESTATE;
    }
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    gapk_nr_batch b = s->batch;
    const int nb = s->plan.h.nb;
    k_crhs<<<blocks_for(nb, 256), 256, 0, st>>>(nb, s->d_bon.as<int>(), s->d_rp.as<int>(),
                                                  reinterpret_cast<const double2*>(d_rhs),
                                                  b->dev.rhs);
    launch_solve<double, 1>(b, st, b->dev.rhs, b->dev.dx, 0);
    k_csol<<<blocks_for(nb, 256), 256, 0, st>>>(nb, s->d_bon.as<int>(), b->dev.dx,
                                                  reinterpret_cast<double2*>(d_x));
    return check_launch();
}

int gapk_splu_size(gapk_splu s) { return s ? s->plan.h.nb : GAPK_EINVAL; }

}  // extern "C"

// ===========================================================================================
// Allocation-free single-scenario solve.
//
// Some callers cannot call cudaMalloc at solve time: hosts that hand out device memory only
// from their own pools, and real-time loops that must not touch the allocator (cudaMalloc and
// cudaFree can block on the whole device).  gapk_nr_solve_noalloc serves them: it solves one
// scenario in FP64 with the same kernels as gapk_nr_solve, but every buffer it needs (a copy
// of the plan's index lists and the whole Newton state) is carved out of one file-scope device
// array of fixed size.  The caller passes only inputs and outputs.
// ===========================================================================================
namespace {

constexpr size_t kNoAllocScratchBytes = size_t(32) << 20;  // 32 MiB, held by every device
                                                             // that loads the library
static __device__ __align__(256) unsigned char g_noalloc_scratch[kNoAllocScratchBytes];

constexpr int kMaxDevices = 64;
std::mutex g_noalloc_mutex;
void* g_noalloc_ptr[kMaxDevices] = {};

// Device address of g_noalloc_scratch on the current device.  In host code the array's name
// is only a host-side stand-in, so the address must come from cudaGetSymbolAddress, once per
// device, with that device current.
int noalloc_scratch_ptr(void** out) {
    int dev = 0;
    GAPK_CUDA_TRY(cudaGetDevice(&dev));
    if (dev < 0 || dev >= kMaxDevices) {
        set_error("gapk_nr_solve_noalloc: device index out of range");
        return GAPK_EINVAL;
    }
    std::lock_guard<std::mutex> lock(g_noalloc_mutex);
    if (!g_noalloc_ptr[dev]) {
        void* p = nullptr;
        GAPK_CUDA_TRY(cudaGetSymbolAddress(&p, g_noalloc_scratch));
        for (int w : {32, 16, 8})
            GAPK_CUDA_TRY(dense_lu_attributes<double>(w, false));
        g_noalloc_ptr[dev] = p;
    }
    *out = g_noalloc_ptr[dev];
    return GAPK_OK;
}

struct Carver {
    size_t off = 0;
    size_t take(size_t bytes) {
        size_t o = off;
        off += (bytes + 255) & ~size_t(255);
        return o;
    }
};

}  // namespace

extern "C" int gapk_nr_solve_noalloc(gapk_nr_plan p, const gapk_nr_inputs* in,
                                     const gapk_nr_outputs* out, void* stream) {
    if (!p || !in || !in->d_y || !in->d_s_spec) {
        set_error("gapk_nr_solve_noalloc: plan, d_y and d_s_spec are required");
        return GAPK_EINVAL;
    }
    if (in->max_iterations < 0 || in->refine != 0 ||
        (in->policy < GAPK_POLICY_REFERENCE || in->policy > GAPK_POLICY_CLAMPED)) {
        set_error("gapk_nr_solve_noalloc: bad max_iterations / policy, or refine != 0 "
                  "(this entry point solves in FP64 only)");
        return GAPK_EINVAL;
    }
    auto const& h = p->h;
    const size_t n = h.n_bus, nb = h.nb, nnz = h.nnz_y, N = 2 * (size_t)h.n_tail;
    // plan index lists copied into the scratch, in this order
    std::vector<int> const* lists[] = {&p->y_row_ptr, &p->y_col, &h.bus_type, &h.node_of_bus,
                                       &h.slot_info, &h.slot_src, &h.level_ptr,
                                       &h.fa_ptr, &h.targets, &h.pairs,
                                       &h.fb_ptr, &h.scale, &h.lptr, &h.lidx, &h.rptr,
                                       &h.rlist, &h.schur, &p->a_rec};
    constexpr int kLists = sizeof(lists) / sizeof(lists[0]);
    Carver c;
    size_t loff[kLists];
    for (int i = 0; i < kLists; ++i) loff[i] = c.take(lists[i]->size() * sizeof(int));
    const size_t oV = c.take(n * 16), oS = c.take(n * 16), oSc = c.take(n * 16),
                 oY = c.take(nnz * 16), oF = c.take((size_t)h.n_slots * 32),
                 oRhs = c.take(nb * 16), oDx = c.take(nb * 16), oRes = c.take(nb * 16),
                 oX = c.take(nb * 16), oDt = c.take(N * dense_ld((int)N) * 8), oMis = c.take(8),
                 oState = c.take(4), oSolv = c.take(4), oSing = c.take(4), oIt = c.take(4),
                 oSt = c.take(4), oFm = c.take(8), oGs = c.take(4), oGi = c.take(4),
                 oCtrl = c.take(8 * 4), oTol = c.take(8);
    if (c.off > kNoAllocScratchBytes) {
        set_error("gapk_nr_solve_noalloc: this grid needs " + std::to_string(c.off) +
                  " bytes of working memory; the static scratch holds " +
                  std::to_string(kNoAllocScratchBytes) + " bytes (32 MiB)");
        return GAPK_ERANGE;
    }
    size_t dense_smem = 0;
    int dense_w = 0;
    if (h.n_tail > 0) {
        // the panel width rule of gapk_nr_batch_create for FP64 tails
        for (int w : {32, 16, 8}) {
            size_t bytes = dense_lu_elems((int)N, w) * 8;
            if (bytes <= DENSE_LU_SMEM_MAX && (w < 32 || N <= 200)) {
                dense_w = w;
                dense_smem = bytes;
                break;
            }
        }
        if (!dense_w) {
            set_error("gapk_nr_solve_noalloc: dense tail exceeds the shared-memory panel limit");
            return GAPK_ERANGE;
        }
    }
    void* base = nullptr;
    int rc = noalloc_scratch_ptr(&base);
    if (rc) return rc;
    unsigned char* B0 = static_cast<unsigned char*>(base);
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    for (int i = 0; i < kLists; ++i)
        if (!lists[i]->empty())
            GAPK_CUDA_TRY(cudaMemcpyAsync(B0 + loff[i], lists[i]->data(),
                                          lists[i]->size() * sizeof(int),
                                          cudaMemcpyHostToDevice, st));
    auto L = [&](int i) { return reinterpret_cast<const int*>(B0 + loff[i]); };
    PlanDev P{};
    P.n_bus = h.n_bus;
    P.nb = h.nb;
    P.nnz_y = h.nnz_y;
    P.n_slots = h.n_slots;
    P.nnz_l = h.nnz_l;
    P.n_levels = h.n_levels;
    P.n_a = h.n_a;
    P.jac_mode = h.jac_mode;
    P.ns = h.ns;
    P.n_tail = h.n_tail;
    P.n_schur = static_cast<int>(h.schur.size() / 4);
    P.y_row_ptr = L(0);
    P.y_col = L(1);
    P.bus_type = L(2);
    P.node_of_bus = L(3);
    P.slot_info = reinterpret_cast<const int4*>(L(4));
    P.slot_src = L(5);
    P.level_ptr = L(6);
    P.fa_ptr = L(7);
    P.targets = reinterpret_cast<const int4*>(L(8));
    P.pairs = reinterpret_cast<const int2*>(L(9));
    P.fb_ptr = L(10);
    P.scale = reinterpret_cast<const int2*>(L(11));
    P.lptr = L(12);
    P.lidx = L(13);
    P.rptr = L(14);
    P.rlist = reinterpret_cast<const int2*>(L(15));
    P.schur = reinterpret_cast<const int4*>(L(16));
    P.a_rec = reinterpret_cast<const int4*>(L(17));
    BatchDev D{};
    D.n_scen = 1;
    D.n_groups = 1;
    D.sw = 1;
    D.y_shared = 1;
    D.V = reinterpret_cast<double2*>(B0 + oV);
    D.Sspec = reinterpret_cast<double2*>(B0 + oS);
    D.Scalc = reinterpret_cast<double2*>(B0 + oSc);
    D.Y = reinterpret_cast<double2*>(B0 + oY);
    D.F = B0 + oF;
    D.A64 = nullptr;
    D.rhs = reinterpret_cast<double2*>(B0 + oRhs);
    D.dx = reinterpret_cast<double2*>(B0 + oDx);
    D.res = reinterpret_cast<double2*>(B0 + oRes);
    D.X = B0 + oX;
    D.Dt = B0 + oDt;
    D.mis_bits = reinterpret_cast<unsigned long long*>(B0 + oMis);
    D.state = reinterpret_cast<int*>(B0 + oState);
    D.solving = reinterpret_cast<int*>(B0 + oSolv);
    D.singular = reinterpret_cast<int*>(B0 + oSing);
    D.iters = reinterpret_cast<int*>(B0 + oIt);
    D.status = reinterpret_cast<int*>(B0 + oSt);
    D.final_mis = reinterpret_cast<double*>(B0 + oFm);
    D.gsolve = reinterpret_cast<int*>(B0 + oGs);
    D.giter = reinterpret_cast<int*>(B0 + oGi);
    D.ctrl = reinterpret_cast<int*>(B0 + oCtrl);
    D.tol = reinterpret_cast<double*>(B0 + oTol);
    // control words and state start fresh on every call (the scratch keeps the last call's)
    int ctrl[8] = {0, in->max_iterations, 1, in->policy, 0, 0, 0, 0};
    GAPK_CUDA_TRY(cudaMemcpyAsync(D.ctrl, ctrl, sizeof(ctrl), cudaMemcpyHostToDevice, st));
    double tol = in->tolerance;
    GAPK_CUDA_TRY(cudaMemcpyAsync(D.tol, &tol, sizeof(double), cudaMemcpyHostToDevice, st));
    k_load<1><<<blocks_for((long)n, 256), 256, 0, st>>>(
        P, D, reinterpret_cast<const double2*>(in->d_y),
        reinterpret_cast<const double2*>(in->d_s_spec),
        reinterpret_cast<const double2*>(in->d_v_init), in->d_u_pu, 0, SolveOpts{});
    rc = check_launch();
    if (rc) return rc;
    const int thr = 512;
    for (int it = 0; it < in->max_iterations; ++it) {
        k_mismatch<1><<<mismatch_grid<1>(P, 1), 256, 0, st>>>(P, D);
        k_check<1><<<1, 1024, 0, st>>>(D, 0, cudaGraphConditionalHandle{});
        k_jfill<double, 1><<<blocks_for((long)h.n_a, 256), 256, 0, st>>>(P, D);
        k_factor<double, 1, false><<<1, thr, 0, st>>>(P, D, 0);
        if (h.n_tail > 0) {
            k_schur<double, 1><<<blocks_for((long)P.n_schur, 256), 256, 0, st>>>(P, D);
            launch_dense_lu<double>(dense_w, 1, dense_smem, st, D, (int)N, false);
        }
        k_solve_fwd<double, 1, false><<<1, thr, 0, st>>>(P, D, D.rhs, 0);
        if (h.n_tail > 0)
            k_dense_solve<double, 1><<<1, 256, dense_solve_smem(P.n_tail, sizeof(double)), st>>>(P, D, D.dx, 0);
        k_solve_bwd<double, 1, false><<<1, thr, 0, st>>>(P, D, D.dx, 0);
        k_update<1><<<blocks_for((long)n, 256), 256, 0, st>>>(P, D);
        rc = check_launch();
        if (rc) return rc;
        int any = 0;
        GAPK_CUDA_TRY(cudaMemcpyAsync(&any, D.ctrl + 2, sizeof(int), cudaMemcpyDeviceToHost, st));
        GAPK_CUDA_TRY(cudaStreamSynchronize(st));
        if (!any) break;
    }
    if (out) {
        k_store<1><<<blocks_for((long)n, 256), 256, 0, st>>>(
            P, D, reinterpret_cast<double2*>(out->d_v), out->d_iterations, out->d_status,
            out->d_final_mismatch);
        rc = check_launch();
        if (rc) return rc;
    }
    // the outputs are read from the shared scratch: wait for them, so that a later call from
    // this thread (on any stream) cannot overwrite the scratch before they are written
    GAPK_CUDA_TRY(cudaStreamSynchronize(st));
    return GAPK_OK;
}

// NVTX range helper of internal.h
gapk::TraceRange::TraceRange(const char* name) { nvtxRangePushA(name); }
gapk::TraceRange::~TraceRange() { nvtxRangePop(); }
