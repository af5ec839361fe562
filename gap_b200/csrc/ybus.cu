// Y-bus value assembly on the device and the gapk_ybus_* C ABI.
//
// One thread per (scenario, CSR slot), whole rows per CTA.  An off-diagonal slot holds the stamp
// of the one branch triplet that produced it; a diagonal slot sums its bus's shunt and branch-end
// stamps sequentially in the reference's accumulation order (shunts in appliance order, then
// branch ends in branch order), so the result is deterministic and, in reference mode,
// bit-identical to src/admittance/cpu/cpu_admittance_matrix.cpp:88-145.  No floating atomics.
//
// All reference-mode arithmetic uses explicitly rounded intrinsics (__dmul_rn, __dadd_rn,
// __ddiv_rn) so that no multiply-add is contracted into an FMA: the reference computes
// r*r + x*x with two roundings.
#include <cuda_runtime.h>

#include <algorithm>
#include <memory>
#include <new>
#include <string>
#include <utility>
#include <vector>

#include "../../include/gapk.h"
#include "internal.h"

namespace gapk {
namespace {

struct Stamps {
    double2 ff, tt, ft, tf;
};

// Untapped stamps of one branch: y = 1 / (r + jx) and the end stamp e = y + g1 + j b1/2
// (cpu_admittance_matrix.cpp:130-135).
struct SeriesStamp {
    double yr, yi, er, ei;
};
__device__ __forceinline__ SeriesStamp series_stamp(double r, double x, double g, double b) {
    const double z2 = __dadd_rn(__dmul_rn(r, r), __dmul_rn(x, x));
    SeriesStamp s = {0.0, 0.0, 0.0, 0.0};
    if (z2 > 1e-12) {
        s.yr = __ddiv_rn(r, z2);
        s.yi = __ddiv_rn(-x, z2);
    }
    s.er = __dadd_rn(__dadd_rn(s.yr, g), 0.0);
    s.ei = __dadd_rn(__dadd_rn(s.yi, 0.0), __dmul_rn(b, 0.5));  // b / 2, exact either way
    return s;
}
__device__ __forceinline__ bool is_tapped(int mode, double k, double th) {
    return mode != GAPK_YBUS_REFERENCE && !(k == 1.0 && th == 0.0);
}
// The branch's stamps with the tap t = k e^{j th} on the from side: Y_ff = (y+ysh)/k^2,
// Y_ft = -y/conj(t) = -y t / k^2, Y_tf = -y/t = -y conj(t) / k^2, Y_tt = y+ysh.
__device__ __forceinline__ Stamps tapped_stamps(SeriesStamp const& q, double k, double th) {
    double sn, cs;
    sincos(th, &sn, &cs);
    const double k2 = k * k;
    const double tr = k * cs, ti = k * sn;
    Stamps s;
    s.ff = make_double2(q.er / k2, q.ei / k2);
    s.tt = make_double2(q.er, q.ei);
    s.ft = make_double2(-(q.yr * tr - q.yi * ti) / k2, -(q.yr * ti + q.yi * tr) / k2);
    s.tf = make_double2(-(q.yr * tr + q.yi * ti) / k2, -(q.yi * tr - q.yr * ti) / k2);
    return s;
}
__device__ __forceinline__ Stamps branch_stamps(const double* __restrict__ br, int mode) {
    const SeriesStamp q = series_stamp(br[0], br[1], br[2], br[3]);
    if (is_tapped(mode, br[4], br[5])) return tapped_stamps(q, br[4], br[5]);
    Stamps s;
    s.ff = make_double2(q.er, q.ei);
    s.tt = s.ff;
    s.ft = make_double2(-q.yr, -q.yi);
    s.tf = s.ft;
    return s;
}

// Columns c, c + 1 of a branch row: one 16-byte load when every row starts on one (VEC).
template <bool VEC>
__device__ __forceinline__ double2 row_pair(const double* __restrict__ row, int c) {
    if constexpr (VEC) return *reinterpret_cast<const double2*>(row + c);
    return make_double2(row[c], row[c + 1]);
}

// One CTA per run of whole rows of at most YB_SLOTS slots and NS scenarios, one thread per
// slot.  Every off-diagonal slot is one end of one branch: its thread computes the branch's
// stamps once per scenario and leaves the end's diagonal stamp in shared memory, where the
// diagonal slot's thread sums its row's ends in the reference's order (diag_pos: the slot each
// end's stamp sits in, or -(s + 1) for shunt s).  Tapped branches (a sine, a cosine and four more
// divisions) are collected first, from all the CTA's scenarios, and worked off by consecutive
// threads, so that a warp with one of them does not carry its 31 plain neighbours through that
// code and the CTA waits for it once per NS scenarios.
// Bound by the L1 wavefronts of the 48-byte row gathers (67 % busy; FP64 pipe 16 %, DRAM 25 %).
// 512 scenarios x 38,000 slots (0.66 GB compulsory), with taps / without: 669 / 479 us with the
// stamps recomputed for every slot and diagonal term, 467 / 350 with one scenario per CTA, 362 /
// 287 with four; the off-diagonal values kept in registers instead of `val` spill (401 / 297).
// NS is 4 where that still leaves the GPU several waves of CTAs, 1 up to YB_FEW of those: there a
// CTA's own chain is the time.  With taps, one scenario of 50 / 1,000 / 10,000 / 30,000 buses 5.5 /
// 6.4 / 7.1 / 10.5 us with NS = 4, 3.9 / 4.5 / 4.6 / 5.8 with 1; 3,000 buses x 16 (736 CTAs) 9.0 / 6.8,
// 1,000 x 64 (1,024) 9.4 / 9.4, 10,000 x 12 (1,824) 12.2 / 14.3.
constexpr int YB_SLOTS = 256, YB_SCEN = 4, YB_FEW = 1024;

template <bool VEC, int NS>
__global__ void __launch_bounds__(YB_SLOTS)
    k_ybus(int n_scen, int n_tiles, const int* __restrict__ tile_slot, const int* __restrict__ slot_src,
           const int* __restrict__ diag_ptr, const int* __restrict__ diag_src,
           const int* __restrict__ diag_pos, const double* __restrict__ br, long long br_stride,
           const double* __restrict__ sh, long long sh_stride, int mode, double scale,
           double2* __restrict__ out, long long out_stride) {
    __shared__ double2 val[NS][YB_SLOTS], end[NS][YB_SLOTS];
    __shared__ short tapped[NS * YB_SLOTS];  // scenario << 8 | slot
    __shared__ int n_tapped;
    const int tile = blockIdx.x % n_tiles;
    const int s0 = (blockIdx.x / n_tiles) * NS, s1 = min(n_scen, s0 + NS);
    const int p0 = tile_slot[tile], cnt = tile_slot[tile + 1] - p0;
    const int t = threadIdx.x;
    const bool taps = mode != GAPK_YBUS_REFERENCE;
    auto put = [&](int s, int p, double2 v) {
        if (scale != 1.0) v = make_double2(__dmul_rn(v.x, scale), __dmul_rn(v.y, scale));
        out[(size_t)s * out_stride + p0 + p] = v;
    };
    if (cnt > YB_SLOTS) {
        // a single row longer than the tile: every end of its bus recomputed for the diagonal
        for (int s = s0; s < s1; ++s) {
            const double* B = br + (size_t)s * br_stride;
            const double* S = sh + (size_t)s * sh_stride;
            for (int p = t; p < cnt; p += YB_SLOTS) {
                const int src = slot_src[p0 + p];
                double2 v = make_double2(0.0, 0.0);
                if (src >= 0) {
                    const Stamps st = branch_stamps(B + (size_t)(src >> 1) * 6, mode);
                    v = (src & 1) ? st.tf : st.ft;
                } else {
                    for (int c = diag_ptr[-src - 1]; c < diag_ptr[-src]; ++c) {
                        const int d = diag_src[c];
                        double2 a;
                        if (d < 0) {
                            a = make_double2(S[(size_t)(-d - 1) * 2], S[(size_t)(-d - 1) * 2 + 1]);
                        } else {
                            const Stamps st = branch_stamps(B + (size_t)(d >> 1) * 6, mode);
                            a = (d & 1) ? st.tt : st.ff;
                        }
                        v = make_double2(__dadd_rn(v.x, a.x), __dadd_rn(v.y, a.y));
                    }
                }
                put(s, p, v);
            }
        }
        return;
    }
    if (t == 0) n_tapped = 0;
    const int src = t < cnt ? slot_src[p0 + t] : 0;
    __syncthreads();
    if (t < cnt && src >= 0) {
        const double* row = br + (size_t)(src >> 1) * 6;
        double2 rx[NS], gb[NS], kt[NS];
#pragma unroll
        for (int k = 0; k < NS; ++k) {
            const double* q = row + (size_t)min(s0 + k, s1 - 1) * br_stride;
            rx[k] = row_pair<VEC>(q, 0);
            gb[k] = row_pair<VEC>(q, 2);
            if (taps) kt[k] = row_pair<VEC>(q, 4);
        }
#pragma unroll
        for (int k = 0; k < NS; ++k) {
            const SeriesStamp q = series_stamp(rx[k].x, rx[k].y, gb[k].x, gb[k].y);
            end[k][t] = make_double2(q.er, q.ei);
            val[k][t] = make_double2(-q.yr, -q.yi);
            if (taps && is_tapped(mode, kt[k].x, kt[k].y))
                tapped[atomicAdd(&n_tapped, 1)] = (short)(k << 8 | t);
        }
    }
    __syncthreads();
    if (taps) {
        for (int j = t; j < n_tapped; j += YB_SLOTS) {
            const int k = tapped[j] >> 8, p = tapped[j] & 255, ps = slot_src[p0 + p];
            const double* q = br + (size_t)min(s0 + k, s1 - 1) * br_stride + (size_t)(ps >> 1) * 6;
            const double2 kt = row_pair<VEC>(q, 4);
            const Stamps st = tapped_stamps({-val[k][p].x, -val[k][p].y, end[k][p].x, end[k][p].y}, kt.x, kt.y);
            end[k][p] = (ps & 1) ? st.tt : st.ff;
            val[k][p] = (ps & 1) ? st.tf : st.ft;
        }
        __syncthreads();
    }
    if (t >= cnt) return;
    if (src >= 0) {
#pragma unroll
        for (int k = 0; k < NS; ++k)
            if (s0 + k < s1) put(s0 + k, t, val[k][t]);
        return;
    }
    double2 v[NS];
#pragma unroll
    for (int k = 0; k < NS; ++k) v[k] = make_double2(0.0, 0.0);
    for (int c = diag_ptr[-src - 1]; c < diag_ptr[-src]; ++c) {
        const int d = diag_pos[c];
#pragma unroll
        for (int k = 0; k < NS; ++k) {
            double2 a;
            if (d >= 0) {
                a = end[k][d - p0];
            } else {
                const double* S = sh + (size_t)min(s0 + k, s1 - 1) * sh_stride + (size_t)(-d - 1) * 2;
                a = make_double2(S[0], S[1]);
            }
            v[k] = make_double2(__dadd_rn(v[k].x, a.x), __dadd_rn(v[k].y, a.y));
        }
    }
#pragma unroll
    for (int k = 0; k < NS; ++k)
        if (s0 + k < s1) put(s0 + k, t, v[k]);
}

// Branch status changes on existing values, one thread per (scenario, touched CSR slot).
// Each thread applies the deltas of its slot in change order, so the result of every slot is
// the one the reference's sequential loop gives (src/admittance/cpu/cpu_admittance_matrix.cpp:
// 214-297: different slots never interact), whatever the number of threads.
//   item  = (scenario, slot, first, last) into seg; seg[e] = change index << 2 | role, role
//           0 / 1 the from / to diagonal, 2 the (from, to) entry, 3 the (to, from) entry
//   prm   = (r1, x1, g1, b1, k, theta, status) per change, Ohm / S
// Delta of one change (sign + when the branch comes into service, - when it leaves):
//   GAPK_DELTA_REFERENCE   the reference's update: diagonals y + g1 + j b1 + j b1/2 (unlike its
//                          build, which stamps y + g1 + j b1/2), off-diagonals -y; taps ignored
//   GAPK_DELTA_FIXED       the builder's own stamps, taps ignored (GAPK_YBUS_REFERENCE)
//   GAPK_DELTA_FIXED_TAPS  the builder's pi-model stamps with the tap (GAPK_YBUS_TAPS)
// scale multiplies every delta (1 = Siemens, Z_base = per unit).
__device__ __forceinline__ double2 change_delta(const double* __restrict__ q, int role, int mode) {
    double2 d;
    if (mode == GAPK_DELTA_REFERENCE) {
        const double r = q[0], x = q[1], g = q[2], b = q[3];
        const double z2 = __dadd_rn(__dmul_rn(r, r), __dmul_rn(x, x));
        double yr = 0.0, yi = 0.0;
        if (z2 > 1e-12) {
            yr = __ddiv_rn(r, z2);
            yi = __ddiv_rn(-x, z2);
        }
        if (role < 2) {
            // (y + (g1 + j b1)) + j b1/2, each sum rounded as the reference's complex adds
            d = make_double2(__dadd_rn(__dadd_rn(yr, g), 0.0),
                             __dadd_rn(__dadd_rn(yi, b), __ddiv_rn(b, 2.0)));
        } else {
            d = make_double2(-yr, -yi);
        }
    } else {
        const Stamps st = branch_stamps(q, mode == GAPK_DELTA_FIXED ? GAPK_YBUS_REFERENCE
                                                                    : GAPK_YBUS_TAPS);
        d = role == 0 ? st.ff : role == 1 ? st.tt : role == 2 ? st.ft : st.tf;
    }
    if (q[6] == 0.0) d = make_double2(-d.x, -d.y);
    return d;
}

__global__ void k_ybus_delta(int n_items, const int4* __restrict__ items,
                             const int* __restrict__ seg, const double* __restrict__ prm,
                             int mode, double scale, double2* __restrict__ values,
                             long long stride) {
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= n_items) return;
    const int4 it = items[t];
    double2* v = values + (size_t)it.x * stride + it.y;
    double vr = v->x, vi = v->y;
    for (int e = it.z; e < it.w; ++e) {
        const int c = seg[e] >> 2, role = seg[e] & 3;
        double2 d = change_delta(prm + (size_t)c * 7, role, mode);
        if (scale != 1.0) d = make_double2(__dmul_rn(d.x, scale), __dmul_rn(d.y, scale));
        if (mode == GAPK_DELTA_REFERENCE && role >= 2) {
            // values[idx] -= series change: -(+-y)
            vr = __dsub_rn(vr, -d.x);
            vi = __dsub_rn(vi, -d.y);
        } else {
            vr = __dadd_rn(vr, d.x);
            vi = __dadd_rn(vi, d.y);
        }
    }
    *v = make_double2(vr, vi);
}

}  // namespace
}  // namespace gapk

using namespace gapk;

struct gapk_ybus_s {
    YbusPatternHost h;
    int device = -1;
    std::vector<int> tile_slot;  // first slot of each CTA's run of rows, then nnz
    std::vector<int> diag_pos;   // diag_src with each branch end replaced by its slot
    // the device's copies, one allocation
    int* d_lists = nullptr;
    const int *d_tile_slot = nullptr, *d_slot_src = nullptr, *d_diag_ptr = nullptr,
              *d_diag_src = nullptr, *d_diag_pos = nullptr;
    ~gapk_ybus_s() {
        if (d_lists) cudaFree(d_lists);
    }
    // Runs of whole rows of at most YB_SLOTS slots (a longer row is a run of its own), and the
    // slot of every branch end.
    void tile() {
        tile_slot.assign(1, 0);
        for (int r = 0; r < h.n_bus; ++r)
            if (h.row_ptr[r] > tile_slot.back() && h.row_ptr[r + 1] - tile_slot.back() > YB_SLOTS)
                tile_slot.push_back(h.row_ptr[r]);
        if (h.n_bus > 0) tile_slot.push_back(h.nnz);
        std::vector<int> slot_of(2 * static_cast<size_t>(h.n_branch), -1);
        for (int p = 0; p < h.nnz; ++p)
            if (h.slot_src[p] >= 0) slot_of[h.slot_src[p]] = p;
        diag_pos = h.diag_src;
        for (int& d : diag_pos)
            if (d >= 0) d = slot_of[d];
    }
    int upload() {
        if (d_slot_src) return GAPK_OK;
        std::vector<int> host;
        size_t at[5], n = 0;
        try {
            for (std::vector<int> const* v : {&tile_slot, &h.slot_src, &h.diag_ptr, &h.diag_src, &diag_pos}) {
                at[n++] = host.size();
                host.insert(host.end(), v->begin(), v->end());
            }
            host.push_back(0);  // no list starts past the allocation
        } catch (std::bad_alloc const&) {
            set_error("ybus upload: host allocation failed");
            return GAPK_ENOMEM;
        }
        cudaError_t e = d_lists ? cudaSuccess : cudaMalloc(&d_lists, host.size() * sizeof(int));
        if (e == cudaSuccess)
            e = cudaMemcpy(d_lists, host.data(), host.size() * sizeof(int), cudaMemcpyHostToDevice);
        if (e != cudaSuccess) {
            set_error(std::string("ybus upload: ") + cudaGetErrorString(e));
            return e == cudaErrorMemoryAllocation ? GAPK_ENOMEM : GAPK_ECUDA;
        }
        d_tile_slot = d_lists + at[0];
        d_slot_src = d_lists + at[1];
        d_diag_ptr = d_lists + at[2];
        d_diag_src = d_lists + at[3];
        d_diag_pos = d_lists + at[4];
        cudaGetDevice(&device);
        return GAPK_OK;
    }
};

// Branch results of solved scenarios.  The stamps are the Y-bus builder's (same arithmetic,
// scaled to per unit), so the flows are those of the network the Newton loop solved.
// out[(s * m + j) * 9 ..] = p_from, q_from, i_from, s_from, p_to, q_to, i_to, s_to, loading
// (W, var, A, VA); zeros for out-of-service branches (from < 0).
//
// One thread per branch, BF_SCEN scenarios per CTA in turn: with one set of branch data for all
// scenarios (branch_stride 0) the stamps, whose divisions and sine cost as much as a scenario's
// results, are computed once per CTA.  A scenario's 9 values per branch are collected in shared
// memory (stride 9, no bank conflicts) and written as one contiguous run; straight from the
// threads they would be 72 bytes apart, nine partial passes over the same sectors.
// 512 scenarios x 14,000 branches (0.60 GB compulsory): 312 us with a thread per
// (scenario, branch) storing its own values, 168 us so.
constexpr int BF_THREADS = 128, BF_SCEN = 8;

__global__ void __launch_bounds__(BF_THREADS, 8)
    k_branch_flows(int n_scen, int n_bus, int m, int tiles, const int* __restrict__ from,
                   const int* __restrict__ to, const double* __restrict__ br,
                   int64_t branch_stride, const double2* __restrict__ v, double zb,
                   double base_power, double u_base, const double* __restrict__ i_n,
                   const double* __restrict__ sn, int mode, double* __restrict__ out) {
    __shared__ double o[BF_THREADS * 9];
    const int t = threadIdx.x, j0 = (int)(blockIdx.x % tiles) * BF_THREADS, j = j0 + t;
    const int s0 = (int)(blockIdx.x / tiles) * BF_SCEN, s1 = min(n_scen, s0 + BF_SCEN);
    const int count = min(BF_THREADS, m - j0) * 9;
    const int f = j < m ? from[j] : -1, tb = j < m ? to[j] : -1;
    const bool on = f >= 0 && tb >= 0;
    const double rated_i = on && i_n ? i_n[j] : 0.0, rated_s = on && sn ? sn[j] : 0.0;
    Stamps st;
    if (on && branch_stride == 0) st = branch_stamps(br + (size_t)j * 6, mode);
    double2 vf{}, vt{};
    if (on) {
        vf = v[(size_t)s0 * n_bus + f];
        vt = v[(size_t)s0 * n_bus + tb];
    }
    for (int s = s0; s < s1; ++s) {
        double2 nf{}, nt{};  // the next scenario's voltages, on their way during this one
        if (on && s + 1 < s1) {
            nf = v[(size_t)(s + 1) * n_bus + f];
            nt = v[(size_t)(s + 1) * n_bus + tb];
        }
        double r[9] = {0.0, 0.0, 0.0, 0.0, 0.0, 0.0, 0.0, 0.0, 0.0};
        if (on) {
            if (branch_stride != 0)
                st = branch_stamps(br + (size_t)s * branch_stride + (size_t)j * 6, mode);
            // currents into the branch at each end, per unit
            const double ifr = zb * (st.ff.x * vf.x - st.ff.y * vf.y + st.ft.x * vt.x - st.ft.y * vt.y);
            const double ifi = zb * (st.ff.x * vf.y + st.ff.y * vf.x + st.ft.x * vt.y + st.ft.y * vt.x);
            const double itr = zb * (st.tf.x * vf.x - st.tf.y * vf.y + st.tt.x * vt.x - st.tt.y * vt.y);
            const double iti = zb * (st.tf.x * vf.y + st.tf.y * vf.x + st.tt.x * vt.y + st.tt.y * vt.x);
            // S = V conj(I), in VA
            r[0] = (vf.x * ifr + vf.y * ifi) * base_power;
            r[1] = (vf.y * ifr - vf.x * ifi) * base_power;
            r[4] = (vt.x * itr + vt.y * iti) * base_power;
            r[5] = (vt.y * itr - vt.x * iti) * base_power;
            r[3] = hypot(r[0], r[1]);
            r[7] = hypot(r[4], r[5]);
            const double k3 = 1.7320508075688772 * u_base;  // sqrt(3) x line-to-line base voltage
            r[2] = r[3] / (k3 * hypot(vf.x, vf.y));
            r[6] = r[7] / (k3 * hypot(vt.x, vt.y));
            if (rated_i > 0.0)
                r[8] = fmax(r[2], r[6]) / rated_i;
            else if (rated_s > 0.0)
                r[8] = fmax(r[3], r[7]) / rated_s;
        }
#pragma unroll
        for (int c = 0; c < 9; ++c) o[t * 9 + c] = r[c];
        __syncthreads();
        double* O = out + ((size_t)s * m + j0) * 9;
        for (int c = t; c < count; c += BF_THREADS) O[c] = o[c];
        __syncthreads();
        vf = nf;
        vt = nt;
    }
}

extern "C" {

int gapk_ybus_create(int n_bus, int n_branch, const int* h_from_idx, const int* h_to_idx,
                     const int* h_in_service, int n_shunt, const int* h_shunt_bus,
                     gapk_ybus* out) {
    TraceRange tr("gapk_ybus_create: Y-bus pattern");
    if (!out || n_bus < 0 || n_branch < 0 || n_shunt < 0 ||
        (n_branch && (!h_from_idx || !h_to_idx || !h_in_service)) || (n_shunt && !h_shunt_bus)) {
        set_error("gapk_ybus_create: bad arguments");
        return GAPK_EINVAL;
    }
    auto y = std::make_unique<gapk_ybus_s>();
    build_ybus_pattern(n_bus, n_branch, h_from_idx, h_to_idx, h_in_service, n_shunt,
                       h_shunt_bus, y->h);
    y->tile();
    *out = y.release();
    return GAPK_OK;
}

int gapk_ybus_destroy(gapk_ybus y) {
    delete y;
    return GAPK_OK;
}

int gapk_ybus_nnz(gapk_ybus y) { return y ? y->h.nnz : GAPK_EINVAL; }

int gapk_ybus_pattern(gapk_ybus y, int* h_row_ptr, int* h_col_idx) {
    if (!y || !h_row_ptr || (y->h.nnz && !h_col_idx)) {
        set_error("gapk_ybus_pattern: bad arguments");
        return GAPK_EINVAL;
    }
    std::copy(y->h.row_ptr.begin(), y->h.row_ptr.end(), h_row_ptr);
    std::copy(y->h.col_idx.begin(), y->h.col_idx.end(), h_col_idx);
    return GAPK_OK;
}

int gapk_ybus_assemble(gapk_ybus y, int n_scen, const double* d_branch, int64_t branch_stride,
                       const double* d_shunt, int64_t shunt_stride, int mode, double scale,
                       double* d_values, int64_t values_stride, void* stream) {
    TraceRange tr("gapk_ybus_assemble");
    if (!y || n_scen <= 0 || !d_values || (y->h.n_branch && !d_branch) ||
        (y->h.n_shunt && !d_shunt) || (mode != GAPK_YBUS_REFERENCE && mode != GAPK_YBUS_TAPS) ||
        branch_stride < 0 || shunt_stride < 0 || (n_scen > 1 && values_stride < y->h.nnz)) {
        set_error("gapk_ybus_assemble: bad arguments");
        return GAPK_EINVAL;
    }
    int rc = y->upload();
    if (rc) return rc;
    const long long total = (long long)y->h.nnz * n_scen;
    if (total == 0) return GAPK_OK;
    const int n_tiles = static_cast<int>(y->tile_slot.size()) - 1;
    // 16-byte loads need every branch row on a 16-byte boundary (a row is 48 bytes)
    const bool vec = reinterpret_cast<uintptr_t>(d_branch) % 16 == 0 && branch_stride % 2 == 0;
    const bool few = (long long)n_tiles * n_scen <= YB_FEW;
    const int ns = few ? 1 : YB_SCEN;
    const long long blocks = (long long)n_tiles * ((n_scen + ns - 1) / ns);
    auto kernel = few ? (vec ? k_ybus<true, 1> : k_ybus<false, 1>)
                      : (vec ? k_ybus<true, YB_SCEN> : k_ybus<false, YB_SCEN>);
    kernel<<<static_cast<unsigned>(blocks), YB_SLOTS, 0, static_cast<cudaStream_t>(stream)>>>(
        n_scen, n_tiles, y->d_tile_slot, y->d_slot_src, y->d_diag_ptr, y->d_diag_src, y->d_diag_pos,
        d_branch, branch_stride, d_shunt, shunt_stride, mode, scale,
        reinterpret_cast<double2*>(d_values), values_stride);
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) {
        set_error(std::string("k_ybus launch: ") + cudaGetErrorString(e));
        return GAPK_ECUDA;
    }
    return GAPK_OK;
}

}  // extern "C"

// Segmented plan of branch changes: for every scenario, the CSR slots its changes touch, each
// with its (change, role) list in change order.
struct gapk_ybus_delta_s {
    int n_scen = 0, n_changes = 0;
    std::vector<int> items;  // int4 per (scenario, slot): scenario, slot, seg begin, seg end
    std::vector<int> seg;
    int device = -1;
    void* d_items = nullptr;
    void* d_seg = nullptr;
    ~gapk_ybus_delta_s() {
        if (d_items) cudaFree(d_items);
        if (d_seg) cudaFree(d_seg);
    }
    int upload() {
        if (d_items || items.empty()) return GAPK_OK;
        cudaError_t e = cudaMalloc(&d_items, items.size() * sizeof(int));
        if (e == cudaSuccess) e = cudaMalloc(&d_seg, std::max<size_t>(seg.size(), 1) * sizeof(int));
        if (e == cudaSuccess)
            e = cudaMemcpy(d_items, items.data(), items.size() * sizeof(int), cudaMemcpyHostToDevice);
        if (e == cudaSuccess && !seg.empty())
            e = cudaMemcpy(d_seg, seg.data(), seg.size() * sizeof(int), cudaMemcpyHostToDevice);
        if (e != cudaSuccess) {
            set_error(std::string("ybus delta upload: ") + cudaGetErrorString(e));
            return e == cudaErrorMemoryAllocation ? GAPK_ENOMEM : GAPK_ECUDA;
        }
        cudaGetDevice(&device);
        return GAPK_OK;
    }
};

namespace {

int delta_build(int n_scen, const int* change_ptr, const int* pos, gapk_ybus_delta_s& d) {
    d.n_scen = n_scen;
    d.n_changes = change_ptr[n_scen];
    std::vector<std::pair<int, int>> touch;  // (slot, change << 2 | role), per scenario
    for (int s = 0; s < n_scen; ++s) {
        if (change_ptr[s + 1] < change_ptr[s]) return GAPK_EINVAL;
        touch.clear();
        for (int c = change_ptr[s]; c < change_ptr[s + 1]; ++c)
            for (int r = 0; r < 4; ++r)
                if (pos[4 * c + r] >= 0) touch.emplace_back(pos[4 * c + r], c << 2 | r);
        // by slot; within a slot in change order (stable: the list is built in change order)
        std::stable_sort(touch.begin(), touch.end(),
                         [](auto const& a, auto const& b) { return a.first < b.first; });
        for (size_t i = 0; i < touch.size();) {
            size_t j = i;
            while (j < touch.size() && touch[j].first == touch[i].first) ++j;
            d.items.insert(d.items.end(), {s, touch[i].first, static_cast<int>(d.seg.size()),
                                           static_cast<int>(d.seg.size() + (j - i))});
            for (size_t k = i; k < j; ++k) d.seg.push_back(touch[k].second);
            i = j;
        }
    }
    return GAPK_OK;
}

int delta_launch(gapk_ybus_delta_s& d, const double* d_params, int mode, double scale,
                 double* d_values, int64_t stride, cudaStream_t st) {
    int rc = d.upload();
    if (rc) return rc;
    const int n_items = static_cast<int>(d.items.size() / 4);
    if (n_items == 0) return GAPK_OK;
    k_ybus_delta<<<(n_items + 255) / 256, 256, 0, st>>>(
        n_items, static_cast<const int4*>(d.d_items), static_cast<const int*>(d.d_seg), d_params,
        mode, scale, reinterpret_cast<double2*>(d_values), stride);
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) {
        set_error(std::string("k_ybus_delta launch: ") + cudaGetErrorString(e));
        return GAPK_ECUDA;
    }
    return GAPK_OK;
}

}  // namespace

extern "C" {

int gapk_ybus_delta_create(int n_scen, const int* h_change_ptr, const int* h_pos,
                           gapk_ybus_delta* out) {
    if (!out || n_scen <= 0 || !h_change_ptr || h_change_ptr[0] != 0 ||
        (h_change_ptr[n_scen] > 0 && !h_pos)) {
        set_error("gapk_ybus_delta_create: bad arguments");
        return GAPK_EINVAL;
    }
    auto d = std::make_unique<gapk_ybus_delta_s>();
    if (delta_build(n_scen, h_change_ptr, h_pos, *d)) {
        set_error("gapk_ybus_delta_create: change_ptr must be non-decreasing");
        return GAPK_EINVAL;
    }
    *out = d.release();
    return GAPK_OK;
}

int gapk_ybus_delta_destroy(gapk_ybus_delta d) {
    delete d;
    return GAPK_OK;
}

int gapk_ybus_delta_apply(gapk_ybus_delta d, const double* d_params, int mode, double scale,
                          double* d_values, int64_t values_stride, void* stream) {
    if (!d || !d_values ||
        (mode != GAPK_DELTA_REFERENCE && mode != GAPK_DELTA_FIXED &&
         mode != GAPK_DELTA_FIXED_TAPS) ||
        (d->n_changes > 0 && !d_params) || (d->n_scen > 1 && values_stride <= 0)) {
        set_error("gapk_ybus_delta_apply: bad arguments");
        return GAPK_EINVAL;
    }
    return delta_launch(*d, d_params, mode, scale, d_values, values_stride,
                        static_cast<cudaStream_t>(stream));
}

int gapk_ybus_apply_changes(int n_changes, const int* h_pos, const double* d_params, int mode,
                            double* d_values, void* stream) {
    if (n_changes < 0 || (n_changes > 0 && (!h_pos || !d_params || !d_values))) {
        set_error("gapk_ybus_apply_changes: bad arguments");
        return GAPK_EINVAL;
    }
    if (n_changes == 0) return GAPK_OK;
    const int ptr[2] = {0, n_changes};
    gapk_ybus_delta_s d;
    if (delta_build(1, ptr, h_pos, d)) return GAPK_EINVAL;
    return gapk_ybus_delta_apply(&d, d_params, mode, 1.0, d_values, 0, stream);
}

int gapk_branch_flows(int n_scen, int n_bus, int n_branch, const int* d_from, const int* d_to,
                      const double* d_branch, int64_t branch_stride, const double* d_v,
                      double base_power, double u_base, const double* d_i_n, const double* d_sn,
                      int mode, double* d_out, void* stream) {
    if (n_scen <= 0 || n_bus <= 0 || n_branch < 0 || base_power <= 0.0 || u_base <= 0.0 ||
        (n_branch && (!d_from || !d_to || !d_branch || !d_v || !d_out)) || branch_stride < 0 ||
        (n_scen > 1 && branch_stride != 0 && branch_stride < (int64_t)n_branch * 6) ||
        (mode != GAPK_YBUS_REFERENCE && mode != GAPK_YBUS_TAPS)) {
        set_error("gapk_branch_flows: bad arguments");
        return GAPK_EINVAL;
    }
    if (n_branch == 0) return GAPK_OK;
    const int tiles = (n_branch + BF_THREADS - 1) / BF_THREADS;
    const long long blocks = (long long)tiles * ((n_scen + BF_SCEN - 1) / BF_SCEN);
    const double zb = u_base * u_base / base_power;
    k_branch_flows<<<(unsigned)blocks, BF_THREADS, 0, static_cast<cudaStream_t>(stream)>>>(
        n_scen, n_bus, n_branch, tiles, d_from, d_to, d_branch, branch_stride,
        reinterpret_cast<const double2*>(d_v), zb, base_power, u_base, d_i_n, d_sn, mode, d_out);
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) {
        set_error(std::string("k_branch_flows launch: ") + cudaGetErrorString(e));
        return GAPK_ECUDA;
    }
    return GAPK_OK;
}

}  // extern "C"
