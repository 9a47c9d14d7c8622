// CUDA kernels of the B200 QuickSampling (QS) hot path, sm_100a.
//
// Per batch of independent path nodes ("slots"):
//   k_prep_sim     neighbour values -> per-node term list, border bounds
//                  (G2S include/simulation.hpp:447-537, quantileSamplingModule.hpp:368-457,
//                   DataImage.hpp:626-710, CPUThreadDevice.cpp:352-366,454-477)
//   k_map_records  mismatch map of every scan position in FP32 (direct sum in
//                  the reference's layer decomposition, CPUThreadDevice.cpp:349-490)
//                  fused with a warp prefix-top-K filter that keeps only the
//                  positions that can enter the running k-best ("records")
//   k_replay       exact replay of the reference's k-biggest scan with its
//                  mt19937 reservoir tie-breaking (fKb.hpp:58-92,121-132,
//                  quantileSamplingModule.hpp:45-49,525-557) over the records,
//                  then the draw and the write-back (quantileSamplingModule.hpp:90-126,
//                  CPUThreadDevice.cpp:257-268, simulation.hpp:586-666)
//   k_map_bits     the same map for categorical patterns with unit weights,
//                  bit-sliced (one bit plane per category), same records
// Setup kernels: k_build_layers (DataImage.hpp:538-599), k_neighbours
// (simulation.hpp:447-511, run for every path node at once), k_level_flow /
// k_level_count / k_level_scatter (dependency levels of the path DAG, nodes
// grouped by level).
#include <cuda_runtime.h>

#include <atomic>
#include <math_constants.h>
#include <cstdint>

#include "qsk_internal.h"
#include "qsk_pdl.cuh"
#include "qsk_tc_nodes.cuh"

namespace qsk {

// ---------------------------------------------------------------------------
// small helpers
// ---------------------------------------------------------------------------
__device__ __forceinline__ unsigned lanemask_lt() {
    unsigned m;
    asm("mov.u32 %0, %%lanemask_lt;" : "=r"(m));
    return m;
}

// merge two descending top-K lists (register arrays, static indices only):
// c_t = max_{i=0..t+1} min(a_{i-1}, b_{t-i}), with a_{-1} = b_{-1} = +inf.
template <int K>
__device__ __forceinline__ void topk_merge(const float (&a)[K], const float (&b)[K], float (&c)[K]) {
#pragma unroll
    for (int t = 0; t < K; ++t) {
        float best = -CUDART_INF_F;
#pragma unroll
        for (int i = 0; i <= t + 1; ++i) {
            float ai = (i == 0) ? CUDART_INF_F : a[i - 1];
            float bj = (t - i >= 0) ? b[t - i] : CUDART_INF_F;
            best = fmaxf(best, fminf(ai, bj));
        }
        c[t] = best;
    }
}

template <int KF>
__device__ __forceinline__ void topk_insert(float (&st)[KF], float x) {
    // insert x into the descending list st, dropping the smallest
#pragma unroll
    for (int s = KF - 1; s >= 0; --s) {
        float prev = (s > 0) ? st[s > 0 ? s - 1 : 0] : CUDART_INF_F;
        // new st[s] = max(min(prev, x), st[s])
        st[s] = fmaxf(st[s], fminf(prev, x));
    }
}

// ---------------------------------------------------------------------------
// layers: flipped copy of each TI variable (DataImage.hpp:538-599)
// continuous: value with NaN -> 0 ; categorical: value kept as the category
// code (NaN stays NaN, so it never equals a code).  Positions of the fft grid
// outside the TI hold 0 (continuous) / NaN (categorical).
// ---------------------------------------------------------------------------
__global__ void k_build_layers(const float *__restrict__ ti, int nvar, const int *__restrict__ types, Geom g,
                               float *__restrict__ layers, int missing) {
    long long q = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (q >= g.N) return;
    // q is an fft-grid flat index of the flipped array: coord = fft-1-digit
    long long src_flat = 0, sstr = 1;
    bool inside = true;
    for (int d = 0; d < g.nd; ++d) {
        long long digit = (q / g.sstride[d]) % g.fft[d];
        long long c = g.fft[d] - 1 - digit;
        inside &= c < g.src[d];
        src_flat += c * sstr;
        sstr *= g.src[d];
    }
    for (int v = 0; v < nvar; ++v) {
        float x;
        if (inside) {
            x = ti[src_flat * nvar + v];
            if (types[v] == 0 && isnan(x) && !missing) x = 0.f;
        } else {
            x = types[v] == 0 ? 0.f : CUDART_NAN_F;
        }
        layers[(long long)v * g.N + q] = x;
    }
    if (missing) {
        // mask layer (DataImage.hpp:582-595): 1 where the TI cell is informed
        layers[(long long)nvar * g.N + q] = (inside && !isnan(ti[src_flat * nvar])) ? 1.f : 0.f;
    }
}

// ---------------------------------------------------------------------------
// neighbour search for every path node (simulation.hpp:447-511, single n,
// non-strict informed rule: cells with path order <= the node's, the node
// itself included).
// ---------------------------------------------------------------------------
// one warp per node: 32 template offsets tested per step, accepted ones
// appended in template order
__global__ void k_neighbours(GridDesc dg, const int *__restrict__ tpl, int ntpl, const unsigned *__restrict__ path,
                             unsigned begin, long long nodes, const unsigned *__restrict__ posterior, int n,
                             int *__restrict__ nb_count, int *__restrict__ nb_tpl, unsigned *__restrict__ nb_cell,
                             const int *__restrict__ node_kernel, const int *__restrict__ tpl_range,
                             const int *__restrict__ node_lim) {
    const long long i = ((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int lane = threadIdx.x & 31;
    if (i >= nodes) return;
    const unsigned cell = path[begin + i];
    const unsigned order = posterior[cell];
    int c0[QSK_MAXD];
    long long rem = cell;
    for (int d = 0; d < dg.nd; ++d) {
        c0[d] = int(rem % dg.dims[d]);
        rem /= dg.dims[d];
    }
    // template of this node's kernel (-kii) and its neighbour limit (-n per variable / -ni)
    int tb = 0, tn = ntpl, lim = n;
    if (node_kernel) {
        const int q = node_kernel[i];
        tb = tpl_range[2 * q];
        tn = tpl_range[2 * q + 1];
    }
    if (node_lim) lim = min(node_lim[i], n);
    int cnt = 0;
    for (int t0 = 0; t0 < tn && cnt < lim; t0 += 32) {
        const int t = t0 + lane;
        bool acc = false;
        long long nc = 0;
        if (t < tn) {
            bool ok = true;
            for (int d = 0; d < dg.nd; ++d) {
                int c = c0[d] + tpl[(tb + t) * dg.nd + d];
                ok &= (c >= 0) && (c < dg.dims[d]);
                nc += (long long)c * dg.stride[d];
            }
            acc = ok && posterior[nc] <= order;
        }
        const unsigned bal = __ballot_sync(0xffffffffu, acc);
        const int pos = cnt + __popc(bal & ((1u << lane) - 1u));
        if (acc && pos < lim) {
            nb_tpl[i * n + pos] = tb + t;
            nb_cell[i * n + pos] = unsigned(nc);
        }
        cnt += __popc(bal);
    }
    if (lane == 0) nb_count[i] = cnt < lim ? cnt : lim;
}

// -fs: one warp per (cell, variable) node.  A cell is taken when a variable
// that still needs neighbours was simulated there strictly before the node
// (posterior < order, simulation.hpp:822-872); the variables it contributes
// are recorded in nb_mask.  The 32 offsets of a step are tested in parallel,
// then taken in template order with the per-variable counts.
__global__ void k_neighbours_full(GridDesc dg, const int *__restrict__ tpl, int ntpl, const unsigned *__restrict__ path,
                                  unsigned begin, long long nodes, const unsigned *__restrict__ posterior, int nvar,
                                  int n, const int *__restrict__ node_nv, int *__restrict__ nb_count,
                                  int *__restrict__ nb_tpl, unsigned *__restrict__ nb_cell,
                                  unsigned char *__restrict__ nb_mask, const int *__restrict__ node_kernel,
                                  const int *__restrict__ tpl_range) {
    const long long i = ((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int lane = threadIdx.x & 31;
    if (i >= nodes) return;
    const unsigned value = path[begin + i];
    const unsigned cell = value / unsigned(nvar);
    const unsigned order = posterior[value];
    int c0[QSK_MAXD];
    long long rem = cell;
    for (int d = 0; d < dg.nd; ++d) {
        c0[d] = int(rem % dg.dims[d]);
        rem /= dg.dims[d];
    }
    int tb = 0, tn = ntpl;
    if (node_kernel) {
        const int q = node_kernel[i];
        tb = tpl_range[2 * q];
        tn = tpl_range[2 * q + 1];
    }
    int need[4] = {0, 0, 0, 0};   // remaining count per variable
    unsigned needm = 0;
    for (int v = 0; v < nvar && v < 4; ++v) {
        need[v] = node_nv ? node_nv[i * nvar + v] : n;
        if (need[v] > 0) needm |= 1u << v;
    }
    int cnt = 0;
    for (int t0 = 0; t0 < tn && needm && cnt < n; t0 += 32) {
        const int t = t0 + lane;
        unsigned im = 0;
        long long nc = 0;
        if (t < tn) {
            bool ok = true;
            for (int d = 0; d < dg.nd; ++d) {
                int c = c0[d] + tpl[(tb + t) * dg.nd + d];
                ok &= (c >= 0) && (c < dg.dims[d]);
                nc += (long long)c * dg.stride[d];
            }
            if (ok)
                for (int v = 0; v < nvar && v < 4; ++v)
                    if (posterior[nc * nvar + v] < order) im |= 1u << v;
        }
        unsigned cand = __ballot_sync(0xffffffffu, (im & needm) != 0u);
        while (cand && needm && cnt < n) {
            const int l = __ffs(cand) - 1;
            cand &= cand - 1u;
            const unsigned m = __shfl_sync(0xffffffffu, im, l) & needm;
            if (!m) continue;
            if (lane == l) {
                nb_tpl[i * n + cnt] = tb + t;
                nb_cell[i * n + cnt] = unsigned(nc);
                nb_mask[i * n + cnt] = (unsigned char)m;
            }
            for (int v = 0; v < 4; ++v)
                if ((m >> v) & 1u && --need[v] == 0) needm &= ~(1u << v);
            ++cnt;
        }
    }
    if (lane == 0) nb_count[i] = cnt;
}

// ---------------------------------------------------------------------------
// dependency levels: level(i) = 1 + max level(j) over the node's informed
// neighbours j that are themselves path nodes (0 without any) -- the longest
// path to i in the path DAG (dependencies always point to smaller path
// indices).  One pass in path order (k_level_flow), then a counting sort of
// the nodes by level (k_level_count, the scan, k_level_scatter).
// ---------------------------------------------------------------------------
// dependency nodes of neighbour j of node i: the cell's node, or (-fs, with
// nb_mask) the nodes of the cell's values that the neighbour contributes
template <class F>
__device__ __forceinline__ void for_each_dep(long long i, int j, int n, const unsigned *__restrict__ nb_cell,
                                             const unsigned char *__restrict__ nb_mask, int nvar,
                                             const int *__restrict__ node_of, F f) {
    const unsigned c = nb_cell[i * n + j];
    if (!nb_mask) {
        const int d = node_of[c];
        if (d >= 0 && (long long)d != i) f(d);
        return;
    }
    const unsigned m = nb_mask[i * n + j];
    for (int v = 0; v < nvar; ++v)
        if ((m >> v) & 1u) {
            const int d = node_of[(long long)c * nvar + v];
            if (d >= 0 && (long long)d != i) f(d);
        }
}

// One warp per node, nodes taken in path order from a ticket.  A node's
// dependencies have smaller path indices, so they were taken earlier by warps
// that are running; the smallest unfinished node waits on finished nodes only,
// so every wait ends.  The waits are bounded all the same: past `spin_limit`
// polls of one dependency (2^22 by default, about a second with the back-off)
// the kernel records DEV_LEVEL_WAIT and moves on (the host then fails the
// run).  `hold` (normally -1) names a node whose level is never published:
// a host-side injection that makes its dependants' waits run out, so that the
// failure path can be exercised without a fault.
// The level words start at -1; a level is published with one volatile store
// and read with volatile loads (it carries no other data).
__global__ void k_level_flow(long long nodes, int n, const int *__restrict__ nb_count,
                             const unsigned *__restrict__ nb_cell, const unsigned char *__restrict__ nb_mask, int nvar,
                             const int *__restrict__ node_of, int *level, int *ticket, int *nl_out, int *status,
                             unsigned spin_limit, long long hold) {
    const int lane = threadIdx.x & 31;
    volatile int *vlevel = level;
    for (;;) {
        int i = 0;
        if (lane == 0) i = atomicAdd(ticket, 1);
        i = __shfl_sync(0xffffffffu, i, 0);
        if ((long long)i >= nodes) return;
        const int c = nb_count[i];
        int mx = -1;
        bool bad = false, late = false;
        for (int j = lane; j < c; j += 32)
            for_each_dep(i, j, n, nb_cell, nb_mask, nvar, node_of, [&](int d) {
                if (d >= i) {
                    bad = true;
                    return;
                }
                int lv = vlevel[d];
                unsigned spins = 0;
                while (lv < 0) {
                    if (++spins > spin_limit) {
                        late = true;
                        lv = 0;
                        break;
                    }
                    __nanosleep(128);
                    lv = vlevel[d];
                }
                mx = max(mx, lv);
            });
#pragma unroll
        for (int off = 16; off > 0; off >>= 1) mx = max(mx, __shfl_xor_sync(0xffffffffu, mx, off));
        const bool any_bad = __any_sync(0xffffffffu, bad), any_late = __any_sync(0xffffffffu, late);
        if (lane == 0) {
            if (any_bad) atomicExch(status, DEV_BAD_INDEX);
            if (any_late) atomicExch(status, DEV_LEVEL_WAIT);
            if ((long long)i != hold) {
                vlevel[i] = mx + 1;
                atomicMax(nl_out, mx + 2);
            }
        }
    }
}

__global__ void k_level_count(long long nodes, const int *__restrict__ level, int *__restrict__ cnt) {
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i < nodes && level[i] >= 0) atomicAdd(&cnt[level[i]], 1);   // < 0: held back (the run fails)
}

// exclusive scan in three passes: 1024-element tiles, tile sums, add
__global__ void __launch_bounds__(1024) k_scan_tiles(long long count, const int *__restrict__ in, int *__restrict__ out,
                                                     int *__restrict__ tile_sum) {
    __shared__ int warp_sum[32];
    const long long i = (long long)blockIdx.x * 1024 + threadIdx.x;
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const int x = i < count ? in[i] : 0;
    int incl = x;
#pragma unroll
    for (int off = 1; off < 32; off <<= 1) {
        const int y = __shfl_up_sync(0xffffffffu, incl, off);
        if (lane >= off) incl += y;
    }
    if (lane == 31) warp_sum[w] = incl;
    __syncthreads();
    if (w == 0) {
        int ws = warp_sum[lane];
#pragma unroll
        for (int off = 1; off < 32; off <<= 1) {
            const int y = __shfl_up_sync(0xffffffffu, ws, off);
            if (lane >= off) ws += y;
        }
        warp_sum[lane] = ws;   // inclusive
    }
    __syncthreads();
    const int base = w > 0 ? warp_sum[w - 1] : 0;
    if (i < count) out[i] = base + incl - x;
    if (threadIdx.x == 1023) tile_sum[blockIdx.x] = base + incl;
}

__global__ void k_scan_sums(int ntiles, int *__restrict__ tile_sum) {
    if (threadIdx.x == 0) {
        int s = 0;
        for (int t = 0; t < ntiles; ++t) {
            const int v = tile_sum[t];
            tile_sum[t] = s;
            s += v;
        }
        tile_sum[ntiles] = s;
    }
}

__global__ void k_scan_add(long long count, int *__restrict__ out, int *__restrict__ cursor,
                           const int *__restrict__ tile_sum) {
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i < count) {
        const int v = out[i] + tile_sum[i / 1024];
        out[i] = v;
        cursor[i] = v;
    } else if (i == count) {
        const int v = tile_sum[(count + 1023) / 1024];
        out[i] = v;
    }
}

// nodes grouped by level (order inside a level is free: its nodes are independent)
__global__ void k_level_scatter(long long nodes, const int *__restrict__ level, int *__restrict__ cursor,
                                int *__restrict__ level_nodes) {
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i < nodes && level[i] >= 0) level_nodes[atomicAdd(&cursor[level[i]], 1)] = int(i);
}

// ---------------------------------------------------------------------------
// selected rank of the draw, exactly as compiled in the reference
// (quantileSamplingModule.hpp:113 with the double overloads of ceil/floor)
// ---------------------------------------------------------------------------
__device__ __forceinline__ int selected_index(float seed, float k, unsigned nti) {
    double prod = (double)__fmul_rn(seed, k);
    double c = ceil((double)__fdiv_rn((float)nti, k));
    return int(floor(prod * (c / (double)nti)));
}

// ---------------------------------------------------------------------------
// prep for the simulation: one warp per slot
// ---------------------------------------------------------------------------
// The part of a node's slot that follows from the neighbour lists and the
// initial grid alone (not from simulated values), shared by k_prep_sim and
// k_mt_prep: candidate count, neighbour offset minima, first valid scan
// coordinate per dimension, number of valid positions, marginal draw.
struct NodeGeom {
    float lk;
    int Ki;
    int mn[QSK_MAXD];
    int lo[QSK_MAXD];
    long long nvalid;
    bool skip;
};

__device__ NodeGeom node_geometry(const SimPrepArgs &A, int i, unsigned cell, int lane) {
    NodeGeom r;
    const int cnt = A.nb_count[i];
    const int nd = A.g.nd;
    // candidate count of this node: -kvi or k (quantileSamplingModule.hpp:90-113)
    r.lk = A.node_k ? A.node_k[i] : A.k;
    int Ki = int(ceilf(r.lk));
    r.Ki = Ki < 1 ? 1 : (Ki > QSK_KMAX ? QSK_KMAX : Ki);
    // vector simulation: data at the centre also forces a search
    // (simulation.hpp:565-584); -fs draws from the marginal below two
    // neighbours (simulation.hpp:952-965)
    bool centreData = false;
    if (!A.full)
        for (int v = 0; v < A.nvar; ++v) centreData |= !isnan(A.init[(long long)cell * A.nvar + v]);
    // min / max of the neighbour offsets, starting from 0 (AcceleratorDevice.cpp:95-112)
    int mn[QSK_MAXD], mx[QSK_MAXD];
#pragma unroll
    for (int d = 0; d < QSK_MAXD; ++d) { mn[d] = 0; mx[d] = 0; }
    for (int j = lane; j < cnt; j += 32) {
        int t = A.nb_tpl[(long long)i * A.n + j];
        for (int d = 0; d < nd; ++d) {
            int o = A.tpl[t * nd + d];
            mn[d] = min(mn[d], o);
            mx[d] = max(mx[d], o);
        }
    }
#pragma unroll
    for (int d = 0; d < QSK_MAXD; ++d) {
        for (int off = 16; off > 0; off >>= 1) {
            mn[d] = min(mn[d], __shfl_xor_sync(0xffffffffu, mn[d], off));
            mx[d] = max(mx[d], __shfl_xor_sync(0xffffffffu, mx[d], off));
        }
    }
    r.nvalid = 1;
    for (int d = 0; d < QSK_MAXD; ++d) {
        r.mn[d] = mn[d];
        int lo = 0;
        if (d < nd) {
            lo = A.g.fft[d] - (A.g.src[d] - (mx[d] - mn[d]));
            lo = lo < 0 ? 0 : (lo > A.g.fft[d] ? A.g.fft[d] : lo);
            r.nvalid *= (A.g.fft[d] - lo);
        }
        r.lo[d] = lo;
    }
    r.skip = cnt <= 1 && !centreData;   // marginal draw (simulation.hpp:586-605)
    return r;
}

// -nV: scan index of the TI cell that continues neighbour 1's source (cell
// id_src, template offset tpl1) (simulation.hpp:556-583,
// quantileSamplingModule.hpp:518-523), or -1 outside the scan
__device__ int verbatim_excl(const Geom &g, const int *tpl1, unsigned id_src, const int *mn) {
    const int nd = g.nd;
    unsigned src = id_src;
    long long pf = 0, st = 1;
    for (int d = 0; d < nd; ++d) {
        int dim = g.src[d];
        int c = int(src % (unsigned)dim) - tpl1[d];
        src /= (unsigned)dim;
        c = ((c % dim) + dim) % dim;
        pf += (long long)c * st;
        st *= dim;
    }
    // cvtPositionToIndex (CPUThreadDevice.cpp:270-284), unsigned arithmetic
    unsigned position = (unsigned)pf, index = 0, div = 1;
    for (int d = nd - 1; d >= 0; --d) div *= (unsigned)g.src[d];
    for (int d = nd - 1; d >= 0; --d) {
        unsigned f = (unsigned)g.fft[d], sr = (unsigned)g.src[d];
        div /= sr;
        index = index * f + (f - (position / div + (unsigned)mn[d]) % sr - 1u);
    }
    return index < (unsigned)g.N ? int(index) : -1;
}

// slot `warp` of a batch (one warp)
__device__ __forceinline__ void prep_sim_warp(const SimPrepArgs &A, const int warp, const int lane) {
    if (warp >= A.nslots) return;
    const int i = A.nodes[warp];
    const unsigned pv = A.path[A.begin + i];
    // -fs: the path entry is a cell value (cell * nvar + variable)
    const unsigned cell = A.full ? pv / unsigned(A.nvar) : pv;
    const int cnt = A.nb_count[i];
    const int nd = A.g.nd;
    const NodeGeom ng = node_geometry(A, i, cell, lane);
    // launched programmatically: what is read above follows from the path
    // alone; simulated values, slots and terms come below
    griddep_wait();
    griddep_launch();   // (no later grid reads or writes anything before this one has completed)
    Slot s;
    s.node = i;
    s.cell = cell;
    s.var = A.full ? int(pv % unsigned(A.nvar)) : 0;
    s.seed = A.seeds[i];
    const float lk = ng.lk;
    const int Ki = ng.Ki;
    s.K = Ki;
    s.sel = selected_index(s.seed, lk, A.nti);
    if (s.sel < 0) s.sel = 0;
    if (s.sel > Ki - 1) s.sel = Ki - 1;   // unreachable for k >= 1 and seeds in [0,1)
    s.flags = 0;
    s.nterms = 0;
    s.excl = -1;
    s.cmask_base = 0;
    int mn[QSK_MAXD];
#pragma unroll
    for (int d = 0; d < QSK_MAXD; ++d) {
        mn[d] = ng.mn[d];
        s.mn[d] = ng.mn[d];
        s.lo[d] = ng.lo[d];
    }
    if (ng.skip) {
        s.flags |= SLOT_SKIP;
    } else {
        if (ng.nvalid < Ki) s.flags |= SLOT_EMIT_MASKED;
        // terms: neighbours in order, variables in order; zero-weight / NaN skipped
        int base_out = 0;
        for (int j0 = 0; j0 < cnt; j0 += 32) {
            int j = j0 + lane;
            Term tl[8];
            int nt = 0;
            if (j < cnt) {
                int t = A.nb_tpl[(long long)i * A.n + j];
                unsigned nc = A.nb_cell[(long long)i * A.n + j];
                long long d_flat = 0;
                for (int d = 0; d < nd; ++d) d_flat += (long long)(A.tpl[t * nd + d] - mn[d]) * A.g.sstride[d];
                for (int v = 0; v < A.nvar && v < 4; ++v) {
                    // a variable takes values from its first n_v neighbours only
                    // (simulation.hpp:476-497)
                    if (A.full) {
                        if (!((A.nb_mask[(long long)i * A.n + j] >> v) & 1u)) continue;
                    } else if (A.node_nv && j >= A.node_nv[(long long)i * A.nvar + v]) {
                        continue;
                    }
                    float val = (nc == cell && !A.full) ? A.init[(long long)nc * A.nvar + v]
                                                        : A.state[(long long)nc * A.nvar + v];
                    float w = A.wtab[t * A.nvar + v];
                    if (isnan(val) || w == 0.f) continue;
                    Term tm;
                    tm.base = int((long long)v * A.g.N - d_flat);
                    if (A.types[v] == 0 && A.missing) {
                        // regular output: -w TI^2 + 2wv TI - ((w v) v) mask; overlap: w mask
                        tm.op = OP_SQLINM;
                        tm.a = -w;
                        tm.b = 2.f * __fmul_rn(w, val);
                        tl[nt++] = tm;
                        Term pl;
                        pl.base = tm.base;
                        pl.op = OP_NOP;
                        pl.a = -__fmul_rn(__fmul_rn(w, val), val);
                        pl.b = w;
                        tl[nt++] = pl;
                        continue;
                    }
                    if (A.types[v] == 0) {
                        tm.op = OP_SQLIN;
                        tm.a = -w;
                        tm.b = 2.f * __fmul_rn(w, val);
                    } else {
                        tm.op = OP_EQ;
                        tm.a = w;
                        tm.b = val;
                    }
                    tl[nt++] = tm;
                }
            }
            // order-preserving compaction across the warp
            int incl = nt;
            for (int off = 1; off < 32; off <<= 1) {
                int y = __shfl_up_sync(0xffffffffu, incl, off);
                if (lane >= off) incl += y;
            }
            int excl = incl - nt;
            int total = __shfl_sync(0xffffffffu, incl, 31);
            for (int q = 0; q < nt; ++q) {
                int o = base_out + excl + q;
                if (o < A.maxterms) A.terms[(long long)warp * A.maxterms + o] = tl[q];
            }
            base_out += total;
        }
        if (base_out > A.maxterms) {
            if (lane == 0) atomicExch(A.status, DEV_TOO_MANY_TERMS);
            base_out = A.maxterms;
        }
        s.nterms = base_out;
        if (A.missing) {
            s.flags |= SLOT_MISSING;
            long long fmn = 0;
            for (int d = 0; d < nd; ++d) fmn += (long long)mn[d] * A.g.sstride[d];
            s.cmask_base = int((long long)A.mask_layer * A.g.N + fmn);
        }
        if (A.no_verbatim && cnt > 1 && !A.full) {
            // the TI cell continuing neighbour 1's source is excluded
            const int t1 = A.nb_tpl[(long long)i * A.n + 1];
            const unsigned c1 = A.nb_cell[(long long)i * A.n + 1];
            s.excl = verbatim_excl(A.g, A.tpl + t1 * nd, A.id_image[c1], mn);
        }
    }
    s.vcell = 0;
    s.vtpl = -1;
    if (lane == 0) A.slots[warp] = s;
}

__global__ void k_prep_sim(SimPrepArgs A) {
    prep_sim_warp(A, int((blockIdx.x * blockDim.x + threadIdx.x) >> 5), int(threadIdx.x & 31));
}

// A tensor-core level's exact terms (k_prep_sim) and node rows (k_tc_nodes)
// in one grid: blocks [0, prep_blocks) prepare the slots, the others write
// the rows.  Neither part reads what the other writes (both read only the
// neighbours, values and seeds of earlier levels), so they need no order.
__global__ void k_prep_tc_nodes(SimPrepArgs P, TcNodeArgs T, unsigned prep_blocks) {
    griddep_launch();   // the shortlist (a programmatic successor) may begin launching
    const int lane = int(threadIdx.x & 31);
    if (blockIdx.x < prep_blocks) prep_sim_warp(P, int((blockIdx.x * blockDim.x + threadIdx.x) >> 5), lane);
    else tc_nodes_warp(T, int(((blockIdx.x - prep_blocks) * blockDim.x + threadIdx.x) >> 5), lane);
}

// ---------------------------------------------------------------------------
// mt19937 (published algorithm: Matsumoto & Nishimura 1998) with the
// conversion of std::uniform_real_distribution<float>(0,1) in libstdc++
// (generate_canonical<float,24>: float(u32) * 2^-32, values >= 1 clamped to
// the largest float below 1).
// ---------------------------------------------------------------------------
__device__ __forceinline__ unsigned mt_temper(unsigned y) {
    y ^= y >> 11;
    y ^= (y << 7) & 0x9d2c5680u;
    y ^= (y << 15) & 0xefc60000u;
    y ^= y >> 18;
    return y;
}

__device__ __forceinline__ float mt_unit(unsigned y) {
    float u = __fmul_rn(__uint2float_rn(y), 2.3283064365386963e-10f);
    return u >= 1.f ? 0x1.fffffep-1f : u;
}

__device__ __forceinline__ unsigned mt_mix(unsigned a, unsigned b, unsigned c) {
    unsigned y = (a & 0x80000000u) | (b & 0x7fffffffu);
    return c ^ (y >> 1) ^ ((y & 1u) ? 0x9908b0dfu : 0u);
}


// generator.seed(seedFromUnitFloat(seed) + 0)  (quantileSamplingModule.hpp:45-49,533-534):
// the standard mt19937 initialisation, serial, on the calling thread
__device__ __forceinline__ void mt_seed(unsigned *mt, float sd) {
    unsigned x;
    if (!isfinite(sd) || sd <= 0.f) x = 0u;
    else if (sd >= 1.f) x = 0xffffffffu;
    else x = (unsigned)floor((double)sd * 4294967295.0);
    mt[0] = x;
    for (int i = 1; i < 624; ++i) {
        x = 1812433253u * (x ^ (x >> 30)) + (unsigned)i;
        mt[i] = x;
    }
}

// The blocks roll through registers: a step makes the next 224 words, seven
// consecutive ones per lane (the recurrence reaches back 227 words at the
// least, so a step depends on earlier steps only), from the three steps
// before it: eleven shuffles, no shared memory and no barrier.  512 slots of a
// 128^3 image (up to 600 blocks each): in shared memory, three phases a block,
// five launches of 126 slots or fewer took 107 to 634 us, 1.30 ms in all; now
// two, of 126 and 386 slots, take 405 and 367.
__device__ __forceinline__ void mt_step(unsigned (&n)[7], const unsigned (&a)[7], const unsigned (&b)[7],
                                        const unsigned (&c)[7], int lane) {
    // word t = 7 lane + i of the step needs words t - 3 of the last step (a),
    // t + 48 and t + 49 of the third last (c); past the step's ends the word
    // lies in the one before (b), supplied by the lanes at that end
    unsigned g[7], q[3];
    const unsigned f = __shfl_sync(0xffffffffu, lane < 6 ? b[6] : c[6], (lane + 6) & 31);
#pragma unroll
    for (int i = 0; i < 7; ++i) g[i] = __shfl_sync(0xffffffffu, lane < 7 ? b[i] : c[i], (lane + 7) & 31);
#pragma unroll
    for (int i = 0; i < 3; ++i) q[i] = __shfl_sync(0xffffffffu, lane == 31 ? b[4 + i] : a[4 + i], (lane + 31) & 31);
#pragma unroll
    for (int i = 0; i < 7; ++i) n[i] = mt_mix(i == 0 ? f : g[i > 0 ? i - 1 : 0], g[i], i < 3 ? q[i < 3 ? i : 0] : a[i >= 3 ? i - 3 : 0]);
}

// `blocks` > 0 blocks further from the state mt[624] (shared memory), in place
__device__ void mt_roll(unsigned *mt, long long blocks, int lane) {
    unsigned r0[7], r1[7], r2[7], r3[7];
#pragma unroll
    for (int i = 0; i < 7; ++i) {
        const int t = 7 * lane + i;
        r0[i] = mt[400 + t];
        r1[i] = mt[176 + t];
        r2[i] = t >= 48 ? mt[t - 48] : 0u;   // words below 48 of this step are read by none
        r3[i] = 0u;
    }
    const long long steps = (624 * blocks + 223) / 224;
    for (long long s = 0; s + 4 <= steps; s += 4) {
        mt_step(r3, r0, r1, r2, lane);
        mt_step(r2, r3, r0, r1, lane);
        mt_step(r1, r2, r3, r0, lane);
        mt_step(r0, r1, r2, r3, lane);
    }
    __syncwarp();
    // word 7 lane + i of step `step` is word k of the state
    auto put = [&](const unsigned (&r)[7], long long step) {
#pragma unroll
        for (int i = 0; i < 7; ++i) {
            const long long k = 224 * step + 7 * lane + i - 624 * (blocks - 1);
            if (k >= 0 && k < 624) mt[k] = r[i];
        }
    };
    const int rest = int(steps & 3);
    if (rest > 0) mt_step(r3, r0, r1, r2, lane);
    if (rest > 1) mt_step(r2, r3, r0, r1, lane);
    if (rest > 2) mt_step(r1, r2, r3, r0, lane);
    // the last four steps hold the 624 words (and at most 223 beyond them)
    put(r0, rest == 0 ? steps - 1 : steps - 1 - rest);
    put(r1, rest == 3 ? steps - 1 : steps - 2 - rest);
    put(r2, rest >= 2 ? steps + 1 - rest : steps - 3 - rest);
    put(r3, rest >= 1 ? steps - rest : steps - 4);
    __syncwarp();
}

// the state mt[624] (shared memory) and the blocks it skipped to row b, one warp
__device__ void store_generator(const unsigned *mt, long long blocks, int b, unsigned *state, int *pre, int lane) {
    // a state row is 624 words, a multiple of 16 bytes
    uint4 *row = reinterpret_cast<uint4 *>(state + (long long)b * 624);
    for (int i = lane; i < 156; i += 32) row[i] = *reinterpret_cast<const uint4 *>(&mt[4 * i]);
    if (lane == 0) pre[b] = int(blocks);
}

// GenArgs: slot b's generator state by the first warp of a CTA
__device__ void slot_generator(const Geom &g, const Slot &sl, int b, const GenArgs &gen, unsigned *mt) {
    if (threadIdx.x >= 32 || (sl.flags & SLOT_SKIP)) return;
    const int lane = threadIdx.x;
    if (lane == 0) mt_seed(mt, sl.seed);
    __syncwarp();
    long long blocks = 0;
    if (!(sl.flags & (SLOT_EMIT_MASKED | SLOT_MISSING))) {
        long long nvalid = 1;
        int lo[QSK_MAXD];
        for (int d = 0; d < QSK_MAXD; ++d) lo[d] = sl.lo[d];
        for (int d = 0; d < g.nd; ++d) nvalid *= g.fft[d] - lo[d];
        blocks = skipped_blocks(g, lo, nvalid, sl.K);
    }
    if (blocks > 0) mt_roll(mt, blocks, lane);
    store_generator(mt, blocks, b, gen.state, gen.pre, lane);
}

// ---------------------------------------------------------------------------
// fused map + record filter
//
// A warp takes MR_SEGS consecutive 128-position segments at once, eight
// positions per lane (base + 32 r + lane): a term's shared-memory read, its
// address and the loop are paid once for eight gathers, which all go to one
// pointer at immediate offsets, and the products run on packed FP32 pairs
// (each half rounded as the scalar instruction rounds it).  In cache the
// kernel is bound by L1 wavefronts, one per 32 gathers and one per term read:
// eight positions a lane reach 23 position-terms per clock and SM of the 28
// that nine wavefronts per 256 allow.  Positions outside the border are
// gathered like the others where every address of the warp's span lies in the
// layers (their scores are not used); at the two ends of the scan, and for
// the rarer operations, they gather from a valid dummy address instead.
// Spans without a valid position gather nothing.
//
// The filter keeps the prefix top-K of the positions the warp has seen over
// all its spans (a CTA's warps take interleaved spans in scan order, so
// everything a warp has seen lies before its next span): a segment, and a
// round of 32 positions, whose maximum is below that K-th best holds no
// record, and a few candidates are inserted one by one.
// ---------------------------------------------------------------------------
namespace {
typedef unsigned long long f32x2;
__device__ __forceinline__ f32x2 pack2(float a, float b) {
    f32x2 r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
    return r;
}
__device__ __forceinline__ void unpack2(f32x2 v, float &a, float &b) {
    asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(v));
}
__device__ __forceinline__ f32x2 mul2(f32x2 a, f32x2 b) {
    f32x2 r;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ f32x2 fma2(f32x2 a, f32x2 b, f32x2 c) {
    f32x2 r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
    return r;
}
// x / d for x < 2^31
__device__ __forceinline__ unsigned fast_div(unsigned x, FastDiv f) { return f.shift < 0 ? x : __umulhi(x, f.mul) >> f.shift; }

constexpr int MR_SEGS = 2;               // segments a warp takes at once
constexpr int MR_P = 4 * MR_SEGS;        // positions per lane

// one pass over the terms at in-bounds addresses: p is the span's first
// layer element of this lane
template <bool ALL_SQ>
__device__ __forceinline__ void map_terms_fast(const Term *__restrict__ sterm, int nt, const float *__restrict__ p,
                                               float (&acc)[MR_P]) {
    f32x2 a2[MR_P / 2];
#pragma unroll
    for (int i = 0; i < MR_P / 2; ++i) a2[i] = 0ull;
#pragma unroll 2
    for (int t = 0; t < nt; ++t) {
        const Term tm = sterm[t];
        const float *lp = p + tm.base;
        float x[MR_P];
#pragma unroll
        for (int r = 0; r < MR_P; ++r) x[r] = __ldg(lp + 32 * r);
        if (ALL_SQ || tm.op == OP_SQLIN) {
            const f32x2 ta = pack2(tm.a, tm.a), tb = pack2(tm.b, tm.b);
#pragma unroll
            for (int i = 0; i < MR_P / 2; ++i) {
                const f32x2 xx = pack2(x[2 * i], x[2 * i + 1]);
                a2[i] = fma2(ta, mul2(xx, xx), a2[i]);
                a2[i] = fma2(tb, xx, a2[i]);
            }
        } else if (tm.op == OP_EQ) {
#pragma unroll
            for (int i = 0; i < MR_P / 2; ++i) {
                float u, v;
                unpack2(a2[i], u, v);
                u = (x[2 * i] == tm.b) ? __fadd_rn(u, tm.a) : u;
                v = (x[2 * i + 1] == tm.b) ? __fadd_rn(v, tm.a) : v;
                a2[i] = pack2(u, v);
            }
        } else {   // OP_LIN
            const f32x2 ta = pack2(tm.a, tm.a);
#pragma unroll
            for (int i = 0; i < MR_P / 2; ++i) a2[i] = fma2(ta, pack2(x[2 * i], x[2 * i + 1]), a2[i]);
        }
    }
#pragma unroll
    for (int i = 0; i < MR_P / 2; ++i) unpack2(a2[i], acc[2 * i], acc[2 * i + 1]);
}

// the same for every operation, with the positions outside the border (or
// the scan) gathered at usafe
__device__ void map_terms_any(const Term *__restrict__ sterm, int nt, const float *__restrict__ layers, unsigned base,
                              unsigned vm, unsigned usafe, float (&acc)[MR_P], float (&crs)[MR_P]) {
    unsigned mm[MR_P];
#pragma unroll
    for (int r = 0; r < MR_P; ++r) mm[r] = ((vm >> r) & 1u) ? base + 32 * r : usafe;
    for (int t = 0; t < nt; ++t) {
        const Term tm = sterm[t];
        const float *lp = layers + tm.base;
        float x[MR_P];
#pragma unroll
        for (int r = 0; r < MR_P; ++r) x[r] = __ldg(lp + mm[r]);
        if (tm.op == OP_SQLIN) {
#pragma unroll
            for (int r = 0; r < MR_P; ++r) {
                acc[r] = __fmaf_rn(tm.a, __fmul_rn(x[r], x[r]), acc[r]);
                acc[r] = __fmaf_rn(tm.b, x[r], acc[r]);
            }
        } else if (tm.op == OP_EQ) {
#pragma unroll
            for (int r = 0; r < MR_P; ++r) acc[r] = (x[r] == tm.b) ? __fadd_rn(acc[r], tm.a) : acc[r];
        } else if (tm.op == OP_LIN) {
#pragma unroll
            for (int r = 0; r < MR_P; ++r) acc[r] = __fmaf_rn(tm.a, x[r], acc[r]);
        } else if (tm.op == OP_LINX) {
#pragma unroll
            for (int r = 0; r < MR_P; ++r) crs[r] = __fmaf_rn(tm.a, x[r], crs[r]);
        } else if (tm.op == OP_SQLINM) {
            const Term pl = sterm[t + 1];
#pragma unroll
            for (int r = 0; r < MR_P; ++r) {
                const bool in = !isnan(x[r]);
                const float x0 = in ? x[r] : 0.f;
                const float mk = in ? 1.f : 0.f;
                acc[r] = __fmaf_rn(tm.a, __fmul_rn(x0, x0), acc[r]);
                acc[r] = __fmaf_rn(tm.b, x0, acc[r]);
                acc[r] = __fmaf_rn(pl.a, mk, acc[r]);
                crs[r] = __fmaf_rn(pl.b, mk, crs[r]);
            }
            ++t;
        }
    }
}
}  // namespace

template <int KF, bool GEN>
__global__ void __launch_bounds__(256, KF <= 4 ? 4 : 2) k_map_records(MapArgs A) {
    extern __shared__ __align__(16) Term sterm[];
    __shared__ Slot ss;
    // smallest and largest layer offset of the terms; bit 0: a term that is not
    // OP_SQLIN, bit 1: one that the fast loop does not know
    __shared__ int s_lo, s_hi, s_ops;
    const int b = blockIdx.y;
    if (GEN && blockIdx.x == 0) {
        slot_generator(A.g, A.slots[b], b, A.gen, reinterpret_cast<unsigned *>(sterm));
        return;
    }
    const int part = int(blockIdx.x) - (GEN ? 1 : 0);
    griddep_wait();
    griddep_launch();
    const Term *src = A.terms + (long long)b * A.maxterms;
    // a thread's first term is read beside the slot (the slot's block of terms
    // is maxterms long; what lies beyond its own terms is not used)
    Term first;
    if ((int)threadIdx.x < A.maxterms) first = src[threadIdx.x];
    if (threadIdx.x == 0) {
        ss = A.slots[b];
        s_lo = INT_MAX;
        s_hi = INT_MIN;
        s_ops = 0;
    }
    __syncthreads();
    if (ss.flags & SLOT_SKIP) return;
    const int nt = ss.nterms;
    {
        int lo = INT_MAX, hi = INT_MIN, ops = 0;
        for (int t = threadIdx.x; t < nt; t += blockDim.x) {
            const Term tm = t < (int)blockDim.x ? first : src[t];
            sterm[t] = tm;
            lo = min(lo, tm.base);
            hi = max(hi, tm.base);
            ops |= (tm.op == OP_SQLIN ? 0 : 1) | (tm.op == OP_SQLIN || tm.op == OP_EQ || tm.op == OP_LIN ? 0 : 2);
        }
        lo = __reduce_min_sync(0xffffffffu, lo);
        hi = __reduce_max_sync(0xffffffffu, hi);
        ops = (int)__reduce_or_sync(0xffffffffu, (unsigned)ops);
        if ((threadIdx.x & 31) == 0 && lo <= hi) {
            atomicMin(&s_lo, lo);
            atomicMax(&s_hi, hi);
            if (ops) atomicOr(&s_ops, ops);
        }
    }
    __syncthreads();
    const bool all_sq = s_ops == 0, all_plain = s_ops < 2;

    const Geom &g = A.g;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, nwarps = blockDim.x >> 5;
    const bool emit_masked = (ss.flags & SLOT_EMIT_MASKED) != 0;
    const bool missing = (ss.flags & SLOT_MISSING) != 0;
    // a valid scan position used for address-safe dummy gathers
    unsigned usafe = 0;
    bool any_valid = true;
    for (int d = 0; d < g.nd; ++d) {
        usafe += (unsigned)(ss.lo[d] * g.sstride[d]);
        any_valid &= ss.lo[d] < g.fft[d];
    }
    const unsigned uN = (unsigned)g.N;

    const int seg_begin = part * A.segs_per_cta;
    const int seg_end = min(seg_begin + A.segs_per_cta, g.nseg);
    float *rv = A.rec_val + (long long)b * g.nseg * QSK_SEG;
    int *ri = A.rec_idx + (long long)b * g.nseg * QSK_SEG;
    float carry[KF];   // prefix top-KF of what this warp has seen
#pragma unroll
    for (int q = 0; q < KF; ++q) carry[q] = -CUDART_INF_F;

    for (int sg0 = seg_begin + MR_SEGS * warp; sg0 < seg_end; sg0 += MR_SEGS * nwarps) {
        const unsigned base = (unsigned)sg0 * QSK_SEG;
        // bit r: the position base + 32 r + lane lies inside the border
        unsigned vm = 0u;
        if (any_valid) {
#pragma unroll
            for (int r = 0; r < MR_P; ++r) {
                const unsigned m = base + 32 * r + lane;
                bool ok = m < uN;
                unsigned rest = m;
#pragma unroll
                for (int d = 0; d < QSK_MAXD; ++d)
                    if (d < g.nd) {
                        const unsigned q = fast_div(rest, A.div[d]);
                        ok &= (int)(rest - q * (unsigned)g.fft[d]) >= ss.lo[d];
                        rest = q;
                    }
                vm |= ok ? (1u << r) : 0u;
            }
        }
        float acc[MR_P];
#pragma unroll
        for (int r = 0; r < MR_P; ++r) acc[r] = 0.f;
        const unsigned vany = __reduce_or_sync(0xffffffffu, vm);
        if (vany) {
            const bool inside = (long long)base + s_lo >= 0 && (long long)base + (32 * MR_P - 1) + s_hi < A.layer_elems;
            if (inside && all_sq && !missing) {
                map_terms_fast<true>(sterm, nt, A.layers + base + lane, acc);
            } else if (inside && all_plain && !missing) {
                map_terms_fast<false>(sterm, nt, A.layers + base + lane, acc);
            } else {
                float crs[MR_P];
#pragma unroll
                for (int r = 0; r < MR_P; ++r) crs[r] = 0.f;
                map_terms_any(sterm, nt, A.layers, base + lane, vm, usafe, acc, crs);
                if (missing) {
                    // overlap masked by the centre, then -|S/c^4| (-inf where c == 0);
                    // positions outside the border are NaN in the reference
                    // (quantileSamplingModule.hpp:507-516, CPUThreadDevice.cpp:501-524)
#pragma unroll
                    for (int r = 0; r < MR_P; ++r) {
                        const bool v = (vm >> r) & 1u;
                        const float cm = v ? __ldg(A.layers + ss.cmask_base + (long long)(base + 32 * r + lane)) : 0.f;
                        const float c = __fmul_rn(crs[r], cm);
                        const float c4 = __fmul_rn(__fmul_rn(__fmul_rn(c, c), c), c);
                        float e = -fabsf(__fdiv_rn(acc[r], c4));
                        if (c == 0.f) e = -CUDART_INF_F;
                        acc[r] = e;
                    }
                }
            }
        }
        // verbatim exclusion (one index, or the radius mask): -inf written over
        // the map after the compensation, at masked positions too, where it
        // replaces the NaN border of a missing-data map
        // (quantileSamplingModule.hpp:518-523, CPUThreadDevice.cpp:310-342)
        unsigned hit = 0u;
        if (ss.excl >= 0) {
            const unsigned o = (unsigned)ss.excl - base - (unsigned)lane;   // 32 r for one lane of the span
            if ((o & 31u) == 0u && o < 32u * MR_P) hit = 1u << (o >> 5);
        }
        if (A.xmask) {
            const unsigned *xm = A.xmask + (long long)b * A.xwords;
#pragma unroll
            for (int r = 0; r < MR_P; ++r)
                if (base + 32 * r < uN) hit |= ((xm[(base >> 5) + r] >> lane) & 1u) << r;
        }
        // a masked position is an explicit record when the slot emits masked
        // entries, or when it is an excluded one of a missing-data map (-inf
        // instead of NaN); otherwise the replay counts it as an implicit -inf
#pragma unroll
        for (int s = 0; s < MR_SEGS; ++s) {
            const int sg = sg0 + s;
            if (sg >= seg_end) break;
            const unsigned sbase = base + s * QSK_SEG;
            float xv[4];
            float segmax = -CUDART_INF_F;
#pragma unroll
            for (int r = 0; r < 4; ++r) {
                const int q = 4 * s + r;
                xv[r] = ((hit >> q) & 1u)  ? -CUDART_INF_F
                        : ((vm >> q) & 1u) ? acc[q]
                                           : (missing ? CUDART_NAN_F : -CUDART_INF_F);
                segmax = fmaxf(segmax, xv[r]);
            }
#pragma unroll
            for (int off = 16; off > 0; off >>= 1) segmax = fmaxf(segmax, __shfl_xor_sync(0xffffffffu, segmax, off));
            int count = 0;
            if (!(segmax < carry[KF - 1])) {
                // warp prefix top-KF in scan order: records are the positions not
                // below the K-th best of everything before them (a superset of the
                // global triggers)
#pragma unroll
                for (int r = 0; r < 4; ++r) {
                    const int q = 4 * s + r;
                    const bool exists = sbase + 32 * r + lane < uN;
                    const float xval = xv[r];
                    const float kth0 = carry[KF - 1];
                    unsigned bal = __ballot_sync(0xffffffffu, exists && xval >= kth0);
                    if (bal == 0u) continue;
                    if (kth0 != -CUDART_INF_F && __popc(bal) <= 6) {
                        // finite candidates only, inserted in scan order
                        unsigned cand = bal;
                        while (cand) {
                            const int l = __ffs(cand) - 1;
                            cand &= cand - 1u;
                            const float y = __shfl_sync(0xffffffffu, xval, l);
                            if (y >= carry[KF - 1]) topk_insert<KF>(carry, y);
                            else bal &= ~(1u << l);
                        }
                    } else {
                        // a NaN score never compares true in the reservoir (fKb.hpp), so it
                        // is never a record and must not raise the prefix K-th best: it
                        // enters the scan as -inf (fminf/fmaxf would turn it into +inf)
                        float st[KF];
                        st[0] = isnan(xval) ? -CUDART_INF_F : xval;
#pragma unroll
                        for (int k = 1; k < KF; ++k) st[k] = -CUDART_INF_F;
#pragma unroll
                        for (int off = 1; off < 32; off <<= 1) {
                            float rcv[KF], mrg[KF];
#pragma unroll
                            for (int k = 0; k < KF; ++k) rcv[k] = __shfl_up_sync(0xffffffffu, st[k], off);
                            if (lane >= off) {
                                topk_merge<KF>(st, rcv, mrg);
#pragma unroll
                                for (int k = 0; k < KF; ++k) st[k] = mrg[k];
                            }
                        }
                        float ex[KF], pre[KF];
#pragma unroll
                        for (int k = 0; k < KF; ++k) {
                            const float y = __shfl_up_sync(0xffffffffu, st[k], 1);
                            ex[k] = lane == 0 ? -CUDART_INF_F : y;
                        }
                        topk_merge<KF>(carry, ex, pre);
                        const bool rec = exists && xval >= pre[KF - 1] &&
                                         (((vm >> q) & 1u) || emit_masked || (((hit >> q) & 1u) && missing));
                        bal = __ballot_sync(0xffffffffu, rec);
                        float last[KF], nc[KF];
#pragma unroll
                        for (int k = 0; k < KF; ++k) last[k] = __shfl_sync(0xffffffffu, st[k], 31);
                        topk_merge<KF>(carry, last, nc);
#pragma unroll
                        for (int k = 0; k < KF; ++k) carry[k] = nc[k];
                    }
                    if ((bal >> lane) & 1u) {
                        const unsigned o = sbase + count + __popc(bal & lanemask_lt());
                        rv[o] = xval;
                        ri[o] = int(sbase + 32 * r + lane);
                    }
                    count += __popc(bal);
                }
            }
            if (lane == 0) {
                A.rec_cnt[(long long)b * g.nseg + sg] = count;
                A.rec_max[(long long)b * g.nseg + sg] = segmax;
            }
        }
    }
}

// ---------------------------------------------------------------------------
// replay of the k-biggest scan + draw + write-back; one CTA per slot
// ---------------------------------------------------------------------------
#define RP_WARPS 4            // slots (warps) per CTA of k_mt_prep
#define RP_TEAM 8             // warps of one slot's team
#define RP_THREADS (32 * RP_TEAM)
#define REC_CAP 2048          // records staged at once
#define RNG_BUF (2 * REC_CAP + 640)   // two draws per staged record + one block
#define SEG_AHEAD 4           // windows of one segment per thread read at once

struct __align__(16) ReplayShared {
    // staged records in scan order, a segment's padded to a multiple of four
    // with NaN (which no comparison takes for a record), and their scan indices
    float rv_s[REC_CAP];
    int ri_s[REC_CAP];
    unsigned mt[2][624];      // generator state, the next block written beside the last
    float buf[RNG_BUF];       // draws
    float w_top[RP_TEAM][QSK_KMAX];   // per warp: top-K of its part
    int w_sum[RP_TEAM];       // per warp: records to stage, or ties
    int4 w_fun[RP_TEAM];      // per warp: cpt function and draws of its part
    int w_map[RP_TEAM][QSK_KMAX];     // per warp: slot map of its part
    int stop, staged;         // first thread whose segment did not fit, records staged
};

// The next MT19937 block by the team, written beside the last one (the
// recurrence reaches back 624, 623 and 227 words, so 227 words are
// independent of one another): three phases, one barrier after each; with
// OUT, draw k of the block goes to out[k].
template <bool OUT>
__device__ __forceinline__ void mt_block(const unsigned *old, unsigned *nw, int tid, float *out) {
    auto put = [&](int k, unsigned y) {
        nw[k] = y;
        if (OUT) out[k] = mt_unit(mt_temper(y));
    };
    static_assert(RP_THREADS >= 227, "one word per thread and phase");
    if (tid < 227) put(tid, mt_mix(old[tid], old[tid + 1], old[tid + 397]));
    __syncthreads();
    if (tid < 227) put(227 + tid, mt_mix(old[227 + tid], old[228 + tid], nw[tid]));
    __syncthreads();
    if (tid < 170) put(454 + tid, mt_mix(old[454 + tid], tid < 169 ? old[455 + tid] : nw[0], nw[227 + tid]));
    __syncthreads();
}

// A slot's draws: buf[rp, len) unread, the state in mt[par]; every thread of
// the team holds the same values.
struct Rng {
    int rp = 0, len = 0, par = 0;
};

// at least `need` (<= 2 * REC_CAP) unread draws in the buffer
__device__ __forceinline__ void rng_need(ReplayShared &w, int tid, Rng &g, int need) {
    if (g.len - g.rp >= need) return;
    __syncthreads();   // every thread has read the draws it took so far
    const int unread = g.len - g.rp;
    // the unread ones to the front (destinations never overtake sources)
    for (int at = 0; at < unread && g.rp > 0; at += 4 * RP_THREADS) {
        float v[4];
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            const int i = at + q * RP_THREADS + tid;
            v[q] = i < unread ? w.buf[g.rp + i] : 0.f;
        }
        __syncthreads();
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            const int i = at + q * RP_THREADS + tid;
            if (i < unread) w.buf[i] = v[q];
        }
        __syncthreads();
    }
    g.rp = 0;
    g.len = unread;
    while (g.len < need) {
        mt_block<true>(w.mt[g.par], w.mt[g.par ^ 1], tid, w.buf + g.len);
        g.par ^= 1;
        g.len += 624;
    }
}

// advance the stream by n draws; whole blocks only regenerate the state
__device__ __forceinline__ void rng_skip(ReplayShared &w, int tid, Rng &g, long long n) {
    const long long avail = g.len - g.rp;
    if (n <= avail) {
        g.rp += int(n);
        return;
    }
    n -= avail;
    g.rp = g.len = 0;
    for (; n > 624; n -= 624) {
        mt_block<false>(w.mt[g.par], w.mt[g.par ^ 1], tid, nullptr);
        g.par ^= 1;
    }
    rng_need(w, tid, g, 1);
    g.rp += int(n);
}

template <int KM>
__device__ __forceinline__ float sel_f(const float (&a)[KM], int i) {
    float r = a[0];
#pragma unroll
    for (int s = 1; s < KM; ++s) r = (s == i) ? a[s] : r;
    return r;
}
template <int KM>
__device__ __forceinline__ int sel_i(const int (&a)[KM], int i) {
    int r = a[0];
#pragma unroll
    for (int s = 1; s < KM; ++s) r = (s == i) ? a[s] : r;
    return r;
}
template <int KM>
__device__ __forceinline__ unsigned sel_u(const unsigned (&a)[KM], int i) {
    unsigned r = a[0];
#pragma unroll
    for (int s = 1; s < KM; ++s) r = (s == i) ? a[s] : r;
    return r;
}

// One trigger of the reference's scan (fKb.hpp): a value v >= the K-th draws x
// among the xes tail slots holding the K-th and swaps it with slot K-1; above
// the K-th it is inserted after the values >= v (the last slot drops out, cpt
// restarts at 0 when the K-th was unique and counts on otherwise); equal to
// the K-th it replaces slot K-1 with probability xes / (xes + cpt + 1) (a
// second draw) and cpt counts on.  `slot` are the K positions, or a map of
// slots (T int, an index i entering as -(i + 1)); returns the draws used.
template <int KM, class T>
__device__ __forceinline__ int replay_trigger(int K, float v, T entry, float (&cv)[KM], T (&slot)[KM], unsigned &cpt,
                                              const float *u) {
    const float kth = sel_f<KM>(cv, K - 1);
    const bool gt = v > kth;
    int xes = 0, q = 0;
#pragma unroll
    for (int s = 0; s < KM; ++s) {
        if (s < K && cv[s] == kth) xes++;
        if (s < K - 1 && cv[s] >= v) q++;
    }
    int x = K - xes + int(floorf(__fmul_rn(u[0], (float)xes)));
    if (x > K - 1) x = K - 1;
    T px = slot[0], pk = slot[0];
#pragma unroll
    for (int s = 1; s < KM; ++s) {
        px = s == x ? slot[s] : px;
        pk = s == K - 1 ? slot[s] : pk;
    }
    T sw[KM];
#pragma unroll
    for (int s = 0; s < KM; ++s) sw[s] = (s == x) ? pk : ((s == K - 1) ? px : slot[s]);
    if (gt) {
#pragma unroll
        for (int s = 0; s < KM; ++s)
            if (s < K) slot[s] = s < q ? sw[s] : (s == q ? entry : sw[s > 0 ? s - 1 : 0]);
        topk_insert<KM>(cv, v);
        cpt = (xes == 1) ? 0u : cpt + 1u;
        return 1;
    }
    cpt += 1u;
    const bool write = __fmul_rn(__uint2float_rn(unsigned(xes) + cpt), u[1]) < (float)xes;
#pragma unroll
    for (int s = 0; s < KM; ++s)
        if (s < K) slot[s] = (write && s == K - 1) ? entry : sw[s];
    return 2;
}

// The position updates of a run: every thread's slot map o, composed in thread
// order (each warp's to its lane 0, then the warps'), applied to cp.
template <int KM>
__device__ __forceinline__ void compose_maps(ReplayShared &w, int tid, int (&o)[KM], unsigned (&cp)[KM]) {
    const unsigned FULL = 0xffffffffu;
    const int lane = tid & 31, wid = tid >> 5;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
        int later[KM];
#pragma unroll
        for (int k = 0; k < KM; ++k) later[k] = __shfl_down_sync(FULL, o[k], d);
        if ((lane & (2 * d - 1)) == 0) {
            int c[KM];
#pragma unroll
            for (int k = 0; k < KM; ++k) c[k] = later[k] < 0 ? later[k] : sel_i<KM>(o, later[k]);
#pragma unroll
            for (int k = 0; k < KM; ++k) o[k] = c[k];
        }
    }
    if (lane == 0) {
#pragma unroll
        for (int k = 0; k < KM; ++k) w.w_map[wid][k] = o[k];
    }
    __syncthreads();
#pragma unroll
    for (int k = 0; k < KM; ++k) o[k] = k;
    for (int q = 0; q < RP_TEAM; ++q) {
        int c[KM];
#pragma unroll
        for (int k = 0; k < KM; ++k) {
            const int later = w.w_map[q][k];
            c[k] = later < 0 ? later : sel_i<KM>(o, later);
        }
#pragma unroll
        for (int k = 0; k < KM; ++k) o[k] = c[k];
    }
    unsigned np[KM];
#pragma unroll
    for (int k = 0; k < KM; ++k) np[k] = o[k] < 0 ? unsigned(-(o[k] + 1)) : sel_u<KM>(cp, o[k]);
#pragma unroll
    for (int k = 0; k < KM; ++k) cp[k] = np[k];
}

// The staged records [r, n) when none exceeds the K-th value V of a full
// state: the state's values stay as they are and every record equal to V is a
// tie (two draws, cpt + 1, a swap inside the xes tail slots that hold V and a
// possible replacement at K-1).  Thread t takes P consecutive records; ties
// are ranked by a scan over the team.
template <int KM>
__device__ __forceinline__ void team_ties(ReplayShared &w, int tid, int r, int n, int K, const float (&cv)[KM],
                                          unsigned (&cp)[KM], unsigned &cpt, Rng &g) {
    const unsigned FULL = 0xffffffffu;
    const int lane = tid & 31, wid = tid >> 5;
    const float V = sel_f<KM>(cv, K - 1);
    int xes = 0;
#pragma unroll
    for (int q = 0; q < KM; ++q) xes += (q < K && cv[q] == V) ? 1 : 0;
    // P odd keeps a warp's reads on distinct banks; P <= REC_CAP / RP_THREADS + 1 bits
    const int P = ((n - r + RP_THREADS - 1) / RP_THREADS) | 1;
    const int j0 = min(n, r + tid * P), j1 = min(n, j0 + P);
    unsigned tm = 0u;
#pragma unroll 1
    for (int j = j0; j < j1; ++j) tm |= unsigned(w.rv_s[j] == V) << (j - j0);
    const int mine = __popc(tm);
    int incl = mine;
#pragma unroll
    for (int off = 1; off < 32; off <<= 1) {
        const int y = __shfl_up_sync(FULL, incl, off);
        if (lane >= off) incl += y;
    }
    if (lane == 31) w.w_sum[wid] = incl;
    __syncthreads();
    int before = 0, total = 0;
#pragma unroll
    for (int q = 0; q < RP_TEAM; ++q) {
        const int t = w.w_sum[q];
        before += q < wid ? t : 0;
        total += t;
    }
    if (total == 0) return;
    rng_need(w, tid, g, 2 * total);
    int o[KM];
#pragma unroll
    for (int k = 0; k < KM; ++k) o[k] = k;
    int rank = before + incl - mine;
    const float fx = (float)xes;
    while (tm) {
        const int j = j0 + __ffs(tm) - 1;
        tm &= tm - 1u;
        const float u1 = w.buf[g.rp + 2 * rank], u2 = w.buf[g.rp + 2 * rank + 1];
        int x = K - xes + int(floorf(__fmul_rn(u1, fx)));
        if (x > K - 1) x = K - 1;
        const unsigned after = cpt + unsigned(rank) + 1u;
        const bool write = __fmul_rn(__uint2float_rn(unsigned(xes) + after), u2) < fx;
        const int ox = sel_i<KM>(o, x), ok1 = sel_i<KM>(o, K - 1);
        const int wr = -(w.ri_s[j] + 1);
#pragma unroll
        for (int k = 0; k < KM; ++k) {
            if (k == x) o[k] = ok1;
            if (k == K - 1) o[k] = write ? wr : ox;
        }
        ++rank;
    }
    compose_maps<KM>(w, tid, o, cp);
    cpt += unsigned(total);
    g.rp += 2 * total;
}

// The scan over the staged records [r, n) by the whole team, thread t taking P
// consecutive ones.  What a record does follows from prefixes: the K-th best
// before it (a top-K scan), its draws (a count) and cpt (a composition of
// "add" / "reset" functions); the position updates are slot maps, composed
// in record order.  Three walks over a thread's records, one scan over the
// team after each of the first two, a reduction of the maps after the third.
// The state (cv, cp, cpt) is replicated in every thread.
template <int KM>
__device__ __forceinline__ void team_scan(ReplayShared &w, int tid, int r, int n, int K, float (&cv)[KM],
                                          unsigned (&cp)[KM], unsigned &cpt, Rng &g) {
    const unsigned FULL = 0xffffffffu;
    const int lane = tid & 31, wid = tid >> 5;
    // P odd keeps a warp's reads on distinct banks
    const int P = ((n - r + RP_THREADS - 1) / RP_THREADS) | 1;
    const int j0 = min(n, r + tid * P), j1 = min(n, j0 + P);
    // 1. the K best before this thread's records
    float pre[KM];
    float top = -CUDART_INF_F;
    {
        float st[KM];
#pragma unroll
        for (int k = 0; k < KM; ++k) st[k] = -CUDART_INF_F;
#pragma unroll 1
        for (int j = j0; j < j1; ++j) {
            const float v = w.rv_s[j];
            topk_insert<KM>(st, isnan(v) ? -CUDART_INF_F : v);
        }
        top = st[0];
#pragma unroll
        for (int off = 1; off < 32; off <<= 1) {
            float rcv[KM], mrg[KM];
#pragma unroll
            for (int k = 0; k < KM; ++k) rcv[k] = __shfl_up_sync(FULL, st[k], off);
            if (lane >= off) {
                topk_merge<KM>(st, rcv, mrg);
#pragma unroll
                for (int k = 0; k < KM; ++k) st[k] = mrg[k];
            }
        }
        if (lane == 31) {
#pragma unroll
            for (int k = 0; k < KM; ++k) w.w_top[wid][k] = st[k];
        }
#pragma unroll
        for (int k = 0; k < KM; ++k) {
            const float y = __shfl_up_sync(FULL, st[k], 1);
            pre[k] = lane == 0 ? -CUDART_INF_F : y;
        }
        __syncthreads();
        float e[KM], mrg[KM];
        topk_merge<KM>(pre, cv, mrg);
#pragma unroll
        for (int k = 0; k < KM; ++k) pre[k] = mrg[k];
        for (int q = 0; q < RP_TEAM; ++q) {
#pragma unroll
            for (int k = 0; k < KM; ++k) e[k] = w.w_top[q][k];
            if (q < wid) {
                topk_merge<KM>(pre, e, mrg);
#pragma unroll
                for (int k = 0; k < KM; ++k) pre[k] = mrg[k];
            }
            topk_merge<KM>(cv, e, mrg);   // the state after the run
#pragma unroll
            for (int k = 0; k < KM; ++k) cv[k] = mrg[k];
        }
    }
    // 2. this thread's draws and cpt function c -> fr ? fa : c + fa
    const bool active = j0 < j1 && top >= sel_f<KM>(pre, K - 1);
    int nd = 0, fr = 0, fa = 0;
    if (active) {
        float st[KM];
#pragma unroll
        for (int k = 0; k < KM; ++k) st[k] = pre[k];
#pragma unroll 1
        for (int j = j0; j < j1; ++j) {
            const float v = w.rv_s[j];
            const float kth = sel_f<KM>(st, K - 1);
            if (!(v >= kth)) continue;
            if (v > kth) {
                int xes = 0;
#pragma unroll
                for (int k = 0; k < KM; ++k) xes += (k < K && st[k] == kth) ? 1 : 0;
                nd += 1;
                fr = xes == 1 ? 1 : fr;
                fa = xes == 1 ? 0 : fa + 1;
                topk_insert<KM>(st, v);
            } else {
                nd += 2;
                fa += 1;
            }
        }
    }
    int id = nd, ir = fr, ia = fa;
#pragma unroll
    for (int off = 1; off < 32; off <<= 1) {
        const int dd = __shfl_up_sync(FULL, id, off), rr = __shfl_up_sync(FULL, ir, off), ra = __shfl_up_sync(FULL, ia, off);
        if (lane >= off) {
            id += dd;
            if (!ir) {   // earlier (rr, ra) then later (0, ia)
                ir = rr;
                ia += ra;
            }
        }
    }
    if (lane == 31) w.w_fun[wid] = make_int4(id, ir, ia, 0);
    int ed = __shfl_up_sync(FULL, id, 1), er = __shfl_up_sync(FULL, ir, 1), ea = __shfl_up_sync(FULL, ia, 1);
    if (lane == 0) ed = er = ea = 0;
    __syncthreads();
    int total = 0;
    unsigned mycpt = cpt;   // before this thread's records
    {
        unsigned cur = cpt;
#pragma unroll
        for (int q = 0; q < RP_TEAM; ++q) {
            const int4 f = w.w_fun[q];
            if (q == wid) {
                ed += total;
                mycpt = er ? unsigned(ea) : cur + unsigned(ea);
            }
            cur = f.y ? unsigned(f.z) : cur + unsigned(f.z);
            total += f.x;
        }
        cpt = cur;
    }
    if (total == 0) return;   // nothing reaches the K-th
    rng_need(w, tid, g, total);
    // 3. this thread's slot map
    int o[KM];
#pragma unroll
    for (int k = 0; k < KM; ++k) o[k] = k;
    if (nd > 0) {
        const float *u = w.buf + g.rp + ed;
#pragma unroll 1
        for (int j = j0; j < j1; ++j) {
            const float v = w.rv_s[j];
            if (!(v >= sel_f<KM>(pre, K - 1))) continue;
            u += replay_trigger<KM, int>(K, v, -(w.ri_s[j] + 1), pre, o, mycpt, u);
        }
    }
    compose_maps<KM>(w, tid, o, cp);
    g.rp += total;
}

// the cell of a slot without neighbours (one thread)
__device__ unsigned marginal_cell(const ReplayArgs &A, const Slot &s) {
    // marginal draw over the TI cells (simulation.hpp:586-605; complete TI)
    unsigned chosen_cell = unsigned(int(floor((double)__fmul_rn(s.seed, __uint2float_rn((unsigned)A.ti_cells)))));
    // float rounding of seed*cells can reach `cells` only for grids above 2^24 cells
    if ((long long)chosen_cell >= A.ti_cells) chosen_cell = (unsigned)(A.ti_cells - 1);
    if (A.complete_prefix) {
        bool hasNaN = false;
        for (int v = 0; v < A.nvar; ++v) hasNaN |= isnan(A.ti[(long long)chosen_cell * A.nvar + v]);
        if (hasNaN) {
            // NaN-safe draw (simulation.hpp:616-652): the first cell whose
            // running count of complete cells reaches floor(seed*(complete/nvar))*nvar
            const unsigned complete = (unsigned)A.complete_prefix[A.ti_cells - 1];
            const unsigned pos2 = unsigned(int(floor((double)__fmul_rn(
                                      s.seed, __uint2float_rn(complete / (unsigned)A.nvar))))) *
                                  (unsigned)A.nvar;
            long long lo2 = 0, hi2 = A.ti_cells;   // first index with prefix >= pos2
            while (lo2 < hi2) {
                long long mid = (lo2 + hi2) >> 1;
                if ((unsigned)A.complete_prefix[mid] < pos2) lo2 = mid + 1;
                else hi2 = mid;
            }
            chosen_cell = (unsigned)(lo2 < A.ti_cells ? lo2 : A.ti_cells - 1);
        }
    }
    return chosen_cell;
}

// write-back of a slot's draw (one thread)
__device__ __forceinline__ void replay_write(const ReplayArgs &A, const Slot &s, unsigned chosen_cell) {
    if (A.node_cell) A.node_cell[s.node] = chosen_cell;
    if (A.full) {
        // -fs: the node's variable only (simulation.hpp:1016-1024)
        const long long val = (long long)s.cell * A.nvar + s.var;
        if (A.state && isnan(A.state[val])) A.state[val] = A.ti[(long long)chosen_cell * A.nvar + s.var];
        if (A.id_image) A.id_image[val] = chosen_cell * A.nti + A.ti_id;
    } else {
        if (A.state) {
            for (int v = 0; v < A.nvar; ++v) {
                float *dst = A.state + (long long)s.cell * A.nvar + v;
                if (isnan(*dst)) *dst = A.ti[(long long)chosen_cell * A.nvar + v];
            }
        }
        if (A.id_image) A.id_image[s.cell] = chosen_cell * A.nti + A.ti_id;
    }
}

__device__ __forceinline__ void cp_async16(void *smem_dst, const void *gmem_src) {
    const unsigned d = (unsigned)__cvta_generic_to_shared(smem_dst);
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(d), "l"(gmem_src) : "memory");
}
__device__ __forceinline__ void cp_async_wait_all() { asm volatile("cp.async.wait_all;\n" ::: "memory"); }

// The k best of one slot, one CTA: the reference's findKBiggest replayed over
// the map's records in scan order.
//
// Windows of one segment per thread are filtered by the whole team: a segment
// can hold a candidate only if its maximum reaches the K-th best of the state
// and of the window's earlier segment maxima (a lower bound of the K-th at
// its turn).  The records of the segments left, a few dozen on a continuous
// map, thousands where most positions tie, go to shared memory in scan order
// and the team scans them from there (team_scan).  What bounds a slot is the
// chain of global reads (two or three per 1024 segments), of barriers, and
// the draws.  Every thread runs the same control flow.  Against one warp
// that read each candidate segment on its own and replayed 32 records a step
// (mean of a level, launch to end): a 200x200 continuous simulation (n = 50)
// 47 -> 14 us, categorical 101x90 (n = 20) 40 -> 25 us, 250x250 -> 500x500
// (n = 80) 65 -> 54 us; then with 16-byte staging copies, tie runs of their own
// (team_ties) and three CTAs of 80 registers per SM the slots of the last two
// took 54 k -> 35 k and 83 k -> 50 k cycles.  One slot of 26,000 segments takes
// 64 us; 559 in the old form, most of them the generator blocks of its first
// masked stretch, which now run beside the map (GenArgs).
template <int KM>
__global__ void __launch_bounds__(RP_THREADS, KM <= 4 ? 3 : 1) k_replay(ReplayArgs A) {
    __shared__ ReplayShared w;
    constexpr int NT = RP_THREADS;
    const unsigned FULL = 0xffffffffu;
    const int tid = threadIdx.x, wid = tid >> 5, lane = tid & 31;
    const int b = blockIdx.x;
    // the slot and its generator state come from kernels that had completed
    // when the map let this grid launch; everything else is read below
    const Slot &sl = A.slots[b];
    const int flags = sl.flags;
    // only_flagged: the slots the hash select leaves (fewer valid positions
    // than k)
    if (A.only_flagged && (flags & (SLOT_SKIP | SLOT_EMIT_MASKED)) != SLOT_EMIT_MASKED) return;
    const Geom &g = A.g;
    if (flags & SLOT_SKIP) {
        griddep_wait();
        if (tid != 0 || !(A.state || A.node_cell)) return;
        replay_write(A, sl, marginal_cell(A, sl));
        return;
    }
    const Slot &s = sl;
    const int K = s.K;
    Rng rng;
    // generator state: seeded here, or prepared by k_mt_prep together with
    // the blocks that the first masked stretch of the scan skips
    long long preskip = 0;
    if (A.mt_state) {
        // 156 16-byte copies (state rows and w.mt are 16-byte aligned), awaited
        // with the first records
        for (int q = tid; q < 156; q += NT) cp_async16(&w.mt[0][4 * q], A.mt_state + (long long)b * 624 + 4 * q);
        preskip = skipped_draws(A.mt_pre[b]);
    } else if (tid == 0) {
        mt_seed(w.mt[0], s.seed);
    }
    float cv[KM];
    unsigned cp[KM];
#pragma unroll
    for (int q = 0; q < KM; ++q) { cv[q] = -CUDART_INF_F; cp[q] = 0xffffffffu; }
    unsigned cpt = 0;
    long long last = -1;
    griddep_wait();
    griddep_launch();
    const bool emit_masked = (flags & (SLOT_EMIT_MASKED | SLOT_MISSING)) != 0;
    long long first_valid = 0;
    for (int d = 0; d < g.nd; ++d) first_valid += (long long)s.lo[d] * g.sstride[d];
    const float *rv = A.rec_val + (long long)b * g.nseg * QSK_SEG;
    const int *ri = A.rec_idx + (long long)b * g.nseg * QSK_SEG;
    const int *rc = A.rec_cnt + (long long)b * g.nseg;
    const float *rm = A.rec_max + (long long)b * g.nseg;

    int sg = 0;
    while (sg < g.nseg) {
        int c[SEG_AHEAD];
        float m[SEG_AHEAD];
#pragma unroll
        for (int i = 0; i < SEG_AHEAD; ++i) {
            const int q = sg + i * NT + tid;
            c[i] = q < g.nseg ? rc[q] : 0;
            m[i] = q < g.nseg ? rm[q] : -CUDART_INF_F;
        }
        // (one copy of the loop's code; the selects cost less than its fetches)
#pragma unroll 1
        for (int i = 0; i < SEG_AHEAD; ++i) {
            const int q0 = sg + i * NT;
            if (q0 >= g.nseg) break;
            int ci = sel_i<SEG_AHEAD>(c, i);
            const float mx = sel_f<SEG_AHEAD>(m, i);
            for (;;) {   // until the window's segments are staged and scanned
                const float kth = sel_f<KM>(cv, K - 1);
                if (!__syncthreads_or(ci > 0 && mx >= kth)) break;
                bool fl = ci > 0 && mx >= kth;
                // (a state that is not full takes the general scan)
                const bool above = __syncthreads_or(fl && (mx > kth || kth == -CUDART_INF_F));
                if (above) {
                    // K-th best of the state and the earlier segments of the window
                    float st[KM], pre[KM];
                    st[0] = ci > 0 ? mx : -CUDART_INF_F;
#pragma unroll
                    for (int k = 1; k < KM; ++k) st[k] = -CUDART_INF_F;
#pragma unroll
                    for (int off = 1; off < 32; off <<= 1) {
                        float rcv[KM], mrg[KM];
#pragma unroll
                        for (int k = 0; k < KM; ++k) rcv[k] = __shfl_up_sync(FULL, st[k], off);
                        if (lane >= off) {
                            topk_merge<KM>(st, rcv, mrg);
#pragma unroll
                            for (int k = 0; k < KM; ++k) st[k] = mrg[k];
                        }
                    }
                    if (lane == 31) {
#pragma unroll
                        for (int k = 0; k < KM; ++k) w.w_top[wid][k] = st[k];
                    }
#pragma unroll
                    for (int k = 0; k < KM; ++k) {
                        const float y = __shfl_up_sync(FULL, st[k], 1);
                        pre[k] = lane == 0 ? -CUDART_INF_F : y;
                    }
                    __syncthreads();
                    float mrg[KM], e[KM];
                    topk_merge<KM>(pre, cv, mrg);
#pragma unroll
                    for (int k = 0; k < KM; ++k) pre[k] = mrg[k];
                    for (int q = 0; q < wid; ++q) {
#pragma unroll
                        for (int k = 0; k < KM; ++k) e[k] = w.w_top[q][k];
                        topk_merge<KM>(pre, e, mrg);
#pragma unroll
                        for (int k = 0; k < KM; ++k) pre[k] = mrg[k];
                    }
                    fl = fl && mx >= sel_f<KM>(pre, K - 1);
                }
                const int cnt = fl ? (ci + 3) & ~3 : 0;   // padded
                int incl = cnt;
#pragma unroll
                for (int off = 1; off < 32; off <<= 1) {
                    const int y = __shfl_up_sync(FULL, incl, off);
                    if (lane >= off) incl += y;
                }
                if (lane == 31) w.w_sum[wid] = incl;
                if (tid == 0) w.stop = INT_MAX;
                __syncthreads();
                int before = 0, all = 0;
#pragma unroll
                for (int q = 0; q < RP_TEAM; ++q) {
                    const int t = w.w_sum[q];
                    before += q < wid ? t : 0;
                    all += t;
                }
                const int dst = before + incl - cnt;
                const bool take = fl && dst + cnt <= REC_CAP;
                if (fl && !take) atomicMin(&w.stop, tid);
                // the segments' records in 16-byte copies (a segment's start on
                // 512 bytes), one segment of the warp after the other: the lower
                // lanes the values, the upper ones the indices
                unsigned todo = __ballot_sync(FULL, take);
                while (todo) {
                    const int l = __ffs(todo) - 1;
                    todo &= todo - 1u;
                    const int n = __shfl_sync(FULL, cnt, l), d = __shfl_sync(FULL, dst, l);
                    const long long from = (long long)(q0 + 32 * wid + l) * QSK_SEG;
                    for (int k = 4 * (lane & 15); k < n; k += 64) {
                        if (lane < 16) cp_async16(&w.rv_s[d + k], rv + from + k);
                        else cp_async16(&w.ri_s[d + k], ri + from + k);
                    }
                }
                cp_async_wait_all();
                __syncthreads();
                if (take)
                    for (int k = ci; k < cnt; ++k) w.rv_s[dst + k] = CUDART_NAN_F;
                __syncthreads();
                const int stop = w.stop;
                int n = all;
                if (stop != INT_MAX) {
                    if (stop == tid) w.staged = dst;
                    __syncthreads();
                    n = w.staged;
                }
                // while fewer than K finite values have been seen the masked
                // positions between two records are -inf ties: two draws and
                // one cpt increment each, no visible slot change
                int r = 0;
                while (!emit_masked && r < n && sel_f<KM>(cv, K - 1) == -CUDART_INF_F) {
                    const float v = w.rv_s[r];
                    if (isnan(v)) {
                        ++r;
                        continue;
                    }
                    const int mm = w.ri_s[r];
                    // (the first record is the first valid position as a rule:
                    // all before it are masked)
                    long long gap = mm - (last + 1);
                    if (gap > 0 && !(last < 0 && mm == first_valid))
                        gap -= valid_prefix(g, s.lo, mm) - (last < 0 ? 0 : valid_prefix(g, s.lo, last + 1));
                    if (gap > 0) {
                        // the first skip covers the prepared blocks (gap >= the masked
                        // positions before the first valid one, so 2 gap > preskip)
                        rng_skip(w, tid, rng, 2 * gap - preskip);
                        preskip = 0;
                        cpt += unsigned(gap);
                    }
                    rng_need(w, tid, rng, 2);
                    rng.rp += replay_trigger<KM, unsigned>(K, v, unsigned(mm), cv, cp, cpt, w.buf + rng.rp);
                    last = mm;
                    ++r;
                }
                if (r < n) {
                    if (above) team_scan<KM>(w, tid, r, n, K, cv, cp, cpt, rng);
                    else team_ties<KM>(w, tid, r, n, K, cv, cp, cpt, rng);
                }
                if (stop == INT_MAX) break;
                if (tid < stop) ci = 0;   // done; the rest of the window once more
            }
        }
        sg += SEG_AHEAD * NT;
    }
    cp_async_wait_all();
    if (wid != 0) return;
    // merge loop (quantileSamplingModule.hpp:546-557): repeated first-max extraction
    float fv[KM];
    unsigned fp[KM];
#pragma unroll
    for (int j = 0; j < KM; ++j) {
        fv[j] = -CUDART_INF_F;
        fp[j] = 0xffffffffu;
        if (j < K) {
            int best = 0;
            float bv = cv[0];
#pragma unroll
            for (int l2 = 1; l2 < KM; ++l2)
                if (l2 < K && cv[l2] > bv) { best = l2; bv = cv[l2]; }
            fv[j] = bv;
            fp[j] = sel_u<KM>(cp, best);
#pragma unroll
            for (int l2 = 0; l2 < KM; ++l2)
                if (l2 == best) cv[l2] = -CUDART_INF_F;
        }
    }
    // sample(): std::sort by score — insertion sort (stable) for K <= 16
#pragma unroll
    for (int a2 = 1; a2 < KM; ++a2) {
        if (a2 < K) {
#pragma unroll
            for (int c = a2; c > 0; --c) {
                if (fv[c] > fv[c - 1]) {
                    float tv = fv[c]; fv[c] = fv[c - 1]; fv[c - 1] = tv;
                    unsigned tp = fp[c]; fp[c] = fp[c - 1]; fp[c - 1] = tp;
                }
            }
        }
    }
    if (lane == 0 && A.out_val) {
#pragma unroll
        for (int j = 0; j < KM; ++j)
            if (j < K) {
                unsigned out = fp[j];
                if (A.out_cells) {
                    // cvtIndexToPosition (CPUThreadDevice.cpp:257-268)
                    unsigned position = 0, div = (unsigned)g.N;
                    for (int d = g.nd - 1; d >= 0; --d) {
                        unsigned f = (unsigned)g.fft[d], sr = (unsigned)g.src[d];
                        div /= f;
                        position = position * sr + ((f - (out / div) % f - (unsigned)s.mn[d] - 1u) + sr) % sr;
                    }
                    out = position;
                }
                A.out_val[(long long)b * K + j] = fv[j];
                A.out_pos[(long long)b * K + j] = out;
            }
    }
    if (!(A.state || A.node_cell)) return;
    // cvtIndexToPosition (CPUThreadDevice.cpp:257-268), unsigned arithmetic
    unsigned index = sel_u<KM>(fp, s.sel);
    unsigned position = 0;
    unsigned div = (unsigned)g.N;
    for (int d = g.nd - 1; d >= 0; --d) {
        unsigned f = (unsigned)g.fft[d], sr = (unsigned)g.src[d];
        div /= f;
        position = position * sr + ((f - (index / div) % f - (unsigned)s.mn[d] - 1u) + sr) % sr;
    }
    if (lane == 0) replay_write(A, s, position);
}

// ---------------------------------------------------------------------------
// k best with hash tie-breaks over the map's records (the draw rule of the
// tensor-core form, for the nodes it leaves to the plain map).  Every position
// scoring at least the k-th best is a record (the filter keeps ties), so the
// k largest (score, tie hash) over the records are the k largest over the map.
// One CTA per slot; slots with SLOT_EMIT_MASKED are left to the replay
// (only_flagged).
// ---------------------------------------------------------------------------
namespace {
template <int W>
__device__ __forceinline__ void hs_insert(unsigned long long (&k)[W], unsigned (&p)[W], unsigned long long key,
                                          unsigned pos) {
    k[0] = key;
    p[0] = pos;
#pragma unroll
    for (int i = 0; i + 1 < W; ++i) {
        const bool sw = k[i] > k[i + 1];
        const unsigned long long a = k[i], c = k[i + 1];
        const unsigned pa = p[i], pc = p[i + 1];
        k[i] = sw ? c : a;
        k[i + 1] = sw ? a : c;
        p[i] = sw ? pc : pa;
        p[i + 1] = sw ? pa : pc;
    }
}
__device__ __forceinline__ unsigned hs_ordered(float f) {
    if (f != f) return 0u;
    const unsigned u = __float_as_uint(f);
    return (u & 0x80000000u) ? ~u : (u | 0x80000000u);
}
}  // namespace

constexpr int HS_THREADS = 256;
template <int KM>
__global__ void __launch_bounds__(HS_THREADS) k_hash_select(ReplayArgs A) {
    __shared__ unsigned long long sk[HS_THREADS * KM];
    __shared__ unsigned sp[HS_THREADS * KM];
    const int b = blockIdx.x;
    if (b >= A.nslots) return;
    const Slot s = A.slots[b];   // (complete when the map let this grid launch)
    griddep_wait();
    griddep_launch();
    if (s.flags & SLOT_SKIP) {
        if (threadIdx.x == 0 && (A.state || A.node_cell)) replay_write(A, s, marginal_cell(A, s));
        return;
    }
    if (s.flags & SLOT_EMIT_MASKED) return;
    const Geom &g = A.g;
    const int K = s.K < KM ? s.K : KM;
    const unsigned seed = __float_as_uint(s.seed) ^ (unsigned(s.node) * 0x85EBCA6Bu);
    unsigned long long rk[KM];
    unsigned rp[KM];
#pragma unroll
    for (int i = 0; i < KM; ++i) {
        rk[i] = 0ull;
        rp[i] = 0u;
    }
    // the thread's K best in rk[KM-K .. KM-1] (ascending array of
    // KM; its minimum rk[0] bounds what may enter)
    const long long base = (long long)b * g.nseg;
    for (int sg = threadIdx.x; sg < g.nseg; sg += HS_THREADS) {
        const int cnt = A.rec_cnt[base + sg];
        if (cnt == 0) continue;
        if (hs_ordered(A.rec_max[base + sg]) < (unsigned)(rk[KM - K] >> 32)) continue;
        const float *rv = A.rec_val + (base + sg) * QSK_SEG;
        const int *ri = A.rec_idx + (base + sg) * QSK_SEG;
        for (int i = 0; i < cnt; ++i) {
            const unsigned idx = (unsigned)ri[i];
            const unsigned long long key = ((unsigned long long)hs_ordered(rv[i]) << 32) | tie_hash(seed, idx);
            if (key > rk[KM - K]) {
                // keep the array's top K: entries below KM-K stay at 0
                hs_insert<KM>(rk, rp, key, idx);
            }
        }
    }
#pragma unroll
    for (int i = 0; i < KM; ++i) {
        sk[i * HS_THREADS + threadIdx.x] = rk[i];
        sp[i * HS_THREADS + threadIdx.x] = rp[i];
    }
    __syncthreads();
    if (threadIdx.x >= 32) return;
    const int lane = threadIdx.x;
    // K rounds of warp argmax over the block's entries, descending
    unsigned chosen = 0xFFFFFFFFu;
    float cval[KM];
    unsigned cpos[KM];
    int got = 0;
    for (int r = 0; r < K; ++r) {
        unsigned long long bk = 0ull;
        int bi = -1;
        for (int e = lane; e < HS_THREADS * KM; e += 32) {
            const unsigned long long k2 = sk[e];
            if (k2 > bk) {
                bk = k2;
                bi = e;
            }
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            const unsigned long long ok = __shfl_xor_sync(0xffffffffu, bk, o);
            const int oi = __shfl_xor_sync(0xffffffffu, bi, o);
            if (ok > bk || (ok == bk && oi > bi)) {
                bk = ok;
                bi = oi;
            }
        }
        if (bk == 0ull) break;
        const unsigned ord = (unsigned)(bk >> 32);
        cval[r] = __uint_as_float((ord & 0x80000000u) ? (ord & 0x7FFFFFFFu) : ~ord);
        cpos[r] = sp[bi];
        __syncwarp();
        if (lane == 0) sk[bi] = 0ull;
        __syncwarp();
        ++got;
    }
    if (lane != 0 || got == 0) return;
    const int sel = s.sel < got ? s.sel : got - 1;
    if (A.out_val)
        for (int j = 0; j < K; ++j) {
            A.out_val[(long long)b * K + j] = j < got ? cval[j] : -CUDART_INF_F;
            A.out_pos[(long long)b * K + j] = j < got ? cpos[j] : 0u;
        }
    // cvtIndexToPosition (CPUThreadDevice.cpp:257-268), unsigned arithmetic
    const unsigned index = cpos[sel];
    unsigned position = 0;
    unsigned div = (unsigned)g.N;
    for (int d = g.nd - 1; d >= 0; --d) {
        unsigned f = (unsigned)g.fft[d], sr = (unsigned)g.src[d];
        div /= f;
        position = position * sr + ((f - (index / div) % f - (unsigned)s.mn[d] - 1u) + sr) % sr;
    }
    chosen = position;
    if (A.drawn_score) {
        A.drawn_score[s.node] = cval[sel];
        A.drawn_scale[s.node] = 0.f;   // the audit's k best come from the same FP32 map: no tolerance
    }
    if (A.node_cell) A.node_cell[s.node] = chosen;
    if (A.state)
        for (int v = 0; v < A.nvar; ++v) {
            float *dst = A.state + (long long)s.cell * A.nvar + v;
            if (isnan(*dst)) *dst = A.ti[(long long)chosen * A.nvar + v];
        }
    if (A.id_image) A.id_image[s.cell] = chosen * A.nti + A.ti_id;
}

// ---------------------------------------------------------------------------
// bit-sliced map for categorical patterns with unit weights
//
// One bit plane per (categorical variable, category) in the flipped scan
// order: bit q of plane (v,c) = [layer_v[q] == c].  For 32 consecutive scan
// positions m0..m0+31 the matches of term t are bits m0-d_t.. of its plane,
// read as one funnel-shifted 32-bit word; an 8-plane bit-sliced counter adds
// them.  With every weight equal to 1 the reference's sum of weights is the
// match count, exact in FP32 (< 2^24), so the scores equal the FP32 map bit
// for bit.  Records, counts and maxima are written in the same 128-position
// segment layout as k_map_records.
// ---------------------------------------------------------------------------
__global__ void k_build_planes(const float *__restrict__ layers, Geom g, int nvar, const int *__restrict__ ncat,
                               const float *__restrict__ catv, int pw, unsigned *__restrict__ planes) {
    long long idx = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    long long total = (long long)nvar * (QSK_CMAX + 1) * pw;
    if (idx >= total) return;
    const int w = int(idx % pw) - plane_guard(g.N);   // data word (negative: guard)
    int vc = int(idx / pw);
    int c = vc % (QSK_CMAX + 1), v = vc / (QSK_CMAX + 1);
    unsigned word = 0;
    if (w >= 0 && c < ncat[v]) {
        float cv = catv[v * QSK_CMAX + c];
        for (int b = 0; b < 32; ++b) {
            long long q = (long long)w * 32 + b;
            if (q < g.N && layers[(long long)v * g.N + q] == cv) word |= 1u << b;
        }
    }
    planes[idx] = word;
}

// bits [a, b) of a word, 0 <= a, b <= 32
__device__ __forceinline__ unsigned bits_range(int a, int b) {
    if (a >= b) return 0u;
    const unsigned hi = b >= 32 ? 0xffffffffu : ((1u << b) - 1u);
    return hi & ~((1u << a) - 1u);
}

// K <= 4: 64 registers, 32 warps per SM.  A warp's later segments are cheap
// once its carried K-th best is near the map's (no scan, no records), so fewer
// CTAs with more segments each do less work than 48 warps of one or two
// segments: 250x250 -> 500x500 (n = 80, plain) 110.5 ms with 40 registers and
// one or two segments a warp, 103.5 with more segments, 95.8 with 64 registers
// (no spills) as well.
// GEN: the first CTA of a slot makes its generator state (GenArgs)
template <int KF, bool GEN>
__global__ void __launch_bounds__(256, KF <= 4 ? 4 : 1) k_map_bits(BitArgs A) {
    extern __shared__ __align__(16) int2 bterm[];
    __shared__ Slot ss;
    __shared__ int nbt, s_multi, s_total;
    // staged plane windows of a single-variable slot, per category: lowest and
    // highest word offset of its terms, and where its window starts
    __shared__ int s_lo[QSK_CMAX], s_hi[QSK_CMAX], s_base[QSK_CMAX];
    const int b = blockIdx.y;
    if (GEN && blockIdx.x == 0) {   // (the staged planes leave room for a state)
        slot_generator(A.g, A.slots[b], b, A.gen, reinterpret_cast<unsigned *>(bterm));
        return;
    }
    const int part = int(blockIdx.x) - (GEN ? 1 : 0);
    // static slots and terms (k_mt_prep, a group of levels ahead) are read
    // before the previous level has completed, the values below
    if (!A.sterms) griddep_wait();
    if (threadIdx.x == 0) {
        ss = A.slots[b];
        nbt = 0;
        s_multi = 0;
    }
    if (threadIdx.x < QSK_CMAX) {
        s_lo[threadIdx.x] = INT_MAX;
        s_hi[threadIdx.x] = INT_MIN;
    }
    __syncthreads();
    griddep_wait();
    griddep_launch();
    if (ss.flags & SLOT_SKIP) return;
    const Geom &g = A.g;
    const int seg_begin = part * A.segs_per_cta;
    const int nseg1k = (int)((g.N + 1023) / 1024);
    int seg_end = seg_begin + A.segs_per_cta;
    if (seg_end > nseg1k) seg_end = nseg1k;
    {
        // terms -> (category, word offset), one thread per term; a code that is
        // no category of the TI (or a NaN value) matches nowhere and adds
        // nothing to the counts, so the term is dropped (the count is a sum of
        // 0/1 matches: its order is free)
        const Term *src = A.terms + (long long)b * A.maxterms;
        const StaticTerm *ssrc = A.sterms ? A.sterms + (long long)b * A.maxterms : nullptr;
        const int N32 = (int)g.N;
        for (int t = threadIdx.x; t < ss.nterms; t += blockDim.x) {
            int base;
            float val;
            if (ssrc) {
                const StaticTerm st = ssrc[t];
                base = st.base;
                val = st.src >= 0 ? A.state[st.src] : A.init[-(long long)st.src - 1];
            } else {
                const Term tm = src[t];
                base = tm.base;
                val = tm.b;
            }
            // base = v*N - d with 0 <= d < N
            const int v = base > 0 ? (base + N32 - 1) / N32 : 0;
            const int d = v * N32 - base;
            int c = QSK_CMAX;
            const int nc = A.ncat[v];
            for (int q = 0; q < nc; ++q)
                if (A.catv[v * QSK_CMAX + q] == val) { c = q; break; }
            if (c == QSK_CMAX) continue;
            // positions 32k..32k+31 read source bits from word k + floor(-d/32),
            // shifted right by (-d) mod 32
            const int off = plane_guard(g.N) + ((-d) >> 5);
            const int o = atomicAdd(&nbt, 1);
            if (v > 0) {
                s_multi = 1;
                bterm[o] = make_int2((v * (QSK_CMAX + 1) + c) * A.pw + off, (-d) & 31);
            } else {
                atomicMin(&s_lo[c], off);
                atomicMax(&s_hi[c], off);
                bterm[o] = make_int2(c * A.pw + off, ((-d) & 31) | (c << 8));
            }
        }
        if (threadIdx.x == 0 && ssrc && A.no_verbatim && ss.vtpl >= 0)
            ss.excl = verbatim_excl(g, A.tpl + ss.vtpl * g.nd, A.id_image[ss.vcell], ss.mn);
    }
    __syncthreads();
    const int nt = nbt;
    // Staging: the words of each category plane that this CTA's segments read
    // ([lo + 32*seg_begin, hi + 32*seg_end + 1)) go to shared memory, where a
    // warp's 32 consecutive words are one conflict-free access at any word
    // alignment (from global memory they span two cache lines).
    unsigned *stage = reinterpret_cast<unsigned *>(bterm + A.maxterms);
    if (threadIdx.x < 32) {
        const int c = threadIdx.x;
        const int len = s_lo[c] <= s_hi[c] ? s_hi[c] - s_lo[c] + 32 * (seg_end - seg_begin) + 1 : 0;
        int inc = len;
#pragma unroll
        for (int off = 1; off < 32; off <<= 1) {
            const int y = __shfl_up_sync(0xffffffffu, inc, off);
            if (c >= off) inc += y;
        }
        s_base[c] = inc - len;
        if (c == 31) s_total = inc;
    }
    __syncthreads();
    const bool staged = !s_multi && s_total <= A.stage_words && A.stage_words > 0;
    if (staged) {
        for (int c = 0; c < QSK_CMAX; ++c) {
            if (s_lo[c] > s_hi[c]) continue;
            const int len = s_hi[c] - s_lo[c] + 32 * (seg_end - seg_begin) + 1;
            const unsigned *src = A.planes + (long long)c * A.pw + s_lo[c] + 32 * seg_begin;
            unsigned *dst = stage + s_base[c];
            for (int w = threadIdx.x; w < len; w += blockDim.x) dst[w] = __ldg(src + w);
        }
        for (int t = threadIdx.x; t < nt; t += blockDim.x) {
            const int2 bt = bterm[t];
            const int c = bt.y >> 8;
            const int off = bt.x - c * A.pw;
            bterm[t] = make_int2(s_base[c] + off - s_lo[c] - 32 * seg_begin, bt.y & 31);
        }
    } else {
        for (int t = threadIdx.x; t < nt; t += blockDim.x) bterm[t].y &= 31;
    }
    __syncthreads();
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, nwarps = blockDim.x >> 5;
    const bool emit_masked = (ss.flags & SLOT_EMIT_MASKED) != 0;
    float *rv = A.rec_val + (long long)b * g.nseg * QSK_SEG;
    int *ri = A.rec_idx + (long long)b * g.nseg * QSK_SEG;

    // prefix top-KF of what this warp has seen: a CTA's warps take interleaved
    // segments in scan order, so all of it lies before the next segment
    float carry[KF];
#pragma unroll
    for (int q = 0; q < KF; ++q) carry[q] = -CUDART_INF_F;
    for (int sg = seg_begin + warp; sg < seg_end; sg += nwarps) {
        const long long m0 = (long long)sg * 1024 + 32 * lane;
        // validity of the lane's 32 positions
        unsigned vmask = 0, emask = 0;
        if (m0 < g.N && g.fft[0] >= 32) {
            // the 32 positions lie in at most two rows of the x dimension
            const long long rem = g.N - m0;
            emask = rem >= 32 ? 0xffffffffu : ((1u << rem) - 1u);
            // scan indices are below 2^31: 32-bit digits (row r holds digits 1..)
            const unsigned X = (unsigned)g.fft[0];
            const unsigned r0 = (unsigned)m0 / X;
            const int x0 = int((unsigned)m0 - r0 * X);
            auto row_ok = [&](unsigned r) {
                bool ok = true;
#pragma unroll
                for (int d = 1; d < QSK_MAXD; ++d)
                    if (d < g.nd) {
                        const unsigned f = (unsigned)g.fft[d];
                        ok &= int(r % f) >= ss.lo[d];
                        r /= f;
                    }
                return ok;
            };
            auto range = [](int a, int b) -> unsigned {   // bits [a, b), 0 <= a, b <= 32
                if (a >= b) return 0u;
                const unsigned hi = b >= 32 ? 0xffffffffu : ((1u << b) - 1u);
                return hi & ~((1u << a) - 1u);
            };
            const int first = X - x0;   // positions p < first are in row r0
            unsigned m = 0;
            if (row_ok(r0)) m |= range(max(0, ss.lo[0] - x0), min(32, first));
            if (first < 32 && row_ok(r0 + 1)) m |= range(min(32, first + ss.lo[0]), 32);
            vmask = m & emask;
        } else if (m0 < g.N) {
            // narrow x dimension: incremental digits
            int dig[QSK_MAXD];
#pragma unroll
            for (int d = 0; d < QSK_MAXD; ++d)
                dig[d] = d < g.nd ? int(((unsigned)m0 / (unsigned)g.sstride[d]) % (unsigned)g.fft[d]) : 0;
            bool rowok = true;
#pragma unroll
            for (int d = 1; d < QSK_MAXD; ++d)
                if (d < g.nd) rowok &= dig[d] >= ss.lo[d];
            for (int bit = 0; bit < 32; ++bit) {
                if (m0 + bit >= g.N) break;
                emask |= 1u << bit;
                if (rowok && dig[0] >= ss.lo[0]) vmask |= 1u << bit;
                if (++dig[0] == g.fft[0]) {
                    dig[0] = 0;
                    for (int d = 1; d < g.nd; ++d) {
                        if (++dig[d] < g.fft[d]) break;
                        dig[d] = 0;
                    }
                    rowok = true;
                    for (int d = 1; d < g.nd; ++d) rowok &= dig[d] >= ss.lo[d];
                }
            }
        }
        // bit-sliced counter: c0 (ones), c1 (twos), c2 (fours), c3 (eights)
        // fed by carry-save adders (Harley-Seal) over groups of 16 match
        // words, c4..c7 count sixteens; a tail of 8 and single words ripples
        unsigned c0 = 0, c1 = 0, c2 = 0, c3 = 0, c4 = 0, c5 = 0, c6 = 0, c7 = 0;
        if (vmask) {
            const int mw = int(m0) >> 5;
            auto count = [&](auto match) {
                auto csa = [](unsigned &h, unsigned &l, unsigned a, unsigned b, unsigned c) {
                    const unsigned u = a ^ b;
                    h = (a & b) | (u & c);
                    l = u ^ c;
                };
                int t = 0;
                for (; t + 16 <= nt; t += 16) {
                    unsigned twosA, twosB, foursA, foursB, eightsA, eightsB, sixteens;
                    csa(twosA, c0, c0, match(t), match(t + 1));
                    csa(twosB, c0, c0, match(t + 2), match(t + 3));
                    csa(foursA, c1, c1, twosA, twosB);
                    csa(twosA, c0, c0, match(t + 4), match(t + 5));
                    csa(twosB, c0, c0, match(t + 6), match(t + 7));
                    csa(foursB, c1, c1, twosA, twosB);
                    csa(eightsA, c2, c2, foursA, foursB);
                    csa(twosA, c0, c0, match(t + 8), match(t + 9));
                    csa(twosB, c0, c0, match(t + 10), match(t + 11));
                    csa(foursA, c1, c1, twosA, twosB);
                    csa(twosA, c0, c0, match(t + 12), match(t + 13));
                    csa(twosB, c0, c0, match(t + 14), match(t + 15));
                    csa(foursB, c1, c1, twosA, twosB);
                    csa(eightsB, c2, c2, foursA, foursB);
                    csa(sixteens, c3, c3, eightsA, eightsB);
                    unsigned x = sixteens, t0;
                    t0 = c4 & x; c4 ^= x; x = t0;
                    t0 = c5 & x; c5 ^= x; x = t0;
                    t0 = c6 & x; c6 ^= x; x = t0;
                    c7 ^= x;
                }
                for (; t + 8 <= nt; t += 8) {
                    unsigned twosA, twosB, foursA, foursB, eights;
                    csa(twosA, c0, c0, match(t), match(t + 1));
                    csa(twosB, c0, c0, match(t + 2), match(t + 3));
                    csa(foursA, c1, c1, twosA, twosB);
                    csa(twosA, c0, c0, match(t + 4), match(t + 5));
                    csa(twosB, c0, c0, match(t + 6), match(t + 7));
                    csa(foursB, c1, c1, twosA, twosB);
                    csa(eights, c2, c2, foursA, foursB);
                    unsigned x = eights, t0;
                    t0 = c3 & x; c3 ^= x; x = t0;
                    t0 = c4 & x; c4 ^= x; x = t0;
                    t0 = c5 & x; c5 ^= x; x = t0;
                    t0 = c6 & x; c6 ^= x; x = t0;
                    c7 ^= x;
                }
                for (; t < nt; ++t) {
                    unsigned x = match(t), t0;
                    t0 = c0 & x; c0 ^= x; x = t0;
                    t0 = c1 & x; c1 ^= x; x = t0;
                    t0 = c2 & x; c2 ^= x; x = t0;
                    t0 = c3 & x; c3 ^= x; x = t0;
                    t0 = c4 & x; c4 ^= x; x = t0;
                    t0 = c5 & x; c5 ^= x; x = t0;
                    t0 = c6 & x; c6 ^= x; x = t0;
                    c7 ^= x;
                }
            };
            if (staged) {
                const unsigned *S = stage + mw;
                count([&](int t) -> unsigned {
                    const int2 bt = bterm[t];
                    return __funnelshift_r(S[bt.x], S[bt.x + 1], unsigned(bt.y));
                });
            } else {
                const unsigned *P = A.planes + mw;
                count([&](int t) -> unsigned {
                    const int2 bt = bterm[t];
                    return __funnelshift_r(__ldg(P + bt.x), __ldg(P + bt.x + 1), unsigned(bt.y));
                });
            }
        }
        // Scores stay bit-sliced: position p of the lane holds the count
        // sum_b ((c_b >> p) & 1) << b where it is valid and not excluded, -inf
        // elsewhere.  Lane top-K by repeated bit-sliced maximum extraction.
        unsigned vm = vmask;
        if (ss.excl >= 0 && (long long)ss.excl >= m0 && (long long)ss.excl < m0 + 32)
            vm &= ~(1u << unsigned(ss.excl - m0));
        auto count_at = [&](int p) -> int {
            return int(((c0 >> p) & 1u) | (((c1 >> p) & 1u) << 1) | (((c2 >> p) & 1u) << 2) |
                       (((c3 >> p) & 1u) << 3) | (((c4 >> p) & 1u) << 4) | (((c5 >> p) & 1u) << 5) |
                       (((c6 >> p) & 1u) << 6) | (((c7 >> p) & 1u) << 7));
        };
        float lst[KF];
#pragma unroll
        for (int q = 0; q < KF; ++q) lst[q] = -CUDART_INF_F;
        float lmax = -CUDART_INF_F;
        {
            unsigned rest = vm;
            int filled = 0;
            for (int q = 0; q < KF && rest != 0u && filled < KF; ++q) {
                unsigned cand = rest;
                int val = 0;
                const unsigned cb[8] = {c0, c1, c2, c3, c4, c5, c6, c7};
#pragma unroll
                for (int bb = 7; bb >= 0; --bb) {
                    const unsigned t = cand & cb[bb];
                    if (t) {
                        cand = t;
                        val |= 1 << bb;
                    }
                }
                const int mult = __popc(cand);
                const float fv = (float)val;
#pragma unroll
                for (int q2 = 0; q2 < KF; ++q2)
                    if (q2 >= filled && q2 < filled + mult) lst[q2] = fv;
                if (q == 0) lmax = fv;
                filled += mult;
                rest &= ~cand;
            }
        }
        // largest score of each 128-position sub-segment (4 lanes) and of all
        const long long sub = (long long)sg * 8 + (lane >> 2);
        float gmax = lmax;
        gmax = fmaxf(gmax, __shfl_xor_sync(0xffffffffu, gmax, 1));
        gmax = fmaxf(gmax, __shfl_xor_sync(0xffffffffu, gmax, 2));
        float smax = gmax;
#pragma unroll
        for (int off = 4; off < 32; off <<= 1) smax = fmaxf(smax, __shfl_xor_sync(0xffffffffu, smax, off));
        if (smax < carry[KF - 1]) {
            // nothing reaches the K-th best before the segment: no record
            if (sub < g.nseg && (lane & 3) == 0) {
                A.rec_cnt[(long long)b * g.nseg + sub] = 0;
                A.rec_max[(long long)b * g.nseg + sub] = gmax;
            }
            continue;
        }
        // exclusive prefix of the lane states across the 1024-position segment
        // and all before it
        float inc[KF];
#pragma unroll
        for (int q = 0; q < KF; ++q) inc[q] = lst[q];
#pragma unroll
        for (int off = 1; off < 32; off <<= 1) {
            float rcv[KF], mrg[KF];
#pragma unroll
            for (int q = 0; q < KF; ++q) rcv[q] = __shfl_up_sync(0xffffffffu, inc[q], off);
            if (lane >= off) {
                topk_merge<KF>(inc, rcv, mrg);
#pragma unroll
                for (int q = 0; q < KF; ++q) inc[q] = mrg[q];
            }
        }
        float st[KF], before[KF];
#pragma unroll
        for (int q = 0; q < KF; ++q) {
            const float y = __shfl_up_sync(0xffffffffu, inc[q], 1);
            before[q] = lane == 0 ? -CUDART_INF_F : y;
        }
        topk_merge<KF>(carry, before, st);
        // Before the warp has seen K values, lane 0's running K-th starts from
        // (almost) nothing and most of its positions would be visited one by one
        // below.  The warp decides them instead: position p of lane 0 on lane p,
        // and an exclusive prefix top-K over the lanes gives the K-th before each.
        const bool special = carry[KF - 1] == -CUDART_INF_F;
        float x0v = 0.f;
        unsigned rmask0 = 0u;
        if (special) {
            const unsigned vm0 = __shfl_sync(0xffffffffu, vm, 0);
            const unsigned recok0 = __shfl_sync(0xffffffffu, emit_masked ? emask : (emask & vmask), 0);
            const unsigned cnt = ((__shfl_sync(0xffffffffu, c0, 0) >> lane) & 1u) |
                                 (((__shfl_sync(0xffffffffu, c1, 0) >> lane) & 1u) << 1) |
                                 (((__shfl_sync(0xffffffffu, c2, 0) >> lane) & 1u) << 2) |
                                 (((__shfl_sync(0xffffffffu, c3, 0) >> lane) & 1u) << 3) |
                                 (((__shfl_sync(0xffffffffu, c4, 0) >> lane) & 1u) << 4) |
                                 (((__shfl_sync(0xffffffffu, c5, 0) >> lane) & 1u) << 5) |
                                 (((__shfl_sync(0xffffffffu, c6, 0) >> lane) & 1u) << 6) |
                                 (((__shfl_sync(0xffffffffu, c7, 0) >> lane) & 1u) << 7);
            const bool val = (vm0 >> lane) & 1u;
            x0v = val ? (float)cnt : -CUDART_INF_F;
            float in0[KF];
            in0[0] = x0v;
#pragma unroll
            for (int q = 1; q < KF; ++q) in0[q] = -CUDART_INF_F;
#pragma unroll
            for (int off = 1; off < 32; off <<= 1) {
                float rcv[KF], mrg[KF];
#pragma unroll
                for (int q = 0; q < KF; ++q) rcv[q] = __shfl_up_sync(0xffffffffu, in0[q], off);
                if (lane >= off) {
                    topk_merge<KF>(in0, rcv, mrg);
#pragma unroll
                    for (int q = 0; q < KF; ++q) in0[q] = mrg[q];
                }
            }
            float ex0[KF], pre0[KF];
#pragma unroll
            for (int q = 0; q < KF; ++q) {
                const float y = __shfl_up_sync(0xffffffffu, in0[q], 1);
                ex0[q] = lane == 0 ? -CUDART_INF_F : y;
            }
            topk_merge<KF>(carry, ex0, pre0);
            const float kth = pre0[KF - 1];
            // before K finite values every position that can be a candidate is
            // a record; afterwards the valid ones not below the K-th
            const bool rec = kth == -CUDART_INF_F ? ((recok0 >> lane) & 1u) != 0u : (val && x0v >= kth);
            rmask0 = __ballot_sync(0xffffffffu, rec);
        }
        {
            float all[KF], nc[KF];
#pragma unroll
            for (int q = 0; q < KF; ++q) all[q] = __shfl_sync(0xffffffffu, inc[q], 31);
            topk_merge<KF>(carry, all, nc);
#pragma unroll
            for (int q = 0; q < KF; ++q) carry[q] = nc[q];
        }
        const bool decided = special && lane == 0;   // by the warp, above
        // record flags: value not below the K-th best of everything before it
        // (earlier lanes, then earlier positions of this lane)
        unsigned rmask = decided ? rmask0 : 0u;
        const float T0s = st[KF - 1];
        unsigned eqm = 0u;       // records whose value is tval (no count extraction)
        float tval = 0.f;
        unsigned from = decided ? 0u : 0xffffffffu;   // positions decided by the threshold path below
        float T0 = T0s;
        if (!decided && T0 == -CUDART_INF_F) {
            // Fewer than K finite values before this lane: every position is a
            // record until K finite values are held (masked ones only when they
            // can be candidates).  Only the valid positions up to that point are
            // visited one by one; the rest of the lane takes the threshold path.
            const unsigned recok = emit_masked ? emask : (emask & vmask);
            unsigned vv = vm;
            int cur = 0;
            while (vv && st[KF - 1] == -CUDART_INF_F) {
                const int bit = __ffs(vv) - 1;
                vv &= vv - 1u;
                rmask |= recok & bits_range(cur, bit);
                rmask |= 1u << bit;
                topk_insert<KF>(st, (float)count_at(bit));
                cur = bit + 1;
            }
            if (st[KF - 1] == -CUDART_INF_F) {
                rmask |= recok & bits_range(cur, 32);
                from = 0u;
            } else {
                from = bits_range(cur, 32);
            }
            T0 = st[KF - 1];
        }
        if (from) {
            // only positions with count >= T0 can be records (the running K-th
            // never drops below T0; a smaller value leaves the state unchanged)
            const int T = (int)T0;
            unsigned gt = 0u, eq = vm;
            const unsigned cb[8] = {c0, c1, c2, c3, c4, c5, c6, c7};
#pragma unroll
            for (int bb = 7; bb >= 0; --bb) {
                if ((T >> bb) & 1) {
                    eq &= cb[bb];
                } else {
                    gt |= eq & cb[bb];
                    eq &= ~cb[bb];
                }
            }
            if (T > 255) gt = eq = 0u;
            gt &= from;
            eq &= from;
            // Positions equal to T0 are records while the running K-th is still
            // T0 and never change the state; only positions above T0 need their
            // count and an insertion.  The first insertion that lifts the K-th
            // above T0 ends the equal records.
            unsigned eqcut = 0xffffffffu;
            unsigned g = gt;
            while (g) {
                const int bit = __ffs(g) - 1;
                g &= g - 1u;
                const float x = (float)count_at(bit);
                if (x >= st[KF - 1]) rmask |= 1u << bit;
                topk_insert<KF>(st, x);
                if (eqcut == 0xffffffffu && st[KF - 1] > T0) eqcut = bit >= 31 ? 0xffffffffu : ((2u << bit) - 1u);
            }
            rmask |= eq & eqcut;
            eqm = eq;
            tval = T0;
        }
        // offsets inside each 128-position sub-segment (4 lanes)
        const int rc = __popc(rmask);
        int pre = rc;
        int y1 = __shfl_up_sync(0xffffffffu, pre, 1);
        if ((lane & 3) >= 1) pre += y1;
        int y2 = __shfl_up_sync(0xffffffffu, pre, 2);
        if ((lane & 3) >= 2) pre += y2;
        const int excl = pre - rc;
        const int tot = __shfl_sync(0xffffffffu, pre, (lane | 3));
        // lane 0's records, one per lane (the first ones of its sub-segment)
        if ((rmask0 >> lane) & 1u) {
            const long long r0 = (long long)sg * 8 * QSK_SEG + __popc(rmask0 & lanemask_lt());
            rv[r0] = x0v;
            ri[r0] = int((long long)sg * 1024 + lane);
        }
        const int rb = int(sub * QSK_SEG) + excl;   // (scan positions are below 2^31)
        unsigned rm = decided || sub >= g.nseg ? 0u : rmask;
        if (__reduce_max_sync(0xffffffffu, (unsigned)__popc(rm)) > 6u) {
            // many records in a lane (ties): one lane's positions after the
            // other, position p on lane p, in coalesced stores
            unsigned todo = __ballot_sync(0xffffffffu, rm != 0u);
            while (todo) {
                const int l = __ffs(todo) - 1;
                todo &= todo - 1u;
                const unsigned mask = __shfl_sync(0xffffffffu, rm, l), eq = __shfl_sync(0xffffffffu, eqm, l);
                const unsigned in = __shfl_sync(0xffffffffu, vm, l);
                const int at = __shfl_sync(0xffffffffu, rb, l);
                float x = __shfl_sync(0xffffffffu, tval, l);
                if (mask & ~eq) {
                    const unsigned cnt = ((__shfl_sync(0xffffffffu, c0, l) >> lane) & 1u) |
                                         (((__shfl_sync(0xffffffffu, c1, l) >> lane) & 1u) << 1) |
                                         (((__shfl_sync(0xffffffffu, c2, l) >> lane) & 1u) << 2) |
                                         (((__shfl_sync(0xffffffffu, c3, l) >> lane) & 1u) << 3) |
                                         (((__shfl_sync(0xffffffffu, c4, l) >> lane) & 1u) << 4) |
                                         (((__shfl_sync(0xffffffffu, c5, l) >> lane) & 1u) << 5) |
                                         (((__shfl_sync(0xffffffffu, c6, l) >> lane) & 1u) << 6) |
                                         (((__shfl_sync(0xffffffffu, c7, l) >> lane) & 1u) << 7);
                    if (!((eq >> lane) & 1u)) x = ((in >> lane) & 1u) ? (float)cnt : -CUDART_INF_F;
                }
                if ((mask >> lane) & 1u) {
                    const int o = at + __popc(mask & lanemask_lt());
                    rv[o] = x;
                    ri[o] = int((long long)sg * 1024 + 32 * l + lane);
                }
            }
        } else {
            int o = rb;
            while (rm) {
                const int bit = __ffs(rm) - 1;
                rm &= rm - 1u;
                rv[o] = ((eqm >> bit) & 1u) ? tval : (((vm >> bit) & 1u) ? (float)count_at(bit) : -CUDART_INF_F);
                ri[o] = int(m0 + bit);
                o++;
            }
        }
        if (sub < g.nseg && (lane & 3) == 0) {
            A.rec_cnt[(long long)b * g.nseg + sub] = tot;
            A.rec_max[(long long)b * g.nseg + sub] = gmax;
        }
    }
}

// The slot of path node i and its terms without their values (bit-sliced
// simulations: unit weights, categorical variables, complete TI): everything
// k_prep_sim derives from the neighbour lists, computed a group of batches
// ahead.
// The map reads the values (and derives the -nV exclusion) when it runs.
__device__ void write_static_slot(const SimPrepArgs &A, int b, int i, unsigned pv, unsigned cell, const NodeGeom &ng,
                                  int lane) {
    const int cnt = A.nb_count[i];
    const int nd = A.g.nd;
    Slot s;
    s.node = i;
    s.cell = cell;
    s.var = A.full ? int(pv % unsigned(A.nvar)) : 0;
    s.seed = A.seeds[i];
    s.K = ng.Ki;
    s.sel = selected_index(s.seed, ng.lk, A.nti);
    if (s.sel < 0) s.sel = 0;
    if (s.sel > ng.Ki - 1) s.sel = ng.Ki - 1;
    s.flags = 0;
    s.nterms = 0;
    s.excl = -1;
    s.cmask_base = 0;
    s.vcell = 0;
    s.vtpl = -1;
#pragma unroll
    for (int d = 0; d < QSK_MAXD; ++d) {
        s.mn[d] = ng.mn[d];
        s.lo[d] = ng.lo[d];
    }
    if (ng.skip) {
        s.flags |= SLOT_SKIP;
    } else {
        if (ng.nvalid < ng.Ki) s.flags |= SLOT_EMIT_MASKED;
        int base_out = 0;
        for (int j0 = 0; j0 < cnt; j0 += 32) {
            const int j = j0 + lane;
            StaticTerm tl[4];
            int nt = 0;
            if (j < cnt) {
                const int t = A.nb_tpl[(long long)i * A.n + j];
                const unsigned nc = A.nb_cell[(long long)i * A.n + j];
                long long d_flat = 0;
                for (int d = 0; d < nd; ++d) d_flat += (long long)(A.tpl[t * nd + d] - ng.mn[d]) * A.g.sstride[d];
                for (int v = 0; v < A.nvar && v < 4; ++v) {
                    if (A.full) {
                        if (!((A.nb_mask[(long long)i * A.n + j] >> v) & 1u)) continue;
                    } else if (A.node_nv && j >= A.node_nv[(long long)i * A.nvar + v]) {
                        continue;
                    }
                    if (A.wtab[t * A.nvar + v] == 0.f) continue;
                    const long long sidx = (long long)nc * A.nvar + v;
                    StaticTerm st;
                    st.base = int((long long)v * A.g.N - d_flat);
                    st.src = (nc == cell && !A.full) ? int(-sidx - 1) : int(sidx);
                    tl[nt++] = st;
                }
            }
            int incl = nt;
            for (int off = 1; off < 32; off <<= 1) {
                int y = __shfl_up_sync(0xffffffffu, incl, off);
                if (lane >= off) incl += y;
            }
            const int excl = incl - nt;
            const int total = __shfl_sync(0xffffffffu, incl, 31);
            for (int q = 0; q < nt; ++q) {
                const int o = base_out + excl + q;
                if (o < A.maxterms) A.sterms[(long long)b * A.maxterms + o] = tl[q];
            }
            base_out += total;
        }
        if (base_out > A.maxterms) {
            if (lane == 0) atomicExch(A.status, DEV_TOO_MANY_TERMS);
            base_out = A.maxterms;
        }
        s.nterms = base_out;
        if (A.no_verbatim && cnt > 1 && !A.full) {
            s.vtpl = A.nb_tpl[(long long)i * A.n + 1];
            s.vcell = A.nb_cell[(long long)i * A.n + 1];
        }
    }
    if (lane == 0) A.slots[b] = s;
}

// MT19937 state of each slot ahead of its replay (one warp per slot; the
// host runs it for the next group of batches while the current one is
// simulated, as it reads the neighbour lists only): the seeding and, with masked positions
// not emitted as records, the state-only blocks of the replay's first
// skip.  That skip covers the c
// masked positions before the first record (two draws each); c is at least
// the number c0 of masked positions before the first valid one, so the
// blocks that rng_skip regenerates without output for 2*c0 draws,
// (2*c0 - 1) / 624 of them, are the first blocks of the real skip too.
__global__ void __launch_bounds__(32 * RP_WARPS) k_mt_prep(SimPrepArgs A, unsigned *__restrict__ state,
                                                           int *__restrict__ pre) {
    __shared__ __align__(16) unsigned mt[RP_WARPS][624];
    const int wib = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int b = blockIdx.x * RP_WARPS + wib;
    if (b >= A.nslots) return;
    const int i = A.nodes[b];
    const unsigned pv = A.path[A.begin + i];
    const unsigned cell = A.full ? pv / unsigned(A.nvar) : pv;
    const NodeGeom ng = node_geometry(A, i, cell, lane);
    if (A.sterms) write_static_slot(A, b, i, pv, cell, ng, lane);
    if (ng.skip) return;
    if (lane == 0) mt_seed(mt[wib], A.seeds[i]);
    __syncwarp();
    const long long blocks = A.missing ? 0 : skipped_blocks(A.g, ng.lo, ng.nvalid, ng.Ki);
    if (blocks > 0) mt_roll(mt[wib], blocks, lane);
    store_generator(mt[wib], blocks, b, state, pre, lane);
}

// Verbatim exclusion with a radius (CPUThreadDevice::setValueInErrorArrayWithRadius,
// G2S src/CPUThreadDevice.cpp:310-342): from the scan index c, level L = nd..2
// steps i_L in [-r, r] with r = ceil(sqrt(R2 - d2)) by fft[L-1] (d2 the sum of
// the squares of the outer steps, a level entered only while d2 <= R2), and
// level 1 steps by fft[0], marking (c + offset + N) mod N in 32-bit unsigned
// arithmetic as the reference does.  One CTA per slot: the outer steps are a
// box [-R, R]^(nd-1) enumerated by the threads, each thread runs the level-1
// loop of its tuples.
__global__ void k_radius_mask(const int *__restrict__ center, const float *__restrict__ radius, Geom g,
                              unsigned *__restrict__ mask, long long xwords) {
    const int b = blockIdx.x;
    unsigned *xm = mask + (long long)b * xwords;
    for (long long q = threadIdx.x; q < xwords; q += blockDim.x) xm[q] = 0u;
    __syncthreads();
    const int c = center[b];
    const float rad = radius[b];
    if (c < 0 || !(rad >= 1.f)) return;
    const float R2 = rad * rad;
    const int R = int(ceil(sqrt((double)R2)));
    const unsigned s = (unsigned)g.N;
    const int nouter = g.nd - 1;
    long long box = 1;
    for (int L = 0; L < nouter; ++L) box *= 2 * R + 1;
    for (long long t = threadIdx.x; t < box; t += blockDim.x) {
        // outer tuple (i_nd, ..., i_2), outermost first
        long long rest = t;
        unsigned pos = (unsigned)c;
        unsigned d2 = 0;
        bool ok = true;
        for (int L = g.nd; L >= 2 && ok; --L) {
            const int i = int(rest % (2 * R + 1)) - R;
            rest /= (2 * R + 1);
            // level L is entered with d2 <= R2 and runs i in [-r, r]
            if (!((float)d2 <= R2)) { ok = false; break; }
            const int r = int(ceil(sqrt((double)(R2 - (float)d2))));
            if (i < -r || i > r) { ok = false; break; }
            pos += (unsigned)(i * (int)g.fft[L - 1]);
            d2 += (unsigned)(i * i);
        }
        if (!ok || !((float)d2 <= R2)) continue;
        const int r1 = int(ceil(sqrt((double)(R2 - (float)d2))));
        for (int i = -r1; i <= r1; ++i) {
            const unsigned m = (pos + (unsigned)(i * (int)g.fft[0]) + s) % s;
            atomicOr(xm + (m >> 5), 1u << (m & 31));
        }
    }
}

// ---------------------------------------------------------------------------
// launch wrappers (called by the host engine)
// ---------------------------------------------------------------------------
cudaError_t launch_build_layers(const float *ti, int nvar, const int *types, const Geom &g, float *layers, int missing,
                                cudaStream_t st) {
    long long blocks = (g.N + 255) / 256;
    k_build_layers<<<(unsigned)blocks, 256, 0, st>>>(ti, nvar, types, g, layers, missing);
    return cudaGetLastError();
}

cudaError_t launch_neighbours(const GridDesc &dg, const int *tpl, int ntpl, const unsigned *path, unsigned begin,
                              long long nodes, const unsigned *posterior, int n, int *nb_count, int *nb_tpl,
                              unsigned *nb_cell, const int *node_kernel, const int *tpl_range, const int *node_lim,
                              cudaStream_t st) {
    if (nodes <= 0) return cudaSuccess;
    k_neighbours<<<(unsigned)((nodes * 32 + 255) / 256), 256, 0, st>>>(dg, tpl, ntpl, path, begin, nodes, posterior, n,
                                                                       nb_count, nb_tpl, nb_cell, node_kernel,
                                                                       tpl_range, node_lim);
    return cudaGetLastError();
}

cudaError_t launch_neighbours_full(const GridDesc &dg, const int *tpl, int ntpl, const unsigned *path, unsigned begin,
                                   long long nodes, const unsigned *posterior, int nvar, int n, const int *node_nv,
                                   int *nb_count, int *nb_tpl, unsigned *nb_cell, unsigned char *nb_mask,
                                   const int *node_kernel, const int *tpl_range, cudaStream_t st) {
    if (nodes <= 0) return cudaSuccess;
    k_neighbours_full<<<(unsigned)((nodes * 32 + 255) / 256), 256, 0, st>>>(dg, tpl, ntpl, path, begin, nodes, posterior,
                                                                            nvar, n, node_nv, nb_count, nb_tpl, nb_cell,
                                                                            nb_mask, node_kernel, tpl_range);
    return cudaGetLastError();
}

cudaError_t launch_levels(const LevelArgs &a, cudaStream_t st) {
    long long nodes = a.nodes;
    if (nodes <= 0) return cudaSuccess;
    const unsigned nb = (unsigned)((nodes + 255) / 256);
    const long long ntiles = (nodes + 1023) / 1024;
    cudaError_t e;
    if ((e = cudaMemsetAsync(a.level, 0xff, sizeof(int) * size_t(nodes), st)) != cudaSuccess) return e;
    if ((e = cudaMemsetAsync(a.cnt, 0, sizeof(int) * size_t(nodes + 2), st)) != cudaSuccess) return e;
    int dev = 0, sms = 0;
    if ((e = cudaGetDevice(&dev)) != cudaSuccess) return e;
    if ((e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev)) != cudaSuccess) return e;
    long long blocks = (long long)sms * 8;
    const long long need = (nodes * 32 + 255) / 256;
    if (blocks > need) blocks = need;
    k_level_flow<<<(unsigned)blocks, 256, 0, st>>>(nodes, a.n, a.nb_count, a.nb_cell, a.nb_mask, a.nvar, a.node_of_cell,
                                                   a.level, a.cnt + nodes + 1, a.nl_out, a.status,
                                                   a.spin_limit ? a.spin_limit : (1u << 22), a.hold);
    k_level_count<<<nb, 256, 0, st>>>(nodes, a.level, a.cnt);
    k_scan_tiles<<<(unsigned)ntiles, 1024, 0, st>>>(nodes, a.cnt, a.start, a.tile_sum);
    k_scan_sums<<<1, 32, 0, st>>>((int)ntiles, a.tile_sum);
    k_scan_add<<<(unsigned)((nodes + 1 + 255) / 256), 256, 0, st>>>(nodes, a.start, a.cursor, a.tile_sum);
    k_level_scatter<<<nb, 256, 0, st>>>(nodes, a.level, a.cursor, a.level_nodes);
    return cudaGetLastError();
}

cudaError_t launch_prep_tc_nodes(const SimPrepArgs &p, const TcNodeArgs &a, bool after_select, cudaStream_t st) {
    if (!a.A || a.nslots != p.nslots || a.rows < a.nslots || (a.Kp * (a.fmt == 1 ? 1 : 2)) % 16 != 0)
        return cudaErrorInvalidValue;
    const long long prep_blocks = ((long long)p.nslots * 32 + 255) / 256;
    const long long node_blocks = (a.rows * 32 + 255) / 256;
    const dim3 grid((unsigned)(prep_blocks + node_blocks));
    if (after_select) return launch_pdl(k_prep_tc_nodes, grid, dim3(256), 0, st, p, a, (unsigned)prep_blocks);
    k_prep_tc_nodes<<<grid, 256, 0, st>>>(p, a, (unsigned)prep_blocks);
    return cudaGetLastError();
}

cudaError_t launch_prep_sim(const SimPrepArgs &a, bool chained, cudaStream_t st) {
    int threads = 256;
    long long blocks = ((long long)a.nslots * 32 + threads - 1) / threads;
    return launch_chain(chained, k_prep_sim, dim3((unsigned)blocks), dim3(threads), 0, st, a);
}

// (148: the SMs of a B200, here and below)
int map_segs_per_cta(const Geom &g, int nslots, int K) {
    // a CTA takes 8 warps x MR_SEGS segments a turn; more turns (up to 8)
    // tighten the filter and share the set-up while the grid still fills the
    // GPU's 4 resident CTAs per SM three times.  Beyond K = 4 (2 resident
    // CTAs) a warp's first turns, which hold no bound yet, cost the most, and
    // one wave of CTAs is best: 80x70x60 continuous (n = 25), K = 15, map and
    // replay of all levels 205 ms by the rule for K <= 4 (196 with a prefix per
    // segment), 183 with three waves of two CTAs, 178 with two, 175 with one;
    // K = 8 51, 51, 50, 51
    const long long turn = 8 * MR_SEGS;
    const long long turns = (g.nseg + turn - 1) / turn * nslots;
    long long per = turns / (K <= 4 ? 148LL * 4 * 3 : 148LL * 2);
    per = per < 1 ? 1 : (per > 8 ? 8 : per);
    return (int)(per * turn);
}

template <bool GEN>
static cudaError_t launch_map_records_k(const MapArgs &a, dim3 grid, size_t smem, int K, bool chained, cudaStream_t st) {
    const dim3 block(256);
    if (K <= 1) return launch_chain(chained, k_map_records<1, GEN>, grid, block, smem, st, a);
    if (K <= 2) return launch_chain(chained, k_map_records<2, GEN>, grid, block, smem, st, a);
    if (K <= 4) return launch_chain(chained, k_map_records<4, GEN>, grid, block, smem, st, a);
    if (K <= 8) return launch_chain(chained, k_map_records<8, GEN>, grid, block, smem, st, a);
    return launch_chain(chained, k_map_records<16, GEN>, grid, block, smem, st, a);
}

cudaError_t launch_map_records(const MapArgs &args, int nslots, int K, int maxterms_in_batch, bool chained,
                               cudaStream_t st) {
    MapArgs a = args;
    for (int d = 0; d < QSK_MAXD; ++d) a.div[d] = make_fast_div((unsigned)a.g.fft[d]);
    dim3 grid((unsigned)((a.g.nseg + a.segs_per_cta - 1) / a.segs_per_cta) + (a.gen.state ? 1u : 0u), (unsigned)nslots);
    size_t smem = sizeof(Term) * (size_t)(maxterms_in_batch > 0 ? maxterms_in_batch : 1);
    if (a.gen.state && smem < 624 * sizeof(unsigned)) smem = 624 * sizeof(unsigned);
    return a.gen.state ? launch_map_records_k<true>(a, grid, smem, K, chained, st)
                       : launch_map_records_k<false>(a, grid, smem, K, chained, st);
}

cudaError_t launch_build_planes(const float *layers, const Geom &g, int nvar, const int *ncat, const float *catv,
                                int pw, unsigned *planes, cudaStream_t st) {
    long long total = (long long)nvar * (QSK_CMAX + 1) * pw;
    k_build_planes<<<(unsigned)((total + 255) / 256), 256, 0, st>>>(layers, g, nvar, ncat, catv, pw, planes);
    return cudaGetLastError();
}

// shared-memory words for the staged plane windows of k_map_bits (30 KB)
#define MAP_BITS_STAGE_WORDS 7680

int map_bits_segs_per_cta(const Geom &g, int nslots) {
    // a CTA takes 8 segments of 1024 positions a turn; more turns (up to 8, in
    // equal shares) tighten the filter of its later segments, whose records
    // and threshold work are most of the kernel, while three CTAs per SM stay
    const long long per_slot = (g.N + 8191) / 8192;
    long long turns = per_slot * nslots / (148LL * 3);
    turns = turns < 1 ? 1 : (turns > 8 ? 8 : turns);
    const long long ctas = (per_slot + turns - 1) / turns;
    return (int)((per_slot + ctas - 1) / ctas * 8);
}

template <bool GEN>
static cudaError_t launch_map_bits_k(const BitArgs &a, dim3 grid, size_t smem, int K, bool chained, cudaStream_t st) {
    const dim3 block(256);
    if (K <= 1) return launch_chain(chained, k_map_bits<1, GEN>, grid, block, smem, st, a);
    if (K <= 2) return launch_chain(chained, k_map_bits<2, GEN>, grid, block, smem, st, a);
    if (K <= 4) return launch_chain(chained, k_map_bits<4, GEN>, grid, block, smem, st, a);
    if (K <= 8) return launch_chain(chained, k_map_bits<8, GEN>, grid, block, smem, st, a);
    return launch_chain(chained, k_map_bits<16, GEN>, grid, block, smem, st, a);
}

cudaError_t launch_map_bits(const BitArgs &args, int nslots, int K, int maxterms_in_batch, bool chained,
                            cudaStream_t st) {
    BitArgs a = args;
    if (a.maxterms < maxterms_in_batch) return cudaErrorInvalidValue;
    a.stage_words = MAP_BITS_STAGE_WORDS;
    long long nseg1k = (a.g.N + 1023) / 1024;
    dim3 grid((unsigned)((nseg1k + a.segs_per_cta - 1) / a.segs_per_cta) + (a.gen.state ? 1u : 0u), (unsigned)nslots);
    size_t smem = sizeof(int2) * (size_t)(a.maxterms > 0 ? a.maxterms : 1) + sizeof(unsigned) * (size_t)a.stage_words;
    return a.gen.state ? launch_map_bits_k<true>(a, grid, smem, K, chained, st)
                       : launch_map_bits_k<false>(a, grid, smem, K, chained, st);
}

template <int KF>
static cudaError_t map_smem_limit(int bytes) {
    cudaError_t e = cudaFuncSetAttribute(k_map_records<KF, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
    if (e != cudaSuccess) return e;
    return cudaFuncSetAttribute(k_map_records<KF, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
}

cudaError_t set_map_smem_limit(int bytes) {
    cudaError_t e;
    if ((e = map_smem_limit<1>(bytes)) != cudaSuccess || (e = map_smem_limit<2>(bytes)) != cudaSuccess ||
        (e = map_smem_limit<4>(bytes)) != cudaSuccess || (e = map_smem_limit<8>(bytes)) != cudaSuccess)
        return e;
    return map_smem_limit<16>(bytes);
}

cudaError_t launch_radius_mask(const int *center, const float *radius, int nslots, const Geom &g, unsigned *mask,
                               long long xwords, cudaStream_t st) {
    if (nslots <= 0) return cudaSuccess;
    k_radius_mask<<<(unsigned)nslots, 256, 0, st>>>(center, radius, g, mask, xwords);
    return cudaGetLastError();
}

// Several training images: one thread per slot merges every TI's K best
// and draws (see MultiDrawArgs).  The merge is the reference's std::sort of
// the TIs x K candidates by score (quantileSamplingModule.hpp:101-104),
// which for at most 16 candidates is libstdc++'s insertion sort: stable.
__global__ void k_multi_draw(MultiDrawArgs A) {
    const int b = blockIdx.x * blockDim.x + threadIdx.x;
    if (b >= A.nslots) return;
    const Slot s = A.slots[b];
    const int nvar = A.nvar;
    unsigned ti = 0, tcell = 0;
    if (s.flags & SLOT_SKIP) {
        // marginal: the TIs' cells end to end (simulation.hpp:586-610)
        unsigned cumulated = 0;
        for (int t = 0; t < A.nti; ++t) cumulated += (unsigned)A.ti_cells[t] * (unsigned)nvar;
        const unsigned position =
            (unsigned)(int)floorf(__fmul_rn(s.seed, __uint2float_rn(cumulated / (unsigned)nvar)));
        cumulated = 0;
        for (int t = 0; t < A.nti; ++t) {
            const unsigned size = (unsigned)A.ti_cells[t] * (unsigned)nvar;
            if (position * (unsigned)nvar < cumulated + size) {
                ti = (unsigned)t;
                tcell = position - cumulated / (unsigned)nvar;
                break;
            }
            cumulated += size;
        }
    } else {
        // delta = sum over continuous variables, then neighbours, of
        // -1 * (w * v * v) in the reference's float order
        // (quantileSamplingModule.hpp:412-457)
        float delta = 0.f;
        const int cnt = A.nb_count[s.node];
        for (int i = 0; i < nvar; ++i) {
            if (A.types[i] != 0) continue;
            for (int j = 0; j < cnt; ++j) {
                const unsigned c = A.nb_cell[(long long)s.node * A.n + j];
                const float v = A.state[(long long)c * nvar + i];
                if (isnan(v)) continue;
                const float w = A.wtab[(long long)A.nb_tpl[(long long)s.node * A.n + j] * nvar + i];
                delta = __fadd_rn(delta, __fmul_rn(-1.f, __fmul_rn(__fmul_rn(w, v), v)));
            }
        }
        const int req = A.ii ? (int)A.ii[s.cell] : -1;
        float v[16];
        int o[16];
        const int m = A.nti * A.K;
        for (int q = 0; q < m; ++q) {
            const int t = q / A.K;
            v[q] = (req < 0 || t == req) ? __fadd_rn(A.vals[t * A.ti_stride + (long long)b * A.K + q % A.K], delta)
                                         : -CUDART_INF_F;
            o[q] = q;
        }
        for (int q = 1; q < m; ++q) {
            const float x = v[q];
            const int y = o[q];
            int j = q;
            while (j > 0 && x > v[j - 1]) {
                v[j] = v[j - 1];
                o[j] = o[j - 1];
                --j;
            }
            v[j] = x;
            o[j] = y;
        }
        const int q = o[s.sel < m ? s.sel : m - 1];
        ti = (unsigned)(q / A.K);
        tcell = A.cells[ti * A.ti_stride + (long long)b * A.K + q % A.K];
    }
    if (A.node_cell) A.node_cell[s.node] = tcell;
    if (A.state) {
        for (int v2 = 0; v2 < nvar; ++v2) {
            float *dst = A.state + (long long)s.cell * nvar + v2;
            if (isnan(*dst)) *dst = A.ti[ti][(long long)tcell * nvar + v2];
        }
    }
    if (A.id_image) A.id_image[s.cell] = tcell * (unsigned)A.nti + ti;
}

cudaError_t launch_multi_draw(const MultiDrawArgs &a, cudaStream_t st) {
    if (a.nslots <= 0) return cudaSuccess;
    if (a.nti < 1 || a.nti > QSK_MAX_TIS || a.nti * a.K > 16) return cudaErrorInvalidValue;
    k_multi_draw<<<(unsigned)((a.nslots + 127) / 128), 128, 0, st>>>(a);
    return cudaGetLastError();
}

cudaError_t launch_mt_prep(const SimPrepArgs &a, unsigned *state, int *pre, cudaStream_t st) {
    k_mt_prep<<<(unsigned)((a.nslots + RP_WARPS - 1) / RP_WARPS), 32 * RP_WARPS, 0, st>>>(a, state, pre);
    return cudaGetLastError();
}

cudaError_t launch_hash_select(const ReplayArgs &a, bool chained, cudaStream_t st) {
    if (a.nslots <= 0) return cudaSuccess;
    const dim3 grid((unsigned)a.nslots), block(HS_THREADS);
    if (a.K <= 2) return launch_chain(chained, k_hash_select<2>, grid, block, 0, st, a);
    if (a.K <= 4) return launch_chain(chained, k_hash_select<4>, grid, block, 0, st, a);
    if (a.K <= 8) return launch_chain(chained, k_hash_select<8>, grid, block, 0, st, a);
    return launch_chain(chained, k_hash_select<16>, grid, block, 0, st, a);
}

cudaError_t launch_replay(const ReplayArgs &a, bool chained, cudaStream_t st) {
    if (a.nslots <= 0) return cudaSuccess;
    const dim3 grid((unsigned)a.nslots), block(RP_THREADS);
    if (a.K <= 1) return launch_chain(chained, k_replay<1>, grid, block, 0, st, a);
    if (a.K <= 2) return launch_chain(chained, k_replay<2>, grid, block, 0, st, a);
    if (a.K <= 4) return launch_chain(chained, k_replay<4>, grid, block, 0, st, a);
    if (a.K <= 8) return launch_chain(chained, k_replay<8>, grid, block, 0, st, a);
    return launch_chain(chained, k_replay<16>, grid, block, 0, st, a);
}

}  // namespace qsk
