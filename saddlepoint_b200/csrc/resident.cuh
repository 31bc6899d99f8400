// resident.cuh — a whole small LP on chip: many PDHG iterations in one launch.
//
// On a small LP the two launches of an iteration are latency: each is a launch gap, two L2
// round trips (entries, then gathers) and a handful of CTAs on 148 SMs. Here one CTA, or one
// cluster of CTAs, keeps the LP in shared memory — the gathered vectors whole in every CTA,
// the row inputs and the matrix entries of its own rows (the entries in L2 where they do not
// fit) — and runs epochs of iterations with their checks inside one launch, its only
// synchronisation the CTA's or the cluster's hardware barrier (nothing spins).
//
// Rows are renumbered. Each matrix's rows are ordered by decreasing length and cut into
// tasks: slices of 32 short rows (at most SEQ_MAX entries) stored column-major, so that
// lane `lane` of a warp walks its own row with loads coalesced across the warp, and groups
// of warp rows stored as 32-entry chunks. Tasks are dealt to the warps longest first, each
// to the least loaded warp; positions number the rows in the order of the warps that own
// them, and the column indices of the other matrix are renamed to positions, so every row
// vector is read and written in place of its thread without a permutation.
//
// What bounds an iteration here is latency: the chain of instructions of the longest warp, at
// 4-9 clocks each, shared memory's (a gather of 32 entries takes about six of its clocks, bank
// conflicts included, which keeps it 30 % busy), L2's where the entries are there, and with a
// cluster its barrier and the fence of the release. So the first entries of each warp's first rows stay in registers; an entry
// in shared memory is its value and the place of its vector entry in 16 bits; slots of padding
// hold -0.0 and the place of a 1.0, so that their product -0.0 changes no sum and the loops
// carry no predicates; the vectors' places in shared memory are constants of the kernel; and
// the dual step's division by sigma is five multiply-adds (SigmaDivisor).
//
// Measured (µs per iteration with its share of the checks, FP64, tile engine -> here; B200):
// 200 x 400 with 1.8k nonzeros 8.8 -> 1.55; 1,417 x 2,834 with 15.6k 9.5 -> 2.8; 3,000 x 6,000
// with 30k (entries in shared memory still) 9.6 -> 4.2. Half of the small ones' time is the two
// barriers and the check (16-26 µs each).
//
// Results are the tile engine's, bit for bit: a short row is summed by one thread in column
// order from -0.0, a warp row as lane-strided partials and the fixed shuffle tree; a pass
// with partial sums stores each row's contributions and res_fold adds them per tile in the
// tile engine's order, res_total over the tiles in the controller's. The engine takes LPs
// without rows longer than TILE_NNZ whose vectors fit.
#pragma once

#include <algorithm>
#include <queue>
#include <vector>

#include "solver_kernels.cuh"

namespace sp {

constexpr int RES_BT = 512;             // threads per CTA
constexpr int RES_W = RES_BT / 32;      // warps per CTA
constexpr int RES_GROUPS = RES_BT / NT; // tiles a CTA folds at once
constexpr int RES_CLUSTER = 8;          // CTAs of a cluster (the portable size)
constexpr int RES_WTAB = 64;            // Halpern weights formed ahead
constexpr int RES_HEAVY_CHUNKS = 16;    // chunks of a group of warp rows (a longer row is alone)
constexpr int RES_MAX_ROWS = 65534;     // 16-bit positions, and one for the padding's 1.0
static_assert(RES_BT % NT == 0 && RES_GROUPS >= 1, "whole tile groups");

// A task: x = its first slot and y = its first position (both from its CTA's first), z = its
// rows, w = the width of a slice, or minus the chunks of each of a group of warp rows (both
// even in a plan of pairs).
using ResTask = int4;

// The plan of one matrix (host), but for which row is at which position.
struct ResCuts {
    std::vector<ResTask> tasks;   // by CTA, then warp
    std::vector<int> first;       // [tasks] each task's first row in the order of decreasing length
    std::vector<int> wt;          // [ctas * RES_W + 1] first task of each warp
    std::vector<int> p0, s0;      // [ctas + 1] first position and first slot of each CTA
    int64_t slots = 0;
    int most_rows = 0, most_slots = 0, most_tasks = 0;  // of one CTA
    bool heavy = false;
};

// Host: cuts the rows, `count[l]` of them with l entries, into tasks and deals these to the
// warps of `ctas` CTAs. pairs: widths and chunks are even. Nothing else about the rows matters.
inline void res_cut(const std::vector<int> &count, int ctas, bool pairs, ResCuts *P) {
    const int odd = pairs ? 1 : 0;
    struct Cut {
        int first, cnt, width, slots, cost;
    };
    std::vector<Cut> cuts;
    int o = 0;
    int l = (int)count.size() - 1;
    auto chunks = [&](int len) { return ((len + 31) / 32 + odd) & ~odd; };
    while (l > SEQ_MAX) {  // groups of rows of the same number of chunks
        const int ch = chunks(l), most = std::max(1, RES_HEAVY_CHUNKS / ch);
        int n = 0;
        for (; l > SEQ_MAX && chunks(l) == ch; --l) n += count[l];
        for (; n > 0; n -= std::min(n, most)) {
            const int cnt = std::min(n, most);
            cuts.push_back(Cut{o, cnt, -ch, 32 * ch * cnt, 8 + cnt * (4 + ch)});
            o += cnt;
        }
    }
    int rest = 0;  // rows that the open slice still takes
    for (; l >= 0; --l)
        for (int n = count[l]; n > 0;) {
            if (rest == 0) {
                const int w = (l + odd) & ~odd;
                cuts.push_back(Cut{o, 0, w, 32 * w, 8 + w});
                rest = 32;
            }
            const int k = std::min(n, rest);
            cuts.back().cnt += k;
            o += k;
            rest -= k;
            n -= k;
        }
    // a few tasks to a warp: longest first, each to the least loaded warp (ties: CTA after CTA);
    // many: in turn, there and back. Turn k counts CTAs fastest: warp k / ctas of CTA k % ctas.
    const int nw = ctas * RES_W, nc = (int)cuts.size();
    std::vector<int> of((size_t)nc), by((size_t)nc);
    for (int c = 0; c < nc; ++c) by[c] = c;
    if (nc <= 16 * nw) {
        std::stable_sort(by.begin(), by.end(), [&](int a, int b) { return cuts[a].cost > cuts[b].cost; });
        using Load = std::pair<int, int>;
        std::priority_queue<Load, std::vector<Load>, std::greater<Load>> heap;
        for (int k = 0; k < nw; ++k) heap.push({0, k});
        for (int c : by) {
            const Load x = heap.top();
            heap.pop();
            of[c] = x.second;
            heap.push({x.first + cuts[c].cost, x.second});
        }
    } else {
        for (int c = 0; c < nc; ++c) of[c] = (c / nw) & 1 ? nw - 1 - c % nw : c % nw;
    }
    P->wt.assign((size_t)nw + 1, 0);
    auto warp_of = [&](int c) { return of[c] % ctas * RES_W + of[c] / ctas; };
    for (int c = 0; c < nc; ++c) ++P->wt[warp_of(c) + 1];
    for (int w = 0; w < nw; ++w) P->wt[w + 1] += P->wt[w];
    std::vector<int> at(P->wt.begin(), P->wt.end() - 1), list((size_t)nc);
    for (int c : by) list[at[warp_of(c)]++] = c;
    P->tasks.resize((size_t)nc);
    P->first.resize((size_t)nc);
    P->p0.assign((size_t)ctas + 1, 0);
    P->s0.assign((size_t)ctas + 1, 0);
    int pos = 0, slot = 0;
    for (int w = 0; w < nw; ++w) {
        const int c = w / RES_W;
        if (w % RES_W == 0) {
            P->p0[c] = pos;
            P->s0[c] = slot;
        }
        for (int t = P->wt[w]; t < P->wt[w + 1]; ++t) {
            const Cut &q = cuts[list[t]];
            P->heavy |= q.width < 0;
            P->tasks[t] = make_int4(slot - P->s0[c], pos - P->p0[c], q.cnt, q.width);
            P->first[t] = q.first;
            pos += q.cnt;
            slot += q.slots;
        }
    }
    P->p0[ctas] = pos;
    P->s0[ctas] = slot;
    P->slots = slot;
    for (int c = 0; c < ctas; ++c) {
        P->most_rows = std::max(P->most_rows, P->p0[c + 1] - P->p0[c]);
        P->most_slots = std::max(P->most_slots, P->s0[c + 1] - P->s0[c]);
        P->most_tasks = std::max(P->most_tasks, P->wt[(c + 1) * RES_W] - P->wt[c * RES_W]);
    }
}

// The whole plan of a small matrix.
struct ResPlan : ResCuts {
    std::vector<uint16_t> perm;   // [rows] the row at each position
    std::vector<uint16_t> inv;    // [rows] the position of each row
};

// Host: the plan of the matrix with row pointers rp, for `ctas` CTAs.
template <class I>
inline void res_plan(const I *rp, int rows, int ctas, bool pairs, ResPlan *P) {
    int maxlen = 0;
    for (int r = 0; r < rows; ++r) maxlen = std::max(maxlen, (int)(rp[r + 1] - rp[r]));
    std::vector<int> count((size_t)maxlen + 1, 0), start((size_t)maxlen + 2, 0), order((size_t)rows);
    for (int r = 0; r < rows; ++r) ++count[(size_t)(rp[r + 1] - rp[r])];
    res_cut(count, ctas, pairs, P);
    // rows by decreasing length, ties in row order
    for (int l = maxlen; l >= 0; --l) start[(size_t)(maxlen - l) + 1] = start[(size_t)(maxlen - l)] + count[l];
    for (int r = 0; r < rows; ++r) order[(size_t)start[(size_t)(maxlen - (int)(rp[r + 1] - rp[r]))]++] = r;
    P->perm.resize((size_t)rows);
    P->inv.resize((size_t)rows);
    for (int c = 0; c < ctas; ++c)
        for (int t = P->wt[c * RES_W]; t < P->wt[(c + 1) * RES_W]; ++t)
            for (int i = 0; i < P->tasks[t].z; ++i) {
                const int pos = P->p0[c] + P->tasks[t].y + i, r = order[P->first[t] + i];
                P->perm[pos] = (uint16_t)r;
                P->inv[r] = (uint16_t)pos;
            }
}

// ------------------------------------------------------------------ cluster primitives

__device__ __forceinline__ unsigned cluster_rank() {
    unsigned r;
    asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
    return r;
}
__device__ __forceinline__ unsigned cluster_size() {
    unsigned r;
    asm volatile("mov.u32 %0, %%cluster_nctarank;" : "=r"(r));
    return r;
}
// The barrier of a solve's CTAs, a cluster of NC or one: what was written before it, in shared
// memory of any of them and in global memory, is visible after it.
template <int NC>
__device__ __forceinline__ void res_sync() {
    if constexpr (NC > 1) {
        asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
        asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
    } else {
        __syncthreads();
    }
}
// This CTA's number among the solve's, and how many there are (NC = 0: the grid).
template <int NC>
__device__ __forceinline__ int res_rank() {
    return NC > 1 ? (int)cluster_rank() : NC == 1 ? 0 : (int)blockIdx.x;
}
template <int NC>
__device__ __forceinline__ int res_size() {
    return NC > 0 ? NC : (int)gridDim.x;
}
// Writes v to the place of shared variable *p in CTA `rank` of the cluster.
__device__ __forceinline__ void cluster_store(double *p, unsigned rank, double v) {
    unsigned a;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(a) : "r"(smem_u32(p)), "r"(rank));
    asm volatile("st.shared::cluster.f64 [%0], %1;" ::"r"(a), "d"(v) : "memory");
}
__device__ __forceinline__ void cluster_store(float *p, unsigned rank, float v) {
    unsigned a;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(a) : "r"(smem_u32(p)), "r"(rank));
    asm volatile("st.shared::cluster.f32 [%0], %1;" ::"r"(a), "f"(v) : "memory");
}
// Copies this thread's own *p to the same place in the other CTAs of the cluster.
template <int NC, class T>
__device__ __forceinline__ void publish(T *p) {
    if constexpr (NC > 1) {
        const unsigned me = cluster_rank(), n = cluster_size();
        const T v = *p;
        for (unsigned r = 1; r < n; ++r) cluster_store(p, me + r < n ? me + r : me + r - n, v);
    }
}

// ------------------------------------------------------------------ shared memory

// Places in dynamic shared memory. The row inputs of at most PT columns and PA rows lie at
// constant places from 0; the others follow: y and x̄ of the whole LP with a 1.0 past their
// ends (FP32 ones too in the mixed form's FP32 phase), the tasks, and the entries of both
// matrices if they fit: the values by slot, and for each lane's pair of slots o + lane and
// o + 32 + lane (o a multiple of 64) the two places, in units of the value's size.
template <int PT, int PA>
struct ResPlaces {
    static constexpr int X = 0, XA = 8 * PT, C = 16 * PT, LV = 24 * PT, UV = 32 * PT;
    static constexpr int YA = 40 * PT, LC = YA + 8 * PA, UC = YA + 16 * PA, END = YA + 24 * PA;
    int y, xbar, y32, xbar32, tasksA, tasksT, wtA, wtT, valA, valT, atA, atT, total;
    __host__ __device__ static int up(int b) { return (b + 15) & ~15; }
    // lo: with the FP32 vectors; tasks and slots: the most of one CTA (A', A'ᵀ); entries: with
    // entries of vb bytes a value in shared memory
    __host__ __device__ ResPlaces(int m, int n, bool lo, int ta, int tt, int sa, int st, bool entries, int vb) {
        int at = END;
        auto take = [&](int bytes) {
            const int a = at;
            at += up(bytes);
            return a;
        };
        y = take(8 * (m + 1));
        xbar = take(8 * (n + 1));
        y32 = lo ? take(4 * (m + 1)) : 0;
        xbar32 = lo ? take(4 * (n + 1)) : 0;
        tasksA = take((int)sizeof(ResTask) * ta);
        tasksT = take((int)sizeof(ResTask) * tt);
        wtA = take(4 * (RES_W + 1));
        wtT = take(4 * (RES_W + 1));
        valA = entries ? take(vb * sa) : 0;
        valT = entries ? take(vb * st) : 0;
        atA = entries ? take(2 * sa) : 0;
        atT = entries ? take(2 * st) : 0;
        total = at;
    }
};

// One matrix as a CTA sees it: its part of the plan, its entries in global memory (positions
// and values; in shared memory too where the kernel says so), and what the fold needs.
template <class IX>
struct ResSide {
    int rows, p0, p1;       // all rows; this CTA's positions
    int slots, ntasks;      // this CTA's
    int heavy;              // whether the matrix has warp rows
    int ntiles;
    int tasks, wt;          // their places in dynamic shared memory
    const IX *ci;           // [slots]
    const double *v;
    const float *v32;
    const IX *perm;         // all positions
    const int *rp;          // the CSR row pointers, for the fold's row lengths
    const Tile *tiles;
};

// One matrix in global memory: the whole plan and all slots.
template <class IX>
struct ResSrc {
    int rows, heavy, ntiles;
    int most_rows, most_slots, most_tasks;
    const ResTask *tasks;
    const int *wt, *p0, *s0;
    const IX *perm;
    IX *ci;
    double *v;
    float *v32;
    const int *rp;
    const Tile *tiles;
};

template <class IX>
struct ResCtx {
    ResSide<IX> A, T;       // A' (rows i) and A'ᵀ (rows j)
    SolverPtrs S;           // vectors over positions (in any memory)
    double *contrib;        // [8 rows] row contributions of a pass, in row order
    double *contribD, *contribT;
};

// Vectors over positions in global memory that only the checks use.
struct ResVecs {
    double *xt, *aty, *df;  // columns
    double *yt, *pf;        // rows
};

// A CTA's shared variables: the problem's arrays, its copy of the solver's state, and what the
// epochs need between their iterations (kept out of the iterations' registers).
template <class IX>
struct ResShared {
    ResCtx<IX> R;
    DevState st;
    DevParams prm;
    unsigned long long until;   // iterations at which to stop
    sp_check_record *trace;
    long long trace_cap;
    int mixed;
    int count_bad_first;        // a non-finite first iteration counts (the batch's rule)
    float stop;                 // 1: the batch's hand-off is due (every CTA's copy, by rank 0)
    double sh[RES_GROUPS * NP_P * (NT / 32) + NP_P];
    double wtab[RES_WTAB];
};

template <class T>
__device__ __forceinline__ T &dsm_at(int place) {
    extern __shared__ __align__(16) unsigned char dsm[];
    return *reinterpret_cast<T *>(dsm + place);
}

template <class IX>
__device__ __forceinline__ ResSide<IX> res_side(const ResSrc<IX> &M, int c, int tasks, int wt) {
    ResSide<IX> d;
    d.rows = M.rows;
    d.p0 = M.p0[c];
    d.p1 = M.p0[c + 1];
    d.slots = M.s0[c + 1] - M.s0[c];
    d.ntasks = M.wt[(c + 1) * RES_W] - M.wt[c * RES_W];
    d.heavy = M.heavy;
    d.ntiles = M.ntiles;
    d.tasks = tasks;
    d.wt = wt;
    d.ci = M.ci + M.s0[c];
    d.v = M.v + M.s0[c];
    d.v32 = M.v32 ? M.v32 + M.s0[c] : nullptr;
    d.perm = M.perm;
    d.rp = M.rp;
    d.tiles = M.tiles;
    return d;
}

// Sets sh.R up for CTA c and copies the plan into shared memory (not the entries). R.S keeps
// its other pointers. Ends with a barrier.
template <int PT, int PA, class IX>
__device__ inline void res_open(ResShared<IX> &sh, const ResPlaces<PT, PA> &L, const ResSrc<IX> &A, const ResSrc<IX> &T,
                                const SolverPtrs &g, const ResVecs &vec, double *contrib, int c) {
    if (threadIdx.x == 0) {
        ResCtx<IX> &R = sh.R;
        R.A = res_side(A, c, L.tasksA, L.wtA);
        R.T = res_side(T, c, L.tasksT, L.wtT);
        R.S = g;
        SolverPtrs &S = R.S;
        const int pt = R.T.p0, pa = R.A.p0;
        using P = ResPlaces<PT, PA>;
        S.x = &dsm_at<double>(P::X) - pt;
        S.xa = &dsm_at<double>(P::XA) - pt;
        S.c = &dsm_at<double>(P::C) - pt;
        S.lv = &dsm_at<double>(P::LV) - pt;
        S.uv = &dsm_at<double>(P::UV) - pt;
        S.ya = &dsm_at<double>(P::YA) - pa;
        S.lc = &dsm_at<double>(P::LC) - pa;
        S.uc = &dsm_at<double>(P::UC) - pa;
        S.y = &dsm_at<double>(L.y);
        S.xbar = &dsm_at<double>(L.xbar);
        S.y32 = L.y32 ? &dsm_at<float>(L.y32) : nullptr;
        S.xbar32 = L.xbar32 ? &dsm_at<float>(L.xbar32) : nullptr;
        S.xt = vec.xt;
        S.aty = vec.aty;
        S.df = vec.df;
        S.yt = vec.yt;
        S.pf = vec.pf;
        R.contrib = contrib;
        R.contribD = contrib + 8ll * T.rows;
        R.contribT = R.contribD + 8ll * A.rows;
        S.y[A.rows] = 1.0;
        S.xbar[T.rows] = 1.0;
        if (S.y32) {
            S.y32[A.rows] = 1.0f;
            S.xbar32[T.rows] = 1.0f;
        }
        // the padding's records in the checks' gathers
        S.pk[T.rows] = CheckQuad{1.0, 1.0, 1.0, 1.0};
        S.pky[A.rows] = make_double2(1.0, 1.0);
    }
    for (const ResSrc<IX> *M : {&A, &T}) {
        const int *wt = M->wt + c * RES_W;
        const int tasks = M == &A ? L.tasksA : L.tasksT, to = M == &A ? L.wtA : L.wtT, n = wt[RES_W] - wt[0];
        for (int i = threadIdx.x; i < n; i += RES_BT) (&dsm_at<ResTask>(tasks))[i] = M->tasks[wt[0] + i];
        if (threadIdx.x <= RES_W) (&dsm_at<int>(to))[threadIdx.x] = wt[threadIdx.x] - wt[0];
    }
    __syncthreads();
}

// The CTA's entries of one matrix into shared memory; `base` is the place of the vector they
// gather.
template <class VT, class IX>
__device__ inline void res_load_entries(const ResSide<IX> &M, const VT *v, int val, int at, int base) {
    for (int i = threadIdx.x; i < M.slots; i += RES_BT) (&dsm_at<VT>(val))[i] = v[i];
    for (int i = threadIdx.x; i < M.slots / 2; i += RES_BT) {
        const int o = (i & ~31) * 2 + (i & 31);
        const unsigned b = (unsigned)base / (unsigned)sizeof(VT);
        (&dsm_at<unsigned>(at))[i] = (b + M.ci[o]) | (b + M.ci[o + 32]) << 16;
    }
}

// ------------------------------------------------------------------ sums of a task's rows

// Two entries of a lane's row: values, and the places of what they multiply.
template <class VT>
struct ResPair {
    VT v0, v1;
    unsigned at;
    __device__ __forceinline__ VT p0() const { return v0 * dsm_at<const VT>((int)((at & 0xffffu) * sizeof(VT))); }
    __device__ __forceinline__ VT p1() const { return v1 * dsm_at<const VT>((int)((at >> 16) * sizeof(VT))); }
};
constexpr int RES_HEAD = 4;  // pairs of a warp's first task that stay in registers

// Entries of one matrix for this lane: in shared memory (ES), or positions and values in
// global memory.
template <class VT, bool ES>
struct ResEntries {
    int val, at;         // ES: their places; else at = the place of the gathered vector
    const uint16_t *ci;
    const VT *v;
    __device__ __forceinline__ ResEntries(const ResSide<uint16_t> &M, const VT *vals, int val_, int at_, int base) {
        const int lane = threadIdx.x & 31;
        const unsigned b = (unsigned)base / (unsigned)sizeof(VT);
        if constexpr (ES) {
            val = val_ + (int)sizeof(VT) * lane;
            at = at_ + 4 * lane;
        } else {
            at = (int)b;
            ci = M.ci + lane;
            v = vals + lane;
        }
    }
    // the pair at slots o, o + 32 (o a multiple of 64)
    __device__ __forceinline__ ResPair<VT> pair(int o) const {
        ResPair<VT> q;
        if constexpr (ES) {
            q.v0 = dsm_at<const VT>(val + (int)sizeof(VT) * o);
            q.v1 = dsm_at<const VT>(val + (int)sizeof(VT) * (o + 32));
            q.at = dsm_at<const unsigned>(at + 2 * o);
        } else {
            q.v0 = v[o];
            q.v1 = v[o + 32];
            q.at = ((unsigned)at + ci[o]) | ((unsigned)at + ci[o + 32]) << 16;
        }
        return q;
    }
};

// The first pairs of a slice, padded with pairs whose products are -0.0 (`one`: the place of
// a 1.0 behind the gathered vector).
template <class VT>
struct ResHead {
    ResPair<VT> q[RES_HEAD];
    template <bool ES>
    __device__ __forceinline__ void load(const ResEntries<VT, ES> &E, const ResTask &t, int one) {
        const unsigned u = (unsigned)one / (unsigned)sizeof(VT);
#pragma unroll
        for (int i = 0; i < RES_HEAD; ++i) {
            if (2 * i < t.w) q[i] = E.pair(t.x + 64 * i);
            else q[i] = ResPair<VT>{VT(-0.0), VT(-0.0), u | u << 16};
        }
    }
};

template <int N, class VT>
__device__ __forceinline__ void res_add(const ResPair<VT> *q, VT &s) {
    VT p[2 * N];
#pragma unroll
    for (int i = 0; i < N; ++i) {
        p[2 * i] = q[i].p0();
        p[2 * i + 1] = q[i].p1();
    }
#pragma unroll
    for (int i = 0; i < 2 * N; ++i) s += p[i];
}

// Adds `w` entries (even) from slot `o` on, 32 slots apart, in order; the next four are
// loaded before these are added.
template <class VT, bool ES>
__device__ __forceinline__ void res_walk(const ResEntries<VT, ES> &E, int o, int w, VT &s) {
    if (w >= 4) {
        ResPair<VT> q[2] = {E.pair(o), E.pair(o + 64)};
#pragma unroll 1
        for (; w >= 8; w -= 4) {
            o += 128;
            const ResPair<VT> n0 = E.pair(o), n1 = E.pair(o + 64);
            res_add<2>(q, s);
            q[0] = n0;
            q[1] = n1;
        }
        res_add<2>(q, s);
        o += 128;
        w -= 4;
    }
    if (w > 0) {
        const ResPair<VT> q = E.pair(o);
        res_add<1>(&q, s);
    }
}

// The sums of task t's rows: lane `lane` returns that of the task's row `lane`. `head`: the
// task's first pairs, or null.
template <class VT, bool ES>
__device__ __forceinline__ double res_sum(const ResEntries<VT, ES> &E, const ResTask &t, const ResHead<VT> *head) {
    if (t.w >= 0) {
        VT s = VT(-0.0);
        if (head) {
            res_add<RES_HEAD / 2>(head->q, s);
            if (t.w > RES_HEAD) res_add<RES_HEAD / 2>(head->q + RES_HEAD / 2, s);
            if (t.w > 2 * RES_HEAD) res_walk<VT, ES>(E, t.x + 64 * RES_HEAD, t.w - 2 * RES_HEAD, s);
        } else {
            res_walk<VT, ES>(E, t.x, t.w, s);
        }
        return double(s);
    }
    const int lane = threadIdx.x & 31;
    double r = 0.0;
    int o = t.x;
#pragma unroll 1
    for (int i = 0; i < t.z; ++i, o -= 32 * t.w) {
        VT s = VT(-0.0);
        res_walk<VT, ES>(E, o, -t.w, s);
        const VT tot = __shfl_sync(0xffffffffu, warp_sum_down(s), 0);
        if (lane == i) r = double(tot);
    }
    return r;
}

// ------------------------------------------------------------------ partial sums

// The warp sums (warp_sum_down's tree) of K values at once, K a power of two up to 8: at
// each step the lower lanes keep one half of the values and the upper lanes the other, so
// that K = 8 costs 9 exchanges instead of 40. Value q ends in the lanes with
// lane / (32 / K) == q. The pairs that are added are the tree's (an addition commutes).
template <int K>
__device__ __forceinline__ double warp_sums(const double (&v)[K], int o = 16) {
    const int lane = threadIdx.x & 31;
    if constexpr (K == 1) {
        double s = v[0];
        for (; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
        return s;
    } else {
        double h[K / 2];
        const bool up = (lane & o) != 0;
#pragma unroll
        for (int q = 0; q < K / 2; ++q) {
            const double keep = up ? v[q + K / 2] : v[q], send = up ? v[q] : v[q + K / 2];
            h[q] = keep + __shfl_xor_sync(0xffffffffu, send, o);
        }
        return warp_sums<K / 2>(h, o / 2);
    }
}
__host__ __device__ constexpr int pow2_up(int k) { return k <= 1 ? 1 : k <= 2 ? 2 : k <= 4 ? 4 : 8; }

// First half of a block tree over NT threads: warp `warp`'s sums into sh[q][warp].
template <int NP>
__device__ __forceinline__ void tree_warps(const double (&v)[NP], double *sh, int warp) {
    constexpr int K = pow2_up(NP), L = 32 / K;
    const int lane = threadIdx.x & 31, q = lane / L;
    double w[K];
#pragma unroll
    for (int i = 0; i < K; ++i) w[i] = i < NP ? v[i < NP ? i : 0] : 0.0;
    const double s = warp_sums<K>(w);
    if (lane % L == 0 && q < NP) sh[q * (NT / 32) + warp] = s;
}
// Second half, by one warp: calls out(q, sum) on one lane for each value.
template <int NP, class Out>
__device__ __forceinline__ void tree_total(const double *sh, Out out) {
    constexpr int W = NT / 32;
    static_assert(W == 8, "groups of 8 lanes");
    const int lane = threadIdx.x & 31;
#pragma unroll
    for (int q0 = 0; q0 < NP; q0 += 4) {
        const int q = q0 + lane / W;
        double s = q < NP ? sh[q * W + lane % W] : 0.0;
#pragma unroll
        for (int o = W / 2; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
        if (lane % W == 0 && q < NP) out(q, s);
    }
}

// The block tree over the values of the CTA's first NT threads; every thread returns the sums.
template <int NP>
__device__ __forceinline__ void res_tree(double (&v)[NP], double *sh) {
    if (threadIdx.x < NT) tree_warps<NP>(v, sh, threadIdx.x >> 5);
    __syncthreads();
    if (threadIdx.x < 32) {
        double *o = sh + NP * (NT / 32);
        tree_total<NP>(sh, [&](int q, double t) { o[q] = t; });
    }
    __syncthreads();
#pragma unroll
    for (int q = 0; q < NP; ++q) v[q] = sh[NP * (NT / 32) + q];
    __syncthreads();
}

// The tile partials [ntiles][NP] of a pass from its contributions, in the tile engine's
// order: thread u of a tile its short rows u, u + NT, ..., lane 0 of warp w the warp rows
// w, w + 8, ..., then the block tree. Groups of NT threads take a tile each, over all of the
// solve's CTAs. Contributions are read from L2 (another CTA may have written them).
template <int NC, int NP, class IX>
__device__ __forceinline__ void res_fold(const ResSide<IX> &M, const double *contrib, double *part, double *sh) {
    constexpr int W = NT / 32;
    const int g = threadIdx.x / NT, tid = threadIdx.x % NT, warp = tid >> 5, lane = tid & 31;
    const int c = res_rank<NC>(), nc = res_size<NC>();
    const int step = nc * RES_GROUPS;
    double *gsh = sh + g * NP * W;
    for (int base = c * RES_GROUPS; base < M.ntiles; base += step) {
        const int tile = base + g;
        if (tile < M.ntiles) {
            const Tile t = M.tiles[tile];
            const int r0 = t.x, nr = t.y - t.x;
            double v[NP];
#pragma unroll
            for (int q = 0; q < NP; ++q) v[q] = 0.0;
            for (int u = tid; u < nr; u += NT) {
                if (M.heavy && M.rp[r0 + u + 1] - M.rp[r0 + u] > SEQ_MAX) continue;
#pragma unroll
                for (int q = 0; q < NP; ++q) v[q] += __ldcg(contrib + (int64_t)q * M.rows + r0 + u);
            }
            for (int b = warp; M.heavy && b < nr; b += 32 * W) {
                const int i = b + lane * W;
                const bool heavy = i < nr && M.rp[r0 + i + 1] - M.rp[r0 + i] > SEQ_MAX;
                for (unsigned mask = __ballot_sync(0xffffffffu, heavy); mask; mask &= mask - 1) {
                    const int r = r0 + b + (__ffs(mask) - 1) * W;
                    if (lane == 0) {
#pragma unroll
                        for (int q = 0; q < NP; ++q) v[q] += __ldcg(contrib + (int64_t)q * M.rows + r);
                    }
                }
            }
            tree_warps<NP>(v, gsh, warp);
        }
        __syncthreads();
        if (tile < M.ntiles && warp == 0) tree_total<NP>(gsh, [&](int q, double t) { part[(int64_t)tile * NP + q] = t; });
        __syncthreads();
    }
}

// The controller's sum over the tiles (control.cuh: sum_slots).
template <int NP>
__device__ __forceinline__ void res_total(const double *part, int tiles, double (&out)[NP], double *sh) {
#pragma unroll
    for (int q = 0; q < NP; ++q) out[q] = 0.0;
    if (threadIdx.x < NT)
        for (int t = threadIdx.x; t < tiles; t += NT)
#pragma unroll
            for (int q = 0; q < NP; ++q) out[q] += __ldcg(part + (int64_t)t * NP + q);
    res_tree<NP>(out, sh);
}

// ------------------------------------------------------------------ the checks' passes

// The solver's passes on positions. Their row() is the solver's.
template <int NC, bool LO, int MODE>
struct ResPrimal : PrimalPass<LO, MODE> {
    using Base = PrimalPass<LO, MODE>;
    using Pre = typename Base::Pre;
    using VT = typename Base::VT;
    using ST = typename Base::ST;
    __device__ __forceinline__ void prod(int c, VT v, ST (&p)[1]) const {
        if constexpr (LO) p[0] = v * this->s.y32[c];
        else p[0] = v * this->s.y[c];
    }
    __device__ __forceinline__ Pre pre_at(int k) const {
        const SolverPtrs &s = this->s;
        return Pre{s.x[k], s.c[k], s.lv[k], s.uv[k], MODE == 1 ? 0.0 : s.xa[k]};
    }
    __device__ __forceinline__ void publish_at(int) const {}  // the dual pass gathers the column records
};

template <int NC, bool LO, int MODE>
struct ResDual : DualPass<LO, MODE> {
    using Base = DualPass<LO, MODE>;
    using Pre = typename Base::Pre;
    using VT = typename Base::VT;
    using ST = typename Base::ST;
    __device__ __forceinline__ void prod(int c, VT v, ST (&p)[Base::G]) const {
        const double2 *q = reinterpret_cast<const double2 *>(this->s.pk + c);
        const double2 q0 = __ldcg(q);
        if constexpr (LO) p[0] = ST((float)v * (float)q0.x);
        else p[0] = v * q0.x;
        p[1] = v * q0.y;
        if constexpr (MODE == 2) {
            const double2 q1 = __ldcg(q + 1);
            p[2] = v * q1.x;
            p[3] = v * q1.y;
        }
    }
    __device__ __forceinline__ Pre pre_at(int k) const {
        const SolverPtrs &s = this->s;
        return Pre{s.y[k], s.lc[k], s.uc[k], s.ya[k], MODE == 2 ? s.pf[k] : 0.0};
    }
    __device__ __forceinline__ void publish_at(int k) const {
        if constexpr (MODE == 1) {
            if constexpr (LO) publish<NC>(this->s.y32 + k);
            else publish<NC>(this->s.y + k);
        }
    }
};

struct ResCheckT : CheckPassT {
    __device__ __forceinline__ void prod(int c, double v, double (&p)[2]) const {
        const double2 q = __ldcg(s.pky + c);
        p[0] = v * q.x;
        p[1] = v * q.y;
    }
    __device__ __forceinline__ Pre pre_at(int k) const {
        return Pre{s.lv[k], s.uv[k], s.df[k], s.c[k], s.aty[k], s.xt[k], s.x[k]};
    }
    __device__ __forceinline__ void publish_at(int) const {}
};

// A check pass over this CTA's rows of M, its entries from global memory: each row's NP
// contributions are left in contrib ([NP][rows], row order).
template <class Op, class IX>
__device__ __forceinline__ void res_pass(const ResSide<IX> &M, const Op &op, double *contrib) {
    using VT = typename Op::VT;
    using ST = typename Op::ST;
    constexpr int G = Op::G, NP = Op::NP;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const VT *vals;
    if constexpr (sizeof(VT) == 4) vals = M.v32;
    else vals = M.v;
    const int t1 = (&dsm_at<int>(M.wt))[warp + 1];
#pragma unroll 1
    for (int ti = (&dsm_at<int>(M.wt))[warp]; ti < t1; ++ti) {
        const ResTask t = (&dsm_at<ResTask>(M.tasks))[ti];
        const int k = M.p0 + t.y + lane;
        const bool live = lane < t.z;
        typename Op::Pre pre{};
        if (live) pre = op.pre_at(k);
        double s[G];
        int o = t.x + lane;
        auto add = [&](SlotSums<G, Op::F32> &acc, auto count) {
            constexpr int N = decltype(count)::value;
            ST p[N][G];
#pragma unroll
            for (int u = 0; u < N; ++u) op.prod(M.ci[o + 32 * u], vals[o + 32 * u], p[u]);
#pragma unroll
            for (int u = 0; u < N; ++u) acc.add(p[u]);
        };
        SlotSums<G, Op::F32> acc;
        if (t.w >= 0) {
            acc.clear();
            int j = 0;
#pragma unroll 2
            for (; j + 2 <= t.w; j += 2, o += 64) add(acc, std::integral_constant<int, 2>{});
            if (j < t.w) add(acc, std::integral_constant<int, 1>{});
#pragma unroll
            for (int q = 0; q < G; ++q) s[q] = acc.get(q);
        } else {
#pragma unroll
            for (int q = 0; q < G; ++q) s[q] = 0.0;
#pragma unroll 1
            for (int i = 0; i < t.z; ++i) {
                acc.clear();
#pragma unroll 1
                for (int c = 0; c < -t.w; ++c, o += 32) {
                    ST p[G];
                    op.prod(M.ci[o], vals[o], p);
                    acc.add(p);
                }
#pragma unroll
                for (int q = 0; q < G; ++q) {
                    double tot;
                    if ((Op::F32 >> q) & 1u) tot = double(__shfl_sync(0xffffffffu, warp_sum_down(acc.f[q]), 0));
                    else tot = __shfl_sync(0xffffffffu, warp_sum_down(acc.d[q]), 0);
                    if (lane == i) s[q] = tot;
                }
            }
        }
        if (live) {
            double part[NP];
#pragma unroll
            for (int q = 0; q < NP; ++q) part[q] = 0.0;
            op.row(k, s, part, pre);
            op.publish_at(k);
            const int r = M.perm[k];
#pragma unroll
            for (int q = 0; q < NP; ++q) contrib[(int64_t)q * M.rows + r] = part[q];
        }
    }
}

template <int NC, bool LO, int MODE, class IX>
__device__ __forceinline__ void res_primal(const ResCtx<IX> &R, const IterScalars &sc) {
    ResPrimal<NC, LO, MODE> o{};
    o.s = R.S;
    o.sc = sc;
    res_pass(R.T, o, R.contrib);
}
template <int NC, bool LO, int MODE, class IX>
__device__ __forceinline__ void res_dual(const ResCtx<IX> &R, const IterScalars &sc) {
    ResDual<NC, LO, MODE> o{};
    o.s = R.S;
    o.sc = sc;
    res_pass(R.A, o, R.contribD);
}

// ------------------------------------------------------------------ the iterations

// Places of a shared array's elements in the other CTAs of the cluster.
template <int NC>
struct ResPeers {
    unsigned base[NC > 1 ? NC - 1 : 1];
    __device__ __forceinline__ ResPeers() {
        if constexpr (NC > 1) {
            const unsigned me = cluster_rank();
#pragma unroll
            for (int u = 0; u < NC - 1; ++u)
                asm volatile("mapa.shared::cluster.u32 %0, %1, %2;"
                             : "=r"(base[u])
                             : "r"(smem_u32(&dsm_at<int>(0))), "r"((me + 1 + u) % NC));
        }
    }
    __device__ __forceinline__ void put(int place, double v) const {
        if constexpr (NC > 1) {
#pragma unroll
            for (int u = 0; u < NC - 1; ++u)
                asm volatile("st.shared::cluster.f64 [%0], %1;" ::"r"(base[u] + place), "d"(v) : "memory");
        }
    }
    __device__ __forceinline__ void put(int place, float v) const {
        if constexpr (NC > 1) {
#pragma unroll
            for (int u = 0; u < NC - 1; ++u)
                asm volatile("st.shared::cluster.f32 [%0], %1;" ::"r"(base[u] + place), "f"(v) : "memory");
        }
    }
};

// `its` FUSED iterations from Halpern counter k0. HEADS: each pass's first head stays in registers.
// With entries in global memory that suits a kernel with room for it (a 3,500 x 7,000 LP in
// the solver's: 5.7 µs an iteration, 6.1 without), not the batch's, whose shorter paths then
// spill (its 1,024 LPs of 50-2,000 rows: 32.0 ms, 30.5 without).
template <int NC, bool LO, bool ES, bool HEADS, int PT, int PA>
__device__ __forceinline__ void res_iterate(ResShared<uint16_t> &sh, const ResPlaces<PT, PA> &L, unsigned long long k0,
                                            unsigned long long its) {
    using VT = typename std::conditional<LO, float, double>::type;
    using P = ResPlaces<PT, PA>;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const double rho = sh.prm.reflection, tau = sh.prm.eta / sh.st.omega, sigma = sh.prm.eta * sh.st.omega;
    const SigmaDivisor by_sigma(sigma);
    const ResPeers<NC> peers;
    const VT *vT, *vA;
    if constexpr (LO) {
        vT = sh.R.T.v32;
        vA = sh.R.A.v32;
    } else {
        vT = sh.R.T.v;
        vA = sh.R.A.v;
    }
    const int gy = LO ? L.y32 : L.y, gx = LO ? L.xbar32 : L.xbar;  // the gathered vectors
    const ResEntries<VT, ES> ET(sh.R.T, vT, L.valT, L.atT, gy), EA(sh.R.A, vA, L.valA, L.atA, gx);
    const int xg = (LO ? L.xbar32 : L.xbar) + (int)sizeof(VT) * sh.R.T.p0;  // this CTA's part of x̄ and y
    const int yg = (LO ? L.y32 : L.y) + (int)sizeof(VT) * sh.R.A.p0;
    const int yd = L.y + 8 * sh.R.A.p0;
    const int t0 = (&dsm_at<int>(L.wtT))[warp], t1 = (&dsm_at<int>(L.wtT))[warp + 1];
    const int a0 = (&dsm_at<int>(L.wtA))[warp], a1 = (&dsm_at<int>(L.wtA))[warp + 1];
    ResHead<VT> hT, hA;
    if (HEADS && t0 < t1) hT.load(ET, (&dsm_at<ResTask>(L.tasksT))[t0], gy + (int)sizeof(VT) * sh.R.A.rows);
    if (HEADS && a0 < a1) hA.load(EA, (&dsm_at<ResTask>(L.tasksA))[a0], gx + (int)sizeof(VT) * sh.R.T.rows);
    double w = 0.0;
    // A task's rows: PrimalPass and DualPass with MODE 0 (solver_kernels.cuh) on positions.
    auto primal = [&](const ResTask t, const ResHead<VT> *head) {
        const double aty = res_sum<VT, ES>(ET, t, head);
        if (lane < t.z) {
            const int k = t.y + lane, k8 = 8 * k;
            const double xj = dsm_at<double>(P::X + k8);
            const double xt = clampd(xj - tau * (dsm_at<double>(P::C + k8) - aty), dsm_at<double>(P::LV + k8),
                                     dsm_at<double>(P::UV + k8));
            const VT xb = VT(2.0 * xt - xj);
            dsm_at<VT>(xg + (int)sizeof(VT) * k) = xb;
            peers.put(xg + (int)sizeof(VT) * k, xb);
            dsm_at<double>(P::X + k8) = halpern(xj, xt, dsm_at<double>(P::XA + k8), w, rho);
        }
    };
    auto dual = [&](const ResTask t, const ResHead<VT> *head) {
        const double a = res_sum<VT, ES>(EA, t, head);
        if (lane < t.z) {
            const int k = t.y + lane, k8 = 8 * k;
            const double yi = dsm_at<double>(yd + k8);
            const double v = a - by_sigma(yi);
            const double yt = yi - sigma * (a - clampd(v, dsm_at<double>(P::LC + k8), dsm_at<double>(P::UC + k8)));
            const double yn = halpern(yi, yt, dsm_at<double>(P::YA + k8), w, rho);
            dsm_at<double>(yd + k8) = yn;
            if constexpr (LO) dsm_at<float>(yg + 4 * k) = (float)yn;
            peers.put(yg + (int)sizeof(VT) * k, VT(yn));
        }
    };
#pragma unroll 1
    while (its > 0) {
        const int cnt = (int)min((unsigned long long)RES_WTAB, its);
        if (threadIdx.x < RES_WTAB) {  // every reader of the last weights is past a barrier
            const unsigned long long k = k0 + threadIdx.x;
            sh.wtab[threadIdx.x] = (double)(k + 1) / (double)(k + 2);
        }
        k0 += (unsigned long long)cnt;
        its -= (unsigned long long)cnt;
        __syncthreads();
#pragma unroll 1
        for (int i = 0; i < cnt; ++i) {
            w = sh.wtab[i];
            if (t0 < t1) primal((&dsm_at<ResTask>(L.tasksT))[t0], HEADS ? &hT : nullptr);
#pragma unroll 1
            for (int ti = t0 + 1; ti < t1; ++ti) primal((&dsm_at<ResTask>(L.tasksT))[ti], nullptr);
            res_sync<NC>();
            if (a0 < a1) dual((&dsm_at<ResTask>(L.tasksA))[a0], HEADS ? &hA : nullptr);
#pragma unroll 1
            for (int ti = a0 + 1; ti < a1; ++ti) dual((&dsm_at<ResTask>(L.tasksA))[ti], nullptr);
            res_sync<NC>();
        }
    }
}

template <class IX>
__device__ __forceinline__ IterScalars res_scalars(const ResShared<IX> &sh, double w) {
    IterScalars sc;
    sc.tau = sh.prm.eta / sh.st.omega;
    sc.sigma = sh.prm.eta * sh.st.omega;
    sc.w = w;
    sc.rho = sh.prm.reflection;
    return sc;
}

// The k = 0 iteration that opens an epoch: both passes with their residual sums, x's
// Halpern step, and the anchor's residual (solver.rs:341-346). Non-finite iterates end the solve.
template <int NC, bool LO, class IX>
__device__ __noinline__ void res_first(ResShared<IX> &sh) {
    const ResCtx<IX> &R = sh.R;
    const IterScalars sc = res_scalars(sh, 1.0 / 2.0);
    res_primal<NC, LO, 1>(R, sc);
    res_sync<NC>();
    res_dual<NC, LO, 1>(R, sc);
    for (int k = R.T.p0 + threadIdx.x; k < R.T.p1; k += RES_BT)
        R.S.x[k] = halpern(R.S.x[k], R.S.xt[k], R.S.xa[k], sc.w, sc.rho);
    res_sync<NC>();
    res_fold<NC, NP_P0>(R.T, R.contrib, R.S.partP0, sh.sh);
    res_fold<NC, NP_D0>(R.A, R.contribD, R.S.partD0, sh.sh);
    res_sync<NC>();
    double P0[NP_P0], D0[NP_D0];
    res_total<NP_P0>(R.S.partP0, R.T.ntiles, P0, sh.sh);
    res_total<NP_D0>(R.S.partD0, R.A.ntiles, D0, sh.sh);
    if (threadIdx.x == 0) {
        bool bad = false;
        DevState &st = sh.st;
        st.anchor_residual = fixed_point_residual(sh.prm.eta, st.omega, P0[0], D0[0], D0[1], &bad);
        if (bad) {
            st.error = ERR_NUMERICAL_ITERATES;
            st.done = 1;
            if (sh.count_bad_first) {
                st.k += 1;
                st.total += 1;
            }
        }
    }
    __syncthreads();
}

// The check iteration that ends an epoch of E iterations: its passes, the decisions (every CTA
// takes the same ones from the same sums, on its own copy of the state), and the Halpern step
// or the restart's copies. `stop` says whether an unfinished solve stops here for the batch's
// hand-off: one CTA of a cluster asks it, so that all of them agree.
template <int NC, bool LO, class IX, class Stop>
__device__ __noinline__ void res_check(ResShared<IX> &sh, unsigned long long E, Stop stop) {
    const ResCtx<IX> &R = sh.R;
    const SolverPtrs &S = R.S;
    DevState *st = &sh.st;
    if (threadIdx.x == 0 && (NC == 1 || cluster_rank() == 0)) {
        sh.stop = stop() ? 1.0f : 0.0f;
        publish<NC>(&sh.stop);
    }
    {
        const IterScalars sc = res_scalars(sh, 0.0);
        res_primal<NC, LO, 2>(R, sc);
        res_sync<NC>();
        res_dual<NC, LO, 2>(R, sc);
        res_sync<NC>();
        ResCheckT o{};
        o.s = S;
        o.inv_tau = 1.0 / sc.tau;
        res_pass(R.T, o, R.contribT);
    }
    res_fold<NC, NP_P>(R.T, R.contrib, S.partP, sh.sh);
    res_fold<NC, NP_D>(R.A, R.contribD, S.partD, sh.sh);
    res_sync<NC>();
    res_fold<NC, NP_T>(R.T, R.contribT, S.partT, sh.sh);
    res_sync<NC>();
    double P[NP_P], D[NP_D], T[NP_T];
    res_total<NP_P>(S.partP, R.T.ntiles, P, sh.sh);
    res_total<NP_D>(S.partD, R.A.ntiles, D, sh.sh);
    res_total<NP_T>(S.partT, R.T.ntiles, T, sh.sh);
    if (threadIdx.x == 0) {
        bool bad = false;
        sp_check_record rec;
        check_decide(st, &sh.prm, P, D, T, st->k + E - 1, st->total + E, &bad, &rec);
        if (!bad && sh.trace) {
            if (res_rank<NC>() == 0)
                if ((long long)st->checks - 1 < sh.trace_cap) sh.trace[st->checks - 1] = rec;
            st->trace_len = st->checks;
        }
        if (!st->done && sh.stop != 0.0f) {
            st->done = 1;
            st->status = SP_STATUS_ITERATION_LIMIT;
            st->handoff = 1;
        }
    }
    __syncthreads();
    if (st->done) return;
    // k_finish: the Halpern step, or the restart's copies
    const double w = st->w_last, rho = sh.prm.reflection;
    const bool rs = st->restart_flag != 0, y32 = sh.mixed && !st->fp64;
    for (int k = R.T.p0 + threadIdx.x; k < R.T.p1; k += RES_BT) {
        if (rs) S.x[k] = S.xa[k] = S.xt[k];
        else S.x[k] = halpern(S.x[k], S.xt[k], S.xa[k], w, rho);
    }
    for (int k = R.A.p0 + threadIdx.x; k < R.A.p1; k += RES_BT) {
        double v;
        if (rs) v = S.ya[k] = S.yt[k];
        else v = halpern(S.y[k], S.yt[k], S.ya[k], w, rho);
        S.y[k] = v;
        publish<NC>(S.y + k);
        if (y32) {
            S.y32[k] = (float)v;
            publish<NC>(S.y32 + k);
        }
    }
    res_sync<NC>();
}

// Epochs of check_every iterations (the last one cut at max_iterations), each ended by its
// check, until the state is done, its total has reached sh.until, or (mixed form) the other
// precision is due: LO runs the FP32 phase.
template <int NC, bool LO, bool ES, bool HEADS, int PT, int PA, class Stop>
__device__ __forceinline__ void res_epochs(ResShared<uint16_t> &sh, const ResPlaces<PT, PA> &L, Stop stop) {
    while (!sh.st.done && sh.st.total < sh.until && LO == (sh.mixed && !sh.st.fp64)) {
        unsigned long long E = sh.prm.max_iterations > sh.st.total ? sh.prm.max_iterations - sh.st.total : 1;
        if (sh.prm.check_every && sh.prm.check_every < E) E = sh.prm.check_every;
        const bool first = sh.st.k == 0 && E > 1;
        if (first) {
            res_first<NC, LO>(sh);
            if (sh.st.done) break;
        }
        res_iterate<NC, LO, ES, HEADS>(sh, L, sh.st.k + first, E - 1 - first);
        res_check<NC, LO>(sh, E, stop);
    }
}

// ------------------------------------------------------------------ power iteration

// Power iteration on A'ᵀA' (solver.rs:215-242) as the solver's launches run it (the same
// start, sums and stopping rule); leaves λ, the iteration count and any error in the pi_
// fields and error of *st. part: one double per tile of A'ᵀ.
template <int NC, bool ES, int PT, int PA>
__device__ __noinline__ void res_power(ResShared<uint16_t> &sh, const ResPlaces<PT, PA> &L, unsigned long long max_iters,
                                       double *part) {
    const ResCtx<uint16_t> &R = sh.R;
    const int n = R.T.rows, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    for (int k = threadIdx.x; k < n; k += RES_BT) dsm_at<double>(L.xbar + 8 * k) = 1.0 + 0.01 * (double)(R.T.perm[k] % 7);
    double s[1] = {0.0};
    if (threadIdx.x < NT) {
        int r = threadIdx.x % 7;
        for (int j = threadIdx.x; j < n; j += NT) {
            const double x = 1.0 + 0.01 * (double)r;
            s[0] += x * x;
            r += NT % 7;
            if (r >= 7) r -= 7;
        }
    }
    res_tree<1>(s, sh.sh);
    double scale = 1.0 / sqrt(s[0]), lambda = 0.0;
    int iters = 0, error = ERR_NONE;
    bool done = max_iters == 0;
    const ResPeers<NC> peers;
    const ResEntries<double, ES> ET(R.T, R.T.v, L.valT, L.atT, L.y), EA(R.A, R.A.v, L.valA, L.atA, L.xbar);
    const int vp = L.xbar + 8 * R.T.p0, tp = L.y + 8 * R.A.p0;
    const int t0 = (&dsm_at<int>(L.wtT))[warp], t1 = (&dsm_at<int>(L.wtT))[warp + 1];
    const int a0 = (&dsm_at<int>(L.wtA))[warp], a1 = (&dsm_at<int>(L.wtA))[warp + 1];
    double *const contrib = R.contrib;
    const uint16_t *const perm = R.T.perm + R.T.p0;
    res_sync<NC>();
    while (!done) {
        // tmp = A'(v·scale): the gathered vector is v after the scaling
        for (int k = threadIdx.x; k < n; k += RES_BT) dsm_at<double>(L.xbar + 8 * k) *= scale;
        __syncthreads();
#pragma unroll 1
        for (int ti = a0; ti < a1; ++ti) {
            const ResTask t = (&dsm_at<ResTask>(L.tasksA))[ti];
            const double a = res_sum<double, ES>(EA, t, nullptr);
            if (lane < t.z) {
                const int at = tp + 8 * (t.y + lane);
                dsm_at<double>(at) = a;
                peers.put(at, a);
            }
        }
        res_sync<NC>();
        // v = A'ᵀ tmp, with ‖v‖²
#pragma unroll 1
        for (int ti = t0; ti < t1; ++ti) {
            const ResTask t = (&dsm_at<ResTask>(L.tasksT))[ti];
            const double a = res_sum<double, ES>(ET, t, nullptr);
            if (lane < t.z) {
                const int k = t.y + lane;
                dsm_at<double>(vp + 8 * k) = a;
                peers.put(vp + 8 * k, a);
                contrib[perm[k]] = 0.0 + a * a;
            }
        }
        res_sync<NC>();
        res_fold<NC, 1>(R.T, contrib, part, sh.sh);
        res_sync<NC>();
        res_total<1>(part, R.T.ntiles, s, sh.sh);
        const double norm = sqrt(s[0]);
        if (isnan(norm) || norm <= 0.0 || isinf(norm)) {
            error = ERR_NUMERICAL_POWER;
            break;
        }
        scale = 1.0 / norm;
        done = fabs(norm - lambda) <= 1e-6 * norm;
        lambda = norm;
        iters += 1;
        if ((unsigned long long)iters >= max_iters) done = true;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        DevState &st = sh.st;
        st.pi_scale = scale;
        st.pi_lambda = lambda;
        st.pi_iters = iters;
        st.pi_done = 1;
        st.error = error;
    }
    __syncthreads();
}

// ------------------------------------------------------------------ the solver's kernels

constexpr int RES_PT = 1024, RES_PA = 512;  // columns and rows of a CTA in the solver's kernels
using ResSolverPlaces = ResPlaces<RES_PT, RES_PA>;

// What the kernels of a solver need. `g` holds the solver's vectors in row order.
struct ResArgs {
    SolverPtrs g;
    ResSrc<uint16_t> A, T;
    ResVecs vec;
    double *contrib;                // [8n + 8m + 5n]
    double *ppart;
    sp_check_record *trace;
    long long trace_cap;
    int mixed;
};

__host__ __device__ inline ResSolverPlaces res_solver_places(const ResSrc<uint16_t> &A, const ResSrc<uint16_t> &T, bool lo, bool entries) {
    return ResSolverPlaces(A.rows, T.rows, lo, A.most_tasks, T.most_tasks, A.most_slots, T.most_slots, entries,
                           lo ? 4 : 8);
}

struct ResNoStop {
    __device__ bool operator()() const { return false; }
};

// Epochs of the solver's state in one precision until its total is `until`. In the mixed
// form the FP64 kernel follows the FP32 one, and the one that is not due returns at once.
template <int NC, bool LO, bool ES>
__global__ void __launch_bounds__(RES_BT, 1) k_res_epochs(const __grid_constant__ ResArgs a, unsigned long long until) {
    __shared__ ResShared<uint16_t> s;
    // the same for every CTA: the state is written after the last barrier
    if (a.g.st->done || a.g.st->total >= until || LO != (a.mixed && !a.g.st->fp64)) return;
    const int c = res_rank<NC>();
    if (threadIdx.x == 0) {
        s.st = *a.g.st;
        s.prm = *a.g.prm;
        s.until = until;
        s.trace = a.trace;
        s.trace_cap = a.trace_cap;
        s.mixed = a.mixed;
        s.count_bad_first = 0;
    }
    const ResSolverPlaces L = res_solver_places(a.A, a.T, LO, ES);
    res_open(s, L, a.A, a.T, a.g, a.vec, a.contrib, c);
    const ResCtx<uint16_t> &R = s.R;
    const SolverPtrs &S = R.S, &g = a.g;
    if constexpr (ES) {
        if constexpr (LO) {
            res_load_entries<float>(R.A, R.A.v32, L.valA, L.atA, L.xbar32);
            res_load_entries<float>(R.T, R.T.v32, L.valT, L.atT, L.y32);
        } else {
            res_load_entries<double>(R.A, R.A.v, L.valA, L.atA, L.xbar);
            res_load_entries<double>(R.T, R.T.v, L.valT, L.atT, L.y);
        }
    }
    for (int k = R.T.p0 + threadIdx.x; k < R.T.p1; k += RES_BT) {
        const int j = R.T.perm[k];
        S.x[k] = g.x[j];
        S.xa[k] = g.xa[j];
        S.xt[k] = g.xt[j];
        const_cast<double *>(S.c)[k] = g.c[j];
        const_cast<double *>(S.lv)[k] = g.lv[j];
        const_cast<double *>(S.uv)[k] = g.uv[j];
        const_cast<double *>(S.df)[k] = g.df[j];
    }
    for (int k = R.A.p0 + threadIdx.x; k < R.A.p1; k += RES_BT) {
        const int i = R.A.perm[k];
        S.ya[k] = g.ya[i];
        S.yt[k] = g.yt[i];
        const_cast<double *>(S.lc)[k] = g.lc[i];
        const_cast<double *>(S.uc)[k] = g.uc[i];
        const_cast<double *>(S.pf)[k] = g.pf[i];
    }
    for (int k = threadIdx.x; k < R.A.rows; k += RES_BT) {
        const double v = g.y[R.A.perm[k]];
        S.y[k] = v;
        if (LO) S.y32[k] = (float)v;
    }
    res_sync<NC>();
    res_epochs<NC, LO, ES, true>(s, L, ResNoStop{});
    res_sync<NC>();
    for (int k = R.T.p0 + threadIdx.x; k < R.T.p1; k += RES_BT) {
        const int j = R.T.perm[k];
        g.x[j] = S.x[k];
        g.xa[j] = S.xa[k];
        g.xt[j] = S.xt[k];
    }
    for (int k = R.A.p0 + threadIdx.x; k < R.A.p1; k += RES_BT) {
        const int i = R.A.perm[k];
        const double v = S.y[k];
        g.y[i] = v;
        if (a.mixed) g.y32[i] = (float)v;
        g.ya[i] = S.ya[k];
        g.yt[i] = S.yt[k];
    }
    if (c == 0 && threadIdx.x == 0) *a.g.st = s.st;
}

// The solver's power iteration.
template <int NC, bool ES>
__global__ void __launch_bounds__(RES_BT, 1) k_res_power(const __grid_constant__ ResArgs a, unsigned long long max_iters) {
    __shared__ ResShared<uint16_t> s;
    const int c = res_rank<NC>();
    const ResSolverPlaces L = res_solver_places(a.A, a.T, false, ES);
    res_open(s, L, a.A, a.T, a.g, a.vec, a.contrib, c);
    if constexpr (ES) {
        res_load_entries<double>(s.R.A, s.R.A.v, L.valA, L.atA, L.xbar);
        res_load_entries<double>(s.R.T, s.R.T.v, L.valT, L.atT, L.y);
    }
    res_sync<NC>();
    res_power<NC, ES>(s, L, max_iters, a.ppart);
    if (c == 0 && threadIdx.x == 0) {
        a.g.st->pi_scale = s.st.pi_scale;
        a.g.st->pi_lambda = s.st.pi_lambda;
        a.g.st->pi_iters = s.st.pi_iters;
        a.g.st->pi_done = 1;
        a.g.st->error = s.st.error;
    }
}

// The CTA of task ti: the last whose first task is at most ti.
template <class IX>
__device__ __forceinline__ int res_cta_of(const ResSrc<IX> &M, int ti, int ctas) {
    int c = 0;
    for (int hi = ctas; hi - c > 1;) {
        const int mid = (c + hi) / 2;
        if (M.wt[mid * RES_W] <= ti) c = mid;
        else hi = mid;
    }
    return c;
}

// The slots of one matrix from its CSR arrays, one warp per task: columns renamed to the
// positions of the other matrix's rows; padding holds -0.0 and a position past them (`spread`
// such positions of which 0, 4, 8, ... are used, task by task).
template <class IX>
__global__ void __launch_bounds__(NT) k_res_fill(ResSrc<IX> M, int ctas, int ntasks, int other_rows, int spread,
                                                 const IX *__restrict__ other_inv, const int *__restrict__ ci,
                                                 const double *__restrict__ v) {
    const int lane = threadIdx.x & 31;
    for (int ti = (blockIdx.x * NT + threadIdx.x) >> 5; ti < ntasks; ti += gridDim.x * (NT / 32)) {
        const int c = res_cta_of(M, ti, ctas);
        const ResTask t = M.tasks[ti];
        const IX none = (IX)(other_rows + 4 * ti % spread);
        auto put = [&](int d, int k, bool in) {
            const double x = in ? v[k] : -0.0;
            M.ci[d] = in ? other_inv[ci[k]] : none;
            M.v[d] = x;
            if (M.v32) M.v32[d] = (float)x;
        };
        int base = M.s0[c] + t.x + lane;
        const int p = M.p0[c] + t.y;
        if (t.w >= 0) {
            const int r = lane < t.z ? M.perm[p + lane] : -1;
            const int a = r >= 0 ? M.rp[r] : 0, l = r >= 0 ? M.rp[r + 1] - a : 0;
            for (int j = 0; j < t.w; ++j) put(base + 32 * j, a + j, j < l);
            continue;
        }
        for (int i = 0; i < t.z; ++i) {
            const int r = M.perm[p + i], a = M.rp[r], l = M.rp[r + 1] - a;
            for (int e = lane; e < -32 * t.w; e += 32, base += 32) put(base, a + e, e < l);
        }
    }
}

}  // namespace sp
