// grid.cuh — a mid-sized LP on the whole chip: the FUSED iterations of an epoch in one launch.
//
// Between the LPs that one cluster holds (resident.cuh) and those whose passes fill the chip for
// long, an iteration is two launches of 5-6 µs of which the work is a fraction, and each ends in
// a wave that leaves SMs idle. Here one CTA per SM keeps its rows of both matrices — entries and
// row inputs in shared memory as far as they fit — and runs an epoch's iterations between its
// first and its check; x̄ and y lie in global memory over positions, and the grid's barrier
// (grid_sync, 1.2 µs) separates the passes. The epoch's first iteration and its check stay
// launches on the row-ordered vectors, which the kernel reads at its start and writes at its
// end. Plan and sums are resident.cuh's, so results are the tile engine's, bit for bit.
//
// An iteration is bound by its gathers (two a nonzero, about one a clock and SM) and, from some
// 5M nonzeros on, by the L2 sectors that they move: random LP of 200k nonzeros 10.5 µs by
// launches, 8.5 here; 2M 36.1 and 28.7; 10M power law 128 and 107 (GridPlan, solver.cu: more sizes).
#pragma once

#include "resident.cuh"

namespace sp {

// The grid's barrier: counts arrivals in global memory and waits for them. All CTAs are running
// then (grid_start), and a CTA that runs goes on running. What was written to global memory
// before it is visible after it. The wait is bounded (GRID_WAIT_NS, or another CTA's giving up);
// a CTA that gives up marks itself and all later barriers let it through, so that the kernel
// ends, and the solve is reported as failed. 1.2 µs for 148 CTAs (B200); counting in two levels
// took 1.7.
//
// Whether all CTAs run is found out by the kernel's first wait, grid_start: all have come to its
// gate, or one that has waited GRID_START_NS marks the gate, by compare-and-swap with a count
// short of all, and all CTAs return without effect. That happens where
// another stream's long kernel (a batch) holds SMs; the host then runs these iterations by
// launches, which share the SMs (solver.cu: grid_resume). A cooperative launch would wait for
// that kernel's end: 640 iterations of a 200k-nonzero LP beside a batch of 0.12 s solved over
// and over took 0.9-1.3 s so, and take 0.01-0.24 s (the batch holds all SMs most of the time).
// 0.1 to 1 ms of waiting did alike there, 3 ms and more worse; CTAs of a launch that has the SMs
// start within some 10 µs.
// The count wraps (148 arrivals twice an iteration: after 14.5M iterations of a launch), so
// counts are compared by their difference, which is at most one barrier's arrivals; it starts
// one below the wrap, so that every launch passes it.
constexpr unsigned long long GRID_START_NS = 300000ull, GRID_WAIT_NS = 10000000000ull, GRID_SPIN_NS = 100000ull;
struct GridBar {
    unsigned count, alive;  // alive: 0 once a wait has given up
    unsigned gate;          // CTAs that have started, as `count`; GRID_LEFT: the launch is left
};
constexpr unsigned GRID_COUNT0 = ~0u;  // all words at a launch's start (one fill)
constexpr unsigned GRID_LEFT = 1u << 30;
__host__ __device__ constexpr bool grid_before(unsigned count, unsigned target) { return (int)(count - target) < 0; }
static_assert(grid_before(GRID_COUNT0, GRID_COUNT0 + 148u) && grid_before(147u, 148u) && !grid_before(148u, 148u) &&
                  !grid_before(3u, GRID_COUNT0) && grid_before(0xfffffff0u, 16u),
              "counts on both sides of the wrap");
struct GridState {
    GridBar *bar;
    unsigned passed;  // the count after the barriers so far
    int dead;         // a wait gave up
    int left;         // the launch is left without effect
    int leader;       // ... by this CTA
    unsigned long long wait_ns;
};

__device__ __forceinline__ unsigned ld_acquire(const unsigned *p) {
    unsigned v;
    asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
}

// Whether all CTAs have started, the same answer in all of them: yes once gridDim.x have
// arrived (and `absent` more, a test's that never come), no once one whose wait exceeds `limit`
// has marked the gate before that.
__device__ __forceinline__ bool grid_start(GridState &g, unsigned long long limit, unsigned absent) {  // g: a shared variable
    __syncthreads();
    if (threadIdx.x == 0) {
        const unsigned all = GRID_COUNT0 + gridDim.x + absent;
        asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(&g.bar->gate) : "memory");
        unsigned gate = ld_acquire(&g.bar->gate);
        const unsigned long long t0 = global_ns();
        while (gate != all && !(gate & GRID_LEFT)) {
            const unsigned long long waited = global_ns() - t0;
            if (waited >= limit) {
                if (atomicCAS(&g.bar->gate, gate, gate | GRID_LEFT) == gate) {
                    g.leader = 1;
                    gate |= GRID_LEFT;
                    break;
                }  // else another CTA came or left just now
            } else if (waited > GRID_SPIN_NS) {
                __nanosleep(1000);
            }
            gate = ld_acquire(&g.bar->gate);
        }
        g.left = gate != all;
    }
    __syncthreads();
    return !g.left;
}

__device__ __forceinline__ void grid_sync(GridState &g) {  // g: a shared variable
    __syncthreads();
    if (threadIdx.x == 0 && !g.dead) {
        const unsigned target = g.passed + gridDim.x;
        asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(&g.bar->count) : "memory");
        if (grid_before(ld_acquire(&g.bar->count), target)) {
            const unsigned long long t0 = global_ns();
            while (grid_before(ld_acquire(&g.bar->count), target)) {
                const unsigned long long waited = global_ns() - t0;
                if (!ld_acquire(&g.bar->alive) || waited >= g.wait_ns) {
                    atomicExch(&g.bar->alive, 0u);
                    g.dead = 1;
                    break;
                }
                if (waited > GRID_SPIN_NS) __nanosleep(1000);
            }
        }
        g.passed = target;
    }
    __syncthreads();
}

// Places in dynamic shared memory: the row inputs of at most PT columns and PA rows (VS), the
// tasks, and the entries (ES), values and 32-bit positions.
template <bool VS, bool ES, int PT, int PA>
struct GridPlaces {
    static constexpr int X = 0, XA = 8 * PT, C = 16 * PT, LV = 24 * PT, UV = 32 * PT;
    static constexpr int YA = 40 * PT, LC = YA + 8 * PA, UC = YA + 16 * PA, END = VS ? YA + 24 * PA : 0;
    int tasksA, tasksT, wtA, wtT, valA, valT, idxA, idxT, total;
    __host__ __device__ GridPlaces(int ta, int tt, int sa, int st, int vb) {
        int at = END;
        auto take = [&](int bytes) {
            const int a = at;
            at += (bytes + 15) & ~15;
            return a;
        };
        tasksA = take((int)sizeof(ResTask) * ta);
        tasksT = take((int)sizeof(ResTask) * tt);
        wtA = take(4 * (RES_W + 1));
        wtT = take(4 * (RES_W + 1));
        valA = ES ? take(vb * sa) : 0;
        valT = ES ? take(vb * st) : 0;
        idxA = ES ? take(4 * sa) : 0;
        idxT = ES ? take(4 * st) : 0;
        total = at;
    }
};

// 1.0s behind each gathered vector: all padding on one of them would have every SM ask the
// same sector of L2.
constexpr int GRID_ONES = 1024;

struct GridArgs {
    SolverPtrs g;                   // the solver's vectors in row order
    ResSrc<int> A, T;
    double *x, *xa, *c, *lv, *uv;   // over positions: the columns' inputs
    double *ya, *lc, *uc;           // ... the rows'
    double *y, *xbar;               // ... the gathered vectors; GRID_ONES 1.0 behind each
    float *y32, *xbar32;
    double *contrib, *ppart;        // the power iteration's
    GridBar *bar;                   // all ones before each launch
    unsigned long long start_ns, wait_ns;  // limits of the first wait and of the others
    unsigned absent;                       // grid_start's
    int mixed;
};

template <bool VS, bool ES, int PT, int PA>
__host__ __device__ inline GridPlaces<VS, ES, PT, PA> grid_places(const GridArgs &a, bool lo) {
    return GridPlaces<VS, ES, PT, PA>(a.A.most_tasks, a.T.most_tasks, a.A.most_slots, a.T.most_slots, lo ? 4 : 8);
}

struct GridShared {
    ResSide<int> A, T;
    GridState grid;
    int due;
    double wtab[RES_WTAB];
    double sh[RES_GROUPS * (NT / 32) + 1];
};

// This CTA's part of the plan into shared memory. Ends with a barrier.
template <bool VS, bool ES, int PT, int PA>
__device__ inline void grid_open(GridShared &sh, const GridPlaces<VS, ES, PT, PA> &L, const GridArgs &a) {
    const int c = (int)blockIdx.x;
    if (threadIdx.x == 0) {
        sh.grid = GridState{a.bar, GRID_COUNT0, 0, 0, 0, a.wait_ns};
        sh.A = res_side(a.A, c, L.tasksA, L.wtA);
        sh.T = res_side(a.T, c, L.tasksT, L.wtT);
    }
    for (const ResSrc<int> *M : {&a.A, &a.T}) {
        const int *wt = M->wt + c * RES_W;
        const int tasks = M == &a.A ? L.tasksA : L.tasksT, to = M == &a.A ? L.wtA : L.wtT, n = wt[RES_W] - wt[0];
        for (int i = threadIdx.x; i < n; i += RES_BT) (&dsm_at<ResTask>(tasks))[i] = M->tasks[wt[0] + i];
        if (threadIdx.x <= RES_W) (&dsm_at<int>(to))[threadIdx.x] = wt[threadIdx.x] - wt[0];
    }
    __syncthreads();
}

template <class VT>
__device__ inline void grid_load_entries(const ResSide<int> &M, const VT *v, int val, int idx) {
    for (int i = threadIdx.x; i < M.slots; i += RES_BT) {
        (&dsm_at<VT>(val))[i] = v[i];
        (&dsm_at<int>(idx))[i] = M.ci[i];
    }
}

// Entries of one matrix for this lane, and the vector that they gather.
template <class VT, bool ES>
struct GridEntries {
    int val, idx;
    const int *ci;
    const VT *v;
    const VT *g;
    __device__ __forceinline__ GridEntries(const ResSide<int> &M, const VT *vals, int val_, int idx_, const VT *g_) : g(g_) {
        const int lane = threadIdx.x & 31;
        if constexpr (ES) {
            val = val_ + (int)sizeof(VT) * lane;
            idx = idx_ + 4 * lane;
        } else {
            ci = M.ci + lane;
            v = vals + lane;
        }
    }
    __device__ __forceinline__ VT value(int o) const {
        if constexpr (ES) return dsm_at<const VT>(val + (int)sizeof(VT) * o);
        else return ld_stream(v + o);
    }
    __device__ __forceinline__ int pos(int o) const {
        if constexpr (ES) return dsm_at<const int>(idx + 4 * o);
        else return ld_stream(ci + o);
    }
};

// Entries of a step. µs an iteration at 2 | 4 | 6 | 8 of them: random LP of 200k nonzeros 9.4 | 8.3 |
// 8.1 | 8.4, 2M 34.2 | 29.2 | 46.0 | 53.5 (6 and 8 spill where entries are in global memory),
// 12M 155 | 139 | 226 | 297, 10M power law 129 | 109 | 197 | 247; mixed 9.6 | 8.5 | 8.3 | 8.5,
// 33.3 | 28.2 | 28.0 | 27.3, 150 | 132 | 129 | 138, 125 | 102 | 102 | 105.
constexpr int GRID_B = 4;

// One step of a warp: GRID_B entries of each lane's row. A row's last step is filled up with
// padding; a row without entries takes a step too.
struct GridStep {
    int o, cnt;      // first slot (for lane 0) and how many slots
    int y, z;        // the task's first position and rows
    int i;           // of a group of warp rows: the row; -1: a slice
    bool row, task;  // the row's, the task's last step
};
// The steps of tasks t0 … t1 - 1 in order.
struct GridCursor {
    int tasks, ti, t1;  // the tasks' place, the next task
    ResTask t;
    int i, j;           // row of a group of warp rows, entry
    bool ok;            // there is a step
    __device__ __forceinline__ GridCursor(int tasks_, int t0, int t1_) : tasks(tasks_), ti(t0), t1(t1_) { open(); }
    __device__ __forceinline__ void open() {
        ok = ti < t1;
        i = j = 0;
        if (ok) t = (&dsm_at<ResTask>(tasks))[ti];
    }
    __device__ __forceinline__ GridStep step() {  // and on to the next one
        const int w = abs(t.w);
        GridStep q;
        q.o = t.x + 32 * (i * w + j);
        q.cnt = w - j;
        q.y = t.y;
        q.z = t.z;
        q.i = t.w < 0 ? i : -1;
        q.row = j + GRID_B >= w;
        q.task = q.row && (t.w >= 0 || i + 1 >= t.z);
        j += GRID_B;
        if (q.row) {
            j = 0;
            ++i;
        }
        if (q.task) {
            ++ti;
            open();
        }
        return q;
    }
};

// The sums of a warp's rows: row(y, z, sum) is called for each task (first position, rows)
// with the sum of the lane's row `lane`. A pass is bound by its gathers — an SM looks up one a
// clock — as long as enough of them are under way: a step's gathers are issued before the last
// step's are used. Entries in global memory are asked for a step earlier still (positions), or
// with the gathers (values).
template <class VT, bool ES, class Mul, class Row>
__device__ __forceinline__ void grid_rows(const GridEntries<VT, ES> &E, int tasks, int t0, int t1, const Mul &mul,
                                          const Row &row) {
    const int lane = threadIdx.x & 31;
    GridCursor cur(tasks, t0, t1);
    if (!cur.ok) return;
    int c[GRID_B];                 // positions of the step whose gathers are next
    VT x0[GRID_B], g0[GRID_B];     // values (global memory) and gathers under way
    auto positions = [&](const GridStep &q) {
#pragma unroll
        for (int u = 0; u < GRID_B; ++u)
            if (u < q.cnt) c[u] = E.pos(q.o + 32 * u);
    };
    auto values = [&](const GridStep &q, VT (&x)[GRID_B]) {
#pragma unroll
        for (int u = 0; u < GRID_B; ++u) x[u] = u < q.cnt ? E.value(q.o + 32 * u) : VT(-0.0);
    };
    auto gather = [&](const GridStep &q, VT (&g)[GRID_B]) {
#pragma unroll
        for (int u = 0; u < GRID_B; ++u) g[u] = u < q.cnt ? E.g[c[u]] : VT(1.0);
    };
    GridStep here = cur.step(), then{};
    positions(here);
    gather(here, g0);
    if (!ES) values(here, x0);
    bool more = cur.ok;
    if (more) {
        then = cur.step();
        if (!ES) positions(then);
    }
    VT s = VT(-0.0);
    double r = 0.0;
#pragma unroll 1
    for (;;) {
        VT x1[GRID_B], g1[GRID_B];
        GridStep after{};
        const bool last = !cur.ok;
        if (more) {
            if (ES) positions(then);
            gather(then, g1);
            if (!ES) values(then, x1);
            if (!last) {
                after = cur.step();
                if (!ES) positions(after);
            }
        }
        if (ES) values(here, x0);
#pragma unroll
        for (int u = 0; u < GRID_B; ++u) s += mul(x0[u], g0[u]);
        if (here.row) {
            if (here.i < 0) {
                r = double(s);
            } else {
                const VT tot = __shfl_sync(0xffffffffu, warp_sum_down(s), 0);
                if (lane == here.i) r = double(tot);
            }
            s = VT(-0.0);
            if (here.task) row(here.y, here.z, r);
        }
        if (!more) return;
        here = then;
        then = after;
        more = !last;
#pragma unroll
        for (int u = 0; u < GRID_B; ++u) {
            g0[u] = g1[u];
            if (!ES) x0[u] = x1[u];
        }
    }
}

// The iterations 1 … E - 2 of an epoch of E (its first and its check are launches). The
// vectors' initial state is read from the row-ordered vectors and left there again; x, c, lv, uv
// and the like lie over positions: c, lv, uv, lc, uc since the solver was made.
template <bool LO, bool VS, bool ES, int PT, int PA>
__global__ void __launch_bounds__(RES_BT, 1) k_grid_mid(const __grid_constant__ GridArgs a, long long E) {
    using VT = typename std::conditional<LO, float, double>::type;
    using P = GridPlaces<VS, ES, PT, PA>;
    __shared__ GridShared sh;
    // The same for every thread of a CTA. A CTA that starts after the launch was left may see
    // the state that says so.
    if (threadIdx.x == 0) {
        const DevState *st = a.g.st;
        sh.due = !st->done && LO == (a.mixed && !st->fp64);
    }
    const P L = grid_places<VS, ES, PT, PA>(a, LO);
    grid_open(sh, L, a);
    if (!sh.due) return;
    const VT *vT, *vA;
    VT *gy, *gx;
    if constexpr (LO) {
        vT = sh.T.v32;
        vA = sh.A.v32;
        gy = a.y32;
        gx = a.xbar32;
    } else {
        vT = sh.T.v;
        vA = sh.A.v;
        gy = a.y;
        gx = a.xbar;
    }
    const int pT = sh.T.p0, pA = sh.A.p0, nT = sh.T.p1 - pT, nA = sh.A.p1 - pA;
    if constexpr (ES) {
        grid_load_entries<VT>(sh.A, vA, L.valA, L.idxA);
        grid_load_entries<VT>(sh.T, vT, L.valT, L.idxT);
    }
    for (int k = threadIdx.x; k < nT; k += RES_BT) {
        const int j = sh.T.perm[pT + k];
        if (VS) {
            dsm_at<double>(P::X + 8 * k) = a.g.x[j];
            dsm_at<double>(P::XA + 8 * k) = a.g.xa[j];
            dsm_at<double>(P::C + 8 * k) = a.c[pT + k];
            dsm_at<double>(P::LV + 8 * k) = a.lv[pT + k];
            dsm_at<double>(P::UV + 8 * k) = a.uv[pT + k];
        } else {
            a.x[pT + k] = a.g.x[j];
            a.xa[pT + k] = a.g.xa[j];
        }
    }
    for (int k = threadIdx.x; k < nA; k += RES_BT) {
        const int i = sh.A.perm[pA + k];
        const double v = a.g.y[i];
        a.y[pA + k] = v;
        if (LO) gy[pA + k] = (VT)v;
        if (VS) {
            dsm_at<double>(P::YA + 8 * k) = a.g.ya[i];
            dsm_at<double>(P::LC + 8 * k) = a.lc[pA + k];
            dsm_at<double>(P::UC + 8 * k) = a.uc[pA + k];
        } else {
            a.ya[pA + k] = a.g.ya[i];
        }
    }
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const double rho = a.g.prm->reflection, tau = a.g.prm->eta / a.g.st->omega, sigma = a.g.prm->eta * a.g.st->omega;
    const SigmaDivisor by_sigma(sigma);
    const GridEntries<VT, ES> ET(sh.T, vT, L.valT, L.idxT, gy), EA(sh.A, vA, L.valA, L.idxA, gx);
    auto mul = [](VT v, VT g) { return v * g; };
    const int t0 = (&dsm_at<int>(L.wtT))[warp], t1 = (&dsm_at<int>(L.wtT))[warp + 1];
    const int a0 = (&dsm_at<int>(L.wtA))[warp], a1 = (&dsm_at<int>(L.wtA))[warp + 1];
    double w = 0.0;
    // A task's rows: PrimalPass and DualPass with MODE 0 (solver_kernels.cuh) on positions.
    auto primal = [&](int ty, int tz, double aty) {
        if (lane >= tz) return;
        const int k8 = 8 * (ty + lane), k = pT + ty + lane;
        double xj, cj, lo, hi, xaj;
        if (VS) {
            xj = dsm_at<double>(P::X + k8);
            cj = dsm_at<double>(P::C + k8);
            lo = dsm_at<double>(P::LV + k8);
            hi = dsm_at<double>(P::UV + k8);
            xaj = dsm_at<double>(P::XA + k8);
        } else {
            xj = a.x[k];
            cj = a.c[k];
            lo = a.lv[k];
            hi = a.uv[k];
            xaj = a.xa[k];
        }
        const double xt = clampd(xj - tau * (cj - aty), lo, hi);
        gx[k] = VT(2.0 * xt - xj);
        const double xn = halpern(xj, xt, xaj, w, rho);
        if (VS) dsm_at<double>(P::X + k8) = xn;
        else a.x[k] = xn;
    };
    auto dual = [&](int ty, int tz, double s) {
        if (lane >= tz) return;
        const int k8 = 8 * (ty + lane), k = pA + ty + lane;
        double lo, hi, yai;
        const double yi = a.y[k];
        if (VS) {
            lo = dsm_at<double>(P::LC + k8);
            hi = dsm_at<double>(P::UC + k8);
            yai = dsm_at<double>(P::YA + k8);
        } else {
            lo = a.lc[k];
            hi = a.uc[k];
            yai = a.ya[k];
        }
        const double v = s - by_sigma(yi);
        const double yt = yi - sigma * (s - clampd(v, lo, hi));
        const double yn = halpern(yi, yt, yai, w, rho);
        a.y[k] = yn;
        if constexpr (LO) gy[k] = (float)yn;
    };
    if (!grid_start(sh.grid, a.start_ns, a.absent)) {  // so far nothing but this engine's own vectors was written
        if (threadIdx.x == 0 && sh.grid.leader) {
            a.g.st->error = ERR_GRID_BUSY;
            a.g.st->done = 1;
        }
        return;
    }
    const unsigned long long k0 = a.g.st->k;
#pragma unroll 1
    for (unsigned long long i = 1; i + 1 < (unsigned long long)E && !sh.grid.dead; ++i) {
        if (i == 1 || i % RES_WTAB == 0) {  // every reader of the last weights is past a barrier
            if (threadIdx.x < RES_WTAB) {
                const unsigned long long k = k0 + i / RES_WTAB * RES_WTAB + threadIdx.x;
                sh.wtab[threadIdx.x] = (double)(k + 1) / (double)(k + 2);
            }
            __syncthreads();
        }
        w = sh.wtab[i % RES_WTAB];
        grid_rows(ET, L.tasksT, t0, t1, mul, primal);
        grid_sync(sh.grid);
        grid_rows(EA, L.tasksA, a0, a1, mul, dual);
        grid_sync(sh.grid);
    }
    for (int k = threadIdx.x; k < nT; k += RES_BT) {
        const int j = sh.T.perm[pT + k];
        a.g.x[j] = VS ? dsm_at<double>(P::X + 8 * k) : a.x[pT + k];
    }
    for (int k = threadIdx.x; k < nA; k += RES_BT) {
        const int i = sh.A.perm[pA + k];
        const double v = a.y[pA + k];
        a.g.y[i] = v;
        if (LO) a.g.y32[i] = (float)v;
    }
    if (threadIdx.x == 0 && sh.grid.dead) {
        a.g.st->error = ERR_GRID_STALL;
        a.g.st->done = 1;
    }
}

// The 1.0s behind the gathered vectors.
static __global__ void k_grid_ones(GridArgs a) {
    for (int k = (int)(blockIdx.x * blockDim.x + threadIdx.x); k < GRID_ONES; k += (int)(gridDim.x * blockDim.x)) {
        a.y[a.A.rows + k] = 1.0;
        a.xbar[a.T.rows + k] = 1.0;
        if (a.mixed) {
            a.y32[a.A.rows + k] = 1.0f;
            a.xbar32[a.T.rows + k] = 1.0f;
        }
    }
}

// The inputs that no iteration changes, over positions.
static __global__ void k_grid_inputs(GridArgs a) {
    const int step = (int)(gridDim.x * blockDim.x), first = (int)(blockIdx.x * blockDim.x + threadIdx.x);
    for (int k = first; k < a.T.rows; k += step) {
        const int j = a.T.perm[k];
        a.c[k] = a.g.c[j];
        a.lv[k] = a.g.lv[j];
        a.uv[k] = a.g.uv[j];
    }
    for (int k = first; k < a.A.rows; k += step) {
        const int i = a.A.perm[k];
        a.lc[k] = a.g.lc[i];
        a.uc[k] = a.g.uc[i];
    }
}

// The solver's power iteration (res_power's: the same start, sums and stopping rule).
template <bool ES>
__global__ void __launch_bounds__(RES_BT, 1) k_grid_power(const __grid_constant__ GridArgs a, long long max_iters) {
    __shared__ GridShared sh;
    const auto L = grid_places<false, ES, 0, 0>(a, false);
    grid_open(sh, L, a);
    if constexpr (ES) {
        grid_load_entries<double>(sh.A, sh.A.v, L.valA, L.idxA);
        grid_load_entries<double>(sh.T, sh.T.v, L.valT, L.idxT);
    }
    const int n = sh.T.rows, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    double *const v = a.xbar, *const tmp = a.y, *const contrib = a.contrib;
    const GridEntries<double, ES> ET(sh.T, sh.T.v, L.valT, L.idxT, tmp), EA(sh.A, sh.A.v, L.valA, L.idxA, v);
    const int t0 = (&dsm_at<int>(L.wtT))[warp], t1 = (&dsm_at<int>(L.wtT))[warp + 1];
    const int a0 = (&dsm_at<int>(L.wtA))[warp], a1 = (&dsm_at<int>(L.wtA))[warp + 1];
    const int pT = sh.T.p0, pA = sh.A.p0;
    const int *const perm = sh.T.perm;
    for (int k = pT + threadIdx.x; k < sh.T.p1; k += RES_BT) v[k] = 1.0 + 0.01 * (double)(perm[k] % 7);
    double s[1] = {0.0};
    if (threadIdx.x < NT) {  // k_power_init
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
    bool done = false;
    if (!grid_start(sh.grid, a.start_ns, a.absent)) {
        if (threadIdx.x == 0 && sh.grid.leader) {
            a.g.st->error = ERR_GRID_BUSY;
            a.g.st->pi_done = 1;
        }
        return;
    }
    while (!done && !sh.grid.dead) {
        grid_rows(EA, L.tasksA, a0, a1, [&](double x, double g) { return x * (g * scale); },
                  [&](int ty, int tz, double q) {
                      if (lane < tz) tmp[pA + ty + lane] = q;
                  });
        grid_sync(sh.grid);
        grid_rows(ET, L.tasksT, t0, t1, [](double x, double g) { return x * g; },
                  [&](int ty, int tz, double q) {
                      if (lane >= tz) return;
                      const int k = pT + ty + lane;
                      v[k] = q;
                      contrib[perm[k]] = 0.0 + q * q;
                  });
        grid_sync(sh.grid);
        res_fold<0, 1>(sh.T, contrib, a.ppart, sh.sh);
        grid_sync(sh.grid);
        res_total<1>(a.ppart, sh.T.ntiles, s, sh.sh);
        const double norm = sqrt(s[0]);
        if (isnan(norm) || norm <= 0.0 || isinf(norm)) {
            error = ERR_NUMERICAL_POWER;
            break;
        }
        scale = 1.0 / norm;
        done = fabs(norm - lambda) <= 1e-6 * norm;
        lambda = norm;
        iters += 1;
        if (iters >= max_iters) done = true;
    }
    if (threadIdx.x == 0 && (sh.grid.dead || blockIdx.x == 0)) {
        a.g.st->pi_scale = scale;
        a.g.st->pi_lambda = lambda;
        a.g.st->pi_iters = iters;
        a.g.st->pi_done = 1;
        if (sh.grid.dead) error = ERR_GRID_STALL;
        if (error != ERR_NONE) a.g.st->error = error;
    }
}

}  // namespace sp
