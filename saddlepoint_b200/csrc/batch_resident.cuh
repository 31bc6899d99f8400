// batch_resident.cuh — the batched form's instances on chip: one CTA, or a cluster of 2 or 4,
// takes the next instance of its size class and runs its whole solve in shared memory — the
// scaling passes (scaling.rs:53-103), the power iteration and the PDHG epochs of resident.cuh —
// so an instance's result is sp_solve's, bit for bit, alone and in any mix.
//
// Against the variants of batch_kernels.cuh (one CTA of 256 threads walking tiles or lane
// groups through L2, each a chain of round trips): the vectors and, where they fit, the
// entries are read from shared memory, by 16 warps that own their rows. Entries in L2 (most
// instances of some 900 rows and more) are what the warps wait for most: their latency, with four warps
// a scheduler, not the rate of L2 (11 % of it) or of the shared memory (30 %).
#pragma once

#include "batch_kernels.cuh"
#include "resident.cuh"

namespace sp {

constexpr int RES_BATCH_MAX = 4;  // CTAs of an instance at most
constexpr int RES_CLASSES = 4;    // the classes of instances (res_class, batch.cu)
// Columns and rows of a CTA: classes of small and of large parts.
constexpr int RES_SMALL_PT = 1024, RES_SMALL_PA = 512, RES_LARGE_PT = 2048, RES_LARGE_PA = 1024;

// The plan of one instance: offsets into the plan arenas (BatchRes) and sizes.
struct ResBatchInst {
    int id, es;                     // the instance; whether its entries fit in shared memory
    long long tasksA, tasksT;
    int wtA, wtT;
    int heavyA, heavyT;
    int mostA[3], mostT[3];         // rows, slots, tasks of one CTA
    int pA[RES_BATCH_MAX + 1], sA[RES_BATCH_MAX + 1], pT[RES_BATCH_MAX + 1], sT[RES_BATCH_MAX + 1];
};

// Where an instance runs on chip, for sp_batch_engine (0 CTAs: not there).
struct BatchChip {
    int ctas = 0, cols = 0, entries = 0;
};

// The instances of one class (cluster size) and what their kernel needs.
struct ResBatchClass {
    const ResBatchInst *inst;       // largest first
    int count;
    int *counter;
    unsigned char *scratch;         // per cluster
    size_t scratch_bytes;
};
struct BatchRes {
    const uint16_t *permA, *permT, *invA, *invT;  // at the instance's m- and n-offsets
    const ResTask *tasks;
    const int *wt;
};

// Offsets into a cluster's scratch.
struct ResScratch {
    size_t vA, vT, v32A, v32T, ciA, ciT, vecs, contrib, pk, pky, part, total;
    __host__ __device__ ResScratch(long long slotsA, long long slotsT, int m, int n, int nta, int ntt, bool mixed) {
        size_t at = 0;
        auto take = [&](size_t b) {
            const size_t a = at;
            at += (b + 255) & ~size_t(255);
            return a;
        };
        vA = take(8 * (size_t)slotsA);
        vT = take(8 * (size_t)slotsT);
        v32A = take(mixed ? 4 * (size_t)slotsA : 0);
        v32T = take(mixed ? 4 * (size_t)slotsT : 0);
        ciA = take(2 * (size_t)slotsA);
        ciT = take(2 * (size_t)slotsT);
        vecs = take(8 * (3 * (size_t)n + 2 * (size_t)m));
        contrib = take(8 * (13 * (size_t)n + 8 * (size_t)m));
        pk = take(sizeof(CheckQuad) * ((size_t)n + 1));
        pky = take(sizeof(double2) * ((size_t)m + 1));
        part = take(8 * ((size_t)nta * (NP_D + NP_D0) + (size_t)ntt * (NP_P + NP_T + NP_P0 + 1)));
        total = at;
    }
};

// Calls f(position, first slot, slot step, slots) for each row of this warp, lane by lane:
// the slots of a slice's row are 32 apart, those of a warp row consecutive; both end in padding.
template <class F>
__device__ __forceinline__ void res_rows(const ResSide<uint16_t> &M, const F &f) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int t1 = (&dsm_at<int>(M.wt))[warp + 1];
#pragma unroll 1
    for (int ti = (&dsm_at<int>(M.wt))[warp]; ti < t1; ++ti) {
        const ResTask t = (&dsm_at<ResTask>(M.tasks))[ti];
        if (lane >= t.z) continue;
        if (t.w >= 0) f(M.p0 + t.y + lane, t.x + lane, 32, t.w);
        else f(M.p0 + t.y + lane, t.x - 32 * t.w * lane, 1, -32 * t.w);
    }
}

// This CTA's slots from the instance's CSR arrays (k_res_fill's layout).
__device__ __forceinline__ void res_fill(const ResSide<uint16_t> &M, uint16_t *ci_out, double *v_out, const int *rp, const int *ci,
                                         const double *v, const uint16_t *other_inv, int other_rows) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int t1 = (&dsm_at<int>(M.wt))[warp + 1];
    auto put = [&](int d, int k, bool in) {
        ci_out[d] = in ? other_inv[ci[k]] : (uint16_t)other_rows;
        v_out[d] = in ? v[k] : -0.0;
    };
#pragma unroll 1
    for (int ti = (&dsm_at<int>(M.wt))[warp]; ti < t1; ++ti) {
        const ResTask t = (&dsm_at<ResTask>(M.tasks))[ti];
        int base = t.x + lane;
        const int p = M.p0 + t.y;
        if (t.w >= 0) {
            const int r = lane < t.z ? M.perm[p + lane] : -1;
            const int a = r >= 0 ? rp[r] : 0, l = r >= 0 ? rp[r + 1] - a : 0;
#pragma unroll 4
            for (int j = 0; j < t.w; ++j) put(base + 32 * j, a + j, j < l);
        } else {
            for (int i = 0; i < t.z; ++i) {
                const int r = M.perm[p + i], a = rp[r], l = rp[r + 1] - a;
                for (int e = lane; e < -32 * t.w; e += 32, base += 32) put(base, a + e, e < l);
            }
        }
    }
}

__device__ __forceinline__ double factor_geo(double lo, double hi) {  // scaling.rs:62-63, :159-178
    const double v = (hi == 0.0 ? 0.0 : lo) * hi;
    return (v > 0.0 && isfinite(v)) ? 1.0 / sqrt(v) : 1.0;
}
__device__ __forceinline__ double factor_of(double v) { return (v > 0.0 && isfinite(v)) ? 1.0 / sqrt(v) : 1.0; }

// The scaling passes on this CTA's slots: vA, vT its values (in any memory), cA, cT their
// columns. Row factors go through y and column factors through x̄ (whole in every CTA, the
// padding's 1.0 behind them); new factors wait in xn and yn (this CTA's positions) while the
// old ones are read. rs, cs: the products of all factors, over positions.
template <int NC>
__device__ __noinline__ void res_scale(ResShared<uint16_t> &sh, const BatchArgs &A, double *vA, double *vT, double *rs, double *cs) {
    const ResCtx<uint16_t> &R = sh.R;
    const ResSide<uint16_t> &MA = R.A, &MT = R.T;
    double *fr = R.S.y, *fc = R.S.xbar, *yn = R.S.ya, *xn = R.S.xa;
    const int noneA = MT.rows, noneT = MA.rows;  // the padding's columns
    auto span = [](const uint16_t *ci, const double *v, int none, int o, int step, int n, double &lo, double &hi) {
#pragma unroll 4
        for (int j = 0; j < n; ++j, o += step)
            if (ci[o] != none) {
                const double a = fabs(v[o]);
                lo = fmin(lo, a);
                hi = fmax(hi, a);
            }
    };
    res_rows(MA, [&](int k, int, int, int) { rs[k] = 1.0; });
    res_rows(MT, [&](int k, int, int, int) { cs[k] = 1.0; });
    if (A.geo_passes > 0) {
        res_rows(MA, [&](int k, int o, int step, int n) {
            double lo = INFINITY, hi = 0.0;
            span(MA.ci, vA, noneA, o, step, n, lo, hi);
            fr[k] = factor_geo(lo, hi);
            publish<NC>(fr + k);
        });
    }
    for (unsigned long long ps = 0; ps < A.geo_passes; ++ps) {
        res_sync<NC>();
        // columns: the row factors first, then the column factor of what they leave
        res_rows(MT, [&](int k, int o, int step, int n) {
            double lo = INFINITY, hi = 0.0;
#pragma unroll 4
            for (int j = 0, d = o; j < n; ++j, d += step)
                if (MT.ci[d] != noneT) {
                    const double a = fabs(vT[d] * fr[MT.ci[d]]);
                    lo = fmin(lo, a);
                    hi = fmax(hi, a);
                }
            const double f = factor_geo(lo, hi);
#pragma unroll 4
            for (int j = 0, d = o; j < n; ++j, d += step)
                if (MT.ci[d] != noneT) vT[d] = (vT[d] * fr[MT.ci[d]]) * f;
            fc[k] = f;
            publish<NC>(fc + k);
            cs[k] *= f;
        });
        res_sync<NC>();
        const bool more = ps + 1 < A.geo_passes;
        res_rows(MA, [&](int k, int o, int step, int n) {
            const double f = fr[k];
            double lo = INFINITY, hi = 0.0;
#pragma unroll 4
            for (int j = 0; j < n; ++j, o += step)
                if (MA.ci[o] != noneA) {
                    const double a = (vA[o] * f) * fc[MA.ci[o]];
                    vA[o] = a;
                    lo = fmin(lo, fabs(a));
                    hi = fmax(hi, fabs(a));
                }
            rs[k] *= f;
            if (more) {
                fr[k] = factor_geo(lo, hi);
                publish<NC>(fr + k);
            }
        });
    }
    const unsigned long long steps = A.ruiz_iterations + (A.pc_enabled ? 1 : 0);
    for (unsigned long long it = 0; it < steps; ++it) {
        const bool pc = it == A.ruiz_iterations;  // Pock-Chambolle: sums in index order
        auto factor = [&](const ResSide<uint16_t> &M, const double *v, int none, int o, int step, int n, double alpha) {
            if (!pc) {
                double lo = INFINITY, hi = 0.0;
                span(M.ci, v, none, o, step, n, lo, hi);
                return factor_of(hi);
            }
            double s = 0.0;
            for (int j = 0; j < n; ++j, o += step)
                if (M.ci[o] != none) {
                    const double a = fabs(v[o]);
                    s = s + (alpha == 1.0 ? a : pow(a, alpha));
                }
            return factor_of(s);
        };
        res_sync<NC>();
        res_rows(MA, [&](int k, int o, int step, int n) { yn[k] = factor(MA, vA, noneA, o, step, n, A.pc_alpha); });
        res_rows(MT, [&](int k, int o, int step, int n) { xn[k] = factor(MT, vT, noneT, o, step, n, 2.0 - A.pc_alpha); });
        res_rows(MA, [&](int k, int, int, int) {
            fr[k] = yn[k];
            publish<NC>(fr + k);
        });
        res_rows(MT, [&](int k, int, int, int) {
            fc[k] = xn[k];
            publish<NC>(fc + k);
        });
        res_sync<NC>();
        res_rows(MA, [&](int k, int o, int step, int n) {
            const double f = fr[k];
#pragma unroll 4
            for (int j = 0; j < n; ++j, o += step)
                if (MA.ci[o] != noneA) vA[o] *= f * fc[MA.ci[o]];
            rs[k] *= f;
        });
        res_rows(MT, [&](int k, int o, int step, int n) {
            const double f = fc[k];
#pragma unroll 4
            for (int j = 0; j < n; ++j, o += step)
                if (MT.ci[o] != noneT) vT[o] *= f * fr[MT.ci[o]];
            cs[k] *= f;
        });
    }
    res_sync<NC>();
}

// The four norms (scaling.rs:186-201, solver.rs:317-318), each a sum in index order from -0.0:
// the CTA forms a chunk's terms, then one thread of each of four warps adds one norm's. out:
// bound norm and cost norm of the scaled problem, then of the original.
__device__ __noinline__ void res_norms(const double *olc, const double *ouc, const double *oc, const double *rs,
                                       const double *cs, int m, int n, double (&out)[4]) {
    constexpr int CH = RES_SMALL_PT;  // terms of a chunk: X, XA, C and LV hold one norm's each
    double *term = &dsm_at<double>(0);
    double s = -0.0;
    for (int base = 0; base < max(m, n); base += CH) {
        __syncthreads();
        for (int u = threadIdx.x; u < CH; u += RES_BT) {
            const int i = base + u;
            auto bound = [&](double l, double h) {
                l = isfinite(l) ? l : 0.0;
                h = isfinite(h) ? h : 0.0;
                return (l == h) ? l * l : l * l + h * h;
            };
            if (i < m) {
                const double l = olc[i], h = ouc[i], r = __ldcg(rs + i);
                term[u] = bound(l * r, h * r);
                term[2 * CH + u] = bound(l, h);
            }
            if (i < n) {
                const double c = oc[i], v = c * __ldcg(cs + i);
                term[CH + u] = v * v;
                term[3 * CH + u] = c * c;
            }
        }
        __syncthreads();
        if ((threadIdx.x & 31) == 0 && threadIdx.x < 128) {
            const int q = threadIdx.x >> 5, cnt = min(CH, ((q & 1) ? n : m) - base);
            const double *t = term + q * CH;
            int i = 0;
            for (; i + 8 <= cnt; i += 8) {
                double v[8];
#pragma unroll
                for (int u = 0; u < 8; ++u) v[u] = t[i + u];
#pragma unroll
                for (int u = 0; u < 8; ++u) s += v[u];
            }
            for (; i < cnt; ++i) s += t[i];
        }
    }
    __syncthreads();
    if ((threadIdx.x & 31) == 0 && threadIdx.x < 128) term[threadIdx.x >> 5] = sqrt(s);
    __syncthreads();
#pragma unroll
    for (int q = 0; q < 4; ++q) out[q] = term[q];
    __syncthreads();
}

struct ResTailStop {
    const BatchArgs *A;
    __device__ bool operator()() const { return tail_due(*A); }
};

struct ResBatchShared {
    ResShared<uint16_t> s;
    double bs, os;  // the scalar rescalings
    float next;     // the instance's number (below 2^24), by cluster_store
};

template <int PT, int PA>
__device__ __forceinline__ ResPlaces<PT, PA> res_batch_places(const ResBatchInst &I, int m, int n, bool mixed, bool es) {
    return ResPlaces<PT, PA>(m, n, mixed, I.mostA[2], I.mostT[2], I.mostA[1], I.mostT[1], es, 8);
}

// Everything before the PDHG epochs: the entries, the scaling, the norms, ‖A'‖₂ and the start.
template <int NC, bool MIXED, bool ES, int PT, int PA>
__device__ __noinline__ void res_batch_setup(const BatchArgs &A, const BatchRes &B, const ResBatchInst &I,
                                             unsigned char *scratch, ResBatchShared &bsh) {
    ResShared<uint16_t> &s = bsh.s;
    const BatchInst &D = A.inst[I.id];
    const int m = D.m, n = D.n, c = res_rank<NC>();
    const auto L = res_batch_places<PT, PA>(I, m, n, MIXED, ES);
    const ResScratch W(I.sA[NC], I.sT[NC], m, n, D.nta, D.ntt, MIXED);
    auto src = [&](bool a) {
        ResSrc<uint16_t> q{};
        const int *most = a ? I.mostA : I.mostT;
        q.rows = a ? m : n;
        q.heavy = a ? I.heavyA : I.heavyT;
        q.ntiles = a ? D.nta : D.ntt;
        q.most_rows = most[0];
        q.most_slots = most[1];
        q.most_tasks = most[2];
        q.tasks = B.tasks + (a ? I.tasksA : I.tasksT);
        q.wt = B.wt + (a ? I.wtA : I.wtT);
        q.p0 = a ? I.pA : I.pT;
        q.s0 = a ? I.sA : I.sT;
        q.perm = a ? B.permA + D.mo : B.permT + D.no;
        q.ci = (uint16_t *)(scratch + (a ? W.ciA : W.ciT));
        q.v = (double *)(scratch + (a ? W.vA : W.vT));
        q.v32 = MIXED ? (float *)(scratch + (a ? W.v32A : W.v32T)) : nullptr;
        q.rp = a ? A.a_rp + D.rpa : A.t_rp + D.rpt;
        q.tiles = a ? A.a_tiles + D.ta : A.t_tiles + D.tt;
        return q;
    };
    const ResSrc<uint16_t> SA = src(true), ST = src(false);
    SolverPtrs g{};
    g.pk = (CheckQuad *)(scratch + W.pk);
    g.pky = (double2 *)(scratch + W.pky);
    double *part = (double *)(scratch + W.part);
    g.partP = part;
    g.partT = part + (size_t)D.ntt * NP_P;
    g.partP0 = g.partT + (size_t)D.ntt * NP_T;
    double *ppart = g.partP0 + D.ntt;
    g.partD = ppart + D.ntt;
    g.partD0 = g.partD + (size_t)D.nta * NP_D;
    double *vecs = (double *)(scratch + W.vecs);
    const ResVecs vec{vecs, vecs + n, vecs + 2 * n, vecs + 3 * n, vecs + 3 * n + m};
    res_open(s, L, SA, ST, g, vec, (double *)(scratch + W.contrib), c);
    const ResCtx<uint16_t> &R = s.R;
    const ResSide<uint16_t> &MA = R.A, &MT = R.T;
    const SolverPtrs &S = R.S;

    // the entries as given, then the scaling passes on them
    double *gvA = SA.v + SA.s0[c], *gvT = ST.v + ST.s0[c];
    double *vA = ES ? &dsm_at<double>(L.valA) : gvA, *vT = ES ? &dsm_at<double>(L.valT) : gvT;
    res_fill(MA, SA.ci + SA.s0[c], vA, SA.rp, A.a_ci + D.nz, A.av0 + D.nz, B.invT + D.no, n);
    res_fill(MT, ST.ci + ST.s0[c], vT, ST.rp, A.t_ci + D.nz, A.tv0 + D.nz, B.invA + D.mo, m);
    __syncthreads();
    // rs and cs over positions in pf and df, and in row order for the norms and the solution
    double *rs = vec.pf, *cs = vec.df, *grs = A.rs + D.mo, *gcs = A.cs + D.no;
    res_scale<NC>(s, A, vA, vT, rs, cs);
    for (int k = MA.p0 + threadIdx.x; k < MA.p1; k += RES_BT) grs[MA.perm[k]] = rs[k];
    for (int k = MT.p0 + threadIdx.x; k < MT.p1; k += RES_BT) gcs[MT.perm[k]] = cs[k];
    auto finish = [&](const ResSide<uint16_t> &M, const double *v, double *gv, float *gv32) {
        for (int i = threadIdx.x; i < M.slots; i += RES_BT) {
            const double x = v[i];
            if (ES) gv[i] = x;
            if (MIXED) gv32[i] = (float)x;
        }
    };
    finish(MA, vA, gvA, MIXED ? SA.v32 + SA.s0[c] : nullptr);
    finish(MT, vT, gvT, MIXED ? ST.v32 + ST.s0[c] : nullptr);
    res_sync<NC>();
    const double *oc = A.oc + D.no, *olv = A.olv + D.no, *ouv = A.ouv + D.no, *olc = A.olc + D.mo, *ouc = A.ouc + D.mo;
    double norms[4];
    res_norms(olc, ouc, oc, grs, gcs, m, n, norms);
    const double bs = A.rescale ? 1.0 / (1.0 + norms[0]) : 1.0, os = A.rescale ? 1.0 / (1.0 + norms[1]) : 1.0;
    if (ES) {
        res_load_entries<double>(MA, gvA, L.valA, L.atA, L.xbar);
        res_load_entries<double>(MT, gvT, L.valT, L.atT, L.y);
    }
    if (threadIdx.x == 0) {
        bsh.bs = bs;
        bsh.os = os;
        s.prm = A.base;
        s.prm.b_norm = norms[2];
        s.prm.c_norm = norms[3];
        s.prm.c0 = D.c0;
        s.prm.obj_factor = 1.0 / (bs * os);
        s.until = ~0ull;
        s.trace = nullptr;
        s.trace_cap = 0;
        s.mixed = MIXED;
        s.count_bad_first = 1;
    }
    for (int k = MT.p0 + threadIdx.x; k < MT.p1; k += RES_BT) {
        const int j = MT.perm[k];
        const double f = cs[k];
        double cj = oc[j] * f, lo = olv[j] / f, hi = ouv[j] / f;
        if (A.rescale) {
            lo *= bs;
            hi *= bs;
            cj *= os;
        }
        const_cast<double *>(S.c)[k] = cj;
        const_cast<double *>(S.lv)[k] = lo;
        const_cast<double *>(S.uv)[k] = hi;
        vec.df[k] = 1.0 / (f * os);
        S.x[k] = S.xa[k] = S.xt[k] = 0.0;  // x_t and y_t: a solve that ends before its first pass returns them
    }
    for (int k = MA.p0 + threadIdx.x; k < MA.p1; k += RES_BT) {
        const int i = MA.perm[k];
        const double f = rs[k];
        double lo = olc[i] * f, hi = ouc[i] * f;
        if (A.rescale) {
            lo *= bs;
            hi *= bs;
        }
        const_cast<double *>(S.lc)[k] = lo;
        const_cast<double *>(S.uc)[k] = hi;
        vec.pf[k] = 1.0 / (f * bs);
        S.ya[k] = S.yt[k] = 0.0;
    }
    res_sync<NC>();
    if (D.nnz > 0) res_power<NC, ES>(s, L, A.power_iterations, ppart);
    res_sync<NC>();  // y is the power iteration's until here
    if (threadIdx.x == 0) {
        const bool numerical = D.nnz > 0 && s.st.error == ERR_NUMERICAL_POWER;
        const double norm_est = D.nnz > 0 ? sqrt(s.st.pi_lambda) * 1.01 : 1.0;
        DevState &st = s.st;
        s.prm.eta = A.step_size_factor / norm_est;
        st = DevState{};
        st.omega = A.rescale ? 1.0 : (1.0 + s.prm.c_norm) / (1.0 + s.prm.b_norm);
        st.status = -1;
        st.fp64 = MIXED ? 0 : 1;
        st.anchor_residual = INFINITY;
        st.prev_residual = INFINITY;
        st.pid_best_weight = st.omega;
        st.pid_best_balance = INFINITY;
        st.mx_best = INFINITY;
        st.pi_done = 1;
        if (numerical) {
            st.done = 1;
            st.error = ERR_NUMERICAL_POWER;
        }
    }
    for (int k = threadIdx.x; k < m; k += RES_BT) {
        S.y[k] = 0.0;
        if (MIXED) S.y32[k] = 0.0f;
    }
    if (MIXED && ES) {
        res_load_entries<float>(MA, MA.v32, L.valA, L.atA, L.xbar32);
        res_load_entries<float>(MT, MT.v32, L.valT, L.atT, L.y32);
    }
    res_sync<NC>();
}

// The result and the solution in the original space (solver.rs:422-437).
template <int NC>
__device__ __noinline__ void res_batch_finish(const BatchArgs &A, const ResBatchInst &I, ResBatchShared &bsh) {
    ResShared<uint16_t> &s = bsh.s;
    const BatchInst &D = A.inst[I.id];
    const ResSide<uint16_t> &MA = s.R.A, &MT = s.R.T;
    const double bs = bsh.bs, os = bsh.os, *grs = A.rs + D.mo, *gcs = A.cs + D.no;
    double *ox = A.ox + D.no, *oy = A.oy + D.mo;
    for (int k = MT.p0 + threadIdx.x; k < MT.p1; k += RES_BT) {
        const int j = MT.perm[k];
        ox[j] = s.R.S.xt[k] * gcs[j] / bs;
    }
    for (int k = MA.p0 + threadIdx.x; k < MA.p1; k += RES_BT) {
        const int i = MA.perm[k];
        oy[i] = s.R.S.yt[k] * grs[i] / os;
    }
    if (threadIdx.x == 0 && res_rank<NC>() == 0) {
        const DevState &st = s.st;
        sp_batch_result r;
        const double sign = D.maximize ? -1.0 : 1.0;
        r.status = st.error ? -1 - st.error : st.status;
        r.objective = sign * st.primal_obj;
        r.dual_objective = sign * st.dual_obj;
        r.primal_residual = st.primal_res;
        r.dual_residual = st.dual_res;
        r.gap = fabs(st.primal_obj - st.dual_obj);
        r.iterations = st.total;
        r.restarts = st.restarts;
        r.lanes_per_row = 0;
        r.handed_off = st.handoff ? 2 : 0;  // 2: the host finishes it
        A.res[I.id] = r;
    }
    res_sync<NC>();
}

// One class of instances: clusters of NC CTAs take them from the class's counter.
template <int NC, bool MIXED, int PT, int PA>
__global__ void __launch_bounds__(RES_BT, 1)
    k_batch_res(const __grid_constant__ BatchArgs A, const __grid_constant__ BatchRes B,
                const __grid_constant__ ResBatchClass K) {
    __shared__ ResBatchShared b;
    unsigned char *scratch = K.scratch + (size_t)(blockIdx.x / NC) * K.scratch_bytes;
    const ResTailStop stop{&A};
    for (;;) {
        if (threadIdx.x == 0 && res_rank<NC>() == 0) {
            b.next = (float)batch_claim(A, K.counter, K.count);
            publish<NC>(&b.next);
        }
        res_sync<NC>();
        const int slot = (int)b.next;
        res_sync<NC>();
        if (slot >= K.count) return;
        const ResBatchInst &I = K.inst[slot];
        auto solve = [&](auto in_shared) {
            constexpr bool ES = decltype(in_shared)::value;
            res_batch_setup<NC, MIXED, ES, PT, PA>(A, B, I, scratch, b);
            const auto L = res_batch_places<PT, PA>(I, b.s.R.A.rows, b.s.R.T.rows, MIXED, ES);
            if constexpr (MIXED) {
                res_epochs<NC, true, ES, ES>(b.s, L, stop);
                res_sync<NC>();
                if (ES && !b.s.st.done) {
                    res_load_entries<double>(b.s.R.A, b.s.R.A.v, L.valA, L.atA, L.xbar);
                    res_load_entries<double>(b.s.R.T, b.s.R.T.v, L.valT, L.atT, L.y);
                    __syncthreads();
                }
            }
            res_epochs<NC, false, ES, ES>(b.s, L, stop);
            res_sync<NC>();
        };
        if (I.es) solve(std::true_type{});
        else solve(std::false_type{});
        res_batch_finish<NC>(A, I, b);
    }
}

}  // namespace sp
