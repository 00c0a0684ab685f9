// Device-resident L-BFGS for the dual weights.
//
// Replaces the solver loop of direct_ot (ot_op.cuh:289-537).  The reference
// runs the two-loop recursion with one kernel per vector operation and moves
// every dot product to the host (2m+1 device->host copies of N doubles per
// iteration, ot_op.cuh:298-337).  Here the two-loop runs on the Gram matrix of
// the basis {s_0..s_{m-1}, y_0..y_{m-1}, g} (the vector-free form of the
// recursion): after each accepted step one pass over N computes the 5m+1 new
// dot products, and one launch runs the recursion on the (2m+1)^2 matrix and
// forms d = sum_j delta_j b_j.  Every reduction is a fixed-order
// tree (per-block partials summed in block order by the last block), so a
// solve is bit-reproducible run to run.  Line-search decisions are taken by
// one device thread as well; the host only reads a flag.
#include "cot_common.cuh"
#include "../../include/causticot.h"
#include <math.h>
#include <algorithm>

namespace cot {

#define FULLMASK 0xffffffffu
#define RED_THREADS 256

// Blocks of the reductions: a cell a thread up to 296 blocks (two an SM),
// whose sums a warp adds in at most ten loads a lane.  With four cells a thread
// and a thread that added the blocks one after the other, k_reduce_eval took
// 11 us at 4,096 sites (4 blocks) and 23 at 262,144 (256 blocks); now 7 and
// 12.
int reduce_blocks(int n) { return std::max(1, std::min((n + RED_THREADS - 1) / RED_THREADS, 2 * 148)); }

__device__ __forceinline__ double wsum(double v)
{
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(FULLMASK, v, o);
    return v;
}
__device__ __forceinline__ double wmax(double v)
{
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v = fmax(v, __shfl_xor_sync(FULLMASK, v, o));
    return v;
}

// Sum (or max) of the blocks' partials of one value by a warp: lane l blocks l,
// l + 32, ..., then the lanes, always in that order (L2 reads: partials of other
// blocks are never taken from a stale L1 line).  lane_partials is a lane's part.
template <bool MAX>
__device__ __forceinline__ double lane_partials(const double *p, unsigned nblocks)
{
    double r = MAX ? -INFINITY : 0.0;
#pragma unroll 5
    for (unsigned b = threadIdx.x & 31; b < nblocks; b += 32) {
        const double v = __ldcg(p + b);
        r = MAX ? fmax(r, v) : r + v;
    }
    return r;
}
template <bool MAX>
__device__ __forceinline__ double warp_partials(const double *p, unsigned nblocks)
{
    const double r = lane_partials<MAX>(p, nblocks);
    return MAX ? wmax(r) : wsum(r);
}

// Fixed-order block reduction of one value (sum or max).  All threads call it.
template <bool MAX>
__device__ double block_reduce(double v, double *sh)
{
    int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, nw = blockDim.x >> 5;
    v = MAX ? wmax(v) : wsum(v);
    __syncthreads();
    if (lane == 0) sh[wid] = v;
    __syncthreads();
    double r = MAX ? -INFINITY : 0.0;
    if (threadIdx.x == 0) {
        for (int k = 0; k < nw; k++) r = MAX ? fmax(r, sh[k]) : r + sh[k];
        sh[32] = r;
    }
    __syncthreads();
    return sh[32];
}

#define COT_F_NOISE 1e-12  // relative noise of the objective the line search tolerates

// Line-search decision for the trial just reduced (one thread).  The control
// block's fields are read together first and written together last: one after
// the other, each waiting for the store before it, they took longer than the
// reduction.
__device__ void ls_decide(CotSolver *S, const CotEvalOut &o)
{
    const int mode = S->mode, stop_nonempty = S->stop_nonempty, final_eval = S->final_eval, max_ls = S->max_ls;
    const int evals = S->evals, rejects = S->ring_rejects, trials = S->trials;
    const double t = S->t, t0 = S->t0, f = S->f, f_lo = S->f_lo, gd = S->gd, c1 = S->c1, c2 = S->c2;
    const double hi = S->hi, lo = S->lo;
    const bool bad = o.overflow > 0;
    bool accepted = false, active = true;
    double nt = t, nhi = hi, nlo = lo, nf_lo = f_lo;
    int ntrials = trials, nfinal = final_eval;
    bool count_reject = false;
    if (mode == COT_SOLVE_REFERENCE) {
        // ot_op.cuh:360-426
        if (bad) {
            count_reject = true;
            nt = t * 0.5;
        } else if (o.f < f) {
            accepted = true;
        } else {
            nt = t * 0.5;
        }
        if (!accepted && nt <= 1e-4 * t0) active = false;  // restart
    } else if (stop_nonempty && o.empty == 0 && !bad) {
        // a solve that only has to give every cell mass takes the first trial
        // point where none is empty
        accepted = true;
    } else if (final_eval) {
        accepted = true;
    } else {
        // strong Wolfe: bracket by doubling, zoom by bisection
        count_reject = bad;
        // approximate Wolfe (Hager and Zhang): near convergence the objective's
        // evaluation noise (rounding in every cell's terms, about 1e-16 of |f|
        // per cell) exceeds the decrease a step can still make, and comparisons
        // of f stop telling steps apart.  A change of f within COT_F_NOISE |f|
        // is then not held against the step, provided the slope at the trial
        // point g(t).d <= (2 c1 - 1) g.d: the directional derivative decides.
        const bool approx = o.f <= f + COT_F_NOISE * fabs(f) && o.gtd <= (2.0 * c1 - 1.0) * gd;
        if (bad || (!approx && (!(o.f <= f + c1 * t * gd) || o.f >= f_lo))) {
            nhi = t;
        } else if (fabs(o.gtd) <= c2 * fabs(gd)) {
            accepted = true;
        } else if (o.gtd > 0.0) {
            nhi = t;
        } else {
            // a step taken on the approximate conditions may sit a rounding
            // above f_lo: it moves the bracket's low end but never raises f_lo
            nlo = t;
            nf_lo = fmin(f_lo, o.f);
        }
        if (!accepted) {
            ntrials = trials + 1;
            if (ntrials >= max_ls) {
                if (nlo > 0.0) {
                    nt = nlo;
                    nfinal = 1;
                } else {
                    active = false;  // failed
                }
            } else {
                nt = isinf(nhi) ? 2.0 * t : 0.5 * (nlo + nhi);
            }
        }
    }
    S->evals = evals + 1;
    S->last = o;
    S->accepted = accepted ? 1 : 0;
    if (accepted || !active) S->ls_active = 0;
    S->ring_rejects = rejects + (count_reject ? 1 : 0);
    S->t = nt;
    S->hi = nhi;
    S->lo = nlo;
    S->f_lo = nf_lo;
    S->trials = ntrials;
    S->final_eval = nfinal;
}

// One pass over the cells: objective, gradient statistics, directional
// derivative; the last block finishes the sums and (in a solve) decides.
__global__ void __launch_bounds__(RED_THREADS) k_reduce_eval(int n, const double *__restrict__ mu,
                                                            const double *__restrict__ fc, const int *__restrict__ nv,
                                                            const double *__restrict__ wt,
                                                            const double *__restrict__ nu, const double *__restrict__ d,
                                                            int max_ring, double *partials, unsigned int *ticket,
                                                            CotEvalOut *out, CotSolver *S)
{
    __shared__ double sh[8], red[7][RED_THREADS / 32];
    __shared__ bool last;
    if (S != nullptr && (S->done || !S->ls_active)) return;
    double f = 0.0, gtd = 0.0, mx = 0.0, gn = 0.0, emp = 0.0, ovf = 0.0, mnv = 0.0;
    int per = (n + gridDim.x - 1) / gridDim.x;
    int b0 = blockIdx.x * per, b1 = min(n, b0 + per);
    for (int i = b0 + threadIdx.x; i < b1; i += blockDim.x) {
        double g = mu[i] - nu[i];
        f += fc[i] - wt[i] * nu[i];
        if (d != nullptr) gtd += g * d[i];
        double rel = nu[i] > 0.0 ? fabs(g) / nu[i] : (g != 0.0 ? INFINITY : 0.0);
        mx = (rel == rel) ? fmax(mx, rel) : INFINITY;  // a NaN mass counts as unconverged
        gn += g * g;
        emp += (mu[i] == 0.0) ? 1.0 : 0.0;
        ovf += (nv[i] > max_ring) ? 1.0 : 0.0;
        mnv = fmax(mnv, (double)nv[i]);
    }
    // warps' sums in shared memory, added in warp order by a thread a value
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    f = wsum(f);
    gtd = wsum(gtd);
    mx = wmax(mx);
    gn = wsum(gn);
    emp = wsum(emp);
    ovf = wsum(ovf);
    mnv = wmax(mnv);
    if (lane == 0) {
        red[0][wid] = f;
        red[1][wid] = gtd;
        red[2][wid] = mx;
        red[3][wid] = gn;
        red[4][wid] = emp;
        red[5][wid] = ovf;
        red[6][wid] = mnv;
    }
    __syncthreads();
    if (threadIdx.x < 7) {
        const int k = threadIdx.x;
        const bool top = k == 2 || k == 6;
        double r = top ? -INFINITY : 0.0;
        for (int w = 0; w < RED_THREADS / 32; w++) r = top ? fmax(r, red[k][w]) : r + red[k][w];
        partials[k * gridDim.x + blockIdx.x] = r;
        __threadfence();
    }
    __syncthreads();
    if (threadIdx.x == 0) last = atomicAdd(ticket, 1u) == gridDim.x - 1;
    __syncthreads();
    if (!last) return;
    __threadfence();
    // a warp a value
    if (wid < 7) {
        const double *p = partials + wid * gridDim.x;
        const double r = (wid == 2 || wid == 6) ? warp_partials<true>(p, gridDim.x) : warp_partials<false>(p, gridDim.x);
        if (lane == 0) sh[wid] = r;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        const double *r = sh;
        CotEvalOut o;
        o.f = r[0];
        o.gtd = r[1];
        o.maxrel = r[2];
        o.gnorm2 = r[3];
        o.empty = (int)r[4];
        o.overflow = (int)r[5];
        o.maxnv = (int)r[6];
        o.pad = 0;
        *out = o;
        *ticket = 0u;
        if (S != nullptr) ls_decide(S, o);
    }
}

void launch_reduce(const CotGeo &g, const double *mu, const double *fc, const int *nv, const double *wt,
                   const double *d, int max_ring, double *partials, unsigned int *ticket, CotEvalOut *out,
                   CotSolver *solver, CotCtx &c)
{
    int nb = reduce_blocks(g.n);
    k_reduce_eval<<<nb, RED_THREADS, 0, c.s>>>(g.n, mu, fc, nv, wt, g.nu, d, max_ring, partials, ticket, out, solver);
    c.launches++;
}

// ---------------------------------------------------------------------------
// the start of an iteration
// ---------------------------------------------------------------------------
// Two-loop recursion on the Gram matrix (ot_op.cuh:291-351): delta gives
// d = sum_j delta_j basis_j; then the descent safeguard.  Every block runs the
// recursion for itself (its first warp, the (2m+1)^2 matrix in shared memory)
// and forms its part of d; the block that finishes last, when all have read
// the control block, writes the iteration's start into it.  The recursion
// keeps r = G delta in the lanes and updates it with every change of delta, so
// a step is a shuffle and a fused multiply-add and not a dot product; as a
// kernel of its own, with dot products, it took 12 us and its launch.
__global__ void __launch_bounds__(RED_THREADS) k_begin_direction(int n, CotSolver *S, const double *__restrict__ Sv,
                                                                 const double *__restrict__ Yv,
                                                                 const double *__restrict__ mu,
                                                                 const double *__restrict__ nu, double *__restrict__ d,
                                                                 unsigned int *ticket)
{
    __shared__ double G[COT_BASIS * COT_BASIS];
    __shared__ double dl[COT_BASIS];
    __shared__ double gd_s;
    __shared__ bool reset_s, last;
    // only at an iteration boundary: inside a device-driven loop this kernel
    // also runs before every further trial of a line search
    if (S->done || !S->need_begin) return;
    const int m = S->m, B = 2 * m + 1, gi = 2 * m;
    const int k = S->k;
    for (int q = threadIdx.x; q < B * B; q += blockDim.x) G[q] = S->G[(q / B) * COT_BASIS + q % B];
    const int lane = threadIdx.x & 31;
    const double rho = lane < m ? S->rho[lane] : 0.0;
    const double H0 = S->H0;
    const bool skip = (S->mode == COT_SOLVE_REFERENCE) && S->restart;
    __syncthreads();
    if (threadIdx.x < 32) {
        constexpr int Q = (COT_BASIS + 31) / 32;
        double x[Q], r[Q];  // delta and G delta, entry c in lane c % 32
#pragma unroll
        for (int q = 0; q < Q; q++) {
            const int c = lane + 32 * q;
            x[q] = c == gi ? -1.0 : 0.0;
            r[q] = c < B ? -G[c * B + gi] : 0.0;
        }
        const auto at = [&](int c) {
            double v = r[0];
#pragma unroll
            for (int q = 1; q < Q; q++)
                if (c >= 32 * q) v = r[q];
            return __shfl_sync(FULLMASK, v, c & 31);
        };
        const auto add = [&](int c, double v) {  // delta_c += v
#pragma unroll
            for (int q = 0; q < Q; q++) {
                if (lane + 32 * q == c) x[q] += v;
                if (lane + 32 * q < B) r[q] += v * G[(lane + 32 * q) * B + c];
            }
        };
        const int cnt = k < m ? k : m;
        if (!skip) {
            double alpha = 0.0;  // of step i in lane i - 1
            for (int i = 1; i <= cnt; i++) {
                const int idx = ((k - i) % m + m) % m;
                const double a = at(idx) * __shfl_sync(FULLMASK, rho, idx);
                if (lane == i - 1) alpha = a;
                add(m + idx, -a);
            }
#pragma unroll
            for (int q = 0; q < Q; q++) {
                x[q] *= H0;
                r[q] *= H0;
            }
            for (int i = cnt; i > 0; i--) {
                const int idx = ((k - i) % m + m) % m;
                const double beta = __shfl_sync(FULLMASK, rho, idx) * at(m + idx);
                add(idx, __shfl_sync(FULLMASK, alpha, i - 1) - beta);
            }
        }
        double gd = at(gi);
        const bool reset = !(gd < 0.0);  // not a descent direction: steepest descent
        if (reset) gd = -G[gi * B + gi];
#pragma unroll
        for (int q = 0; q < Q; q++) {
            const int c = lane + 32 * q;
            if (c < B) dl[c] = reset ? (c == gi ? -1.0 : 0.0) : x[q];
        }
        if (lane == 0) {
            gd_s = gd;
            reset_s = reset;
        }
    }
    __syncthreads();
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        double r = dl[2 * m] * (mu[i] - nu[i]);
        for (int j = 0; j < m; j++) {
            double a = dl[j], b = dl[m + j];
            if (a != 0.0) r += a * Sv[(size_t)j * n + i];
            if (b != 0.0) r += b * Yv[(size_t)j * n + i];
        }
        d[i] = r;
    }
    if (threadIdx.x == 0) last = atomicAdd(ticket, 1u) == gridDim.x - 1;
    __syncthreads();
    if (!last || threadIdx.x != 0) return;
    *ticket = 0u;
    const int evals = S->evals, empty = S->empty;
    const double gnorm2 = S->gnorm2, t0 = S->t0, f = S->f;
    if (reset_s) {
        S->k = 0;
        S->H0 = 1.0;
    }
    S->need_begin = 0;
    S->eval_mark = evals;
    S->gnorm_stale = sqrt(gnorm2);
    S->empty_stale = empty;
    S->gd = gd_s;
    S->t = t0;
    S->lo = 0.0;
    S->hi = INFINITY;
    S->f_lo = f;
    S->trials = 0;
    S->ls_active = 1;
    S->accepted = 0;
    S->final_eval = 0;
}

void launch_begin_direction(const CotGeo &g, CotSolver *S, const double *Sv, const double *Yv, const double *mu,
                            double *d, unsigned int *ticket, CotCtx &c)
{
    int blocks = (g.n + RED_THREADS - 1) / RED_THREADS;
    if (blocks > 2 * 148) blocks = 2 * 148;
    k_begin_direction<<<blocks, RED_THREADS, 0, c.s>>>(g.n, S, Sv, Yv, mu, g.nu, d, ticket);
    c.launches++;
}

// Line search gave up (ot_op.cuh:413-425): keep the point, drop the history.
__device__ __forceinline__ void reject(CotSolver *S)
{
    if (S->done || S->accepted || S->ls_active) return;
    const int mode = S->mode, k = S->k, restarts = S->restarts, iter = S->iter, max_iter = S->max_iter;
    S->need_begin = 1;
    if (mode == COT_SOLVE_REFERENCE) {
        S->restart = 1;
    } else if (k == 0) {
        S->failed = 1;
        S->done = 1;
        return;
    }
    S->k = 0;
    S->H0 = 1.0;
    S->restarts = restarts + 1;
    S->iter = iter + 1;
    if (iter + 1 >= max_iter) S->done = 1;
}

// Condition of the device-driven trial loop (a WHILE node of a CUDA graph):
// go on until the solve is done or reaches the iteration where the host
// wants to look (a progress report).
__device__ __forceinline__ void loop_condition(cudaGraphConditionalHandle hc, const CotSolver *S)
{
    cudaGraphSetConditional(hc, (!S->done && S->iter < S->pause_iter) ? 1u : 0u);
}

// Accept the trial: s_h = t d, y_h = mu_t - mu, w = w_t, mu = mu_t, then the
// new Gram entries s_h.y_j, y_h.s_j, y_h.y_j, g.s_j, g.y_j, g.g; the last
// block updates the matrix, the history scalars (ot_op.cuh:434-466) and the
// stop test (ot_op.cuh:468-476, 510).
// LOOP: the end of a pass of the device-driven trial loop.  A pass whose trial
// was not accepted ends here too (the rejection, where the line search gave
// up), and the loop's condition is set.
template <bool LOOP>
__global__ void __launch_bounds__(RED_THREADS) k_accept(int n, CotSolver *S, double *Sv, double *Yv, double *w,
                                                       const double *__restrict__ wt, double *mu,
                                                       const double *__restrict__ mut, const double *__restrict__ nu,
                                                       const double *__restrict__ d, double *partials,
                                                       unsigned int *ticket, int initial,
                                                       cudaGraphConditionalHandle hc)
{
    constexpr int NW = RED_THREADS / 32, SLOTS = (COT_MAX_HIST + NW - 1) / NW;
    __shared__ double sn_s[RED_THREADS], yn_s[RED_THREADS], g_s[RED_THREADS], red[NW];
    __shared__ double tot[5 * COT_MAX_HIST + 1];
    __shared__ bool last;
    // (a rejection may raise `done` while blocks of the same launch read it:
    // they leave either way)
    if (S->done || (!initial && !S->accepted)) {
        if (LOOP && blockIdx.x == 0 && threadIdx.x == 0) {
            reject(S);
            loop_condition(hc, S);
        }
        return;
    }
    const int m = S->m, k0 = S->k;
    const double t = S->t;
    const int h = k0 % m;
    const int nvals = 5 * m + 1;
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    int per = (n + gridDim.x - 1) / gridDim.x;
    int b0 = blockIdx.x * per, b1 = min(n, b0 + per);
    const int cnt = initial ? 0 : (k0 + 1 < m ? k0 + 1 : m);  // slots that hold pairs after this update
    const auto held = [&](int j) { return j < m && ((h - j) % m + m) % m < cnt; };
    // 256 cells at a time: a thread a cell for the new vectors, which go to
    // shared memory, then a warp a slot for the dot products with its pair, so
    // that the slots' loads and sums run side by side (all threads on one slot
    // after the other took 30 us for ten of them at 4,096 sites, this 12)
    double acc[SLOTS][5], gg = 0.0;
#pragma unroll
    for (int s = 0; s < SLOTS; s++)
        for (int v = 0; v < 5; v++) acc[s][v] = 0.0;
    for (int base = b0; base < b1; base += RED_THREADS) {
        const int i = base + threadIdx.x;
        double sn = 0.0, yn = 0.0, g = 0.0;
        if (i < b1) {
            const double mt = mut[i];
            if (!initial) {
                sn = __dmul_rn(t, d[i]);
                yn = mt - mu[i];
                Sv[(size_t)h * n + i] = sn;
                Yv[(size_t)h * n + i] = yn;
                w[i] = wt[i];
            }
            mu[i] = mt;
            g = mt - nu[i];
        }
        sn_s[threadIdx.x] = sn;
        yn_s[threadIdx.x] = yn;
        g_s[threadIdx.x] = g;
        gg += g * g;
        __syncthreads();
#pragma unroll
        for (int s = 0; s < SLOTS; s++) {
            const int j = wid + NW * s;
            if (!held(j)) continue;
            double sj[NW], yj[NW];
#pragma unroll
            for (int q = 0; q < NW; q++) {
                const int c = lane + 32 * q;
                const bool in = base + c < b1;
                sj[q] = j == h ? sn_s[c] : (in ? Sv[(size_t)j * n + base + c] : 0.0);
                yj[q] = j == h ? yn_s[c] : (in ? Yv[(size_t)j * n + base + c] : 0.0);
            }
#pragma unroll
            for (int q = 0; q < NW; q++) {
                const int c = lane + 32 * q;
                acc[s][0] += sn_s[c] * yj[q];
                acc[s][1] += yn_s[c] * sj[q];
                acc[s][2] += yn_s[c] * yj[q];
                acc[s][3] += g_s[c] * sj[q];
                acc[s][4] += g_s[c] * yj[q];
            }
        }
        __syncthreads();
    }
    gg = wsum(gg);
    if (lane == 0) red[wid] = gg;
#pragma unroll
    for (int s = 0; s < SLOTS; s++) {
        const int j = wid + NW * s;
        if (j >= m) continue;
#pragma unroll
        for (int v = 0; v < 5; v++) {
            const double r = wsum(acc[s][v]);
            if (lane == 0) partials[(size_t)(5 * j + v) * gridDim.x + blockIdx.x] = r;
        }
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        double r = 0.0;
        for (int k = 0; k < NW; k++) r += red[k];
        partials[(size_t)5 * m * gridDim.x + blockIdx.x] = r;
    }
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0) {
        unsigned int tk = atomicAdd(ticket, 1u);
        last = (tk == gridDim.x - 1);
    }
    __syncthreads();
    if (!last) return;
    __threadfence();
    // a warp a value, four values' loads at once
    for (int v0 = wid; v0 < nvals; v0 += 4 * NW) {
        double r[4];
#pragma unroll
        for (int q = 0; q < 4; q++) {
            const int v = v0 + NW * q;
            r[q] = v < nvals ? lane_partials<false>(partials + (size_t)v * gridDim.x, gridDim.x) : 0.0;
        }
#pragma unroll
        for (int q = 0; q < 4; q++) {
            r[q] = wsum(r[q]);
            if (lane == 0 && v0 + NW * q < nvals) tot[v0 + NW * q] = r[q];
        }
    }
    __syncthreads();
    const int gi = 2 * m;
    double *G = S->G;
    // a thread a slot for the matrix
    for (int j = threadIdx.x; j < m; j += blockDim.x) {
        const int age = ((h - j) % m + m) % m;
        if (cnt == 0 || age >= cnt) continue;
        if (!initial) {
            G[h * COT_BASIS + (m + j)] = G[(m + j) * COT_BASIS + h] = tot[5 * j + 0];
            if (j != h) G[(m + h) * COT_BASIS + j] = G[j * COT_BASIS + (m + h)] = tot[5 * j + 1];
            G[(m + h) * COT_BASIS + (m + j)] = G[(m + j) * COT_BASIS + (m + h)] = tot[5 * j + 2];
        }
        G[gi * COT_BASIS + j] = G[j * COT_BASIS + gi] = tot[5 * j + 3];
        G[gi * COT_BASIS + (m + j)] = G[(m + j) * COT_BASIS + gi] = tot[5 * j + 4];
    }
    if (threadIdx.x != 0) return;
    // the control block's fields are read together before the first is written
    const CotEvalOut o = S->last;
    const int mode = S->mode, iter = S->iter, max_iter = S->max_iter, stop_nonempty = S->stop_nonempty;
    const int empty_stale = S->empty_stale, pause = S->pause_iter;
    const double tol = S->tol, gnorm_stale = S->gnorm_stale;
    *ticket = 0u;
    G[gi * COT_BASIS + gi] = tot[5 * m];
    // current point
    S->f = o.f;
    S->maxrel = o.maxrel;
    S->gnorm2 = o.gnorm2;
    S->empty = o.empty;
    bool done = stop_nonempty && o.empty == 0, converged = false;
    int it = iter;
    if (initial) {
        // a Wolfe-mode solve whose start already meets the tolerance stops at
        // its first evaluation (as the oracle's restatement does); the
        // reference mode always takes an iteration, as direct_ot does
        converged = mode == COT_SOLVE_WOLFE && o.maxrel <= tol;
    } else {
        const double ys = tot[5 * h + 1], yy = tot[5 * h + 2];
        if (mode == COT_SOLVE_REFERENCE) {
            S->rho[h] = 1.0 / ys;
            S->H0 = (yy > 1e-5) ? ys / yy : 1.0;
            S->k = k0 + 1;
            S->restart = 0;
            converged = gnorm_stale < tol && empty_stale == 0;
        } else {
            if (ys > 0.0) {
                S->rho[h] = 1.0 / ys;
                S->H0 = ys / yy;
                S->k = k0 + 1;
            }
            converged = o.maxrel <= tol;
        }
        it = iter + 1;
        S->iter = it;
        S->need_begin = 1;
        done = done || it >= max_iter;
    }
    if (converged) S->converged = 1;
    done = done || converged;
    if (done) S->done = 1;
    if (LOOP) cudaGraphSetConditional(hc, (!done && it < pause) ? 1u : 0u);
}

void launch_accept(const CotGeo &g, CotSolver *S, double *Sv, double *Yv, double *w, const double *wt, double *mu,
                   const double *mut, const double *d, double *partials, unsigned int *ticket, int initial,
                   const cudaGraphConditionalHandle *loop, CotCtx &c)
{
    int nb = reduce_blocks(g.n);
    if (loop != nullptr)
        k_accept<true><<<nb, RED_THREADS, 0, c.s>>>(g.n, S, Sv, Yv, w, wt, mu, mut, g.nu, d, partials, ticket, initial,
                                                    *loop);
    else
        k_accept<false><<<nb, RED_THREADS, 0, c.s>>>(g.n, S, Sv, Yv, w, wt, mu, mut, g.nu, d, partials, ticket, initial,
                                                     cudaGraphConditionalHandle{});
    c.launches++;
}

__global__ void k_reject(CotSolver *S) { reject(S); }

void launch_reject(CotSolver *S, CotCtx &c)
{
    k_reject<<<1, 1, 0, c.s>>>(S);
    c.launches++;
}

// The first evaluation becomes the current point without a line search.
__global__ void k_init_from_eval(CotSolver *S, const CotEvalOut *out)
{
    S->last = *out;
    S->evals++;
}

void launch_init_from_eval(CotSolver *S, const CotEvalOut *out, CotCtx &c)
{
    k_init_from_eval<<<1, 1, 0, c.s>>>(S, out);
    c.launches++;
}

// ---------------------------------------------------------------------------
// helpers of cot_eval and of the Fresnel-reweighted Anderson solve
// ---------------------------------------------------------------------------

// fresnel_T_unpolarized (basic_function.cuh:407-435)
__device__ double fresnel_t(const double wi[3], const double wt[3], const double nrm[3], double eta_i, double eta_t)
{
    const double eps = 1e-12;
    double ci = fabs(wi[0] * nrm[0] + wi[1] * nrm[1] + wi[2] * nrm[2]);
    double ct = fabs(wt[0] * nrm[0] + wt[1] * nrm[1] + wt[2] * nrm[2]);
    ci = fmin(1.0, fmax(0.0, ci));
    ct = fmin(1.0, fmax(0.0, ct));
    double ds = eta_i * ci + eta_t * ct;
    double dp = eta_i * ct + eta_t * ci;
    if (fabs(ds) < eps) ds = eps;
    if (fabs(dp) < eps) dp = eps;
    double rs = (eta_i * ci - eta_t * ct) / ds;
    double rp = (eta_i * ct - eta_t * ci) / dp;
    rs *= rs;
    rp *= rp;
    return 1.0 - 0.5 * (rs + rp);
}

__device__ void normalize3(double v[3])
{
    double nn = sqrt(v[0] * v[0] + v[1] * v[1] + v[2] * v[2]);
    if (nn < 1e-12) {
        v[0] = v[1] = v[2] = 0.0;
        return;
    }
    v[0] /= nn;
    v[1] /= nn;
    v[2] /= nn;
}

// compute_energy_remain_rate (basic_function.cuh:437-494) times the source
// mass: energy_i = lambda_i * T1_i * T2_i, from the cell centroids.
__global__ void k_fresnel_energy(int n, const double *__restrict__ cen, const double *__restrict__ src,
                                 const double *__restrict__ inl, const double *__restrict__ insl,
                                 const double *__restrict__ hgt, const double *__restrict__ lam, double zl,
                                 double zr, double eta, double *__restrict__ energy)
{
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    double p[3] = {src[2 * i], src[2 * i + 1], zl};
    double wi[3] = {inl[3 * i], inl[3 * i + 1], inl[3 * i + 2]};
    double ins[3] = {insl[3 * i], insl[3 * i + 1], insl[3 * i + 2]};
    double op[3] = {p[0] + hgt[i] * ins[0], p[1] + hgt[i] * ins[1], p[2] + hgt[i] * ins[2]};
    double wo[3] = {cen[2 * i] - op[0], cen[2 * i + 1] - op[1], zr - op[2]};
    normalize3(wo);
    double n2[3] = {eta * ins[0] - wo[0], eta * ins[1] - wo[1], eta * ins[2] - wo[2]};
    normalize3(n2);
    const double n1[3] = {0.0, 0.0, 1.0};
    double t1 = fresnel_t(wi, ins, n1, 1.0, eta);
    double t2 = fresnel_t(ins, wo, n2, eta, 1.0);
    energy[i] = lam[i] * (t1 * t2);
}

// Fixed-order sum of x: block partials, which every block of the scale kernel
// adds in the same order.
__global__ void __launch_bounds__(RED_THREADS) k_sum_partials(int n, const double *__restrict__ x, double *partials)
{
    __shared__ double sh[33];
    int per = (n + gridDim.x - 1) / gridDim.x;
    int b0 = blockIdx.x * per, b1 = min(n, b0 + per);
    double v = 0.0;
    for (int i = b0 + threadIdx.x; i < b1; i += blockDim.x) v += x[i];
    v = block_reduce<false>(v, sh);
    if (threadIdx.x == 0) partials[blockIdx.x] = v;
}

// nu_i = energy_i / sum(energy) * total, unless the evaluation it comes from
// had rings that are too complex
__global__ void k_scale_to_total(int n, const double *__restrict__ energy, const double *__restrict__ partials,
                                 int nparts, double total, const CotEvalOut *__restrict__ eval,
                                 double *__restrict__ nu)
{
    if (eval->overflow > 0) return;
    const double s = warp_partials<false>(partials, nparts);
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) nu[i] = energy[i] / s * total;
}

void launch_fresnel_nu(int n, const double *cen, const double *src, const double *inl, const double *insl,
                       const double *hgt, const double *lam, double zl, double zr, double eta, double total,
                       double *energy, double *partials, const CotEvalOut *eval, double *nu, CotCtx &c)
{
    k_fresnel_energy<<<(n + 255) / 256, 256, 0, c.s>>>(n, cen, src, inl, insl, hgt, lam, zl, zr, eta, energy);
    int nb = reduce_blocks(n);
    k_sum_partials<<<nb, RED_THREADS, 0, c.s>>>(n, energy, partials);
    k_scale_to_total<<<(n + 255) / 256, 256, 0, c.s>>>(n, energy, partials, nb, total, eval, nu);
    c.launches += 3;
}

// Anderson history slot h: G_h = mu - nu, F_h = w + alpha G_h
// (storage + compute_fixed_function, ot_op.cuh:1139-1142)
__global__ void k_aa_store(int n, const double *__restrict__ w, const double *__restrict__ mu,
                           const double *__restrict__ nu, double alpha, double *__restrict__ gh,
                           double *__restrict__ fh)
{
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    double g = mu[i] - nu[i];
    gh[i] = g;
    fh[i] = w[i] + alpha * g;
}

// row[j] = G_h . G_j for j < cnt (fixed order: warps' and blocks' partials, the
// last block sums)
__global__ void __launch_bounds__(RED_THREADS) k_aa_gram_row(int n, const double *__restrict__ G, int h, int cnt,
                                                            double *partials, unsigned int *ticket, double *row)
{
    constexpr int NW = RED_THREADS / 32;
    __shared__ double red[COT_MAX_HIST][NW];
    __shared__ bool last;
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    int per = (n + gridDim.x - 1) / gridDim.x;
    int b0 = blockIdx.x * per, b1 = min(n, b0 + per);
    const double *gh = G + (size_t)h * n;
#pragma unroll 4
    for (int j = 0; j < cnt; j++) {
        const double *gj = G + (size_t)j * n;
        double v = 0.0;
        for (int i = b0 + threadIdx.x; i < b1; i += blockDim.x) v += gh[i] * gj[i];
        v = wsum(v);
        if (lane == 0) red[j][wid] = v;
    }
    __syncthreads();
    if ((int)threadIdx.x < cnt) {
        double r = 0.0;
        for (int k = 0; k < NW; k++) r += red[threadIdx.x][k];
        partials[(size_t)threadIdx.x * gridDim.x + blockIdx.x] = r;
    }
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0) last = atomicAdd(ticket, 1u) == gridDim.x - 1;
    __syncthreads();
    if (!last) return;
    __threadfence();
    for (int j = wid; j < cnt; j += NW) {
        const double r = warp_partials<false>(partials + (size_t)j * gridDim.x, gridDim.x);
        if (lane == 0) row[j] = r;
    }
    if (threadIdx.x == 0) *ticket = 0u;
}

void launch_aa_store_gram(int n, const double *w, const double *mu, const double *nu, double alpha, double *G,
                          double *F, int h, int cnt, double *partials, unsigned int *ticket, double *row, CotCtx &c)
{
    k_aa_store<<<(n + 255) / 256, 256, 0, c.s>>>(n, w, mu, nu, alpha, G + (size_t)h * n, F + (size_t)h * n);
    k_aa_gram_row<<<reduce_blocks(n), RED_THREADS, 0, c.s>>>(n, G, h, cnt, partials, ticket, row);
    c.launches += 2;
}

// d = sum_j coef_j F_j - w   (compute_weighted_sum + compute_subtract, ot_op.cuh:1172-1173)
__global__ void k_aa_combine(int n, const double *__restrict__ F, const double *__restrict__ coef, int cnt,
                             const double *__restrict__ w, double *__restrict__ d)
{
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    double s = 0.0;
    for (int j = 0; j < cnt; j++) s += coef[j] * F[(size_t)j * n + i];
    d[i] = s - w[i];
}

void launch_aa_combine(int n, const double *F, const double *coef, int cnt, const double *w, double *d, CotCtx &c)
{
    k_aa_combine<<<(n + 255) / 256, 256, 0, c.s>>>(n, F, coef, cnt, w, d);
    c.launches++;
}

}  // namespace cot
