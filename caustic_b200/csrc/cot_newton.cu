// Kernels of the damped Newton solve (cot_solve_newton; no counterpart in the
// reference, whose solvers are L-BFGS and Anderson acceleration).
//
//  - k_hessian: the mass Jacobian dmu/dw at the rings the last evaluation
//    left in the ring buffer: one warp per cell, one lane per edge, each
//    edge's density line integral (cot_edge.cuh) over 2|s_i - s_j|.  Rows go
//    to an ELL layout, entry k of cell i at [k * n + i], so that a thread per
//    row reads coalesced in the solver's matrix products; rings above 32
//    vertices have their rows built by the large-ring pass of the cell kernel.
//  - k_newton_stats: |g|^2, min mu, max relative error, empty cells and the
//    largest ring at a trial point, in fixed order (last block sums).
//  - k_pcg: the Jacobi-preconditioned conjugate gradient for dmu/dw d = nu -
//    mu as ONE persistent launch: a thread owns rows, and the blocks meet at
//    two reductions an iteration, which are its barriers too (the new search
//    direction is formed on the fly from z and the previous direction inside
//    the matrix product).
#include "cot_common.cuh"
#include "cot_edge.cuh"

#include <algorithm>

namespace cot {

#define HESS_THREADS 128
#define PCG_THREADS 512
#define PCG_THREADS_R 256  // a thread owns up to 4 rows, in registers
#define PCG_CLUSTER_ROWS 16384  // 16 blocks of 4 rows a thread
#define PCG_SPIN_LIMIT (1u << 21)  // polls of a slot: about a second

__device__ __forceinline__ double hsum32(double v)
{
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

__global__ void __launch_bounds__(HESS_THREADS) k_hessian(CotGeo g, const double2 *__restrict__ rbuf,
                                                         const int *__restrict__ lbuf, const int *__restrict__ nv,
                                                         double *__restrict__ hval, int *__restrict__ hcol,
                                                         int *__restrict__ hcnt, double *__restrict__ hdiag)
{
    const int lane = threadIdx.x & 31;
    const int i = blockIdx.x * (HESS_THREADS / 32) + (threadIdx.x >> 5);
    if (i >= g.n) return;
    const int m = nv[i];
    if (m > 32) return;  // a big row, built by the large-ring pass
    if (m < 3) {
        if (lane == 0) {
            hcnt[i] = 0;
            hdiag[i] = 0.0;
        }
        return;
    }
    const double2 si = g.xy[i];
    double a = 0.0;
    int j = -1;
    if (lane < m) {
        j = lbuf[ring_at(i, lane)];
        if (j >= 0) {
            const double2 p = rbuf[ring_at(i, lane)];
            const double2 q = rbuf[ring_at(i, lane + 1 == m ? 0 : lane + 1)];
            const double2 sj = g.xy[j];
            const double ex = sj.x - si.x, ey = sj.y - si.y;
            a = edge_rho_integral(g, si.x + p.x, si.y + p.y, si.x + q.x, si.y + q.y) / (2.0 * sqrt(ex * ex + ey * ey));
        }
    }
    const unsigned site = __ballot_sync(0xffffffffu, j >= 0);
    const int pos = __popc(site & ((1u << lane) - 1u));
    if (j >= 0) {
        hval[(size_t)pos * g.n + i] = a;
        hcol[(size_t)pos * g.n + i] = j;
    }
    const double d = hsum32(a);
    if (lane == 0) {
        hcnt[i] = __popc(site);
        hdiag[i] = d;
    }
}

void launch_hessian(const CotGeo &g, const double2 *rbuf, const int *lbuf, const int *nv, double *hval, int *hcol,
                    int *hcnt, double *hdiag, CotCtx &c)
{
    const int per = HESS_THREADS / 32;
    k_hessian<<<(g.n + per - 1) / per, HESS_THREADS, 0, c.s>>>(g, rbuf, lbuf, nv, hval, hcol, hcnt, hdiag);
    c.launches++;
}

// ---------------------------------------------------------------------------
// statistics of a trial point
// ---------------------------------------------------------------------------
#define NST_THREADS 256
#define NST_VALS 5

__device__ __forceinline__ double nmax_keep_nan(double a, double b) { return (a != a || b != b) ? INFINITY : fmax(a, b); }

__global__ void __launch_bounds__(NST_THREADS) k_newton_stats(int n, const double *__restrict__ mu,
                                                             const double *__restrict__ nu, const int *__restrict__ nv,
                                                             double *partials, unsigned int *ticket,
                                                             NewtonEvalStats *out)
{
    __shared__ double sh[NST_VALS][NST_THREADS / 32];
    __shared__ bool last;
    double g2 = 0.0, mn = INFINITY, mx = 0.0, emp = 0.0, mnv = 0.0;
    const int per = (n + gridDim.x - 1) / gridDim.x;
    const int b0 = blockIdx.x * per, b1 = min(n, b0 + per);
    for (int i = b0 + threadIdx.x; i < b1; i += blockDim.x) {
        const double m = mu[i], g = m - nu[i];
        g2 += g * g;
        mn = fmin(mn, m);
        const double rel = nu[i] > 0.0 ? fabs(g) / nu[i] : (g != 0.0 ? INFINITY : 0.0);
        mx = (rel == rel) ? fmax(mx, rel) : INFINITY;
        emp += m == 0.0 ? 1.0 : 0.0;
        mnv = fmax(mnv, (double)nv[i]);
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        g2 += __shfl_xor_sync(0xffffffffu, g2, o);
        mn = fmin(mn, __shfl_xor_sync(0xffffffffu, mn, o));
        mx = nmax_keep_nan(mx, __shfl_xor_sync(0xffffffffu, mx, o));
        emp += __shfl_xor_sync(0xffffffffu, emp, o);
        mnv = fmax(mnv, __shfl_xor_sync(0xffffffffu, mnv, o));
    }
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    if (lane == 0) {
        sh[0][wid] = g2;
        sh[1][wid] = mn;
        sh[2][wid] = mx;
        sh[3][wid] = emp;
        sh[4][wid] = mnv;
    }
    __syncthreads();
    // a thread a value for the warps, then a warp a value for the blocks (their
    // partials, never NaN but in the sums, in one fixed order)
    const auto join = [](int k, double x, double y) {
        return k == 1 ? fmin(x, y) : (k == 2 || k == 4 ? fmax(x, y) : x + y);
    };
    if (threadIdx.x < NST_VALS) {
        const int k = threadIdx.x;
        double r = sh[k][0];
        for (int w = 1; w < NST_THREADS / 32; w++) r = join(k, r, sh[k][w]);
        partials[(size_t)k * gridDim.x + blockIdx.x] = r;
        __threadfence();
    }
    __syncthreads();
    if (threadIdx.x == 0) last = atomicAdd(ticket, 1u) == gridDim.x - 1;
    __syncthreads();
    if (!last) return;
    __threadfence();
    if (wid < NST_VALS) {
        double r = wid == 1 ? INFINITY : 0.0;
#pragma unroll 5
        for (unsigned b = lane; b < gridDim.x; b += 32) r = join(wid, r, __ldcg(partials + (size_t)wid * gridDim.x + b));
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) r = join(wid, r, __shfl_xor_sync(0xffffffffu, r, o));
        if (lane == 0) sh[wid][0] = r;
    }
    __syncthreads();
    if (threadIdx.x != 0) return;
    const double r[NST_VALS] = {sh[0][0], sh[1][0], sh[2][0], sh[3][0], sh[4][0]};
    NewtonEvalStats o;
    o.gnorm2 = r[0];
    o.minmu = r[1];
    o.maxrel = r[2];
    o.empty = (int)r[3];
    o.maxnv = (int)r[4];
    *out = o;
    *ticket = 0u;
}

void launch_newton_stats(int n, const double *mu, const double *nu, const int *nv, double *partials,
                         unsigned int *ticket, NewtonEvalStats *out, CotCtx &c)
{
    k_newton_stats<<<reduce_blocks(n), NST_THREADS, 0, c.s>>>(n, mu, nu, nv, partials, ticket, out);
    c.launches++;
}

// ---------------------------------------------------------------------------
// conjugate gradient, one persistent launch
// ---------------------------------------------------------------------------
// An iteration is two reductions that every block needs the result of, each
// also the barrier that publishes the vectors written before it.  What it
// costs is their latency: at 16,384 rows 10 us an iteration went into an
// atomic counter, a polled generation, a fence and a second read of the
// partials, twice.  Here a block hands its total to the others directly:
//  - up to PCG_CLUSTER_ROWS rows the blocks are one thread-block cluster
//    (at most 16): totals through distributed shared memory, the hardware's
//    cluster barrier;
//  - above, a slot per block in global memory that block 0 watches; it adds
//    the totals and hands the result on in one more slot.  (Every block
//    reading every slot took 11 to 13 us an iteration at 148 blocks.)  The
//    waits are bounded: a block that waits too long sets an error flag and
//    leaves, as do the others at their next reduction, and the host falls back.
// The totals are added in one fixed order, so a solve repeats bit for bit.  Up
// to 4 rows a thread keep their vectors and matrix entries in registers: what
// an iteration reads is the neighbours' z and direction.
// A Newton solve's time over its CG iterations, evaluations included (us,
// before and now): 4,096 sites 11 to 13, 5.6 to 6.1; 16,384 12.0, 6.4;
// 25,600 12.6, 9.0; 65,536 12.8, 9.7; 102,400 16.1, 10.9.
#define PCG_MAX_CLUSTER 16
#define PCG_ROW 8                        // matrix entries of a row kept in registers
#define PCG_POLL 5                       // slots a lane of block 0 watches at once (160 blocks)
#define PCG_SLOTS(nb) (6 * (nb) + 48)    // doubles: three sets of two per block, three results
#define PCG_EMPTY 0xffffffffffffffffull  // an unwritten slot (no sum has these bits)

struct PcgShared {
    double2 warp[32];
    double2 total[2][PCG_MAX_CLUSTER];  // cluster: every block's total, by parity of the reduction
    double2 sum;
    int ok;
};

__device__ __forceinline__ unsigned long long ld_relaxed(const unsigned long long *p)
{
    unsigned long long v;
    asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ void st_relaxed(unsigned long long *p, unsigned long long v)
{
    asm volatile("st.relaxed.gpu.global.u64 [%0], %1;" ::"l"(p), "l"(v) : "memory");
}

// The sums of v0 (and v1, where TWO) over the whole launch, in a fixed order;
// a barrier for everything written before it.  t: the number of reductions so
// far.  slots: three sets of two values per block (a set is emptied again
// while the next ones are in use).  Returns false when a wait gave up.
template <bool CL, bool TWO>
__device__ __forceinline__ bool pcg_reduce(double v0, double v1, double2 &out, int t, PcgShared &sh,
                                           unsigned long long *slots, PcgState *st)
{
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, nw = blockDim.x >> 5;
    const unsigned nb = gridDim.x;
    v0 = hsum32(v0);
    if (TWO) v1 = hsum32(v1);
    if (lane == 0) sh.warp[wid] = make_double2(v0, v1);
    __syncthreads();
    if constexpr (CL) {
        if (wid == 0) {
            const double2 w = lane < nw ? sh.warp[lane] : make_double2(0.0, 0.0);
            const double b0 = hsum32(w.x), b1 = TWO ? hsum32(w.y) : 0.0;
            if (lane < (int)nb) {
                // this block's total into block `lane`'s table
                uint32_t local = (uint32_t)__cvta_generic_to_shared(&sh.total[t & 1][blockIdx.x]), remote;
                asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(remote) : "r"(local), "r"(lane));
                asm volatile("st.shared::cluster.v2.f64 [%0], {%1, %2};" ::"r"(remote), "d"(b0), "d"(b1) : "memory");
            }
        }
        asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
        asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
        double2 b = (lane & 15) < (int)nb ? sh.total[t & 1][lane & 15] : make_double2(0.0, 0.0);
#pragma unroll
        for (int o = 8; o > 0; o >>= 1) {
            b.x += __shfl_xor_sync(0xffffffffu, b.x, o);
            if (TWO) b.y += __shfl_xor_sync(0xffffffffu, b.y, o);
        }
        out = b;
        return true;
    } else {
        if (wid == 0) {
            const double2 w = lane < nw ? sh.warp[lane] : make_double2(0.0, 0.0);
            double b0 = hsum32(w.x), b1 = TWO ? hsum32(w.y) : 0.0;
            unsigned long long *set = slots + (size_t)(t % 3) * 2 * nb;
            if (lane == 0) {
                if (b0 != b0) b0 = __longlong_as_double(0x7ff8000000000000ll);
                if (b1 != b1) b1 = __longlong_as_double(0x7ff8000000000000ll);
                __threadfence();
                st_relaxed(set + blockIdx.x, (unsigned long long)__double_as_longlong(b0));
                if (TWO) st_relaxed(set + nb + blockIdx.x, (unsigned long long)__double_as_longlong(b1));
            }
            // block 0 adds the totals (lane l blocks l, l + 32, ..., then the
            // lanes) and hands the result on: were every block to read every
            // slot, the few L2 lines that hold them would be the limit
            unsigned long long *res = slots + (size_t)6 * nb + 16 * (t % 3);
            double a0 = 0.0, a1 = 0.0;
            bool ok = true;
            const auto gave_up = [&](unsigned spins) {
                if (spins <= PCG_SPIN_LIMIT && ((spins & 1023u) != 1023u || *(volatile int *)&st->error == 0)) return false;
                atomicExch(&st->error, 1);
                return true;
            };
            if (blockIdx.x == 0) {
                for (unsigned k0 = 0; k0 < nb && ok; k0 += 32 * PCG_POLL) {
                    unsigned long long x0[PCG_POLL], x1[PCG_POLL];
#pragma unroll
                    for (int u = 0; u < PCG_POLL; u++) {
                        const bool there = k0 + 32 * u + lane < nb;
                        x0[u] = there ? PCG_EMPTY : 0ull;
                        x1[u] = there && TWO ? PCG_EMPTY : 0ull;
                    }
                    bool all = false;
                    for (unsigned spins = 0; !all && ok; spins++) {
                        all = true;
#pragma unroll
                        for (int u = 0; u < PCG_POLL; u++) {
                            if (x0[u] == PCG_EMPTY) x0[u] = ld_relaxed(set + k0 + 32 * u + lane);
                            if (x1[u] == PCG_EMPTY) x1[u] = ld_relaxed(set + nb + k0 + 32 * u + lane);
                        }
#pragma unroll
                        for (int u = 0; u < PCG_POLL; u++) all = all && x0[u] != PCG_EMPTY && x1[u] != PCG_EMPTY;
                        if (!all && gave_up(spins)) ok = false;
                    }
#pragma unroll
                    for (int u = 0; u < PCG_POLL; u++) {
                        a0 += __longlong_as_double((long long)x0[u]);
                        a1 += __longlong_as_double((long long)x1[u]);
                    }
                }
                ok = __all_sync(0xffffffffu, ok);
                a0 = hsum32(a0);
                if (TWO) a1 = hsum32(a1);
                // each lane's fence after the slots that it read, then the warp's
                // barrier: what the blocks wrote before their totals is ordered
                // before lane 0's result (votes and shuffles order no memory)
                __threadfence();
                __syncwarp();
                if (lane == 0 && ok) {
                    if (a0 != a0) a0 = __longlong_as_double(0x7ff8000000000000ll);
                    if (a1 != a1) a1 = __longlong_as_double(0x7ff8000000000000ll);
                    st_relaxed(res, (unsigned long long)__double_as_longlong(a0));
                    if (TWO) st_relaxed(res + 1, (unsigned long long)__double_as_longlong(a1));
                }
            } else if (lane == 0) {
                unsigned long long x0 = PCG_EMPTY, x1 = TWO ? PCG_EMPTY : 0ull;
                for (unsigned spins = 0; ok; spins++) {
                    if (x0 == PCG_EMPTY) x0 = ld_relaxed(res);
                    if (TWO && x1 == PCG_EMPTY) x1 = ld_relaxed(res + 1);
                    if (x0 != PCG_EMPTY && x1 != PCG_EMPTY) break;
                    if (gave_up(spins)) ok = false;
                }
                a0 = __longlong_as_double((long long)x0);
                a1 = __longlong_as_double((long long)x1);
                __threadfence();
            }
            if (lane == 0) {
                // every block has left the sets before this one
                unsigned long long *old = slots + (size_t)((t + 2) % 3) * 2 * nb;
                st_relaxed(old + blockIdx.x, PCG_EMPTY);
                st_relaxed(old + nb + blockIdx.x, PCG_EMPTY);
                if (blockIdx.x == 0) {
                    unsigned long long *ro = slots + (size_t)6 * nb + 16 * ((t + 2) % 3);
                    st_relaxed(ro, PCG_EMPTY);
                    st_relaxed(ro + 1, PCG_EMPTY);
                }
                sh.sum = make_double2(a0, a1);
                sh.ok = ok;
            }
        }
        __syncthreads();
        out = sh.sum;
        return sh.ok != 0;
    }
}

// Entries k0 .. of row i (all of it, or what does not fit the registers)
// applied to the direction p = z + beta * pold, which is formed on the fly
// from the two vectors (final at this point), subtracted from acc.
__device__ __forceinline__ double pcg_row(int n, int i, const double *__restrict__ hval, const int *__restrict__ hcol,
                                          int c, int k0, const double *__restrict__ hbig_val,
                                          const int *__restrict__ hbig_col, const double *z, const double *pold,
                                          double beta, double acc)
{
    if (c >= 0) {
        for (int k = k0; k < c; k++) {
            const int j = hcol[(size_t)k * n + i];
            acc -= hval[(size_t)k * n + i] * (__ldcg(z + j) + beta * __ldcg(pold + j));
        }
    } else {
        const size_t base = (size_t)(-c - 1) * COT_HBIG_W;
        for (int k = 0; k < COT_HBIG_W; k++) {
            const int j = hbig_col[base + k];
            if (j < 0) break;
            acc -= hbig_val[base + k] * (__ldcg(z + j) + beta * __ldcg(pold + j));
        }
    }
    return acc;
}

// CL: the launch is one cluster.  R > 0: a thread owns R rows, with their
// vectors and first PCG_ROW matrix entries in registers; z and the direction
// are also written out for the neighbours.  R = 0: any number of rows.
template <bool CL, int R>
__global__ void __launch_bounds__(R > 0 ? PCG_THREADS_R : PCG_THREADS)
    k_pcg(int n, const double *__restrict__ hval, const int *__restrict__ hcol, const int *__restrict__ hcnt,
          const double *__restrict__ hbig_val, const int *__restrict__ hbig_col, const double *__restrict__ hdiag,
          const double *__restrict__ b, double *x, double *r, double *z, double *pa, double *pb, double *q,
          double *slots_mem, PcgState *st, double rtol, int max_it)
{
    __shared__ PcgShared sh;
    unsigned long long *slots = reinterpret_cast<unsigned long long *>(slots_mem);
    const int stride = gridDim.x * blockDim.x;
    const int t0 = blockIdx.x * blockDim.x + threadIdx.x;
    int t = 0;
    double2 s2;
    // a cluster's blocks are all running before one writes to another
    if constexpr (CL) {
        asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
        asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
    }
    // mean of the right-hand side (the Jacobian's range is mean-free)
    double sb = 0.0;
    for (int i = t0; i < n; i += stride) sb += b[i];
    if (!pcg_reduce<CL, false>(sb, 0.0, s2, t++, sh, slots, st)) return;
    const double mean = s2.x / (double)n;
    double *pold = pa, *pnew = pb;
    int it = 0;
    double beta = 0.0, rz, rr, rr0;
    if constexpr (R > 0) {
        const int i0 = blockIdx.x * (R * blockDim.x) + threadIdx.x;
        double xo[R], ro[R], zo[R], po[R], qo[R], di[R], h[R][PCG_ROW];
        int c[R], j[R][PCG_ROW];
        double rz_l = 0.0, rr_l = 0.0;
#pragma unroll
        for (int a = 0; a < R; a++) {
            const int i = i0 + a * blockDim.x;
            const bool row = i < n;
            di[a] = row && hdiag[i] > 0.0 ? hdiag[i] : 1.0;  // an empty cell's row is zero and keeps a unit diagonal
            c[a] = row ? hcnt[i] : 0;
            ro[a] = row ? b[i] - mean : 0.0;
            zo[a] = ro[a] / di[a];
            xo[a] = po[a] = qo[a] = 0.0;
#pragma unroll
            for (int k = 0; k < PCG_ROW; k++) {
                j[a][k] = k < c[a] ? hcol[(size_t)k * n + i] : -1;
                h[a][k] = k < c[a] ? hval[(size_t)k * n + i] : 0.0;
            }
            if (row) {
                z[i] = zo[a];
                pa[i] = 0.0;
            }
            rz_l += ro[a] * zo[a];
            rr_l += ro[a] * ro[a];
        }
        if (!pcg_reduce<CL, true>(rz_l, rr_l, s2, t++, sh, slots, st)) return;
        rz = s2.x;
        rr = rr0 = s2.y;
        const double stop = rtol * rtol * rr0;
        while (it < max_it && rr > stop && rz > 0.0) {
            // p = z + beta pold; q = J p; partial p.q
            double pq_l = 0.0;
#pragma unroll
            for (int a = 0; a < R; a++) {
                const int i = i0 + a * blockDim.x;
                double zj[PCG_ROW], pj[PCG_ROW];
#pragma unroll
                for (int k = 0; k < PCG_ROW; k++) {
                    zj[k] = j[a][k] >= 0 ? __ldcg(z + j[a][k]) : 0.0;
                    pj[k] = j[a][k] >= 0 ? __ldcg(pold + j[a][k]) : 0.0;
                }
                po[a] = zo[a] + beta * po[a];
                if (i < n) pnew[i] = po[a];
                double acc = di[a] * po[a];
#pragma unroll
                for (int k = 0; k < PCG_ROW; k++) acc -= h[a][k] * (zj[k] + beta * pj[k]);
                if (c[a] > PCG_ROW || c[a] < 0)
                    acc = pcg_row(n, i, hval, hcol, c[a], PCG_ROW, hbig_val, hbig_col, z, pold, beta, acc);
                qo[a] = acc;
                pq_l += po[a] * acc;
            }
            if (!pcg_reduce<CL, false>(pq_l, 0.0, s2, t++, sh, slots, st)) return;
            const double pq = s2.x;
            if (!(pq > 0.0)) break;
            const double alpha = rz / pq;
            double rz2_l = 0.0, rr2_l = 0.0;
#pragma unroll
            for (int a = 0; a < R; a++) {
                const int i = i0 + a * blockDim.x;
                xo[a] += alpha * po[a];
                ro[a] -= alpha * qo[a];
                zo[a] = ro[a] / di[a];
                if (i < n) z[i] = zo[a];
                rz2_l += ro[a] * zo[a];
                rr2_l += ro[a] * ro[a];
            }
            if (!pcg_reduce<CL, true>(rz2_l, rr2_l, s2, t++, sh, slots, st)) return;
            beta = s2.x / rz;
            rz = s2.x;
            rr = s2.y;
            double *tp = pold;
            pold = pnew;
            pnew = tp;
            it++;
        }
#pragma unroll
        for (int a = 0; a < R; a++) {
            const int i = i0 + a * blockDim.x;
            if (i < n) x[i] = xo[a];
        }
    } else {
        double rz_l = 0.0, rr_l = 0.0;
        for (int i = t0; i < n; i += stride) {
            const double ri = b[i] - mean;
            const double di = hdiag[i] > 0.0 ? hdiag[i] : 1.0;
            const double zi = ri / di;
            r[i] = ri;
            z[i] = zi;
            x[i] = 0.0;
            pa[i] = 0.0;
            rz_l += ri * zi;
            rr_l += ri * ri;
        }
        if (!pcg_reduce<CL, true>(rz_l, rr_l, s2, t++, sh, slots, st)) return;
        rz = s2.x;
        rr = rr0 = s2.y;
        const double stop = rtol * rtol * rr0;
        while (it < max_it && rr > stop && rz > 0.0) {
            double pq_l = 0.0;
            for (int i = t0; i < n; i += stride) {
                const double di = hdiag[i] > 0.0 ? hdiag[i] : 1.0;
                const double pi = z[i] + beta * pold[i];
                pnew[i] = pi;
                const double qi = pcg_row(n, i, hval, hcol, hcnt[i], 0, hbig_val, hbig_col, z, pold, beta, di * pi);
                q[i] = qi;
                pq_l += pi * qi;
            }
            if (!pcg_reduce<CL, false>(pq_l, 0.0, s2, t++, sh, slots, st)) return;
            const double pq = s2.x;
            if (!(pq > 0.0)) break;
            const double alpha = rz / pq;
            double rz2_l = 0.0, rr2_l = 0.0;
            for (int i = t0; i < n; i += stride) {
                const double di = hdiag[i] > 0.0 ? hdiag[i] : 1.0;
                x[i] += alpha * pnew[i];
                const double ri = r[i] - alpha * q[i];
                const double zi = ri / di;
                r[i] = ri;
                z[i] = zi;
                rz2_l += ri * zi;
                rr2_l += ri * ri;
            }
            if (!pcg_reduce<CL, true>(rz2_l, rr2_l, s2, t++, sh, slots, st)) return;
            beta = s2.x / rz;
            rz = s2.x;
            rr = s2.y;
            double *tp = pold;
            pold = pnew;
            pnew = tp;
            it++;
        }
    }
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        st->iterations = it;
        st->rr0 = rr0;
        st->rr = rr;
    }
}

int pcg_max_blocks(int n, int num_sms)
{
    // one block per SM at most (the kernels' registers allow one), so that
    // every block of a cooperative launch is resident
    const int want = (n + PCG_THREADS_R - 1) / PCG_THREADS_R;
    return std::max(1, std::min(want, num_sms));
}

// Whether the device takes a cluster of this launch.
static bool pcg_cluster_fits(const void *kernel, const cudaLaunchConfig_t &cfg)
{
    int clusters = 0;
    bool ok = cudaFuncSetAttribute(kernel, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) == cudaSuccess;
    ok = ok && cudaOccupancyMaxActiveClusters(&clusters, kernel, &cfg) == cudaSuccess && clusters > 0;
    if (!ok) cudaGetLastError();
    return ok;
}

cudaError_t launch_pcg(int n, const double *hval, const int *hcol, const int *hcnt, const double *hbig_val,
                       const int *hbig_col, const double *hdiag, const double *b, double *x, double *r, double *z,
                       double *pa, double *pb, double *q, double *partials, PcgState *st, double rtol, int max_it,
                       int blocks, CotCtx &c)
{
    void *args[] = {&n, &hval, &hcol, &hcnt, &hbig_val, &hbig_col, &hdiag, &b, &x, &r, &z, &pa, &pb, &q,
                    &partials, &st, &rtol, &max_it};
    c.launches++;
    const int want = (n + PCG_THREADS_R - 1) / PCG_THREADS_R;  // blocks of a row a thread
    if (n <= PCG_CLUSTER_ROWS) {
        const int cb = std::min(want, PCG_MAX_CLUSTER), rows = (want + cb - 1) / cb;
        const void *kernel = rows == 1 ? (const void *)k_pcg<true, 1>
                                       : (rows == 2 ? (const void *)k_pcg<true, 2> : (const void *)k_pcg<true, 4>);
        cudaLaunchConfig_t cfg = {};
        cudaLaunchAttribute at[1];
        at[0].id = cudaLaunchAttributeClusterDimension;
        at[0].val.clusterDim.x = (unsigned)cb;
        at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
        cfg.gridDim = dim3((unsigned)cb);
        cfg.blockDim = dim3(PCG_THREADS_R);
        cfg.stream = c.s;
        cfg.attrs = at;
        cfg.numAttrs = 1;
        if (pcg_cluster_fits(kernel, cfg)) return cudaLaunchKernelExC(&cfg, kernel, args);
    }
    const int rows = (want + blocks - 1) / blocks;
    const void *kernel = rows == 1   ? (const void *)k_pcg<false, 1>
                         : rows == 2 ? (const void *)k_pcg<false, 2>
                         : rows <= 4 ? (const void *)k_pcg<false, 4>
                                     : (const void *)k_pcg<false, 0>;
    cudaError_t e = cudaMemsetAsync(partials, 0xff, (size_t)PCG_SLOTS(blocks) * sizeof(double), c.s);
    if (e != cudaSuccess) return e;
    return cudaLaunchCooperativeKernel(kernel, dim3(blocks), dim3(rows <= 4 ? PCG_THREADS_R : PCG_THREADS), args, 0, c.s);
}

}  // namespace cot
