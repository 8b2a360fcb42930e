// cufsp_bdf_step.cu -- one step attempt of the BDF integrator (cufsp_bdf.cu) as ONE persistent launch,
// for generators whose slices fit the CTAs' registers and shared memory (up to 148 x 1056 = 156,288 states).
//
// The launch sequence spends a step on some 60 launches and 8 waits of the host for scalars: 344 us a step
// on the 131,072-state gene model (5.4 GMRES iterations), nearly all of it launch and round-trip latency.
// Here one cooperative grid runs the whole attempt -- prediction, right-hand side, GMRES with
// re-orthogonalisation, error test, update of the difference history and weights -- and the host reads
// one small block.  Same arithmetic as the sequence, in another summation order; two things are arranged
// differently:
//  * the residual is published before its norm beta is known, and A r / beta stands for A V_0;
//  * (I - c A) V_j is V_j plus q = -c A V_j, so q alone is orthogonalised and 1 is added to its coefficient
//    h_j: what is left of q is not a small difference from V_j;
//  * the norm of q travels with the dots h = V^T q, and ||q - V h||^2 = ||q||^2 - ||h||^2 (V is orthonormal
//    to rounding).  A second orthogonalisation pass follows only where the first has taken more than
//    three quarters of ||q||^2, the criterion of Daniel, Gragg, Kaufman and Stewart (Math. Comp. 30, 1976)
//    with eta = 1/2: above it one pass leaves V orthonormal to rounding, and the difference of squares
//    keeps its digits.  Where the second pass, too, takes that much, the norm is summed explicitly.
// Each CTA owns a slice of the states (cufsp_slice.cuh): generator coefficients, weights and the vector
// being orthogonalised in registers, the basis in shared memory (what does not fit is read from the
// published vectors in L2).  An extra warp collects totals and runs the Givens rotations beside the
// update.  What bounds it is the chain of exchanges, two and one gather per iteration (cufsp_grid.cuh).
// Measured on the 131,072-state gene model to t = 6 (315 steps): 0.34 ms a step with the launch
// sequence, 0.088 ms so.
// The coefficients c_r(t_new): tables of unit propensities, gain and outflow, are built once per
// generator, a table of the terms' coefficients from them for the reactions with constant rates; the
// launch adds the reactions whose rates have changed.  Waits are bounded; on expiry the error word is set and every CTA leaves.
#include <algorithm>
#include <atomic>
#include <chrono>
#include <climits>
#include <cmath>
#include <cstdlib>
#include <cstring>
#include <mutex>

#include "cufsp_bdf_step.h"
#include "cufsp_grid.cuh"
#include "cufsp_slice.cuh"

namespace cufsp {
namespace {

// 11 warps that own states, up to three per thread, and one for control: 168 registers a thread, what
// 12 warps can have.  The dots are taken by the first 2^kLog warps.
constexpr int kThreads = 352, kLog = 3, kWarps = kThreads / 32;
constexpr int kCtaStates = 256;  // a CTA per so many states, up to one per SM
constexpr int kMaxR = 32;
constexpr int kMaxL = 60;

struct StepArgs {
    SliceTerms terms;
    int chunk, slots, maxl;
    int nr, diag;                     // diag: near term of the outflow
    short term[kMaxR];                // reaction's term: near t, n_near + far t, -1: none
    double coef[kMaxR];
    const double *gain, *out;         // unit propensities [nr][n]: at the source state (0 outside), at the state
    const double *base;               // [n_near + n_far][n] coefficients of the reactions not in var
    int n_var;
    short var[kMaxR];
    double *D[kBdfHist], *w;
    int k;
    double g[kBdfOrder + 1], inv_alpha, c, econst, atol, rtol, sqrt_n, eps_lin;
    double *X, *X_clear;              // published vectors of this launch (all unset): y_pred, r, V_1 ..
    int n_clear;                      // vectors and exchange rows the launch before has used
    int rows_clear;
    double *ex, *ex_clear;
    int ex_rows;
    double *h_out;                    // report block (pinned host or device memory) and its sequence word
    unsigned *h_seq, seq;
    Waits waits;
};

struct StepSmem {
    double part[16][4];
    double wsum[2][kWarps];
    double h1[kMaxL + 2], h2[kMaxL + 2], col[kMaxL + 2];
    double cs[kMaxL], sn[kMaxL], gv[kMaxL + 2], y[kMaxL + 2];
    double beta, hn, inv, err;
    int conv, more;
};

// The owners' part of an exchange, by the compute warps but the first, which publishes.
__device__ __forceinline__ bool own(double *ex, int ex_rows, int row, int rows, const Waits &waits) {
    return threadIdx.x >= kThreads || exchange_own(ex, ex_rows, row, rows, 1, kWarps, false, waits);
}

template <int NS, int TN, int TF>
__global__ void __launch_bounds__(kThreads + 32, 1) k_bdf_step(const __grid_constant__ StepArgs a) {
    extern __shared__ __align__(16) double ws[];  // [chunk] | [halo][chunk][halo] | [slots][chunk] | packed R of GMRES
    __shared__ __align__(16) StepSmem sm;
    constexpr int NT = kThreads;
    const int n = a.terms.n, lo = (int)blockIdx.x * a.chunk, len = min(a.chunk, n - lo);
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const bool work = tid < NT;               // else: the control warp
    const int hi = work ? len : 0;            // bound of the state loops
    double *const xs = ws + a.chunk + a.terms.halo;
    double *const slot0 = xs + a.chunk + a.terms.halo;
    double *const R = slot0 + a.slots * a.chunk;  // column j at R + j (j + 1) / 2
    const int G = (int)gridDim.x, pitch = exchange_pitch(G);
    const int gt = (int)blockIdx.x * (NT + 32) + tid, gn = G * (NT + 32);
    int row = 0;

#pragma unroll 1
    for (int p = gt; p < a.rows_clear * pitch; p += gn) a.ex_clear[p] = unset_value();
#pragma unroll 1
    for (int p = gt; p < a.rows_clear * kCopies; p += gn)
        a.ex_clear[(size_t)a.ex_rows * pitch + (size_t)(p % kCopies) * a.ex_rows + p / kCopies] = unset_value();
#pragma unroll 1
    for (long long p = gt; p < (long long)a.n_clear * n; p += gn) a.X_clear[p] = unset_value();
    // coefficients: the base table, and the reactions whose rates have changed since it was built (summed
    // through shared memory: registers need constant indices)
    double cn[NS][TN], cf[NS][TF], w2[NS];
    if (work && a.n_var > 0) {
#pragma unroll 1
        for (int e = 0; e < (a.terms.n_near + a.terms.n_far) * NS; ++e) ws[e * NT + tid] = 0.0;
#pragma unroll 1
        for (int v = 0; v < a.n_var; ++v) {
            const int r = a.var[v], t = max(0, (int)a.term[r]);
            const double c = a.coef[r], cg = a.term[r] >= 0 ? c : 0.0;
            double g[NS], o[NS];
#pragma unroll
            for (int s = 0; s < NS; ++s) {
                const size_t i = (size_t)r * n + lo + (tid + s * NT < hi ? tid + s * NT : 0);
                g[s] = __ldcg(a.gain + i);
                o[s] = __ldcg(a.out + i);
            }
#pragma unroll
            for (int s = 0; s < NS; ++s) {
                ws[(t * NS + s) * NT + tid] += cg * g[s];
                ws[(a.diag * NS + s) * NT + tid] -= c * o[s];
            }
        }
    }
#pragma unroll
    for (int s = 0; s < NS; ++s) {
        const int il = tid + s * NT;
        const bool in = il < hi;
        const double *const p = a.base + lo + (in ? il : 0);
        const double wi = in ? __ldcg(a.w + lo + il) : 0.0;
        w2[s] = wi * wi;
#pragma unroll
        for (int t = 0; t < TN; ++t) cn[s][t] = in && t < a.terms.n_near ? __ldcg(p + (size_t)t * n) : 0.0;
#pragma unroll
        for (int t = 0; t < TF; ++t)
            cf[s][t] = in && t < a.terms.n_far ? __ldcg(p + (size_t)(a.terms.n_near + t) * n) : 0.0;
    }
    if (work && a.n_var > 0) {
#pragma unroll
        for (int s = 0; s < NS; ++s) {
            if (tid + s * NT < hi) {
#pragma unroll
                for (int t = 0; t < TN; ++t)
                    if (t < a.terms.n_near) cn[s][t] += ws[(t * NS + s) * NT + tid];
#pragma unroll
                for (int t = 0; t < TF; ++t)
                    if (t < a.terms.n_far) cf[s][t] += ws[((a.terms.n_near + t) * NS + s) * NT + tid];
            }
        }
    }
    __syncthreads();
#pragma unroll 1
    for (int r = warp; r <= a.slots; r += kWarps + 1)  // the last CTA's padding
        for (int il = len + lane; il < a.chunk; il += 32) (r ? slot0 + (r - 1) * a.chunk : ws)[il] = 0.0;
    __syncthreads();
    // y_pred = sum_{j<=k} D_j to the neighbours;  ws = -(sum_{1<=j<=k} gamma_j D_j) / alpha
#pragma unroll 1
    for (int il = tid; il < hi; il += NT) {
        double yp = 0.0, ps = 0.0;
#pragma unroll
        for (int j = 0; j <= kBdfOrder; ++j)
            if (j <= a.k) {
                const double dj = __ldcg(a.D[j] + lo + il);
                yp += dj;
                if (j >= 1) ps = fma(a.g[j], dj, ps);
            }
        xs[il] = yp;
        st_relaxed(a.X + lo + il, settled(yp));
        ws[il] = -ps * a.inv_alpha;
    }
    __syncthreads();

    // report to the host (one thread of CTA 0)
    auto report = [&](int status, int iters, double err, double em, double ep) {
        a.h_out[0] = status;
        a.h_out[1] = iters;
        a.h_out[2] = err;
        a.h_out[3] = em;
        a.h_out[4] = ep;
        a.h_out[5] = row;
        __threadfence_system();
        *(volatile unsigned *)a.h_seq = a.seq;
    };
    const bool teller = blockIdx.x == 0 && tid == NT;
    bool bad = false;
    // sum over the block's warps of v, left in slot `at` of wsum
    auto block_part = [&](int at, double v) {
        v = warp_sum(v);
        if (work && lane == 0) sm.wsum[at][warp] = v;
    };
    auto publish_part = [&](int at, int r) {  // by the control warp
        const double v = warp_sum(lane < kWarps ? sm.wsum[at][lane] : 0.0);
        if (lane == 0) st_relaxed(a.ex + (size_t)(row + r) * pitch + blockIdx.x, settled(v));
    };
    double q[NS], acc = 0.0, scale = 1.0;
    int J = -1;  // -1: the right-hand side r = c A y_pred + ws
#pragma unroll 1
    for (;;) {
        const int K = J + 1, Kres = min(K, a.slots);
        const double *const x = a.X + (size_t)K * n;
        const double *const gb = a.X + n + lo;  // V_r at gb + r n (r >= 1)
        acc = 0.0;
        {
            double v[NS][TF];
            if (work) bad = !gather_begin<NT, NS, TF, true>(a.terms, x, lo, len, true, xs, v, a.waits);
            if (work && !gather_end<NT, NS, TN, TF>(a.terms, x, lo, len, true, xs, cn, cf, v, q, a.waits)) bad = true;
        }
        if (J < 0) {
            if (__syncthreads_or(bad)) return;
#pragma unroll
            for (int s = 0; s < NS; ++s) {
                const int il = tid + s * NT;
                if (il < hi) {
                    q[s] = fma(a.c, q[s], ws[il]);
                    xs[il] = q[s];
                    st_relaxed(a.X + n + lo + il, settled(q[s]));
                    acc = fma(q[s] * q[s], w2[s], acc);
                }
            }
            block_part(0, acc);
            __syncthreads();
            if (!work) publish_part(0, 0);
            if (!own(a.ex, a.ex_rows, row, 1, a.waits)) bad = true;
            if (!work) {
                double v;
                if (!exchange_total(a.ex, a.ex_rows, row, 0, a.waits, v)) bad = true;
                sm.beta = sqrt(v);
                sm.inv = 1.0 / sm.beta;
                sm.gv[0] = sm.beta;
                sm.conv = 0;
            }
            row += 1;
            if (__syncthreads_or(bad)) return;
            const double beta = sm.beta;
            if (!isfinite(beta)) {
                if (teller) report(kBdfRhsNonfinite, 0, 0.0, 0.0, 0.0);
                return;
            }
            J = 0;
            if (beta <= a.eps_lin) break;  // d = 0
            scale = sm.inv;  // of the published vector: V_0 = r / beta
#pragma unroll
            for (int s = 0; s < NS; ++s) {
                const int il = tid + s * NT;
                if (il < hi) slot0[il] = q[s] * scale;
            }
            continue;
        }
        {
#pragma unroll
            for (int s = 0; s < NS; ++s) {  // q = -c A V_J; the V_J of (I - c A) V_J goes into its coefficient
                const int il = tid + s * NT;
                if (il < hi) {
                    q[s] *= -a.c * scale;
                    ws[il] = q[s] * w2[s];
                    acc = fma(q[s] * q[s], w2[s], acc);
                }
            }
            block_part(0, acc);
            scale = 1.0;
            if (__syncthreads_or(bad)) return;
            double *const mine = a.ex + blockIdx.x;
#pragma unroll 1
            for (int pass = 0;; ++pass) {  // h = V^T q, q -= V h
                double *const h = pass ? sm.h2 : sm.h1;
                if (work) slice_dots<kLog>(ws, a.chunk, len, K, Kres, slot0, gb, gb, n, sm.part);
                else publish_part(0, K);
                __syncthreads();
                if (tid < K) st_relaxed(mine + (size_t)(row + tid) * pitch, settled(dots_sum<kLog>(sm.part, K, tid)));
                if (!own(a.ex, a.ex_rows, row, K + 1, a.waits)) bad = true;
                if (!work) {
                    double s2 = 0.0, v = 0.0;
#pragma unroll 1
                    for (int r = lane; r <= K; r += 32) {
                        double u;
                        if (!exchange_total(a.ex, a.ex_rows, row, r, a.waits, u)) bad = true;
                        if (r == K) {
                            v = u;
                        } else {
                            h[r] = u;
                            if (pass == 0) sm.h2[r] = 0.0;
                            s2 = fma(u, u, s2);
                        }
                    }
                    v = __shfl_sync(0xffffffffu, v, K & 31);
                    s2 = warp_sum(s2);
                    sm.more = !(v - s2 >= 0.25 * v);  // also for NaN
                    sm.hn = sqrt(v - s2);
                    sm.inv = 1.0 / sm.hn;
                }
                row += K + 1;
                if (__syncthreads_or(bad)) return;
                acc = 0.0;
                double u[NS];
                int off[NS];
#pragma unroll
                for (int s = 0; s < NS; ++s) {
                    u[s] = q[s];
                    off[s] = tid + s * NT < hi ? s * NT : 0;
                }
                if (tid < hi) {
#pragma unroll 2
                    for (int r = 0; r < Kres; ++r) {
                        const double hr = h[r];
                        const double *p = slot0 + r * a.chunk + tid;
#pragma unroll
                        for (int s = 0; s < NS; ++s) u[s] = fma(-hr, p[off[s]], u[s]);
                    }
#pragma unroll 1
                    for (int r = Kres; r < K; ++r) {
                        const double hr = h[r];
                        const double *p = gb + (size_t)r * n + tid;
#pragma unroll
                        for (int s = 0; s < NS; ++s) u[s] = fma(-hr, __ldcg(p + off[s]), u[s]);
                    }
                }
#pragma unroll
                for (int s = 0; s < NS; ++s) q[s] = u[s];
                if (pass == 1 || !sm.more) break;
#pragma unroll
                for (int s = 0; s < NS; ++s) {
                    const int il = tid + s * NT;
                    if (il < hi) {
                        ws[il] = q[s] * w2[s];
                        acc = fma(q[s] * q[s], w2[s], acc);
                    }
                }
                block_part(0, acc);
                __syncthreads();
            }
            if (sm.more) {  // the difference of squares would cancel: the norm itself
                acc = 0.0;
#pragma unroll
                for (int s = 0; s < NS; ++s)
                    if (tid + s * NT < hi) acc = fma(q[s] * q[s], w2[s], acc);
                block_part(1, acc);
                __syncthreads();
                if (!work) publish_part(1, 0);
                if (!own(a.ex, a.ex_rows, row, 1, a.waits)) bad = true;
                if (!work) {
                    double v;
                    if (!exchange_total(a.ex, a.ex_rows, row, 0, a.waits, v)) bad = true;
                    sm.hn = sqrt(v);
                    sm.inv = 1.0 / sm.hn;
                }
                row += 1;
                if (__syncthreads_or(bad)) return;
            }
            const double hn = sm.hn, inv = sm.inv;
            if (!isfinite(hn)) {
                if (teller) report(kBdfBasisNonfinite, J + 1, 0.0, 0.0, 0.0);
                return;
            }
            if (work) {  // V_{J+1} to its slot and to the neighbours
                const bool more = K < a.maxl;
                double *const sl = K < a.slots ? slot0 + K * a.chunk : nullptr;
#pragma unroll
                for (int s = 0; s < NS; ++s) {
                    const int il = tid + s * NT;
                    if (il < hi) {
                        const double v = settled(q[s] * inv);
                        if (more) st_relaxed(a.X + (size_t)(K + 1) * n + lo + il, v);
                        xs[il] = v;
                        if (sl) sl[il] = v;
                    }
                }
            } else {  // Givens rotations of column J
                for (int r = lane; r < K; r += 32) sm.col[r] = (sm.h1[r] + sm.h2[r]) + (r == J ? 1.0 : 0.0);
                __syncwarp();
                if (lane == 0) {
                    double *const Rj = R + J * (J + 1) / 2;
                    double u = sm.col[0];
#pragma unroll 1
                    for (int l = 0; l < J; ++l) {
                        const double b = sm.col[l + 1];
                        Rj[l] = sm.cs[l] * u + sm.sn[l] * b;
                        u = -sm.sn[l] * u + sm.cs[l] * b;
                    }
                    const double r = hypot(u, hn);
                    const double cs = r > 0.0 ? u / r : 1.0, sn = r > 0.0 ? hn / r : 0.0;
                    Rj[J] = r;
                    sm.cs[J] = cs;
                    sm.sn[J] = sn;
                    const double gn1 = -sn * sm.gv[J];
                    sm.gv[J] = cs * sm.gv[J];
                    sm.gv[J + 1] = gn1;
                    sm.conv = fabs(gn1) <= a.eps_lin || hn == 0.0;
                }
            }
            __syncthreads();
            ++J;
            if (sm.conv || J == a.maxl) break;
        }
    }
    if (J > 0) {
        if (!sm.conv) {
            if (teller) report(kBdfNotConverged, J, 0.0, 0.0, 0.0);
            return;
        }
        if (!work) {  // back substitution
#pragma unroll 1
            for (int i = J - 1; i >= 0; --i) {
                const double *const Ri = R + i * (i + 1) / 2;
                const double yi = sm.gv[i] / Ri[i];
                __syncwarp();
                for (int l = lane; l < i; l += 32) sm.gv[l] -= Ri[l] * yi;
                if (lane == 0) sm.y[i] = yi;
                __syncwarp();
            }
        }
        __syncthreads();
    }
    // d = V y in ws, and its weighted norm
    acc = 0.0;
#pragma unroll
    for (int s = 0; s < NS; ++s) {
        const int il = tid + s * NT;
        if (il < hi) {
            double d = 0.0;
#pragma unroll 2
            for (int r = 0; r < min(J, a.slots); ++r) d = fma(sm.y[r], slot0[r * a.chunk + il], d);
#pragma unroll 1
            for (int r = a.slots; r < J; ++r) d = fma(sm.y[r], __ldcg(a.X + (size_t)(r + 1) * n + lo + il), d);
            ws[il] = d;
            acc = fma(d * d, w2[s], acc);
        }
    }
    block_part(0, acc);
    __syncthreads();
    if (!work) publish_part(0, 0);
    if (!own(a.ex, a.ex_rows, row, 1, a.waits)) bad = true;
    if (!work) {
        double v;
        if (!exchange_total(a.ex, a.ex_rows, row, 0, a.waits, v)) bad = true;
        sm.err = a.econst * sqrt(v);
    }
    row += 1;
    if (__syncthreads_or(bad)) return;
    const double err = sm.err;
    if (!isfinite(err) || err > 1.0) {
        if (teller) report(isfinite(err) ? kBdfRejected : kBdfErrNonfinite, J, err, 0.0, 0.0);
        return;
    }
    // accepted: D_{k+2} = d - D_{k+1}, D_{k+1} = d, D_j += D_{j+1} (j = k..0); weights of the new D_0
    double am = 0.0, ap = 0.0;
    const int k = a.k;
#pragma unroll 1
    for (int il = tid; il < hi; il += NT) {
        double v[kBdfHist];
#pragma unroll
        for (int j = 0; j < kBdfHist; ++j) v[j] = j <= k + 1 ? __ldcg(a.D[j] + lo + il) : 0.0;
        const double di = ws[il];
        double top = 0.0;
#pragma unroll
        for (int j = 0; j < kBdfHist; ++j)
            if (j == k + 1) {
                top = di - v[j];
                v[j] = di;
            }
#pragma unroll
        for (int j = kBdfHist - 2; j >= 0; --j)
            if (j <= k) v[j] += v[j + 1];
        double dk = 0.0;
#pragma unroll
        for (int j = 0; j < kBdfHist; ++j) {
            if (j <= k + 1) a.D[j][lo + il] = v[j];
            if (j == k + 2) a.D[j][lo + il] = top;
            if (j == k) dk = v[j];
        }
        const double wi = 1.0 / ((a.atol + a.rtol * fabs(v[0])) * a.sqrt_n);
        a.w[lo + il] = wi;
        am = fma(dk * dk, wi * wi, am);
        ap = fma(top * top, wi * wi, ap);
    }
    block_part(0, am);
    block_part(1, ap);
    __syncthreads();
    if (!work) {
        publish_part(0, 0);
        publish_part(1, 1);
    }
    own(a.ex, a.ex_rows, row, 2, a.waits);
    if (blockIdx.x == 0 && !work) {
        double em, ep;
        const bool ok = exchange_total(a.ex, a.ex_rows, row, 0, a.waits, em) && exchange_total(a.ex, a.ex_rows, row, 1, a.waits, ep);
        row += 2;
        if (ok && teller) report(kBdfAccepted, J, err, sqrt(em), sqrt(ep));
    }
}

struct UnitArgs {
    int64_t n;
    int ns, nr, tab_stride;
    int dims[CUFSP_MAX_SPECIES], tab_off[CUFSP_MAX_SPECIES];
    const double *tables;  // [nr][tab_stride], or null
    const double *props;   // [nr][n] propensities, or null
    const int *nu;
    const int64_t *d;
    double *gain, *out;    // [nr][n]
};

// Unit-rate propensities of every reaction at the state's source (0 outside the box) and at the state.
// Reactions without net change cancel (both 0).
__global__ void k_unit_propensities(const UnitArgs b) {
    const int64_t stride = (int64_t)gridDim.x * blockDim.x;
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < b.n; i += stride) {
        int xs[CUFSP_MAX_SPECIES];
        int64_t rem = i;
        for (int s = 0; s < b.ns; ++s) {
            xs[s] = (int)(rem % b.dims[s]);
            rem /= b.dims[s];
        }
        for (int r = 0; r < b.nr; ++r) {
            const double *tr = b.tables ? b.tables + (size_t)r * b.tab_stride : nullptr;
            double here = 1.0, there = 1.0;
            bool in = true, moves = false;
            for (int s = 0; s < b.ns; ++s) {
                const int v = b.nu[r * b.ns + s], y = xs[s] - v;
                moves = moves || v != 0;
                in = in && y >= 0 && y < b.dims[s];
                if (tr) {
                    here *= tr[b.tab_off[s] + xs[s]];
                    if (in) there *= tr[b.tab_off[s] + y];
                }
            }
            if (!tr) {
                here = b.props[(size_t)r * b.n + i];
                there = in ? b.props[(size_t)r * b.n + i - b.d[r]] : 0.0;
            }
            b.out[(size_t)r * b.n + i] = moves ? here : 0.0;
            b.gain[(size_t)r * b.n + i] = moves && in ? there : 0.0;
        }
    }
}

struct BaseArgs {
    int64_t n;
    int nr, terms, diag;
    unsigned skip;          // reactions left out
    short term[kMaxR];
    double coef[kMaxR];
    const double *gain, *out;
    double *base;           // [terms][n]
};

// Term coefficients of the reactions outside `skip`.
__global__ void k_bdf_base(const BaseArgs b) {
    const int64_t stride = (int64_t)gridDim.x * blockDim.x;
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < b.n; i += stride)
        for (int t = 0; t < b.terms; ++t) {
            double v = 0.0;
            for (int r = 0; r < b.nr; ++r) {
                if (b.skip >> r & 1u) continue;
                if (b.term[r] == t) v = fma(b.coef[r], b.gain[(size_t)r * b.n + i], v);
                if (t == b.diag) v = fma(-b.coef[r], b.out[(size_t)r * b.n + i], v);
            }
            b.base[(size_t)t * b.n + i] = v;
        }
}

using StepKernel = void (*)(const StepArgs);
struct StepVariant {
    StepKernel kern;
    int states, near, far;
};
#define CUFSP_SV(NS, TN, TF) {k_bdf_step<NS, TN, TF>, kThreads * NS, TN, TF}
const StepVariant kVariants[] = {CUFSP_SV(1, 4, 2), CUFSP_SV(1, 10, 4), CUFSP_SV(1, 4, 8), CUFSP_SV(2, 4, 2), CUFSP_SV(2, 10, 4),
                                 CUFSP_SV(2, 4, 8), CUFSP_SV(3, 4, 2),  CUFSP_SV(3, 10, 4), CUFSP_SV(3, 4, 8)};
#undef CUFSP_SV

size_t step_smem_max() { return (size_t)device_info().max_smem_optin - sizeof(StepSmem) - 1024; }

cudaError_t step_smem_attribute() {  // once per device, for every variant (as in cufsp_arnoldi.cu)
    constexpr int kMaxDevices = 64;
    static std::mutex mu;
    static bool done[kMaxDevices] = {};
    static cudaError_t result[kMaxDevices] = {};
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    if (dev < 0 || dev >= kMaxDevices) return cudaErrorInvalidDevice;
    std::lock_guard<std::mutex> lk(mu);
    if (!done[dev]) {
        for (const StepVariant &v : kVariants)
            if (result[dev] == cudaSuccess)
                result[dev] = cudaFuncSetAttribute((const void *)v.kern, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                                   (int)step_smem_max());
        done[dev] = true;
    }
    return result[dev];
}

}  // namespace

struct BdfStepper {
    StepArgs a;
    const StepVariant *var = nullptr;
    int grid = 0;
    size_t smem = 0;
    double *d_units = nullptr;  // gain and outflow tables, then the base table
    double base_coef[kMaxR];    // rates in the base table
    unsigned varying = 0;       // reactions left out of it: their rates have changed before
    bool have_base = false;     // (the launch that followed its build has reported)
    double *d_X = nullptr;      // two sets of published vectors: a launch uses one and clears the other
    double *d_ex = nullptr;     // two exchange areas, likewise
    int *d_err = nullptr;
    int turn = 0, used_vecs = 0, used_rows = 0;  // of the last launch
    cudaStream_t last = nullptr;  // stream of the launches, unless they were on several (mixed)
    bool used = false, mixed = false;
    bool fresh = false;         // both sets are unset
    bool copied = false;        // the last report was copied, not polled
};

void bdf_stepper_new_rates(BdfStepper *B) {
    B->have_base = false;
    B->varying = 0;
}

void bdf_stepper_destroy(BdfStepper *B) {
    if (!B) return;
    for (void *p : {(void *)B->d_units, (void *)B->d_X, (void *)B->d_ex, (void *)B->d_err}) {
        if (B->used && !B->mixed) cache_free(p, B->last);
        else cache_free(p);
    }
    delete B;
}

std::string bdf_stepper_describe(const BdfStepper *B) {
    const StepArgs &a = B->a;
    return "one persistent launch per step attempt, " + std::to_string(B->grid) + " CTAs x " + std::to_string(kThreads + 32) +
           " threads, variant of " + std::to_string(B->var->states / kThreads) + " states per thread, " +
           std::to_string(B->var->near) + " near and " + std::to_string(B->var->far) + " far terms, " + std::to_string(a.slots) +
           " of " + std::to_string(a.maxl + 1) + " basis vectors in shared memory, " + std::to_string(a.n_var) +
           " rates added per launch, report " + (B->copied ? "copied" : "polled");
}

cufsp_status bdf_stepper_create(cufsp_mat *A, int maxl, cudaStream_t st, BdfStepper **out) {
    *out = nullptr;
    static const bool on = [] {
        const char *e = getenv("CUFSP_BDF_PERSISTENT");
        return !e || atoi(e) != 0;
    }();
    const ModelHost &m = A->model;
    const int ns = m.ns, nr = m.nr;
    const int64_t n = m.n;
    const int sms = std::min(device_info().sm_count, 64 * kMaxGridPairs);
    const bool kron = A->format == CUFSP_FORMAT_KRONECKER;
    if (!on || nr > kMaxR || maxl > kMaxL || n > (int64_t)sms * kVariants[8].states || (kron ? m.tables.empty() : !A->sparse))
        return CUFSP_SUCCESS;
    std::vector<int64_t> d(nr, 0), stride(ns, 1);
    for (int s = 1; s < ns; ++s) stride[s] = stride[s - 1] * ((int64_t)m.bounds[s - 1] + 1);
    for (int r = 0; r < nr; ++r)
        for (int s = 0; s < ns; ++s) d[r] += (int64_t)m.nu[(size_t)r * ns + s] * stride[s];
    // distinct shifts, the diagonal (0) first; a shift of n or more has no source in the box
    std::vector<int> shifts(1, 0);
    for (int r = 0; r < nr; ++r)
        if (d[r] != 0 && std::llabs(d[r]) < n && std::find(shifts.begin(), shifts.end(), (int)d[r]) == shifts.end())
            shifts.push_back((int)d[r]);
    BdfStepper *B = new BdfStepper();
    StepArgs &a = B->a;
    std::memset(&a, 0, sizeof(a));
    split_terms((int)shifts.size(), shifts.data(), a.terms);
    a.terms.n = (int)n;
    const int64_t want = std::max<int64_t>(1, std::min<int64_t>(sms, (n + kCtaStates - 1) / kCtaStates));
    a.chunk = (int)(((n + want - 1) / want + 1) & ~int64_t(1));
    B->grid = (int)((n + a.chunk - 1) / a.chunk);
    const StepVariant *var = nullptr;
    for (const StepVariant &v : kVariants)
        if (!var && a.chunk <= v.states && a.terms.n_near <= v.near && a.terms.n_far <= v.far) var = &v;
    if (!var) {
        delete B;
        return CUFSP_SUCCESS;
    }
    B->var = var;
    a.nr = nr;
    for (int r = 0; r < nr; ++r) {
        a.term[r] = -1;
        if (d[r] == 0) continue;
        for (int t = 0; t < a.terms.n_near; ++t)
            if (a.terms.near_shift[t] == d[r]) a.term[r] = (short)t;
        for (int t = 0; t < a.terms.n_far; ++t)
            if (a.terms.far_shift[t] == d[r]) a.term[r] = (short)(a.terms.n_near + t);
    }
    for (int t = 0; t < a.terms.n_near; ++t)
        if (a.terms.near_shift[t] == 0) a.diag = t;
    const size_t row = sizeof(double) * (size_t)a.chunk;
    const size_t fixed = 2 * row + sizeof(double) * (2 * kHaloMax + (size_t)maxl * (maxl + 1) / 2);
    a.maxl = maxl;
    a.slots = (int)std::min<size_t>(maxl + 1, (step_smem_max() - fixed) / row);
    const size_t coefs = sizeof(double) * (size_t)(shifts.size() * (var->states / kThreads) * kThreads);
    B->smem = std::max(fixed + row * (size_t)a.slots, coefs);
    a.ex_rows = 4;
    for (int j = 0; j < maxl; ++j) a.ex_rows += 2 * (j + 2) + 1;
    const size_t units = (size_t)nr * n, base = shifts.size() * (size_t)n, xbytes = sizeof(double) * 2 * (size_t)(maxl + 2) * n;
    const size_t ebytes = sizeof(double) * 2 * (size_t)exchange_doubles(a.ex_rows, B->grid);
    // the model's data for the unit tables, needed only while they are built
    double *d_tab = nullptr;
    int *d_nu = nullptr;
    int64_t *d_d = nullptr;
    const size_t tab = kron ? m.tables.size() : units;
    cudaError_t e = step_smem_attribute();
    if (e == cudaSuccess) e = cache_alloc((void **)&B->d_units, sizeof(double) * (2 * units + base));
    if (e == cudaSuccess) e = cache_alloc((void **)&B->d_X, xbytes);
    if (e == cudaSuccess) e = cache_alloc((void **)&B->d_ex, ebytes);
    if (e == cudaSuccess) e = cache_alloc((void **)&B->d_err, sizeof(int));
    if (e == cudaSuccess) e = cache_alloc((void **)&d_tab, sizeof(double) * tab);
    if (e == cudaSuccess) e = cache_alloc((void **)&d_nu, sizeof(int) * (size_t)nr * ns);
    if (e == cudaSuccess) e = cache_alloc((void **)&d_d, sizeof(int64_t) * nr);
    if (e == cudaSuccess) e = cudaMemcpyAsync(d_nu, m.nu.data(), sizeof(int) * (size_t)nr * ns, cudaMemcpyHostToDevice, st);
    if (e == cudaSuccess) e = cudaMemcpyAsync(d_d, d.data(), sizeof(int64_t) * nr, cudaMemcpyHostToDevice, st);
    if (e == cudaSuccess && kron) e = cudaMemcpyAsync(d_tab, m.tables.data(), sizeof(double) * tab, cudaMemcpyHostToDevice, st);
    cufsp_status s = CUFSP_SUCCESS;
    if (e == cudaSuccess && !kron) s = sparse_export(A->sparse, d_tab, st);
    if (e == cudaSuccess && s == CUFSP_SUCCESS) {
        UnitArgs u;
        std::memset(&u, 0, sizeof(u));
        u.n = n;
        u.ns = ns;
        u.nr = nr;
        u.tab_stride = m.tab_stride;
        for (int s = 0; s < ns; ++s) {
            u.dims[s] = m.bounds[s] + 1;
            u.tab_off[s] = m.tab_off.empty() ? 0 : m.tab_off[s];
        }
        (kron ? u.tables : u.props) = d_tab;
        u.nu = d_nu;
        u.d = d_d;
        u.gain = B->d_units;
        u.out = B->d_units + units;
        k_unit_propensities<<<stream_grid(n, 1, device_info().sm_count * 8), 256, 0, st>>>(u);
        e = cudaGetLastError();
    }
    // the uploads above read pageable host memory and the scratch goes back to the cache
    if (e == cudaSuccess) e = cudaStreamSynchronize(st);
    cache_free(d_tab, st);
    cache_free(d_nu, st);
    cache_free(d_d, st);
    int per_sm = 0;
    if (e == cudaSuccess)
        e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, (const void *)var->kern, kThreads + 32, B->smem);
    if (e != cudaSuccess || s != CUFSP_SUCCESS || per_sm < 1) {
        bdf_stepper_destroy(B);
        if (e != cudaSuccess && e != cudaErrorMemoryAllocation) return cuda_error(e, "cufsp_bdf: persistent step");
        cudaGetLastError();
        return s;
    }
    a.gain = B->d_units;
    a.out = B->d_units + units;
    a.base = B->d_units + 2 * units;
    B->used = true;  // the unit tables were built on st
    B->last = st;
    *out = B;
    return CUFSP_SUCCESS;
}

cufsp_status bdf_stepper_run(BdfStepper *B, const BdfStepIn &in, BdfStepOut &out, cudaStream_t st) {
    StepArgs &a = B->a;
    const size_t xset = (size_t)(a.maxl + 2) * a.terms.n, area = (size_t)exchange_doubles(a.ex_rows, B->grid);
    if (!B->fresh) {
        CUFSP_CUDA_TRY(cudaMemsetAsync(B->d_X, kUnsetByte, sizeof(double) * 2 * xset, st));
        CUFSP_CUDA_TRY(cudaMemsetAsync(B->d_ex, kUnsetByte, sizeof(double) * 2 * area, st));
        CUFSP_CUDA_TRY(cudaMemsetAsync(B->d_err, 0, sizeof(int), st));
        if (in.d_out) CUFSP_CUDA_TRY(cudaMemsetAsync(in.d_out, 0, sizeof(double) * (kBdfOutWords + 1), st));
        B->used_vecs = B->used_rows = 0;
        B->have_base = false;  // nor is the base table known to have been built
        B->varying = 0;
    }
    B->fresh = false;  // until the launch has reported
    for (int j = 0; j < kBdfHist; ++j) a.D[j] = in.D[j];
    a.w = in.w;
    a.k = in.k;
    for (int j = 0; j <= kBdfOrder; ++j) a.g[j] = in.g[j];
    a.inv_alpha = in.inv_alpha;
    a.c = in.c;
    a.econst = in.econst;
    a.atol = in.atol;
    a.rtol = in.rtol;
    a.sqrt_n = in.sqrt_n;
    a.eps_lin = in.eps_lin;
    // The base table holds the reactions whose rates have never changed; the others are added per launch.
    unsigned varying = B->varying;
    for (int r = 0; r < a.nr; ++r) {
        a.coef[r] = in.coefs[r];
        if (B->have_base && in.coefs[r] != B->base_coef[r]) varying |= 1u << r;
    }
    if (!B->have_base || varying != B->varying) {
        BaseArgs b;
        std::memset(&b, 0, sizeof(b));
        b.n = a.terms.n;
        b.nr = a.nr;
        b.terms = a.terms.n_near + a.terms.n_far;
        b.diag = a.diag;
        b.skip = B->varying = varying;
        std::copy(a.term, a.term + kMaxR, b.term);
        std::copy(a.coef, a.coef + kMaxR, b.coef);
        std::copy(a.coef, a.coef + kMaxR, B->base_coef);
        b.gain = a.gain;
        b.out = a.out;
        b.base = const_cast<double *>(a.base);
        k_bdf_base<<<stream_grid(b.n, 1, device_info().sm_count * 8), 256, 0, st>>>(b);
        CUFSP_CUDA_TRY(cudaGetLastError());
        B->have_base = true;
    }
    a.n_var = 0;
    for (int r = 0; r < a.nr; ++r)
        if (varying >> r & 1u) a.var[a.n_var++] = (short)r;
    a.X = B->d_X + (size_t)B->turn * xset;
    a.X_clear = B->d_X + (size_t)(1 - B->turn) * xset;
    a.ex = B->d_ex + (size_t)B->turn * area;
    a.ex_clear = B->d_ex + (size_t)(1 - B->turn) * area;
    a.n_clear = B->used_vecs;
    a.rows_clear = B->used_rows;
    a.h_out = in.d_out ? in.d_out : in.h_out;
    a.h_seq = in.d_out ? reinterpret_cast<unsigned *>(in.d_out + kBdfOutWords) : in.h_seq;
    a.seq = ++*in.seq;
    a.waits = launch_waits(B->d_err);
    B->copied = in.d_out != nullptr;
    if (B->last != st) B->mixed = true;
    B->last = st;
    void *args[] = {&a};
    CUFSP_CUDA_TRY(cudaLaunchCooperativeKernel((const void *)B->var->kern, dim3(B->grid), dim3(kThreads + 32), args, B->smem, st));
    const volatile unsigned *seq = in.h_seq;
    if (in.d_out) {
        CUFSP_CUDA_TRY(cudaMemcpyAsync(in.h_out, in.d_out, sizeof(double) * (kBdfOutWords + 1), cudaMemcpyDeviceToHost, st));
        CUFSP_CUDA_TRY(cudaStreamSynchronize(st));
        seq = reinterpret_cast<unsigned *>(in.h_out + kBdfOutWords);
    }
    // bounded poll of the report, as the integrator's scalar reads
    const auto t0 = std::chrono::steady_clock::now();
    for (unsigned it = 1; *seq != a.seq; ++it) {
        if ((it & 1023) == 0) {
            if (cudaStreamQuery(st) != cudaErrorNotReady) break;
            if (std::chrono::steady_clock::now() - t0 > std::chrono::seconds(10)) break;
        }
    }
    if (*seq != a.seq) {
        CUFSP_CUDA_TRY(cudaStreamSynchronize(st));
        if (*seq != a.seq)
            return set_error(CUFSP_ERR_CUDA, "cufsp_bdf: a wait between the CTAs of a persistent step expired");
    }
    std::atomic_thread_fence(std::memory_order_acquire);
    out.status = (int)in.h_out[0];
    out.iters = (int)in.h_out[1];
    out.err = in.h_out[2];
    out.em = in.h_out[3];
    out.ep = in.h_out[4];
    B->used_rows = (int)in.h_out[5];
    B->used_vecs = std::min(a.maxl + 2, out.iters + 2);
    B->turn = 1 - B->turn;
    B->fresh = true;
    return CUFSP_SUCCESS;
}

}  // namespace cufsp
