// cufsp_batch.cuh -- batched adaptive Krylov exp(tA)p over many FSP instances in ONE persistent launch.
//
// The single-instance Krylov driver (cufsp_krylov.cu, replacing cuFSP::KryExpvFSP,
// src/KryExpvFSP.cu:38-188) runs its step control on the host, one synchronisation per step.  Here
// every part of the solve runs on the device, for hundreds of instances of one reaction network that
// differ in their box (truncation bounds), their factor tables and their rate coefficients:
//  * Work split: the grid is a set of thread-block clusters; each cluster takes instances from a
//    global work counter (largest first) and solves one instance at a time with all its CTAs.  The
//    cluster's CTAs split the instance's states into contiguous chunks.
//  * Reductions (norms, the Gram-Schmidt dots) go through distributed shared memory: every CTA
//    writes its partial sums, one cluster barrier (barrier.cluster: hardware, no spinning), then
//    every CTA sums the partials of all CTAs in rank order -- identical, deterministic results in all
//    CTAs, so every CTA holds the same Hessenberg matrix and takes the same step-control decisions
//    without further communication.
//  * Per Arnoldi iteration, over the own chunk: the generator action w = rho_j A W_j, the dots of w against
//    the basis, a cluster reduction, the update w -= V h fused with ||w||^2, a second cluster reduction.  The basis is stored unnormalised (v_k = rho_k W_k) as in the
//    single-instance driver.
//  * The small (m+2)^2 exponential is Pade(13,13) with scaling and squaring (Higham 2005, the same
//    algorithm as the host path cufsp_expm.cpp), computed by every CTA in its shared memory; the
//    Expokit step control (delta = 1.2, gamma = 0.9, phi1/phi2 estimate, 2-significant-digit
//    rounding, first-step formula) follows the host driver.
//  * Every loop is bounded (max steps and rejections per instance); an instance that exhausts them
//    or meets NaN/Inf gets an error status and the cluster moves on.  There are no spin waits.
//
// This file is compiled by NVRTC per reaction network (cufsp_batch.cu writes the prefix): species and
// reaction counts, the Krylov dimension M, the threads per CTA, and per reaction and species the net
// change nu(r, s) and the factor kind(r, s) (0: f = 1, 1: f(x) = x, 2: table lookup) are constants.

#ifndef CUFSP_BATCH_CUH
#define CUFSP_BATCH_CUH

#define CUFSP_BATCH_MAXS 8
#define CUFSP_BATCH_MAXR 32

struct CufspBatchDiv {  // unsigned division by a runtime constant d (round-up multiplier method)
    unsigned d, mul, shift;
};

struct CufspBatchInst {
    long long off;       // offset of the instance's vector in the packed array
    long long tab;       // offset of its factor tables in the packed table array
    int n;               // states
    int tab_stride;      // sum_s (b_s + 1)
    int dims[CUFSP_BATCH_MAXS];
    int tab_off[CUFSP_BATCH_MAXS];
    int delta[CUFSP_BATCH_MAXR];  // flat shift of reaction r: sum_s nu_{r,s} stride_s
    CufspBatchDiv div[CUFSP_BATCH_MAXS];
    double coef[CUFSP_BATCH_MAXR];
};

struct CufspBatchStat {
    double t;            // time reached
    double err;          // last local error estimate
    int steps, rejects, matvecs, status;  // status: 0 ok, 1 step limit, 2 NaN/Inf
};

struct CufspBatchArgs {
    const CufspBatchInst *inst;
    const int *order;        // processing order (largest instances first)
    const double *tables;    // packed factor tables
    double *p;               // packed state vectors (in: p(0), out: p(t_final))
    double *work;            // per-cluster basis workspace, work_stride doubles each
    long long work_stride;   // >= (M + 1) ld_max, and the cluster's tables where they are not in shared memory; even
    unsigned *counter;       // work counter (zero before the launch)
    CufspBatchStat *stats;   // per instance
    int n_inst;
    int ld_max;              // longest basis vector (even)
    int max_steps, max_reject;
    double t_final, tol, anorm;
};

#ifdef __CUDACC_RTC__

#include <cooperative_groups.h>
namespace cg = cooperative_groups;

namespace cufsp_batch {

constexpr int NS = CUFSP_BATCH_NS;
constexpr int NR = CUFSP_BATCH_NR;
constexpr int M = CUFSP_BATCH_M;          // Krylov dimension
constexpr int MP2 = M + 2;
constexpr int T = CUFSP_BATCH_THREADS;    // threads per CTA
constexpr int WARPS = T / 32;
constexpr int KR = M + 1;                 // most partial sums one reduction carries
constexpr bool IOP = CUFSP_BATCH_IOP != 0;
constexpr int QIOP = CUFSP_BATCH_QIOP;

// Generated: nu(r, s) and kind(r, s), constexpr functions of constant indices.

__device__ __forceinline__ unsigned fdiv(unsigned n, const CufspBatchDiv &f) {
    const unsigned t = __umulhi(n, f.mul);
    return (t + n) >> f.shift;
}

// ---- per-CTA shared state -------------------------------------------------------------------
struct Shared {
    double red[2][KR];          // this CTA's partial sums (double-buffered; read remotely)
    double warp_part[WARPS][KR];
    double tot[KR];             // cluster totals
    double H[MP2 * MP2];        // Hessenberg matrix (column-major), identical in every CTA
    double rho[MP2], gam[MP2 + 8];
    double pade[8][MP2 * MP2];  // exponential workspace
    double coefc[MP2 + 8];          // combination coefficients
    double dpiv[MP2], dinv[MP2];  // pivots of the exponential's LU and their inverses
    int piv[MP2];
    CufspBatchInst in;          // current instance
    int inst_idx;
    double sc[8];               // scalars broadcast inside the CTA
    int flag[4];
};

// Cluster-wide sum of one value per thread: every CTA ends with the total in s.tot[0].
__device__ __forceinline__ void cluster_sum1(cg::cluster_group &cl, Shared &s, double v, int &buf);

// ---- generator action from per-instance tables ----------------------------------------------------
// At the start of an instance the rates are written into tables (every CTA its own in shared memory when they
// fit beside the solver's state, else the cluster's CTAs one in its workspace): gain[r][s][x_s], the factor of reaction r at the
// source state x - nu_r, 0 where that leaves the box, with the rate in the first species' factor; and
// loss[s][x_s], the summed outflow of the reactions whose propensity depends on species s alone.  A state
// then needs no bounds tests, conversions or factor products of its own: 5 + 16 table reads for the
// 12-reaction gene network instead of about 300 instructions.
__device__ constexpr bool used(int r, int sp) { return kind(r, sp) != 0 || nu(r, sp) != 0; }
__device__ constexpr int first_used(int r) {
    for (int sp = 0; sp < NS; ++sp)
        if (used(r, sp)) return sp;
    return -1;
}
__device__ constexpr bool same_nu(int a, int b) {
    for (int sp = 0; sp < NS; ++sp)
        if (nu(a, sp) != nu(b, sp)) return false;
    return true;
}
__device__ constexpr int leader(int r) {  // first reaction with r's net change: they share the source entry
    for (int a = 0; a < r; ++a)
        if (same_nu(a, r)) return a;
    return r;
}
__device__ constexpr int own_species(int r) {  // the species r's propensity depends on; -1 none, -2 several
    int at = -1;
    for (int sp = 0; sp < NS; ++sp)
        if (kind(r, sp) != 0) at = at == -1 ? sp : -2;
    return at;
}

struct Tables {
    const double *gain;  // [NR][tab_stride]
    const double *loss;  // [tab_stride]
};

template <int R, int SP>
__device__ __forceinline__ double gain_factor(const CufspBatchInst &in, const Tables &t, const int (&x)[NS], double f) {
    if constexpr (SP < NS) {
        if constexpr (used(R, SP)) {
            const double g = t.gain[R * in.tab_stride + in.tab_off[SP] + x[SP]];
            f = SP == first_used(R) ? g : f * g;
        }
        return gain_factor<R, SP + 1>(in, t, x, f);
    }
    return f;
}

template <int R, int L>  // reactions R, R + 1, .. that share leader L's net change
__device__ __forceinline__ double gain_sum(const CufspBatchInst &in, const Tables &t, const int (&x)[NS]) {
    if constexpr (R < NR) {
        if constexpr (leader(R) == L) {
            const double f = first_used(R) < 0 ? in.coef[R] : gain_factor<R, 0>(in, t, x, 1.0);
            if constexpr (R + 1 < NR) return f + gain_sum<R + 1, L>(in, t, x);
            return f;
        } else {
            return gain_sum<R + 1, L>(in, t, x);
        }
    }
    return 0.0;
}

template <int R, int SP>
__device__ __forceinline__ double own_product(const CufspBatchInst &in, const double *__restrict__ tab, const int (&x)[NS],
                                              double f) {
    if constexpr (SP < NS) {
        if constexpr (kind(R, SP) == 1) f *= (double)x[SP];
        else if constexpr (kind(R, SP) == 2) f *= __ldg(tab + R * in.tab_stride + in.tab_off[SP] + x[SP]);
        return own_product<R, SP + 1>(in, tab, x, f);
    }
    return f;
}

template <int R>
__device__ __forceinline__ void accumulate(const CufspBatchInst &in, const Tables &t, const double *__restrict__ tab,
                                           const double *v, int i, const int (&x)[NS], double &acc, double &dg) {
    if constexpr (R < NR) {
        if constexpr (leader(R) == R)  // a source outside the box has gain 0; its index is kept in range
            acc = fma(gain_sum<R, R>(in, t, x), v[min(max(i - in.delta[R], 0), in.n - 1)], acc);
        if constexpr (own_species(R) == -1) dg += in.coef[R];
        if constexpr (own_species(R) == -2) dg += own_product<R, 0>(in, tab, x, in.coef[R]);
        accumulate<R + 1>(in, t, tab, v, i, x, acc, dg);
    }
}

// rho * (A v)[i]
__device__ __forceinline__ double apply_at(const CufspBatchInst &in, const Tables &t, const double *__restrict__ tab,
                                           const double *v, int i, double rho) {
    int x[NS];
    unsigned rem = (unsigned)i;
#pragma unroll
    for (int sp = 0; sp < NS - 1; ++sp) {
        const unsigned q = fdiv(rem, in.div[sp]);
        x[sp] = (int)(rem - q * (unsigned)in.dims[sp]);
        rem = q;
    }
    x[NS - 1] = (int)rem;
    double acc = 0.0, dg = 0.0;
#pragma unroll
    for (int sp = 0; sp < NS; ++sp) dg += t.loss[in.tab_off[sp] + x[sp]];
    accumulate<0>(in, t, tab, v, i, x, acc, dg);
    return rho * fma(-dg, v[i], acc);
}

template <int R, int SP>  // by threads `me` of `step`
__device__ __forceinline__ void fill_tables(const CufspBatchInst &in, const double *__restrict__ tab, double *gain,
                                            double *loss, int me, int step) {
    if constexpr (R < NR) {
        if constexpr (SP < NS) {
            const double *own = tab + R * in.tab_stride + in.tab_off[SP];
            for (int x = me; x < in.dims[SP]; x += step) {
                if constexpr (used(R, SP)) {
                    const int y = x - nu(R, SP);
                    double g = y < 0 || y >= in.dims[SP] ? 0.0 : kind(R, SP) == 0 ? 1.0 : __ldg(own + y);
                    if (SP == first_used(R)) g *= in.coef[R];
                    gain[R * in.tab_stride + in.tab_off[SP] + x] = g;
                }
                if constexpr (own_species(R) == SP) loss[in.tab_off[SP] + x] += in.coef[R] * __ldg(own + x);
            }
            fill_tables<R, SP + 1>(in, tab, gain, loss, me, step);
        } else {
            fill_tables<R + 1, 0>(in, tab, gain, loss, me, step);
        }
    }
}

// ---- a thread's states: pairs (i, i + 1), i even, 16 bytes a load -----------------------------------
// Every basis vector starts on a 16-byte boundary (stride rounded up to even), so a pass over the chunk
// keeps eight 16-byte loads per thread in flight: the passes over the basis are bound by how many bytes
// are on their way from L2 and HBM.  With 8-byte loads (and four at a time in the update) 48 gene models
// of 13K-113K states took 104 ms, so (and with the tables below) 63 ms.  The last state of an odd instance is a pair of one.
__device__ __forceinline__ double2 ld2(const double *p, bool two) {
    return two ? *reinterpret_cast<const double2 *>(p) : make_double2(*p, 0.0);
}
__device__ __forceinline__ void st2(double *p, double2 v, bool two) {
    if (two) *reinterpret_cast<double2 *>(p) = v;
    else *p = v.x;
}
template <int U, class F>  // U: pairs in flight per thread
__device__ __forceinline__ void for_pairs(int i0, int i1, F &&f) {  // f(i, two)
    int i = i0 + 2 * (int)threadIdx.x;
#pragma unroll U
    for (; i + 1 < i1; i += 2 * T) f(i, true);
    if (i < i1) f(i, false);
}
// the same from the end of the chunk
template <class F>
__device__ __forceinline__ void for_pairs_back(int i0, int i1, F &&f) {
    const int pairs = (i1 - i0 + 1) >> 1, first = (int)threadIdx.x;
    if (first >= pairs) return;
    int i = i0 + 2 * (first + (pairs - 1 - first) / T * T);
    if (i + 1 >= i1) {
        f(i, false);
        i -= 2 * T;
    }
#pragma unroll 1
    for (; i >= i0; i -= 2 * T) f(i, true);
}

// Warp partial sums of up to 8 values into s.warp_part[warp][k0 + k].
__device__ __forceinline__ void warp_partials8(Shared &s, const double (&acc)[8], int k0, int kused) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
    for (int k = 0; k < 8; ++k) {
        if (k0 + k < kused) {
            double v = acc[k];
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
            if (lane == 0) s.warp_part[warp][k0 + k] = v;
        }
    }
}

// CTA totals of s.warp_part[.][0..kused) into s.red[buf], one cluster barrier, then every CTA sums
// the partials of all CTAs in rank order into s.tot.
__device__ __forceinline__ void cluster_finish(cg::cluster_group &cl, Shared &s, int kused, int &buf) {
    __syncthreads();
    for (int k = threadIdx.x; k < kused; k += T) {
        double v = 0.0;
        for (int w = 0; w < WARPS; ++w) v += s.warp_part[w][k];
        s.red[buf][k] = v;
    }
    cl.sync();
    const int nb = (int)cl.num_blocks();
    for (int k = threadIdx.x; k < kused; k += T) {
        double v = 0.0;
        for (int b = 0; b < nb; ++b) v += cl.map_shared_rank(&s.red[buf][0], b)[k];
        s.tot[k] = v;
    }
    __syncthreads();
    buf ^= 1;
}

__device__ __forceinline__ void cluster_sum1(cg::cluster_group &cl, Shared &s, double v, int &buf) {
    double acc[8] = {v, 0.0, 0.0, 0.0, 0.0, 0.0, 0.0, 0.0};
    warp_partials8(s, acc, 0, 1);
    cluster_finish(cl, s, 1, buf);
}

// ---- small dense kernels for the (m+2)^2 exponential (column-major, k = MP2) -------------------
__device__ void mm(const double *A, const double *B, double *C) {  // C = A B, two columns per thread
    for (int e = threadIdx.x; e < MP2 * ((MP2 + 1) / 2); e += T) {
        const int i = e % MP2, j0 = e / MP2 * 2, j1 = min(j0 + 1, MP2 - 1);
        double c0 = 0.0, c1 = 0.0;
#pragma unroll 8
        for (int l = 0; l < MP2; ++l) {
            const double al = A[i + l * MP2];
            c0 = fma(al, B[l + j0 * MP2], c0);
            c1 = fma(al, B[l + j1 * MP2], c1);
        }
        C[i + j0 * MP2] = c0;
        C[i + j1 * MP2] = c1;
    }
    __syncthreads();
}

__device__ __forceinline__ double nan_value() { return __longlong_as_double(0x7ff8000000000000ll); }

// F = exp(A) by scaling and squaring Pade(13,13); false on NaN/Inf or a singular denominator.
// Workspace: s.pade[0..7]; A is read from s.pade[7] and F is left in s.pade[0].
__device__ __noinline__ bool expm_dev(Shared &s) {
    double *A = s.pade[7];
    double *B = s.pade[0], *B2 = s.pade[1], *B4 = s.pade[2], *B6 = s.pade[3], *Tm = s.pade[4], *U = s.pade[5],
           *V = s.pade[6];
    __shared__ double norm1;
    __shared__ int sq;
    if (threadIdx.x < 32) {  // 1-norm: a column per lane
        double nm = 0.0;
        bool nan = false;
        for (int j = threadIdx.x; j < MP2; j += 32) {
            double c = 0.0;
#pragma unroll 4
            for (int i = 0; i < MP2; ++i) c += fabs(A[i + j * MP2]);
            nan = nan || !isfinite(c);
            nm = fmax(nm, c);
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) nm = fmax(nm, __shfl_xor_sync(0xffffffffu, nm, o));
        nan = __any_sync(0xffffffffu, nan);
        if (threadIdx.x == 0) {
            norm1 = nan ? nan_value() : nm;
            const double theta13 = 5.371920351148152;
            sq = (!nan && nm > theta13) ? (int)ceil(log2(nm / theta13)) : 0;
        }
    }
    __syncthreads();
    if (!isfinite(norm1)) return false;
    double c[14];
    c[0] = 1.0;
#pragma unroll
    for (int j = 0; j < 13; ++j) c[j + 1] = c[j] * (double)(13 - j) / ((double)(j + 1) * (double)(26 - j));
    const double scale = ldexp(1.0, -sq);
    for (int e = threadIdx.x; e < MP2 * MP2; e += T) B[e] = A[e] * scale;
    __syncthreads();
    mm(B, B, B2);
    mm(B2, B2, B4);
    mm(B4, B2, B6);
    for (int e = threadIdx.x; e < MP2 * MP2; e += T) Tm[e] = c[13] * B6[e] + c[11] * B4[e] + c[9] * B2[e];
    __syncthreads();
    mm(B6, Tm, A);  // A is free now: W = B6 (c13 B6 + c11 B4 + c9 B2)
    for (int e = threadIdx.x; e < MP2 * MP2; e += T) {
        A[e] += c[7] * B6[e] + c[5] * B4[e] + c[3] * B2[e];
        if (e % MP2 == e / MP2) A[e] += c[1];
    }
    __syncthreads();
    mm(B, A, U);  // U = B W
    for (int e = threadIdx.x; e < MP2 * MP2; e += T) Tm[e] = c[12] * B6[e] + c[10] * B4[e] + c[8] * B2[e];
    __syncthreads();
    mm(B6, Tm, V);
    for (int e = threadIdx.x; e < MP2 * MP2; e += T) {
        double vv = V[e] + c[6] * B6[e] + c[4] * B4[e] + c[2] * B2[e];
        if (e % MP2 == e / MP2) vv += c[0];
        const double u = U[e];
        B2[e] = vv - u;  // P = V - U
        B4[e] = vv + u;  // Q = V + U (becomes the solution)
    }
    __syncthreads();
    // LU with partial pivoting of P (B2), applied to Q (B4): one column per step; a warp takes every WARPS-th
    // column of [P Q], its lanes the rows (the other way round all lanes meet in one bank).
    constexpr int RN = (MP2 + 31) / 32;  // rows per lane
    double *P = B2, *Q = B4;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    __shared__ int singular;
    if (threadIdx.x == 0) singular = 0;
    __syncthreads();
    for (int col = 0; col < MP2; ++col) {
        if (threadIdx.x < 32) {  // the first largest entry of the column on or below the diagonal
            double best = -1.0;
            int p = col;
            for (int i = col + (int)threadIdx.x; i < MP2; i += 32) {
                const double vv = fabs(P[i + col * MP2]);
                if (vv > best) {
                    best = vv;
                    p = i;
                }
            }
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) {
                const double ob = __shfl_xor_sync(0xffffffffu, best, o);
                const int op = __shfl_xor_sync(0xffffffffu, p, o);
                if (ob > best || (ob == best && op < p)) {
                    best = ob;
                    p = op;
                }
            }
            if (threadIdx.x == 0) {
                s.piv[col] = p;
                s.dpiv[col] = P[p + col * MP2];
                s.dinv[col] = 1.0 / s.dpiv[col];
                if (!(best > 0.0)) singular = 1;
            }
        }
        __syncthreads();
        if (singular) return false;
        const int p = s.piv[col];
        const double inv = s.dinv[col];
        double l[RN];  // multipliers; rows p and col change places as the columns are read
#pragma unroll
        for (int q = 0; q < RN; ++q) {
            const int i = lane + 32 * q;
            l[q] = i > col && i < MP2 ? P[(i == p ? col : i) + col * MP2] * inv : 0.0;
        }
        for (int j = warp; j < 2 * MP2; j += WARPS) {
            if (j <= col) continue;
            double *c = j < MP2 ? P + j * MP2 : Q + (j - MP2) * MP2;
            const double pivot = c[p], other = c[col];
            double x[RN];
#pragma unroll
            for (int q = 0; q < RN; ++q) {
                const int i = lane + 32 * q;
                x[q] = i > col && i < MP2 ? fma(-l[q], pivot, i == p ? other : c[i]) : 0.0;
            }
            __syncwarp();
#pragma unroll
            for (int q = 0; q < RN; ++q) {
                const int i = lane + 32 * q;
                if (i > col && i < MP2) c[i] = x[q];
                if (i == col) c[i] = pivot;
            }
        }
        __syncthreads();
    }
    // back substitution: a column of Q in the lanes of one warp
    for (int j = warp; j < MP2; j += WARPS) {
        double x[RN];
#pragma unroll
        for (int q = 0; q < RN; ++q) x[q] = lane + 32 * q < MP2 ? Q[lane + 32 * q + j * MP2] : 0.0;
#pragma unroll
        for (int q = RN - 1; q >= 0; --q)
            for (int c2 = min(MP2, 32 * (q + 1)) - 1; c2 >= 32 * q; --c2) {
                const double t = __shfl_sync(0xffffffffu, x[q], c2 & 31) / s.dpiv[c2];
#pragma unroll
                for (int r = 0; r <= q; ++r) {
                    const int i = lane + 32 * r;
                    if (i < c2) x[r] = fma(-P[i + c2 * MP2], t, x[r]);
                    else if (i == c2) x[r] = t;
                }
            }
#pragma unroll
        for (int q = 0; q < RN; ++q)
            if (lane + 32 * q < MP2) Q[lane + 32 * q + j * MP2] = x[q];
    }
    __syncthreads();
    double *R = Q, *Tmp = B6;
    for (int k = 0; k < sq; ++k) {
        mm(R, R, Tmp);
        double *t0 = R;
        R = Tmp;
        Tmp = t0;
    }
    bool bad = false;
    for (int e = threadIdx.x; e < MP2 * MP2; e += T) {
        s.pade[0][e] = R[e];
        bad = bad || !isfinite(R[e]);
    }
    return !__syncthreads_or(bad);
}

__device__ __forceinline__ double round2(double t) {
    const double sc = pow(10.0, floor(log10(t)) - 1.0);
    return ceil(t / sc) * sc;
}

// ---- passes over the own chunk [i0, i1) of the states ---------------------------------------------
// Called functions: each has the registers for its eight 16-byte loads, and what the solve keeps is
// saved once per pass (inlined, 560 bytes a thread were spilled inside the loops of the 512-thread shape).
// Basis vector k starts at v (k = 0) or W + (k - 1) ld.

// w = rho A x, or (w null) the sum of squares of rho A x
__device__ __noinline__ double pass_apply(const CufspBatchInst &in, const Tables &t, const double *tab, const double *x,
                                          double *__restrict__ w, int i0, int i1, double rho) {
    double acc = 0.0;
    for_pairs<1>(i0, i1, [&](int i, bool two) {
        double2 r;
        r.x = apply_at(in, t, tab, x, i, rho);
        r.y = two ? apply_at(in, t, tab, x, i + 1, rho) : 0.0;
        if (w) st2(w + i, r, two);
        acc = fma(r.y, r.y, fma(r.x, r.x, acc));
    });
    return acc;
}

// Warp partial sums of W_k . w for the K vectors from k0 on
__device__ __noinline__ void pass_dots(Shared &s, const double *v, const double *W, int ld, int k0, int K, const double *w,
                                       int i0, int i1) {
#pragma unroll 1
    for (int g0 = 0; g0 < K; g0 += 8) {
        double acc[8] = {0.0, 0.0, 0.0, 0.0, 0.0, 0.0, 0.0, 0.0};
        const int used = K - g0;
        const double *const pn = W + (size_t)(k0 + g0) * ld, *const p0 = k0 + g0 == 0 ? v : pn - ld;
        for_pairs<1>(i0, i1, [&](int i, bool two) {
            const double2 wi = ld2(w + i, two);
            double2 x[8];
#pragma unroll
            for (int k = 0; k < 8; ++k) {
                x[k] = make_double2(0.0, 0.0);
                if (k < used) x[k] = ld2((k ? pn + (size_t)(k - 1) * ld : p0) + i, two);
            }
#pragma unroll
            for (int k = 0; k < 8; ++k) acc[k] = fma(x[k].y, wi.y, fma(x[k].x, wi.x, acc[k]));
        });
        warp_partials8(s, acc, g0, K);
    }
}

// w -= sum of c_k W_k over the K vectors from k0 on, returns the sum of squares of w.  Backwards: what
// the dots have read last is still in L2 (15 bases of 14 MB do not fit it).
__device__ __noinline__ double pass_update(const double *v, const double *W, int ld, int k0, int K, const double *c, double *w,
                                           int i0, int i1) {
    double acc = 0.0;
    for_pairs_back(i0, i1, [&](int i, bool two) {
        double2 r = ld2(w + i, two);
#pragma unroll 1
        for (int g0 = 0; g0 < K; g0 += 8) {
            const double *const pn = W + (size_t)(k0 + g0) * ld + i, *const p0 = k0 + g0 == 0 ? v + i : pn - ld;
            double2 x[8];
#pragma unroll
            for (int k = 0; k < 8; ++k) {
                x[k] = make_double2(0.0, 0.0);
                if (g0 + k < K) x[k] = ld2(k ? pn + (size_t)(k - 1) * ld : p0, two);
            }
#pragma unroll
            for (int k = 0; k < 8; ++k) {
                const double ck = -c[g0 + k];  // past K: any finite number, times 0
                r.x = fma(ck, x[k].x, r.x);
                r.y = fma(ck, x[k].y, r.y);
            }
        }
        st2(w + i, r, two);
        acc = fma(r.y, r.y, fma(r.x, r.x, acc));
    });
    return acc;
}

// v = sum of c_k W_k over the first K vectors (W_0 = v: every pair is read before it is written)
__device__ __noinline__ void pass_combine(double *v, const double *W, int ld, int K, const double *c, int i0, int i1) {
    for_pairs<1>(i0, i1, [&](int i, bool two) {
        double2 r = make_double2(0.0, 0.0);
#pragma unroll 1
        for (int g0 = 0; g0 < K; g0 += 8) {
            const double *const pn = W + (size_t)g0 * ld + i, *const p0 = g0 == 0 ? v + i : pn - ld;
            double2 x[8];
#pragma unroll
            for (int k = 0; k < 8; ++k) {
                x[k] = make_double2(0.0, 0.0);
                if (g0 + k < K) x[k] = ld2(k ? pn + (size_t)(k - 1) * ld : p0, two);
            }
#pragma unroll
            for (int k = 0; k < 8; ++k) {
                r.x = fma(c[g0 + k], x[k].x, r.x);
                r.y = fma(c[g0 + k], x[k].y, r.y);
            }
        }
        st2(v + i, r, two);
    });
}

// ---- one instance --------------------------------------------------------------------------
__device__ void solve_instance(const CufspBatchArgs &a, cg::cluster_group &cl, Shared &s, double *W, double *tabs,
                               int ld_max, int &buf) {
    const int n = s.in.n;
    const int nb = (int)cl.num_blocks(), rank = (int)cl.block_rank();
    const int chunk = ((n + nb - 1) / nb + 63) & ~63;
    const int ld = (n + 1) & ~1;
    const int i0 = min(n, rank * chunk), i1 = min(n, i0 + chunk);
    double *v = a.p + s.in.off;
    const double *tab = a.tables + s.in.tab;
    auto vec = [&](int k) -> double * { return k == 0 ? v : W + (size_t)(k - 1) * ld; };
    const double delta = 1.2, gamma = 0.9;
    double t_now = 0.0, t_new = 0.0, xm = 1.0 / M, err_loc = 0.0;
    const double btol = a.anorm * a.tol;
    int steps = 0, rejects = 0, matvecs = 0, status = 0;
    Tables tb;
    {  // behind the solver's state in shared memory, or behind the basis in the cluster's workspace
        constexpr bool OWN = CUFSP_BATCH_TABSMEM != 0;
        const int me = OWN ? (int)threadIdx.x : rank * T + (int)threadIdx.x, step = OWN ? T : nb * T;
        double *gain = OWN ? tabs : W + (size_t)(M + 1) * ld_max;
        double *loss = gain + (size_t)NR * s.in.tab_stride;
        auto sync = [&] {
            if constexpr (OWN) __syncthreads();
            else cl.sync();
        };
        for (int x = me; x < s.in.tab_stride; x += step) loss[x] = 0.0;
        sync();
        fill_tables<0, 0>(s.in, tab, gain, loss, me, step);
        sync();
        tb.gain = gain;
        tb.loss = loss;
    }

    while (t_now < a.t_final && status == 0) {
        if (steps >= a.max_steps) {
            status = 1;
            break;
        }
        // beta = ||v||
        double acc1 = 0.0;
        for_pairs<1>(i0, i1, [&](int i, bool two) {
            const double2 x = ld2(v + i, two);
            acc1 = fma(x.y, x.y, fma(x.x, x.x, acc1));
        });
        cluster_sum1(cl, s, acc1, buf);
        const double beta = sqrt(s.tot[0]);
        if (!isfinite(beta)) {
            status = 2;
            break;
        }
        if (beta == 0.0) {  // exp(tA) 0 = 0
            t_now = a.t_final;
            break;
        }
        for (int e = threadIdx.x; e < MP2 * MP2; e += T) s.H[e] = 0.0;
        for (int e = threadIdx.x; e < MP2; e += T) s.rho[e] = 0.0;
        for (int e = threadIdx.x; e < MP2 + 8; e += T) s.gam[e] = s.coefc[e] = 0.0;
        __syncthreads();
        if (threadIdx.x == 0) s.rho[0] = 1.0 / beta;
        __syncthreads();
        if (steps == 0) {  // first-step size (src/KryExpvFSP.cu:45-51)
            const double fact = pow((M + 1) / exp(1.0), M + 1) * sqrt(2.0 * 3.14159265358979323846 * (M + 1));
            t_new = (1.0 / a.anorm) * pow((fact * a.tol) / (4.0 * beta * a.anorm), 1.0 / M);
        }
        // Arnoldi
        int mb = M, k1 = 2;
        double avnorm = 0.0;
        for (int j = 0; j < M; ++j) {
            const int istart = IOP ? max(0, j - QIOP + 1) : 0;
            const int K = j - istart + 1;
            const double *vj = vec(j);
            double *w = vec(j + 1);
            const double rj = s.rho[j];
            // generator action (own chunk; neighbours read anywhere in the instance), Gram-Schmidt dots (each
            // thread reads only its own w entries)
            pass_apply(s.in, tb, tab, vj, w, i0, i1, rj);
            pass_dots(s, v, W, ld, istart, K, w, i0, i1);
            cluster_finish(cl, s, K, buf);
            for (int k = threadIdx.x; k < K; k += T) {
                const double h = s.rho[istart + k] * s.tot[k];
                s.H[(istart + k) + j * MP2] = h;
                s.gam[istart + k] = h * s.rho[istart + k];
            }
            __syncthreads();
            const double acc2 = pass_update(v, W, ld, istart, K, s.gam + istart, w, i0, i1);
            cluster_sum1(cl, s, acc2, buf);
            const double sn = sqrt(s.tot[0]);
            ++matvecs;
            if (!isfinite(sn)) {
                status = 2;
                break;
            }
            // happy breakdown (src/KryExpvFSP.cu:90-98) with the threshold divided by the remaining time
            // (when above 1): the jump to t_final then stays within tol
            if (sn < btol / fmax(1.0, a.t_final - t_now)) {
                k1 = 0;
                mb = j + 1;
                break;
            }
            if (threadIdx.x == 0) {
                s.H[(j + 1) + j * MP2] = sn;
                s.rho[j + 1] = 1.0 / sn;
            }
            __syncthreads();
        }
        if (status) break;
        double tau = fmin(a.t_final - t_now, t_new);
        if (k1 == 0) {
            tau = a.t_final - t_now;
        } else {  // avnorm = ||A v_m|| (src/KryExpvFSP.cu:114-120)
            const double *vm = vec(M);
            const double rm = s.rho[M];
            const double acc3 = pass_apply(s.in, tb, tab, vm, nullptr, i0, i1, rm);
            cluster_sum1(cl, s, acc3, buf);
            avnorm = sqrt(s.tot[0]);
            ++matvecs;
            if (!isfinite(avnorm)) {
                status = 2;
                break;
            }
            if (threadIdx.x == 0) s.H[(M + 1) + M * MP2] = 1.0;
            __syncthreads();
        }
        // rejection loop (src/KryExpvFSP.cu:122-158)
        bool accepted = false;
        int mx = mb + k1;
        while (rejects <= a.max_reject) {
            for (int e = threadIdx.x; e < MP2 * MP2; e += T) s.pade[7][e] = tau * s.H[e];
            __syncthreads();
            if (!expm_dev(s)) {
                status = 2;
                break;
            }
            const double *F = s.pade[0];
            if (k1 == 0) {
                err_loc = btol;
                accepted = true;
                break;
            }
            const double phi1 = fabs(beta * F[mx - 2]);
            const double phi2 = fabs(beta * F[mx - 1] * avnorm);
            if (phi1 > phi2 * 10.0) {
                err_loc = phi2;
                xm = 1.0 / (double)mx;
            } else if (phi1 > phi2) {
                err_loc = (phi1 * phi2) / (phi1 - phi2);
                xm = 1.0 / (double)mx;
            } else {
                err_loc = phi1;
                xm = 1.0 / (double)(mx - 1);
            }
            if (!isfinite(err_loc)) {
                status = 2;
                break;
            }
            if (err_loc <= delta * tau * a.tol) {
                accepted = true;
                break;
            }
            tau = round2(gamma * tau * pow(tau * a.tol / err_loc, xm));
            ++rejects;
        }
        if (status) break;
        if (!accepted) {
            status = 1;
            break;
        }
        // v = beta V[:, 0:mx] F(0:mx, 0) = sum_k (beta F_k0 rho_k) W_k
        mx = mb + max(0, k1 - 1);
        for (int k = threadIdx.x; k < mx; k += T) s.coefc[k] = beta * s.pade[0][k] * s.rho[k];
        __syncthreads();
        pass_combine(v, W, ld, mx, s.coefc, i0, i1);
        const bool last = tau >= a.t_final - t_now;
        t_now = last ? a.t_final : t_now + tau;
        if (err_loc > 0.0) t_new = round2(gamma * tau * pow(tau * a.tol / err_loc, xm));
        if (!(t_new > 0.0) || !isfinite(t_new)) t_new = a.t_final - t_now;
        ++steps;
        cl.sync();  // v complete before the next step's generator action reads it
    }
    if (rank == 0 && threadIdx.x == 0) {
        CufspBatchStat st;
        st.t = t_now;
        st.err = err_loc;
        st.steps = steps;
        st.rejects = rejects;
        st.matvecs = matvecs;
        st.status = status;
        a.stats[s.inst_idx] = st;
    }
}

}  // namespace cufsp_batch

// Dynamic shared memory the kernel needs (read by the host after loading).
extern "C" __device__ const int cufsp_batch_smem_bytes = (int)sizeof(cufsp_batch::Shared);

extern "C" __global__ void __launch_bounds__(CUFSP_BATCH_THREADS, CUFSP_BATCH_MINB)
    cufsp_batch_expv(const CufspBatchArgs a) {
    using namespace cufsp_batch;
    extern __shared__ __align__(16) unsigned char dsm[];
    Shared &s = *reinterpret_cast<Shared *>(dsm);
    cg::cluster_group cl = cg::this_cluster();
    const int nb = (int)cl.num_blocks();
    const int cid = (int)(blockIdx.x / nb);
    double *W = a.work + (size_t)cid * (size_t)a.work_stride;
    int buf = 0;
    for (int it = 0; it < a.n_inst; ++it) {  // at most one instance per iteration and cluster
        if (cl.block_rank() == 0 && threadIdx.x == 0) s.inst_idx = (int)atomicAdd(a.counter, 1u);
        cl.sync();
        if (threadIdx.x == 0) s.inst_idx = *cl.map_shared_rank(&s.inst_idx, 0);
        cl.sync();  // every CTA has read rank 0's index before rank 0 can overwrite it
        if (s.inst_idx >= a.n_inst) break;
        const int idx = a.order[s.inst_idx];
        if (threadIdx.x == 0) s.inst_idx = idx;
        for (int e = threadIdx.x; e < (int)(sizeof(CufspBatchInst) / sizeof(int)); e += T)
            reinterpret_cast<int *>(&s.in)[e] = reinterpret_cast<const int *>(a.inst + idx)[e];
        __syncthreads();
        solve_instance(a, cl, s, W, reinterpret_cast<double *>(dsm + sizeof(Shared)), a.ld_max, buf);
        cl.sync();  // the cluster's workspace is free again
    }
}

#endif  // __CUDACC_RTC__
#endif  // CUFSP_BATCH_CUH
