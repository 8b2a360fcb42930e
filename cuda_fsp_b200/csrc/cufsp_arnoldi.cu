// cufsp_arnoldi.cu -- the Arnoldi pass of one Krylov step as ONE persistent launch, for generators
// whose Krylov basis stays on the chip (single-instance solves of 32K-1M states).
//
// Same arithmetic contract as the launch sequence of cufsp_krylov.cu (src/KryExpvFSP.cu:38-120,
// restated there): basis W_k with v_k = rho_k W_k, h = V^T w, w -= V h, ||w||, happy breakdown,
// ||A v_m||, results in the same device state block.  At these sizes every one of the ~3m kernels
// of that sequence is latency-bound; here one cooperative grid walks all m iterations.  What bounds an
// iteration is the chain of waits between CTAs, so the chain is as short as the recurrence allows:
//  * ONE all-to-all exchange per iteration.  The norm of W_j is not waited for before A W_j is formed:
//    each CTA publishes its partial sums of ||W_j||^2 together with those of W_k . (A W_j), k <= j, and
//      rho_j = 1/||W_j||,  h_k = rho_k rho_j W_k . (A W_j),  W_{j+1} = rho_j (A W_j - sum_k rho_k^2 (W_k . A W_j) W_k)
//    follow from the totals: the same quantities as with a normalisation first, to rounding.  The
//    breakdown test of W_j then runs one iteration later, after one generator application too many.
//  * no grid barrier (cufsp_grid.cuh): partial sums and the entries of W_j that other CTAs gather are
//    polled as data.  Every CTA sums the partials in the same fixed order, so all take identical
//    decisions.
//  * the generator is applied from a per-state term table built once per coefficient vector:
//      (A x)[i] = sum_t coef[t][i] x[i - shift_t]   (last term: shift 0, the diagonal),
//    coefficient 0 wherever the source state leaves the box (its index is clamped to [0, n)).  A CTA
//    owns a contiguous slice of the states; up to 4 states per thread, 10 near and 8 far terms the coefficients
//    stay in registers for the whole launch, and sources inside the slice come from shared memory.
//  * the CTA's slices of as many basis vectors as fit live in shared memory (all 30 of them up to 148 x
//    ~890 = 131K states); the dots and the update read them there and the rest from L2.
// Measured, a Krylov step of m = 30 (pass, host step control and combination): 32,768 states 0.35 ms with
// two barriers per iteration, 0.19 ms so; 134,088 states 0.50 and 0.26 ms.
// Waits are bounded; on expiry the kernel sets an error word, every CTA leaves, and the host reports
// CUFSP_ERR_CUDA.  The launch is cooperative, so all CTAs are co-resident.
#include <algorithm>
#include <cmath>
#include <cstdlib>
#include <cstring>
#include <map>

#include <mutex>

#include "cufsp_internal.h"
#include "cufsp_grid.cuh"
#include "cufsp_slice.cuh"

namespace cufsp {

namespace {

constexpr int kMaxTerms = 64;
constexpr int kPThreadsMax = 512;
constexpr int kPWarpsMax = kPThreadsMax / 32;

struct PArgs {
    SliceTerms terms;           // register variants
    int n;
    int chunk;                  // states per CTA, even (the last CTA may have fewer)
    int slots;                  // basis vectors whose slices live in shared memory
    int ring;                   // > 0: W_k is in slot k % ring (incomplete orthogonalisation); 0: W_k in slot k < slots
    int T;
    const double *coef;         // [T][n]
    int shift[kMaxTerms];       // source index i - shift[t] (clamped)
    const double *v0;           // W_0 (the caller's vector)
    double *W;                  // W_1 .. W_{m+1}
    double *H, *rho, *beta, *avnorm;
    int *flag;                  // 0 ok, >0 happy breakdown at mb = flag, -1 NaN/Inf, -2 zero vector
    int mp2, m, iop, q;
    double btol;
    int with_avnorm;
    double *ex;                 // exchange area of this launch, all unset
    double *ex_next;            // that of the next launch, set back to unset here
    int ex_rows;                // rows of an area
    Waits waits;
    double *h_state;            // pinned host copy of the state block (nullable), its length and sequence word
    int words;
    unsigned *h_seq, seq;
};

struct PSmem {
    double2 c2[(CUFSP_MAX_KRYLOV + 4) / 2];  // c_r = rho_k^2 W_k . (A W_j) of the vector at position r; 0 for W_j
    double part[kPWarpsMax][4];              // dots of one warp's four vectors over its part of the slice
    double wsum[kPWarpsMax], asum[kPWarpsMax];  // per-warp sums of ||W_j||^2 and of ||A W_m||^2
    double dot[CUFSP_MAX_KRYLOV + 2];        // W_k . (A W_j) by position
    double rho[CUFSP_MAX_KRYLOV + 2];        // by k
    double sn, rj;                           // ||W_j||, 1 / ||W_j||
};

// NT threads.  TN > 0: at most NS states per thread, TN near and TF far terms (cufsp_slice.cuh), their
// coefficients in registers.  TN = 0: any.
// 8 warps with up to 4 states per thread rather than 16 or 32 with fewer: at these sizes the instructions
// that every warp spends on addresses, reductions and waits, not the data, fill an iteration between two
// waits, and a thread of 8 warps has 255 registers, so that nothing spills (a spill goes to L2: shared
// memory leaves little L1).
template <int NT, int NS, int TN, int TF>
__global__ void __launch_bounds__(NT, 1) k_arnoldi_persistent(const __grid_constant__ PArgs a) {
    extern __shared__ __align__(16) double ws[];  // [chunk] slice of A W_j | [halo][chunk][halo] of W_j | [slots][chunk] basis
    __shared__ __align__(16) PSmem sm;
    constexpr bool REG = TN > 0;
    constexpr int NW = NT / 32, LNW = NW == 16 ? 4 : 3;
    static_assert(NW == 1 << LNW, "8 or 16 warps");
    const int lo = (int)blockIdx.x * a.chunk;
    const int len = min(a.chunk, a.n - lo);
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const bool lead = blockIdx.x == 0 && tid == 0;
    double *const xs = ws + a.chunk + a.terms.halo;
    double *const slot0 = xs + a.chunk + a.terms.halo;
    double *const c = reinterpret_cast<double *>(sm.c2);
    const int pitch = exchange_pitch((int)gridDim.x);

#pragma unroll 1
    for (int p = (int)blockIdx.x * NT + tid; p < exchange_doubles(a.ex_rows, (int)gridDim.x); p += (int)gridDim.x * NT)
        a.ex_next[p] = unset_value();
    if (blockIdx.x == 0) {
#pragma unroll 1
        for (int i = tid; i < a.mp2 * (a.mp2 + 2); i += NT) a.H[i] = 0.0;  // H, rho and the launch sequence's gamma are contiguous
    }
#pragma unroll 1
    for (int il = tid; il < (a.slots + 2) * a.chunk + 2 * a.terms.halo; il += NT) ws[il] = 0.0;
    if (tid < CUFSP_MAX_KRYLOV + 4) c[tid] = 0.0;  // positions a loop rounded up to four may read
    __syncthreads();
    double cn[NS][REG ? TN : 1], cfar[NS][REG ? TF : 1];
    if constexpr (REG) {
#pragma unroll
        for (int s = 0; s < NS; ++s) {
            const int il = tid + s * NT;
            const double *cp = a.coef + lo + il;
#pragma unroll
            for (int t = 0; t < TN; ++t) cn[s][t] = t < a.terms.n_near && il < len ? __ldcg(cp + (size_t)a.terms.near_t[t] * a.n) : 0.0;
#pragma unroll
            for (int t = 0; t < TF; ++t) cfar[s][t] = t < a.terms.n_far && il < len ? __ldcg(cp + (size_t)a.terms.far_t[t] * a.n) : 0.0;
        }
    }
    double acc = 0.0;
#pragma unroll 1
    for (int il = tid; il < len; il += NT) {
        const double t = __ldcg(a.v0 + lo + il);
        xs[il] = t;
        if (a.slots > 0) slot0[il] = t;
        acc = fma(t, t, acc);
        double *w = a.W + lo + il;
#pragma unroll 2
        for (int k = 0; k < a.m; ++k, w += a.n) st_relaxed(w, unset_value());
    }
    acc = warp_sum(acc);
    if (lane == 0) sm.wsum[warp] = acc;
    __syncthreads();

    int pj = 0;                // position of W_j in its window
    int row = 0;               // first exchange row of this iteration
    const double *x = a.v0;    // W_j
#pragma unroll 1
    for (int j = 0;; ++j) {
        const bool last = j == a.m;
        const int istart = a.iop ? max(0, j - a.q + 1) : 0;
        const int K = last ? 0 : j - istart + 1;
        const int rows = last ? 1 + a.with_avnorm : K + 1;
        const int Kres = a.ring > 0 ? K : max(0, min(K, a.slots - istart));  // positions in shared memory
        const double *const base = slot0 + (a.ring > 0 ? 0 : istart * a.chunk);
        const double *const gbase = a.W + lo + ((long long)istart - 1) * a.n;   // position r > 0: + r n
        double *const mine = a.ex + (size_t)row * pitch + blockIdx.x;
        double w[NS];
        double aw2 = 0.0;
        bool bad = false;
        if (warp == NW - 1 && j > 0) {  // row 0: ||W_j||^2, on its way while A W_j is formed
            const double v = warp_sum(lane < NW ? sm.wsum[lane] : 0.0);
            if (lane == 0) st_relaxed(mine, settled(v));
        }
        if (!last || a.with_avnorm) {
            if constexpr (REG) {
                double v[NS][TF];
                bad = !gather_begin<NT, NS, TF, false>(a.terms, x, lo, len, j > 0, xs, v, a.waits);
                __syncthreads();
                if (!gather_end<NT, NS, TN, TF>(a.terms, x, lo, len, j > 0, xs, cn, cfar, v, w, a.waits)) bad = true;
#pragma unroll
                for (int s = 0; s < NS; ++s) {
                    if (tid + s * NT < len) ws[tid + s * NT] = w[s];
                    aw2 = fma(w[s], w[s], aw2);
                }
            } else {
#pragma unroll 1
                for (int il = tid; il < len; il += NT) {
                    Patience wait;
                    double sum;
                    bool miss;
                    do {
                        sum = 0.0;
                        miss = false;
#pragma unroll 4
                        for (int t = 0; t < a.T; ++t) {
                            const int rel = il - a.shift[t];
                            double v;
                            if ((unsigned)rel < (unsigned)len) v = xs[rel];
                            else v = far_entry(x, lo, rel, a.n);
                            miss = miss || is_unset(v);
                            sum = fma(__ldg(a.coef + (size_t)t * a.n + lo + il), v, sum);
                        }
                        if (j == 0 || !miss) break;
                        bad = bad || wait.give_up(a.waits);
                    } while (!bad);
                    ws[il] = sum;
                    aw2 = fma(sum, sum, aw2);
                }
            }
        }
        if (last) {
            aw2 = warp_sum(aw2);
            if (lane == 0) sm.asum[warp] = aw2;
        }
        if (__syncthreads_or(bad)) return;
        slice_dots<LNW>(ws, a.chunk, len, K, Kres, base, istart == 0 ? a.v0 + lo : gbase, gbase, a.n, sm.part);
        __syncthreads();
        // publish the other rows: the dots, or ||A W_m||^2
        if (j == 0) __threadfence();  // the cleared basis is visible before any CTA passes this exchange
        if (tid < K) {
            st_relaxed(mine + (size_t)(1 + tid) * pitch, settled(dots_sum<LNW>(sm.part, K, tid)));
        }
        if (warp == NW - 1 && (last || j == 0)) {
            const double v = warp_sum(lane < NW ? (last ? sm.asum : sm.wsum)[lane] : 0.0);
            if (lane == 0 && (j == 0 || rows == 2)) st_relaxed(mine + (j == 0 ? 0 : pitch), settled(v));
        }
        if (!exchange_own(a.ex, a.ex_rows, row, rows, 1, NW, j == 0, a.waits)) bad = true;
        if (warp == 0) {
#pragma unroll 1
            for (int r = lane + 1; r < rows; r += 32) {
                const int pos = r - 1;
                const int k = a.ring > 0 ? pos + a.ring * ((j - pos) / a.ring) : istart + pos;
                const double rk = k < j ? sm.rho[k] : 0.0;
                double v;
                if (!exchange_total(a.ex, a.ex_rows, row, r, a.waits, v)) bad = true;
                sm.dot[pos] = v;
                c[pos] = v * (rk * rk);
            }
        } else if (warp == NW - 1) {  // the norm has come earlier: its root and inverse hide behind the dots
            double v;
            if (!exchange_total(a.ex, a.ex_rows, row, 0, a.waits, v)) bad = true;
            const double sn = sqrt(v);
            sm.sn = sn;
            sm.rj = sn > 0.0 ? 1.0 / sn : 0.0;
        }
        if (j == 0) __threadfence();
        if (__syncthreads_or(bad)) return;
        row += rows;
        const double sn = sm.sn, rj = sm.rj;
        // 0: go on, else the flag that ends the pass: happy breakdown (src/KryExpvFSP.cu:90-98) at W_j
        const int stop = !isfinite(sn) ? -1 : j == 0 ? (sn == 0.0 ? -2 : 0) : (sn < a.btol ? j : 0);
        if (stop || last) {
            if (lead) {
                if (j == 0) {
                    *a.beta = sn;
                    *a.avnorm = 0.0;
                    a.rho[0] = rj;
                }
                *a.flag = stop;
                if (last && !stop) {
                    a.H[j + (j - 1) * a.mp2] = sn;
                    a.rho[j] = rj;
                    if (rows == 2) {  // ||A v_m|| (src/KryExpvFSP.cu:114-120)
                        const double av = rj * sqrt(sm.dot[0]);
                        *a.avnorm = av;
                        if (!isfinite(av)) *a.flag = -1;
                    }
                }
            }
            if (blockIdx.x == 0 && a.h_state) {  // to the host: all of it was written by this CTA
                __syncthreads();
                for (int i = tid; i < a.words; i += NT) a.h_state[i] = a.H[i];
                __threadfence_system();
                __syncthreads();
                if (tid == 0) *(volatile unsigned *)a.h_seq = a.seq;
            }
            return;
        }
        // W_{j+1} = rho_j (A W_j - sum_k c_k W_k), and its squared norm
        const double cj = sm.dot[pj] * (rj * rj);
        double *const wn = a.W + (size_t)j * a.n + lo;
        pj = a.ring > 0 ? (pj + 1 == a.ring ? 0 : pj + 1) : j + 1 - (a.iop ? max(0, j + 2 - a.q) : 0);
        double *const xn = a.ring > 0 ? slot0 + pj * a.chunk : j + 1 < a.slots ? slot0 + (j + 1) * a.chunk : nullptr;
        acc = 0.0;
#pragma unroll 1
        for (int il = tid; il < len; il += NS * NT) {
            double u[NS];
            int off[NS];  // of the states; past the slice: the first one again
#pragma unroll
            for (int s = 0; s < NS; ++s) {
                u[s] = REG ? w[s] : ws[il];
                off[s] = il + s * NT < len ? s * NT : 0;
            }
            const double *p = base + il;
            const int r4 = min((Kres + 3) & ~3, max(0, a.ring > 0 ? a.slots : a.slots - istart) & ~3);  // past K: c is zero
            int r = 0;
#pragma unroll 1
            for (; r < r4; r += 4, p += 4 * a.chunk) {
                const double2 c01 = sm.c2[r >> 1], c23 = sm.c2[(r >> 1) + 1];
#pragma unroll
                for (int s = 0; s < NS; ++s) {
                    const double *ps = p + off[s];
                    u[s] = fma(-c01.y, ps[a.chunk], fma(-c01.x, ps[0], u[s]));
                    u[s] = fma(-c23.y, ps[3 * a.chunk], fma(-c23.x, ps[2 * a.chunk], u[s]));
                }
            }
#pragma unroll 1
            for (; r < Kres; ++r, p += a.chunk) {
#pragma unroll
                for (int s = 0; s < NS; ++s) u[s] = fma(-c[r], p[off[s]], u[s]);
            }
            r = Kres;
#pragma unroll 2
            for (; r < K - 1; ++r) {  // positions in L2 (W_j itself follows)
                const double *g = (istart + r == 0 ? a.v0 + lo : gbase + (size_t)r * a.n) + il;
#pragma unroll
                for (int s = 0; s < NS; ++s) u[s] = fma(-c[r], __ldcg(g + off[s]), u[s]);
            }
#pragma unroll
            for (int s = 0; s < NS; ++s) {
                if (s == 0 || off[s] > 0) {
                    const int i = il + s * NT;
                    const double wi = settled(fma(-cj, xs[i], u[s]) * rj);
                    st_relaxed(wn + i, wi);
                    acc = fma(wi, wi, acc);
                    xs[i] = wi;
                    if (xn) xn[i] = wi;
                }
            }
        }
        acc = warp_sum(acc);
        if (lane == 0) sm.wsum[warp] = acc;
        x = a.W + (size_t)j * a.n;
        __syncthreads();
        if (blockIdx.x == 0) {  // column j of H, while the others' entries travel
            if (tid < K) {
                const int k = a.ring > 0 ? tid + a.ring * ((j - tid) / a.ring) : istart + tid;
                a.H[k + j * a.mp2] = (k == j ? rj : sm.rho[k]) * rj * sm.dot[tid];
            }
            if (tid == NT - 1) {
                a.rho[j] = rj;
                if (j > 0) a.H[j + (j - 1) * a.mp2] = sn;
                else {
                    *a.beta = sn;
                    *a.avnorm = 0.0;
                }
            }
        }
        if (tid == 0) sm.rho[j] = rj;
    }
}

// ---- term table ---------------------------------------------------------------------------------

struct TermBuildArgs {
    int64_t n;
    int ns, nr, T, tab_stride, transpose;
    int dims[CUFSP_MAX_SPECIES];
    int tab_off[CUFSP_MAX_SPECIES];
    const double *tables;  // [nr][tab_stride] factor tables, or null
    const double *props;   // [nr][n] propensities a_r(x_i), or null
    const int *nu;         // [nr][ns]
    const double *c;       // [nr] coefficients
    const int *rterm;      // [nr] term of reaction r (-1: no source inside the box, -2: no net change)
    const int64_t *d;      // [nr] flat shift sum_s nu_{r,s} stride_s
    double *coef;          // [T][n]
};

__device__ __forceinline__ double prop_at(const TermBuildArgs &b, int r, int64_t i, const int *xs) {
    if (b.props) return b.props[(size_t)r * b.n + i];
    double f = 1.0;
    const double *tr = b.tables + (size_t)r * b.tab_stride;
    for (int s = 0; s < b.ns; ++s) f *= tr[b.tab_off[s] + xs[s]];
    return f;
}

__global__ void k_build_terms(const TermBuildArgs b) {
    const int64_t stride = (int64_t)gridDim.x * blockDim.x;
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < b.n; i += stride) {
        int xs[CUFSP_MAX_SPECIES], ys[CUFSP_MAX_SPECIES];
        int64_t rem = i;
        for (int s = 0; s < b.ns; ++s) {
            xs[s] = (int)(rem % b.dims[s]);
            rem /= b.dims[s];
        }
        double acc[kMaxTerms];
        for (int t = 0; t < b.T; ++t) acc[t] = 0.0;
        for (int r = 0; r < b.nr; ++r) {
            const int t = b.rterm[r];
            if (t == -2) continue;  // its gain and its outflow cancel
            const double cr = b.c[r];
            const double here = prop_at(b, r, i, xs);
            acc[b.T - 1] -= cr * here;  // the diagonal keeps the full outflow
            if (t < 0) continue;
            const int sg = b.transpose ? 1 : -1;  // A: source x - nu_r;  A^T: target x + nu_r
            bool ok = true;
            for (int s = 0; s < b.ns; ++s) {
                ys[s] = xs[s] + sg * b.nu[r * b.ns + s];
                ok = ok && ys[s] >= 0 && ys[s] < b.dims[s];
            }
            if (!ok) continue;
            if (b.transpose) acc[t] += cr * here;
            else acc[t] += cr * prop_at(b, r, i - b.d[r], ys);
        }
        for (int t = 0; t < b.T; ++t) b.coef[(size_t)t * b.n + i] = acc[t];
    }
}

thread_local bool tl_disabled = false;

}  // namespace

struct PArnoldi {
    struct Terms {
        std::vector<double> coefs;
        bool transpose = false;
        int T = 0;
        std::vector<int64_t> shift;
        double *d_coef = nullptr;
    };
    Terms terms[2];       // forward and transposed, each for its last coefficient vector
    int *d_nu = nullptr;  // model data for the term builder
    double *d_tables = nullptr, *d_c = nullptr;
    int *d_rterm = nullptr;
    int64_t *d_d = nullptr;
    double *d_props = nullptr;  // sparse formats: exported propensities
    bool have_model = false;  // the model data above has arrived
    double *d_ex = nullptr;  // two exchange areas: a launch uses one and clears the other
    bool clean = false;      // so that the next launch's is unset: the last launch has reported
    int ex_rows = 0;         // rows per area
    int turn = 0;            // area of the next launch
    int grid = 0, chunk = 0, slots = 0, ring = 0;
    size_t smem = 0;
};

namespace {
template <class Free>
void parnoldi_release(PArnoldi *pa, Free release) {
    if (!pa) return;
    for (auto &t : pa->terms) release(t.d_coef);
    release(pa->d_nu);
    release(pa->d_tables);
    release(pa->d_c);
    release(pa->d_rterm);
    release(pa->d_d);
    release(pa->d_props);
    release(pa->d_ex);
    delete pa;
}
}  // namespace

void parnoldi_destroy(PArnoldi *pa) {
    parnoldi_release(pa, [](void *p) { cache_free(p); });
}

void parnoldi_destroy(PArnoldi *pa, cudaStream_t last_use) {
    parnoldi_release(pa, [last_use](void *p) { cache_free(p, last_use); });
}

void parnoldi_reported(PArnoldi *pa) { pa->clean = true; }

void parnoldi_thread_disable(bool off) { tl_disabled = off; }

namespace {
thread_local int tl_cta_cap = 0;  // at most this many CTAs per pass launched from this thread (0: all SMs)
}
void parnoldi_thread_cta_cap(int cap) { tl_cta_cap = cap > 0 ? cap : 0; }

namespace {
int persistent_mode() {  // CUFSP_ARNOLDI_PERSISTENT: 0 never, 1 always, unset: by size
    static const int mode = [] {
        const char *e = getenv("CUFSP_ARNOLDI_PERSISTENT");
        return e ? atoi(e) : -1;
    }();
    return mode;
}
}  // namespace

bool parnoldi_size_ok(int64_t n) {
    static const int64_t max_n = [] {
        const char *e = getenv("CUFSP_ARNOLDI_MAX_N");
        return e ? (int64_t)atoll(e) : (int64_t)1 << 20;
    }();
    const int mode = persistent_mode();
    return mode != 0 && (mode == 1 || n <= max_n);
}

namespace {
// Dynamic shared memory the pass may use, and what it needs beside the basis: the CTA's slices of W_j and
// A W_j, and W_j's halo.
size_t persistent_smem_max() { return (size_t)device_info().max_smem_optin - sizeof(PSmem) - 1024; }
size_t persistent_fixed(int64_t chunk) { return sizeof(double) * (2 * (size_t)chunk + 2 * kHaloMax); }

// States per CTA (even) of a pass that may use `ctas` CTAs: one CTA per SM, fewer for small n, each with at
// least 256 states by default (CUFSP_ARNOLDI_CTA_STATES).
int64_t persistent_chunk(int64_t n, int ctas) {
    static const int64_t min_states = [] {
        const char *e = getenv("CUFSP_ARNOLDI_CTA_STATES");
        return e ? std::max<int64_t>(32, atoll(e)) : (int64_t)256;
    }();
    const int64_t want = std::max<int64_t>(1, std::min<int64_t>(ctas, (n + min_states - 1) / min_states));
    return ((n + want - 1) / want + 1) & ~int64_t(1);
}

// CTAs a pass launched from this thread may use.
int persistent_ctas() {
    const int sms = std::min(device_info().sm_count, 64 * kMaxGridPairs);
    return tl_cta_cap > 0 ? std::min(tl_cta_cap, sms) : sms;
}
}  // namespace

bool parnoldi_fits(int64_t n, int ctas) {
    return n <= INT32_MAX / 2 && persistent_fixed(persistent_chunk(n, ctas)) <= persistent_smem_max();
}

bool parnoldi_wanted(const cufsp_mat *A, int64_t n, int m) {
    if (tl_disabled || !A || m > CUFSP_MAX_KRYLOV || !parnoldi_size_ok(n) || !parnoldi_fits(n, persistent_ctas())) return false;
    if (A->model.nr > CUFSP_MAX_REACTIONS_SPARSE || A->model.ns > CUFSP_MAX_SPECIES) return false;
    return A->format == CUFSP_FORMAT_KRONECKER ? !A->model.tables.empty() : A->sparse != nullptr;
}

namespace {

// Term table of A (or A^T) at `coefs`, rebuilt when either changes.
cufsp_status build_terms(PArnoldi *pa, cufsp_mat *A, const std::vector<double> &coefs, bool transpose,
                         PArnoldi::Terms *&out, cudaStream_t st) {
    PArnoldi::Terms &tm = pa->terms[transpose ? 1 : 0];
    out = &tm;
    if (tm.d_coef && tm.transpose == transpose && tm.coefs == coefs) return CUFSP_SUCCESS;
    const ModelHost &m = A->model;
    const int ns = m.ns, nr = m.nr;
    const int64_t n = m.n;
    // flat shifts and their distinct values (shift 0 = no net change)
    std::vector<int64_t> d(nr, 0), stride(ns, 1);
    for (int s = 1; s < ns; ++s) stride[s] = stride[s - 1] * ((int64_t)m.bounds[s - 1] + 1);
    for (int r = 0; r < nr; ++r)
        for (int s = 0; s < ns; ++s) d[r] += (int64_t)m.nu[(size_t)r * ns + s] * stride[s];
    std::map<int64_t, int> idx;
    std::vector<int> rterm(nr, -1);
    std::vector<int64_t> shifts;
    for (int r = 0; r < nr; ++r) {
        if (d[r] == 0 || std::llabs(d[r]) >= n) {  // no source inside the box (shifts fit an int below), or no change
            const int *nu = m.nu.data() + (size_t)r * ns;
            if (std::all_of(nu, nu + ns, [](int v) { return v == 0; })) rterm[r] = -2;
            continue;
        }
        const int64_t sh = transpose ? -d[r] : d[r];
        auto it = idx.find(sh);
        if (it == idx.end()) {
            it = idx.emplace(sh, (int)shifts.size()).first;
            shifts.push_back(sh);
        }
        rterm[r] = it->second;
    }
    const int T = (int)shifts.size() + 1;
    if (T > kMaxTerms) return set_error(CUFSP_ERR_UNSUPPORTED, "persistent Arnoldi: more than 63 distinct shifts");
    shifts.push_back(0);
    // model data on the device (once per generator), in order on st like the build below
    tm.coefs.clear();  // a build that fails leaves no table behind
    if (!pa->have_model) {
        if (!pa->d_nu) CUFSP_CUDA_TRY(cache_alloc((void **)&pa->d_nu, sizeof(int) * (size_t)nr * ns));
        CUFSP_CUDA_TRY(cudaMemcpyAsync(pa->d_nu, m.nu.data(), sizeof(int) * (size_t)nr * ns, cudaMemcpyHostToDevice, st));
        if (!pa->d_c) CUFSP_CUDA_TRY(cache_alloc((void **)&pa->d_c, sizeof(double) * nr));
        if (!pa->d_rterm) CUFSP_CUDA_TRY(cache_alloc((void **)&pa->d_rterm, sizeof(int) * nr * 2));
        if (!pa->d_d) CUFSP_CUDA_TRY(cache_alloc((void **)&pa->d_d, sizeof(int64_t) * nr));
        CUFSP_CUDA_TRY(cudaMemcpyAsync(pa->d_d, d.data(), sizeof(int64_t) * nr, cudaMemcpyHostToDevice, st));
        if (A->format == CUFSP_FORMAT_KRONECKER) {
            if (!pa->d_tables) CUFSP_CUDA_TRY(cache_alloc((void **)&pa->d_tables, sizeof(double) * m.tables.size()));
            CUFSP_CUDA_TRY(cudaMemcpyAsync(pa->d_tables, m.tables.data(), sizeof(double) * m.tables.size(),
                                           cudaMemcpyHostToDevice, st));
        }
    }
    TermBuildArgs b;
    std::memset(&b, 0, sizeof(b));
    b.n = n;
    b.ns = ns;
    b.nr = nr;
    b.T = T;
    b.transpose = transpose ? 1 : 0;
    b.tab_stride = m.tab_stride;
    for (int s = 0; s < ns; ++s) {
        b.dims[s] = m.bounds[s] + 1;
        b.tab_off[s] = m.tab_off.empty() ? 0 : m.tab_off[s];
    }
    if (A->format == CUFSP_FORMAT_KRONECKER) {
        b.tables = pa->d_tables;
    } else {
        if (!pa->d_props) CUFSP_CUDA_TRY(cache_alloc((void **)&pa->d_props, sizeof(double) * (size_t)nr * n));
        cufsp_status s = sparse_export(A->sparse, pa->d_props, st);
        if (s != CUFSP_SUCCESS) return s;
        b.props = pa->d_props;
    }
    // per-call coefficients and term map: small copies in stream order
    int *d_rt = pa->d_rterm + (transpose ? nr : 0);
    CUFSP_CUDA_TRY(cudaMemcpyAsync(pa->d_c, coefs.data(), sizeof(double) * nr, cudaMemcpyHostToDevice, st));
    CUFSP_CUDA_TRY(cudaMemcpyAsync(d_rt, rterm.data(), sizeof(int) * nr, cudaMemcpyHostToDevice, st));
    b.nu = pa->d_nu;
    b.c = pa->d_c;
    b.rterm = d_rt;
    b.d = pa->d_d;
    if (!tm.d_coef || tm.T < T) {
        cache_free(tm.d_coef);
        tm.d_coef = nullptr;
        CUFSP_CUDA_TRY(cache_alloc((void **)&tm.d_coef, sizeof(double) * (size_t)T * n));
    }
    b.coef = tm.d_coef;
    const int grid = stream_grid(n, 1, device_info().sm_count * 8);
    k_build_terms<<<grid, 256, 0, st>>>(b);
    CUFSP_CUDA_TRY(cudaGetLastError());
    // the copies above read pageable host memory: finish before `rterm` goes out of scope
    CUFSP_CUDA_TRY(cudaStreamSynchronize(st));
    pa->have_model = true;
    tm.coefs = coefs;
    tm.transpose = transpose;
    tm.T = T;
    tm.shift = shifts;
    return CUFSP_SUCCESS;
}

}  // namespace

namespace {
using PKernel = void (*)(const PArgs);
struct PVariant {
    PKernel kern;
    int threads, states, near, far;  // states per CTA, near and far terms it takes
};
// the first that fits is used; the last takes everything
#define CUFSP_PV(NS, TN, TF) {k_arnoldi_persistent<256, NS, TN, TF>, 256, 256 * NS, TN, TF}
const PVariant kPVariants[] = {CUFSP_PV(1, 4, 2), CUFSP_PV(1, 10, 4), CUFSP_PV(1, 4, 8), CUFSP_PV(2, 4, 2), CUFSP_PV(2, 10, 4),
                               CUFSP_PV(2, 4, 8), CUFSP_PV(4, 4, 2),  CUFSP_PV(4, 10, 4), CUFSP_PV(4, 4, 8),
                               {k_arnoldi_persistent<512, 1, 0, 0>, 512, INT32_MAX, kMaxTerms, kMaxTerms}};
#undef CUFSP_PV

cudaError_t persistent_smem_attribute() {
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
        for (const PVariant &v : kPVariants)
            if (result[dev] == cudaSuccess)
                result[dev] = cudaFuncSetAttribute((const void *)v.kern, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                                   (int)persistent_smem_max());
        done[dev] = true;
    }
    return result[dev];
}
}  // namespace

cufsp_status parnoldi_run(PArnoldi **ppa, cufsp_mat *A, const std::vector<double> &coefs, bool transpose,
                          int64_t n, const double *v, double *W, double *H, double *rho, double *beta,
                          double *avnorm, int *flag, int *err, int m, int iop, int q, double btol, bool with_avnorm,
                          double *h_state, int words, unsigned *h_seq, unsigned seq, cudaStream_t st) {
    if (!*ppa) *ppa = new PArnoldi();
    PArnoldi *pa = *ppa;
    PArnoldi::Terms *tm = nullptr;
    cufsp_status s = build_terms(pa, A, coefs, transpose, tm, st);
    if (s != CUFSP_SUCCESS) return s;
    if (!pa->grid) {
        // a host thread that shares the GPU with other solves (the batched gradient's workers) takes
        // its share of the SMs, so that the workers' cooperative passes run side by side
        const int64_t chunk = persistent_chunk(n, persistent_ctas());
        const int64_t grid = (n + chunk - 1) / chunk;
        const size_t row = sizeof(double) * (size_t)chunk, room = persistent_smem_max();
        if (n > INT32_MAX / 2) return set_error(CUFSP_ERR_UNSUPPORTED, "persistent Arnoldi: too many states");
        // basis vectors the dots read: W_0..W_{m-1}, or the last q of them
        const bool window = iop && q < m;
        const size_t fixed = persistent_fixed(chunk);
        if (fixed > room) return set_error(CUFSP_ERR_UNSUPPORTED, "persistent Arnoldi: vector slice exceeds shared memory");
        pa->slots = (int)std::min<size_t>((size_t)(window ? q : m), (room - fixed) / row);
        pa->ring = window && pa->slots == q ? q : 0;
        // The attribute belongs to the current device: set it once per device, to the most any
        // driver may ask for, so that drivers of different sizes on different host threads never
        // undercut each other.
        CUFSP_CUDA_TRY(persistent_smem_attribute());
        pa->smem = fixed + row * (size_t)pa->slots;
        for (const PVariant &v : kPVariants) {
            int per_sm = 0;
            CUFSP_CUDA_TRY(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, (const void *)v.kern, v.threads, pa->smem));
            if (per_sm < 1) return set_error(CUFSP_ERR_CUDA, "persistent Arnoldi: kernel does not fit an SM");
        }
        // exchange rows of one launch: K + 1 per iteration, two for the norms at the end
        int rows = 2;
        for (int j = 0; j < m; ++j) rows += (iop ? std::min(j + 1, q) : j + 1) + 1;
        pa->ex_rows = rows;
        const size_t bytes = sizeof(double) * 2 * (size_t)exchange_doubles(rows, (int)grid);
        CUFSP_CUDA_TRY(cache_alloc((void **)&pa->d_ex, bytes));
        pa->chunk = (int)chunk;
        pa->grid = (int)grid;
    }
    PArgs a;
    std::memset(&a, 0, sizeof(a));
    a.n = (int)n;
    a.chunk = pa->chunk;
    a.slots = pa->slots;
    a.ring = pa->ring;
    a.T = tm->T;
    a.coef = tm->d_coef;
    for (int t = 0; t < tm->T; ++t) a.shift[t] = (int)tm->shift[t];
    a.v0 = v;
    a.W = W;
    a.H = H;
    a.rho = rho;
    a.beta = beta;
    a.avnorm = avnorm;
    a.flag = flag;
    a.mp2 = m + 2;
    a.m = m;
    a.iop = iop;
    a.q = q;
    a.btol = btol;
    a.with_avnorm = with_avnorm ? 1 : 0;
    const size_t area = (size_t)exchange_doubles(pa->ex_rows, pa->grid);
    if (!pa->clean) {  // the first launch, or one after a launch that was refused, captured or broke off
        CUFSP_CUDA_TRY(cudaMemsetAsync(pa->d_ex, kUnsetByte, sizeof(double) * 2 * area, st));
        CUFSP_CUDA_TRY(cudaMemsetAsync(err, 0, sizeof(int), st));
    }
    pa->clean = false;  // until this one has reported (parnoldi_reported)
    a.ex = pa->d_ex + (size_t)pa->turn * area;
    a.ex_next = pa->d_ex + (size_t)(1 - pa->turn) * area;
    a.ex_rows = pa->ex_rows;
    a.waits = launch_waits(err);
    a.h_state = h_state;
    a.words = words;
    a.h_seq = h_seq;
    a.seq = seq;
    pa->turn = 1 - pa->turn;
    a.terms.n = (int)n;
    split_terms(a.T, a.shift, a.terms);
    const PVariant *var = kPVariants;
    while (a.chunk > var->states || a.terms.n_near > var->near || a.terms.n_far > var->far) ++var;
    void *args[] = {&a};
    CUFSP_CUDA_TRY(cudaLaunchCooperativeKernel((const void *)var->kern, dim3(pa->grid), dim3(var->threads), args, pa->smem, st));
    return CUFSP_SUCCESS;
}

}  // namespace cufsp
