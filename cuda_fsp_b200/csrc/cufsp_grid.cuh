// cufsp_grid.cuh -- data exchange between the co-resident CTAs of one cooperative launch, without
// grid barriers.
//
// A value that another CTA waits for is stored as one 8-byte word into a place that holds the bit
// pattern kUnset (all ones, a NaN that no arithmetic here produces); the reader polls the word itself
// until it differs.  The data is its own arrival flag, so an exchange costs one store and one L2 round
// trip: no arrival counter, no fence on the way out and no second read after the wait.  Every place is
// written once per launch and set back to kUnset by an earlier launch, or in the same launch before a
// fenced exchange.
//
// Waits are bounded (Waits::ns by the global timer): on expiry the error word is set, every waiting CTA
// sees it, and all CTAs leave.
#pragma once
#include <cuda_runtime.h>

#include <cstdlib>

namespace cufsp {

// What a wait is given: its error word and its limit.
struct Waits {
    int *err;               // set when a wait expired
    unsigned every;         // the limit is looked at every (every + 1) polls, a power of two
    unsigned long long ns;
};
// Of a launch: 0.3 s, or CUFSP_GRID_WAIT_NS (the tests of what follows an expired wait set 0: the second poll
// of a wait that finds nothing gives up).
inline Waits launch_waits(int *err) {
    const char *e = getenv("CUFSP_GRID_WAIT_NS");
    const unsigned long long ns = e && *e ? strtoull(e, nullptr, 10) : 300ull * 1000 * 1000;
    return Waits{err, ns ? 127u : 0u, ns};
}
constexpr int kUnsetByte = 0xff;  // memset value that makes every double kUnset

__device__ __forceinline__ unsigned long long global_ns() {
    unsigned long long t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}

__device__ __forceinline__ double ld_relaxed(const double *p) {
    double v;
    asm volatile("ld.relaxed.gpu.global.f64 %0, [%1];" : "=d"(v) : "l"(p));
    return v;
}

__device__ __forceinline__ double2 ld_relaxed2(const double *p) {
    double2 v;
    asm volatile("ld.relaxed.gpu.global.v2.f64 {%0, %1}, [%2];" : "=d"(v.x), "=d"(v.y) : "l"(p));
    return v;
}

__device__ __forceinline__ void st_relaxed(double *p, double v) {
    asm volatile("st.relaxed.gpu.global.f64 [%0], %1;" ::"l"(p), "d"(v));
}

__device__ __forceinline__ bool is_unset(double v) { return __double_as_longlong(v) == -1ll; }
__device__ __forceinline__ double unset_value() { return __longlong_as_double(-1ll); }
// v, with a NaN that happens to have the unset pattern replaced by another NaN
__device__ __forceinline__ double settled(double v) {
    return is_unset(v) ? __longlong_as_double(0x7ff8000000000000ll) : v;
}

// Bound of one thread's wait: give_up() counts a failed poll and is true once the wait has expired or
// another CTA has set the error word.
struct Patience {
    unsigned polls = 0;
    unsigned long long t0 = 0;
    __device__ __forceinline__ bool give_up(const Waits &w) {
        if ((++polls & w.every) != 0) return false;
        if (*(volatile int *)w.err) return true;
        const unsigned long long t = global_ns();
        if (polls == w.every + 1u) t0 = t;
        else if (t - t0 >= w.ns) {
            atomicExch(w.err, 1);
            return true;
        }
        return false;
    }
};

__device__ __forceinline__ double warp_sum(double v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

// Sums of d0..d3 over the warp in six 8-byte shuffles: lane 8 q holds the sum of d_q.
__device__ __forceinline__ double warp_sum4(double d0, double d1, double d2, double d3) {
    const int lane = threadIdx.x & 31;
    const bool hi = lane & 16, up = lane & 8;
    double a = hi ? d2 : d0, b = hi ? d3 : d1;
    a += __shfl_xor_sync(0xffffffffu, hi ? d0 : d2, 16);
    b += __shfl_xor_sync(0xffffffffu, hi ? d1 : d3, 16);
    double v = up ? b : a;
    v += __shfl_xor_sync(0xffffffffu, up ? a : b, 8);
    v += __shfl_xor_sync(0xffffffffu, v, 4);
    v += __shfl_xor_sync(0xffffffffu, v, 2);
    v += __shfl_xor_sync(0xffffffffu, v, 1);
    return v;
}

// ---- all-to-all sums -----------------------------------------------------------------------------
// One exchange sums `rows` values over the CTAs of the grid.  Every CTA stores its partial of row r at
// ex[r * pitch + CTA]; one CTA per row (its owner) polls the row, sums it in a fixed order and stores
// the total into kCopies places, and every CTA polls the totals from the copy of its own.  Two hops of
// one store and one L2 read each.  Polling all partials in every CTA (one hop) measured 3x slower at 148
// CTAs and 31 rows: 148 pollers on each of the 310 lines queue up in L2.
constexpr int kCopies = 8;
constexpr int kMaxGridPairs = 3;  // double2 loads per lane that cover one row: up to 192 CTAs

__host__ __device__ inline int exchange_pitch(int grid) { return (grid + 1) & ~1; }
// doubles of an exchange area that holds `rows` rows in all
__host__ __device__ inline int exchange_doubles(int rows, int grid) { return rows * (exchange_pitch(grid) + kCopies); }

// Owner's part, one warp per owned row: rows are dealt to CTAs, then to warps [w0, warps) of a CTA.
// `row` is the number of the exchange's first row in the area, `all` the area's rows.  With `fence`,
// what a CTA wrote and fenced before it published is visible to whoever has read a total and fenced.
__device__ __forceinline__ bool exchange_own(double *area, int all, int row, int rows, int w0, int warps, bool fence,
                                             const Waits &waits) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, G = (int)gridDim.x;
    const int pitch = exchange_pitch(G);
    bool ok = true;
    if (warp < w0) return true;
#pragma unroll 1
    for (int r = (int)blockIdx.x + (warp - w0) * G; r < rows; r += (warps - w0) * G) {
        const double *p = area + (size_t)(row + r) * pitch;
        double2 v[kMaxGridPairs];
        Patience w;
        do {
            bool miss = false;
#pragma unroll
            for (int i = 0; i < kMaxGridPairs; ++i) {
                const int b = 2 * lane + 64 * i;
                v[i] = make_double2(0.0, 0.0);
                if (b < G) v[i] = ld_relaxed2(p + b);
                if (b + 1 >= G) v[i].y = 0.0;
                miss = miss || is_unset(v[i].x) || is_unset(v[i].y);
            }
            if (!miss) break;
            ok = !w.give_up(waits);
        } while (ok);
        double s = 0.0;
#pragma unroll
        for (int i = 0; i < kMaxGridPairs; ++i) s += v[i].x + v[i].y;
        s = settled(warp_sum(s));
        ok = __all_sync(0xffffffffu, ok);
        if (fence) __threadfence();
        if (ok && lane < kCopies) st_relaxed(area + (size_t)all * pitch + (size_t)lane * all + row + r, s);
    }
    return ok;
}

// Total of row `r` (< rows) of the exchange, from this CTA's copy.
__device__ __forceinline__ bool exchange_total(const double *area, int all, int row, int r, const Waits &waits, double &v) {
    const double *p = area + (size_t)all * exchange_pitch((int)gridDim.x) + (size_t)(blockIdx.x % kCopies) * all + row + r;
    Patience w;
    for (v = ld_relaxed(p); is_unset(v); v = ld_relaxed(p))
        if (w.give_up(waits)) return false;
    return true;
}

}  // namespace cufsp
