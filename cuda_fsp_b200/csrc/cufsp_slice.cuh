// cufsp_slice.cuh -- generator action and dot products of a CTA that owns a contiguous slice of the
// states and keeps it in shared memory (persistent Arnoldi pass, BDF step).
//
// The generator is a sum of terms (A x)[i] = sum_t coef_t[i] x[i - shift_t], coefficients in registers.
// Near terms (|shift| <= halo) read x from the slice in shared memory, extended on both sides by a halo
// of the neighbours' entries; far terms read it from L2, all loads of a thread in flight together.
// Entries that another CTA owns are polled until they have been stored (cufsp_grid.cuh).
#pragma once
#include "cufsp_grid.cuh"

namespace cufsp {

constexpr int kHaloMax = 64;  // largest |shift| of a near term
constexpr int kMaxNear = 10, kMaxFar = 8;

struct SliceTerms {
    int n;                       // states
    int n_near, n_far, halo;     // halo: largest near |shift|, rounded up to even
    int near_shift[kMaxNear], far_shift[kMaxFar];
    short near_t[kMaxNear], far_t[kMaxFar];  // their numbers in the caller's list
};

// Splits a list of shifts; n_near / n_far count all of them, also past the arrays' ends.
inline void split_terms(int T, const int *shift, SliceTerms &s) {
    s.n_near = s.n_far = s.halo = 0;
    for (int t = 0; t < T; ++t) {
        const int d = shift[t] < 0 ? -shift[t] : shift[t];
        if (d <= kHaloMax) {
            if (s.n_near < kMaxNear) {
                s.near_shift[s.n_near] = shift[t];
                s.near_t[s.n_near] = (short)t;
            }
            ++s.n_near;
            if (d > s.halo) s.halo = d;
        } else {
            if (s.n_far < kMaxFar) {
                s.far_shift[s.n_far] = shift[t];
                s.far_t[s.n_far] = (short)t;
            }
            ++s.n_far;
        }
    }
    s.halo = (s.halo + 1) & ~1;
}

#if defined(__CUDACC__)

// x[lo + rel], the index clamped to the vector (a term whose source is outside has coefficient 0)
__device__ __forceinline__ double far_entry(const double *x, int lo, int rel, int n) {
    return ld_relaxed(x + min(max(lo + rel, 0), n - 1));
}

// First half of a generator action by NT threads: starts the far loads of the thread's states tid, tid +
// NT, .. and fetches the halo into xs (the slice, xs[-halo .. len + halo)).  poll: entries may not have been
// stored yet.  False when a wait expired.
// EDGES false: by the first 2 halo threads; a block barrier must follow.  EDGES true: by the warps whose states
// lie within the halo of an end, each for itself (two may fetch the same entries: the same values), so that
// the others go on to their sums without a barrier.  A BDF step of the 131,072-state gene model takes 87.6 us
// so and 90.5 us with the barrier; an Arnoldi pass gains nothing (134,088 states: 5.96 and 5.97 ms a solve)
// or loses (32,768 states: 5.70 and 5.50 ms), its 7 or 8 warps then poll for far entries all the earlier.
template <int NT, int NS, int TF, bool EDGES>
__device__ __forceinline__ bool gather_begin(const SliceTerms &a, const double *x, int lo, int len, bool poll, double *xs,
                                             double (&v)[NS][TF], const Waits &waits) {
    const int tid = threadIdx.x, lane = tid & 31;
    bool ok = true;
#pragma unroll
    for (int s = 0; s < NS; ++s)
#pragma unroll
        for (int t = 0; t < TF; ++t) {
            v[s][t] = 0.0;
            if (t < a.n_far && s * NT < len) v[s][t] = far_entry(x, lo, tid + s * NT - a.far_shift[t], a.n);
        }
    auto fetch = [&](int e, Patience &wait) {  // halo entry e: the left ones first
        const int rel = e < a.halo ? e - a.halo : len + e - a.halo;
        double h = far_entry(x, lo, rel, a.n);
        while (poll && is_unset(h)) {
            if (wait.give_up(waits)) {
                ok = false;
                break;
            }
            h = far_entry(x, lo, rel, a.n);
        }
        xs[rel] = h;
    };
    Patience wait;
    if constexpr (EDGES) {
        const bool left = tid - lane < a.halo;
        bool right = false;
#pragma unroll
        for (int s = 0; s < NS; ++s) {
            const int base = s * NT + tid - lane;
            right = right || (base < len && base + 32 + a.halo > len);
        }
        if (left || right) {
#pragma unroll 1
            for (int e = lane; e < 2 * a.halo; e += 32)
                if (e < a.halo ? left : right) fetch(e, wait);
            __syncwarp();
        }
    } else {
        if (tid < 2 * a.halo) fetch(tid, wait);
    }
    return ok;
}

// Second half: w[s] = (A x)[lo + tid + s NT] from the near and far coefficients, 0 past the slice.
template <int NT, int NS, int TN, int TF>
__device__ __forceinline__ bool gather_end(const SliceTerms &a, const double *x, int lo, int len, bool poll,
                                           const double *xs, const double (&cn)[NS][TN], const double (&cf)[NS][TF],
                                           double (&v)[NS][TF], double (&w)[NS], const Waits &waits) {
    const int tid = threadIdx.x;
    bool ok = true;
#pragma unroll
    for (int s = 0; s < NS; ++s) w[s] = 0.0;
#pragma unroll
    for (int t = 0; t < TN; ++t) {
        if (t >= a.n_near) break;
        const double *p = xs + tid - a.near_shift[t];
#pragma unroll
        for (int s = 0; s < NS; ++s)
            if (tid + s * NT < len) w[s] = fma(cn[s][t], p[s * NT], w[s]);
    }
    if (poll) {
        Patience wait;
        for (;;) {
            bool miss = false;
#pragma unroll
            for (int s = 0; s < NS; ++s)
#pragma unroll
                for (int t = 0; t < TF; ++t)
                    if (is_unset(v[s][t])) {
                        miss = true;
                        v[s][t] = far_entry(x, lo, tid + s * NT - a.far_shift[t], a.n);
                    }
            if (!miss) break;
            if (wait.give_up(waits)) {
                ok = false;
                break;
            }
        }
    }
#pragma unroll
    for (int s = 0; s < NS; ++s) {
#pragma unroll
        for (int t = 0; t < TF; ++t) w[s] = fma(cf[s][t], v[s][t], w[s]);
        if (tid + s * NT >= len) w[s] = 0.0;
    }
    return ok;
}

// Dot products of the slice ws with K slices by the first NW = 2^LNW warps: a warp takes four of them and
// one part of the slice, so that each entry of ws is read once for four products.  Slices r < Kres are in
// shared memory at base + r chunk, the others in global memory at g0 (r = 0) or gbase + r n.  chunk is
// even; the slices in shared memory are zero past len.  A block barrier, then dots_sum, must follow.
template <int LNW>
__device__ __forceinline__ void slice_dots(const double *ws, int chunk, int len, int K, int Kres, const double *base,
                                           const double *g0, const double *gbase, int n, double (*part)[4]) {
    constexpr int NW = 1 << LNW;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int lnb = K > 32 ? 4 : K > 16 ? 3 : K > 8 ? 2 : K > 4 ? 1 : 0, nb = 1 << lnb;
    const int nsl = NW >> lnb;  // parts (0: more groups of four than warps)
#pragma unroll 1
    for (int r0 = (warp & (nb - 1)) * 4, at = warp; r0 < K; r0 += 4 * NW, at += NW) {
        const int half = chunk >> 1, per = nsl > 1 ? (half + nsl - 1) >> (LNW - lnb) : half;
        const int b0 = nsl > 1 ? (warp >> lnb) * per : 0, b1 = min(half, b0 + per);
        const int q1 = min(r0 + 1, K - 1), q2 = min(r0 + 2, K - 1), q3 = min(r0 + 3, K - 1);
        double d0 = 0.0, d1 = 0.0, d2 = 0.0, d3 = 0.0;
        if (q3 < Kres) {
            const double2 *p0 = reinterpret_cast<const double2 *>(base + r0 * chunk);
            const double2 *p1 = reinterpret_cast<const double2 *>(base + q1 * chunk);
            const double2 *p2 = reinterpret_cast<const double2 *>(base + q2 * chunk);
            const double2 *p3 = reinterpret_cast<const double2 *>(base + q3 * chunk);
            const double2 *pw = reinterpret_cast<const double2 *>(ws);
#pragma unroll 2
            for (int b = b0 + lane; b < b1; b += 32) {
                const double2 u = pw[b], u0 = p0[b], u1 = p1[b], u2 = p2[b], u3 = p3[b];
                d0 = fma(u0.y, u.y, fma(u0.x, u.x, d0));
                d1 = fma(u1.y, u.y, fma(u1.x, u.x, d1));
                d2 = fma(u2.y, u.y, fma(u2.x, u.x, d2));
                d3 = fma(u3.y, u.y, fma(u3.x, u.x, d3));
            }
        } else {
            const double *p0 = r0 == 0 ? g0 : gbase + (size_t)r0 * n;
            const double *p1 = gbase + (size_t)q1 * n, *p2 = gbase + (size_t)q2 * n, *p3 = gbase + (size_t)q3 * n;
            if (q1 == 0) p1 = p2 = p3 = p0;  // K = 1
#pragma unroll 4
            for (int il = 2 * b0 + lane; il < min(len, 2 * b1); il += 32) {
                const double u = ws[il];
                d0 = fma(__ldcg(p0 + il), u, d0);
                d1 = fma(__ldcg(p1 + il), u, d1);
                d2 = fma(__ldcg(p2 + il), u, d2);
                d3 = fma(__ldcg(p3 + il), u, d3);
            }
        }
        d0 = warp_sum4(d0, d1, d2, d3);
        if ((lane & 7) == 0) part[at][lane >> 3] = d0;
    }
}

// Dot product k (< K) from the parts, in a fixed order.
template <int LNW>
__device__ __forceinline__ double dots_sum(const double (*part)[4], int K, int k) {
    const int lnb = K > 32 ? 4 : K > 16 ? 3 : K > 8 ? 2 : K > 4 ? 1 : 0, nsl = (1 << LNW) >> lnb;
    double v = part[k >> 2][k & 3];
#pragma unroll 4
    for (int u = 1; u < nsl; ++u) v += part[(u << lnb) + (k >> 2)][k & 3];
    return v;
}

#endif  // __CUDACC__

}  // namespace cufsp
