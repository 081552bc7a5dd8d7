// Vrms of the output points assembled on the GPU (sm_100a).
//
// The reference's providers are CPU loops (src/velocity_reader.cpp): the text table blends
// every table point into every sample (:320-361), O(points) per sample; an off-grid SEG-Y Vrms
// blends the 2x2 label neighbours (:93-163) and interpolates in time (:124-138, :184-196).
// Here one thread computes one sample (il, xl, t) of the dense Vrms cube with the same
// operations in the same order: double products and sums with explicit round-to-nearest
// intrinsics (the host build has no fused multiply-add), float weights 1 / (1 + float(d)),
// float accumulation in source order.  The result equals the host providers' bit for bit
// (their distance to the reference's -ffast-math build, which reorders those sums, is 1-2 ulp).
#pragma once

#include <cstdint>
#include <cuda_runtime.h>

namespace psm {

constexpr int kTableThreads = 128;  // samples of a work item
constexpr int kTablePoints = 64;    // table points staged in shared memory at a time

// float(sqrt(x)) for the double x, as rounding to double first and to float then gives it; clears
// *sure when the caller has to take the exact root.  Two Newton steps from an approximate
// 1 / sqrt(x) (off by 2^-19 at the worst) leave 4 units of the double's last place at most, so
// float(s) is the wanted float unless s lies about the middle between two floats (32 units
// here), or x is too small (an exact hit may be) or large for the steps.
__device__ __forceinline__ float root_to_float(double x, bool* sure) {
    double q;
    asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(q) : "d"(x));
    const double h = __dmul_rn(0.5, q), y = __dmul_rn(x, q);
    const double r = __fma_rn(__fma_rn(-y, y, x), h, y);
    const double s = __fma_rn(__fma_rn(-r, r, x), h, r);
    constexpr unsigned kMiddle = 1u << 28, kNear = 32u;
    constexpr unsigned kLo = 0x3c400000u, kHi = 0x47000000u;  // high words of 2^-59 and 2^113
    const unsigned low = static_cast<unsigned>(__double2loint(s)) & (2u * kMiddle - 1u);
    *sure &= (low - (kMiddle - kNear) > 2u * kNear) &
             (static_cast<unsigned>(__double2hiint(x)) - kLo < kHi - kLo);
    return __double2float_rn(s);
}

// One table point's share of the weighted sums, at squared distance x: with the fast root (*sure as
// above), and with the exact one, which is true for an exact hit.
__device__ __forceinline__ void blend_fast(double x, float v, float& sv, float& sw, bool* sure) {
    const float w = __frcp_rn(__fadd_rn(1.0f, root_to_float(x, sure)));
    sv = __fadd_rn(sv, __fmul_rn(v, w));
    sw = __fadd_rn(sw, w);
}
__device__ __forceinline__ bool blend_exact(double x, float v, float& sv, float& sw) {
    const double d = __dsqrt_rn(x);
    if (d < 1e-10) return true;
    const float w = __fdiv_rn(1.0f, __fadd_rn(1.0f, __double2float_rn(d)));
    sv = __fadd_rn(sv, __fmul_rn(v, w));
    sw = __fadd_rn(sw, w);
    return false;
}
__device__ __forceinline__ float blend_result(bool hit, float hit_v, float sv, float sw,
                                              float vmin) {
    if (hit) return hit_v;
    const float r = sw > 0.0f ? __fdiv_rn(sv, sw) : vmin;
    return r <= 0.0f ? vmin : r;
}

// Text-table Vrms: every point (il, xl, time, v) weighted by 1 / (1 + dist) with dist mixing
// label units and seconds; an exact hit (dist < 1e-10) returns that point's v; a result <= 0
// (or no weight) gives vmin.  out [n_il][n_xl][n_t], t0 = t * dt.
//
// Bound by instructions, some 45 per point and sample (84% of the issue slots).  A work item is
// kTableThreads samples of one trace; the label part of the squared distances is summed once per
// item and point; a thread whose root_to_float was not sure of one of the staged points (an
// exact hit, or 1 in 2^23) takes those points again with the exact root.
// 81 x 93 x 626 samples, 54 points: 659 us with the exact root and divide everywhere, 466 us with
// a branch to the exact root per point (and one Newton step), 397 us so.
__global__ void __launch_bounds__(kTableThreads)
vrms_table_kernel(const int32_t* __restrict__ p_il, const int32_t* __restrict__ p_xl,
                  const double* __restrict__ p_time, const float* __restrict__ p_v, int n_points,
                  float vmin, const int32_t* __restrict__ il, const int32_t* __restrict__ xl,
                  int n_il, int n_xl, int n_t, double dt, float* __restrict__ out) {
    __shared__ double2 at[kTablePoints];  // label part of the squared distance, time
    __shared__ float vel[kTablePoints];
    const int n_seg = (n_t + kTableThreads - 1) / kTableThreads;
    const int64_t n_items = static_cast<int64_t>(n_il) * n_xl * n_seg;
    for (int64_t item = blockIdx.x; item < n_items; item += gridDim.x) {
        const int64_t tr = item / n_seg;
        const int t = static_cast<int>(item % n_seg) * kTableThreads + threadIdx.x;
        const int32_t a_il = il[tr / n_xl], a_xl = xl[tr % n_xl];
        const double time = __dmul_rn(static_cast<double>(t), dt);
        float sv = 0.0f, sw = 0.0f, hit_v = 0.0f;
        bool hit = false;
        for (int base = 0; base < n_points; base += kTablePoints) {
            const int cnt = min(kTablePoints, n_points - base);
            __syncthreads();  // the readers of the points before these
            for (int p = threadIdx.x; p < cnt; p += kTableThreads) {
                const double a = fabs(static_cast<double>(p_il[base + p] - a_il));
                const double b = fabs(static_cast<double>(p_xl[base + p] - a_xl));
                at[p] = make_double2(__dadd_rn(__dmul_rn(a, a), __dmul_rn(b, b)),
                                     p_time[base + p]);
                vel[p] = p_v[base + p];
            }
            __syncthreads();
            if (t >= n_t || hit) continue;
            const float v0 = sv, w0 = sw;
            bool sure = true;
#pragma unroll 2
            for (int p = 0; p < cnt; ++p) {
                const double2 u = at[p];
                const double c = __dsub_rn(u.y, time);
                blend_fast(__dadd_rn(u.x, __dmul_rn(c, c)), vel[p], sv, sw, &sure);
            }
            if (sure) continue;
            sv = v0;  // again, with the exact root
            sw = w0;
#pragma unroll 1
            for (int p = 0; p < cnt; ++p) {
                const double2 u = at[p];
                const double c = __dsub_rn(u.y, time);
                if (blend_exact(__dadd_rn(u.x, __dmul_rn(c, c)), vel[p], sv, sw)) {
                    hit = true;
                    hit_v = vel[p];
                    break;
                }
            }
        }
        if (t >= n_t) continue;
        out[tr * n_t + t] = blend_result(hit, hit_v, sv, sw, vmin);
    }
}

// The same for a table of few points or traces that leave a work item's threads without samples: a
// thread per sample, which reads the points from global memory and sums their label parts itself.
__global__ void vrms_table_flat_kernel(const int32_t* __restrict__ p_il,
                                       const int32_t* __restrict__ p_xl,
                                       const double* __restrict__ p_time,
                                       const float* __restrict__ p_v, int n_points, float vmin,
                                       const int32_t* __restrict__ il,
                                       const int32_t* __restrict__ xl, int n_il, int n_xl,
                                       int n_t, double dt, float* __restrict__ out) {
    const int64_t n = static_cast<int64_t>(n_il) * n_xl * n_t;
    for (int64_t k = blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x; k < n;
         k += static_cast<int64_t>(gridDim.x) * blockDim.x) {
        const int64_t tr = k / n_t;
        const int32_t a_il = il[tr / n_xl], a_xl = xl[tr % n_xl];
        const double time = __dmul_rn(static_cast<double>(static_cast<int>(k - tr * n_t)), dt);
        auto square = [&](int p) {
            const double a = fabs(static_cast<double>(p_il[p] - a_il));
            const double b = fabs(static_cast<double>(p_xl[p] - a_xl));
            const double c = __dsub_rn(p_time[p], time);
            return __dadd_rn(__dadd_rn(__dmul_rn(a, a), __dmul_rn(b, b)), __dmul_rn(c, c));
        };
        float sv = 0.0f, sw = 0.0f, hit_v = 0.0f;
        bool hit = false, sure = true;
        for (int p = 0; p < n_points; ++p) blend_fast(square(p), p_v[p], sv, sw, &sure);
        if (!sure) {  // again, with the exact root
            sv = sw = 0.0f;
            for (int p = 0; p < n_points && !hit; ++p) {
                hit = blend_exact(square(p), p_v[p], sv, sw);
                if (hit) hit_v = p_v[p];
            }
        }
        out[k] = blend_result(hit, hit_v, sv, sw, vmin);
    }
}

// Linear interpolation in time of a grid trace, clamped at both ends.
__device__ __forceinline__ float grid_in_time(const float* tr, int g_nt, double gdt, double time) {
    if (time <= 0.0) return tr[0];
    if (time >= __dmul_rn(static_cast<double>(g_nt - 1), gdt)) return tr[g_nt - 1];
    const double s = __ddiv_rn(time, gdt);
    const int lo = static_cast<int>(s);
    if (lo >= g_nt - 1) return tr[g_nt - 1];
    const double fr = __dsub_rn(s, static_cast<double>(lo));
    return __double2float_rn(__dadd_rn(__dmul_rn(static_cast<double>(tr[lo]), __dsub_rn(1.0, fr)),
                                       __dmul_rn(static_cast<double>(tr[lo + 1]), fr)));
}

// Index of the label nearest to x in the sorted labels v (ties to the lower one).
__device__ __forceinline__ int nearest_label(const int32_t* v, int n, int32_t x) {
    int lo = 0, hi = n;  // first index with v[i] >= x
    while (lo < hi) {
        const int mid = (lo + hi) >> 1;
        if (v[mid] < x)
            lo = mid + 1;
        else
            hi = mid;
    }
    if (lo == 0) return 0;
    if (lo == n) return n - 1;
    return abs(v[lo] - x) < abs(v[lo - 1] - x) ? lo : lo - 1;
}

// SEG-Y-grid Vrms: grid [g_nil][g_nxl][g_nt] on sorted labels (missing traces zero), sample
// interval gdt.  A point on a grid inline and crossline copies its trace (same dt and n_t) or
// interpolates it in time; any other point blends the 4 neighbours one label below and above
// the nearest grid labels with weights 1 / (1 + |dIL| + |dXL|).
__global__ void vrms_grid_kernel(const float* __restrict__ grid, const int32_t* __restrict__ g_il,
                                 int g_nil, const int32_t* __restrict__ g_xl, int g_nxl, int g_nt,
                                 double gdt, const int32_t* __restrict__ il,
                                 const int32_t* __restrict__ xl, int n_il, int n_xl, int n_t,
                                 double dt, float* __restrict__ out) {
    const int64_t n = static_cast<int64_t>(n_il) * n_xl * n_t;
    const bool same_axis = fabs(dt - gdt) < 1e-6 && n_t == g_nt;
    for (int64_t k = blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x; k < n;
         k += static_cast<int64_t>(gridDim.x) * blockDim.x) {
        const int t = static_cast<int>(k % n_t);
        const int64_t tr = k / n_t;
        const int32_t a_il = il[tr / n_xl], a_xl = xl[tr % n_xl];
        const double time = __dmul_rn(static_cast<double>(t), dt);
        const int ii = nearest_label(g_il, g_nil, a_il), xi = nearest_label(g_xl, g_nxl, a_xl);
        float r;
        if (g_il[ii] == a_il && g_xl[xi] == a_xl) {
            const float* trc = grid + (static_cast<int64_t>(ii) * g_nxl + xi) * g_nt;
            r = same_axis ? trc[t] : grid_in_time(trc, g_nt, gdt, time);
        } else {
            const int is[2] = {ii > 0 ? ii - 1 : 0, ii < g_nil - 1 ? ii + 1 : g_nil - 1};
            const int xs[2] = {xi > 0 ? xi - 1 : 0, xi < g_nxl - 1 ? xi + 1 : g_nxl - 1};
            float sv = 0.0f, sw = 0.0f, v0 = 0.0f;
            for (int p = 0; p < 2; ++p)
                for (int q = 0; q < 2; ++q) {
                    const float* trc = grid + (static_cast<int64_t>(is[p]) * g_nxl + xs[q]) * g_nt;
                    const float val = grid_in_time(trc, g_nt, gdt, time);
                    if (p == 0 && q == 0) v0 = val;
                    const double d_il = fabs(static_cast<double>(g_il[is[p]] - a_il));
                    const double d_xl = fabs(static_cast<double>(g_xl[xs[q]] - a_xl));
                    const float w =
                        __fdiv_rn(1.0f, __fadd_rn(1.0f, __double2float_rn(__dadd_rn(d_il, d_xl))));
                    sv = __fadd_rn(sv, __fmul_rn(val, w));
                    sw = __fadd_rn(sw, w);
                }
            r = sw > 0.0f ? __fdiv_rn(sv, sw) : v0;
        }
        out[k] = r;
    }
}

}  // namespace psm
