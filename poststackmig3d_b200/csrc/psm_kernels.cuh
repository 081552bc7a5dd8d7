// Device code of the B200 Kirchhoff post-stack 3D time migration (sm_100a).
//
// The operator is the reference's diffraction summation (sergeevsn/poststackmig3d,
// src/migration_kernel.cpp:17-383): for every output sample (inline c, crossline x, time t0)
//     out = sum over input traces (i, k) with r^2 = dx^2 + dy^2 <= (v t0 / 2)^2 tan^2(theta)
//           and floor(t / dt) < n_t - 1 of  interp(trace(i,k), t / dt) / (t v^2)
// with t = sqrt(t0^2 + 4 r^2 / v^2), v the output point's Vrms, interp the linear rule
// fma(frac, d[lo+1] - d[lo], d[lo]) (simdInterpolate, :544-550).
//
// This header holds what the forward (psm_forward.cuh) and adjoint (psm_adjoint.cuh) kernels
// share: parameters, PTX helpers, the per-sample constants and the exact masks, trace storage
// and the term count.
//
// HBM layout: traces are [inline][crossline][ns], ns a multiple of 8 samples above n_t with a
// zero tail: fp32 values, or 16-bit values d / scale with one fp32 scale per trace.
//
// Masks: a term passes the reference's aperture and range masks exactly when r^2 <= B, B a
// per-sample bound found once with the reference's IEEE arithmetic (pass_bound).
// Every wait is bounded: on expiry the kernel records PSM_DEV_ERR_TIMEOUT in *err and leaves.
#pragma once

#include <cstdint>
#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <cuda_runtime.h>

namespace psm {

constexpr int kStages = 2;      // ring depth
// mbarrier waits end after FwdParams::wait_us of %globaltimer time (kDefaultWaitUs when 0),
// or after kWaitPollCap polls, whichever comes first
constexpr unsigned kDefaultWaitUs = 4000000u;
constexpr unsigned kWaitPollCap = 1u << 30;
// FwdParams::fault: test-only failure injection, 0 in normal runs.  kFaultStallProducer: the
// producer never arrives on (and issues no copy into) the first stage of its tile, so the
// consumers' bounded wait on it runs out and the launch reports PSM_DEV_ERR_TIMEOUT.
constexpr int kFaultStallProducer = 1;

// Trace storage in HBM: fp32 samples, 16-bit samples (bf16 / fp16 values d / scale with one
// fp32 scale per trace), or the pairs (d[t], d[t+1] - d[t]) of psm_forward_noalloc's callers,
// of which the first member is read.
constexpr int kStoreF32 = 0;
constexpr int kStoreBF16 = 1;
constexpr int kStoreF16 = 2;
constexpr int kStorePairs = 3;
__host__ __device__ constexpr int store_bytes(int store) {
    return store == kStorePairs ? 8 : store == kStoreF32 ? 4 : 2;
}

constexpr int PSM_DEV_ERR_TIMEOUT = 1;
constexpr int PSM_DEV_ERR_WINDOW = 2;  // debug-bounds build (PSM_DEBUG_BOUNDS) only

// One output inline of a launch.
struct Job {
    int row;   // output image row
    int vrow;  // Vrms plane (cube inline of the output point's velocity)
    int pos;   // inline position of the output point (dx = (il_pos[i] - pos) * d_il)
    int i0;    // cube inlines [i0, i1) form the buffer (migration_kernel.cpp:404-409)
    int i1;
};

struct FwdParams {
    const void* traces;   // [n_ci][n_cx][ns] samples of `store`; rows 16 B aligned
    const float* scales;  // [n_ci][n_cx] 16-bit storage: d = q * scale
    const float* vrms;    // Vrms of the output points: (vrow, x, t) at vrow vs_row + x vs_x + t
    long long vs_row, vs_x;  // element strides ([n_vrow][n_vx][n_t]; 0 broadcasts one trace)
    float* image;         // [rows][n_ox][n_t]
    const Job* jobs;
    const int* il_pos;    // [n_ci] inline positions
    const float* t0;      // [n_t]
    int* err;
    unsigned wait_us;  // limit of every mbarrier wait in microseconds (0: kDefaultWaitUs)
    int fault;         // test-only failure injection (kFault*), 0 normally
    int compat_pad;    // trailing padded crosslines take the last real crossline's Vrms
    int store;         // kStore* of `traces`
    int n_ci, n_cx, n_t, ns;
    int n_vx;             // crosslines of a Vrms plane
    int n_ox;             // output crosslines per row
    int xoff;             // cube / Vrms crossline of output x is x + xoff
    int max_inl;          // largest i1 - i0 over the jobs (the adjoint's inline tables)
    int max_rows;         // most rows of a trace list over the jobs (the forward's row tables)
    int stage_cap;        // adjoint: samples per ring stage
    int pairable;         // il_pos consecutive: mirrored inlines c - d, c + d can be paired
    float inv_dt, idt2, d_il, d_xl, inv_dxl, tan2, tanth;
    float ntm1f;          // n_t - 1
    float ntm1m;          // largest float below n_t - 1
};

struct TileStats {
    float vmin, vmax, bmax, t0min, t0max;
    int any;
};

// ----------------------------------------------------------------------------- PTX helpers

__device__ __forceinline__ uint32_t smem_u32(const void* p) {
    return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}

__device__ __forceinline__ void mbar_init(uint64_t* bar, uint32_t count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count)
                 : "memory");
}

__device__ __forceinline__ void fence_barrier_init() {
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}

__device__ __forceinline__ void mbar_arrive(uint64_t* bar) {
    asm volatile(
        "{\n\t.reg .b64 st;\n\t"
        "mbarrier.arrive.release.cta.shared::cta.b64 st, [%0];\n\t}" ::"r"(smem_u32(bar))
        : "memory");
}

__device__ __forceinline__ void mbar_arrive_expect_tx(uint64_t* bar, uint32_t bytes) {
    asm volatile(
        "{\n\t.reg .b64 st;\n\t"
        "mbarrier.arrive.expect_tx.release.cta.shared::cta.b64 st, [%0], %1;\n\t}" ::"r"(
            smem_u32(bar)),
        "r"(bytes)
        : "memory");
}

__device__ __forceinline__ bool mbar_try_wait(uint64_t* bar, uint32_t parity) {
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.acquire.cta.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok)
        : "r"(smem_u32(bar)), "r"(parity)
        : "memory");
    return ok != 0;
}

__device__ __forceinline__ unsigned long long global_ns() {
    unsigned long long t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}

// Bounded wait: false (and *err set) once limit_us (0: kDefaultWaitUs) microseconds of
// globaltimer time have passed without the phase completing (the clock is read every 64
// polls; kWaitPollCap polls at most).
__device__ __forceinline__ bool mbar_wait(uint64_t* bar, uint32_t parity, int* err,
                                          unsigned limit_us) {
    if (mbar_try_wait(bar, parity)) return true;
    const unsigned long long lim = 1000ull * (limit_us ? limit_us : kDefaultWaitUs);
    const unsigned long long start = global_ns();
    for (unsigned it = 1; it < kWaitPollCap; ++it) {
        if (mbar_try_wait(bar, parity)) return true;
        if ((it & 63u) == 0 && global_ns() - start > lim) break;
    }
    atomicOr(err, PSM_DEV_ERR_TIMEOUT);
    return false;
}

// TMA bulk copy global -> shared, completion counted on an mbarrier (bytes % 16 == 0,
// both addresses 16 B aligned).
__device__ __forceinline__ void tma_load_1d(uint32_t dst_smem, const void* src, uint32_t bytes,
                                            uint64_t* bar) {
    asm volatile(
        "cp.async.bulk.shared::cta.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::
            "r"(dst_smem),
        "l"(src), "r"(bytes), "r"(smem_u32(bar))
        : "memory");
}

// packed FP32 pairs (sm_100 f32x2 arithmetic)
__device__ __forceinline__ unsigned long long pk(float2 v) {
    unsigned long long r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(v.x), "f"(v.y));
    return r;
}
__device__ __forceinline__ float2 upk(unsigned long long r) {
    float2 v;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(v.x), "=f"(v.y) : "l"(r));
    return v;
}
__device__ __forceinline__ float2 fma2(float2 a, float2 b, float2 c) {
    unsigned long long r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(pk(a)), "l"(pk(b)), "l"(pk(c)));
    return upk(r);
}
__device__ __forceinline__ float2 mul2(float2 a, float2 b) {
    unsigned long long r;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(pk(a)), "l"(pk(b)));
    return upk(r);
}
__device__ __forceinline__ float2 add2(float2 a, float2 b) {
    unsigned long long r;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(pk(a)), "l"(pk(b)));
    return upk(r);
}
__device__ __forceinline__ float2 add2_rm(float2 a, float2 b) {  // rounding toward -inf
    unsigned long long r;
    asm("add.rm.f32x2 %0, %1, %2;" : "=l"(r) : "l"(pk(a)), "l"(pk(b)));
    return upk(r);
}
__device__ __forceinline__ float2 sub2(float2 a, float2 b) {
    unsigned long long r;
    asm("sub.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(pk(a)), "l"(pk(b)));
    return upk(r);
}

__device__ __forceinline__ float warp_max(float v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, o));
    return v;
}
__device__ __forceinline__ float warp_min(float v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v = fminf(v, __shfl_xor_sync(0xffffffffu, v, o));
    return v;
}

// ----------------------------------------------------------------------------- point setup

// Vrms trace of output point (vrow, xv).
__device__ __forceinline__ const float* vrms_trace(const FwdParams& P, int vrow, int xv) {
    return P.vrms + vrow * P.vs_row + xv * P.vs_x;
}

// Vrms crossline of output crossline x (cube crossline xv = x + xoff), or -1 when the point
// has none: padded crosslines have v = 0 and no terms (migration_kernel.cpp:486-510, the
// serial build).  With compat_pad, trailing padded crosslines take the last real crossline's
// Vrms, as the reference's OpenMP build computes them: there the kernel's crossline loop is a
// nested parallel region (src/main.cpp:255 already runs one output inline per thread), so
// one thread walks every crossline in order, and its per-sample caches
// (migration_kernel.cpp:60-72, :115-144), filled only where v >= 1e-5, still hold the last
// real crossline's values, while r^2 is taken from the padded crossline's own position.
__device__ __forceinline__ int vrms_col(const FwdParams& P, int x) {
    const int xv = x + P.xoff;
    if (x >= P.n_ox || xv < 0) return -1;
    if (xv < P.n_vx) return xv;
    return P.compat_pad ? P.n_vx - 1 : -1;
}

// Per output sample constants in the reference's FP32 order (migration_kernel.cpp:115-144).
// Division and products are pinned to round-to-nearest so the masks see the same numbers
// as the reference build; that build (GCC, -ffp-contract=fast) fuses v*v + 1e-10.
struct PointConst {
    bool valid;
    float t0sq, f4, md2, vsq;
};

__device__ __forceinline__ PointConst point_const(float v, float t0v, float tan2) {
    PointConst p;
    p.valid = (v >= 1e-5f) && (t0v >= 1e-5f);                 // :121
    p.t0sq = __fmul_rn(t0v, t0v);                              // :125
    p.vsq = __fmul_rn(v, v);                                   // :127
    float inv_vsq = __fdiv_rn(1.0f, __fmaf_rn(v, v, 1e-10f));  // :128
    p.f4 = __fmul_rn(4.0f, inv_vsq);                           // :129
    float vth = __fmul_rn(__fmul_rn(v, t0v), 0.5f);            // :133
    p.md2 = __fmul_rn(__fmul_rn(vth, vth), tan2);              // :134
    return p;
}

// The reference keeps a term when floor(s) < n_t - 1 with s = fl(sqrt(fma(f4, r2, t0^2)) *
// inv_dt) in IEEE FP32 (migration_kernel.cpp:209-226, :291-298).  s grows monotonically
// with r2, so the kept r2 form a prefix [0, R].  pass_bound returns B = min(md2, R): a term
// passes both of the reference's masks exactly when r2 <= B (B < 0: no term passes).  Found
// by a search on the bit patterns of the non-negative floats in [0, md2].
__device__ __forceinline__ bool range_ok(float r2, float f4, float t0sq, float inv_dt,
                                         float ntm1f) {
    return __fmul_rn(__fsqrt_rn(__fmaf_rn(f4, r2, t0sq)), inv_dt) < ntm1f;
}

__device__ __forceinline__ float pass_bound(const PointConst& p, float inv_dt, float ntm1f) {
    if (!p.valid || !(p.md2 >= 0.0f)) return -1.0f;
    if (range_ok(p.md2, p.f4, p.t0sq, inv_dt, ntm1f)) return p.md2;
    if (!range_ok(0.0f, p.f4, p.t0sq, inv_dt, ntm1f)) return -1.0f;
    unsigned lo = 0u, hi = __float_as_uint(p.md2);  // ok(lo), !ok(hi)
    if (hi - lo > 1u) {
        // Gallop out from the boundary of the unrounded test, f4 r2 + t0^2 =
        // ((n_t - 1) / inv_dt)^2, to a bracket of doubling width; the bisection below then
        // closes it.  The test is monotone in r2, so any bracket gives the same bound as a
        // bisection of all of [0, md2]; about 7 evaluations instead of 32.
        const float a = __fdividef(ntm1f, inv_dt);
        const float e = __fdividef(__fmaf_rn(a, a, -p.t0sq), p.f4);
        unsigned m = e > 0.0f ? __float_as_uint(e) : 0u;
        m = min(max(m, lo + 1u), hi - 1u);
        unsigned step = 1u;
        if (range_ok(__uint_as_float(m), p.f4, p.t0sq, inv_dt, ntm1f)) {
            lo = m;
            while (hi - lo > step) {
                const unsigned c = lo + step;
                if (!range_ok(__uint_as_float(c), p.f4, p.t0sq, inv_dt, ntm1f)) {
                    hi = c;
                    break;
                }
                lo = c;
                step <<= 1;
            }
        } else {
            hi = m;
            while (hi - lo > step) {
                const unsigned c = hi - step;
                if (range_ok(__uint_as_float(c), p.f4, p.t0sq, inv_dt, ntm1f)) {
                    lo = c;
                    break;
                }
                hi = c;
                step <<= 1;
            }
        }
    }
    while (hi - lo > 1u) {
        const unsigned mid = lo + ((hi - lo) >> 1);
        if (range_ok(__uint_as_float(mid), p.f4, p.t0sq, inv_dt, ntm1f))
            lo = mid;
        else
            hi = mid;
    }
    return __uint_as_float(lo);
}

// dx^2 of a buffer inline (migration_kernel.cpp:51-56).
__device__ __forceinline__ float inline_dx2(int ipos, int pos, float d_il) {
    float dx = __fmul_rn(static_cast<float>(ipos - pos), d_il);
    return __fmul_rn(dx, dx);
}

// r^2 of a trace at crossline distance dk (migration_kernel.cpp:197-204 / :282-284, with the
// multiply-add fused as the reference's GCC build fuses it).
__device__ __forceinline__ float trace_r2(int dk, float d_xl, float dx2) {
    float dy = __fmul_rn(static_cast<float>(dk), d_xl);
    return __fmaf_rn(dy, dy, dx2);
}

// ----------------------------------------------------------------------------- trace storage

// 16-bit storage of rows of ns fp32 samples (zero beyond n_t): one warp per trace.
// scale = max |d| over the trace (1 for an all-zero trace), q[t] = RNE(d[t] / scale) as
// bf16 or fp16.  A lane writes two samples (one word).
template <int STORE>
__device__ __forceinline__ uint32_t q16(float x) {
    if (STORE == kStoreBF16) return __bfloat16_as_ushort(__float2bfloat16_rn(x));
    return __half_as_ushort(__float2half_rn(x));
}

template <int STORE>
__global__ void quantize_kernel(const float* __restrict__ src, uint32_t* __restrict__ halves,
                                float* __restrict__ scales, size_t n_rows, int ns) {
    const int lane = threadIdx.x & 31;
    const size_t warps = static_cast<size_t>(gridDim.x) * (blockDim.x >> 5);
    for (size_t r = blockIdx.x * static_cast<size_t>(blockDim.x >> 5) + (threadIdx.x >> 5);
         r < n_rows; r += warps) {
        const float* row = src + r * ns;
        float m = 0.0f;
        for (int t = lane; t < ns; t += 32) m = fmaxf(m, fabsf(row[t]));
        m = warp_max(m);
        const float scale = m > 0.0f ? m : 1.0f;
        if (lane == 0) scales[r] = scale;
        uint32_t* out = halves + r * (ns / 2);
        for (int t = lane; t < ns / 2; t += 32) {
            const float2 d = reinterpret_cast<const float2*>(row)[t];
            out[t] = q16<STORE>(__fdiv_rn(d.x, scale)) | (q16<STORE>(__fdiv_rn(d.y, scale)) << 16);
        }
    }
}

// ----------------------------------------------------------------------------- trace lists

// Buffer inlines (local indices) of row r of the producer's trace list: with pc < 0 the row is
// inline r; else row r is the mirror distance from the centre inline pc, holding inlines
// pc - r and pc + r (*b = -1 when the row has one inline: r = 0, or one side outside the
// buffer).
__device__ __forceinline__ void row_inlines(int pc, int n_inl, int r, int* a, int* b) {
    if (pc < 0) {
        *a = r;
        *b = -1;
        return;
    }
    *a = pc - r;
    *b = r > 0 && pc + r < n_inl ? pc + r : -1;
    if (*a < 0) {
        *a = pc + r;
        *b = -1;
    }
}

// Producer: lo of every passing term of the tile on trace (dx2, kc) lies in [*lolo, *lohi]
// (with two samples of slack for rounding); false when the trace has no passing term.
// Bounds: t >= t0 and, inside the aperture r <= v t0 tan/2, t0 >= 2 r_min / (v_max tan);
// t^2 = t0^2 + f4 r^2 <= min(t0max^2 + 4 r_max^2 / v_min^2, t0max^2 (1 + tan^2)).
__device__ __forceinline__ bool trace_bounds(const FwdParams& P, const TileStats& S, int xa,
                                             int xb, float dx2, int kc, int* lolo_out,
                                             int* lohi_out) {
    const int dkmin = kc < xa ? xa - kc : (kc > xb ? kc - xb : 0);
    const int dkmax = max(abs(kc - xa), abs(kc - xb));
    const float dymin = static_cast<float>(dkmin) * P.d_xl;
    const float dymax = static_cast<float>(dkmax) * P.d_xl;
    const float rmin2 = fmaf(dymin, dymin, dx2);
    const float rmax2 = fmaf(dymax, dymax, dx2);
    if (rmin2 > S.bmax * 1.0001f + 1e-6f) return false;
    float t0lo = S.t0min;
    if (P.tanth > 0.0f) t0lo = fmaxf(t0lo, 2.0f * sqrtf(rmin2) / (S.vmax * P.tanth));
    const float tlo = sqrtf(fmaf(t0lo, t0lo, 4.0f * rmin2 / fmaf(S.vmax, S.vmax, 1e-10f)));
    const float thi2 =
        fminf(fmaf(S.t0max, S.t0max, 4.0f * rmax2 / fmaf(S.vmin, S.vmin, 1e-10f)),
              S.t0max * S.t0max * (1.0f + P.tan2) * 1.0001f);
    const float slo = tlo * P.inv_dt;
    const float shi = fminf(sqrtf(thi2) * P.inv_dt, 1.0e9f);
    *lolo_out = max(static_cast<int>(floorf(slo)) - 2, 0);
    *lohi_out = min(static_cast<int>(floorf(shi)) + 2, P.n_t - 2);
    return *lolo_out <= *lohi_out;
}

// Both samples of a 16-bit storage word as fp32 (exact conversions).
template <int STORE>
__device__ __forceinline__ float2 unpack16(uint32_t w) {
    if (STORE == kStoreBF16)
        return make_float2(__uint_as_float(w << 16), __uint_as_float(w & 0xffff0000u));
    return make_float2(__half2float(__ushort_as_half(static_cast<unsigned short>(w & 0xffffu))),
                       __half2float(__ushort_as_half(static_cast<unsigned short>(w >> 16))));
}

// Padded output inlines repeat the migrated edge inline (main.cpp:268-285): row copies[k].x of
// the image gets row copies[k].y, every copy in one launch (a source row is never a
// destination).
__global__ void copy_rows_kernel(float* __restrict__ img, const int2* __restrict__ copies,
                                 int n_copies, size_t row) {
    const size_t total = static_cast<size_t>(n_copies) * row;
    for (size_t i = blockIdx.x * static_cast<size_t>(blockDim.x) + threadIdx.x; i < total;
         i += static_cast<size_t>(gridDim.x) * blockDim.x) {
        const int k = static_cast<int>(i / row);
        const size_t e = i - static_cast<size_t>(k) * row;
        const int2 cp = copies[k];
        img[static_cast<size_t>(cp.x) * row + e] = img[static_cast<size_t>(cp.y) * row + e];
    }
}

// ----------------------------------------------------------------------------- term count

// One block per (job, output crossline); threads stride over t.  out[job] += terms.
// A term passes when r^2 <= B (pass_bound); r^2 grows with |k - x|, so for each buffer
// inline the passing crosslines are |k - x| <= d with d found from sqrt(B - dx^2) and exact
// fix-ups.
__global__ void count_kernel(const FwdParams P, unsigned long long* out) {
    __shared__ unsigned long long wsum[32];
    const int x = blockIdx.x;
    const Job job = P.jobs[blockIdx.y];
    const int xv = x + P.xoff;
    // the farthest trace of the cube from crossline xv (xv >= 0; beyond n_cx - 1 with
    // compat_pad), plus one
    const int dcap = max(xv, P.n_cx - 1 - xv) + 1;
    unsigned long long local = 0;
    for (int t = threadIdx.x; t < P.n_t; t += blockDim.x) {
        const int vc = vrms_col(P, x);
        if (vc < 0) break;
        const float v = vrms_trace(P, job.vrow, vc)[t];
        const PointConst pc = point_const(v, P.t0[t], P.tan2);
        const float B = pass_bound(pc, P.inv_dt, P.ntm1f);
        if (B < 0.0f) continue;
        for (int i = job.i0; i < job.i1; ++i) {
            const float dx2 = inline_dx2(P.il_pos[i], job.pos, P.d_il);
            if (dx2 > B) continue;  // d = 0 passes from here on
            int d = static_cast<int>(sqrtf(fmaxf(B - dx2, 0.0f)) * P.inv_dxl);
            d = min(d, dcap);
            while (d > 0 && trace_r2(d, P.d_xl, dx2) > B) --d;
            while (d < dcap && trace_r2(d + 1, P.d_xl, dx2) <= B) ++d;
            const int lo = max(0, xv - d), hi = min(P.n_cx - 1, xv + d);
            if (hi >= lo) local += static_cast<unsigned long long>(hi - lo + 1);
        }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) local += __shfl_xor_sync(0xffffffffu, local, o);
    if ((threadIdx.x & 31) == 0) wsum[threadIdx.x >> 5] = local;
    __syncthreads();
    if (threadIdx.x == 0) {
        unsigned long long s = 0;
        for (int w = 0; w < static_cast<int>(blockDim.x >> 5); ++w) s += wsum[w];
        if (s) atomicAdd(out + blockIdx.y, s);
    }
}

}  // namespace psm
