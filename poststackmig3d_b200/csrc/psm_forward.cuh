// Forward kernel (migration): the diffraction summation of psm_kernels.cuh.
//
// One CTA migrates one tile: an output inline, NX output crosslines and kTileT = 256 samples.
// Its warps have three roles, joined by a ring of kStages shared-memory stages:
//   * producer (warp 0): lists the input traces that can reach the tile, derives for each a
//     window of samples that covers every passing term, and copies the windows with TMA bulk
//     copies (cp.async.bulk).  The traces at inlines c - d and c + d of one crossline (c the
//     output inline) have the same r^2 to every output point, hence the same travel times and
//     weights: they share one slot;
//   * folder (warp 1): adds the two traces of a slot and writes the window as pairs
//     (p[t], p[t + 1] - p[t]), so one 8-byte shared load gives a consumer both interpolation
//     operands of both traces;
//   * consumers (NX warps): two crosslines (16 lanes each) and 128 of the tile's samples a
//     warp, 4 pairs of 16-sample blocks a lane.
//
// What bounds it (B200, shared loads 128 B, rsqrt 16, FMA 128 lanes per clock per SM): one
// evaluation (64 output samples of one slot) needs 2 rsqrt warp instructions (16 cycles of a
// sub-partition's XU), 6 packed and 2 scalar FMA instructions and 2 addresses (16 to 18 cycles
// of its FMA pipe) and 4 wavefronts of shared loads (16 cycles of a quarter of the SM), so the
// three pipes are about equally loaded; the loop runs at 20 to 21 cycles an evaluation.
// Reasons for the layout:
//   * folding a pair before the consumers read it halves their shared loads and takes one
//     packed add a load away; a window of about 150 samples is read by NX crosslines, so the
//     fold is 5% of the instructions;
//   * 16 lanes x 2 crosslines: the lanes of one evaluation span 32 samples and 2 crosslines,
//     over which the aperture's edge moves less than over 64 samples of one crossline (9%
//     against 17% of the evaluated terms fail their masks on the 201 x 201 x 1001 cube below);
//   * the slots of a stage are sorted into four lists per couple of pairs (all lanes pass,
//     both pairs, first or second pair only), so that the evaluations run in loops without
//     tests: the earlier kernel spent half of its instructions on a test tree per slot.
// Measured on 201 x 201 x 1001 samples (Vrms 1500 -> 3500 m/s, 45 degrees): 116.4 ms before
// (one crossline a warp, pairs read unfolded, a test tree per slot), 72.6 ms with NX = 14 (64
// registers, 2 CTAs per SM).  NX = 12 takes 76.0 ms, NX = 10 78.4 ms, NX = 8 (3 CTAs per SM) 82.8
// ms, NX = 4 102 ms; three smaller stages and stages of 3200 samples were 4 to 6% slower (the
// work per stage and warp besides the evaluations is about 230 instructions).  NX = 4 is faster
// where the wide tiles leave SMs idle: 31 x 29 x 251 samples 0.088 against 0.108 ms; there the
// producer's bulk copies (some 50 short windows a stage) are the bound.
#pragma once

#include "psm_kernels.cuh"

namespace psm {

constexpr int kTileT = 256;  // output samples of a tile
constexpr int kSlots = 32;   // slots per ring stage at most (a lane each)

// Tables of one ring stage (NX output crosslines).
template <int NX>
struct FwdStage {
    int n;              // slots, -1 = end of the tile's stream
    int split;          // nonzero: one slot, part of a window longer than a stage holds
    float slo, shi;     // split: this part takes the terms with floor(t / dt) in [slo, shi)
    int tot, tot_pairs; // samples of all windows; of the paired slots' windows, which come first
    int pad[2];
    int base[kSlots];   // byte offset of the window's sample 0, less 8 * bits(2^23)
    int4 win[kSlots];   // window's byte offset, samples, mirror's raw samples (0: none)
    float2 scale[kSlots];  // 16-bit storage: scales of the trace and of its mirror
    float r2[NX][kSlots];  // r^2 to each output crossline
};

// Shared memory of a CTA: CAP samples a stage, folded windows of 8 bytes a sample.  A trace's
// own raw samples are copied into the upper end of the memory that its folded window takes,
// its mirror's into a buffer of their own, one per stage.  Caller-made pairs (8 bytes a sample) have
// one mirror buffer for all stages, so that as many CTAs fit an SM as with fp32 traces: the
// producer waits for the folder to be done with it, which it is long before the consumers
// release a stage.  (psm_forward_noalloc, 101 x 101 x 501 samples: 2.71 ms with a buffer per stage,
// which leaves room for one CTA of the wide tiles, 1.91 ms so.)
template <int NX, int CAP>
struct FwdLayout {
    static_assert(NX % 2 == 0 && CAP % 8 == 0, "crossline pairs; 16-byte aligned windows");
    static constexpr unsigned kFull = 0, kReady = 8 * kStages, kEmpty = 16 * kStages;
    static constexpr unsigned kZero = (24 * kStages + 15) & ~15u;  // 16 zero bytes
    static constexpr unsigned kTab = kZero + 16;
    static constexpr unsigned kList = kTab + kStages * sizeof(FwdStage<NX>);  // [NX][2][kSlots]
    static constexpr unsigned kStat = kList + NX * 2 * kSlots * 8;  // [NX / 2][8] float4
    static constexpr unsigned kBnd = kStat + NX / 2 * 8 * 16;       // [NX][4] float4
    static constexpr unsigned kBlk = kBnd + NX * 4 * 16;            // [8][2] float4
    static constexpr unsigned kRing = (kBlk + 8 * 32 + 127) & ~127u;
    static constexpr unsigned kStageBytes = 8u * CAP;
    static constexpr unsigned kMirror = kRing + kStages * kStageBytes;
    // the row tables, for raw samples of rb bytes
    static __host__ __device__ constexpr unsigned rows_at(int rb) {
        return kMirror + (rb == 8 ? 1 : kStages) * static_cast<unsigned>(CAP) * rb;
    }
    // row tables: running slot counts and dx^2
    static __host__ __device__ constexpr unsigned total(int store, int max_rows) {
        return rows_at(store_bytes(store)) + 4u * (2u * static_cast<unsigned>(max_rows) + 1u);
    }
    static_assert(kTab % 16 == 0 && sizeof(FwdStage<NX>) % 16 == 0, "16-byte aligned tables");
};

// Square root for the bounds of windows and rows, whose slack is two samples or traces (the
// correctly rounded one is 8 to 10 instructions more on the producer's chain: 0.852 ms with it,
// 0.841 without, 101 x 101 x 501 samples).
__device__ __forceinline__ float sqrt_approx(float x) {
    float r;
    asm("sqrt.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
    return r;
}

__device__ __forceinline__ void fence_async_smem() {
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
}

// ----------------------------------------------------------------------------- evaluation

#ifdef PSM_DEBUG_BOUNDS
// The windows of the stage a consumer reads (debug-bounds build).
struct DebugWin {
    const int* base;
    const int4* win;
    int n;
    int* err;
};
__device__ __forceinline__ uint32_t debug_check(const DebugWin& d, uint32_t base, uint32_t o,
                                                uint32_t zero) {
    if (o == zero) return o;
    for (int g = 0; g < d.n; ++g)
        if (static_cast<uint32_t>(d.base[g]) == base && o >= static_cast<uint32_t>(d.win[g].x) &&
            o + 8 <= static_cast<uint32_t>(d.win[g].x + 8 * d.win[g].y))
            return o;
    atomicOr(d.err, PSM_DEV_ERR_WINDOW);
    return zero;
}
#define PSM_DBG_PARAM , const DebugWin& dbg
#define PSM_DBG_ARG , dbg
#else
#define PSM_DBG_PARAM
#define PSM_DBG_ARG
#endif

// One slot at two output samples per lane.  Sample n of the slot's window sits at byte
// base + 8 bits(2^23 + n) (32-bit wrap-around).  A term that passes both masks needs no clamp:
// the producer's bounds (two samples of slack, one extra element) keep its floor(t / dt) inside
// the window.  MASK: a failing term reads a zero sample instead and adds nothing.
template <bool AMP, bool MASK>
__device__ __forceinline__ void eval2(const unsigned char* smem, float r2, uint32_t base,
                                      const float2& T2, const float2& F4, const float2& B,
                                      uint32_t zero, float2& acc PSM_DBG_PARAM) {
    const float2 t2 = fma2(F4, make_float2(r2, r2), T2);       // (t / dt)^2
    const float2 q = make_float2(rsqrtf(t2.x), rsqrtf(t2.y));  // dt / t
    const float2 s = mul2(t2, q);                              // t / dt
    const float2 M = make_float2(8388608.0f, 8388608.0f);
    const float2 mm = add2_rm(s, M);                           // 2^23 + floor(t / dt)
    const float2 fr = sub2(s, sub2(mm, M));                    // frac
    uint32_t oa = base + (__float_as_uint(mm.x) << 3), ob = base + (__float_as_uint(mm.y) << 3);
    if (MASK) {
        oa = r2 <= B.x ? oa : zero;
        ob = r2 <= B.y ? ob : zero;
    }
#ifdef PSM_DEBUG_BOUNDS
    oa = debug_check(dbg, base, oa, zero);
    ob = debug_check(dbg, base, ob, zero);
#endif
    const float2 pa = *reinterpret_cast<const float2*>(smem + oa);
    const float2 pb = *reinterpret_cast<const float2*>(smem + ob);
    const float2 v = make_float2(fmaf(fr.x, pa.y, pa.x), fmaf(fr.y, pb.y, pb.x));
    if (AMP)
        acc = fma2(v, q, acc);
    else
        acc = add2(acc, v);
}

// ----------------------------------------------------------------------------- folding

// Two raw samples i, i + 1 (i even) of a staged window at byte offset a.
template <int STORE>
__device__ __forceinline__ float2 raw_pair(const unsigned char* smem, uint32_t a, int i) {
    if (STORE == kStoreF32) return *reinterpret_cast<const float2*>(smem + a + 4 * i);
    if (STORE == kStorePairs) {
        const float4 v = *reinterpret_cast<const float4*>(smem + a + 8 * i);
        return make_float2(v.x, v.z);
    }
    return unpack16<STORE>(*reinterpret_cast<const uint32_t*>(smem + a + 2 * i));
}

// fp32 storage: the windows of a whole stage as one array, samples [from, to), MIRROR: plus the
// mirrors' samples.  d, a, b: byte offsets of the folded windows, the raw samples and the
// mirrors' raw samples of sample 0.  OWN: a difference is the sum of the two traces' own
// differences, else the difference of the sums.  A lane folds two samples; the 32nd lane only
// supplies its neighbour's next samples, so a step advances by 62.  The folded windows grow over the raw
// samples from below: a step writes to byte 8 (i + 62) of the stage and the raw samples not yet
// read start at 4 tot + 4 (i + 62), which is not less while i + 62 <= tot.  A window's last
// element takes its second value from the next window and is never read: windows end one
// sample past the last element used (fp32 rows end in a zero sample).
template <bool MIRROR, bool OWN>
__device__ __forceinline__ void fold_range(unsigned char* smem, uint32_t d, uint32_t a, uint32_t b,
                                           int from, int to, int lane) {
    constexpr int U = 4;  // steps in flight: one alone is a chain of load, shuffle and store
    for (int i0 = from; i0 < to; i0 += 62 * U) {
        float2 p[U], m[MIRROR ? U : 1];
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const int i = min(i0 + 62 * u + 2 * lane, to - 2);
            p[u] = *reinterpret_cast<const float2*>(smem + a + 4 * i);
            if (MIRROR) {
                const float2 q = *reinterpret_cast<const float2*>(smem + b + 4 * i);
                if (OWN)
                    m[MIRROR ? u : 0] = q;
                else
                    p[u] = add2(p[u], q);
            }
        }
        __syncwarp();
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const int i = i0 + 62 * u + 2 * lane;
            const float pn = __shfl_down_sync(0xffffffffu, p[u].x, 1);
            float4 o = make_float4(p[u].x, p[u].y - p[u].x, p[u].y, pn - p[u].y);
            if (MIRROR && OWN) {
                const float2 q = m[MIRROR ? u : 0];
                const float qn = __shfl_down_sync(0xffffffffu, q.x, 1);
                o = make_float4(o.x + q.x, o.y + (q.y - q.x), o.z + q.y, o.w + (qn - q.y));
            }
            if (lane < 31 && i < to) *reinterpret_cast<float4*>(smem + d + 8 * i) = o;
        }
        __syncwarp();
    }
}

// 16-bit storage and caller-made pairs: one window, its raw samples at the upper end of its own
// memory (pairs: in place), the mirror's at offset b (0: none); the sample after the window is
// taken as zero.
template <int STORE>
__device__ __forceinline__ void fold_window(unsigned char* smem, uint32_t d, int size, uint32_t b,
                                            float2 scale, int lane) {
    constexpr bool Q = STORE == kStoreBF16 || STORE == kStoreF16;
    constexpr int U = 3;
    const uint32_t a = d + (8 - store_bytes(STORE)) * size;
    for (int i0 = 0; i0 < size; i0 += 62 * U) {
        float2 p[U];
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const int i = min(i0 + 62 * u + 2 * lane, size - 2);
            p[u] = raw_pair<STORE>(smem, a, i);
            if (Q) p[u] = mul2(p[u], make_float2(scale.x, scale.x));
            if (b) {
                const float2 m = raw_pair<STORE>(smem, b, i);
                p[u] = Q ? fma2(m, make_float2(scale.y, scale.y), p[u]) : add2(p[u], m);
            }
        }
        __syncwarp();
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const int i = i0 + 62 * u + 2 * lane;
            float pn = __shfl_down_sync(0xffffffffu, p[u].x, 1);
            if (i + 2 >= size) pn = 0.0f;
            if (lane < 31 && i < size)
                *reinterpret_cast<float4*>(smem + d + 8 * i) =
                    make_float4(p[u].x, p[u].y - p[u].x, p[u].y, pn - p[u].y);
        }
        __syncwarp();
    }
}

// ----------------------------------------------------------------------------- one tile

// One tile of a batched launch: problem, job of that problem, first crossline and sample.
struct BatchItem {
    int prob, job, x0, T0;
};

struct True {
    static constexpr bool value = true;
};
struct False {
    static constexpr bool value = false;
};

// ORDERED (fp32 storage): every output sample adds its terms in the order of the trace list
// (mirror distance, then crossline), with the traces' own differences; else the order within a
// stage is that of the slots' kinds.  Least-squares migration runs the ordered form: conjugate
// gradients carry a change of rounding in the operator into their step lengths and residual
// norms, which are reproducible to 1e-9 this way.  By kind saves the control of short runs:
// 0.84 against 0.91 ms on 101 x 101 x 501 samples (201 x 201 x 1001: 72.6, 72.7 ms).
//
// KAHAN: compensated summation.  Each ring stage (at most kSlots slots) is summed into a fresh
// partial, and the partials are added to the accumulator with Kahan's compensation, so the long
// sum over the aperture carries no growing rounding error.
//
// PAIRS: caller-made pairs (kStorePairs), else any other storage.
//
// All warps of the CTA call fwd_tile; `it` counts the ring stages the CTA has used, so that
// consecutive tiles of a persistent CTA continue the ring's phases (every stage, the
// end-of-stream marker included, is released).  Returns false when a bounded wait expired.
template <bool AMP, bool KAHAN, bool ORDERED, int NX, int CAP, bool PAIRS = false>
__device__ __forceinline__ bool fwd_tile(const FwdParams& P, const Job job, int x0, int T0,
                                         unsigned char* smem, uint32_t& it) {
    using L = FwdLayout<NX, CAP>;
    using Stage = FwdStage<NX>;
    uint64_t* full = reinterpret_cast<uint64_t*>(smem + L::kFull);
    uint64_t* ready = reinterpret_cast<uint64_t*>(smem + L::kReady);
    uint64_t* empty = reinterpret_cast<uint64_t*>(smem + L::kEmpty);
    Stage* tabs = reinterpret_cast<Stage*>(smem + L::kTab);
    float4* stat = reinterpret_cast<float4*>(smem + L::kStat);
    // (read through a shuffle, which makes the compiler lay out the evaluation loops otherwise:
    // 79.2 ms without, 72.6 with, 201 x 201 x 1001 samples)
    const int warp = __shfl_sync(0xffffffffu, static_cast<int>(threadIdx.x >> 5), 0);
    const int lane = threadIdx.x & 31;

    // ---- consumers: per-sample constants.  Warp cw owns crosslines x0 + 2 xp + {0, 1} (16 lanes
    // each) and every other 32 samples of the tile (phase ph), so the warps of a crossline
    // pair share the deep samples, whose aperture is the widest: pair p holds samples
    // 64 p + 32 ph + {0, 16} + (lane & 15).
    const int cw = warp - 2;
    const int xl = lane >> 4, xp = cw >> 1, ph = cw & 1;
    const int x = x0 + 2 * xp + xl;
    float2 T2[4], F4[4], BB[4], ACC[4], CMP[KAHAN ? 4 : 1];
    if (cw >= 0) {
        const int vc = vrms_col(P, x);
        const float* vp = vrms_trace(P, job.vrow, vc >= 0 ? vc : 0);
        float4* bnd = reinterpret_cast<float4*>(smem + L::kBnd) + cw * 4;
#pragma unroll
        for (int p = 0; p < 4; ++p) {
            float bj[2], t2[2], f4[2];
            int vmn = 0x7f000000, vmx = 0;
#pragma unroll
            for (int c = 0; c < 2; ++c) {
                const int t = T0 + 64 * p + 32 * ph + 16 * c + (lane & 15);
                float v = 0.0f, t0v = 0.0f;
                if (vc >= 0 && t < P.n_t) {
                    v = __ldg(vp + t);
                    t0v = __ldg(P.t0 + t);
                }
                const PointConst pc = point_const(v, t0v, P.tan2);
                const float b = pass_bound(pc, P.inv_dt, P.ntm1f);
                bj[c] = b;
                t2[c] = b >= 0.0f ? pc.t0sq * P.idt2 : 1.0f;
                f4[c] = b >= 0.0f ? pc.f4 * P.idt2 : 0.0f;
                if (b >= 0.0f) {
                    vmn = min(vmn, __float_as_int(v));
                    vmx = max(vmx, __float_as_int(v));
                }
            }
            T2[p] = make_float2(t2[0], t2[1]);
            F4[p] = make_float2(f4[0], f4[1]);
            BB[p] = make_float2(bj[0], bj[1]);
            ACC[p] = make_float2(0.0f, 0.0f);
            if (KAHAN) CMP[KAHAN ? p : 0] = make_float2(0.0f, 0.0f);
            // largest and smallest bound of the pair per crossline (non-negative floats order
            // as their bits, -1 below them all), and the Vrms range of its passing samples
            const int bx = __float_as_int(fmaxf(bj[0], bj[1]));
            const int bn = __float_as_int(fminf(bj[0], bj[1]));
            const int none = static_cast<int>(0x80000000u);
            const int mx0 = __reduce_max_sync(0xffffffffu, xl == 0 ? bx : none);
            const int mx1 = __reduce_max_sync(0xffffffffu, xl == 1 ? bx : none);
            const int mn0 = __reduce_min_sync(0xffffffffu, xl == 0 ? bn : 0x7fffffff);
            const int mn1 = __reduce_min_sync(0xffffffffu, xl == 1 ? bn : 0x7fffffff);
            vmn = __reduce_min_sync(0xffffffffu, vmn);
            vmx = __reduce_max_sync(0xffffffffu, vmx);
            if (lane == 0) {
                bnd[p] = make_float4(__int_as_float(mx0), __int_as_float(mx1),
                                     __int_as_float(mn0), __int_as_float(mn1));
                stat[xp * 8 + 2 * p + ph] = make_float4(__int_as_float(vmn), __int_as_float(vmx),
                                                        __int_as_float(max(mx0, mx1)), 0.0f);
            }
        }
    }
    // The producer's share of the wait: smallest and largest t0 of each block of 32 samples (lane
    // b holds block b), whatever their order (the per-inline call takes the caller's times).
    // A sample has terms only with t0 > 0; every other counts as 0.  (Unrolled, the loop moves the
    // evaluation loops: 8.86 against 8.84 ms, 133 x 87 x 733 samples.)
    float t0min = 0.0f, t0max = 0.0f;
    if (warp == 0) {
#pragma unroll 1
        for (int b = 0; b < kTileT / 32; ++b) {
            const float t = __ldg(P.t0 + min(T0 + 32 * b + lane, P.n_t - 1));
            const int bits = t > 0.0f ? __float_as_int(t) : 0;
            const int mn = __reduce_min_sync(0xffffffffu, bits);
            const int mx = __reduce_max_sync(0xffffffffu, bits);
            if (lane == b) {
                t0min = __int_as_float(mn);
                t0max = __int_as_float(mx);
            }
        }
    }
    __syncthreads();

    if (warp == 0) {
        // ---------------------------------------------------------------- producer
        const int store = PAIRS ? kStorePairs : P.store;
        const int rb = PAIRS ? 8 : store == kStoreF32 ? 4 : 2;
        const int A = store == kStoreBF16 || store == kStoreF16 ? 8 : 4;  // window alignment
        // bounds of each block of 32 samples over the tile's crosslines, in two float4: (largest
        // B, smallest t0, 2 / (v_max tan), 4 / v_max^2), (largest t0^2, 4 / v_min^2, largest t0^2
        // (1 + tan^2), 1 when a sample passes)
        float4* blk = reinterpret_cast<float4*>(smem + L::kBlk);
        float bmax;
        {
            float vmn = 3.0e38f, vmx = 0.0f, bmx = -1.0f;
            for (int w = lane >> 3; w < NX / 2; w += 4) {
                const float4 s = stat[w * 8 + (lane & 7)];
                vmn = fminf(vmn, s.x);
                vmx = fmaxf(vmx, s.y);
                bmx = fmaxf(bmx, s.z);
            }
#pragma unroll
            for (int o = 8; o < 32; o <<= 1) {
                vmn = fminf(vmn, __shfl_xor_sync(0xffffffffu, vmn, o));
                vmx = fmaxf(vmx, __shfl_xor_sync(0xffffffffu, vmx, o));
                bmx = fmaxf(bmx, __shfl_xor_sync(0xffffffffu, bmx, o));
            }
            bmax = warp_max(bmx);
            if (lane < 8) {
                blk[2 * lane] = make_float4(
                    bmx * 1.0001f + 1e-6f, t0min,
                    P.tanth > 0.0f && vmx > 0.0f ? 2.0f / (vmx * P.tanth) : 0.0f,
                    4.0f / fmaf(vmx, vmx, 1e-10f));
                blk[2 * lane + 1] = make_float4(
                    t0max * t0max, 4.0f / fmaf(vmn, vmn, 1e-10f),
                    t0max * t0max * (1.0f + P.tan2) * 1.0001f, bmx >= 0.0f ? 1.0f : 0.0f);
            }
            __syncwarp();
        }
        // cube crossline range of the tile's output points
        const int xa = max(x0 + P.xoff, 0);
        const int xb = min(min(x0 + NX, P.n_ox) - 1 + P.xoff,
                           P.compat_pad ? 0x3fffffff : P.n_vx - 1);
        int* row_pre = reinterpret_cast<int*>(smem + L::rows_at(rb));
        float* row_dx2 = reinterpret_cast<float*>(row_pre + P.max_rows + 1);
        const int n_inl = max(job.i1 - job.i0, 0);
        // rows of the trace list: the buffer inlines, or the mirror distances d from the centre
        // inline pc (row d holds inlines pc - d and pc + d)
        int pc = -1;
        if (P.pairable && n_inl > 0) {
            const int c = job.pos - __ldg(P.il_pos + job.i0);
            if (c >= 0 && c < n_inl) pc = c;
        }
        const int n_rows = pc >= 0 ? max(pc, n_inl - 1 - pc) + 1 : n_inl;
        // first crossline of a row's traces: none beyond bmax reaches the tile
        auto row_first = [&](float dx2, int* reach) {
            *reach = static_cast<int>(sqrt_approx(fmaxf(bmax - dx2, 0.0f)) * P.inv_dxl) + 2;
            return max(0, xa - *reach);
        };
        int total = 0;
        if (bmax >= 0.0f && xa <= xb) {
            for (int base = 0; base < n_rows; base += 32) {
                const int n = base + lane;
                int cnt = 0;
                if (n < n_rows) {
                    int a, b;
                    row_inlines(pc, n_inl, n, &a, &b);
                    const float dx2 = inline_dx2(__ldg(P.il_pos + job.i0 + a), job.pos, P.d_il);
                    if (dx2 <= bmax) {
                        int reach;
                        const int klo = row_first(dx2, &reach);
                        cnt = max(0, min(P.n_cx - 1, xb + reach) - klo + 1);
                    }
                    row_dx2[n] = dx2;
                }
                int incl = cnt;
#pragma unroll
                for (int o = 1; o < 32; o <<= 1) {
                    const int v = __shfl_up_sync(0xffffffffu, incl, o);
                    if (lane >= o) incl += v;
                }
                if (n < n_rows) row_pre[n] = total + incl - cnt;
                total += __shfl_sync(0xffffffffu, incl, 31);
            }
            if (lane == 0) row_pre[n_rows] = total;
            __syncwarp();
        }
        bool alive = true;
        const uint32_t it_begin = it;    // the ring iteration of this tile's first stage
        uint32_t stalled = 0xffffffffu;  // test-only stall: the stage left unfilled
        int f = 0;                       // traces of the list consumed
        int part = 0;                    // samples of a window longer than a stage already staged
        while (f < total) {
            const int idx = f + lane;
            int ws = 0, size = 0, kc = 0, row = 0, rowb = -1;
            float dx2 = 0.0f;
            if (idx < total) {
                int lo = 0, hi = n_rows - 1;  // the last row with row_pre <= idx
                while (lo < hi) {
                    const int mid = (lo + hi + 1) >> 1;
                    if (row_pre[mid] <= idx)
                        lo = mid;
                    else
                        hi = mid - 1;
                }
                dx2 = row_dx2[lo];
                int reach;
                kc = row_first(dx2, &reach) + (idx - row_pre[lo]);
                int a, b;
                row_inlines(pc, n_inl, lo, &a, &b);
                row = job.i0 + a;
                rowb = b >= 0 ? job.i0 + b : -1;
                // window: over the blocks that the trace can reach, t^2 lies in [e^2 + 4 r_min^2 /
                // v_max^2, min(t0^2 + 4 r_max^2 / v_min^2, t0^2 (1 + tan^2))] with e the later of
                // the block's smallest t0 and the aperture's entry 2 r_min / (v_max tan)
                const int dkmin = kc < xa ? xa - kc : (kc > xb ? kc - xb : 0);
                const int dkmax = max(abs(kc - xa), abs(kc - xb));
                const float dymin = static_cast<float>(dkmin) * P.d_xl;
                const float dymax = static_cast<float>(dkmax) * P.d_xl;
                const float rmin2 = fmaf(dymin, dymin, dx2), rmax2 = fmaf(dymax, dymax, dx2);
                const float rmin = sqrt_approx(rmin2);
                float tlo2 = 3.0e38f, thi2 = -1.0f;
#pragma unroll
                for (int p = 0; p < 8; ++p) {
                    const float4 u = blk[2 * p], w = blk[2 * p + 1];
                    if (w.w > 0.0f && rmin2 <= u.x) {
                        const float e = fmaxf(u.y, u.z * rmin);
                        tlo2 = fminf(tlo2, fmaf(e, e, u.w * rmin2));
                        thi2 = fmaxf(thi2, fminf(fmaf(w.y, rmax2, w.x), w.z));
                    }
                }
                if (thi2 >= 0.0f) {
                    const float slo = fminf(sqrt_approx(tlo2) * P.inv_dt, 1.0e9f);
                    const float shi = fminf(sqrt_approx(thi2) * P.inv_dt, 1.0e9f);
                    const int lolo = max(static_cast<int>(floorf(slo)) - 2, 0);
                    const int lohi = min(static_cast<int>(floorf(shi)) + 2, P.n_t - 2);
                    if (lolo <= lohi) {
                        // floor(t / dt) of a passing term lies in [lolo, lohi + 1], and its
                        // element holds the next sample too
                        ws = lolo & ~(A - 1);
                        size = ((lohi + 2 + A) & ~(A - 1)) - ws;
                    }
                }
            }
            // the lanes whose windows fit one stage
            int cum = size;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const int v = __shfl_up_sync(0xffffffffu, cum, o);
                if (lane >= o) cum += v;
            }
            unsigned taken = __ballot_sync(0xffffffffu, cum <= CAP);
            int split = 0;
            float slo = 0.0f, shi = 0.0f;
            if (!taken) {  // the first window alone exceeds a stage: stage it in parts
                split = 1;
                const int ws0 = __shfl_sync(0xffffffffu, ws, 0);
                const int rest = __shfl_sync(0xffffffffu, size, 0) - part;
                const bool last = rest <= CAP;
                slo = part ? static_cast<float>(ws0 + part) : -1.0f;
                shi = last ? 3.0e38f : static_cast<float>(ws0 + part + CAP - 8);
                ws = ws0 + part;
                size = lane ? 0 : (last ? rest : CAP);
                cum = last ? rest : CAP;
                part = last ? 0 : part + CAP - 8;  // (an element needs the sample after it)
                taken = 1u;
            }
            const int consumed = split && part ? 0 : __popc(taken);
            const bool mine = ((taken >> lane) & 1u) && size > 0;
            const unsigned slots = __ballot_sync(0xffffffffu, mine);
            const int n = __popc(slots);
            // windows of mirrored pairs first, then those of single traces
            const int own = mine && rowb >= 0 ? size : 0;
            int cump = own;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const int v = __shfl_up_sync(0xffffffffu, cump, o);
                if (lane >= o) cump += v;
            }
            const int totp = __shfl_sync(0xffffffffu, cump, 31);
            const int tot = __shfl_sync(0xffffffffu, cum, __popc(taken) - 1);
            if (n > 0) {
                const int stage = it % kStages;
                const uint32_t par = ((it / kStages) & 1u) ^ 1u;
                int ok = lane == 0 ? mbar_wait(&empty[stage], par, P.err, P.wait_us) : 0;
                if (PAIRS && lane == 0 && ok && it > it_begin)  // the mirror buffer
                    ok = mbar_wait(&ready[(it - 1) % kStages], ((it - 1) / kStages) & 1u, P.err,
                                   P.wait_us);
                if (!__shfl_sync(0xffffffffu, ok, 0)) {
                    alive = false;
                    break;
                }
                // test-only: the tile's first stage is never filled nor arrived on
                const bool stall = (P.fault & kFaultStallProducer) && it == it_begin;
                Stage& m = tabs[stage];
                const int copy = min(size, P.ns - ws);  // (rows of caller-made pairs may end here)
                const int bytes = __reduce_add_sync(
                    0xffffffffu, mine ? (rowb >= 0 ? 2 * copy : copy) * rb : 0);
                const uint32_t off =
                    static_cast<uint32_t>(rowb >= 0 ? cump - own : totp + (cum - size) - cump);
                const uint32_t dst = L::kRing + stage * L::kStageBytes + 8u * off;
                const uint32_t dst_raw =
                    store == kStoreF32 ? L::kRing + stage * L::kStageBytes + 4u * (tot + off)
                                       : dst + (8u - rb) * copy;
                const uint32_t dst_mir =
                    L::kMirror + ((PAIRS ? 0u : static_cast<uint32_t>(stage) * CAP) + off) * rb;
                const int slot = __popc(slots & ((1u << lane) - 1u));
                if (mine) {
                    m.base[slot] = static_cast<int>(dst - 8u * ws - 0x58000000u);
                    m.win[slot] = make_int4(static_cast<int>(dst), copy,
                                            rowb >= 0 ? static_cast<int>(dst_mir) : 0, 0);
                    if (store == kStoreBF16 || store == kStoreF16)
                        m.scale[slot] = make_float2(
                            __ldg(P.scales + static_cast<size_t>(row) * P.n_cx + kc),
                            rowb >= 0 ? __ldg(P.scales + static_cast<size_t>(rowb) * P.n_cx + kc)
                                      : 0.0f);
#pragma unroll
                    for (int w = 0; w < NX; ++w)
                        m.r2[w][slot] = trace_r2(kc - (x0 + w + P.xoff), P.d_xl, dx2);
                }
                if (lane == 0) {
                    m.n = n;
                    m.split = split;
                    m.slo = slo;
                    m.shi = shi;
                    m.tot = tot;
                    m.tot_pairs = totp;
                }
                fence_async_smem();  // the stage's last readers and writers, then the copies
                __threadfence_block();
                __syncwarp();
                if (lane == 0 && !stall)
                    mbar_arrive_expect_tx(&full[stage], static_cast<uint32_t>(bytes));
                __syncwarp();
                if (stall) {
                    stalled = it;
                } else if (mine) {
                    const unsigned char* src = static_cast<const unsigned char*>(P.traces);
                    const size_t o = (static_cast<size_t>(row) * P.n_cx + kc) * P.ns + ws;
                    tma_load_1d(smem_u32(smem) + dst_raw, src + o * rb,
                                static_cast<uint32_t>(copy) * rb, &full[stage]);
                    if (rowb >= 0) {
                        const size_t ob = (static_cast<size_t>(rowb) * P.n_cx + kc) * P.ns + ws;
                        tma_load_1d(smem_u32(smem) + dst_mir, src + ob * rb,
                                    static_cast<uint32_t>(copy) * rb, &full[stage]);
                    }
                }
                ++it;
            }
            f += consumed;
        }
        // end-of-stream marker
        if (alive) {
            int ok = 1;
            if (lane == 0) {
                const int stage = it % kStages;
                ok = mbar_wait(&empty[stage], ((it / kStages) & 1u) ^ 1u, P.err, P.wait_us);
                if (ok) {
                    tabs[stage].n = -1;
                    __threadfence_block();
                    mbar_arrive(&full[stage]);
                }
            }
            alive = __shfl_sync(0xffffffffu, ok, 0) != 0;
            ++it;
        }
        if (!alive && lane == 0) {
            // a wait ran out: before the CTA can exit, let the bulk copies of this tile's last
            // fills land (earlier fills of a stage were consumed before it was refilled); each
            // of these waits is bounded too
            for (uint32_t i = it > it_begin + kStages ? it - kStages : it_begin; i < it; ++i)
                if (i != stalled)
                    mbar_wait(&full[i % kStages], (i / kStages) & 1u, P.err, P.wait_us);
        }
        __syncwarp();
        return alive;
    }

    if (warp == 1) {
        // ---------------------------------------------------------------- folder
        const int store = PAIRS ? kStorePairs : P.store;
        bool alive = true;
        while (true) {
            const int stage = it % kStages;
            if (!mbar_wait(&full[stage], (it / kStages) & 1u, P.err, P.wait_us)) {
                alive = false;
                break;
            }
            const Stage& m = tabs[stage];
            const int n = m.n;
            if (store == kStoreF32) {
                if (n > 0) {
                    const uint32_t d = L::kRing + stage * L::kStageBytes, a = d + 4u * m.tot;
                    const uint32_t b = L::kMirror + static_cast<uint32_t>(stage) * CAP * 4u;
                    fold_range<true, ORDERED>(smem, d, a, b, 0, m.tot_pairs, lane);
                    fold_range<false, false>(smem, d, a, b, m.tot_pairs, m.tot, lane);
                }
            } else if (!ORDERED) {
                for (int g = 0; g < n; ++g) {
                    const int4 w = m.win[g];
                    if constexpr (PAIRS)
                        fold_window<kStorePairs>(smem, w.x, w.y, w.z, make_float2(0.f, 0.f), lane);
                    else if (store == kStoreBF16)
                        fold_window<kStoreBF16>(smem, w.x, w.y, w.z, m.scale[g], lane);
                    else
                        fold_window<kStoreF16>(smem, w.x, w.y, w.z, m.scale[g], lane);
                }
            }
            fence_async_smem();  // the next fill of this stage is the async proxy's
            __syncwarp();
            if (lane == 0) mbar_arrive(&ready[stage]);
            ++it;
            if (n < 0) break;
        }
        __syncwarp();
        return alive;
    }

    // -------------------------------------------------------------------- consumers
    bool alive = true;
    // lists of (r^2, window base), one per half-warp (its crossline's r^2)
    float2* list = reinterpret_cast<float2*>(smem + L::kList) + cw * 2 * kSlots;
    const float2* mylist = list + xl * kSlots;
    const float4* bnd = reinterpret_cast<const float4*>(smem + L::kBnd) + cw * 4;
    while (true) {
        const int stage = it % kStages;
        if (!mbar_wait(&ready[stage], (it / kStages) & 1u, P.err, P.wait_us)) {
            alive = false;
            break;
        }
        const Stage& m = tabs[stage];
        const int n = m.n;
        if (n < 0) {  // end of stream: release the marker's stage too
            __syncwarp();
            if (lane == 0) mbar_arrive(&empty[stage]);
            ++it;
            break;
        }
#ifdef PSM_DEBUG_BOUNDS
        const DebugWin dbg{m.base, m.win, n, P.err};
#endif
        if (m.split) {  // part of one window: its terms one at a time
            const float r2 = m.r2[2 * xp + xl][0];
            const uint32_t base = static_cast<uint32_t>(m.base[0]);
            const float slo = m.slo, shi = m.shi;
            auto one = [&](float t2c, float f4c, float b, float& acc, float& cmp) {
                const float t2 = __fmaf_rn(f4c, r2, t2c);
                const float q = rsqrtf(t2);
                const float s = t2 * q;
                const float mm = __fadd_rd(s, 8388608.0f);
                const float lo = mm - 8388608.0f;
                if (r2 <= b && lo >= slo && lo < shi) {
                    uint32_t o = base + (__float_as_uint(mm) << 3);
#ifdef PSM_DEBUG_BOUNDS
                    o = debug_check(dbg, base, o, L::kZero);
#endif
                    const float2 a = *reinterpret_cast<const float2*>(smem + o);
                    const float v = fmaf(s - lo, a.y, a.x);
                    const float add = AMP ? v * q : v;
                    if (KAHAN) {
                        const float y = add - cmp, t = acc + y;
                        cmp = (t - acc) - y;
                        acc = t;
                    } else {
                        acc += add;
                    }
                }
            };
#pragma unroll
            for (int p = 0; p < 4; ++p) {
                one(T2[p].x, F4[p].x, BB[p].x, ACC[p].x, CMP[KAHAN ? p : 0].x);
                one(T2[p].y, F4[p].y, BB[p].y, ACC[p].y, CMP[KAHAN ? p : 0].y);
            }
        } else {
            const float* r2x = m.r2[2 * xp + xl];
            const bool in = lane < n;
            const float ra = in ? m.r2[2 * xp][lane] : 3.0e38f;
            const float rb = in ? m.r2[2 * xp + 1][lane] : 3.0e38f;
            const float base = __int_as_float(m.base[lane]);
            const unsigned lt = (1u << lane) - 1u;
#pragma unroll
            for (int h = 0; h < 4; h += 2) {  // a couple of pairs at a time
                const float4 b0 = bnd[h], b1 = bnd[h + 1];
                const bool any0 = in && (ra <= b0.x || rb <= b0.y);
                const bool any1 = in && (ra <= b1.x || rb <= b1.y);
                const bool all = in && ra <= b0.z && rb <= b0.w && ra <= b1.z && rb <= b1.w;
                const unsigned A0 = __ballot_sync(0xffffffffu, any0);
                const unsigned A1 = __ballot_sync(0xffffffffu, any1);
                if (!(A0 | A1)) continue;
                // four kinds of slots: every lane of both pairs passes; some lane of both; some
                // lane of the first pair only; of the second only
                const unsigned F = __ballot_sync(0xffffffffu, all);
                float2 s0 = KAHAN ? make_float2(0.0f, 0.0f) : ACC[h];
                float2 s1 = KAHAN ? make_float2(0.0f, 0.0f) : ACC[h + 1];
                auto both = [&](auto masked, float r2, float b) {
                    eval2<AMP, decltype(masked)::value>(smem, r2, __float_as_uint(b), T2[h], F4[h],
                                                        BB[h], L::kZero, s0 PSM_DBG_ARG);
                    eval2<AMP, decltype(masked)::value>(smem, r2, __float_as_uint(b), T2[h + 1],
                                                        F4[h + 1], BB[h + 1], L::kZero,
                                                        s1 PSM_DBG_ARG);
                };
                auto first = [&](float r2, float b) {
                    eval2<AMP, true>(smem, r2, __float_as_uint(b), T2[h], F4[h], BB[h], L::kZero,
                                     s0 PSM_DBG_ARG);
                };
                auto second = [&](float r2, float b) {
                    eval2<AMP, true>(smem, r2, __float_as_uint(b), T2[h + 1], F4[h + 1], BB[h + 1],
                                     L::kZero, s1 PSM_DBG_ARG);
                };
                if (ORDERED) {
                    // runs of one kind, in slot order
                    const float* bf = reinterpret_cast<const float*>(m.base);
                    unsigned todo = A0 | A1;
                    while (todo) {
                        int i = __clz(__brev(todo));
                        const unsigned bit = 1u << i;
                        const bool f = F & bit, p0 = A0 & bit, p1 = A1 & bit;
                        const unsigned kind = f ? F : (p0 ? A0 : ~A0) & (p1 ? A1 : ~A1) & ~F;
                        const int e = i + __clz(__brev(~(kind >> i)));
                        todo &= ~(0xffffffffu >> (kSlots - e));
                        if (f) {
                            if (i & 1) {
                                both(False{}, r2x[i], bf[i]);
                                ++i;
                            }
#pragma unroll 1
                            for (; i + 1 < e; i += 2) {
                                const float2 r = *reinterpret_cast<const float2*>(r2x + i);
                                const float2 b = *reinterpret_cast<const float2*>(bf + i);
                                both(False{}, r.x, b.x);
                                both(False{}, r.y, b.y);
                            }
                            if (i < e) both(False{}, r2x[i], bf[i]);
                        } else if (p0 && p1) {
#pragma unroll 2
                            for (; i < e; ++i) both(True{}, r2x[i], bf[i]);
                        } else if (p0) {
#pragma unroll 2
                            for (; i < e; ++i) first(r2x[i], bf[i]);
                        } else {
#pragma unroll 2
                            for (; i < e; ++i) second(r2x[i], bf[i]);
                        }
                    }
                } else {
                    // a list per kind, one after the other
                    const unsigned B = A0 & A1 & ~F, S0 = A0 & ~A1, S1 = A1 & ~A0;
                    const int nf = __popc(F), nb = nf + __popc(B), n0 = nb + __popc(S0),
                              n1 = n0 + __popc(S1);
                    const unsigned peers = all ? F : any0 && any1 ? B : any0 ? S0 : S1;
                    const int off = all ? 0 : any0 && any1 ? nf : any0 ? nb : n0;
                    if (h) __syncwarp();
                    if (any0 || any1) {
                        float2* e = list + off + __popc(peers & lt);
                        e[0] = make_float2(ra, base);
                        e[kSlots] = make_float2(rb, base);
                    }
                    __syncwarp();
                    int i = 0;
#pragma unroll 1
                    for (; i + 1 < nf; i += 2) {
                        const float4 e = *reinterpret_cast<const float4*>(mylist + i);
                        both(False{}, e.x, e.y);
                        both(False{}, e.z, e.w);
                    }
                    // (the last of an odd number joins the masked ones: its masks pass)
#pragma unroll 2
                    for (; i < nb; ++i) {
                        const float2 e = mylist[i];
                        both(True{}, e.x, e.y);
                    }
#pragma unroll 2
                    for (; i < n0; ++i) {
                        const float2 e = mylist[i];
                        first(e.x, e.y);
                    }
#pragma unroll 2
                    for (; i < n1; ++i) {
                        const float2 e = mylist[i];
                        second(e.x, e.y);
                    }
                }
                if (KAHAN) {  // ACC += partial, compensated
                    const int k0 = KAHAN ? h : 0, k1 = KAHAN ? h + 1 : 0;
                    const float2 y0 = sub2(s0, CMP[k0]), t0 = add2(ACC[h], y0);
                    CMP[k0] = sub2(sub2(t0, ACC[h]), y0);
                    ACC[h] = t0;
                    const float2 y1 = sub2(s1, CMP[k1]), t1 = add2(ACC[h + 1], y1);
                    CMP[k1] = sub2(sub2(t1, ACC[h + 1]), y1);
                    ACC[h + 1] = t1;
                } else {
                    ACC[h] = s0;
                    ACC[h + 1] = s1;
                }
            }
        }
        __syncwarp();
        if (lane == 0) mbar_arrive(&empty[stage]);
        ++it;
    }

    // ---- write the tile: weight 1/(t v^2) = (dt/t) * inv_dt / v^2 applied per output sample
    if (x < P.n_ox) {
        const int vc = vrms_col(P, x);
        const float* vp = vrms_trace(P, job.vrow, vc >= 0 ? vc : 0);
        float* op = P.image + (static_cast<size_t>(job.row) * P.n_ox + x) * P.n_t;
#pragma unroll
        for (int p = 0; p < 4; ++p) {
#pragma unroll
            for (int c = 0; c < 2; ++c) {
                const int t = T0 + 64 * p + 32 * ph + 16 * c + (lane & 15);
                if (t < P.n_t) {
                    float o = 0.0f;
                    if ((c ? BB[p].y : BB[p].x) >= 0.0f) {
                        o = c ? ACC[p].y : ACC[p].x;
                        if (AMP) {
                            const float v = __ldg(vp + t);
                            o *= __fdiv_rn(P.inv_dt, __fmul_rn(v, v));
                        }
                    }
                    op[t] = o;
                }
            }
        }
    }
    return alive;
}

// The ring's mbarriers: full (one producer arrival + the TMA bytes), ready (the folder), empty
// (every consumer); and the zero sample that failing terms read.
template <int NX, int CAP>
__device__ __forceinline__ void ring_init(unsigned char* smem) {
    using L = FwdLayout<NX, CAP>;
    uint64_t* bar = reinterpret_cast<uint64_t*>(smem);
    for (int s = 0; s < kStages; ++s) {
        mbar_init(bar + s, 1);
        mbar_init(bar + kStages + s, 1);
        mbar_init(bar + 2 * kStages + s, NX);
    }
    *reinterpret_cast<float4*>(smem + L::kZero) = make_float4(0.f, 0.f, 0.f, 0.f);
    fence_barrier_init();
}

// ----------------------------------------------------------------------------- kernels

// One tile per CTA: grid (crossline tiles, jobs, time tiles).  The time tile is the slowest
// dimension, deepest first: the block scheduler starts CTAs in grid order, and a deep tile
// holds several times the terms of a shallow one (the aperture grows with t0), so the light
// tiles come last and the launch's tail is short.
template <bool AMP, bool KAHAN, bool ORDERED, int NX, int CAP, int MINB>
__global__ void __launch_bounds__(32 * (NX + 2), MINB) fwd_kernel(const FwdParams P) {
    extern __shared__ __align__(128) unsigned char smem_raw[];
    if (threadIdx.x == 0) ring_init<NX, CAP>(smem_raw);  // ordered by the tile's first barrier
    uint32_t it = 0;
    fwd_tile<AMP, KAHAN, ORDERED, NX, CAP>(P, P.jobs[blockIdx.y], blockIdx.x * NX,
                                           static_cast<int>(gridDim.z - 1 - blockIdx.z) * kTileT,
                                           smem_raw, it);
}

// The same on caller-made pairs, a kernel of its own, so that the others carry none of it.
template <bool AMP, int NX, int CAP, int MINB>
__global__ void __launch_bounds__(32 * (NX + 2), MINB) fwd_pairs_kernel(const FwdParams P) {
    extern __shared__ __align__(128) unsigned char smem_raw[];
    if (threadIdx.x == 0) ring_init<NX, CAP>(smem_raw);
    uint32_t it = 0;
    fwd_tile<AMP, false, false, NX, CAP, true>(
        P, P.jobs[blockIdx.y], blockIdx.x * NX,
        static_cast<int>(gridDim.z - 1 - blockIdx.z) * kTileT, smem_raw, it);
}

// Parameters of every problem of a batched launch, passed by value: they live in the
// kernel-parameter constant bank, whose loads are cached and uniform across the CTA.
constexpr int kMaxBatchProblems = 184;
struct BatchParams {
    FwdParams p[kMaxBatchProblems];
};
static_assert(sizeof(BatchParams) + 64 <= 32764, "kernel parameters are limited to 32764 bytes");

// Persistent batched launch: each CTA takes tiles from the shared list in order (an atomic
// counter) until the list is exhausted, with the ring kept across tiles.  Problems (velocity
// panels, sub-volumes) each have their own FwdParams.  A device error (bounded wait expired)
// stops every CTA at its next tile.
template <bool AMP, bool KAHAN, int NX, int CAP, int MINB>
__global__ void __launch_bounds__(32 * (NX + 2), MINB)
    fwd_batch_kernel(const __grid_constant__ BatchParams B, const BatchItem* __restrict__ items,
                     int n_items, int* next, const int* err) {
    extern __shared__ __align__(128) unsigned char smem_raw[];
    __shared__ BatchItem s_item;
    __shared__ Job s_job;
    if (threadIdx.x == 0) ring_init<NX, CAP>(smem_raw);
    uint32_t it = 0;
    while (true) {
        if (threadIdx.x == 0) {
            const int k = *reinterpret_cast<const volatile int*>(err) ? n_items
                                                                      : atomicAdd(next, 1);
            s_item = k < n_items ? items[k] : BatchItem{-1, 0, 0, 0};
            if (k < n_items) s_job = B.p[s_item.prob].jobs[s_item.job];
        }
        __syncthreads();
        const BatchItem w = s_item;
        if (w.prob < 0) break;
        const bool ok =
            fwd_tile<AMP, KAHAN, false, NX, CAP>(B.p[w.prob], s_job, w.x0, w.T0, smem_raw, it);
        // barrier: the tile's tables, statistics, s_item and s_job are reused next
        if (__syncthreads_or(!ok)) break;
    }
}

// The same tile list in ONE grid launch: CTA b migrates tile items[b] (deepest tiles first in
// the depth-first order), and the hardware's block scheduler hands tiles to SMs as others
// finish, so the CTAs carry no state from tile to tile.
template <bool AMP, bool KAHAN, int NX, int CAP, int MINB>
__global__ void __launch_bounds__(32 * (NX + 2), MINB)
    fwd_items_kernel(const __grid_constant__ BatchParams B,
                     const BatchItem* __restrict__ items) {
    extern __shared__ __align__(128) unsigned char smem_raw[];
    if (threadIdx.x == 0) ring_init<NX, CAP>(smem_raw);
    const BatchItem w = items[blockIdx.x];
    const FwdParams& P = B.p[w.prob];
    uint32_t it = 0;
    fwd_tile<AMP, KAHAN, false, NX, CAP>(P, P.jobs[w.job], w.x0, w.T0, smem_raw, it);
}

}  // namespace psm
