// Recursive Gaussian blurs (Young and van Vliet, third order) over whole lines held in shared memory,
// evaluated block-parallel.
//
// The recurrence of one line (reference kernels/fx_blur.metal:125-170):
//   forward   w[i] = B x[i] + B1 w[i-1] + B2 w[i-2] + B3 w[i-3],  w[-1] = w[-2] = w[-3] = x[0];  u[i] = float(w[i])
//   backward  y[i] = B u[i] + B1 y[i+1] + B2 y[i+2] + B3 y[i+3],  y[n] = y[n+1] = y[n+2] = u[n-1]
// is a linear time-invariant system, so a line cut into segments of L samples can be solved in three
// steps (the block decomposition of Nehab, Maximo, Lima and Hoppe, "GPU-efficient recursive filtering
// and summed-area tables", SIGGRAPH Asia 2011):
//   1. every segment runs the recurrence from a zero state (the first segment from the true edge
//      state) and keeps its last three values e_s;
//   2. the true state entering segment s+1 is S_s = e_s + M S_{s-1}, with M the 3 x 3 map of an
//      entry state through L steps of the homogeneous recurrence (a parallel scan over the segments);
//   3. every segment recomputes from its true entry state and stores its values.
// State and the carries are binary64 (the reference keeps double-float state on its GPU and double
// state on its host copy); x, u and y are stored as binary32 exactly as there.
//
// k_iir_rows: one CTA per image row, 3 lines x kSegRows segments; the row (3 w floats) in shared memory,
//             loaded afresh for every mixture component, blurred and written to the component's plane.
// k_iir_cols: one CTA per strip of 4 pixel columns (12 lines); every component's row result blurred
//             down the columns in turn; the mixture accumulated as the reference's fused passes do
//             (acc = 0 + w0 y0, acc = acc + w_k y_k) in tensor memory, and the halation mix raw := a raw +
//             b acc written in place of raw; a plain blur (one component) stores its lines as they are.
//             A strip comes into shared memory by TMA: the component's plane, its rows padded to a multiple
//             of 4 pixels, is a 2-D tensor (3 pitch floats x h rows), and the strip is a column of 12-float
//             boxes of up to 256 rows, all completing on one mbarrier.
//             Column pass, the sum in a global plane and scalar copies at odd widths before: 3840 x 2160, two
//             components 0.290 -> 0.239 ms; 6000 x 4000, two 1.06 -> 0.88; 1999 x 1333, two 0.219 -> 0.100.
//             With three components at 6000 x 4000 the loads take 0.29 ms, raw 0.28, the recurrences the rest
//             (one strip of twelve warps per SM; the 32-to-64-bit conversions' unit is the busiest there).
//             Loading and converting eight samples ahead of their chain made the recurrences slower (0.88 ->
//             1.09 ms; rows at 4K 0.150 -> 0.187): the unrolled loop already overlaps them. Short frames with
//             many strips run three strips an SM instead of two (three_strips).
//             Its waits are bounded: one that gives up counts
//             itself (g_iir_gave_up), waits again under the full limit for the copies in flight, and if
//             even they never land the CTA loads this and every later strip with plain copies.
#include <cuda.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include <atomic>
#include <mutex>

#include "../kernel_args.h"
#include "iir.hpp"

namespace spkb::dev {

namespace {

#ifndef SPKB_IIR_SEG_ROWS
#define SPKB_IIR_SEG_ROWS 64
#endif
constexpr int kSegRows = SPKB_IIR_SEG_ROWS;  // segments per channel line in a row (4K rows: 0.185 ms at 128, 0.152 at 64)
static_assert(kSegRows <= (1 << kIirScanSteps), "the carry scan composes at most 2^kIirScanSteps segments");
constexpr int kRowThreads = 3 * kSegRows;
constexpr int kColPixels = 4;       // pixels per column strip
constexpr int kColLines = 3 * kColPixels;
#ifndef SPKB_IIR_SEG_COLS
#define SPKB_IIR_SEG_COLS 32
#endif
constexpr int kSegCols = SPKB_IIR_SEG_COLS;  // segments per column line (32: two 4K strips per SM)
static_assert(kSegCols <= (1 << kIirScanSteps), "the carry scan composes at most 2^kIirScanSteps segments");
constexpr int kColThreads = kColLines * kSegCols;

// One pass's coefficients for up to N components, as a kernel argument: both passes of eight components by
// value are 26 KB, which a small frame's launches copy longer than its blur takes.
template <int N>
struct IirPass {
    int32_t seg_len, adjoint;
    IirChannel ch[3 * N];
    IirPass(const IirLaunch& q, uint32_t ncomp) : seg_len(q.seg_len), adjoint(q.adjoint) {
        for (uint32_t i = 0; i < 3 * ncomp; ++i) ch[i] = q.ch[i];
    }
};

// The column pass's tensor maps, one per component plane, and the strip's box geometry: `boxes` boxes of
// `box_rows` rows (a multiple of 8, at most 256) cover the frame's rows; the strip buffer holds
// boxes * box_rows rows, and the rows past the frame are zero-filled by the copy and never read.
struct IirColMaps {
    CUtensorMap map[SPKB_MAX_COMPONENTS];
    long long wait_limit;  // SM clocks a strip wait may take before it gives up
    uint32_t box_rows, boxes;
    uint32_t use_tma;      // 0: plain copies (a pitch that is not a multiple of 4, or no tensor map)
    uint32_t tmem_cols;    // tensor-memory columns of the mixture's sum; 0: one component, no sum to keep
};

#ifndef SPKB_IIR_COL_TMA
#define SPKB_IIR_COL_TMA 1
#endif
constexpr bool kColTma = SPKB_IIR_COL_TMA != 0;  // 0: every strip by plain 16-byte copies

constexpr long long kWaitCycles = 4000000000LL;  // about 2 s at the B200's clocks
__device__ unsigned int g_iir_gave_up;           // strip waits that gave up, since the last read

__device__ __forceinline__ uint32_t smem_addr(const void* p) { return uint32_t(__cvta_generic_to_shared(p)); }

__device__ __forceinline__ void mbar_init(uint32_t bar, uint32_t count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count) : "memory");
}
__device__ __forceinline__ void fence_mbar_init() { asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory"); }

// this thread's earlier shared-memory accesses ordered before the asynchronous (TMA) proxy's next ones
__device__ __forceinline__ void fence_proxy_async() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }

__device__ __forceinline__ void mbar_arrive_expect_tx(uint32_t bar, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
}

__device__ __forceinline__ bool mbar_try(uint32_t bar, uint32_t parity) {
    uint32_t done;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(done)
        : "r"(bar), "r"(parity)
        : "memory");
    return done != 0;
}

// the phase's completion tested without waiting
__device__ __forceinline__ bool mbar_test(uint32_t bar, uint32_t parity) {
    uint32_t done;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.test_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(done)
        : "r"(bar), "r"(parity)
        : "memory");
    return done != 0;
}

// the barrier's phase of the given parity completed; false once `limit` SM clocks have passed without it.
// try_wait may suspend the thread for a while by itself, so a shortened limit (the test hook) polls with
// the non-blocking test_wait instead.
__device__ __forceinline__ bool mbar_wait(uint32_t bar, uint32_t parity, long long limit) {
    if (limit < kWaitCycles) {
        const long long t0 = clock64();
        for (;;) {
            if (mbar_test(bar, parity)) return true;
            if (clock64() - t0 > limit) return false;
        }
    }
    if (mbar_try(bar, parity)) return true;
    const long long t0 = clock64();
    for (;;) {
        if (mbar_try(bar, parity)) return true;
        if (clock64() - t0 > limit) return false;
    }
}

// one box of a 2-D tensor map at element coordinates (x, y) into shared memory, completing on `bar`
__device__ __forceinline__ void tma_load_2d(uint32_t dst, const CUtensorMap* map, int x, int y, uint32_t bar) {
    asm volatile(
        "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];" ::"r"(dst),
        "l"(reinterpret_cast<uint64_t>(map)), "r"(x), "r"(y), "r"(bar)
        : "memory");
}

struct Coef {
    double B, B1, B2, B3;
};

// A step of the recurrence takes the oldest state first and the newest last: each state is j steps old when
// it enters the j-th multiply-add from the end, so the chain costs one multiply-add latency per sample.
// One pass over the segment [a, b) of a line in shared memory (element i at base[i * stride]), ascending or
// descending. Zero-state run: returns the end state. Writing run: from the state given, stores float(w)
// back.

template <bool FORWARD, bool WRITE>
__device__ __forceinline__ void seg_run(const Coef& k, float* base, int stride, int a, int b, double& s1, double& s2,
                                        double& s3) {
    const int n = b - a, dir = FORWARD ? stride : -stride;
    float* p = base + (FORWARD ? a : b - 1) * stride;
    const auto chain = [&](double kx) {
        const double t = fma(k.B1, s1, fma(k.B2, s2, fma(k.B3, s3, kx)));
        s3 = s2;
        s2 = s1;
        s1 = t;
        return float(t);
    };
#pragma unroll 4
    for (int i = 0; i < n; ++i, p += dir) {
        const float v = chain(k.B * double(*p));
        if (WRITE) *p = v;
    }
}

// The true entry states of the segments, by a Kogge-Stone scan of the zero-state end states e_s held in
// carry (log2 of the segment count in steps rather than one serial pass per line):
//   forward   S_s = e_s + M S_{s-1}, s = 1 .. last-1; S_0 = e_0 is already true (the edge state)
//   backward  S_s = e_s + M S_{s+1}, s = last-1 .. 0; S_last = e_last is already true
// Step p adds M^(2^p) times the carry 2^p segments away. The segments whose maps are composed are full
// length, so M is the same for each. Every thread of the block runs the loop (it has barriers).
__device__ void carry_scan(double* carry, int nt, int cstep, int seg, int last, const IirChannel& ch, bool active,
                           bool forward) {
    // component i of thread t's carry at carry[i * nt + t]; the neighbouring segment's is cstep away
    double* cs = carry + threadIdx.x;
    for (int p = 0, k = 1; k <= last; ++p, k <<= 1) {
        const int src = forward ? seg - k : seg + k;
        const bool upd = active && (forward ? (src >= 0 && seg <= last - 1) : src <= last);
        double n0 = 0.0, n1 = 0.0, n2 = 0.0;
        if (upd) {
            const double* ps = cs + (forward ? -k : k) * cstep;
            const double p0 = ps[0], p1 = ps[nt], p2 = ps[2 * nt];
            const double(&M)[3][3] = ch.Mp[p];
            n0 = cs[0] + (M[0][0] * p0 + M[0][1] * p1 + M[0][2] * p2);
            n1 = cs[nt] + (M[1][0] * p0 + M[1][1] * p1 + M[1][2] * p2);
            n2 = cs[2 * nt] + (M[2][0] * p0 + M[2][1] * p1 + M[2][2] * p2);
        }
        __syncthreads();
        if (upd) {
            cs[0] = n0;
            cs[nt] = n1;
            cs[2 * nt] = n2;
        }
        __syncthreads();
    }
}

// The transpose's edge term: v[e] += ((B1 + B2 + B3) v[e] + (B2 + B3) v[e + step] + B3 v[e + 2 step]) / B,
// with the samples that exist (a line shorter than three samples folds what it has)
__device__ __forceinline__ void edge_fold(const Coef& k, float* base, int e, int step, int n, bool doit) {
    if (!doit) return;
    const double v0 = base[e];
    const double v1 = n > 1 ? double(base[e + step]) : 0.0;
    const double v2 = n > 2 ? double(base[e + 2 * step]) : 0.0;
    base[e] = float(v0 + (((k.B1 + k.B2) + k.B3) * v0 + (k.B2 + k.B3) * v1 + k.B3 * v2) / k.B);
}

// One full forward + backward blur of `nlines` interleaved lines of length n held in shared memory
// (line j, element i at buf[i * pitch + j]), nseg segments per line, threads = nlines * nseg. Thread t
// handles line t / nseg, segment t % nseg when seg_major, else line t % nlines, segment t / nlines; the
// channel of line j is 3 comp + j % 3. carry: shared scratch of 3 * nlines * nseg doubles, component i of
// thread t's segment at carry[i * nlines * nseg + t].
template <int N>
__device__ __forceinline__ void blur_lines(float* buf, int pitch, int nlines, int n, int nseg, const IirPass<N>& q, int comp,
                           double* carry, bool seg_major) {
    const int t = threadIdx.x;
    const int line = seg_major ? t / nseg : t % nlines;
    const int seg = seg_major ? t % nseg : t / nlines;
    const int cstep = seg_major ? 1 : nlines;  // carry distance between neighbouring segments of a line
    const int L = q.seg_len;
    const int a = seg * L;
    const int b = min(n, a + L);
    const IirChannel& ch = q.ch[3 * comp + line % 3];
    const bool active = ch.active != 0 && line < nlines;
    const Coef k{ch.B, ch.B1, ch.B2, ch.B3};
    float* base = buf + line;
    const int nt = nlines * nseg;
    double* cs = carry + t;

    const bool adj = q.adjoint != 0;
    // ---- forward ----
    if (active && a < n) {
        double s1 = 0.0, s2 = 0.0, s3 = 0.0;
        if (seg == 0 && !adj) s1 = s2 = s3 = double(base[0]);
        seg_run<true, false>(k, base, pitch, a, b, s1, s2, s3);
        cs[0] = s1;
        cs[nt] = s2;
        cs[2 * nt] = s3;
    }
    __syncthreads();
    const int nseg_used = (n + L - 1) / L;
    const int last = nseg_used - 1;
    carry_scan(carry, nt, cstep, seg, last, ch, active, true);
    if (active && a < n) {
        double s1, s2, s3;
        if (seg == 0) {
            s1 = s2 = s3 = adj ? 0.0 : double(base[0]);
        } else {
            const double* prev = cs - cstep;
            s1 = prev[0];
            s2 = prev[nt];
            s3 = prev[2 * nt];
        }
        seg_run<true, true>(k, base, pitch, a, b, s1, s2, s3);
    }
    __syncthreads();
    if (adj) {
        // the forward blur's anticausal pass starts from y[n..n+2] = u[n-1]: its transpose adds
        // ((B1 + B2 + B3) l[n-1] + (B2 + B3) l[n-2] + B3 l[n-3]) / B to sample n-1
        edge_fold(k, base, (n - 1) * pitch, -pitch, n, active && seg == 0);
        __syncthreads();
    }
    // ---- backward ----
    if (active && a < n) {
        double s1 = 0.0, s2 = 0.0, s3 = 0.0;
        if (seg == last && !adj) s1 = s2 = s3 = double(base[(n - 1) * pitch]);
        seg_run<false, false>(k, base, pitch, a, b, s1, s2, s3);
        cs[0] = s1;
        cs[nt] = s2;
        cs[2 * nt] = s3;
    }
    __syncthreads();
    carry_scan(carry, nt, cstep, seg, last, ch, active, false);
    if (active && a < n) {
        double s1, s2, s3;
        if (seg == last) {
            s1 = s2 = s3 = adj ? 0.0 : double(base[(n - 1) * pitch]);
        } else {
            const double* prev = cs + cstep;
            s1 = prev[0];
            s2 = prev[nt];
            s3 = prev[2 * nt];
        }
        seg_run<false, true>(k, base, pitch, a, b, s1, s2, s3);
    }
    __syncthreads();
    if (adj) {
        // the forward blur's causal pass starts from w[-1..-3] = x[0]: its transpose folds into sample 0
        edge_fold(k, base, 0, pitch, n, active && seg == 0);
        __syncthreads();
    }
}

// 16-byte asynchronous copy global -> shared (both addresses 16-byte aligned), and the wait for all of
// this thread's copies
// blur_lines as a call: with registers for three CTAs an SM the inlined body spills into its loops (1600 x 200, eight
// components 0.121 ms inlined, 0.089 called)
template <int N>
__device__ __noinline__ void blur_lines_call(float* buf, int pitch, int nlines, int n, int nseg, const IirPass<N>& q,
                                             int comp, double* carry, bool seg_major) {
    blur_lines(buf, pitch, nlines, n, nseg, q, comp, carry, seg_major);
}

__device__ __forceinline__ void cp_async16(void* dst, const void* src) {
    const unsigned d = static_cast<unsigned>(__cvta_generic_to_shared(dst));
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(d), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async_wait_all() { asm volatile("cp.async.wait_all;" ::: "memory"); }

__device__ __forceinline__ void cp_async4(void* dst, const void* src) {
    const unsigned d = static_cast<unsigned>(__cvta_generic_to_shared(dst));
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(d), "l"(src) : "memory");
}

template <int N>
__global__ void __launch_bounds__(kRowThreads) k_iir_rows(const float* __restrict__ in, const __grid_constant__ IirPlanes outs, uint32_t w,
                                                          uint32_t h, const __grid_constant__ IirSum mix,
                                                          const __grid_constant__ IirPass<N> pass) {
    extern __shared__ __align__(128) unsigned char smem[];
    const uint32_t y = blockIdx.x;
    if (y >= h) return;
    const int n3 = int(3 * w), p3 = int(3 * mix.pitch);
    const int n3r = (p3 + 3) & ~3;  // keeps carry 16-byte aligned
    float* work = reinterpret_cast<float*>(smem);
    double* carry = reinterpret_cast<double*>(work + n3r);
    const float* src = in + size_t(y) * n3;
    const bool vec = (n3 & 3) == 0;  // the source's rows start on 16-byte boundaries
    for (int i = n3 + int(threadIdx.x); i < p3; i += blockDim.x) work[i] = 0.0f;  // the padding
    for (int c = 0; c < int(mix.ncomp); ++c) {
        // each component blurs the row afresh: the source row is read again (from L2 after the first)
        if (vec) {
            for (int i = threadIdx.x; i < n3 / 4; i += blockDim.x) cp_async16(work + 4 * i, src + 4 * i);
        } else {
#pragma unroll 4
            for (int i = threadIdx.x; i < n3; i += blockDim.x) cp_async4(work + i, src + i);
        }
        cp_async_wait_all();
        __syncthreads();
        blur_lines(work, 3, 3, int(w), kSegRows, pass, c, carry, true);
        float* dst = outs.p[c] + size_t(y) * p3;
        if ((p3 & 3) == 0) {
            for (int i = threadIdx.x; i < p3 / 4; i += blockDim.x)
                reinterpret_cast<float4*>(dst)[i] = reinterpret_cast<const float4*>(work)[i];
        } else {
            for (int i = threadIdx.x; i < p3; i += blockDim.x) dst[i] = work[i];
        }
        __syncthreads();
    }
}

// The mixture's sum lives in tensor memory, used as the strip's scratch: the 12 n floats that a global plane
// would have to hold (written, read and written again for every component but one) do not fit beside
// the strip in shared memory, but they fill at most 435 of the SM's 512 columns of 128 words. Quad i (four
// floats of a strip row, three to a row) belongs to thread i % kColThreads, which keeps it in its own lane at
// columns 4 (i / 128) ..: warp w's lanes start at 32 (w % 4), and its 32 quads of turn k are 384 k + 32 w ...
// Only the owner ever reads a quad, so no barrier orders the accesses.
__device__ __forceinline__ void tmem_alloc(uint32_t slot, uint32_t cols) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(slot), "r"(cols) : "memory");
}
__device__ __forceinline__ void tmem_relinquish() {
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_dealloc(uint32_t taddr, uint32_t cols) {
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(cols) : "memory");
}
__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
__device__ __forceinline__ float4 tmem_ld4(uint32_t taddr) {
    uint32_t r[4];
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x4.b32 {%0, %1, %2, %3}, [%4];\n\t"
        "tcgen05.wait::ld.sync.aligned;"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
        : "r"(taddr)
        : "memory");
    return make_float4(__uint_as_float(r[0]), __uint_as_float(r[1]), __uint_as_float(r[2]), __uint_as_float(r[3]));
}
__device__ __forceinline__ void tmem_st4(uint32_t taddr, const float4& v) {
    asm volatile("tcgen05.st.sync.aligned.32x32b.x4.b32 [%0], {%1, %2, %3, %4};" ::"r"(taddr),
                 "r"(__float_as_uint(v.x)), "r"(__float_as_uint(v.y)), "r"(__float_as_uint(v.z)), "r"(__float_as_uint(v.w))
                 : "memory");
}
__device__ __forceinline__ void tmem_wait_st() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }

constexpr int kQuads = kColLines / 4, kQuadRows = kColThreads / kQuads;
static_assert(kQuads == 3 && kColThreads == 384, "the tensor-memory layout above");

// One thread's weights of its four channels
struct QuadWeights {
    float w[4];
};
__device__ __forceinline__ QuadWeights quad_weights(const float (&w)[3]) {
    const int j = 4 * (int(threadIdx.x) % kQuads);
    return {{w[j % 3], w[(j + 1) % 3], w[(j + 2) % 3], w[j % 3]}};
}
template <bool MULTI>
__device__ __forceinline__ float4 sum_quad(const QuadWeights& wc, const float4& v, bool first, uint32_t taddr) {
    if (!MULTI || first) return make_float4(0.0f + wc.w[0] * v.x, 0.0f + wc.w[1] * v.y, 0.0f + wc.w[2] * v.z, 0.0f + wc.w[3] * v.w);
    const float4 a = tmem_ld4(taddr);
    return make_float4(a.x + wc.w[0] * v.x, a.y + wc.w[1] * v.y, a.z + wc.w[2] * v.z, a.w + wc.w[3] * v.w);
}

// mix_a raw + mix_b sum with the product of x unrounded. Frames whose width is a multiple of 4 take x = mix_a
// raw and the others x = mix_b sum: either is within the sum's rounding, and each keeps the bits that the
// renders of its frames have always had.
__device__ __forceinline__ float mix2(float mx, float x, float my, float y) { return __fmaf_rn(mx, x, __fmul_rn(my, y)); }

// The blurred strip of component c joins the sum: acc := 0 + w v or acc + w v. The result goes back to the
// tensor memory, or (to_strip) over the strip. Every lane of a warp with a quad left takes part in the
// tensor-memory accesses, those past the frame's rows with zeros: a strip row is read and written by its
// owner alone.
template <bool MULTI>
__device__ __forceinline__ void strip_sum(float* strip, int n, const IirSum& mix, int c, uint32_t tmem, bool to_strip) {
    const int warp = int(threadIdx.x) >> 5, qd = int(threadIdx.x) % kQuads, last = n - 1;
    const QuadWeights wc = quad_weights(mix.weight[c]);
    uint32_t taddr = tmem + (uint32_t(32 * (warp & 3)) << 16) + 4u * uint32_t(warp >> 2);
    for (int q0 = 32 * warp, row = int(threadIdx.x) / kQuads; q0 < kQuads * n; q0 += kColThreads, row += kQuadRows, taddr += 12u) {
        float4* at = reinterpret_cast<float4*>(strip + size_t(min(row, last)) * kColLines + 4 * qd);
        const float4 v = row <= last ? *at : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        const float4 a = sum_quad<MULTI>(wc, v, c == 0, taddr);
        if (MULTI && !to_strip) tmem_st4(taddr, a);
        else if (row <= last) *at = a;
    }
    if (MULTI && !to_strip) tmem_wait_st();
}

// raw := mix_a raw + mix_b (the sum after the last component c), or the strip as it is (plain), in float4.
// A thread steps down the rows BATCH at a time, their reads issued before the first store (4K 0.239 ms at one and
// two, 0.258 at four; 6000 x 4000 0.93, 0.88, 0.87).
template <bool MULTI, int BATCH>
__device__ __forceinline__ void strip_to_raw(const float* strip, float* raw, size_t pitch, int n, const IirSum& mix,
                                             int c, uint32_t tmem) {
    const int warp = int(threadIdx.x) >> 5, qd = int(threadIdx.x) % kQuads;
    const QuadWeights wc = quad_weights(mix.weight[c]), ma = quad_weights(mix.mix_a), mb = quad_weights(mix.mix_b);
    const bool plain = mix.plain != 0;
    uint32_t taddr = tmem + (uint32_t(32 * (warp & 3)) << 16) + 4u * uint32_t(warp >> 2);
    int row = int(threadIdx.x) / kQuads;
    float* out = raw + size_t(row) * pitch + 4 * qd;
    const size_t step = size_t(kQuadRows) * pitch;
    for (int q0 = 32 * warp; q0 < kQuads * n; q0 += BATCH * kColThreads) {
        float4 rw[BATCH];
        if (!plain) {
#pragma unroll
            for (int u = 0; u < BATCH; ++u)
                if (row + u * kQuadRows < n) rw[u] = *reinterpret_cast<const float4*>(out + u * step);
        }
#pragma unroll
        for (int u = 0; u < BATCH; ++u) {
            if (q0 + u * kColThreads >= kQuads * n) break;
            const int r = min(row, n - 1);
            float4 v = *reinterpret_cast<const float4*>(strip + size_t(r) * kColLines + 4 * qd);
            if (!plain) {
                const float4 a = sum_quad<MULTI>(wc, v, c == 0, taddr);
                v.x = mix2(ma.w[0], rw[u].x, mb.w[0], a.x);
                v.y = mix2(ma.w[1], rw[u].y, mb.w[1], a.y);
                v.z = mix2(ma.w[2], rw[u].z, mb.w[2], a.z);
                v.w = mix2(ma.w[3], rw[u].w, mb.w[3], a.w);
            }
            if (row < n) *reinterpret_cast<float4*>(out) = v;
            row += kQuadRows;
            out += step;
            taddr += 12u;
        }
    }
}

// The same from a strip that holds the sum (or the plain blur) to a raw whose rows are not aligned, or a
// strip cut by the frame's edge: a float at a time, nl to a row
__device__ __forceinline__ void strip_to_raw_scalar(const float* strip, float* raw, size_t pitch, int nl, int n,
                                                    const IirSum& mix) {
    constexpr int kStep = kColThreads / kColLines, kBatch = 8;
    const int j = int(threadIdx.x) % kColLines;
    if (j >= nl) return;
    const float ma = mix.mix_a[j % 3], mb = mix.mix_b[j % 3];
    for (int r = int(threadIdx.x) / kColLines; r < n; r += kBatch * kStep) {
        float rw[kBatch];
        if (!mix.plain) {
#pragma unroll
            for (int u = 0; u < kBatch; ++u)
                if (r + u * kStep < n) rw[u] = raw[size_t(r + u * kStep) * pitch + j];
        }
#pragma unroll
        for (int u = 0; u < kBatch; ++u) {
            const int row = r + u * kStep;
            if (row >= n) break;
            const float a = strip[size_t(row) * kColLines + j];
            raw[size_t(row) * pitch + j] = mix.plain ? a : mix2(mb, a, ma, rw[u]);
        }
    }
}

// MULTI: more than one component, the sum in tensor memory. CTAS: the strips per SM that the registers allow. Two
// (what shared memory holds at 4K) are faster each; a strip of a short frame is latency from barrier to
// barrier, and where there are more than two for every SM three at a time are faster together (three_strips).
template <bool MULTI, int N, int CTAS>
__global__ void __launch_bounds__(kColThreads, CTAS) k_iir_cols(float* raw, const __grid_constant__ IirPlanes hs, uint32_t w, uint32_t h,
                                                          const __grid_constant__ IirSum mix,
                                                          const __grid_constant__ IirPass<N> pass,
                                                          const __grid_constant__ IirColMaps maps) {
    extern __shared__ __align__(128) unsigned char smem[];
    const uint32_t x0 = blockIdx.x * kColPixels;
    const int px = min(kColPixels, int(w) - int(x0));
    const int nl = 3 * px;  // valid lines in this strip
    const int n = int(h);
    // [row][kColLines], boxes * box_rows rows (each box's first row 128-byte aligned: box_rows is a
    // multiple of 8 and a row is 48 bytes), then the carries, then the strip's mbarrier
    const size_t rows_alloc = size_t(maps.box_rows) * maps.boxes;
    float* strip = reinterpret_cast<float*>(smem);
    double* carry = reinterpret_cast<double*>(strip + rows_alloc * kColLines);
    const uint32_t bar = smem_addr(carry + size_t(kColLines) * kSegCols * 3);
    const size_t pitch = 3 * size_t(mix.pitch), raw_pitch = 3 * size_t(w);
    const size_t off = 3 * size_t(x0);
    // rows of the component planes and the sum (vec), of raw (raw_vec), as three aligned float4 a strip row
    const bool vec = (mix.pitch & 3u) == 0, raw_vec = px == kColPixels && (w & 3u) == 0;
    bool tma = vec && maps.use_tma != 0;  // the same in every thread of the CTA
    if (tma) {
        if (threadIdx.x == 0) {
            mbar_init(bar, 1);
            fence_mbar_init();
        }
        __syncthreads();
    }
    const uint32_t tmem_slot = bar + 8;
    uint32_t tmem = 0;
    if (MULTI) {
        if (threadIdx.x < 32) {
            tmem_alloc(tmem_slot, maps.tmem_cols);
            tmem_relinquish();
        }
        tc_fence_before();
        __syncthreads();
        tc_fence_after();
        asm volatile("ld.shared.u32 %0, [%1];" : "=r"(tmem) : "r"(tmem_slot) : "memory");
    }
    for (int c = 0; c < int(mix.ncomp); ++c) {
        const float* src = hs.p[c];
        if (tma) {
            if (threadIdx.x == 0) {
                fence_proxy_async();  // the previous component's reads and writes of the strip come first
                mbar_arrive_expect_tx(bar, maps.boxes * maps.box_rows * uint32_t(kColLines * sizeof(float)));
                for (uint32_t k = 0; k < maps.boxes; ++k)
                    tma_load_2d(smem_addr(strip + size_t(k) * maps.box_rows * kColLines), &maps.map[c], int(off),
                                int(k * maps.box_rows), bar);
            }
            // component c completes the barrier's phase c
            const uint32_t parity = uint32_t(c) & 1u;
            bool gave_up = false, landed = true;
            if (!mbar_wait(bar, parity, maps.wait_limit)) {
                gave_up = true;
                landed = mbar_wait(bar, parity, kWaitCycles);
            }
            const int any_gave_up = __syncthreads_or(gave_up);
            const int all_landed = __syncthreads_and(landed);
            if (threadIdx.x == 0 && any_gave_up) atomicAdd(&g_iir_gave_up, 1u);
            if (!all_landed) tma = false;  // this strip and every later one by plain copies
        }
        if (tma) {
            // the strip is in place
        } else if (vec) {
            for (int i = threadIdx.x; i < n * kQuads; i += blockDim.x) {
                const int r = i / kQuads, qd = i - r * kQuads;
                cp_async16(strip + size_t(r) * kColLines + 4 * qd, src + size_t(r) * pitch + off + 4 * qd);
            }
            cp_async_wait_all();
        } else {
            for (int i = threadIdx.x; i < n * kColLines; i += blockDim.x) {
                const int r = i / kColLines, j = i % kColLines;
                strip[i] = j < nl ? src[size_t(r) * pitch + off + j] : 0.0f;
            }
        }
        __syncthreads();
        if (CTAS == 2) blur_lines(strip, kColLines, kColLines, n, kSegCols, pass, c, carry, false);
        else blur_lines_call(strip, kColLines, kColLines, n, kSegCols, pass, c, carry, false);
        if (MULTI && c + 1 < int(mix.ncomp)) {
            strip_sum<MULTI>(strip, n, mix, c, tmem, false);
        } else if (raw_vec) {
            strip_to_raw<MULTI, CTAS == 2 ? 2 : 1>(strip, raw + off, raw_pitch, n, mix, c, tmem);
        } else {
            if (mix.plain == 0) {
                strip_sum<MULTI>(strip, n, mix, c, tmem, true);
                __syncthreads();
            }
            strip_to_raw_scalar(strip, raw + off, raw_pitch, nl, n, mix);
        }
        __syncthreads();
    }
    if (MULTI) {
        tc_fence_before();
        __syncthreads();
        tc_fence_after();
        if (threadIdx.x < 32) tmem_dealloc(tmem, maps.tmem_cols);
    }
}

}  // namespace

size_t iir_rows_smem(uint32_t pitch) {
    const size_t n3r = (3 * size_t(pitch) + 3) & ~size_t(3);
    return n3r * sizeof(float) + size_t(3) * kSegRows * 3 * sizeof(double);
}

namespace {
// The strip's boxes: ceil(h / 256) of them, each a multiple of 8 rows (at most 256) and together at least h.
struct ColBoxes {
    uint32_t rows, boxes;
};
ColBoxes col_boxes(uint32_t h) {
    const uint32_t boxes = h > 0 ? (h + 255u) / 256u : 1u;
    const uint32_t per = (h + boxes - 1u) / boxes;
    return {(per + 7u) & ~7u, boxes};
}
}  // namespace

size_t iir_cols_smem(uint32_t h) {
    const ColBoxes cb = col_boxes(h);
    return size_t(cb.rows) * cb.boxes * kColLines * sizeof(float) + size_t(kColLines) * kSegCols * 3 * sizeof(double) +
           2 * sizeof(uint64_t);  // the mbarrier, the tensor memory's base
}

// The column segment length: at least n / nseg, and with nlines L = nlines (mod 32), so that a warp's
// lanes (line t % nlines, segment t / nlines, sample i) address floats equal to t + nlines i modulo 32
// and never share a shared-memory bank (L = 1 (mod 8) for twelve lines).
namespace {
int seg_len(uint32_t n, int nseg, int nlines) {
    int g = 32;
    while (nlines % g != 0) g /= 2;  // gcd(nlines, 32)
    const int m = 32 / g;
    const int L0 = int((n + uint32_t(nseg) - 1) / uint32_t(nseg));
    return L0 + ((1 - L0) % m + m) % m;
}
}  // namespace

// rows run segment-major (a warp's lanes: one line, 32 consecutive segments, addresses 3 L t + const):
// any odd L keeps them in distinct banks
int iir_row_seg_len(uint32_t w) {
    const int L0 = int((w + uint32_t(kSegRows) - 1) / uint32_t(kSegRows));
    return L0 | 1;
}
int iir_col_seg_len(uint32_t h) { return seg_len(h, kSegCols, kColLines); }

namespace {
size_t smem_limit() {
    int dev = 0, optin = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
    return size_t(optin);
}
}  // namespace

bool iir_mixture_fits(uint32_t w, uint32_t h) {
    const size_t limit = smem_limit();
    return iir_rows_smem(w) <= limit && iir_cols_smem(h) <= limit;
}

uint32_t iir_pitch(uint32_t w) {
    const uint32_t padded = (w + 3u) & ~3u;
    return padded == w || iir_rows_smem(padded) <= smem_limit() ? padded : w;
}

namespace {
using EncodeTiled = CUresult (*)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                 const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                 CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

// cuTensorMapEncodeTiled from the driver, looked up once (null when the driver cannot give it)
EncodeTiled encode_tiled() {
    static EncodeTiled fn = nullptr;
    static std::once_flag once;
    std::call_once(once, [] {
        void* f = nullptr;
        cudaDriverEntryPointQueryResult q{};
        if (cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &f, 12000, cudaEnableDefault, &q) ==
                cudaSuccess &&
            q == cudaDriverEntryPointSuccess)
            fn = reinterpret_cast<EncodeTiled>(f);
    });
    return fn;
}

std::atomic<long long> g_wait_limit{0};  // set_iir_wait_limit: 0 the full limit

// The tensor maps of the column pass's component planes, `pitch` pixels a row: each a 2-D tensor of 3 pitch
// floats x h rows, read in 12 x box_rows boxes. False (plain copies) for a pitch that is not a multiple of 4
// (the rows and the strips' x coordinates would leave 16-byte alignment), a plane not on a 16-byte
// boundary, or a map the driver refuses.
bool col_maps(IirColMaps& maps, const IirPlanes& planes, uint32_t ncomp, uint32_t pitch, uint32_t h) {
    const ColBoxes cb = col_boxes(h);
    maps.box_rows = cb.rows;
    maps.boxes = cb.boxes;
    const long long lim = g_wait_limit.load();
    maps.wait_limit = lim > 0 ? lim : kWaitCycles;
    maps.use_tma = 0;
    const EncodeTiled enc = encode_tiled();
    if (!kColTma || !enc || (pitch & 3u) != 0u) return false;
    const cuuint64_t dims[2] = {cuuint64_t(3) * pitch, h};
    const cuuint64_t strides[1] = {cuuint64_t(3) * pitch * sizeof(float)};
    const cuuint32_t box[2] = {cuuint32_t(kColLines), cb.rows};
    const cuuint32_t estr[2] = {1, 1};
    for (uint32_t c = 0; c < ncomp; ++c) {
        if ((reinterpret_cast<uintptr_t>(planes.p[c]) & 15u) != 0u) return false;
        if (enc(&maps.map[c], CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 2, planes.p[c], dims, strides, box, estr,
                CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
                CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) != CUDA_SUCCESS)
            return false;
    }
    maps.use_tma = 1;
    return true;
}

// Whether the column pass runs three strips an SM: more strips than two for every SM, in frames short enough.
// Column pass with two and three, 1, 2 and 3 components: 1600 x 200 0.025 / 0.021, 0.040 / 0.031, 0.056 / 0.042 ms;
// 4096 x 64 0.027 / 0.027, 0.048 / 0.044, 0.064 / 0.060; 1600 x 600 0.033 / 0.029, 0.052 / 0.046, 0.072 / 0.058;
// 1600 x 1067 0.044 / 0.044, 0.070 / 0.064, 0.095 / 0.087; 3552 x 900 one component 9 % slower with three, 3552 x 1300
// 19, 9 and 2 % slower. At 1100 rows three strips take 186 KB of shared memory and 384 columns of tensor memory.
bool three_strips(uint32_t w, uint32_t h, uint32_t ncomp) {
    return (w + kColPixels - 1) / kColPixels > 2 * sm_count() && h <= (ncomp > 1 ? 1100u : 500u);
}

template <int N>
void launch_passes(const float* src, float* raw, const IirPlanes& planes, uint32_t w, uint32_t h, const IirMixture& m,
                   const IirColMaps& maps, cudaStream_t s) {
    const size_t sr = iir_rows_smem(m.pitch), sc = iir_cols_smem(h);
    constexpr bool kMulti = N > 1;
    ensure_smem(reinterpret_cast<const void*>(k_iir_rows<N>), int(sr));
    const auto cols = three_strips(w, h, m.ncomp) ? k_iir_cols<kMulti, N, 3> : k_iir_cols<kMulti, N, 2>;
    ensure_smem(reinterpret_cast<const void*>(cols), int(sc));
    {
        Probe p("iir_rows", s);
        k_iir_rows<N><<<h, kRowThreads, sr, s>>>(src, planes, w, h, m, IirPass<N>(m.rows, m.ncomp));
    }
    {
        Probe p("iir_cols", s);
        const uint32_t g = (w + kColPixels - 1) / kColPixels;
        cols<<<g, kColThreads, sc, s>>>(raw, planes, w, h, m, IirPass<N>(m.cols, m.ncomp), maps);
    }
}
}  // namespace

void set_iir_wait_limit(long long cycles) { g_wait_limit.store(cycles); }

uint32_t take_iir_waits_given_up(cudaStream_t s) {
    unsigned int v = 0, zero = 0;
    cudaMemcpyFromSymbolAsync(&v, g_iir_gave_up, sizeof(v), 0, cudaMemcpyDeviceToHost, s);
    cudaMemcpyToSymbolAsync(g_iir_gave_up, &zero, sizeof(zero), 0, cudaMemcpyHostToDevice, s);
    cudaStreamSynchronize(s);
    return v;
}

void iir_mixture(const float* src, float* raw, float* const* tmp, uint32_t w, uint32_t h, const IirMixture& m,
                 cudaStream_t s) {
    IirPlanes planes{};
    for (uint32_t c = 0; c < m.ncomp; ++c) planes.p[c] = tmp[c];
    IirColMaps maps{};
    col_maps(maps, planes, m.ncomp, m.pitch, h);
    if (m.ncomp > 1) {
        // four columns for every 128 quads; allocations are powers of two from 32
        const uint32_t need = 4u * ((3u * h + 127u) / 128u);
        maps.tmem_cols = 32;
        while (maps.tmem_cols < need) maps.tmem_cols *= 2;
    }
    if (m.ncomp == 1) launch_passes<1>(src, raw, planes, w, h, m, maps, s);
    else if (m.ncomp == 2) launch_passes<2>(src, raw, planes, w, h, m, maps, s);
    else launch_passes<SPKB_MAX_COMPONENTS>(src, raw, planes, w, h, m, maps, s);
}

}  // namespace spkb::dev
