// sm_100a kernels of the render path (first generation: one pass per stage, fused where the reference
// stores and reloads an intermediate plane with no change of value).
//
// Numerics follow the reference kernels (kernels/film.metal, print.metal, fx_blur.metal,
// fx_grain.metal): binary32 arithmetic in the same bracketing; recursive-filter state in binary64
// (the reference keeps it in double-float on its GPU and in double on its host copy); the grain
// sampler from grain_sampler.h, which the host checker compiles too.
#include <cuda.h>
#include <cuda_runtime.h>
#include <math.h>
#include <stdint.h>

#include <algorithm>
#include <atomic>
#include <map>
#include <mutex>

#include "../grain_sampler.h"
#include "../kernel_args.h"
#include "encode.cuh"
#include "launch.hpp"
#include "lookup.cuh"

namespace spkb::dev {

namespace {

__host__ __device__ inline uint32_t div_up(uint32_t a, uint32_t b) { return (a + b - 1) / b; }

// ---------------------------------------------------------------------------------------------------
// expose: reference kernels/film.metal:50-99 (Mitchell-Netravali B = C = 1/3) and :189-227.

__device__ __forceinline__ float mitchell(float u) {
    const float a = fabsf(u);
    if (a < 1.0f) return (1.0f / 6.0f) * (7.0f * a * a * a - 12.0f * a * a + 16.0f / 3.0f);
    if (a < 2.0f) return (1.0f / 6.0f) * ((-7.0f / 3.0f) * a * a * a + 12.0f * a * a - 20.0f * a + 32.0f / 3.0f);
    return 0.0f;
}

// The table comes as 4 x 4 patches. Patch (ba, bb) holds the sixteen texels the bicubic reads when the
// pixel's base indices are (ba, bb) -- row reflect(ba - 1 + i), column reflect(bb - 1 + j) -- as RGB triples
// in the loop order (i outer, j inner): 48 floats, 192 bytes, fetched with six 32-byte loads instead of
// sixteen 16-byte gathers, so a warp's random lookups take about a third of the L1 wavefronts. One pixel per
// thread: a thread's lookups wait on its divisions, so pixels in turn in one thread only add up their waits.

__device__ __forceinline__ void mitchell_base(float t, uint32_t L, int& base, float w[4]) {
    const float last = float(L - 1);
    float u = t * last;
    float frac;
    if (u <= 0.0f) u = 0.0f;
    if (u >= last) {
        base = int(L) - 2;
        frac = 1.0f;
    } else {
        base = int(floorf(u));
        frac = u - float(base);
    }
    w[0] = mitchell(frac + 1.0f);
    w[1] = mitchell(frac);
    w[2] = mitchell(frac - 1.0f);
    w[3] = mitchell(frac - 2.0f);
}

__device__ __forceinline__ void ld32(const float* p, float* r) {
    asm volatile("ld.global.nc.v8.f32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
                 : "=f"(r[0]), "=f"(r[1]), "=f"(r[2]), "=f"(r[3]), "=f"(r[4]), "=f"(r[5]), "=f"(r[6]), "=f"(r[7])
                 : "l"(p));
}

__device__ __forceinline__ void expose_pixel(const ExposeArgs& q, const float* __restrict__ patches, float r, float g,
                                             float b, float* h) {
    if (q.apply_ae) {
        r = __fmul_rn(r, q.ae_gain);
        g = __fmul_rn(g, q.ae_gain);
        b = __fmul_rn(b, q.ae_gain);
    }
    const float X = (q.a[0] * r + q.a[1] * g) + q.a[2] * b;
    const float Y = (q.a[3] * r + q.a[4] * g) + q.a[5] * b;
    const float Z = (q.a[6] * r + q.a[7] * g) + q.a[8] * b;
    const float bs = (X + Y) + Z;
    const float d = bs > 1e-10f ? bs : 1e-10f;
    const float x = X / d, y = Y / d, o = 1.0f - x;
    const float t0 = fminf(fmaxf(o * o, 0.0f), 1.0f);
    const float t1 = fminf(fmaxf(y / (o > 1e-10f ? o : 1e-10f), 0.0f), 1.0f);
    const float bp = isnan(bs) ? 0.0f : bs;
    int ba, bb;
    float wa[4], wb[4];
    mitchell_base(t0, q.L, ba, wa);
    mitchell_base(t1, q.L, bb, wb);
    const float* pt = patches + (size_t(ba) * (q.L - 1) + size_t(bb)) * kPatchFloats;
    float t[kPatchFloats];
#pragma unroll
    for (int k = 0; k < 6; ++k) ld32(pt + 8 * k, t + 8 * k);
    float s = 0.0f, a0 = 0.0f, a1 = 0.0f, a2 = 0.0f;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const float w = wa[i] * wb[j];
            const float* tx = t + 3 * (4 * i + j);
            s += w;
            a0 += w * tx[0];
            a1 += w * tx[1];
            a2 += w * tx[2];
        }
    }
    if (s != 0.0f) {
        a0 = a0 / s;
        a1 = a1 / s;
        a2 = a2 / s;
    }
    float h0 = bp * a0, h1 = bp * a1, h2 = bp * a2;
    if (q.apply_gain) {
        h0 = h0 * q.gain;
        h1 = h1 * q.gain;
        h2 = h2 * q.gain;
    }
    h[0] = h0;
    h[1] = h1;
    h[2] = h2;
}

constexpr uint32_t kExposeThreads = 128;

// At most 40 registers a thread (12 CTAs an SM): 131 x 97 14.0 us with a pixel per thread, 23.7 with four in
// turn; 3840 x 2160 0.188 and 0.206 ms (a photograph; uniform noise, whose lookups fill the L1's tag stage,
// 0.225 either way, 0.237 without the bound on registers); 6000 x 4000 0.524 and 0.556.
__global__ void __launch_bounds__(kExposeThreads, 12) k_expose_patch(const float* __restrict__ rgb,
                                                                     float* __restrict__ hout,
                                                                     const float* __restrict__ patches,
                                                                     const __grid_constant__ ExposeArgs q) {
    const uint32_t p = blockIdx.x * blockDim.x + threadIdx.x;
    if (p >= q.n) return;
    const float* in = rgb + 3 * size_t(p);
    expose_pixel(q, patches, in[0], in[1], in[2], hout + 3 * size_t(p));
}

// ---------------------------------------------------------------------------------------------------
// FIR: reference kernels/fx_blur.metal:20-78: taps -r..r ascending, float accumulator from 0,
// half-sample symmetric reflection at the edges.

__device__ __forceinline__ int reflect_index(int i, int n) {
    if (n <= 1) return 0;
    const int period = 2 * n;
    int m = i % period;
    if (m < 0) m += period;
    return m < n ? m : period - 1 - m;
}

__global__ void k_fir_v(const float* __restrict__ in, float* __restrict__ out, uint32_t w, uint32_t h,
                        const __grid_constant__ FirTaps t) {
    const uint32_t x = blockIdx.x * blockDim.x + threadIdx.x;
    const uint32_t y = blockIdx.y * blockDim.y + threadIdx.y;
    if (x >= w || y >= h) return;
    const int r = t.r;
    float a0 = 0.0f, a1 = 0.0f, a2 = 0.0f;
    for (int i = -r; i <= r; ++i) {
        const int yy = reflect_index(int(y) + i, int(h));
        const float* p = in + 3 * (size_t(yy) * w + x);
        const int k = i + r;
        a0 += t.taps[0][k] * p[0];
        a1 += t.taps[1][k] * p[1];
        a2 += t.taps[2][k] * p[2];
    }
    float* o = out + 3 * (size_t(y) * w + x);
    o[0] = a0;
    o[1] = a1;
    o[2] = a2;
}

__global__ void k_fir_h(const float* __restrict__ in, float* out, const float* acc, uint32_t w, uint32_t h,
                        const __grid_constant__ FirTaps t, int mode, float w0, float w1, float w2) {
    const uint32_t x = blockIdx.x * blockDim.x + threadIdx.x;
    const uint32_t y = blockIdx.y * blockDim.y + threadIdx.y;
    if (x >= w || y >= h) return;
    const int r = t.r;
    const float* row = in + 3 * size_t(y) * w;
    float a0 = 0.0f, a1 = 0.0f, a2 = 0.0f;
    for (int i = -r; i <= r; ++i) {
        const int xx = reflect_index(int(x) + i, int(w));
        const float* p = row + 3 * xx;
        const int k = i + r;
        a0 += t.taps[0][k] * p[0];
        a1 += t.taps[1][k] * p[1];
        a2 += t.taps[2][k] * p[2];
    }
    const size_t o = 3 * (size_t(y) * w + x);
    if (mode == ACC_NONE) {
        out[o] = a0;
        out[o + 1] = a1;
        out[o + 2] = a2;
    } else if (mode == ACC_ZERO) {
        out[o] = 0.0f + w0 * a0;
        out[o + 1] = 0.0f + w1 * a1;
        out[o + 2] = 0.0f + w2 * a2;
    } else {
        const float c0 = acc[o], c1 = acc[o + 1], c2 = acc[o + 2];
        out[o] = c0 + w0 * a0;
        out[o + 1] = c1 + w1 * a1;
        out[o + 2] = c2 + w2 * a2;
    }
}

// ---------------------------------------------------------------------------------------------------
// Recursive Gaussian (Young-van Vliet, third order): reference kernels/fx_blur.metal:125-204.
//   forward:  w[-1..-3] = x[0];  w[i] = B x[i] + B1 w[i-1] + B2 w[i-2] + B3 w[i-3];  u[i] = float(w[i])
//   backward: y[n..n+2] = u[n-1]; y[i] = B u[i] + B1 y[i+1] + B2 y[i+2] + B3 y[i+3]
// State in binary64; x, u and y stored as binary32.

// The line kernels below take the frames and channels that the block-parallel kernels do not (a component
// whose channels are not all recursive, lines too long for shared memory, unaligned planes).

struct LineCoefs {
    double B, B1, B2, B3;
};
__device__ __forceinline__ LineCoefs line_coefs(const IirCoefs& q, uint32_t c) {
    return {q.B[c], q.B1[c], q.B2[c], q.B3[c]};
}
__device__ __forceinline__ double iir_step(const LineCoefs& k, double x, double s1, double s2, double s3) {
    return ((k.B * x + k.B1 * s1) + k.B2 * s2) + k.B3 * s3;
}

// The same line with its tangent along sigma (forward mode): the coefficients' derivatives dq (the same
// layout as q) and the input's tangent src_dot (nullptr: zero) give the output's tangent
//   forward:  w'[i] = dB x[i] + B x'[i] + sum_j (dB_j w[i-j] + B_j w'[i-j]), w'[-1..-3] = x'[0]
//   backward: y'[i] = dB u[i] + B u'[i] + sum_j (dB_j y[i+j] + B_j y'[i+j]), y'[n..n+2] = u'[n-1]
// with u = the forward pass rounded to binary32 (its tangent is not rounded). Work planes: the forward
// pass's value and tangent.
__device__ __forceinline__ void iir_line_tangent(const float* __restrict__ src, const float* __restrict__ src_dot,
                                                 float* __restrict__ work, float* __restrict__ work_dot,
                                                 float* __restrict__ dst, float* __restrict__ dst_dot, size_t base,
                                                 size_t stride, uint32_t n, const IirCoefs& q, const IirCoefs& dq,
                                                 int c) {
    // the line's samples go in chunks of kTanChunk: a chunk's loads are issued together, ahead of its
    // recurrence steps, so that a step waits on the previous step and not on memory
    constexpr uint32_t kTanChunk = 8;
    const double B = q.B[c], B1 = q.B1[c], B2 = q.B2[c], B3 = q.B3[c];
    const double dB = dq.B[c], dB1 = dq.B1[c], dB2 = dq.B2[c], dB3 = dq.B3[c];
    double w1 = double(src[base]), w2 = w1, w3 = w1;
    double t1 = src_dot ? double(src_dot[base]) : 0.0, t2 = t1, t3 = t1;
    for (uint32_t i0 = 0; i0 < n; i0 += kTanChunk) {
        float xs[kTanChunk], xds[kTanChunk];
#pragma unroll
        for (uint32_t j = 0; j < kTanChunk; ++j) {
            const size_t o = base + size_t(i0 + j) * stride;
            xs[j] = i0 + j < n ? src[o] : 0.0f;
            xds[j] = i0 + j < n && src_dot ? src_dot[o] : 0.0f;
        }
#pragma unroll
        for (uint32_t j = 0; j < kTanChunk; ++j) {
            if (i0 + j >= n) break;
            const size_t o = base + size_t(i0 + j) * stride;
            const double x = double(xs[j]), xd = double(xds[j]);
            // the newest state enters last: one multiply-add latency per sample on each recurrence
            const double v = fma(B1, w1, fma(B2, w2, fma(B3, w3, B * x)));
            const double vd = fma(B1, t1, fma(dB1, w1, fma(B2, t2, fma(dB2, w2, fma(B3, t3, fma(dB3, w3, fma(B, xd, dB * x)))))));
            w3 = w2;
            w2 = w1;
            w1 = v;
            t3 = t2;
            t2 = t1;
            t1 = vd;
            work[o] = float(v);
            work_dot[o] = float(vd);
        }
    }
    const size_t last = base + size_t(n - 1) * stride;
    double y1 = double(work[last]), y2 = y1, y3 = y1;
    double s1 = double(work_dot[last]), s2 = s1, s3 = s1;
    for (uint32_t k0 = n; k0 > 0;) {
        const uint32_t m = k0 < kTanChunk ? k0 : kTanChunk;  // samples k0 - 1 down to k0 - m
        float us[kTanChunk], uds[kTanChunk];
#pragma unroll
        for (uint32_t j = 0; j < kTanChunk; ++j) {
            const size_t o = base + size_t(k0 - 1 - (j < m ? j : 0)) * stride;
            us[j] = work[o];
            uds[j] = work_dot[o];
        }
#pragma unroll
        for (uint32_t j = 0; j < kTanChunk; ++j) {
            if (j >= m) break;
            const size_t o = base + size_t(k0 - 1 - j) * stride;
            const double u = double(us[j]), ud = double(uds[j]);
            const double v = fma(B1, y1, fma(B2, y2, fma(B3, y3, B * u)));
            const double vd = fma(B1, s1, fma(dB1, y1, fma(B2, s2, fma(dB2, y2, fma(B3, s3, fma(dB3, y3, fma(B, ud, dB * u)))))));
            y3 = y2;
            y2 = y1;
            y1 = v;
            s3 = s2;
            s2 = s1;
            s1 = vd;
            dst[o] = float(v);
            dst_dot[o] = float(vd);
        }
        k0 -= m;
    }
}

// The same tangent with the lines staged in shared memory and each line cut into kTanSegs segments of L
// samples, a thread per (line, segment). A CTA takes `px` rows (3 px lines, vertical = 0) or a strip of
// `px` pixel columns (3 px lines, vertical = 1); the whole CTA loads and stores them in the frame's order.
// Line j, sample i at [i * nl + j]. The value and its tangent form one linear recurrence on the state
// (w1, w2, w3, t1, t2, t3) (the last three values and tangents), so a segment is solved block-parallel as
// the blur itself is: every segment runs from a zero state (the first from the line's edge state) and
// keeps its end state e_s; one thread per line chains the true entry states, S_{s+1} = A^L S_s + e_s, with
// A^L the homogeneous L-step map (TangentMaps, binary64, formed on the host); every segment then reruns
// from its true entry state and stores float(value) and float(tangent) in place. The backward direction
// cuts its segments from the line's end. The state is binary64 throughout.
constexpr uint32_t kTanSegs = 8;
struct TangentMaps {
    double AL[3][36];  // per channel, row-major over (w1, w2, w3, t1, t2, t3)
    uint32_t L;        // segment length
};

struct TanState {
    double w1, w2, w3, t1, t2, t3;
};

// one step of the recurrence on the sample at smem offset o (x and its tangent), the newest state last in
// each multiply-add chain; writes float(value), float(tangent) back when `store`
__device__ __forceinline__ void tan_step(TanState& st, const double* k, float* val, float* dot, size_t o, bool store) {
    const double x = double(val[o]), xd = double(dot[o]);
    const double v = fma(k[1], st.w1, fma(k[2], st.w2, fma(k[3], st.w3, k[0] * x)));
    const double vd = fma(k[1], st.t1, fma(k[5], st.w1, fma(k[2], st.t2, fma(k[6], st.w2,
                      fma(k[3], st.t3, fma(k[7], st.w3, fma(k[0], xd, k[4] * x)))))));
    st.w3 = st.w2;
    st.w2 = st.w1;
    st.w1 = v;
    st.t3 = st.t2;
    st.t2 = st.t1;
    st.t1 = vd;
    if (store) {
        val[o] = float(v);
        dot[o] = float(vd);
    }
}

__global__ void k_iir_tangent_seg(const float* __restrict__ in, const float* __restrict__ in_dot,
                                  float* __restrict__ out, float* __restrict__ out_dot, uint32_t w, uint32_t h,
                                  int vertical, uint32_t px, const __grid_constant__ IirCoefs q,
                                  const __grid_constant__ IirCoefs dq, const __grid_constant__ TangentMaps maps) {
    extern __shared__ __align__(16) unsigned char tsm_raw[];
    const uint32_t n = vertical ? h : w;
    const uint32_t z0 = blockIdx.x * px;                    // the first pixel column, or row
    const uint32_t npx = min(px, (vertical ? w : h) - z0);  // columns (rows) in this strip
    const uint32_t nl = 3 * px;                              // the strip's line pitch
    const uint32_t nv = 3 * npx;                             // valid lines
    double* carry = reinterpret_cast<double*>(tsm_raw);      // [line][segment][6]
    float* val = reinterpret_cast<float*>(carry + size_t(nl) * kTanSegs * 6);
    float* dot = val + size_t(n) * nl;
    const uint32_t span = vertical ? nv : 3 * n;  // contiguous floats per strip row
    const uint32_t total = vertical ? n * nv : npx * 3 * n;
#pragma unroll 4
    for (uint32_t e = threadIdx.x; e < total; e += blockDim.x) {
        const uint32_t r = e / span, f = e - r * span;
        const size_t g = vertical ? (size_t(r) * w + z0) * 3 + f : (size_t(z0 + r) * w) * 3 + f;
        const uint32_t i = vertical ? r : f / 3, j = vertical ? f : 3 * r + f % 3;
        val[size_t(i) * nl + j] = in[g];
        dot[size_t(i) * nl + j] = in_dot ? in_dot[g] : 0.0f;
    }
    __syncthreads();

    const uint32_t line = threadIdx.x / kTanSegs, seg = threadIdx.x % kTanSegs;
    const int c = int(line % 3u);
    const bool active = line < nv && ((q.mask >> c) & 1u) != 0u;
    const double k[8] = {q.B[c], q.B1[c], q.B2[c], q.B3[c], dq.B[c], dq.B1[c], dq.B2[c], dq.B3[c]};
    const uint32_t L = maps.L;
    double* cs = carry + (size_t(line) * kTanSegs + seg) * 6;
    for (int dir = 0; dir < 2; ++dir) {
        // this segment's samples: forward [a, b) ascending; backward [a, b) descending, cut from the end
        uint32_t a, b;
        if (dir == 0) {
            a = min(n, seg * L);
            b = min(n, a + L);
        } else {
            b = n > seg * L ? n - seg * L : 0u;
            a = b > L ? b - L : 0u;
        }
        // the line's edge state: x[0] (forward) or the forward result u[n-1] (backward)
        TanState edge{};
        if (active) {
            const size_t o0 = size_t(dir == 0 ? 0u : n - 1u) * nl + line;
            const double e0 = double(val[o0]), d0 = double(dot[o0]);
            edge = TanState{e0, e0, e0, d0, d0, d0};
        }
        // pass 1: zero-state run (the first segment from the edge state), its end state kept
        if (active && a < b) {
            TanState st = seg == 0 ? edge : TanState{};
            if (dir == 0) {
                for (uint32_t i = a; i < b; ++i) tan_step(st, k, val, dot, size_t(i) * nl + line, false);
            } else {
                for (uint32_t i = b; i-- > a;) tan_step(st, k, val, dot, size_t(i) * nl + line, false);
            }
            cs[0] = st.w1;
            cs[1] = st.w2;
            cs[2] = st.w3;
            cs[3] = st.t1;
            cs[4] = st.t2;
            cs[5] = st.t3;
        }
        __syncthreads();
        // the true entry states, one thread per line: segment s + 1 enters with A^L S_s + e_s (segment 0's
        // end state is already true); a segment's slot takes its entry state
        if (active && seg == 0) {
            double S[6];
            double* c0 = carry + size_t(line) * kTanSegs * 6;
            for (int m = 0; m < 6; ++m) S[m] = c0[m];
            for (uint32_t sg = 1; sg < kTanSegs && sg * L < n; ++sg) {
                double* cg = c0 + sg * 6;
                double e[6];
                for (int m = 0; m < 6; ++m) {
                    e[m] = cg[m];
                    cg[m] = S[m];
                }
                const double* A = maps.AL[c];
                double T[6];
                for (int r = 0; r < 6; ++r) {
                    double acc = e[r];
                    for (int m = 0; m < 6; ++m) acc = fma(A[r * 6 + m], S[m], acc);
                    T[r] = acc;
                }
                for (int m = 0; m < 6; ++m) S[m] = T[m];
            }
        }
        __syncthreads();
        // pass 2: every segment from its true entry state, storing
        if (active && a < b) {
            TanState st = seg == 0 ? edge : TanState{cs[0], cs[1], cs[2], cs[3], cs[4], cs[5]};
            if (dir == 0) {
                for (uint32_t i = a; i < b; ++i) tan_step(st, k, val, dot, size_t(i) * nl + line, true);
            } else {
                for (uint32_t i = b; i-- > a;) tan_step(st, k, val, dot, size_t(i) * nl + line, true);
            }
        }
        __syncthreads();
    }
#pragma unroll 4
    for (uint32_t e = threadIdx.x; e < total; e += blockDim.x) {
        const uint32_t r = e / span, f = e - r * span;
        const size_t g = vertical ? (size_t(r) * w + z0) * 3 + f : (size_t(z0 + r) * w) * 3 + f;
        const uint32_t i = vertical ? r : f / 3, j = vertical ? f : 3 * r + f % 3;
        out[g] = val[size_t(i) * nl + j];
        out_dot[g] = dot[size_t(i) * nl + j];
    }
}

// the blur's tangent along sigma, one thread per line: rows (vertical = 0) or columns (vertical = 1); a
// channel outside q.mask passes its value and tangent through
__global__ void k_iir_tangent(const float* __restrict__ in, const float* in_dot, float* work, float* work_dot,
                              float* out, float* out_dot, uint32_t w, uint32_t h, int vertical,
                              const __grid_constant__ IirCoefs q, const __grid_constant__ IirCoefs dq) {
    const uint32_t t = blockIdx.x * blockDim.x + threadIdx.x;
    const uint32_t lines = vertical ? 3u * w : 3u * h;
    if (t >= lines) return;
    const uint32_t c = t % 3u;
    const size_t base = vertical ? size_t(t) : 3 * size_t(t / 3u) * w + c;
    const size_t stride = vertical ? 3 * size_t(w) : 3;
    const uint32_t n = vertical ? h : w;
    if (((q.mask >> c) & 1u) == 0u) {
        for (uint32_t i = 0; i < n; ++i) {
            const size_t o = base + i * stride;
            out[o] = in[o];
            out_dot[o] = in_dot ? in_dot[o] : 0.0f;
        }
        return;
    }
    iir_line_tangent(in, in_dot, work, work_dot, out, out_dot, base, stride, n, q, dq, int(c));
}

// Row pass of the line recurrence, one lane per line: a one-warp CTA takes kLineRows rows (30 lines) and
// walks them in chunks of kLinePix pixels that cp.async brings into shared memory kLineStages - 1 chunks
// ahead; a chunk's results replace its samples there and leave in coalesced stores. The bound is the
// recurrence itself (three dependent binary64 multiply-adds a sample, twice a line): a lane per line that
// reads global memory sample by sample waited for a load at each (6000 x 4000: 3.03 ms, 0.62 this way). Pitch 3 kLinePix + 3 keeps the 30 lanes
// (row r, channel c: word r pitch + 3 i + c) in distinct banks.
constexpr uint32_t kLineRows = 10, kLinePix = 32, kLinePitch = 3 * kLinePix + 3, kLineStages = 4;

__device__ __forceinline__ void cp_async4(float* dst, const float* src) {
    const unsigned d = static_cast<unsigned>(__cvta_generic_to_shared(dst));
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(d), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_async_wait() {
    asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}

// chunk q's floats of the CTA's rows, plane -> buf or buf -> plane; rows past nrows and floats past the row
// are left alone
template <bool LOAD>
__device__ __forceinline__ void line_chunk(const float* src, float* dst, float* buf, uint32_t n3, uint32_t nrows,
                                           uint32_t q) {
    const uint32_t lane = threadIdx.x;
#pragma unroll
    for (uint32_t r = 0; r < kLineRows; ++r) {
        if (r >= nrows) break;
#pragma unroll
        for (uint32_t k = 0; k < 3; ++k) {
            const uint32_t f = k * 32u + lane, g = q * 3u * kLinePix + f;
            if (g >= n3) continue;
            if (LOAD) cp_async4(buf + r * kLinePitch + f, src + size_t(r) * n3 + g);
            else dst[size_t(r) * n3 + g] = buf[r * kLinePitch + f];
        }
    }
}

__global__ void __launch_bounds__(32) k_iir_h(uint32_t w, uint32_t h, const __grid_constant__ IirLineJobs jobs) {
    const float* in = jobs.in[blockIdx.y];
    float* out = jobs.work[blockIdx.y];
    const IirCoefs& q = jobs.q[blockIdx.y];
    __shared__ float ring[kLineStages][kLineRows * kLinePitch];
    static_assert(3 * kLinePix == 96, "a row's chunk is three floats a lane");
    const uint32_t lane = threadIdx.x, r0 = blockIdx.x * kLineRows;
    const uint32_t nrows = min(kLineRows, h - r0), n3 = 3 * w, nq = div_up(w, kLinePix);
    const uint32_t row = min(lane / 3u, nrows - 1), c = lane % 3u;
    const bool live = lane < 3u * nrows, active = live && ((q.mask >> c) & 1u) != 0u;
    const float* src = in + size_t(r0) * n3;
    float* dst = out + size_t(r0) * n3;
    const uint32_t o = row * kLinePitch + c;
    const LineCoefs kc = line_coefs(q, c);
    // forward over the chunks 0 .. nq - 1 of the input, then backward over nq - 1 .. 0 of the result
#pragma unroll 1
    for (int dir = 0; dir < 2; ++dir) {
        const float* from = dir == 0 ? src : dst;
        auto chunk = [&](uint32_t k) { return dir == 0 ? k : nq - 1u - k; };
#pragma unroll 1
        for (uint32_t k = 0; k + 1 < kLineStages; ++k) {
            if (k < nq) line_chunk<true>(from, dst, ring[k], n3, nrows, chunk(k));
            cp_async_commit();
        }
        double s1 = 0.0, s2 = 0.0, s3 = 0.0;
#pragma unroll 1
        for (uint32_t k = 0; k < nq; ++k) {
            const uint32_t ahead = k + kLineStages - 1;
            if (ahead < nq) line_chunk<true>(from, dst, ring[ahead % kLineStages], n3, nrows, chunk(ahead));
            cp_async_commit();
            cp_async_wait<kLineStages - 1>();
            __syncwarp();
            float* buf = ring[k % kLineStages];
            const uint32_t np = min(kLinePix, w - chunk(k) * kLinePix);
            if (active) {
                if (k == 0) s1 = s2 = s3 = double(buf[o + (dir == 0 ? 0u : 3u * (np - 1u))]);
                if (dir == 0) {
#pragma unroll 8
                    for (uint32_t i = 0; i < np; ++i) {
                        const double t = iir_step(kc, double(buf[o + 3 * i]), s1, s2, s3);
                        s3 = s2;
                        s2 = s1;
                        s1 = t;
                        buf[o + 3 * i] = float(t);
                    }
                } else {
#pragma unroll 8
                    for (uint32_t i = np; i-- > 0;) {
                        const double t = iir_step(kc, double(buf[o + 3 * i]), s1, s2, s3);
                        s3 = s2;
                        s2 = s1;
                        s1 = t;
                        buf[o + 3 * i] = float(t);
                    }
                }
            }
            __syncwarp();
            line_chunk<false>(src, dst, buf, n3, nrows, chunk(k));
            __syncwarp();  // the chunk's stores are done: its buffer may be filled again, its rows read back
        }
        cp_async_wait<0>();
        __syncwarp();
    }
}

// Column pass of the line recurrence, a thread per line (neighbouring threads on neighbouring floats). Each
// thread holds the next kColChunk samples in registers while it runs the current ones, so that a sample
// costs its three dependent multiply-adds and no memory latency (6000 x 4000: 5.49 ms with a load per
// sample, 0.65 this way). One-warp CTAs spread the lines over the SMs. A channel that is not filtered passes through.
constexpr uint32_t kColChunk = 16;

template <int MODE>
__global__ void __launch_bounds__(32) k_iir_v(const float* acc, uint32_t w, uint32_t h,
                                              const __grid_constant__ IirLineJobs jobs, float w0, float w1, float w2) {
    float* work = jobs.work[blockIdx.y];
    float* out = jobs.out[blockIdx.y];
    const IirCoefs& q = jobs.q[blockIdx.y];
    const uint32_t t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= 3u * w) return;
    const uint32_t c = t % 3u;
    const size_t stride = 3 * size_t(w);
    const bool active = ((q.mask >> c) & 1u) != 0u;
    const float wgt = c == 0 ? w0 : (c == 1 ? w1 : w2);
    const LineCoefs kc = line_coefs(q, c);
    const uint32_t nq = div_up(h, kColChunk);
    float cur[kColChunk], nxt[kColChunk], ca[kColChunk], na[kColChunk];
    // the samples of chunk k: rows k kColChunk + j downwards, or from the bottom row upwards; past the line
    // the last one again
    auto load = [&](const float* p, float* v, uint32_t k, bool up) {
#pragma unroll
        for (uint32_t j = 0; j < kColChunk; ++j) {
            const uint32_t i = min(k * kColChunk + j, h - 1u);
            v[j] = p[t + size_t(up ? h - 1u - i : i) * stride];
        }
    };
    load(work, cur, 0, false);
    double s1 = double(cur[0]), s2 = s1, s3 = s1;
#pragma unroll 1
    for (uint32_t k = 0; k < nq; ++k) {
        if (k + 1 < nq) load(work, nxt, k + 1, false);
        // the chain first, its results stored after it: a store would hold the next step back until the
        // result's conversion is through
#pragma unroll
        for (uint32_t j = 0; j < kColChunk; ++j) {
            const double v = iir_step(kc, double(cur[j]), s1, s2, s3);
            s3 = s2;
            s2 = s1;
            s1 = v;
            cur[j] = float(v);
        }
        float* o = work + t + size_t(k * kColChunk) * stride;
#pragma unroll
        for (uint32_t j = 0; j < kColChunk; ++j, o += stride) {
            if (active && k * kColChunk + j < h) *o = cur[j];
            cur[j] = nxt[j];
        }
    }
    load(work, cur, 0, true);
    if (MODE == ACC_PLANE) load(acc, ca, 0, true);
    s1 = double(cur[0]);
    s2 = s1;
    s3 = s1;
#pragma unroll 1
    for (uint32_t k = 0; k < nq; ++k) {
        if (k + 1 < nq) {
            load(work, nxt, k + 1, true);
            if (MODE == ACC_PLANE) load(acc, na, k + 1, true);
        }
#pragma unroll
        for (uint32_t j = 0; j < kColChunk; ++j) {
            const double v = iir_step(kc, double(cur[j]), s1, s2, s3);
            s3 = s2;
            s2 = s1;
            s1 = v;
            cur[j] = active ? float(v) : cur[j];
        }
#pragma unroll
        for (uint32_t j = 0; j < kColChunk; ++j) {
            const uint32_t i = k * kColChunk + j;
            float r = cur[j];
            if (MODE == ACC_ZERO && active) r = 0.0f + wgt * r;
            if (MODE == ACC_PLANE && active) r = ca[j] + wgt * r;
            if (i < h) out[t + size_t(h - 1u - i) * stride] = r;
            cur[j] = nxt[j];
            if (MODE == ACC_PLANE) ca[j] = na[j];
        }
    }
}

__global__ void k_lincomb(const float* x, const float* y, float* out, size_t n, float a0, float a1, float a2,
                          float b0, float b1, float b2) {
    const size_t i = size_t(blockIdx.x) * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const float a[3] = {a0, a1, a2}, b[3] = {b0, b1, b2};
#pragma unroll
    for (int c = 0; c < 3; ++c) {
        const size_t o = 3 * i + c;
        const float yv = y ? y[o] : 0.0f;
        out[o] = a[c] * x[o] + b[c] * yv;
    }
}

__global__ void k_copy(const float* __restrict__ x, float* __restrict__ out, size_t n) {
    const size_t i = size_t(blockIdx.x) * blockDim.x + threadIdx.x;
    if (i >= n) return;
    out[i] = x[i];
}

// ---------------------------------------------------------------------------------------------------
// develop: log10 exposure (film.metal:242-246), density curves (:84-101, :249-261), grain draw
// (fx_grain.metal:39-97, SUM and SIMPLE modes).

__device__ __forceinline__ float curve_lookup(const float* __restrict__ x, const float* __restrict__ inv,
                                              const float* __restrict__ y, uint32_t K, const AxisGrid& g, float v) {
    if (v <= __ldg(x)) return __ldg(y);
    if (v >= __ldg(x + K - 1)) return __ldg(y + K - 1);
    const uint32_t l = axis_index(x, 1, K, g, v);
    const float t = (v - __ldg(x + l)) * __ldg(inv + l);
    const float y0 = __ldg(y + l);
    return y0 + t * (__ldg(y + l + 1) - y0);
}

// the three sub-layer densities of channel c at density v (reference fx_grain.metal:60-75)
__device__ __forceinline__ void layer_densities(const DevelopArgs& q, uint32_t c, float v, float dl[3]) {
    const uint32_t K = q.gK;
    if (v <= __ldg(q.axis + c)) {
        for (uint32_t l = 0; l < 3u; ++l) dl[l] = __ldg(q.layers + l * 3u + c);
    } else if (v >= __ldg(q.axis + 3u * (K - 1u) + c)) {
        for (uint32_t l = 0; l < 3u; ++l) dl[l] = __ldg(q.layers + ((K - 1u) * 3u + l) * 3u + c);
    } else {
        // a NaN v gives j = 0, in bounds, and NaN densities
        const uint32_t j = axis_index(q.axis + c, 3u, K, q.ggrid[c], v);
        const float t = (v - __ldg(q.axis + 3u * j + c)) * __ldg(q.ginv + 3u * j + c);
        for (uint32_t l = 0; l < 3u; ++l) {
            const float y0 = __ldg(q.layers + (j * 3u + l) * 3u + c);
            const float y1 = __ldg(q.layers + ((j + 1u) * 3u + l) * 3u + c);
            dl[l] = y0 + t * (y1 - y0);
        }
    }
}

// spk_sublayer_draw (grain_sampler.h) with the count kept for the test hook: the same operations.
__device__ __forceinline__ float grain_draw(float d, float D, float n, float u, uint32_t pixel, uint32_t stream,
                                            uint32_t seed, float* count_slot) {
    float sat;
    const float lam = spk_sublayer_lambda(d, D, n, u, &sat);
    const float k = spk_poisson(lam, pixel, stream, seed);
    if (count_slot) *count_slot = k;
    return SPK_MUL(k, SPK_MUL(SPK_DIV(D, n), sat));
}

// DIR couplers' source (reference kernels/film.metal:242-276): L = log10(max(H, 0) + 1e-10), D = the curve at
// L, s_c = positive ? dmax_c - D_c : D_c, chi_m = (s_0 M[0][m] + s_1 M[1][m]) + s_2 M[2][m], each operation
// rounded as written
__global__ void k_coupler_source(const float* __restrict__ exposure, float* __restrict__ chi,
                                 const __grid_constant__ CouplerArgs q) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= q.n) return;
    float sv[3];
#pragma unroll
    for (uint32_t c = 0; c < 3; ++c) {
        const float L = log10f(fmaxf(exposure[3 * size_t(i) + c], 0.0f) + 1e-10f);
        const float D = curve_lookup(q.cx, q.cinv, q.cy + size_t(c) * q.K, q.K, q.cgrid, L);
        sv[c] = q.positive ? __fsub_rn(q.dmax[c], D) : D;
    }
#pragma unroll
    for (uint32_t m = 0; m < 3; ++m)
        chi[3 * size_t(i) + m] = __fadd_rn(__fadd_rn(__fmul_rn(sv[0], q.m[m]), __fmul_rn(sv[1], q.m[3 + m])),
                                           __fmul_rn(sv[2], q.m[6 + m]));
}

__global__ void k_develop(const float* __restrict__ exposure, float* __restrict__ out, uint32_t w, uint32_t h,
                          const __grid_constant__ DevelopArgs q) {
    const uint32_t x = blockIdx.x * blockDim.x + threadIdx.x;
    const uint32_t y = blockIdx.y * blockDim.y + threadIdx.y;
    if (x >= w || y >= h) return;
    const uint32_t pixel = y * q.width + x;
    const size_t o = 3 * (size_t(y) * w + x);
    for (uint32_t c = 0; c < 3; ++c) {
        float L = log10f(fmaxf(exposure[o + c], 0.0f) + 1e-10f);
        if (q.chi) L = __fsub_rn(L, q.chi[o + c]);  // DIR couplers: the corrected log exposure, the y0 curve
        const float D = curve_lookup(q.cx, q.cinv, q.cy + size_t(c) * q.K, q.K, q.cgrid, L);
        if (!q.grain) {
            out[o + c] = D;
            continue;
        }
        if (q.mode == 2) {  // SIMPLE
            const float d = D + q.dmin_c[c];
            float G = 0.0f;
            for (uint32_t l = 0; l < q.n_sub; ++l)
                G = G + grain_draw(d, q.sat_d[c], q.count[c], q.uniformity[c], pixel, SPK_STREAM_GRAIN(c, l), q.seed,
                                   q.counts_out && l < 3 ? q.counts_out + size_t(pixel) * 9 + c * 3 + l : nullptr);
            out[o + c] = G * q.inv_n_sub + (-q.dmin_c[c]);
            continue;
        }
        const float v = q.positive ? -D : D;
        float dl[3];
        layer_densities(q, c, v, dl);
        float val[3];
        for (uint32_t l = 0; l < 3u; ++l) {
            const uint32_t lc = l * 3u + c;
            val[l] = grain_draw(dl[l] + q.dmin_l[lc], q.sat_d[lc], q.count[lc], q.uniformity[c], pixel,
                                SPK_STREAM_GRAIN(c, l), q.seed,
                                q.counts_out ? q.counts_out + size_t(pixel) * 9 + c * 3 + l : nullptr);
        }
        float G = ((0.0f + val[0]) + val[1]) + val[2];
        if (q.shift) G = G * 1.0f + (-q.dmin_c[c]);
        out[o + c] = G;
    }
}

// ---------------------------------------------------------------------------------------------------
// develop with sub-layer grain (SUM mode), the draws compacted per warp.
//
// A pixel's nine Poisson draws take data-dependent paths: most PTRS draws end at the first attempt's
// squeeze, the rest need the logarithm test, further attempts or (lam < 10) the product method. Run
// per lane, a warp would wait on its slowest lane at every draw. Here each lane makes every draw's
// first attempt in lockstep, by approximations that settle it only where their error cannot matter
// (squeeze_certain); every other draw goes to a ring in the warp's shared memory, from which the whole
// warp takes 32 at a time, one attempt per lane, by the sampler's own operations (draw_attempt). Every
// draw consumes the same uniforms in the same order as spk_poisson, so the counts are those of the
// per-lane sampler.

#ifndef SPKB_DEVELOP_WARPS
#define SPKB_DEVELOP_WARPS 4
#endif
constexpr uint32_t kDrawWarps = SPKB_DEVELOP_WARPS;  // warps per block
// resident blocks per SM the register allocation is held to (1: no cap)
#ifndef SPKB_DEVELOP_MIN_BLOCKS
#define SPKB_DEVELOP_MIN_BLOCKS 10
#endif

// log(k!) for k = 0 .. kLgammaTable - 1, each the sampler's own spk_lgamma_k(k + 1) computed by this
// device once per process (k_lgamma_table): the full test's largest single cost, a table read instead.
constexpr uint32_t kLgammaTable = 65536;
__device__ float g_lgamma[kLgammaTable];

__global__ void k_lgamma_table() {
    const uint32_t k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k < kLgammaTable) g_lgamma[k] = spk_lgamma_k(SPK_ADD(float(k), 1.0f));
}

// spk_ptrs_test with log(k!) from the table while k is in it (k >= 0 and integral here)
__device__ __forceinline__ int ptrs_test_table(const spk_ptrs* p, float V, float k, float us) {
    const float L = SPK_SUB(SPK_ADD(spk_logf(V), p->loginvalpha),
                            spk_logf(SPK_ADD(SPK_DIV(p->a, SPK_MUL(us, us)), p->b)));
    const float lg = k < float(kLgammaTable) ? g_lgamma[int(k)] : spk_lgamma_k(SPK_ADD(k, 1.0f));
    const float Rt = SPK_SUB(SPK_ADD(-p->lam, SPK_MUL(k, p->loglam)), lg);
    return L <= Rt;
}

// PTX approximations: sqrt and reciprocal within 2^-23 relative; log2 within 2^-22, relative outside [1/2, 2]
__device__ __forceinline__ float sqrt_approx(float x) {
    float y;
    asm("sqrt.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}
__device__ __forceinline__ float rcp_approx(float x) {
    float y;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}
__device__ __forceinline__ float log2_approx(float x) {
    float y;
    asm("lg2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}

// The sampler's full test (ptrs_test_table) with its left side, log V + log(1 / alpha) - log(a / us^2 + b),
// taken as one approximate logarithm. The right side's rounding reaches far above that, so it is formed by
// the sampler's own operations. The approximate left side lies within 4e-5 of the sampler's (its binary32
// logarithms up to 37 in magnitude: at most 2e-5; lg2.approx: at most 1.4e-5; the argument's rounding
// 1e-6): a test decided by more than 1e-4 stands, any other (about 2 in 10,000) runs the sampler's.
__device__ __forceinline__ bool ptrs_accepts(spk_ptrs* p, float V, float k, float us) {
    const float lg = k < float(kLgammaTable) ? g_lgamma[int(k)] : spk_lgamma_k(SPK_ADD(k, 1.0f));
    p->loglam = spk_logf_normal(p->lam, 0);
    const float Rt = SPK_SUB(SPK_ADD(-p->lam, SPK_MUL(k, p->loglam)), lg);
    const float us2 = us * us, b34 = p->b - 3.4f;
    const float num = (V * us2) * fmaf(1.1239f, b34, 1.1328f), den = b34 * fmaf(p->b, us2, p->a);
    const float L = 0.693147181f * log2_approx(num * rcp_approx(den));
    if (fabsf(L - Rt) > 1e-4f) return L <= Rt;
    spk_ptrs_init_test(p);
    return ptrs_test_table(p, V, k, us);
}

// Draws whose first attempt the lockstep below does not settle are queued as one word each: slot (draw *
// 32 + lane) | attempt << 9.
constexpr uint32_t kDrawRing = 512;  // at most the warp's 288 draws are queued at a time

// Attempt `it` of a queued draw of lambda lm >= 10, exactly as spk_ptrs_from runs it (the squeeze, then the
// full test). The count replaces the lambda in *res; false when the attempt was rejected.
__device__ __forceinline__ bool draw_attempt(float* res, float lm, uint32_t pixel, uint32_t stream, uint32_t seed,
                                             uint32_t it) {
    if (it == 64u) {
        *res = SPK_FLOOR(lm);
        return true;
    }
    spk_ptrs p;
    spk_ptrs_init(&p, lm);
    // uniforms 2 it and 2 it + 1: words x, y (it even) or z, w (it odd) of Philox block it / 2
    spk_u4 c4;
    c4.x = pixel;
    c4.y = stream;
    c4.z = it >> 1;
    c4.w = 0u;
    const spk_u4 b = spk_philox(c4, seed, 0u);
    const bool odd = (it & 1u) != 0u;
    const float V = spk_uniform(odd ? b.w : b.y);
    float k, us;
    const int r = spk_ptrs_squeeze(&p, spk_uniform(odd ? b.z : b.x), V, &k, &us);
    if (r == SPK_PTRS_REJECT || (r == SPK_PTRS_TEST && !ptrs_accepts(&p, V, k, us))) return false;
    *res = k;
    return true;
}

// The rounds of a pixel's first Philox block (counter (pixel, stream, 0, 0), key (seed, 0)) that do not
// depend on the stream, shared by its nine draws: the second round's (x, y) and the third round's first
// product, with the round keys and the words they meet folded in.
struct PhiloxHead {
    uint32_t y3k;       // y of round 2 ^ k0 of round 3
    uint32_t z2;        // lo(M0 pixel) ^ k1 of round 2: z of round 2 is this ^ hi(M0 (stream ^ seed))
    uint32_t z3k, w3;   // hi(M0 x2) ^ k1 of round 3, lo(M0 x2)
};
__device__ __forceinline__ PhiloxHead philox_head(uint32_t pixel, uint32_t seed) {
    const uint64_t p0 = uint64_t(SPK_PHILOX_M0) * pixel;
    const uint64_t p1 = uint64_t(SPK_PHILOX_M1) * uint32_t(p0 >> 32);
    const uint64_t p3 = uint64_t(SPK_PHILOX_M0) * (uint32_t(p1 >> 32) ^ (seed + SPK_PHILOX_W0));
    PhiloxHead h;
    h.y3k = uint32_t(p1) ^ (seed + 2u * SPK_PHILOX_W0);
    h.z2 = uint32_t(p0) ^ SPK_PHILOX_W1;
    h.z3k = uint32_t(p3 >> 32) ^ (2u * SPK_PHILOX_W1);
    h.w3 = uint32_t(p3);
    return h;
}
// the block's words; sh, sl: the halves of M0 (stream ^ seed)
__device__ __forceinline__ spk_u4 philox_first(const PhiloxHead& h, uint32_t sh, uint32_t sl, uint32_t seed) {
    const uint64_t p1 = uint64_t(SPK_PHILOX_M1) * (sh ^ h.z2);
    spk_u4 c;
    c.x = uint32_t(p1 >> 32) ^ h.y3k;
    c.y = uint32_t(p1);
    c.z = h.z3k ^ sl;
    c.w = h.w3;
#pragma unroll
    for (uint32_t r = 3; r < 10; ++r) {
        const uint64_t a = uint64_t(SPK_PHILOX_M0) * c.x, b = uint64_t(SPK_PHILOX_M1) * c.z;
        c.x = uint32_t(b >> 32) ^ c.y ^ (seed + r * SPK_PHILOX_W0);
        c.y = uint32_t(b);
        c.z = uint32_t(a >> 32) ^ c.w ^ (r * SPK_PHILOX_W1);
        c.w = uint32_t(a);
    }
    return c;
}

// Four more uniforms of the product method: prod times each in turn, and how many products stayed above
// E = exp(-lambda) (they never rise, so these come first); the draw is done once one has not
__device__ __forceinline__ uint32_t product_block(const spk_u4& words, float E, float& prod) {
    const uint32_t wd[4] = {words.x, words.y, words.z, words.w};
    uint32_t above = 0;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        prod = SPK_MUL(prod, spk_uniform(wd[i]));
        above += prod > E ? 1u : 0u;
    }
    return above;
}

// spk_poisson_product, a Philox block (four uniforms) per turn
__device__ __forceinline__ float poisson_product(float lam, uint32_t pixel, uint32_t stream, uint32_t seed) {
    const float E = spk_expf(-lam);
    float prod = 1.0f;
    uint32_t n = 0;
#pragma unroll 1
    for (uint32_t j = 0; j < 128u; ++j) {
        spk_u4 c4;
        c4.x = pixel;
        c4.y = stream;
        c4.z = j;
        c4.w = 0u;
        const uint32_t above = product_block(spk_philox(c4, seed, 0u), E, prod);
        n += above;
        if (above < 4u) break;
    }
    return float(n);
}

// A first attempt (uniform words wu, wv) that the sampler's squeeze accepts beyond doubt: true, and k the
// sampler's count. The squeeze is evaluated with approximate square root and reciprocals; it stands when
// V lies more than 1e-6 below v_r and the count's argument lies further from an integer than both
// evaluations' errors: 2 ulp of the argument (below lam + 0.74 b) for the last sums, and 8e-7 relative of
// (2 a / us + b) |U| < 0.74 b before them. U, us and V are the sampler's own values.
__device__ __forceinline__ bool squeeze_certain(float lam, uint32_t wu, uint32_t wv, float& k) {
    const float U = __fmaf_rn(__fadd_rn(float(wu >> 8), 0.5f), 5.9604644775390625e-08f, -0.5f);
    const float us = __fsub_rn(0.5f, fabsf(U));
    const float V = spk_uniform(wv);
    const float b = fmaf(2.53f, sqrt_approx(lam), 0.931f);
    const float vr = fmaf(-3.6224f, rcp_approx(b - 2.0f), 0.9277f - 1e-6f);
    const float g = fmaf(fmaf(fmaf(0.04966f, b, -0.118f), rcp_approx(us), b), U, lam + 0.43f);
    k = floorf(g);
    const float frac = g - k, tol = fmaf(lam, 4e-7f, 1.5e-6f * b);
    return lam >= 10.0f && us >= 0.07f && V <= vr && frac >= tol && frac <= 1.0f - tol;
}

// curve_lookup and layer_densities on the packed tables (DevelopArgs::packed): the same interval and the
// same operations, the interval's values read with one vector load, the ends by clamping onto the first or
// last entry. A NaN stays one. The densities' axis is the film's own curve, far from evenly spaced: its
// bisection took ten dependent loads, the guide's bucket leaves none to four.
__device__ __forceinline__ float curve_packed(const DevelopArgs& q, uint32_t c, float v) {
    const float4* e = reinterpret_cast<const float4*>(q.curve4) + size_t(c) * q.K;
    v = v < q.cgrid.x0 ? q.cgrid.x0 : v;
    v = v > q.curve_last ? q.curve_last : v;
    const int j = min(max(int((v - q.cgrid.x0) * q.cgrid.s), 0), int(q.K) - 2);
    float4 t = __ldg(e + j);
    const float next = __ldg(&e[j + 1].x);
    if (t.x > v) t = __ldg(e + j - 1);
    else if (next <= v) t = __ldg(e + j + 1);
    return t.z + ((v - t.x) * t.y) * t.w;
}
__device__ __forceinline__ void layers_packed(const DevelopArgs& q, uint32_t c, float v, float dl[3]) {
    const float* e = q.layer8 + size_t(c) * q.gK * 8;
    v = v < q.guide_x0[c] ? q.guide_x0[c] : v;
    v = v > q.axis_last[c] ? q.axis_last[c] : v;
    const uint32_t g = __ldg(q.guide + c * kGuide + min(uint32_t(max(int((v - q.guide_x0[c]) * q.guide_s[c]), 0)), kGuide - 1u));
    uint32_t j = g & 0xFFFFu, hi = g >> 16;
    while (j < hi) {
        const uint32_t mid = (j + hi + 1u) / 2u;
        if (__ldg(e + 8 * mid) <= v) j = mid;
        else hi = mid - 1u;
    }
    float t[8];
    ld32(e + 8 * j, t);
    const float f = (v - t[0]) * t[1];
#pragma unroll
    for (int l = 0; l < 3; ++l) dl[l] = t[2 + 2 * l] + f * t[3 + 2 * l];
}

// d / D correctly rounded from D's correctly rounded reciprocal rD, exact after the remainder's correction:
// Brisebarre, Muller and Raina, "Accelerating correctly rounded floating-point division when the divisor is
// known in advance", IEEE Trans. Computers 53 (2004). For quotients and remainders clear of underflow.
__device__ __forceinline__ float div_by_constant(float d, float D, float rD) {
    const float q0 = __fmul_rn(d, rD);
    return __fmaf_rn(__fmaf_rn(-q0, D, d), rD, q0);
}

// spk_sublayer_lambda with the quotients by div_by_constant (one small enough to underflow is clamped to
// 1e-6 in any case) and by spk_div_normal
__device__ __forceinline__ float sublayer_lambda_fast(float d, float D, float rD, float n, float u, float* sat_out) {
    float q = div_by_constant(d, D, rD);
    q = q < 1e-6f ? 1e-6f : (q > 0.999999f ? 0.999999f : q);
    const float sat = SPK_SUB(1.0f, SPK_MUL(SPK_MUL(q, u), 0.999999f));
    *sat_out = sat;
    return SPK_MUL(SPK_DIV_NORMAL(n, sat), q);
}

// PRODUCT: a warp with a draw of lambda below this runs the product method's first four uniforms in
// lockstep (at 4, 6, 8 and 10 the 24-megapixel export measured the same within 0.5 %).
constexpr float kProductLockstep = 6.0f;

// One pixel per lane. Every lane makes the first attempt of its nine draws, straight-line code with no
// branch; a draw that squeeze_certain does not settle (26 % in the 4K benchmark frame) is queued in the
// warp's ring as its slot alone, and the warp then takes 32 queued draws at a time, one attempt each, the
// rejected queued again behind the rest; product-method draws (lambda < 10, or NaN) are set aside and run
// last, so that a warp runs one method at a time. The kernel is bound by instruction issue (73 % of the
// slots, 83 warp instructions a pixel): 4K benchmark frame 1.48 ms with ten-step bisections of the
// densities' axis, general divides and the whole PTRS state in the ring, 0.80 this way.
// Ten blocks per SM: 0.826 ms against 0.840 (nine), 0.865 (no cap); eleven slow the exports by 2 %. Settling the
// full test in the lockstep too (half as many queued draws) cost what it saved (0.84); a queue shared by
// the block's warps lost more to its barriers (0.84 .. 0.90).
// HOOK: the counts or lambdas are written out too (the adjoint, tests).
template <bool PACKED, bool PRODUCT, bool HOOK>
__global__ void __launch_bounds__(kDrawWarps * 32, SPKB_DEVELOP_MIN_BLOCKS) k_develop_layers(const float* __restrict__ exposure,
                                                                    float* __restrict__ out, uint32_t w,
                                                                    uint32_t blocks_per_row,
                                                                    const __grid_constant__ DevelopArgs q) {
    __shared__ uint16_t ring[kDrawWarps][kDrawRing], product_list[kDrawWarps][9 * 32];
    __shared__ float lam[kDrawWarps][9 * 32], scale[9][kDrawWarps * 32];  // [c * 3 + l]; a count replaces its lambda
    const uint32_t lane = threadIdx.x & 31u, wi = threadIdx.x >> 5, tid = threadIdx.x;
    const uint32_t row = blockIdx.x / blocks_per_row, y = q.row0 + row;
    const uint32_t x = (blockIdx.x - row * blocks_per_row) * (kDrawWarps * 32) + threadIdx.x;
    const bool live = x < w;
    const uint32_t pixel = y * q.width + x;
    const size_t o = 3 * (size_t(y) * w + min(x, w - 1));  // a lane past the row works on its last pixel, queues and stores nothing
    uint16_t* ringw = ring[wi];
    uint16_t* productw = product_list[wi];
    float* resw = lam[wi];
    const uint32_t below = (1u << lane) - 1u;
    const PhiloxHead head0 = philox_head(pixel, q.seed);
    uint32_t tail = 0;
#pragma unroll
    for (uint32_t c = 0; c < 3; ++c) {
        float dl[3];
        float L = log10f(fmaxf(exposure[o + c], 0.0f) + 1e-10f);
        if (q.chi) L = __fsub_rn(L, q.chi[o + c]);  // DIR couplers: the corrected log exposure, the y0 curve
        if (PACKED) {
            const float D = curve_packed(q, c, L);
            layers_packed(q, c, q.positive ? -D : D, dl);
        } else {
            const float D = curve_lookup(q.cx, q.cinv, q.cy + size_t(c) * q.K, q.K, q.cgrid, L);
            layer_densities(q, c, q.positive ? -D : D, dl);
        }
#pragma unroll
        for (uint32_t l = 0; l < 3; ++l) {
            const uint32_t lc = l * 3 + c, k = c * 3 + l;
            float sat = 1.0f, value;
            const float d = dl[l] + q.dmin_l[lc];
            const float lm =
                PACKED ? sublayer_lambda_fast(d, q.sat_d[lc], q.rcp_sat_d[lc], q.count[lc], q.uniformity[c], &sat)
                       : spk_sublayer_lambda(d, q.sat_d[lc], q.count[lc], q.uniformity[c], &sat);
            if (HOOK && q.lam_out && live) q.lam_out[size_t(pixel) * 9 + k] = lm;
            scale[k][tid] = SPK_MUL(q.unit[lc], sat);  // unit: SPK_DIV(sat_d, count), formed once
            const spk_u4 words = philox_first(head0, q.stream_hi[k], q.stream_lo[k], q.seed);
            bool settled = squeeze_certain(lm, words.x, words.y, value);
            // the product method's first four uniforms, where some lane's draw is likely to end with them
            if (PRODUCT && __any_sync(0xFFFFFFFFu, lm < kProductLockstep)) {
                float prod = 1.0f;
                const uint32_t above = product_block(words, spk_expf_normal(-fminf(lm, 80.0f)), prod);
                if (lm < 10.0f && above < 4u) {
                    value = float(above);
                    settled = true;
                }
            }
            resw[k * 32u + lane] = settled ? value : lm;
            const uint32_t open = __ballot_sync(0xFFFFFFFFu, live && !settled);
            if (live && !settled) ringw[tail + __popc(open & below)] = uint16_t(k * 32u + lane);
            tail += __popc(open);
        }
    }
    __syncwarp();
    const auto stream_of = [](uint32_t slot) {
        const uint32_t k = slot >> 5, c = k / 3u;
        return SPK_STREAM_GRAIN(c, k - 3u * c);
    };
    const uint32_t pixel0 = pixel - lane;
    uint32_t n_product = 0;
    for (uint32_t head = 0; tail != head;) {
        const uint32_t n = min(tail - head, 32u);
        uint32_t slot = 0, it = 0;
        bool again = false, product = false;
        if (lane < n) {
            const uint32_t e = ringw[(head + lane) & (kDrawRing - 1u)];
            slot = e & 511u;
            it = e >> 9;
            const float lm = resw[slot];
            product = !(lm >= 10.0f);
            if (!product) again = !draw_attempt(resw + slot, lm, pixel0 + (slot & 31u), stream_of(slot), q.seed, it);
        }
        head += n;
        __syncwarp();
        const uint32_t m = __ballot_sync(0xFFFFFFFFu, again), mp = __ballot_sync(0xFFFFFFFFu, product);
        if (again) ringw[(tail + __popc(m & below)) & (kDrawRing - 1u)] = uint16_t(slot | (it + 1u) << 9);
        if (product) productw[n_product + __popc(mp & below)] = uint16_t(slot);
        tail += __popc(m);
        n_product += __popc(mp);
        __syncwarp();
    }
    for (uint32_t i = lane; i < n_product; i += 32u) {
        const uint32_t slot = productw[i];
        resw[slot] = poisson_product(resw[slot], pixel0 + (slot & 31u), stream_of(slot), q.seed);
    }
    __syncwarp();
    if (!live) return;
#pragma unroll
    for (int c = 0; c < 3; ++c) {
        float val[3];
#pragma unroll
        for (int l = 0; l < 3; ++l) {
            const float cnt = resw[(c * 3 + l) * 32 + lane];
            if (HOOK && q.counts_out) q.counts_out[size_t(pixel) * 9 + c * 3 + l] = cnt;
            val[l] = SPK_MUL(cnt, scale[c * 3 + l][tid]);
        }
        float G = ((0.0f + val[0]) + val[1]) + val[2];
        if (q.shift) G = G * 1.0f + (-q.dmin_c[c]);
        out[o + c] = G;
    }
}

// ---------------------------------------------------------------------------------------------------
// encode: reference kernels/print.metal:129-156 and :350-366 (helpers in encode.cuh).

__global__ void k_encode(const float* __restrict__ rgb, const float* __restrict__ gpl, uint16_t* __restrict__ out,
                         uint32_t w, uint32_t h, const __grid_constant__ EncodeArgs e) {
    const uint32_t x = blockIdx.x * blockDim.x + threadIdx.x;
    const uint32_t y = blockIdx.y * blockDim.y + threadIdx.y;
    if (x >= w || y >= h) return;
    const size_t i = 3 * (size_t(y) * w + x);
    float v0 = rgb[i], v1 = rgb[i + 1], v2 = rgb[i + 2];
    if (e.unsharp) {
        v0 = e.lincomb_a * v0 + e.lincomb_b * gpl[i];
        v1 = e.lincomb_a * v1 + e.lincomb_b * gpl[i + 1];
        v2 = e.lincomb_a * v2 + e.lincomb_b * gpl[i + 2];
    }
    edr_tone(e, v0, v1, v2);
    if (e.cctf_active) {
        float m0, m1, m2;
        mat_apply(e.m_nid, v0, v1, v2, m0, m1, m2);
        v0 = cctf_encode(m0, e.cctf_mode);
        v1 = cctf_encode(m1, e.cctf_mode);
        v2 = cctf_encode(m2, e.cctf_mode);
    }
    ushort4 p;
    p.x = encode16(v0);
    p.y = encode16(v1);
    p.z = encode16(v2);
    p.w = 65535;
    reinterpret_cast<ushort4*>(out)[size_t(y) * e.stride + x] = p;
}

// ---------------------------------------------------------------------------------------------------
// source copy: channels 3 or 4 -> interleaved RGB, non-finite -> 0 (reference src/session/session.cpp:164-168)

__global__ void k_source(const float* __restrict__ raw, float* __restrict__ out, size_t n, uint32_t channels) {
    const size_t i = size_t(blockIdx.x) * blockDim.x + threadIdx.x;
    if (i >= n) return;
#pragma unroll
    for (int c = 0; c < 3; ++c) {
        const float v = raw[i * channels + c];
        out[3 * i + c] = isfinite(v) ? v : 0.0f;
    }
}

// L2 flush: write a buffer larger than the L2 cache
__global__ void k_fill(uint4* p, size_t n, uint32_t v) {
    for (size_t i = size_t(blockIdx.x) * blockDim.x + threadIdx.x; i < n; i += size_t(gridDim.x) * blockDim.x)
        p[i] = make_uint4(v, v, v, v);
}

// ---------------------------------------------------------------------------------------------------
// test kernels

__global__ void k_sampler_poisson(const float* lam, float* out, uint32_t n, uint32_t stream, uint32_t seed) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    out[i] = spk_poisson(lam[i], i, stream, seed);
}

// The sampler's branch-free operations against the compiler's correctly rounded ones: how many of n results
// differ (SamplerOp).
__device__ __forceinline__ float ldexp_bits(uint32_t significand, int e) {
    return __uint_as_float(uint32_t(127 + e) << 23 | (significand & 0x007FFFFFu));
}

__global__ void k_sampler_ops(int op, uint64_t n, uint32_t seed, unsigned long long* wrong) {
    uint32_t bad = 0;
    for (uint64_t i = uint64_t(blockIdx.x) * blockDim.x + threadIdx.x; i < n; i += uint64_t(gridDim.x) * blockDim.x) {
        if (op == SAMPLER_OP_RCP || op == SAMPLER_OP_SQRT) {  // every significand, exponents from -100 up
            const float x = ldexp_bits(uint32_t(i), int(i >> 23) - 100);
            const float got = op == SAMPLER_OP_RCP ? SPK_RCP_NORMAL(x) : SPK_SQRT_NORMAL(x);
            const float want = op == SAMPLER_OP_RCP ? __frcp_rn(x) : __fsqrt_rn(x);
            bad += __float_as_uint(got) != __float_as_uint(want);
            continue;
        }
        spk_u4 c;
        c.x = uint32_t(i);
        c.y = uint32_t(i >> 32);
        c.z = uint32_t(op);
        c.w = 0u;
        const spk_u4 r = spk_philox(c, seed, 0u);
        float a = ldexp_bits(r.x, int(r.z % 81u) - 40), b = ldexp_bits(r.y, int(r.w % 121u) - 60);
        if (i & 1u) {
            // a quotient as near the middle of two floats as a 24-bit numerator allows: a = b times an odd
            // 25-bit number, cut to 24 bits, or the next float above
            const uint64_t Q = 0x1000001u | (r.x & 0xFFFFFFu), P = Q * (0x800000u | (r.y & 0x7FFFFFu));
            const uint32_t A = uint32_t(P >> (40 - __clzll((long long)P))) + uint32_t((i >> 1) & 1u);
            a = float(A);
        }
        const float want = __fdiv_rn(a, b);
        const float got = op == SAMPLER_OP_DIV ? SPK_DIV_NORMAL(a, b) : div_by_constant(a, b, __frcp_rn(b));
        bad += __float_as_uint(got) != __float_as_uint(want);
    }
    if (bad) atomicAdd(wrong, (unsigned long long)bad);
}

// The print glare's field (reference kernels/fx_grain.metal:99-116 with same_all): one lognormal value
// per pixel, on stream 200 with the print seed, written to the three channels.
__global__ void k_glare_field(float* out, uint32_t n, float mean, float sd, uint32_t seed) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const float v = spk_lognormal(mean, sd, i, 200u, seed);
    out[3 * size_t(i)] = v;
    out[3 * size_t(i) + 1] = v;
    out[3 * size_t(i) + 2] = v;
}

__global__ void k_sampler_lognormal(float* out, uint32_t n, float mean, float sd, uint32_t stream, uint32_t seed) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    out[i] = spk_lognormal(mean, sd, i, stream, seed);
}

__global__ void k_philox(const uint32_t* ctr, const uint32_t* key, uint32_t* out, uint32_t n) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    spk_u4 c;
    c.x = ctr[4 * i];
    c.y = ctr[4 * i + 1];
    c.z = ctr[4 * i + 2];
    c.w = ctr[4 * i + 3];
    const spk_u4 r = spk_philox(c, key[2 * i], key[2 * i + 1]);
    out[4 * i] = r.x;
    out[4 * i + 1] = r.y;
    out[4 * i + 2] = r.z;
    out[4 * i + 3] = r.w;
}

}  // namespace

// ---- launchers ------------------------------------------------------------------------------------

namespace {
thread_local LaunchHook* t_hook = nullptr;
std::atomic<uint64_t> g_launches{0};
}  // namespace

Probe::Probe(const char* name, cudaStream_t st) : s(st) {
    g_launches.fetch_add(1, std::memory_order_relaxed);
    if (t_hook) t_hook->before(name, s);
}
Probe::~Probe() {
    if (t_hook) t_hook->after(s);
}

unsigned long long current_context_id() {
    using GetCurrent = CUresult (*)(CUcontext*);
    using GetId = CUresult (*)(CUcontext, unsigned long long*);
    static GetCurrent get_current = nullptr;
    static GetId get_id = nullptr;
    static std::once_flag once;
    std::call_once(once, [] {
        void* f0 = nullptr;
        void* f1 = nullptr;
        cudaDriverEntryPointQueryResult q0{}, q1{};
        if (cudaGetDriverEntryPointByVersion("cuCtxGetCurrent", &f0, 12000, cudaEnableDefault, &q0) != cudaSuccess ||
            cudaGetDriverEntryPointByVersion("cuCtxGetId", &f1, 12000, cudaEnableDefault, &q1) != cudaSuccess ||
            !f0 || !f1)
            return;
        get_current = reinterpret_cast<GetCurrent>(f0);
        get_id = reinterpret_cast<GetId>(f1);
    });
    CUcontext ctx = nullptr;
    unsigned long long id = 0;
    if (!get_current || !get_id || get_current(&ctx) != CUDA_SUCCESS || !ctx || get_id(ctx, &id) != CUDA_SUCCESS)
        return 0;
    return id;
}

void ensure_smem(const void* kernel, int bytes) {
    static std::mutex m;
    static std::map<std::pair<const void*, unsigned long long>, int> done;
    unsigned long long ctx = current_context_id();
    if (ctx == 0) {  // no context yet: make the device's primary one current first
        cudaFree(nullptr);
        ctx = current_context_id();
    }
    std::lock_guard<std::mutex> g(m);
    int& cur = done[{kernel, ctx}];
    if (ctx != 0 && bytes <= cur) return;
    cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
    cur = bytes;
}

void set_launch_hook(LaunchHook* hook) { t_hook = hook; }
uint32_t sm_count() {
    static std::atomic<int> known[64];
    int dev = 0, n = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return 148;
    n = known[dev].load(std::memory_order_relaxed);
    if (n == 0) {
        if (cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || n <= 0) return 148;
        known[dev].store(n, std::memory_order_relaxed);
    }
    return uint32_t(n);
}

uint64_t launch_count() { return g_launches.load(); }

void expose(const float* rgb, float* h, const float* patches, const ExposeArgs& a, cudaStream_t s) {
    if (a.n == 0) return;
    Probe p("expose", s);
    k_expose_patch<<<div_up(a.n, kExposeThreads), kExposeThreads, 0, s>>>(rgb, h, patches, a);
}

void iir_tangent(const float* in, const float* in_dot, float* work, float* work_dot, float* out, float* out_dot,
                 uint32_t w, uint32_t h, bool vertical, const IirCoefs& c, const IirCoefs& dc, cudaStream_t s) {
    const uint32_t lines = vertical ? 3u * w : 3u * h;
    if (lines == 0) return;
    Probe p("iir_tangent", s);
    // lines staged in shared memory where they fit, kTanSegs threads per line (strips of up to 10 rows or 4
    // pixel columns, at most 32 lines for the 256-thread CTA); the lines in global memory otherwise
    int dev = 0, optin = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
    const size_t n = vertical ? h : w;
    TangentMaps maps{};
    maps.L = uint32_t((n + kTanSegs - 1) / kTanSegs);
    for (int ch = 0; ch < 3; ++ch) {
        // the homogeneous one-step map A of (w1, w2, w3, t1, t2, t3), raised to the L-th power by squaring
        double A[36] = {0}, R[36] = {0}, T[36];
        A[0] = c.B1[ch], A[1] = c.B2[ch], A[2] = c.B3[ch];
        A[6] = 1.0;
        A[13] = 1.0;
        A[18] = dc.B1[ch], A[19] = dc.B2[ch], A[20] = dc.B3[ch], A[21] = c.B1[ch], A[22] = c.B2[ch], A[23] = c.B3[ch];
        A[27] = 1.0;
        A[34] = 1.0;
        for (int i = 0; i < 6; ++i) R[i * 7] = 1.0;
        auto mul = [&](const double* X, const double* Y, double* Z) {
            for (int r = 0; r < 6; ++r)
                for (int q2 = 0; q2 < 6; ++q2) {
                    double acc = 0.0;
                    for (int m = 0; m < 6; ++m) acc += X[r * 6 + m] * Y[m * 6 + q2];
                    T[r * 6 + q2] = acc;
                }
            for (int i = 0; i < 36; ++i) Z[i] = T[i];
        };
        for (uint32_t e = maps.L; e > 0; e >>= 1) {
            if (e & 1u) mul(R, A, R);
            mul(A, A, A);
        }
        for (int i = 0; i < 36; ++i) maps.AL[ch][i] = R[i];
    }
    for (uint32_t px : {10u, 8u, 4u, 2u, 1u}) {
        if (vertical && px > 4u) continue;
        const size_t smem = size_t(3 * px) * kTanSegs * 6 * sizeof(double) + 2 * n * (3 * px) * sizeof(float);
        if (smem > size_t(optin)) continue;
        ensure_smem(reinterpret_cast<const void*>(k_iir_tangent_seg), int(smem));
        const uint32_t ctas = div_up(vertical ? w : h, px);
        k_iir_tangent_seg<<<ctas, 256, smem, s>>>(in, in_dot, out, out_dot, w, h, vertical ? 1 : 0, px, c, dc, maps);
        return;
    }
    // a thread per line and few lines (3 per row or column): 32-thread CTAs spread them over more SMs
    k_iir_tangent<<<div_up(lines, 32), 32, 0, s>>>(in, in_dot, work, work_dot, out, out_dot, w, h, vertical ? 1 : 0, c,
                                                   dc);
}

void fir_v(const float* in, float* out, uint32_t w, uint32_t h, const FirTaps& t, cudaStream_t s) {
    const dim3 b(32, 8), g(div_up(w, 32), div_up(h, 8));
    Probe p("fir_v", s);
    k_fir_v<<<g, b, 0, s>>>(in, out, w, h, t);
}

void fir_h(const float* in, float* out, const float* acc, uint32_t w, uint32_t h, const FirTaps& t, int mode,
           const float weight[3], cudaStream_t s) {
    const dim3 b(32, 8), g(div_up(w, 32), div_up(h, 8));
    Probe p("fir_h", s);
    k_fir_h<<<g, b, 0, s>>>(in, out, acc, w, h, t, mode, weight[0], weight[1], weight[2]);
}

void iir_h_lines(const IirLineJobs& j, uint32_t w, uint32_t h, cudaStream_t s) {
    if (uint64_t(w) * h == 0 || j.n == 0) return;
    Probe p("iir_h", s);
    k_iir_h<<<dim3(div_up(h, kLineRows), j.n), 32, 0, s>>>(w, h, j);
}

void iir_v_lines(const IirLineJobs& j, uint32_t w, uint32_t h, cudaStream_t s) {
    if (uint64_t(w) * h == 0 || j.n == 0) return;
    Probe p("iir_v", s);
    k_iir_v<ACC_NONE><<<dim3(div_up(3 * w, 32), j.n), 32, 0, s>>>(nullptr, w, h, j, 1.0f, 1.0f, 1.0f);
}

void iir_h(const float* in, float* out, uint32_t w, uint32_t h, const IirCoefs& c, cudaStream_t s) {
    IirLineJobs j{};
    j.n = 1;
    j.in[0] = in;
    j.work[0] = out;
    j.q[0] = c;
    iir_h_lines(j, w, h, s);
}

void iir_v(float* work, float* out, const float* acc, uint32_t w, uint32_t h, const IirCoefs& c, int mode,
           const float weight[3], cudaStream_t s) {
    IirLineJobs j{};
    j.n = 1;
    j.work[0] = work;
    j.out[0] = out;
    j.q[0] = c;
    if (mode == ACC_NONE) {
        iir_v_lines(j, w, h, s);
        return;
    }
    if (uint64_t(w) * h == 0) return;
    Probe p("iir_v", s);
    const uint32_t g = div_up(3 * w, 32);
    if (mode == ACC_ZERO) k_iir_v<ACC_ZERO><<<g, 32, 0, s>>>(acc, w, h, j, weight[0], weight[1], weight[2]);
    else k_iir_v<ACC_PLANE><<<g, 32, 0, s>>>(acc, w, h, j, weight[0], weight[1], weight[2]);
}

void lincomb(const float* x, const float* y, float* out, size_t pixels, const float a[3], const float b[3],
             cudaStream_t s) {
    if (pixels == 0) return;
    Probe p("lincomb", s);
    k_lincomb<<<unsigned((pixels + 255) / 256), 256, 0, s>>>(x, y, out, pixels, a[0], a[1], a[2], b[0], b[1], b[2]);
}

void copy(const float* x, float* out, size_t pixels, cudaStream_t s) {
    const size_t n = 3 * pixels;
    if (n == 0) return;
    Probe p("copy", s);
    k_copy<<<unsigned((n + 255) / 256), 256, 0, s>>>(x, out, n);
}

void develop_prepare(cudaStream_t s) {
    static std::mutex m;
    static bool done[64] = {};
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return;
    std::lock_guard<std::mutex> g(m);
    if (done[dev]) return;
    k_lgamma_table<<<div_up(kLgammaTable, 256), 256, 0, s>>>();
    // once written and waited for, every later launch on any stream reads the table
    if (cudaStreamSynchronize(s) == cudaSuccess && cudaGetLastError() == cudaSuccess) done[dev] = true;
}

void develop(const float* exposure, float* out, const DevelopArgs& a, uint32_t w, uint32_t h, cudaStream_t s) {
    if (uint64_t(w) * h == 0) return;
    if (a.grain && a.mode == 0) {
        develop_prepare(s);
        const uint32_t bx = div_up(w, kDrawWarps * 32);
        Probe p("develop_layers", s);
        // The product method's lockstep pays where many lambdas are below 6: with DIR couplers, whose
        // corrected densities reach far down, and pixels small against a grain. Measured with couplers at
        // 1920 x 1280, without and with it: 52 um (2,800 grains a pixel) 0.28 / 0.31 ms, 18 um (340) 0.38 / 0.41,
        // 12.5 um (160) 0.42 / 0.43 on a photograph and 0.51 / 0.50 on noise, 7.8 um (63) 0.41 / 0.37, 5.7 um
        // (34) 0.38 / 0.32; without couplers it never gained more than 2 %.
        float mean = 0.0f;
        for (int i = 0; i < 9; ++i) mean += a.count[i] / 9.0f;
        const bool product = a.chi && mean < 160.0f;
        const dim3 g(bx * h), b(kDrawWarps * 32);
        auto kernel = k_develop_layers<false, true, true>;
        if (a.counts_out || a.lam_out) {
            if (a.packed) kernel = product ? k_develop_layers<true, true, true> : k_develop_layers<true, false, true>;
        } else {
            kernel = k_develop_layers<false, true, false>;
            if (a.packed) kernel = product ? k_develop_layers<true, true, false> : k_develop_layers<true, false, false>;
        }
        kernel<<<g, b, 0, s>>>(exposure, out, w, bx, a);
        return;
    }
    const dim3 b(32, 4), g(div_up(w, 32), div_up(h, 4));
    Probe p("develop", s);
    k_develop<<<g, b, 0, s>>>(exposure, out, w, h, a);
}

void develop_rows(const float* exposure, float* out, const DevelopArgs& a, uint32_t w, uint32_t row0, uint32_t rows,
                  cudaStream_t s) {
    DevelopArgs b = a;
    b.row0 = row0;
    develop(exposure, out, b, w, rows, s);
}

void coupler_source(const float* exposure, float* chi, const CouplerArgs& a, cudaStream_t s) {
    if (a.n == 0) return;
    Probe p("coupler_source", s);
    k_coupler_source<<<div_up(a.n, 256), 256, 0, s>>>(exposure, chi, a);
}

void encode(const float* rgb, const float* g, uint16_t* out, uint32_t w, uint32_t h, const EncodeArgs& e,
            cudaStream_t s) {
    const dim3 b(32, 8), gr(div_up(w, 32), div_up(h, 8));
    Probe p("encode", s);
    k_encode<<<gr, b, 0, s>>>(rgb, g, out, w, h, e);
}

void source_copy(const float* raw, float* out, size_t pixels, uint32_t channels, cudaStream_t s) {
    if (pixels == 0) return;
    Probe p("source_copy", s);
    k_source<<<unsigned((pixels + 255) / 256), 256, 0, s>>>(raw, out, pixels, channels);
}

void fill(void* p, size_t bytes, uint32_t v, cudaStream_t s) {
    Probe pr("fill", s);
    k_fill<<<sm_count() * 8, 256, 0, s>>>(static_cast<uint4*>(p), bytes / 16, v);
}

void sampler_poisson(const float* lam, float* out, uint32_t n, uint32_t stream, uint32_t seed, cudaStream_t s) {
    if (n == 0) return;
    Probe p("sampler_poisson", s);
    k_sampler_poisson<<<div_up(n, 128), 128, 0, s>>>(lam, out, n, stream, seed);
}

void sampler_ops(int op, uint64_t n, uint32_t seed, unsigned long long* wrong, cudaStream_t s) {
    if (n == 0) return;
    Probe p("sampler_ops", s);
    k_sampler_ops<<<unsigned(std::min<uint64_t>((n + 255) / 256, 4096)), 256, 0, s>>>(op, n, seed, wrong);
}

void glare_field(float* out, uint32_t pixels, float mean, float sd, uint32_t seed, cudaStream_t s) {
    Probe p("glare_field", s);
    k_glare_field<<<div_up(pixels, 256), 256, 0, s>>>(out, pixels, mean, sd, seed);
}

void sampler_lognormal(float* out, uint32_t n, float mean, float stddev, uint32_t stream, uint32_t seed,
                       cudaStream_t s) {
    if (n == 0) return;
    Probe p("sampler_lognormal", s);
    k_sampler_lognormal<<<div_up(n, 128), 128, 0, s>>>(out, n, mean, stddev, stream, seed);
}

void philox_blocks(const uint32_t* ctr, const uint32_t* key, uint32_t* out, uint32_t n, cudaStream_t s) {
    if (n == 0) return;
    Probe p("philox", s);
    k_philox<<<div_up(n, 128), 128, 0, s>>>(ctr, key, out, n);
}

}  // namespace spkb::dev
