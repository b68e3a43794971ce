// The scanner stage in one pass: lens blur (FIR), unsharp mask (FIR + combine), output matrix, transfer
// function and RGBA16 encode, over 32 x 32 pixel tiles staged in shared memory.
//
// Reference: src/fx/scanner.cpp:16-31 (blur, then (1 + a) x - a G(x)), kernels/fx_blur.metal:20-78
// (FIR: taps -r..r ascending, binary32 accumulator from 0, half-sample symmetric reflection at the
// edges, a vertical pass then a horizontal pass) and kernels/print.metal:350-366 (encode).
//
// Every intermediate value is the one the separate passes compute: each pass is evaluated only at
// pixels inside the image, in the same tap order, and where a pass reads past an edge it reads the
// value at the reflected pixel. The vertical passes do not mix columns, so a column loaded from the
// reflected source column already carries the reflected result; after the lens blur's horizontal pass
// the tile copies the reflected values into the (at most r2 wide) border that the unsharp pass reads.
//
// Shared memory (floats, interleaved RGB rows), R = r1 + r2:
//   A: the print output with an R halo (TH + 2R rows x 3 (TW + 2R)), later the lens-blurred tile with an
//      r2 halo (TH + 2 r2 rows x 3 (TW + 2 r2))
//   B: the lens blur's vertical pass (TH + 2 r2 rows x 3 (TW + 2R)), later the unsharp vertical pass
//      (TH rows x 3 (TW + 2 r2))
#include <cuda_runtime.h>
#include <stdint.h>

#include <type_traits>

#include "../kernel_args.h"
#include "encode.cuh"
#include "launch.hpp"

namespace spkb::dev {

namespace {

// threads per tile CTA (4K scanner: 0.326 ms at 128, 0.209 at 256, 0.191 at 512; the pixels are the same)
#ifndef SPKB_SCAN_THREADS
#define SPKB_SCAN_THREADS 512
#endif
constexpr int kTW = 32, kTH = 32, kThreads = SPKB_SCAN_THREADS, kWarps = kThreads / 32;
static_assert(uint32_t(kTH) == scan_tile_rows(), "row bands start on tile rows");

// half-sample symmetric reflection, exact for p in [-n, 2n)
__device__ __forceinline__ int reflect_near(int p, int n) { return p < 0 ? -1 - p : (p >= n ? 2 * n - 1 - p : p); }

// FIR passes over rows in shared memory with register windows: a thread forms kWin outputs of one float
// column (window_v) or of one channel in one row (window_h) and reads each input they share once; every output
// is sum_k t[k] x[i + k] from 0, k ascending. window_v: rows x cols floats of dst from rows + 2 R of src;
// window_h: rows x px pixels of dst from px + 2 R of src. Outputs past the image are formed from whatever
// the rows hold and never used.
// 12 outputs: the 36 rows and pixels of the 4K scanner's lens-blurred tile take three windows each, one turn
// of the CTA (4K scanner 0.185 ms with 6 and 4, two turns, 0.172 with 12).
constexpr int kWin = 12;

template <int R>
__device__ __forceinline__ void window_v(const float* src, int sp, float* dst, int dp, int rows, int cols, const float* t) {
    constexpr int T = 2 * R + 1;
    const int items = cols * ((rows + kWin - 1) / kWin);
    for (int item = threadIdx.x; item < items; item += kThreads) {
        const int blk = item / cols, f = item - blk * cols, i0 = blk * kWin;
        float acc[kWin];
#pragma unroll
        for (int o = 0; o < kWin; ++o) acc[o] = 0.0f;
#pragma unroll
        for (int j = 0; j < kWin + T - 1; ++j)
            if (i0 + j < rows + T - 1) {
                const float v = src[(i0 + j) * sp + f];
#pragma unroll
                for (int o = 0; o < kWin; ++o)
                    if (j - o >= 0 && j - o < T) acc[o] += t[j - o] * v;
            }
#pragma unroll
        for (int o = 0; o < kWin; ++o)
            if (i0 + o < rows) dst[(i0 + o) * dp + f] = acc[o];
    }
}

template <int R>
__device__ __forceinline__ void window_h(const float* src, int sp, float* dst, int dp, int rows, int px, const float* t) {
    constexpr int T = 2 * R + 1;
    const int per = 3 * ((px + kWin - 1) / kWin), items = rows * per;
    for (int item = threadIdx.x; item < items; item += kThreads) {
        const int i = item / per, rem = item - i * per, c = rem % 3, j0 = (rem / 3) * kWin;
        const float* row = src + i * sp + c;
        float acc[kWin];
#pragma unroll
        for (int o = 0; o < kWin; ++o) acc[o] = 0.0f;
#pragma unroll
        for (int q = 0; q < kWin + T - 1; ++q)
            if (j0 + q < px + T - 1) {
                const float v = row[3 * (j0 + q)];
#pragma unroll
                for (int o = 0; o < kWin; ++o)
                    if (q - o >= 0 && q - o < T) acc[o] += t[q - o] * v;
            }
#pragma unroll
        for (int o = 0; o < kWin; ++o)
            if (j0 + o < px) dst[i * dp + 3 * (j0 + o) + c] = acc[o];
    }
}

// f<R>() for the radius r, 1 .. SPKB_FIR_MAX_R; RC >= 0: r is RC, known when compiled
template <int RC, class F>
__device__ __forceinline__ void with_radius(int r, F&& f) {
    if constexpr (RC >= 0) {
        f(std::integral_constant<int, RC>());
    } else {
        switch (r) {
            case 1: f(std::integral_constant<int, 1>()); break;
            case 2: f(std::integral_constant<int, 2>()); break;
            case 3: f(std::integral_constant<int, 3>()); break;
            case 4: f(std::integral_constant<int, 4>()); break;
            case 5: f(std::integral_constant<int, 5>()); break;
            case 6: f(std::integral_constant<int, 6>()); break;
            case 7: f(std::integral_constant<int, 7>()); break;
            case 8: f(std::integral_constant<int, 8>()); break;
            default: f(std::integral_constant<int, 9>()); break;
        }
    }
}

// One 32 x 32 output tile at (x0, y0) of a frame; smem as sized by scan_smem_bytes for the radii.
template <int R1, int R2>
__device__ __forceinline__ void scan_tile(const ScanArgs& a, const float* __restrict__ rgb, uint16_t* __restrict__ out,
                                          int w, int h, int x0, int y0, float* smem) {
    const int r1 = R1 >= 0 ? R1 : a.r1, r2 = R2 >= 0 ? R2 : a.r2, R = r1 + r2;
    const int PC = 3 * (kTW + 2 * R);  // floats per row of the print tile and the first vertical pass
    const int PR = kTH + 2 * R;
    const int BR = kTH + 2 * r2;       // rows of the lens-blurred tile
    const int BC = 3 * (kTW + 2 * r2);
    float* A = smem;
    float* B = smem + PR * PC;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;

    // 1. the print output at (y0 - R + i, x0 - R + j), reflected; pixels more than R past an edge are
    //    never read and load a clamped pixel. A tile whose haloed columns lie inside the frame reads each
    //    row's floats contiguously, with no per-element reflection.
    const bool inner_x = x0 - R >= 0 && x0 + kTW + R <= w;
    for (int i = warp; i < PR; i += kWarps) {
        const int yy = min(max(reflect_near(y0 - R + i, h), 0), h - 1);
        const float* row = rgb + size_t(yy) * size_t(w) * 3;
        if (inner_x) {
            const float* seg = row + 3 * (x0 - R);
            for (int f = lane; f < PC; f += 32) A[i * PC + f] = __ldg(seg + f);
            continue;
        }
        for (int f = lane; f < PC; f += 32) {
            const int j = f / 3, c = f - 3 * j;
            const int xx = min(max(reflect_near(x0 - R + j, w), 0), w - 1);
            A[i * PC + f] = __ldg(row + 3 * xx + c);
        }
    }
    __syncthreads();

    // 2., 3. lens blur, vertical (B: the tile's rows and its r2 halo, every column) and horizontal (back to A);
    // without one the tile as loaded is the lens-blurred tile, its rows at the same pitch
    if (r1 > 0) {
        with_radius<R1>(r1, [&](auto r) { window_v<decltype(r)::value>(A, PC, B, PC, BR, PC, a.t1); });
        __syncthreads();
        with_radius<R1>(r1, [&](auto r) { window_h<decltype(r)::value>(B, PC, A, BC, BR, kTW + 2 * r2, a.t1); });
        __syncthreads();
    }

    if (r2 > 0) {
        // 4. the border up to r2 past an edge takes the lens-blurred value of the reflected pixel
        if (x0 - r2 < 0 || x0 + kTW + r2 > w || y0 - r2 < 0 || y0 + kTH + r2 > h) {
            for (int i = warp; i < BR; i += kWarps) {
                const int yy = y0 - r2 + i;
                if (yy < -r2 || yy >= h + r2) continue;
                const bool row_out = yy < 0 || yy >= h;
                const int is = reflect_near(yy, h) - (y0 - r2);
                for (int fb = lane; fb < BC; fb += 32) {
                    const int jb = fb / 3, c = fb - 3 * jb;
                    const int xx = x0 - r2 + jb;
                    if (xx < -r2 || xx >= w + r2) continue;
                    if (!row_out && xx >= 0 && xx < w) continue;
                    const int js = reflect_near(xx, w) - (x0 - r2);
                    A[i * BC + fb] = A[is * BC + 3 * js + c];
                }
            }
            __syncthreads();
        }
        // 5. unsharp blur, vertical, every column of the blurred tile
        with_radius<R2>(r2, [&](auto r) { window_v<decltype(r)::value>(A, BC, B, BC, kTH, BC, a.t2); });
        __syncthreads();
    }

    // 6. unsharp horizontal pass and combine, matrix, transfer function, RGBA16: a pixel per lane
    const EncodeArgs& e = a.e;
    for (int i = warp; i < kTH; i += kWarps) {
        const int yy = y0 + i, xx = x0 + lane;
        if (yy >= h) break;
        if (xx >= w) continue;
        const float* bc = A + (i + r2) * BC + 3 * (lane + r2);
        float v0 = bc[0], v1 = bc[1], v2 = bc[2];
        if (e.unsharp) {
            // a radius of 0 (a mask of a small tier of a large frame): the one tap on the tile itself, no pass before
            const float* vr = r2 > 0 ? B + i * BC + 3 * lane : bc;
            float g0 = 0.0f, g1 = 0.0f, g2 = 0.0f;
#pragma unroll
            for (int k = 0; k <= 2 * r2; ++k) {
                g0 += a.t2[k] * vr[3 * k];
                g1 += a.t2[k] * vr[3 * k + 1];
                g2 += a.t2[k] * vr[3 * k + 2];
            }
            v0 = e.lincomb_a * v0 + e.lincomb_b * g0;
            v1 = e.lincomb_a * v1 + e.lincomb_b * g1;
            v2 = e.lincomb_a * v2 + e.lincomb_b * g2;
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
        reinterpret_cast<ushort4*>(out)[size_t(yy) * e.stride + xx] = p;
    }
}

template <int R1, int R2>
__global__ void __launch_bounds__(kThreads) k_scan_encode(const float* __restrict__ rgb, uint16_t* __restrict__ out,
                                                          int w, int h, int row0, const __grid_constant__ ScanArgs a) {
    extern __shared__ float smem[];
    scan_tile<R1, R2>(a, rgb, out, w, h, blockIdx.x * kTW, row0 + int(blockIdx.y) * kTH, smem);
}

// The scanner stage of many frames in one persistent launch: the CTAs take tiles t = blockIdx.x,
// blockIdx.x + gridDim.x, ... of the frames' concatenated tile lists (row-major within a frame).
template <int R1, int R2>
__global__ void __launch_bounds__(kThreads) k_scan_encode_batch(const BatchScanFrame* __restrict__ frames,
                                                                uint32_t n_frames, uint32_t n_tiles) {
    extern __shared__ float smem[];
    for (uint32_t t = blockIdx.x; t < n_tiles; t += gridDim.x) {
        uint32_t lo = 0, hi = n_frames;  // the last frame whose first tile is <= t
        while (hi - lo > 1) {
            const uint32_t mid = (lo + hi) / 2;
            if (frames[mid].first_tile <= t) lo = mid;
            else hi = mid;
        }
        const BatchScanFrame& f = frames[lo];
        const uint32_t local = t - f.first_tile;
        const uint32_t ty = local / f.tiles_x, tx = local - ty * f.tiles_x;
        __syncthreads();  // the previous tile's reads of shared memory are done
        scan_tile<R1, R2>(f.args, f.rgb, f.out, int(f.w), int(f.h), int(tx) * kTW, int(ty) * kTH, smem);
    }
}

// A separable FIR Gaussian with one tap vector for the three channels, both passes in one tiled kernel:
// the vertical pass at the tile's rows (every column of the haloed tile; a halo column holds the
// reflected source column, so its vertical result is that of the reflected column), then the horizontal
// pass. out must not alias in (neighbouring tiles read in's halo).
template <int R>
__global__ void __launch_bounds__(kThreads) k_fir_tile(const float* __restrict__ in, float* __restrict__ out, int w,
                                                       int h, int row0, const __grid_constant__ ScanArgs a) {
    extern __shared__ float smem[];
    const int r = R >= 0 ? R : a.r1;
    const int PC = 3 * (kTW + 2 * r), PR = kTH + 2 * r;
    float* A = smem;
    float* B = smem + PR * PC;
    const int x0 = blockIdx.x * kTW, y0 = row0 + int(blockIdx.y) * kTH;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const bool inner_x = x0 - r >= 0 && x0 + kTW + r <= w;  // the haloed columns lie inside the frame
    for (int i = warp; i < PR; i += kWarps) {
        const int yy = min(max(reflect_near(y0 - r + i, h), 0), h - 1);
        const float* row = in + size_t(yy) * size_t(w) * 3;
        if (inner_x) {
            const float* seg = row + 3 * (x0 - r);
            for (int f = lane; f < PC; f += 32) A[i * PC + f] = __ldg(seg + f);
            continue;
        }
        for (int f = lane; f < PC; f += 32) {
            const int j = f / 3, c = f - 3 * j;
            const int xx = min(max(reflect_near(x0 - r + j, w), 0), w - 1);
            A[i * PC + f] = __ldg(row + 3 * xx + c);
        }
    }
    __syncthreads();
    if constexpr (R >= 0) {
        // register windows: a thread takes kFRows consecutive rows of one column and reads each input row
        // once; every output is still sum_k t[k] A[i + k] from 0, k ascending
        constexpr int T = 2 * R + 1, PCc = 3 * (kTW + 2 * R), kFRows = 8, NB = kTH / kFRows;
        for (int item = threadIdx.x; item < PCc * NB; item += kThreads) {
            const int f = item % PCc, i0 = (item / PCc) * kFRows;
            float acc[kFRows];
#pragma unroll
            for (int o = 0; o < kFRows; ++o) acc[o] = 0.0f;
#pragma unroll
            for (int j = 0; j < kFRows + T - 1; ++j) {
                const float v = A[(i0 + j) * PCc + f];
#pragma unroll
                for (int o = 0; o < kFRows; ++o)
                    if (j - o >= 0 && j - o < T) acc[o] += a.t1[j - o] * v;
            }
#pragma unroll
            for (int o = 0; o < kFRows; ++o)
                if (y0 + i0 + o < h) B[(i0 + o) * PCc + f] = acc[o];
        }
    } else {
    for (int i = warp; i < kTH; i += kWarps) {
        if (y0 + i >= h) break;
        for (int f = lane; f < PC; f += 32) {
            float acc = 0.0f;
#pragma unroll
            for (int k = 0; k <= 2 * r; ++k) acc += a.t1[k] * A[(i + k) * PC + f];
            B[i * PC + f] = acc;
        }
    }
    }
    __syncthreads();
    const int OC = 3 * kTW;
    for (int i = warp; i < kTH; i += kWarps) {
        const int yy = y0 + i;
        if (yy >= h) break;
        float* orow = out + size_t(yy) * size_t(w) * 3 + size_t(x0) * 3;
        const int lim = 3 * min(kTW, w - x0);
        for (int f = lane; f < OC; f += 32) {
            if (f >= lim) break;
            float acc = 0.0f;
#pragma unroll
            for (int k = 0; k <= 2 * r; ++k) acc += a.t1[k] * B[i * PC + f + 3 * k];
            orow[f] = acc;
        }
    }
}

// A run of FIR Gaussians of one plane, per-channel taps (fir_mixture): the haloed tile is loaded once for
// every component; a component's vertical pass writes the tile's rows (every column it needs) to a second
// buffer, its horizontal pass keeps eight pixels of one channel per thread, whose running sum stays in
// registers until the tile is written. Both passes slide register windows of eight outputs over their inputs,
// the taps of the thread's channel in registers, each output the sum of tap x sample from 0, taps ascending,
// as the separate passes form it. Those (k_fir_v, k_fir_h: a thread per pixel, 2 r + 1 reads of the plane per
// output and pass, a plane written and read again per pass) took 1.84 ms for a 6000 x 4000 export's scatter
// and couplers, this 0.69; 1999 x 1333 0.34 and 0.13. Bound by the tile's barriers and shared-memory reads.
constexpr int kMixThreads = 384, kMixWin = 8;
static_assert(kMixThreads == kTH * 3 * (kTW / kMixWin), "a thread per row, channel and window");

// the vertical buffer's pitch: at least 3 (kTW + 2 r) floats, 3 modulo 32, so that the horizontal pass's lanes
// (twelve to a row: floats 24 g + c) of neighbouring rows fall in different banks
__host__ __device__ constexpr int mix_pitch(int r) { return (3 * (kTW + 2 * r) - 3 + 31) / 32 * 32 + 3; }

template <int R>
__device__ __forceinline__ void mix_component(const float* A, int pa, int rmax, float* B, int pb, const float* taps,
                                              float (&out)[kMixWin]) {
    constexpr int T = 2 * R + 1, kCols = 3 * (kTW + 2 * R), kItems = kCols * (kTH / kMixWin);
    const float* corner = A + (rmax - R) * (pa + 3);
    for (int item = threadIdx.x; item < kItems; item += kMixThreads) {
        const int f = item % kCols, i0 = (item / kCols) * kMixWin;
        const float* t = taps + (f % 3) * (2 * SPKB_FIR_MAX_R + 1);
        float tp[T], acc[kMixWin];
#pragma unroll
        for (int k = 0; k < T; ++k) tp[k] = t[k];
#pragma unroll
        for (int o = 0; o < kMixWin; ++o) acc[o] = 0.0f;
#pragma unroll
        for (int j = 0; j < kMixWin + T - 1; ++j) {
            const float v = corner[(i0 + j) * pa + f];
#pragma unroll
            for (int o = 0; o < kMixWin; ++o)
                if (j - o >= 0 && j - o < T) acc[o] = __fmaf_rn(tp[j - o], v, acc[o]);
        }
#pragma unroll
        for (int o = 0; o < kMixWin; ++o) B[(i0 + o) * pb + f] = acc[o];
    }
    __syncthreads();
    const int i = threadIdx.x / 12, c = threadIdx.x % 3, g = (threadIdx.x % 12) / 3;
    const float* row = B + i * pb + 3 * kMixWin * g + c;
    const float* t = taps + c * (2 * SPKB_FIR_MAX_R + 1);
    float tp[T];
#pragma unroll
    for (int k = 0; k < T; ++k) tp[k] = t[k];
#pragma unroll
    for (int o = 0; o < kMixWin; ++o) out[o] = 0.0f;
#pragma unroll
    for (int q = 0; q < kMixWin + T - 1; ++q) {
        const float v = row[3 * q];
#pragma unroll
        for (int o = 0; o < kMixWin; ++o)
            if (q - o >= 0 && q - o < T) out[o] = __fmaf_rn(tp[q - o], v, out[o]);
    }
    __syncthreads();  // B is free for the next component
}

__global__ void __launch_bounds__(kMixThreads, 3) k_fir_mixture(const float* __restrict__ in, float* out, const float* acc,
                                                                int w, int h, const __grid_constant__ FirMixArgs a) {
    extern __shared__ float smem[];
    const int rm = a.rmax, pa = 3 * (kTW + 2 * rm), pr = kTH + 2 * rm, pb = mix_pitch(rm);
    float* A = smem;
    float* B = A + pr * pa;
    float* taps = B + kTH * pb;  // the component's [channel][tap]
    const int x0 = blockIdx.x * kTW, y0 = blockIdx.y * kTH;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const bool inner_x = x0 - rm >= 0 && x0 + kTW + rm <= w;
    for (int i = warp; i < pr; i += kMixThreads / 32) {
        const int yy = min(max(reflect_near(y0 - rm + i, h), 0), h - 1);
        const float* row = in + size_t(yy) * size_t(w) * 3;
        if (inner_x) {
            const float* seg = row + 3 * (x0 - rm);
            for (int f = lane; f < pa; f += 32) A[i * pa + f] = __ldg(seg + f);
            continue;
        }
        for (int f = lane; f < pa; f += 32) {
            const int j = f / 3, c = f - 3 * j;
            const int xx = min(max(reflect_near(x0 - rm + j, w), 0), w - 1);
            A[i * pa + f] = __ldg(row + 3 * xx + c);
        }
    }
    // the tile's place in the planes: rows of up to 3 kTW floats, staged in B on the way in and out
    const int rows = min(kTH, h - y0), cols = 3 * min(kTW, w - x0);
    const size_t o0 = (size_t(y0) * w + x0) * 3;
    const auto staged = [&](auto&& f) {
        for (int e = threadIdx.x; e < kTH * 3 * kTW; e += kMixThreads) {
            const int i = e / (3 * kTW), j = e - i * (3 * kTW);
            if (i < rows && j < cols) f(B[i * pb + j], o0 + size_t(i) * w * 3 + j);
        }
    };
    const int ti = threadIdx.x / 12, tc = threadIdx.x % 3, tg = (threadIdx.x % 12) / 3;
    float* mine = B + ti * pb + 3 * kMixWin * tg + tc;
    float sum[kMixWin];
#pragma unroll
    for (int o = 0; o < kMixWin; ++o) sum[o] = 0.0f;
    if (a.mode == ACC_PLANE) {
        staged([&](float& b, size_t o) { b = acc[o]; });
        __syncthreads();
#pragma unroll
        for (int o = 0; o < kMixWin; ++o) sum[o] = mine[3 * o];
    }
    for (uint32_t k = 0; k < a.n; ++k) {
        const FirTaps& t = a.t[k];
        for (int e = threadIdx.x; e < 3 * (2 * SPKB_FIR_MAX_R + 1); e += kMixThreads)
            taps[e] = (&t.taps[0][0])[e];
        __syncthreads();
        float v[kMixWin];
        switch (t.r) {
            case 1: mix_component<1>(A, pa, rm, B, pb, taps, v); break;
            case 2: mix_component<2>(A, pa, rm, B, pb, taps, v); break;
            case 3: mix_component<3>(A, pa, rm, B, pb, taps, v); break;
            case 4: mix_component<4>(A, pa, rm, B, pb, taps, v); break;
            case 5: mix_component<5>(A, pa, rm, B, pb, taps, v); break;
            case 6: mix_component<6>(A, pa, rm, B, pb, taps, v); break;
            case 7: mix_component<7>(A, pa, rm, B, pb, taps, v); break;
            case 8: mix_component<8>(A, pa, rm, B, pb, taps, v); break;
            case 9: mix_component<9>(A, pa, rm, B, pb, taps, v); break;
            default: mix_component<0>(A, pa, rm, B, pb, taps, v); break;
        }
        const float wk = a.weight[k][tc];
#pragma unroll
        for (int o = 0; o < kMixWin; ++o) sum[o] = a.mode == ACC_NONE ? v[o] : __fmaf_rn(wk, v[o], sum[o]);
    }
#pragma unroll
    for (int o = 0; o < kMixWin; ++o) mine[3 * o] = sum[o];
    __syncthreads();
    staged([&](float& b, size_t o) { out[o] = b; });
}

size_t scan_smem_bytes(int r1, int r2) {
    const int R = r1 + r2;
    return size_t((kTH + 2 * R) + (kTH + 2 * r2)) * size_t(3 * (kTW + 2 * R)) * sizeof(float);
}

// f(R1, R2) with the radii known when compiled where they are common (-1: read from the arguments): the unsharp
// mask's 2 px at the full tier and 1 px on the smaller ones, no lens blur, or the 5 px of a 1.5 px one. The last
// step's unsharp sum is what a radius read at run time slows down (4K, no lens blur: 0.113 ms against 0.158).
template <class F>
void with_scan_radii(int r1, int r2, F&& f) {
    const auto lens = [&](auto c2) {
        if (r1 == 0) f(std::integral_constant<int, 0>(), c2);
        else if (r1 == 5) f(std::integral_constant<int, 5>(), c2);
        else f(std::integral_constant<int, -1>(), c2);
    };
    if (r2 == 1) lens(std::integral_constant<int, 1>());
    else if (r2 == 2) lens(std::integral_constant<int, 2>());
    else f(std::integral_constant<int, -1>(), std::integral_constant<int, -1>());
}

template <int R1, int R2>
void launch_scan(const float* rgb, uint16_t* out, uint32_t w, uint32_t h, uint32_t row0, uint32_t row1,
                 const ScanArgs& a, cudaStream_t s) {
    const size_t smem = scan_smem_bytes(a.r1, a.r2);  // at most 96 KB (r1 = r2 = 9)
    ensure_smem(reinterpret_cast<const void*>(k_scan_encode<R1, R2>), int(smem));
    const dim3 g((w + kTW - 1) / kTW, (row1 - row0 + kTH - 1) / kTH);
    k_scan_encode<R1, R2><<<g, kThreads, smem, s>>>(rgb, out, int(w), int(h), int(row0), a);
}

}  // namespace

bool scan_encode_fits(uint32_t w, uint32_t h, int r1, int r2) {
    const int R = r1 + r2;
    return r1 >= 0 && r2 >= 0 && r1 <= SPKB_FIR_MAX_R && r2 <= SPKB_FIR_MAX_R && w >= uint32_t(R) + 1 &&
           h >= uint32_t(R) + 1 && (uint64_t(h) + kTH - 1) / kTH <= 65535u;
}

void scan_encode_rows(const float* rgb, uint16_t* out, uint32_t w, uint32_t h, uint32_t row0, uint32_t row1,
                      const ScanArgs& a, cudaStream_t s) {
    if (uint64_t(w) * h == 0 || row1 <= row0) return;
    Probe p("scan_encode", s);
    with_scan_radii(a.r1, a.r2, [&](auto r1, auto r2) {
        launch_scan<decltype(r1)::value, decltype(r2)::value>(rgb, out, w, h, row0, row1, a, s);
    });
}

void scan_encode(const float* rgb, uint16_t* out, uint32_t w, uint32_t h, const ScanArgs& a, cudaStream_t s) {
    scan_encode_rows(rgb, out, w, h, 0, h, a, s);
}

namespace {
template <int R1, int R2>
void launch_scan_batch(const BatchScanFrame* frames, uint32_t n_frames, uint32_t n_tiles, uint32_t ctas, size_t smem,
                       cudaStream_t s) {
    ensure_smem(reinterpret_cast<const void*>(k_scan_encode_batch<R1, R2>), int(smem));
    k_scan_encode_batch<R1, R2><<<ctas, kThreads, smem, s>>>(frames, n_frames, n_tiles);
}
}  // namespace

void scan_prepare() {
    const int max_smem = int(scan_smem_bytes(SPKB_FIR_MAX_R, SPKB_FIR_MAX_R));
    const auto set = [&](auto r1, auto r2) {
        ensure_smem(reinterpret_cast<const void*>(k_scan_encode<decltype(r1)::value, decltype(r2)::value>), max_smem);
        ensure_smem(reinterpret_cast<const void*>(k_scan_encode_batch<decltype(r1)::value, decltype(r2)::value>), max_smem);
    };
    for (int r1 : {0, 1, 5})
        for (int r2 : {1, 2, 3}) with_scan_radii(r1, r2, set);
}

uint32_t scan_tiles(uint32_t w, uint32_t h) { return ((w + kTW - 1) / kTW) * ((h + kTH - 1) / kTH); }
uint32_t scan_tiles_x(uint32_t w) { return (w + kTW - 1) / kTW; }

void scan_encode_batch(const BatchScanFrame* frames, uint32_t n_frames, uint32_t n_tiles, int r1, int r2,
                       uint32_t ctas, cudaStream_t s) {
    if (n_tiles == 0) return;
    Probe p("scan_encode_batch", s);
    const size_t smem = r1 >= 0 && r2 >= 0 ? scan_smem_bytes(r1, r2) : scan_smem_bytes(SPKB_FIR_MAX_R, SPKB_FIR_MAX_R);
    with_scan_radii(r1, r2, [&](auto c1, auto c2) {
        launch_scan_batch<decltype(c1)::value, decltype(c2)::value>(frames, n_frames, n_tiles, ctas, smem, s);
    });
}

namespace {
template <int R>
void launch_fir_tile(const float* in, float* out, uint32_t w, uint32_t h, uint32_t row0, uint32_t row1, const ScanArgs& a,
                     cudaStream_t s) {
    const size_t smem = size_t(2 * kTH + 2 * a.r1) * size_t(3 * (kTW + 2 * a.r1)) * sizeof(float);
    ensure_smem(reinterpret_cast<const void*>(k_fir_tile<R>), int(smem));
    const dim3 g((w + kTW - 1) / kTW, (row1 - row0 + kTH - 1) / kTH);
    k_fir_tile<R><<<g, kThreads, smem, s>>>(in, out, int(w), int(h), int(row0), a);
}
}  // namespace

bool fir_tile_fits(uint32_t w, uint32_t h, int r) { return scan_encode_fits(w, h, r, 0); }

void fir_tile(const float* in, float* out, uint32_t w, uint32_t h, int r, const float* taps, cudaStream_t s) {
    fir_tile_rows(in, out, w, h, 0, h, r, taps, s);
}

void fir_tile_rows(const float* in, float* out, uint32_t w, uint32_t h, uint32_t row0, uint32_t row1, int r,
                   const float* taps, cudaStream_t s) {
    static_assert(kFirTileRows == uint32_t(kTH), "a row range starts at a tile");
    if (uint64_t(w) * (row1 - row0) == 0) return;
    ScanArgs a{};
    a.r1 = r;
    for (int k = 0; k <= 2 * r; ++k) a.t1[k] = taps[k];
    Probe p("fir_tile", s);
    if (r == 2) launch_fir_tile<2>(in, out, w, h, row0, row1, a, s);
    else if (r == 5) launch_fir_tile<5>(in, out, w, h, row0, row1, a, s);
    else launch_fir_tile<-1>(in, out, w, h, row0, row1, a, s);
}

void fir_mixture(const float* in, float* out, const float* acc, uint32_t w, uint32_t h, const FirMixArgs& a,
                 cudaStream_t s) {
    if (uint64_t(w) * h == 0) return;
    const int rm = a.rmax;
    const size_t smem = (size_t(kTH + 2 * rm) * size_t(3 * (kTW + 2 * rm)) + size_t(kTH) * mix_pitch(rm) +
                         3 * (2 * SPKB_FIR_MAX_R + 1)) * sizeof(float);
    ensure_smem(reinterpret_cast<const void*>(k_fir_mixture), int(smem));
    Probe p("fir_mixture", s);
    const dim3 g((w + kTW - 1) / kTW, (h + kTH - 1) / kTH);
    k_fir_mixture<<<g, kMixThreads, smem, s>>>(in, out, acc, int(w), int(h), a);
}

}  // namespace spkb::dev
