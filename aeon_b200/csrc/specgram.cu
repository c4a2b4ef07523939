// Log-mel spectrogram kernel for sm_100a: framing + window + real DFT magnitude + mel filter
// bank + natural log, one launch per batch of clips.
//
// Follows aeon's specgram::wav_to_specgram and specgram_to_cepsgram (src/specgram.cpp:26-137):
//   frames = (n - L)/S + 1 (capped), sample -> float, * window, length-L DFT, bins 0..L/2,
//   magnitude; then (mag*mag / (2*(L/2))) x filter bank, natural log.  Rows past the last
//   frame of a clip are written as zeros.
//
// One warp owns one frame and never leaves registers for the transform itself: the L real
// samples are packed into L/2 complex values, L/2 = R*32, lane n holds the R values
// z[32*r + n].  An R-point DFT runs in registers, the results are twiddled, and R independent
// 32-point transforms run ACROSS the warp with shuffle butterflies.  The packed spectrum is
// unfolded into the L/2+1 real-signal bins through a small per-warp shared-memory buffer,
// which also feeds the sparse triangular mel filters (at most two filters touch a bin).
#include <cuda_runtime.h>
#include <math_constants.h>
#include <stdint.h>

#include "../../include/aeon_b200.h"

namespace aeonb
{
    namespace
    {
        constexpr int SPEC_WARPS   = 8;
        constexpr int SPEC_THREADS = SPEC_WARPS * 32;
        constexpr int SPEC_MAX_R   = 10;

        struct spec_launch
        {
            const aeonb_specgram_desc* descs;
            aeonb_specgram_config      cfg;
            const float*               window;    // L floats, or nullptr
            const float2*              twiddle;   // L/2 entries of exp(-2*pi*i*k/(L/2)) followed by L/2+1 of exp(-2*pi*i*k/L)
            const int*                 filt_start; // num_filters+1 offsets into filt_weight
            const int*                 filt_bin;   // first bin of every filter
            const float*               filt_weight;
            const float*               dct;       // num_cepstra x dct_n cosine table with the orthonormal scale, or nullptr
            int                        dct_n;     // num_filters rounded up to even
            int                        n_out;     // floats per output row
        };

        __device__ __forceinline__ float2 cmul(float2 a, float2 b)
        {
            return make_float2(a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x);
        }

        // Power row -> sparse mel filters -> log [-> first num_cepstra rows of the orthonormal DCT-II].  `cep` is scratch for
        // the log-mel vector when a DCT follows (num_filters floats, may not alias `power`).
        __device__ __forceinline__ void finish_mel(const spec_launch& P, const float* power, float* cep, float* out, int lane)
        {
            for (int j = lane; j < P.cfg.num_filters; j += 32)
            {
                float acc = 0.f;
                // the bins of a filter follow one another; its weights lie at filt_start[j]
                const int    begin = __ldg(P.filt_start + j), n = __ldg(P.filt_start + j + 1) - begin;
                const float* in = power + __ldg(P.filt_bin + j);
                const float* w  = P.filt_weight + begin;
#pragma unroll 4
                for (int i = 0; i < n; ++i)
                    acc += in[i] * __ldg(w + i);
                if (P.dct)
                    cep[j] = logf(acc);
                else
                    out[j] = logf(acc);
            }
            if (!P.dct)
                return;
            __syncwarp();
            for (int j = lane; j < P.cfg.num_cepstra; j += 32)
            {
                const float* row = P.dct + (size_t)j * P.dct_n;
                float        acc = 0.f;
                for (int k = 0; k < P.cfg.num_filters; ++k)
                    acc += cep[k] * __ldg(row + k);
                out[j] = acc;
            }
        }

        template <int R>
        __global__ void __launch_bounds__(SPEC_THREADS) specgram_kernel(const spec_launch P)
        {
            constexpr int H = R * 32; // complex transform length
            constexpr int L = 2 * H;  // frame length
            __shared__ float2 zbuf[SPEC_WARPS][H + 1];
            __shared__ float  pbuf[SPEC_WARPS][H + 1];

            const int lane = threadIdx.x & 31;
            const int warp = threadIdx.x >> 5;
            const aeonb_specgram_desc d = P.descs[blockIdx.y];
            const int frame = blockIdx.x * SPEC_WARPS + warp;
            if (frame >= P.cfg.max_time_steps)
                return;
            float* out = d.dst + (size_t)frame * P.n_out;
            int    frames = d.n_samples >= L ? (d.n_samples - L) / P.cfg.frame_stride + 1 : 0;
            frames        = min(frames, P.cfg.max_time_steps);
            if (frame >= frames)
            {
                for (int j = lane; j < P.n_out; j += 32)
                    out[j] = 0.f;
                return;
            }

            // ---- load + window + pack: z[m] = x[2m] + i*x[2m+1], lane holds m = 32*r + lane
            const int16_t* x = d.samples + (size_t)frame * P.cfg.frame_stride;
            float2         z[R];
#pragma unroll
            for (int r = 0; r < R; ++r)
            {
                const int m = 32 * r + lane;
                float     a = (float)x[2 * m], b = (float)x[2 * m + 1];
                if (P.window)
                {
                    a *= __ldg(P.window + 2 * m);
                    b *= __ldg(P.window + 2 * m + 1);
                }
                z[r] = make_float2(a, b);
            }

            // ---- R-point DFT over r (in registers), then twiddle by W_H^(lane*k1)
            float2 y[R];
#pragma unroll
            for (int k1 = 0; k1 < R; ++k1)
            {
                float2 acc = z[0];
#pragma unroll
                for (int r = 1; r < R; ++r)
                {
                    // W_R^(r*k1) = W_H^(32*r*k1)
                    const float2 w = __ldg(P.twiddle + ((32 * r * k1) % H));
                    const float2 t = cmul(z[r], w);
                    acc.x += t.x;
                    acc.y += t.y;
                }
                y[k1] = cmul(acc, __ldg(P.twiddle + ((lane * k1) % H)));
            }

            // ---- R independent 32-point transforms across the lanes (decimation in frequency)
#pragma unroll
            for (int half = 16; half >= 1; half >>= 1)
            {
                const bool   upper = (lane & half) != 0;
                // twiddle W_(2*half)^(lane mod half) = W_H^((lane mod half) * H/(2*half))
                const float2 w = __ldg(P.twiddle + ((lane & (half - 1)) * (H / (2 * half))));
#pragma unroll
                for (int k1 = 0; k1 < R; ++k1)
                {
                    const float ox = __shfl_xor_sync(0xffffffffu, y[k1].x, half);
                    const float oy = __shfl_xor_sync(0xffffffffu, y[k1].y, half);
                    if (upper)
                        y[k1] = cmul(make_float2(ox - y[k1].x, oy - y[k1].y), w);
                    else
                        y[k1] = make_float2(y[k1].x + ox, y[k1].y + oy);
                }
            }
            // lane now holds Z[k1 + R*k2] with k2 = bit-reversed lane
            const int k2 = __brev((unsigned)lane) >> 27;
#pragma unroll
            for (int k1 = 0; k1 < R; ++k1)
                zbuf[warp][k1 + R * k2] = y[k1];
            __syncwarp();

            // ---- unfold to the real-signal bins 0..H and take the power
            const float2* wl = P.twiddle + H; // exp(-2*pi*i*k/L)
            const float   scale = 1.0f / (float)(2 * H);
            for (int k = lane; k <= H; k += 32)
            {
                const float2 a = zbuf[warp][k == H ? 0 : k];
                const float2 b = zbuf[warp][k == 0 || k == H ? 0 : H - k];
                // even part (a + conj b)/2, odd part (a - conj b)/(2i)
                const float2 ev = make_float2(0.5f * (a.x + b.x), 0.5f * (a.y - b.y));
                const float2 od = make_float2(0.5f * (a.y + b.y), -0.5f * (a.x - b.x));
                const float2 t  = cmul(od, __ldg(wl + k));
                const float  re = ev.x + t.x, im = ev.y + t.y;
                const float  mag = sqrtf(re * re + im * im);
                if (P.cfg.num_filters > 0)
                    pbuf[warp][k] = scale * mag * mag;
                else
                    out[k] = mag;
            }
            if (P.cfg.num_filters <= 0)
                return;
            __syncwarp();

            finish_mel(P, pbuf[warp], reinterpret_cast<float*>(zbuf[warp]), out, lane);
        }

        // Frame lengths L = N1 * N2 with both factors small (400 = 20 * 20, 441 = 21 * 21): sample n = N2*n1 + n2, bin
        // k = k1 + N1*k2.  A block takes F frames.  First the N1-point transforms of the N2 columns, of which real input needs
        // only k1 <= N1/2; then, turned by exp(-2*pi*i*n2*k1/L), the N2-point transforms of those rows, whose bins above L/2 are
        // the conjugates of the ones below that the missing rows would give.  Samples n and N-n of a transform share a cosine
        // and, up to the sign, a sine, and so do bins k and N-k: sums and differences of sample pairs are taken first, each
        // thread works out four bins (and their mirrors) at a time, and a table entry serves a whole warp or most of it.
        // About 13 thousand multiply-adds for 400 samples, against 161 thousand of the direct sum below.  Bound by the
        // issue of those and of the shared-memory reads; 32 clips of up to 16 s with 400-sample frames, 40 filters and 13 cepstra
        // (27 thousand frames): 0.10 ms, the direct sum 1.76 ms.  Lengths 64*R stay with the kernel above: 0.095 ms for 64 clips
        // with 320-sample frames, 0.140 ms with this one.
        constexpr int SPLIT_THREADS = 256;
        struct split_plan
        {
            int           n1, n2, frames; // frames of a block
            const float2* c1;             // (cos, sin)(2*pi*k*n/N1), k = 0..N1/2, n = 1..(N1-1)/2
            const float2* c2;             // the same for N2
        };
        __host__ __device__ inline int split_terms(int n) { return (n / 2 + 1) * ((n - 1) / 2); }
        __global__ void __launch_bounds__(SPLIT_THREADS) specgram_split_kernel(const spec_launch P, const split_plan S)
        {
            extern __shared__ __align__(16) float2 ssm[];
            const int L = P.cfg.frame_length, H = L / 2, F = S.frames; // bins 0..H
            const int N1 = S.n1, N2 = S.n2, K1 = N1 / 2 + 1, M1 = (N1 - 1) / 2, K2 = N2 / 2 + 1, M2 = (N2 - 1) / 2;
            const int row_stride = N2 | 1; // odd: rows start in different banks
            float2*   c1 = ssm;
            float2*   c2 = c1 + split_terms(N1);
            float2*   y  = c2 + split_terms(N2);                               // F x K1 rows of N2 values
            float*    xs = reinterpret_cast<float*>(y + F * K1 * row_stride);  // F x L windowed samples, then F x (H + 1) bins
            const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
            const aeonb_specgram_desc d = P.descs[blockIdx.y];
            const int first = blockIdx.x * F;
            int       frames = d.n_samples >= L ? (d.n_samples - L) / P.cfg.frame_stride + 1 : 0;
            frames           = min(frames, P.cfg.max_time_steps);
            float* out       = d.dst + (size_t)first * P.n_out;
            const int here = min(F, P.cfg.max_time_steps - first), live = max(0, min(here, frames - first));
            for (int i = live * P.n_out + tid; i < here * P.n_out; i += SPLIT_THREADS)
                out[i] = 0.f;
            if (live == 0)
                return;

            for (int i = tid; i < split_terms(N1) + split_terms(N2); i += SPLIT_THREADS)
                c1[i] = i < split_terms(N1) ? __ldg(S.c1 + i) : __ldg(S.c2 + i - split_terms(N1));
            for (int f = warp; f < live; f += SPLIT_THREADS / 32)
            {
                const int16_t* x = d.samples + (size_t)(first + f) * P.cfg.frame_stride;
                for (int n = lane; n < L; n += 32)
                    xs[f * L + n] = (float)x[n] * (P.window ? __ldg(P.window + n) : 1.f);
            }
            __syncthreads();

            // ---- columns: k = 4*group .. 4*group + 3 of column n2 of frame f
            const int cols = live * N2;
            for (int it = tid; it < (K1 + 3) / 4 * cols; it += SPLIT_THREADS)
            {
                const int    k = it / cols * 4, col = it % cols, f = col / N2, n2 = col - f * N2;
                const float* x    = xs + f * L + n2;
                const float  half = N1 & 1 ? 0.f : x[N1 / 2 * N2]; // sample N1/2 turns by half a circle for odd k
                float        p[4], q[4] = {0.f, 0.f, 0.f, 0.f};
                const float2* c[4];
#pragma unroll
                for (int j = 0; j < 4; ++j)
                {
                    p[j] = x[0] + (j & 1 ? -half : half);
                    c[j] = c1 + min(k + j, K1 - 1) * M1;
                }
                for (int n = 0; n < M1; ++n)
                {
                    const float a = x[(n + 1) * N2], b = x[(N1 - 1 - n) * N2], sum = a + b, dif = a - b;
#pragma unroll
                    for (int j = 0; j < 4; ++j)
                    {
                        const float2 t = c[j][n];
                        p[j]           = __fmaf_rn(sum, t.x, p[j]);
                        q[j]           = __fmaf_rn(dif, t.y, q[j]);
                    }
                }
                float2* row = y + (f * K1 + k) * row_stride + n2;
#pragma unroll
                for (int j = 0; j < 4; ++j)
                    if (k + j < K1)
                    {
                        const float2 w      = __ldg(P.twiddle + n2 * (k + j)); // exp(-2*pi*i*n2*k1/L)
                        row[j * row_stride] = make_float2(__fmaf_rn(p[j], w.x, q[j] * w.y), __fmaf_rn(p[j], w.y, -(q[j] * w.x)));
                    }
            }
            __syncthreads();

            // ---- rows: k2 = 4*group .. 4*group + 3 and N2 - k2 of row k1 of frame f
            const float scale = 1.0f / (float)(2 * H);
            const int   rows  = live * K1;
            float*      bins  = xs;
            for (int it = tid; it < (K2 + 3) / 4 * rows; it += SPLIT_THREADS)
            {
                const int     k = it / rows * 4, row = it % rows, f = row / K1, k1 = row - f * K1;
                const float2* z    = y + row * row_stride;
                const float2  half = N2 & 1 ? make_float2(0.f, 0.f) : z[N2 / 2];
                float2        p[4], q[4];
                const float2* c[4];
#pragma unroll
                for (int j = 0; j < 4; ++j)
                {
                    p[j] = make_float2(z[0].x + (j & 1 ? -half.x : half.x), z[0].y + (j & 1 ? -half.y : half.y));
                    q[j] = make_float2(0.f, 0.f);
                    c[j] = c2 + min(k + j, K2 - 1) * M2;
                }
                for (int n = 0; n < M2; ++n)
                {
                    const float2 a = z[n + 1], b = z[N2 - 1 - n];
                    const float2 sum = make_float2(a.x + b.x, a.y + b.y), dif = make_float2(a.x - b.x, a.y - b.y);
#pragma unroll
                    for (int j = 0; j < 4; ++j)
                    {
                        const float2 t = c[j][n];
                        p[j].x         = __fmaf_rn(sum.x, t.x, p[j].x);
                        p[j].y         = __fmaf_rn(sum.y, t.x, p[j].y);
                        q[j].x         = __fmaf_rn(dif.x, t.y, q[j].x);
                        q[j].y         = __fmaf_rn(dif.y, t.y, q[j].y);
                    }
                }
                auto put = [&](int k2, float re, float im) {
                    int bin = k1 + N1 * k2;
                    if (bin > H)
                    {
                        if (k1 == 0 || 2 * k1 == N1)
                            return; // such a row holds its own conjugates
                        bin = L - bin;
                    }
                    const float mag         = sqrtf(__fmaf_rn(re, re, im * im));
                    bins[f * (H + 1) + bin] = P.cfg.num_filters > 0 ? scale * mag * mag : mag;
                };
#pragma unroll
                for (int j = 0; j < 4; ++j)
                    if (k + j < K2)
                    {
                        put(k + j, p[j].x + q[j].y, p[j].y - q[j].x);
                        if (k + j > 0 && 2 * (k + j) != N2)
                            put(N2 - k - j, p[j].x - q[j].y, p[j].y + q[j].x);
                    }
            }
            __syncthreads();
            if (P.cfg.num_filters <= 0)
            {
                for (int i = tid; i < live * (H + 1); i += SPLIT_THREADS)
                    out[i] = bins[i];
                return;
            }
            for (int f = warp; f < live; f += SPLIT_THREADS / 32)
            {
                finish_mel(P, bins + f * (H + 1), reinterpret_cast<float*>(y) + f * P.cfg.num_filters, out + (size_t)f * P.n_out, lane);
                __syncwarp();
            }
        }

        // Any other frame length (a large prime factor): one warp per frame, lanes take the bins, each bin a direct sum over the
        // frame with the twiddles from a table of L entries (index k*n mod L kept by addition).
        constexpr int SPEC_GENERIC_WARPS = 4;
        __global__ void __launch_bounds__(SPEC_GENERIC_WARPS * 32) specgram_generic_kernel(const spec_launch P)
        {
            extern __shared__ float gsm[];
            const int L = P.cfg.frame_length, H = L / 2; // bins 0..H
            float*    xs   = gsm + (size_t)(threadIdx.x >> 5) * (L + H + 1); // this warp's windowed samples, then its power row
            float*    pw   = xs + L;
            const int lane = threadIdx.x & 31;
            const aeonb_specgram_desc d = P.descs[blockIdx.y];
            const int frame = blockIdx.x * SPEC_GENERIC_WARPS + (threadIdx.x >> 5);
            if (frame >= P.cfg.max_time_steps)
                return;
            float* out = d.dst + (size_t)frame * P.n_out;
            int    frames = d.n_samples >= L ? (d.n_samples - L) / P.cfg.frame_stride + 1 : 0;
            frames        = min(frames, P.cfg.max_time_steps);
            if (frame >= frames)
            {
                for (int j = lane; j < P.n_out; j += 32)
                    out[j] = 0.f;
                return;
            }
            const int16_t* x = d.samples + (size_t)frame * P.cfg.frame_stride;
            for (int n = lane; n < L; n += 32)
                xs[n] = (float)x[n] * (P.window ? __ldg(P.window + n) : 1.f);
            __syncwarp();
            const float scale = 1.0f / (float)(2 * H);
            for (int k = lane; k <= H; k += 32)
            {
                float re = 0.f, im = 0.f;
                int   idx = 0; // k*n mod L
                for (int n = 0; n < L; ++n)
                {
                    const float2 w = __ldg(P.twiddle + idx); // exp(-2*pi*i*idx/L)
                    re += xs[n] * w.x;
                    im += xs[n] * w.y;
                    idx += k;
                    if (idx >= L)
                        idx -= L;
                }
                const float mag = sqrtf(re * re + im * im);
                if (P.cfg.num_filters > 0)
                    pw[k] = scale * mag * mag;
                else
                    out[k] = mag;
            }
            if (P.cfg.num_filters <= 0)
                return;
            __syncwarp();
            finish_mel(P, pw, xs, out, lane);
        }

        template <int R>
        cudaError_t launch_r(const spec_launch& P, int n, cudaStream_t stream)
        {
            dim3 grid((P.cfg.max_time_steps + SPEC_WARPS - 1) / SPEC_WARPS, n, 1);
            specgram_kernel<R><<<grid, SPEC_THREADS, 0, stream>>>(P);
            return cudaGetLastError();
        }
    }

    bool specgram_frame_length_supported(int frame_length)
    {
        const int r = frame_length / 64;
        return frame_length >= 64 && frame_length % 64 == 0 && r <= SPEC_MAX_R && r != 7 && r != 9;
    }

    cudaError_t launch_specgram(const aeonb_specgram_desc* descs_dev, int n, const aeonb_specgram_config& cfg,
                                const float* window_dev, const float2* twiddle_dev, const int* filt_start_dev,
                                const int* filt_bin_dev, const float* filt_weight_dev, const float* dct_dev, int dct_n, int n_out,
                                cudaStream_t stream)
    {
        spec_launch P{descs_dev, cfg, window_dev, twiddle_dev, filt_start_dev, filt_bin_dev, filt_weight_dev, dct_dev, dct_n, n_out};
        switch (cfg.frame_length / 64)
        {
        case 1: return launch_r<1>(P, n, stream);
        case 2: return launch_r<2>(P, n, stream);
        case 3: return launch_r<3>(P, n, stream);
        case 4: return launch_r<4>(P, n, stream);
        case 5: return launch_r<5>(P, n, stream);
        case 6: return launch_r<6>(P, n, stream);
        case 8: return launch_r<8>(P, n, stream);
        case 10: return launch_r<10>(P, n, stream);
        default: return cudaErrorInvalidValue;
        }
    }

    // Shared memory of a block of the split kernel with `frames` frames.
    static size_t split_smem(int n1, int n2, int frames)
    {
        return sizeof(float2) * (split_terms(n1) + split_terms(n2) + (size_t)frames * (n1 / 2 + 1) * (n2 | 1)) + sizeof(float) * (size_t)frames * n1 * n2;
    }

    // The factors with the fewest multiply-adds whose tables (16 KB at most) fit, and as many frames per block, up to one for each
    // warp, as leave room for two blocks on an SM.  False: no such factors.
    bool specgram_split(int frame_length, int& n1, int& n2, int& frames)
    {
        double best = 0;
        for (int a = 1; a <= frame_length; ++a)
        {
            if (frame_length % a)
                continue;
            const int b = frame_length / a;
            if (a > 128 || b > 128 || sizeof(float2) * (split_terms(a) + split_terms(b)) > 16384 || split_smem(a, b, 1) > 200 * 1024)
                continue;
            const double cost = 2.0 * b * split_terms(a) + 4.0 * (a / 2 + 1) * split_terms(b);
            if (best == 0 || cost < best)
                best = cost, n1 = a, n2 = b;
        }
        if (best == 0)
            return false;
        frames = SPLIT_THREADS / 32;
        while (frames > 1 && split_smem(n1, n2, frames) > 100 * 1024)
            frames /= 2;
        return true;
    }

    cudaError_t launch_specgram_split(const aeonb_specgram_desc* descs_dev, int n, const aeonb_specgram_config& cfg, const float* window_dev,
                                      const float2* twiddle_dev, const float2* c1_dev, const float2* c2_dev, int n1, int n2, int frames,
                                      const int* filt_start_dev, const int* filt_bin_dev, const float* filt_weight_dev, const float* dct_dev,
                                      int dct_n, int n_out, cudaStream_t stream)
    {
        spec_launch      P{descs_dev, cfg, window_dev, twiddle_dev, filt_start_dev, filt_bin_dev, filt_weight_dev, dct_dev, dct_n, n_out};
        const split_plan S{n1, n2, frames, c1_dev, c2_dev};
        const size_t     smem = split_smem(n1, n2, frames);
        // the most any frame length takes, so that threads with other lengths do not lower it between this call and the launch
        cudaError_t      err  = cudaFuncSetAttribute(specgram_split_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, 216 * 1024);
        if (err != cudaSuccess)
            return err;
        dim3 grid((cfg.max_time_steps + frames - 1) / frames, n, 1);
        specgram_split_kernel<<<grid, SPLIT_THREADS, smem, stream>>>(P, S);
        return cudaGetLastError();
    }

    size_t specgram_generic_smem(int frame_length) { return (size_t)SPEC_GENERIC_WARPS * (frame_length + frame_length / 2 + 1) * sizeof(float); }

    // Frame lengths the shuffle-FFT kernel does not take: `twiddle_dev` then holds frame_length entries exp(-2*pi*i*k/L).
    cudaError_t launch_specgram_generic(const aeonb_specgram_desc* descs_dev, int n, const aeonb_specgram_config& cfg,
                                        const float* window_dev, const float2* twiddle_dev, const int* filt_start_dev,
                                        const int* filt_bin_dev, const float* filt_weight_dev, const float* dct_dev, int dct_n,
                                        int n_out, cudaStream_t stream)
    {
        spec_launch  P{descs_dev, cfg, window_dev, twiddle_dev, filt_start_dev, filt_bin_dev, filt_weight_dev, dct_dev, dct_n, n_out};
        const size_t smem = specgram_generic_smem(cfg.frame_length);
        // the most specgram_tables lets through, for the same reason as above
        cudaError_t  err  = cudaFuncSetAttribute(specgram_generic_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, 200 * 1024);
        if (err != cudaSuccess)
            return err;
        dim3 grid((cfg.max_time_steps + SPEC_GENERIC_WARPS - 1) / SPEC_GENERIC_WARPS, n, 1);
        specgram_generic_kernel<<<grid, SPEC_GENERIC_WARPS * 32, smem, stream>>>(P);
        return cudaGetLastError();
    }
}
