// Whole-picture pre-passes of the image path for sm_100a.
//
// orient_kernel: the EXIF orientation turn cv::imdecode applies after decoding (a pure permutation of pixels).
//
// rotate_pixels_kernel, rotate_tiles_kernel: aeon's image::rotate (src/image.cpp:53-75), i.e.
// cv::warpAffine(src, dst, getRotationMatrix2D(centre, angle, 1), src.size(), INTER_LINEAR, BORDER_CONSTANT, 0)
// on 8-bit interleaved pictures, bit for bit; and its INTER_NEAREST form (interpolate == false), which the
// pixelmask and depthmap transformers use (src/etl_pixel_mask.cpp:71-73): the same fixed-point source coordinates
// rounded to the nearest whole pixel.
//
// OpenCV maps every destination pixel back through the inverted matrix in 10-bit fixed point -- the products are
// formed in float64 and rounded half to even per column (M0*x*1024, M3*x*1024) and per row ((M1*y+M2)*1024,
// (M4*y+M5)*1024) -- keeps 5 fractional bits, and blends the four neighbours with integer weights
// (32-fx)(32-fy)*32 ... that sum to 2^15; neighbours outside the picture count as zero.  The kernels do exactly
// that per destination pixel: the float64 products with explicit round-to-nearest multiplies (no contraction),
// __double2int_rn for the rounding, then integer arithmetic.  HBM traffic is one read of the source (neighbouring
// threads share their taps through L1/L2) and one write of the destination.
#include <cuda_runtime.h>
#include <stdint.h>

#include <cmath>
#include <sstream>
#include <vector>

#include "context.hpp"

namespace aeonb
{
    namespace
    {
        struct rotate_job
        {
            const uint8_t* src;
            uint8_t*       dst;
            int32_t        src_pitch, src_stride, dst_pitch, dst_stride, width, height;
            int32_t        nearest; // INTER_NEAREST instead of INTER_LINEAR
            double         m[6]; // inverse map: source = m * (x, y, 1)
        };

        // The bytes of pixel `x` of a row and, with `two`, of the one behind it, from the bottom of v[0] on: cut out of aligned words
        // that hold a byte of them (loads of single bytes: 16 pictures of 437 x 437 35 us, 31 so, a thread per pixel in both).
        __device__ __forceinline__ void source_bytes(const rotate_job& J, const uint8_t* row, int x, bool two, uint32_t (&v)[2])
        {
            const uint8_t*  p     = row + (size_t)x * J.src_stride;
            const uint32_t  lead  = (uint32_t)((uintptr_t)p & 3);
            const uint32_t* word  = reinterpret_cast<const uint32_t*>(p - lead);
            const int       bytes = (int)lead + (two ? J.src_stride : 0) + 3; // a word is loaded only if one of them lies in it
            const uint32_t  w0 = __ldg(word), w1 = bytes > 4 ? __ldg(word + 1) : 0, w2 = bytes > 8 ? __ldg(word + 2) : 0;
            v[0] = __funnelshift_r(w0, w1, 8 * lead);
            v[1] = __funnelshift_r(w1, w2, 8 * lead);
        }

        // The destination pixel at the fixed-point source coordinates (fx, fy), B in the lowest byte.
        __device__ __forceinline__ uint32_t rotated_pixel(const rotate_job& J, int fx, int fy)
        {
            uint32_t v[2];
            if (J.nearest)
            {
                // the source pixel the fixed-point coordinate rounds to, zero outside the picture
                const int nx = max(-32768, min(32767, fx >> 10)), ny = max(-32768, min(32767, fy >> 10));
                if (nx < 0 || nx >= J.width || ny < 0 || ny >= J.height)
                    return 0;
                source_bytes(J, J.src + (size_t)ny * J.src_pitch, nx, false, v);
                return v[0] & 0xFFFFFF;
            }
            const int X = fx >> 5, Y = fy >> 5;
            const int sx = max(-32768, min(32767, X >> 5)), sy = max(-32768, min(32767, Y >> 5)); // saturate_cast<short>
            const uint32_t ax = (uint32_t)X & 31, ay = (uint32_t)Y & 31;
            // weights of the two rows, a pixel each in the upper and the lower half
            uint32_t   upper = (32 - ax) * (32 - ay) * 32 | ax * (32 - ay) * 32 << 16, lower = (32 - ax) * ay * 32 | ax * ay * 32 << 16;
            const bool in_x0 = sx >= 0 && sx < J.width, in_x1 = sx + 1 >= 0 && sx + 1 < J.width;
            const bool in_y0 = sy >= 0 && sy < J.height, in_y1 = sy + 1 >= 0 && sy + 1 < J.height;
            uint32_t   low[2] = {0, 0};
            v[0] = v[1] = 0;
            if (in_x0 && in_x1)
            {
                if (in_y0)
                    source_bytes(J, J.src + (size_t)sy * J.src_pitch, sx, true, v);
                if (in_y1)
                    source_bytes(J, J.src + (size_t)(sy + 1) * J.src_pitch, sx, true, low);
            }
            else if (in_x0 || in_x1) // one column of the two: it takes the place of the first one, with its own weight
            {
                if (in_y0)
                    source_bytes(J, J.src + (size_t)sy * J.src_pitch, in_x0 ? sx : sx + 1, false, v);
                if (in_y1)
                    source_bytes(J, J.src + (size_t)(sy + 1) * J.src_pitch, in_x0 ? sx : sx + 1, false, low);
                upper = in_x0 ? upper & 0xFFFF : upper >> 16;
                lower = in_x0 ? lower & 0xFFFF : lower >> 16;
            }
            uint32_t pixel = 0;
#pragma unroll
            for (uint32_t c = 0; c < 3; ++c)
            {
                const uint32_t pair = c | ((uint32_t)J.src_stride + c) << 4; // the channel's bytes of the two pixels
                uint32_t       sum  = __dp2a_lo(upper, __byte_perm(v[0], v[1], pair), 1u << 14);
                sum                 = __dp2a_lo(lower, __byte_perm(low[0], low[1], pair), sum);
                pixel |= (sum >> 15 & 255) << (8 * c);
            }
            return pixel;
        }

        // The parts of a fixed-point source coordinate that depend on the column and on the row (the rounding included).
        __device__ __forceinline__ int2 column_part(const rotate_job& J, int x)
        {
            return make_int2(__double2int_rn(__dmul_rn(__dmul_rn(J.m[0], (double)x), 1024.0)), __double2int_rn(__dmul_rn(__dmul_rn(J.m[3], (double)x), 1024.0)));
        }
        __device__ __forceinline__ int2 row_part(const rotate_job& J, int y)
        {
            const int round = J.nearest ? 512 : 16; // half of the last kept bit: 10 bits dropped, or 5
            return make_int2(__double2int_rn(__dmul_rn(__dadd_rn(__dmul_rn(J.m[1], (double)y), J.m[2]), 1024.0)) + round,
                             __double2int_rn(__dmul_rn(__dadd_rn(__dmul_rn(J.m[4], (double)y), J.m[5]), 1024.0)) + round);
        }
        __device__ __forceinline__ void store_pixel(uint8_t* p, uint32_t v) { p[0] = (uint8_t)v, p[1] = (uint8_t)(v >> 8), p[2] = (uint8_t)(v >> 16); }

        // Few pixels, narrow pictures, destinations with four bytes per pixel: a thread per pixel, as many blocks as the pixels fill.
        __global__ void __launch_bounds__(256) rotate_pixels_kernel(const rotate_job* __restrict__ jobs)
        {
            const rotate_job J      = jobs[blockIdx.y];
            const int        pixels = J.width * J.height;
            for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < pixels; i += gridDim.x * blockDim.x)
            {
                const int  y = i / J.width, x = i - y * J.width;
                const int2 column = column_part(J, x), line = row_part(J, y);
                store_pixel(J.dst + (size_t)y * J.dst_pitch + (size_t)x * J.dst_stride, rotated_pixel(J, line.x + column.x, line.y + column.y));
            }
        }

        // Many pixels: a block takes tiles of ROT_COLS x ROT_ROWS destination pixels.  What depends on the column or the row alone -- the
        // float64 products -- is worked out once per tile; a thread makes four neighbouring pixels, which leave as three words (the
        // destination's rows start on words, three bytes per pixel).  Bound by the issue of integer instructions: 16 pictures and 16 masks
        // of about 437 x 437 take 38 us (tiles of 16 rows 41, of four 39).
        constexpr int ROT_COLS = 512, ROT_ROWS = 8;
        __global__ void __launch_bounds__(256) rotate_tiles_kernel(const rotate_job* __restrict__ jobs)
        {
            __shared__ int2  column[ROT_COLS], line[ROT_ROWS];
            const rotate_job J       = jobs[blockIdx.y];
            const int        tiles_x = (J.width + ROT_COLS - 1) / ROT_COLS, tiles = tiles_x * ((J.height + ROT_ROWS - 1) / ROT_ROWS);
            for (int tile = blockIdx.x; tile < tiles; tile += gridDim.x)
            {
                const int x_first = tile % tiles_x * ROT_COLS, y_first = tile / tiles_x * ROT_ROWS;
                const int cols = min(ROT_COLS, J.width - x_first), rows = min(ROT_ROWS, J.height - y_first);
                __syncthreads(); // the tile before has been used
                for (int i = threadIdx.x; i < cols + rows; i += blockDim.x)
                {
                    if (i < cols)
                        column[i] = column_part(J, x_first + i);
                    else
                        line[i - cols] = row_part(J, y_first + i - cols);
                }
                __syncthreads();
                const int quads = (cols + 3) / 4;
                for (int i = threadIdx.x; i < quads * rows; i += blockDim.x)
                {
                    const int  r = i / quads, x = 4 * (i - r * quads), n = min(4, cols - x);
                    const int2 from = line[r];
                    uint32_t   px[4];
#pragma unroll
                    for (int k = 0; k < 4; ++k)
                        px[k] = k < n ? rotated_pixel(J, from.x + column[x + (k < n ? k : 0)].x, from.y + column[x + (k < n ? k : 0)].y) : 0;
                    uint8_t* const d = J.dst + (size_t)(y_first + r) * J.dst_pitch + (size_t)(x_first + x) * 3;
                    if (n == 4)
                    {
                        uint32_t* const w = reinterpret_cast<uint32_t*>(d);
                        w[0] = px[0] | px[1] << 24;
                        w[1] = px[1] >> 8 | px[2] << 16;
                        w[2] = px[2] >> 16 | px[3] << 8;
                    }
                    else
#pragma unroll
                        for (int k = 0; k < 4; ++k)
                            if (k < n)
                                store_pixel(d + 3 * k, px[k]);
                }
            }
        }
    }

    namespace
    {
        struct orient_job
        {
            const uint8_t* src;
            uint8_t*       dst;
            int32_t        src_pitch, src_stride, dst_pitch, dst_stride, width, height, orientation;
        };

        // EXIF orientation as OpenCV applies it after decoding: destination pixel (x, y) comes from source column /
        // row as below (w, h: source size; the destination is h wide and w high for the transposed cases 5..8).
        __global__ void __launch_bounds__(256) orient_kernel(const orient_job* __restrict__ jobs)
        {
            const orient_job J  = jobs[blockIdx.y];
            const int        w = J.width, h = J.height;
            const bool       swapped = J.orientation >= 5;
            const int        dw = swapped ? h : w, pixels = w * h;
            for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < pixels; i += gridDim.x * blockDim.x)
            {
                const int y = i / dw, x = i - y * dw;
                int       sc, sr;
                switch (J.orientation)
                {
                case 2: sc = w - 1 - x, sr = y; break;         // mirror
                case 3: sc = w - 1 - x, sr = h - 1 - y; break; // half turn
                case 4: sc = x, sr = h - 1 - y; break;         // flip
                case 5: sc = y, sr = x; break;                 // transpose
                case 6: sc = y, sr = h - 1 - x; break;         // quarter turn clockwise
                case 7: sc = w - 1 - y, sr = h - 1 - x; break; // transverse
                case 8: sc = w - 1 - y, sr = x; break;         // quarter turn counter-clockwise
                default: sc = x, sr = y; break;
                }
                const uint8_t* s = J.src + (size_t)sr * J.src_pitch + (size_t)sc * J.src_stride;
                uint8_t*       d = J.dst + (size_t)y * J.dst_pitch + (size_t)x * J.dst_stride;
                d[0] = s[0];
                d[1] = s[1];
                d[2] = s[2];
            }
        }
    }

    // The inverse of getRotationMatrix2D(Point2i(width/2, height/2), angle, 1.0), with the operation order of
    // cv::getRotationMatrix2D and of cv::warpAffine's own inversion, in float64.
    void rotation_inverse_map(int width, int height, int angle, double m[6])
    {
        const double cx = (double)(float)(width / 2), cy = (double)(float)(height / 2);
        const double a     = angle * (3.1415926535897932384626433832795 / 180.);
        const double alpha = std::cos(a), beta = std::sin(a);
        double       M[6]  = {alpha, beta, (1 - alpha) * cx - beta * cy, -beta, alpha, beta * cx + (1 - alpha) * cy};
        double       D     = M[0] * M[4] - M[1] * M[3];
        D                  = D != 0 ? 1. / D : 0;
        const double A11 = M[4] * D, A22 = M[0] * D;
        M[0] = A11;
        M[1] *= -D;
        M[3] *= -D;
        M[4]            = A22;
        const double b1 = -M[0] * M[2] - M[1] * M[5];
        const double b2 = -M[3] * M[2] - M[4] * M[5];
        M[2]            = b1;
        M[5]            = b2;
        for (int i = 0; i < 6; ++i)
            m[i] = M[i];
    }
}

using namespace aeonb;

extern "C" int aeonb_rotate_batch(aeonb_ctx* ctx, const aeonb_rotate_desc* descs, int n)
{
    return guarded([&]() {
        if (!ctx || (n > 0 && !descs))
            throw std::invalid_argument("aeonb_rotate_batch: NULL argument");
        if (n <= 0)
            return AEONB_OK;
        std::vector<rotate_job> jobs(n);
        int64_t                 most = 0, most_tiles = 0, pixels = 0; // (pixels without interpolation four times)
        bool                    wide = true, words = true;
        for (int i = 0; i < n; ++i)
        {
            const aeonb_rotate_desc& r = descs[i];
            std::ostringstream       ss;
            if (!r.src || !r.dst || r.width <= 0 || r.height <= 0 || r.width > 32767 || r.height > 32767)
                ss << "record " << i << ": NULL picture or size outside 1..32767";
            else if ((r.src_pixel_stride != 3 && r.src_pixel_stride != 4) || (r.dst_pixel_stride != 3 && r.dst_pixel_stride != 4))
                ss << "record " << i << ": pixel strides must be 3 or 4";
            else if (r.src_pitch < r.width * r.src_pixel_stride || r.dst_pitch < r.width * r.dst_pixel_stride)
                ss << "record " << i << ": pitch smaller than a row";
            const std::string msg = ss.str();
            if (!msg.empty())
                throw std::invalid_argument(msg);
            rotate_job& j = jobs[i];
            j.src         = r.src;
            j.dst         = r.dst;
            j.src_pitch   = r.src_pitch;
            j.src_stride  = r.src_pixel_stride;
            j.dst_pitch   = r.dst_pitch;
            j.dst_stride  = r.dst_pixel_stride;
            j.width       = r.width;
            j.height      = r.height;
            j.nearest     = r.nearest != 0;
            rotation_inverse_map(r.width, r.height, r.angle, j.m);
            most       = std::max<int64_t>(most, (int64_t)r.width * r.height);
            most_tiles = std::max<int64_t>(most_tiles, (int64_t)((r.width + ROT_COLS - 1) / ROT_COLS) * ((r.height + ROT_ROWS - 1) / ROT_ROWS));
            pixels += (int64_t)r.width * r.height * (r.nearest ? 4 : 1);
            wide &= r.width >= 128;
            words &= r.dst_pixel_stride == 3 && (((uintptr_t)r.dst | (uintptr_t)r.dst_pitch) & 3) == 0;
        }
        AEONB_CUDA(cudaSetDevice(ctx->device));
        auto*      jdev = static_cast<const rotate_job*>(ctx->upload(jobs.data(), sizeof(rotate_job) * n));
        // A tile is a longer chain of work than a pixel, and tiles narrower than 128 pixels leave threads idle: below about four million
        // pixels, of masks one million, there are too few of them to fill the SMs.  Pixels / tiles: one picture of 437 x 437 8.5 / 14.4 us,
        // 16 of them 30.7 / 32.8, 16 of 512 x 512 39.2 / 36.9, 64 of 437 x 437 102 / 87; four masks of 437 x 437 10.6 / 11.9, eight 14.6 / 12.3;
        // 64 pictures of 30 x 3000 41 / 69.  With destinations of four bytes per pixel, which a tile would store by bytes, 16 pictures
        // of 437 x 437 30.7 / 40.5.
        const bool tiles = words && wide && pixels >= 1 << 22;
        const int  per   = (int)std::min<int64_t>(tiles ? most_tiles : (most + 255) / 256, 148 * 8); // blocks per record
        const dim3 grid((unsigned)std::max(per, 1), (unsigned)n);
        launch_timer timer(ctx, AEONB_KERNEL_OTHER, 0);
        if (tiles)
            rotate_tiles_kernel<<<grid, 256, 0, ctx->stream>>>(jdev);
        else
            rotate_pixels_kernel<<<grid, 256, 0, ctx->stream>>>(jdev);
        cudaError_t e = cudaGetLastError();
        if (e != cudaSuccess)
            throw error(AEONB_ERR_CUDA, cuda_message("rotate kernel launch", e));
        ctx->launches++;
        return AEONB_OK;
    });
}

extern "C" int aeonb_orient_batch(aeonb_ctx* ctx, const aeonb_orient_desc* descs, int n)
{
    return guarded([&]() {
        if (!ctx || (n > 0 && !descs))
            throw std::invalid_argument("aeonb_orient_batch: NULL argument");
        if (n <= 0)
            return AEONB_OK;
        std::vector<orient_job> jobs(n);
        int64_t                 most = 0;
        for (int i = 0; i < n; ++i)
        {
            const aeonb_orient_desc& r = descs[i];
            std::ostringstream       ss;
            const int                dw = r.orientation >= 5 ? r.height : r.width;
            if (!r.src || !r.dst || r.width <= 0 || r.height <= 0 || (int64_t)r.width * r.height > (1ll << 30))
                ss << "record " << i << ": NULL picture or bad size";
            else if (r.orientation < 1 || r.orientation > 8)
                ss << "record " << i << ": orientation must be 1..8";
            else if ((r.src_pixel_stride != 3 && r.src_pixel_stride != 4) || (r.dst_pixel_stride != 3 && r.dst_pixel_stride != 4))
                ss << "record " << i << ": pixel strides must be 3 or 4";
            else if (r.src_pitch < r.width * r.src_pixel_stride || r.dst_pitch < dw * r.dst_pixel_stride)
                ss << "record " << i << ": pitch smaller than a row";
            const std::string msg = ss.str();
            if (!msg.empty())
                throw std::invalid_argument(msg);
            jobs[i] = orient_job{r.src, r.dst, r.src_pitch, r.src_pixel_stride, r.dst_pitch, r.dst_pixel_stride, r.width, r.height, r.orientation};
            most    = std::max<int64_t>(most, (int64_t)r.width * r.height);
        }
        AEONB_CUDA(cudaSetDevice(ctx->device));
        auto*      jdev = static_cast<const orient_job*>(ctx->upload(jobs.data(), sizeof(orient_job) * n));
        const int  per  = (int)std::min<int64_t>((most + 255) / 256, 148 * 8);
        const dim3 grid((unsigned)std::max(per, 1), (unsigned)n);
        launch_timer timer(ctx, AEONB_KERNEL_OTHER, 0);
        orient_kernel<<<grid, 256, 0, ctx->stream>>>(jdev);
        cudaError_t e = cudaGetLastError();
        if (e != cudaSuccess)
            throw error(AEONB_ERR_CUDA, cuda_message("orientation kernel launch", e));
        ctx->launches++;
        return AEONB_OK;
    });
}
