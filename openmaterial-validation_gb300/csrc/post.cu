// Image development on the device and the image writers: the reference's
// host-side tail of a render (main.cpp:505-521), after BDPTRenderer::render.
//
//   k_develop   film sums -> PinholeCamera::stop normalisation (rgb / count,
//               PinholeCamera.cpp:70-78) -> gammaCorrection -> 8-bit rgba, in
//               one pass over the film; each output optional
//   k_tonemap   gammaCorrection (ToneMapping.cpp:24-53) in place: per pixel
//               rgb *= A l^gamma / l for the luminance l when l > FLT_EPSILON,
//               every channel clamped to [0, 1], alpha 1
//   k_median3   SimpleDenoiserMedian<1> (Denoiser.h:24-64): per-channel median
//               of the 3x3 window on pixels one away from every edge (alpha 1
//               there), the border copied; sorted row triples shared by the
//               windows of a column
//   k_median    the same for windows of 5x5 and 7x7
//   k_rgba8     saveImage's conversion (main.cpp:92): unsigned char(255 f),
//               rows optionally flipped (ImageSaver::flipVerticallyOnWrite)
//
// All are bound by HBM traffic: 16 B read and 16 B written per pixel for the
// float passes, 28 B read for the film.  The luminance and scaling use
// explicitly rounded operations (no contraction) so they round like the
// reference; only powf differs from the host's within its error bound.
//
// save_image writes PFM as ImageSaver::savePfm does with flipping on, and PNG
// (stored deflate blocks), BMP and TGA (uncompressed) with the same pixels as
// the reference's stb_image_write output.
#include <cuda_runtime.h>

#include <algorithm>
#include <cfloat>
#include <cstdio>
#include <cstring>
#include <string>
#include <vector>

#include "scene.h"

namespace omv {
namespace {

// clamp01f (UtilityFunctions.h:452) with the reference's comparison order:
// max(0, min(v, 1)), so NaN maps to 1
__device__ __forceinline__ float clamp01(float v)
{
    const float m = v < 1.0f ? v : 1.0f;
    return 0.0f > m ? 0.0f : m;
}

__device__ __forceinline__ float4 gamma_correct(float4 p, float A, float gamma)
{
    const float l = __fadd_rn(__fadd_rn(__fmul_rn(0.2126f, p.x), __fmul_rn(0.7152f, p.y)), __fmul_rn(0.0722f, p.z));
    const float o = __fmul_rn(A, powf(l, gamma));
    const float f = l > FLT_EPSILON ? __fdiv_rn(o, l) : 1.0f;
    return make_float4(clamp01(__fmul_rn(f, p.x)), clamp01(__fmul_rn(f, p.y)), clamp01(__fmul_rn(f, p.z)), 1.0f);
}

// unsigned char(255 f); the clamp only matters outside [0, 1], where the
// reference's conversion is undefined
__device__ __forceinline__ uint8_t to_u8(float f)
{
    const float v = __fmul_rn(255.0f, f);
    return v >= 255.0f ? (uint8_t)255 : (v > 0.0f ? (uint8_t)__float2uint_rz(v) : (uint8_t)0);
}

__device__ __forceinline__ uchar4 to_u8x4(float4 p)
{
    return make_uchar4(to_u8(p.x), to_u8(p.y), to_u8(p.z), to_u8(p.w));
}

// (float)(x * (1.0 / c)) of a film sum x (its 64 bits) by FP32 and integer
// arithmetic, where (sh, sl) is 1 / c as a float-float: x is split into its
// leading 24 bits h and the rest l, the product is p + e with p = h sh and e
// its rounding error and the cross terms, within 2^-44 |p| of the exact value
// (the FP64 expression is within 2^-51).  When adding 2^-42 |p| either way
// gives the same float, that is the FP64 expression's value too; about one sum
// in 2^17 lies closer to a rounding boundary, and false sends it, and
// sums beyond 2^-70 .. 2^90, to the FP64 arithmetic.
__device__ __forceinline__ bool scaled(unsigned long long x, float sh, float sl, float& out)
{
    const uint32_t hi = (uint32_t)(x >> 32), lo = (uint32_t)x;
    const uint32_t sign = hi & 0x80000000u, ex = (hi >> 20) & 0x7FFu;
    if (((hi ^ sign) | lo) == 0u) {
        out = __uint_as_float(sign);
        return true;
    }
    if (ex - (1023u - 70u) > 160u) return false;
    const uint32_t e32 = (ex - (1023u - 127u)) << 23;  // 2^(ex - 1023) as a float
    const float h = __uint_as_float(e32 | ((hi & 0xFFFFFu) << 3) | (lo >> 29));
    const float l = __fmul_rn((float)(lo & 0x1FFFFFFFu), __uint_as_float(e32 - (52u << 23)));
    const float p = __fmul_rn(h, sh);
    const float e = fmaf(l, sh, fmaf(h, sl, fmaf(h, sh, -p)));
    const float tol = __fmul_rn(p, 0x1p-42f);
    const float r0 = __fadd_rn(p, __fsub_rn(e, tol)), r1 = __fadd_rn(p, __fadd_rn(e, tol));
    out = __uint_as_float(__float_as_uint(r0) | sign);
    return r0 == r1;
}

// PinholeCamera::stop of one pixel: rgb / count as sum * (1.0 / count)
static __device__ __noinline__ float4 normalised_fp64(const double* __restrict__ sum, uint32_t count)
{
    const double c = (double)count;
    const double s = c < 0.5 ? 1.0 : __drcp_rn(c);  // 1.0 / c, the same correctly rounded bits
    return make_float4((float)(sum[0] * s), (float)(sum[1] * s), (float)(sum[2] * s), 1.0f);
}

__device__ __forceinline__ float4 normalised(const double* __restrict__ sum, uint32_t count)
{
    const unsigned long long* q = reinterpret_cast<const unsigned long long*>(sum);
    const unsigned long long x = q[0], y = q[1], z = q[2];
    const float c = count == 0u ? 1.0f : (float)count;
    const float sh = __fdiv_rn(1.0f, c);
    const float sl = __fmul_rn(fmaf(-sh, c, 1.0f), sh);
    float4 v;
    v.w = 1.0f;
    const bool ok = scaled(x, sh, sl, v.x) & scaled(y, sh, sl, v.y) & scaled(z, sh, sl, v.z);
    return ok && count < (1u << 24) ? v : normalised_fp64(sum, count);  // the count is exact as a float
}

// Bound by HBM (28 B read, up to 36 B written per pixel) once the arithmetic
// of the normalisation is off the FP64 pipe, which runs at about two lanes per
// SM and cycle: 1920x1080 with all three outputs, 51.6 us with three FP64
// multiplies, three conversions and the reciprocal per pixel, 27.3 so.
__global__ void __launch_bounds__(256) k_develop(const double* __restrict__ sum, const uint32_t* __restrict__ count,
                                                 int w, int h, float A, float gamma, float4* __restrict__ linear,
                                                 float4* __restrict__ toned, uchar4* __restrict__ rgba8, int flip)
{
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= (int64_t)w * h) return;
    const float4 lin = normalised(sum + 3 * i, count[i]);
    if (linear) linear[i] = lin;
    if (!toned && !rgba8) return;
    const float4 t = gamma_correct(lin, A, gamma);
    if (toned) toned[i] = t;
    if (rgba8) {  // i < 2^31: a 32-bit division for the row
        const int64_t y = (int64_t)((uint32_t)i / (uint32_t)w), x = i - y * w;
        rgba8[flip ? (h - 1 - y) * (int64_t)w + x : i] = to_u8x4(t);
    }
}

__global__ void k_tonemap(float4* __restrict__ img, int64_t n, float A, float gamma)
{
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
        img[i] = gamma_correct(img[i], A, gamma);
}

// four pixels per thread, all loaded before the first is converted (one load
// in flight per thread left it waiting for latency: 1920x1080 9.8 -> 8.4 us)
constexpr int kRgbaPixels = 4;

__global__ void __launch_bounds__(256) k_rgba8(const float4* __restrict__ in, uchar4* __restrict__ out, int w, int h,
                                               int flip)
{
    const int64_t n = (int64_t)w * h;
    const int64_t i0 = (int64_t)blockIdx.x * blockDim.x * kRgbaPixels + threadIdx.x;
    float4 v[kRgbaPixels];
#pragma unroll
    for (int k = 0; k < kRgbaPixels; ++k) {
        const int64_t i = i0 + k * blockDim.x;
        if (i < n) v[k] = in[i];
    }
#pragma unroll
    for (int k = 0; k < kRgbaPixels; ++k) {
        const int64_t i = i0 + k * blockDim.x;
        if (i >= n) return;
        const int64_t y = (int64_t)((uint32_t)i / (uint32_t)w), x = i - y * w;  // i < 2^31
        out[flip ? (h - 1 - y) * (int64_t)w + x : i] = to_u8x4(v[k]);
    }
}

__device__ __forceinline__ void order(float& a, float& b)
{
    const float lo = fminf(a, b), hi = fmaxf(a, b);
    a = lo;
    b = hi;
}

// median of nine by Paeth's 19-exchange network (A. Paeth, "Median finding on
// a 3x3 grid", Graphics Gems, 1990): after the exchanges p[4] holds the value
// that sorting the nine would put in the middle
__device__ __forceinline__ float median9(float p[9])
{
    order(p[1], p[2]); order(p[4], p[5]); order(p[7], p[8]);
    order(p[0], p[1]); order(p[3], p[4]); order(p[6], p[7]);
    order(p[1], p[2]); order(p[4], p[5]); order(p[7], p[8]);
    order(p[0], p[3]); order(p[5], p[8]); order(p[4], p[7]);
    order(p[3], p[6]); order(p[1], p[4]); order(p[2], p[5]);
    order(p[4], p[7]); order(p[4], p[2]); order(p[6], p[4]);
    order(p[4], p[2]);
    return p[4];
}

__device__ __forceinline__ float med3(float a, float b, float c)
{
    return fmaxf(fminf(a, b), fminf(fmaxf(a, b), c));
}

// the median of a pixel's window by the network above, for windows that may
// hold a NaN (its result then depends on the order of the exchanges)
static __device__ __noinline__ float4 median3_any(const float4* __restrict__ in, int w, int x, int y)
{
    float r[9], g[9], b[9];
#pragma unroll
    for (int dy = 0; dy < 3; ++dy)
#pragma unroll
        for (int dx = 0; dx < 3; ++dx) {
            const float4 p = in[(size_t)(y - 1 + dy) * w + (x - 1 + dx)];
            r[3 * dy + dx] = p.x;
            g[3 * dy + dx] = p.y;
            b[3 * dy + dx] = p.z;
        }
    return make_float4(median9(r), median9(g), median9(b), 1.0f);
}

// one channel of a row's three horizontal neighbours, sorted
struct Sorted3 {
    float lo, mid, hi;
};
__device__ __forceinline__ Sorted3 sort3(float a, float b, float c)
{
    return Sorted3{fminf(fminf(a, b), c), med3(a, b, c), fmaxf(fmaxf(a, b), c)};
}
// the median of nine from three sorted triples: the middle of the largest
// minimum, the middle median and the smallest maximum (J. L. Smith,
// "Implementing median filters in XC4000E FPGAs", XCell 23, 1996)
__device__ __forceinline__ float median9(Sorted3 p, Sorted3 q, Sorted3 r)
{
    return med3(fmaxf(fmaxf(p.lo, q.lo), r.lo), med3(p.mid, q.mid, r.mid), fminf(fminf(p.hi, q.hi), r.hi));
}

struct MedianRow {
    Sorted3 r, g, b;
    float4 mid;   // the row's own pixel
    bool plain;   // no NaN among the nine values (an infinity may clear it too)
};
__device__ __forceinline__ MedianRow median_row(const float4* __restrict__ row)
{
    const float4 a = row[-1], b = row[0], c = row[1];
    MedianRow m;
    m.r = sort3(a.x, b.x, c.x);
    m.g = sort3(a.y, b.y, c.y);
    m.b = sort3(a.z, b.z, c.z);
    m.mid = b;
    const float s = ((a.x + a.y + a.z) + (b.x + b.y + b.z)) + (c.x + c.y + c.z);
    m.plain = s == s;
    return m;
}

// 3x3 median.  A thread walks kMedRows rows of one column: each row's three
// neighbours are loaded and sorted once and serve the three windows that
// contain the row, about 17 min/max per channel and pixel where the
// 19-exchange network of every pixel by itself takes 38.  Neighbouring lanes
// read the same lines, so the loads need no shared tile.  1920x1080: 23.9 us
// with a 34x10 tile and the full network per pixel (ALU bound), 20.2 so.
constexpr int kMedRows = 4, kMedThreads = 128;

__global__ void __launch_bounds__(kMedThreads) k_median3(const float4* __restrict__ in, float4* __restrict__ out,
                                                         int w, int h)
{
    // one-dimensional grid (any width and height): column blocks, then row groups
    const uint32_t cols = ((uint32_t)w + kMedThreads - 1) / kMedThreads, group = blockIdx.x / cols;
    const int x = (int)((blockIdx.x - group * cols) * kMedThreads + threadIdx.x);
    const int y0 = (int)group * kMedRows, y1 = min(y0 + kMedRows, h);
    if (x >= w) return;
    if (x == 0 || x == w - 1) {
        for (int y = y0; y < y1; ++y) out[(size_t)y * w + x] = in[(size_t)y * w + x];
        return;
    }
    MedianRow p = median_row(in + (size_t)max(y0 - 1, 0) * w + x);
    MedianRow q = median_row(in + (size_t)y0 * w + x);
#pragma unroll
    for (int k = 0; k < kMedRows; ++k) {
        const int y = y0 + k;
        if (y >= y1) break;
        const MedianRow r = median_row(in + (size_t)min(y + 1, h - 1) * w + x);
        float4 o = q.mid;  // the border rows copy their input
        if (y > 0 && y < h - 1) {
            if (p.plain && q.plain && r.plain)
                o = make_float4(median9(p.r, q.r, r.r), median9(p.g, q.g, r.g), median9(p.b, q.b, r.b), 1.0f);
            else
                o = median3_any(in, w, x, y);
        }
        out[(size_t)y * w + x] = o;
        p = q;
        q = r;
    }
}

// the value with (n - 1) / 2 window elements before it in sorted order (ties
// broken by position): the element sorting would put in the middle
template <int N>
__device__ float select_median(const float* v)
{
    constexpr int target = (N - 1) / 2;
    for (int a = 0; a < N; ++a) {
        int before = 0;
        for (int b = 0; b < N; ++b) before += (v[b] < v[a] || (v[b] == v[a] && b < a)) ? 1 : 0;
        if (before == target) return v[a];
    }
    return v[target];
}

// the median of a window that holds a NaN
template <int H>
__device__ __noinline__ float4 median_any(const float4* __restrict__ in, int w, int x, int y)
{
    constexpr int S = 2 * H + 1;
    float v[3][S * S];
    for (int dy = 0; dy < S; ++dy)
        for (int dx = 0; dx < S; ++dx) {
            const float4 p = in[(size_t)(y - H + dy) * w + (x - H + dx)];
            v[0][S * dy + dx] = p.x;
            v[1][S * dy + dx] = p.y;
            v[2][S * dy + dx] = p.z;
        }
    return make_float4(select_median<S * S>(v[0]), select_median<S * S>(v[1]), select_median<S * S>(v[2]), 1.0f);
}

// moves the smallest of p[0 .. K) to p[0] and the largest to p[K - 1]
template <int K>
__device__ __forceinline__ void extremes(float* p)
{
#pragma unroll
    for (int i = 0; i < K / 2; ++i) order(p[i], p[K - 1 - i]);
#pragma unroll
    for (int i = 1; i < (K + 1) / 2; ++i) order(p[0], p[i]);
#pragma unroll
    for (int i = K / 2; i < K - 1; ++i) order(p[i], p[K - 1]);
}

// One step of the selection: with K values kept, the extremes go and the
// window's element `at` comes in, until three are left.
template <int H, int K>
struct MedianStep {
    static __device__ __forceinline__ void run(float* r, float* g, float* b, const float4* __restrict__ in, int w,
                                               bool& plain)
    {
        constexpr int S = 2 * H + 1, N = S * S, at = N / 2 + 2 + (N / 2 + 2 - K);
        extremes<K>(r);
        extremes<K>(g);
        extremes<K>(b);
        const float4 p = in[(ptrdiff_t)(at / S - H) * w + (at % S - H)];
        plain = plain && p.x == p.x && p.y == p.y && p.z == p.z;
        r[0] = p.x;
        g[0] = p.y;
        b[0] = p.z;
        MedianStep<H, K - 1>::run(r, g, b, in, w, plain);
    }
};
template <int H>
struct MedianStep<H, 3> {
    static __device__ __forceinline__ void run(float* r, float* g, float* b, const float4* __restrict__, int, bool&)
    {
        extremes<3>(r);
        extremes<3>(g);
        extremes<3>(b);
    }
};

// 5x5 and 7x7 medians by forgetful selection (Perrot, Domas and Couturier,
// "Fine-tuned high-speed implementation of a GPU-based median filter", J. Signal
// Processing Systems 75, 2014): of the first half of the window
// and two more, neither the smallest nor the largest can be the median, so
// both are dropped, one more element is taken in, and so on.  1920x1080, 5x5:
// 673 us with a rank count of every element (N^2 comparisons per channel), 99
// so; 7x7: 2736 and 364.
template <int H>
__global__ void __launch_bounds__(256) k_median(const float4* __restrict__ in, float4* __restrict__ out, int w, int h)
{
    constexpr int S = 2 * H + 1, N = S * S, K = N / 2 + 2;
    const int x = blockIdx.x * blockDim.x + threadIdx.x, y = blockIdx.y * blockDim.y + threadIdx.y;
    if (x >= w || y >= h) return;
    const size_t o = (size_t)y * w + x;
    if (x < H || y < H || x >= w - H || y >= h - H) {
        out[o] = in[o];
        return;
    }
    float r[K], g[K], b[K];
    bool plain = true;
#pragma unroll
    for (int i = 0; i < K; ++i) {
        const float4 p = in[o + (ptrdiff_t)(i / S - H) * w + (i % S - H)];
        plain = plain && p.x == p.x && p.y == p.y && p.z == p.z;
        r[i] = p.x;
        g[i] = p.y;
        b[i] = p.z;
    }
    MedianStep<H, K>::run(r, g, b, in + o, w, plain);
    out[o] = plain ? make_float4(r[1], g[1], b[1], 1.0f) : median_any<H>(in, w, x, y);
}

int stream_grid(int64_t n, int threads)
{
    static int sms = 0;
    if (!sms) {
        int dev = 0;
        if (cudaGetDevice(&dev) != cudaSuccess ||
            cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || sms <= 0)
            sms = 152;
    }
    const int64_t need = (n + threads - 1) / threads;
    return (int)std::max<int64_t>(1, std::min<int64_t>(need, (int64_t)sms * 8));
}

void check_image(int w, int h)
{
    if (w <= 0 || h <= 0) throw ArgError("image width and height must be positive");
    if ((int64_t)w * h > ((int64_t)1 << 31)) throw ArgError("image too large");
}

// ------------------------------------------------------------ writers ---
void put16(std::vector<uint8_t>& v, uint32_t x)
{
    v.push_back(x & 0xFF);
    v.push_back((x >> 8) & 0xFF);
}
void put32(std::vector<uint8_t>& v, uint32_t x)
{
    put16(v, x & 0xFFFF);
    put16(v, x >> 16);
}
void put32be(std::vector<uint8_t>& v, uint32_t x)
{
    v.push_back(x >> 24);
    v.push_back((x >> 16) & 0xFF);
    v.push_back((x >> 8) & 0xFF);
    v.push_back(x & 0xFF);
}

// CRC-32 of ISO 3309 / ITU-T V.42 (the PNG chunk checksum), bitwise
uint32_t crc32(const uint8_t* p, size_t n)
{
    uint32_t c = 0xFFFFFFFFu;
    for (size_t i = 0; i < n; ++i) {
        c ^= p[i];
        for (int k = 0; k < 8; ++k) c = (c >> 1) ^ (0xEDB88320u & (0u - (c & 1u)));
    }
    return ~c;
}

// PNG (RFC 2083): 8-bit RGBA, filter 0 on every row, the zlib stream (RFC 1950)
// made of stored deflate blocks (RFC 1951 section 3.2.4)
std::vector<uint8_t> encode_png(const uint8_t* rgba, int w, int h)
{
    std::vector<uint8_t> raw;
    raw.reserve((size_t)h * (4 * (size_t)w + 1));
    for (int y = 0; y < h; ++y) {
        raw.push_back(0);
        raw.insert(raw.end(), rgba + (size_t)y * 4 * w, rgba + (size_t)(y + 1) * 4 * w);
    }
    std::vector<uint8_t> z{0x78, 0x01};
    z.reserve(raw.size() + raw.size() / 65535 * 5 + 16);
    size_t off = 0;
    do {
        const size_t len = std::min<size_t>(65535, raw.size() - off);
        z.push_back(off + len >= raw.size() ? 1 : 0);
        put16(z, (uint32_t)len);
        put16(z, (uint32_t)(~len & 0xFFFF));
        z.insert(z.end(), raw.begin() + off, raw.begin() + off + len);
        off += len;
    } while (off < raw.size());
    uint32_t a = 1, b = 0;  // Adler-32
    for (uint8_t c : raw) {
        a = (a + c) % 65521u;
        b = (b + a) % 65521u;
    }
    put32be(z, (b << 16) | a);

    std::vector<uint8_t> out{0x89, 'P', 'N', 'G', 0x0D, 0x0A, 0x1A, 0x0A};
    auto chunk = [&out](const char* type, const std::vector<uint8_t>& data) {
        put32be(out, (uint32_t)data.size());
        const size_t start = out.size();
        out.insert(out.end(), type, type + 4);
        out.insert(out.end(), data.begin(), data.end());
        put32be(out, crc32(out.data() + start, out.size() - start));
    };
    std::vector<uint8_t> ihdr;
    put32be(ihdr, (uint32_t)w);
    put32be(ihdr, (uint32_t)h);
    ihdr.insert(ihdr.end(), {8, 6, 0, 0, 0});
    chunk("IHDR", ihdr);
    chunk("IDAT", z);
    chunk("IEND", {});
    return out;
}

// BMP: BITMAPINFOHEADER, 32 bits per pixel BGRA, rows stored bottom-up
std::vector<uint8_t> encode_bmp(const uint8_t* rgba, int w, int h)
{
    const uint32_t data = 4u * (uint32_t)w * (uint32_t)h;
    std::vector<uint8_t> v{'B', 'M'};
    v.reserve(54 + data);
    put32(v, 54 + data);
    put32(v, 0);
    put32(v, 54);
    put32(v, 40);
    put32(v, (uint32_t)w);
    put32(v, (uint32_t)h);
    put16(v, 1);
    put16(v, 32);
    put32(v, 0);
    put32(v, data);
    put32(v, 2835);
    put32(v, 2835);
    put32(v, 0);
    put32(v, 0);
    for (int y = h - 1; y >= 0; --y)
        for (int x = 0; x < w; ++x) {
            const uint8_t* p = rgba + 4 * ((size_t)y * w + x);
            v.insert(v.end(), {p[2], p[1], p[0], p[3]});
        }
    return v;
}

// TGA: uncompressed true colour, 32 bits BGRA, top-left origin
std::vector<uint8_t> encode_tga(const uint8_t* rgba, int w, int h)
{
    std::vector<uint8_t> v{0, 0, 2, 0, 0, 0, 0, 0, 0, 0, 0, 0};
    v.reserve(18 + 4 * (size_t)w * h);
    put16(v, (uint32_t)w);
    put16(v, (uint32_t)h);
    v.push_back(32);
    v.push_back(0x28);
    for (size_t i = 0; i < (size_t)w * h; ++i) {
        const uint8_t* p = rgba + 4 * i;
        v.insert(v.end(), {p[2], p[1], p[0], p[3]});
    }
    return v;
}

}  // namespace

void develop_film(const double* d_sum, const uint32_t* d_count, int w, int h, float A, float gamma, float* d_linear,
                  float* d_toned, uint8_t* d_rgba8, bool flip, cudaStream_t st)
{
    check_image(w, h);
    if (!d_sum || !d_count) throw ArgError("develop: film sums and counts are required");
    const int64_t n = (int64_t)w * h;
    k_develop<<<(unsigned)((n + 255) / 256), 256, 0, st>>>(
        d_sum, d_count, w, h, A, gamma, reinterpret_cast<float4*>(d_linear), reinterpret_cast<float4*>(d_toned),
        reinterpret_cast<uchar4*>(d_rgba8), flip ? 1 : 0);
    OMV_CUDA(cudaGetLastError());
}

void tonemap(float* d_rgba, int64_t pixels, float A, float gamma, cudaStream_t st)
{
    if (pixels < 0) throw ArgError("tonemap: negative pixel count");
    if (pixels == 0) return;
    if (!d_rgba) throw ArgError("tonemap: image is NULL");
    k_tonemap<<<stream_grid(pixels, 256), 256, 0, st>>>(reinterpret_cast<float4*>(d_rgba), pixels, A, gamma);
    OMV_CUDA(cudaGetLastError());
}

void denoise_median(const float* d_in, float* d_out, int w, int h, int half, cudaStream_t st)
{
    check_image(w, h);
    if (!d_in || !d_out) throw ArgError("median: image is NULL");
    if (d_in == d_out) throw ArgError("median: input and output must be distinct buffers");
    const auto* in = reinterpret_cast<const float4*>(d_in);
    auto* out = reinterpret_cast<float4*>(d_out);
    if (half == 1) {
        const int64_t blocks = ((int64_t)w + kMedThreads - 1) / kMedThreads * (((int64_t)h + kMedRows - 1) / kMedRows);
        k_median3<<<(unsigned)blocks, kMedThreads, 0, st>>>(in, out, w, h);
    } else if (half == 2 || half == 3) {
        const dim3 b(16, 8), g((w + 15) / 16, (h + 7) / 8);
        if (half == 2)
            k_median<2><<<g, b, 0, st>>>(in, out, w, h);
        else
            k_median<3><<<g, b, 0, st>>>(in, out, w, h);
    } else {
        throw ArgError("median: half size must be 1, 2 or 3");
    }
    OMV_CUDA(cudaGetLastError());
}

void rgba8(const float* d_in, uint8_t* d_out, int w, int h, bool flip, cudaStream_t st)
{
    check_image(w, h);
    if (!d_in || !d_out) throw ArgError("rgba8: image is NULL");
    const int64_t n = (int64_t)w * h;
    constexpr int64_t per = 256 * kRgbaPixels;
    k_rgba8<<<(unsigned)((n + per - 1) / per), 256, 0, st>>>(reinterpret_cast<const float4*>(d_in),
                                                            reinterpret_cast<uchar4*>(d_out), w, h, flip ? 1 : 0);
    OMV_CUDA(cudaGetLastError());
}

void save_image(const char* path, const float* rgba, int w, int h)
{
    if (!path || !rgba) throw ArgError("save_image: path and image are required");
    check_image(w, h);
    const std::string p(path);
    const size_t dot = p.find_last_of('.');
    std::string ext = dot == std::string::npos ? "" : p.substr(dot + 1);
    for (char& c : ext) c = (char)((c >= 'A' && c <= 'Z') ? c - 'A' + 'a' : c);
    const size_t n = (size_t)w * h;
    std::vector<uint8_t> bytes;
    if (ext == "pfm") {
        // ImageSaver::savePfm with flipping on: rows in stored order, rgb floats
        const std::string head = "PF\n" + std::to_string(w) + " " + std::to_string(h) + "\n-1.000000\n";
        bytes.assign(head.begin(), head.end());
        bytes.reserve(head.size() + 12 * n);
        for (size_t i = 0; i < n; ++i) {
            const auto* b = reinterpret_cast<const uint8_t*>(rgba + 4 * i);
            bytes.insert(bytes.end(), b, b + 12);
        }
    } else if (ext == "png" || ext == "bmp" || ext == "tga") {
        // saveImage (main.cpp:86-120): 8 bits per channel; flipVerticallyOnWrite(true)
        // puts the last row of the buffer at the top of the picture
        std::vector<uint8_t> q(4 * n);
        for (size_t y = 0; y < (size_t)h; ++y) {
            const float* src = rgba + 4 * (h - 1 - y) * (size_t)w;
            uint8_t* dst = q.data() + 4 * y * (size_t)w;
            for (size_t k = 0; k < 4 * (size_t)w; ++k) {
                const float v = 255.0f * src[k];
                dst[k] = v >= 255.0f ? 255 : (v > 0.0f ? (uint8_t)v : 0);
            }
        }
        bytes = ext == "png" ? encode_png(q.data(), w, h) : ext == "bmp" ? encode_bmp(q.data(), w, h)
                                                                          : encode_tga(q.data(), w, h);
    } else {
        throw ArgError("save_image: the extension must be png, bmp, tga or pfm");
    }
    FILE* f = std::fopen(path, "wb");
    if (!f) throw ArgError(std::string("save_image: cannot open ") + path);
    const size_t wr = std::fwrite(bytes.data(), 1, bytes.size(), f);
    const int rc = std::fclose(f);
    if (wr != bytes.size() || rc != 0) throw ArgError(std::string("save_image: short write to ") + path);
}

}  // namespace omv
