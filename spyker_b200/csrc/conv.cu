// Spike x weight convolution: the plain FP32 SIMT path and the dispatcher of
// spk_conv (Core::conv of src/spyker/impl.h:224; semantics shape.cpp:35-50).
//
// out[n, o, y, x] = sum_{c, ky, kx} in[n, c, y*sy + ky - top, x*sx + kx - left]
//                                   * kernel[o, c, ky, kx]     (zero pad)
// N folds batch and time (the reference reshapes [B, T, C, H, W] to
// [B*T, C, H, W], opers.cpp:419-420).  Spikes are read as u8 directly: there
// is no F32 copy of the spike tensor (the reference casts it, opers.cpp:410).
#include <algorithm>

#include "common.cuh"
#include "conv_tc.cuh"

namespace spk
{
namespace
{
constexpr int kTileW = 32, kTileH = 8, kGroup = 16;

// CTA: one image, an 8x32 tile of output pixels, 16 output channels; one
// output pixel per thread with 16 FP32 accumulators.  Input channel by input
// channel, the receptive-field patch and the 16 weight slices are staged in
// shared memory.  Summation order: c, ky, kx (fmaf).
template <typename I>
__global__ void __launch_bounds__(kTileW *kTileH)
    conv_fp32_kernel(const I *__restrict__ in, const float *__restrict__ kernel, float *__restrict__ out, int cin,
                     int h, int w, int cout, int kh, int kw, int oh, int ow, int sy, int sx, int top, int left,
                     int tiles_x)
{
    extern __shared__ __align__(16) float smem[];
    const int ph = (kTileH - 1) * sy + kh, pw = (kTileW - 1) * sx + kw;
    float *patch = smem;                 // [ph][pw]
    float *wsm = smem + ph * pw;         // [kGroup][kh*kw]
    const int n = blockIdx.z;
    const int tile = blockIdx.x;
    const int ty0 = (tile / tiles_x) * kTileH, tx0 = (tile % tiles_x) * kTileW;
    const int o0 = blockIdx.y * kGroup;
    const int lx = threadIdx.x % kTileW, ly = threadIdx.x / kTileW;
    const int oy = ty0 + ly, ox = tx0 + lx;
    const int iy0 = ty0 * sy - top, ix0 = tx0 * sx - left;
    const int taps = kh * kw;
    float acc[kGroup];
#pragma unroll
    for (int g = 0; g < kGroup; ++g) acc[g] = 0.f;

    for (int c = 0; c < cin; ++c)
    {
        const I *plane = in + (int64_t(n) * cin + c) * h * w;
        for (int i = threadIdx.x; i < ph * pw; i += blockDim.x)
        {
            int yy = iy0 + i / pw, xx = ix0 + i % pw;
            patch[i] = (yy >= 0 && yy < h && xx >= 0 && xx < w) ? float(plane[int64_t(yy) * w + xx]) : 0.f;
        }
        for (int i = threadIdx.x; i < kGroup * taps; i += blockDim.x)
        {
            int g = i / taps, r = i % taps;
            wsm[i] = (o0 + g < cout) ? kernel[(int64_t(o0 + g) * cin + c) * taps + r] : 0.f;
        }
        __syncthreads();
        for (int ky = 0; ky < kh; ++ky)
            for (int kx = 0; kx < kw; ++kx)
            {
                float v = patch[(ly * sy + ky) * pw + lx * sx + kx];
                const float *wp = wsm + ky * kw + kx;
#pragma unroll
                for (int g = 0; g < kGroup; ++g) acc[g] = fmaf(v, wp[g * taps], acc[g]);
            }
        __syncthreads();
    }
    if (oy < oh && ox < ow)
    {
#pragma unroll
        for (int g = 0; g < kGroup; ++g)
            if (o0 + g < cout) out[((int64_t(n) * cout + o0 + g) * oh + oy) * ow + ox] = acc[g];
    }
}

// Register-tiled form for a horizontal stride of 1 and kernel widths of 1, 3,
// 5 or 7: every potential is the same fmaf chain (c, ky, kx), so the results
// equal the kernel above bit for bit.
//
// Bound by the FP32 FMA pipe (2 x K x Cout FLOP per output position).  A
// thread keeps PX neighbouring positions x 8 channels in registers, as
// channel pairs for the packed fma.rn.f32x2; a warp's 32 lanes hold 32 groups
// of PX positions and share their 8 channels, so a tap costs two broadcast
// 16-byte weight loads per 4 PX packed FMAs, and the PX + KW - 1 inputs of a
// kernel row are read once for its KW taps.  (The kernel above reads one
// shared-memory word per FMA: 1920 maps of 30 x 14 x 14 to 100 channels, 5 x 5,
// 11.1 ms; here 1.59 ms, 36 TFLOP/s; 240 of 64 x 64 x 64 to 256 channels 54.2 ->
// 16.7 ms, 48 TFLOP/s.  Loading the next channel into registers during the
// current one's FMAs was slower, 23.3 ms: the registers spill.)  The groups run through the output rows of all images, so small
// planes fill a CTA; PX is 5, 7 or 8, whichever leaves fewer idle positions at
// the row's end (28 and 14 wide planes: 7).
//
// A CTA: `wp` x `wc` warps (groups x channel octets), the input rows under its
// output rows as F32 and the octets' weights [tap][channel] in shared memory,
// `cb` input channels per stage, two stages.
constexpr int kTiledWarps = 8, kCb = 4;

struct Fp32Tile
{
    int64_t groups;  // n * oh * gx
    int cin, h, w, cout, kh, oh, ow, sy, top, left;
    int gx, wc, wp, pw, ws;  // groups per row, warps, strides of a patch row and of a tap's weights
    int patch, cb;           // floats of one channel's patch; channels per stage
};

__device__ __forceinline__ unsigned long long pack2(float a, float b)
{
    unsigned long long r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
    return r;
}

__device__ __forceinline__ void fma2(unsigned long long &acc, unsigned long long a, unsigned long long b)
{
    asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(acc) : "l"(a), "l"(b));
}

template <typename I, int KW, int PX>
__global__ void __launch_bounds__(kTiledWarps * 32, 2)
    conv_fp32_tiled_kernel(const I *__restrict__ in, const float *__restrict__ kernel, float *__restrict__ out,
                           Fp32Tile G)
{
    extern __shared__ __align__(16) float smem[];
    constexpr int NV = PX == 8 ? (PX + KW - 1 + 3) / 4 * 4 : PX + KW - 1;  // inputs of a kernel row
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int taps = G.kh * KW;
    const int stage_floats = G.cb * (G.patch + taps * G.ws);
    // this CTA's groups, output rows and input rows (image by image)
    const int64_t g0 = int64_t(blockIdx.x) * G.wp * 32, g1 = min(g0 + G.wp * 32, G.groups) - 1;
    const int64_t r0 = g0 / G.gx, r1 = g1 / G.gx;
    const int64_t n0 = r0 / G.oh, n1 = r1 / G.oh;
    const int oy0 = int(r0 - n0 * G.oh), oy1 = int(r1 - n1 * G.oh);
    const int sfull = (G.oh - 1) * G.sy + G.kh;
    const int sfirst = ((n1 == n0 ? oy1 : G.oh - 1) - oy0) * G.sy + G.kh;
    const int rows = n1 == n0 ? sfirst : sfirst + int(n1 - n0 - 1) * sfull + oy1 * G.sy + G.kh;
    const int o0 = blockIdx.y * G.wc * 8;
    // this thread's group and channels
    const int wi = warp / G.wc, oct = warp - wi * G.wc;
    const int64_t g = min(g0 + wi * 32 + lane, g1);
    const bool mine = g0 + wi * 32 + lane <= g1;
    const int64_t r = g / G.gx, n = r / G.oh;
    const int gi = int(g - r * G.gx), oy = int(r - n * G.oh);
    const int prow = n == n0 ? (oy - oy0) * G.sy : sfirst + int(n - n0 - 1) * sfull + oy * G.sy;
    const bool work = wi < G.wp && o0 + oct * 8 < G.cout;
    const int xbase = prow * G.pw + gi * PX;

    unsigned long long acc[PX][4];
#pragma unroll
    for (int p = 0; p < PX; ++p)
#pragma unroll
        for (int q = 0; q < 4; ++q) acc[p][q] = 0ull;

    // the staged rows' offsets in a channel's planes of image n0 (-1: padding)
    int *roff = reinterpret_cast<int *>(smem + (G.cin > G.cb ? 2 : 1) * stage_floats);
    const int istride = G.cin * G.h * G.w;
    for (int q = tid; q < rows; q += kTiledWarps * 32)
    {
        const int e = q - sfirst, img = e < 0 ? 0 : 1 + e / sfull;
        const int iy = (e < 0 ? oy0 * G.sy + q : e - (img - 1) * sfull) - G.top;
        roff[q] = iy >= 0 && iy < G.h ? img * istride + iy * G.w : -1;
    }
    __syncthreads();
    const I *src0 = in + n0 * istride;
    // weights: 4 taps x 8 channels per warp step (few bank conflicts, 16-byte runs)
    const int tl = lane & 3, wo = oct * 8 + (lane >> 2);
    const float *ksrc = kernel + int64_t(o0 + wo) * G.cin * taps;
    const bool kin = wi < G.wp && o0 + wo < G.cout;
    const int need = (G.gx - 1) * PX + NV;  // columns of a patch row that are read

    // Stages `cb` channels: slot by slot (a column of a patch row), then tap by
    // tap, the channels innermost, so that a slot's addresses are made once.
    const int hw = G.h * G.w;
    auto stage = [&](int c0, float *buf) {
        const int nc = min(G.cb, G.cin - c0);
        const I *src = src0 + c0 * hw;
        for (int x = lane; x < need; x += 32)
        {
            const int ix = x - G.left;
            const bool col = ix >= 0 && ix < G.w;
            for (int q = warp; q < rows; q += 2 * kTiledWarps)
            {
                const int q2 = q + kTiledWarps;
                const int offa = roff[q], offb = q2 < rows ? roff[q2] : -1;
                const bool ina = col && offa >= 0, inb = col && offb >= 0;
                const I *pa = src + offa + ix, *pb = src + offb + ix;
                float *da = buf + q * G.pw + x, *db = buf + q2 * G.pw + x;
                I va[kCb], vb[kCb];
#pragma unroll
                for (int cc = 0; cc < kCb; ++cc)
                {
                    va[cc] = ina && cc < nc ? pa[cc * hw] : I(0);
                    vb[cc] = inb && cc < nc ? pb[cc * hw] : I(0);
                }
#pragma unroll
                for (int cc = 0; cc < kCb; ++cc)
                    if (cc < nc)
                    {
                        da[cc * G.patch] = float(va[cc]);
                        if (q2 < rows) db[cc * G.patch] = float(vb[cc]);
                    }
            }
        }
        float *wdst = buf + G.cb * G.patch + wo;
        for (int tap = wi * 4 + tl; tap < taps; tap += G.wp * 4)
        {
            const float *kc = ksrc + c0 * taps + tap;
            float v[kCb];
#pragma unroll
            for (int cc = 0; cc < kCb; ++cc) v[cc] = kin && cc < nc ? kc[cc * taps] : 0.f;
#pragma unroll
            for (int cc = 0; cc < kCb; ++cc)
                if (cc < nc) wdst[(cc * taps + tap) * G.ws] = v[cc];
        }
    };

    stage(0, smem);
    __syncthreads();
    int cur = 0;
    for (int c0 = 0; c0 < G.cin; c0 += G.cb, cur ^= 1)
    {
        if (c0 + G.cb < G.cin) stage(c0 + G.cb, smem + (cur ^ 1) * stage_floats);
        const float *buf = smem + cur * stage_floats;
        const int nc = work ? min(G.cb, G.cin - c0) : 0;
        for (int cc = 0; cc < nc; ++cc)
        {
            const float *xp = buf + cc * G.patch + xbase;
            const float *wp = buf + G.cb * G.patch + cc * taps * G.ws + oct * 8;
            for (int ky = 0; ky < G.kh; ++ky, xp += G.pw)
            {
                unsigned long long v[NV];
                if (PX == 8)
                {
#pragma unroll
                    for (int j = 0; j < NV; j += 4)
                    {
                        const float4 f = *reinterpret_cast<const float4 *>(xp + j);
                        v[j] = pack2(f.x, f.x), v[j + 1] = pack2(f.y, f.y);
                        v[j + 2] = pack2(f.z, f.z), v[j + 3] = pack2(f.w, f.w);
                    }
                }
                else
                {
#pragma unroll
                    for (int j = 0; j < NV; ++j) v[j] = pack2(xp[j], xp[j]);
                }
#pragma unroll
                for (int kx = 0; kx < KW; ++kx, wp += G.ws)
                {
                    const ulonglong2 wa = *reinterpret_cast<const ulonglong2 *>(wp);
                    const ulonglong2 wb = *reinterpret_cast<const ulonglong2 *>(wp + 4);
#pragma unroll
                    for (int p = 0; p < PX; ++p)
                    {
                        fma2(acc[p][0], v[p + kx], wa.x);
                        fma2(acc[p][1], v[p + kx], wa.y);
                        fma2(acc[p][2], v[p + kx], wb.x);
                        fma2(acc[p][3], v[p + kx], wb.y);
                    }
                }
            }
        }
        __syncthreads();
    }
    if (!work || !mine) return;
    const int ox = gi * PX, nx = min(PX, G.ow - ox);
    float *dst = out + ((n * G.cout + o0 + oct * 8) * G.oh + oy) * int64_t(G.ow) + ox;
    const int64_t plane = int64_t(G.oh) * G.ow;
#pragma unroll
    for (int q = 0; q < 8; ++q)
    {
        if (o0 + oct * 8 + q >= G.cout) break;
        float f[PX];
#pragma unroll
        for (int p = 0; p < PX; ++p)
            f[p] = __uint_as_float(q & 1 ? unsigned(acc[p][q / 2] >> 32) : unsigned(acc[p][q / 2]));
#pragma unroll
        for (int p = 0; p < PX; ++p)
            if (p < nx) dst[q * plane + p] = f[p];
    }
}

template <typename I, int KW, int PX>
bool launch_tiled(const I *in, const float *kernel, float *out, int64_t n, Fp32Tile G, cudaStream_t s)
{
    G.gx = int(ceil_div(G.ow, PX));
    G.groups = n * G.oh * G.gx;
    const int octs = int(ceil_div(G.cout, 8));
    G.wc = octs >= 3 ? 4 : octs;  // 1, 2 or 4 octets per CTA, the other warps over positions
    G.wp = kTiledWarps / G.wc;
    // Patch rows: an odd PX reads words, conflict-free when consecutive groups
    // stay PX words apart across rows; PX = 8 reads 16 bytes, best with an odd
    // number of them per row.
    if (PX != 8)
        G.pw = PX * G.gx + 32 * int(ceil_div(KW - 1, 32));
    else
        G.pw = (8 * G.gx + KW - 1 + 3) / 4 * 4, G.pw += G.pw / 4 % 2 ? 0 : 4;
    G.ws = G.wc * 8 + 4;
    // the most input rows that G.wp * 32 consecutive groups can span
    const int64_t orows = (int64_t(G.wp) * 32 - 1) / G.gx + 2;
    const int64_t imgs = (orows - 1) / G.oh + 2;
    const int64_t rows = std::min(orows * G.sy + imgs * G.kh, imgs * (int64_t(G.oh - 1) * G.sy + G.kh));
    const int64_t patch = (rows * G.pw + 15) / 4 * 4;  // (and what the last row's 16-byte reads take past its end)
    const int64_t per = patch + int64_t(G.kh) * KW * G.ws;
    const int64_t budget = 104 * 1024 / 4 - rows;  // floats, two CTAs per SM
    // (a CTA's offsets from its first image stay below 2^31)
    if (2 * per > budget || imgs * G.cin * G.h * G.w >= (int64_t(1) << 31) ||
        ceil_div(G.groups, int64_t(G.wp) * 32) > 0x7FFFFFFF) return false;
    G.patch = int(patch);
    G.cb = int(std::min<int64_t>(std::min<int64_t>(G.cin, kCb), budget / (2 * per)));
    const size_t smem = size_t((G.cin > G.cb ? 2 : 1) * G.cb * per + rows) * 4;
    auto k = conv_fp32_tiled_kernel<I, KW, PX>;
    allow_smem(k, smem);
    const dim3 grid(unsigned(ceil_div(G.groups, int64_t(G.wp) * 32)), unsigned(ceil_div(octs, G.wc)));
    k<<<grid, kTiledWarps * 32, smem, s>>>(in, kernel, out, G);
    SPK_LAUNCHED();
    return true;
}

template <typename I, int KW>
bool launch_tiled_px(const I *in, const float *kernel, float *out, int64_t n, const Fp32Tile &G, cudaStream_t s)
{
    // the least work at the row's end (5 positions pay more for their loads)
    const int64_t w5 = ceil_div(G.ow, 5) * 5 * 9 / 8, w7 = ceil_div(G.ow, 7) * 7, w8 = ceil_div(G.ow, 8) * 8;
    if (w5 < w7 && w5 < w8) return launch_tiled<I, KW, 5>(in, kernel, out, n, G, s);
    return w7 < w8 ? launch_tiled<I, KW, 7>(in, kernel, out, n, G, s) : launch_tiled<I, KW, 8>(in, kernel, out, n, G, s);
}

// The tiled form of the whole call; false where it does not apply (horizontal
// stride, other kernel widths, rows too long for a patch in shared memory).
template <typename I>
bool conv_fp32_tiled(const I *in, const float *kernel, float *out, int64_t n, int64_t cin, int64_t h, int64_t w,
                     int64_t cout, int64_t kh, int64_t kw, int64_t oh, int64_t ow, int64_t sy, int64_t sx, Pad4 p,
                     cudaStream_t s)
{
    const int64_t big = int64_t(1) << 20;
    if (sx != 1 || kh > 64 || cin > big || cout > big || h > big || w > big || oh > big || ow > big || sy > 64 ||
        p.top > big || p.left > big || ceil_div(cout, 32) > 65535)
        return false;
    Fp32Tile G{};
    G.cin = int(cin), G.h = int(h), G.w = int(w), G.cout = int(cout), G.kh = int(kh), G.oh = int(oh), G.ow = int(ow);
    G.sy = int(sy), G.top = int(p.top), G.left = int(p.left);
    switch (kw)
    {
    case 1: return launch_tiled_px<I, 1>(in, kernel, out, n, G, s);
    case 3: return launch_tiled_px<I, 3>(in, kernel, out, n, G, s);
    case 5: return launch_tiled_px<I, 5>(in, kernel, out, n, G, s);
    case 7: return launch_tiled_px<I, 7>(in, kernel, out, n, G, s);
    default: return false;
    }
}

template <typename I>
void launch_fp32(const I *in, const float *kernel, float *out, int64_t n, int64_t cin, int64_t h, int64_t w,
                 int64_t cout, int64_t kh, int64_t kw, int64_t oh, int64_t ow, int64_t sy, int64_t sx, Pad4 p,
                 cudaStream_t s)
{
    const int tiles_x = int(ceil_div(ow, kTileW)), tiles_y = int(ceil_div(oh, kTileH));
    const int ph = (kTileH - 1) * int(sy) + int(kh), pw = (kTileW - 1) * int(sx) + int(kw);
    const size_t smem = size_t(ph * pw + kGroup * kh * kw) * 4;
    SPK_REQUIRE(smem <= 200 * 1024, "kernel or stride too large for the FP32 path");
    SPK_REQUIRE(n <= 65535, "N (batch x time) is limited to 65535 per call on the FP32 path");
    auto k = conv_fp32_kernel<I>;
    allow_smem(k, smem);
    dim3 grid(unsigned(tiles_x * tiles_y), unsigned(ceil_div(cout, kGroup)), unsigned(n));
    k<<<grid, kTileW * kTileH, smem, s>>>(in, kernel, out, int(cin), int(h), int(w), int(cout), int(kh), int(kw),
                                          int(oh), int(ow), int(sy), int(sx), int(p.top), int(p.left), tiles_x);
    SPK_LAUNCHED();
}
}  // namespace
}  // namespace spk

using namespace spk;

extern "C" {

size_t spk_conv_workspace(int64_t n, int64_t cin, int64_t h, int64_t w, int64_t cout, int64_t kh, int64_t kw,
                          int precision)
{
    if (precision == SPK_CONV_FP32) return 0;
    return conv_tc_workspace(n, cin, h, w, cout, kh, kw, precision);
}

spk_status spk_conv(const void *in, spk_dtype itype, const float *kernel, float *out, int64_t n, int64_t cin, int64_t h,
                    int64_t w, int64_t cout, int64_t kh, int64_t kw, int64_t sy, int64_t sx, const int64_t *pad4,
                    int precision, void *ws, size_t ws_bytes, spk_stream stream)
{
    return guarded([&] {
        Pad4 p = pad_of(pad4);
        SPK_REQUIRE(sy >= 1 && sx >= 1, "stride items are incorrect");
        SPK_REQUIRE(n >= 0 && cin >= 1 && cout >= 1 && kh >= 1 && kw >= 1 && h >= 1 && w >= 1, "invalid dims");
        const int64_t oh = (h + p.top + p.bottom - kh) / sy + 1, ow = (w + p.left + p.right - kw) / sx + 1;
        SPK_REQUIRE(h + p.top + p.bottom >= kh && w + p.left + p.right >= kw && oh > 0 && ow > 0,
                    "input and kernel shapes are not compatible");
        if (n == 0) return;
        cudaStream_t s = stream_of(stream);
        if (precision == SPK_CONV_FP32)
        {
            if (itype == SPK_U8 ? conv_fp32_tiled((const uint8_t *)in, kernel, out, n, cin, h, w, cout, kh, kw, oh, ow, sy,
                                                  sx, p, s)
                                : itype == SPK_F32 && conv_fp32_tiled((const float *)in, kernel, out, n, cin, h, w, cout,
                                                                      kh, kw, oh, ow, sy, sx, p, s))
                return;
            for (int64_t n0 = 0; n0 < n; n0 += 65535)
            {
                int64_t nn = std::min<int64_t>(65535, n - n0);
                float *o = out + n0 * cout * oh * ow;
                if (itype == SPK_U8)
                    launch_fp32<uint8_t>((const uint8_t *)in + n0 * cin * h * w, kernel, o, nn, cin, h, w, cout, kh,
                                         kw, oh, ow, sy, sx, p, s);
                else if (itype == SPK_F32)
                    launch_fp32<float>((const float *)in + n0 * cin * h * w, kernel, o, nn, cin, h, w, cout, kh, kw, oh,
                                       ow, sy, sx, p, s);
                else
                    throw Error(SPK_ERR_UNSUPPORTED, "conv input must be U8 or F32");
            }
            return;
        }
        SPK_REQUIRE(precision == SPK_CONV_BF16X2 || precision == SPK_CONV_BF16X3, "unknown precision");
        conv_tc(in, itype, kernel, out, n, cin, h, w, cout, kh, kw, sy, sx, p, oh, ow, precision, ws, ws_bytes, s);
    });
}

}  // extern "C"
