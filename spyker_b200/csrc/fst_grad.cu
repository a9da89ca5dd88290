// Gradients of a first-spike conv layer (the rule at the top of temporal.cu)
// from the non-zero output gradients.
//
// Behind a pooling layer three quarters of a layer's output gradients are
// exactly zero (a window's gradient goes to its earliest input), so both
// kernels first compact each (sample, map)'s gradients, in position order,
// into shared memory, and then spend one step per non-zero gradient with the
// lanes of a warp over the weight's taps: each lane compares its tap's input
// time with the output's.  Walking every position, a tap or an input pixel per
// thread (the kernels in temporal.cu), took 1811 us for the kernel gradients
// and 1084 us for the input gradients of 256 images through 32 x 5 x 5,
// 64 x 3 x 3 and fc 10; these take 176 and 156 us.
//
// Bound by shared-memory reads (one broadcast entry and one input time per
// lane and step).  The sample's input times are staged with the padding
// around them (+inf: never before an output), in rows and planes padded so
// that 32 neighbouring taps fall on as many banks as a small search finds.
//
//  * kernel gradient: a CTA holds 8 maps x up to 9 groups of 32 taps and runs
//    through a group of samples with FP64 sums in registers; the groups are
//    added in order afterwards.
//  * input gradient: a CTA holds a sample's channels (or a block of them) and
//    their sums in shared memory.  A warp owns whole channels, so within a
//    step its lanes update different pixels and the order of the sums (map,
//    then position) is fixed.
#include <algorithm>
#include <cfloat>
#include <cmath>

#include "fst_grad.cuh"

namespace spk
{
namespace
{
constexpr int kMaps = 8;          // maps per staged block
constexpr int kPositions = 256;   // output positions per staged block
constexpr int kMaxTapGroups = 9;  // of the kernel gradient's CTA

// One non-zero output gradient: its value, its output time, and its window's
// corner in the staged planes.
struct __align__(16) Entry
{
    double go;
    float to;
    int base;
};
struct __align__(16) EntryF
{
    float go, to;
    int base;
};
__device__ __forceinline__ void fill(Entry &e, float go, float to, int base) { e = Entry{double(go), to, base}; }
__device__ __forceinline__ void fill(EntryF &e, float go, float to, int base) { e = EntryF{go, to, base}; }

// Rows and planes of the staged input.
struct Stage
{
    int hp, wp, plane;  // padded height, row stride, plane stride
};

// The first strides from the tight ones on that spread 32 neighbouring taps
// best.
Stage stage_of(const FstGrad &F)
{
    const int hp = std::max((F.oh - 1) * F.sy + F.kh, F.h + F.top), w0 = std::max((F.ow - 1) * F.sx + F.kw, F.w + F.left);
    const int KK = F.kh * F.kw, taps = std::min(32, F.cin * KK);
    int tc[32], ty[32], tx[32];
    for (int k = 0; k < taps; ++k) tc[k] = k / KK, ty[k] = k % KK / F.kw, tx[k] = k % KK % F.kw;
    Stage best{hp, w0, hp * w0};
    int best_ways = taps + 1;
    // (a few microseconds of host time: it stops at the first strides without
    // conflicts, and gives a pair up at the best count so far)
    for (int dw = 0; dw < 8 && best_ways > 1; ++dw)
        for (int dp = 0; dp < 32 && best_ways > 1; ++dp)
        {
            const int wp = w0 + dw, plane = hp * wp + dp;
            uint8_t n[32] = {};
            int ways = 0;
            for (int k = 0; k < taps && ways < best_ways; ++k)
                ways = std::max<int>(ways, ++n[(tc[k] * plane + ty[k] * wp + tx[k]) & 31]);
            if (ways < best_ways) best_ways = ways, best = {hp, wp, plane};
        }
    return best;
}

// Channels c0 .. c0 + nc - 1 of sample s into dst.
__device__ __forceinline__ void stage_input(float *dst, const FstGrad &F, const Stage &S, int64_t s, int c0, int nc)
{
    // a thread per element, 8 in flight
    const int row = S.hp * S.wp, n = nc * row;
    const float *src = F.t_in + (s * F.cin + c0) * F.h * int64_t(F.w);
    for (int i0 = threadIdx.x; i0 < n; i0 += 8 * blockDim.x)
    {
        float v[8];
        int to[8];
#pragma unroll
        for (int u = 0; u < 8; ++u)
        {
            const int i = i0 + u * blockDim.x, c = i / row, q = i - c * row, y = q / S.wp, x = q - y * S.wp;
            const unsigned iy = unsigned(y - F.top), ix = unsigned(x - F.left);
            to[u] = i < n ? c * S.plane + q : -1;
            v[u] = i < n && iy < unsigned(F.h) && ix < unsigned(F.w) ? src[(c * F.h + iy) * F.w + ix] : INFINITY;
        }
#pragma unroll
        for (int u = 0; u < 8; ++u)
            if (to[u] >= 0) dst[to[u]] = v[u];
    }
}

// The non-zero gradients of maps z0 .. z0 + nz - 1 at positions p0 .. of
// sample s, in position order; a warp per map.
template <typename E>
__device__ __forceinline__ void compact(E *list, int *count, const FstGrad &F, const Stage &S, int64_t s, int z0,
                                        int nz, int p0)
{
    const int lane = threadIdx.x & 31, nw = blockDim.x >> 5, P = F.oh * F.ow, np = min(kPositions, P - p0);
    for (int z = threadIdx.x >> 5; z < nz; z += nw)
    {
        const int64_t row = (s * F.cout + z0 + z) * P + p0;
        float g[kPositions / 32], t[kPositions / 32];
#pragma unroll
        for (int u = 0; u < kPositions / 32; ++u)
        {
            const int p = 32 * u + lane;
            g[u] = p < np ? F.grad_out[row + p] : 0.f;
            t[u] = p < np ? F.t_out[row + p] : 0.f;
        }
        int n = 0;
#pragma unroll
        for (int u = 0; u < kPositions / 32; ++u)
        {
            const unsigned on = __ballot_sync(0xffffffffu, g[u] != 0.f);  // (a NaN counts)
            if (g[u] != 0.f)
            {
                const int q = p0 + 32 * u + lane, oy = q / F.ow, ox = q - oy * F.ow;
                fill(list[z * kPositions + n + __popc(on & ((1u << lane) - 1u))], g[u], t[u],
                     oy * F.sy * S.wp + ox * F.sx);
            }
            n += __popc(on);
        }
        if (lane == 0) count[z] = n;
    }
}

// grid (tap blocks, map blocks, sample groups); tg x (kMaps / ZP) warps
template <int ZP>
__global__ void __launch_bounds__(kMaxTapGroups * 32)
    fst_grad_w_kernel(FstGrad F, Stage S, double *__restrict__ part, int tg, int64_t per_group, int max_nc)
{
    extern __shared__ __align__(16) unsigned char gsm[];
    Entry *list = reinterpret_cast<Entry *>(gsm);                      // [kMaps][kPositions]
    int *count = reinterpret_cast<int *>(list + kMaps * kPositions);  // [kMaps]
    float *s_in = reinterpret_cast<float *>(count + kMaps);           // [max_nc][plane]
    const int KK = F.kh * F.kw, K = F.cin * KK, P = F.oh * F.ow;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, tw = warp % tg, zw = warp / tg;
    const int k0 = blockIdx.x * tg * 32, k1 = min(K, k0 + tg * 32);
    const int c0 = k0 / KK, nc = (k1 - 1) / KK + 1 - c0;
    const int z0 = blockIdx.y * kMaps, nz = min(kMaps, F.cout - z0);
    const int k = k0 + tw * 32 + lane, kk = min(k, k1 - 1);
    const int c = kk / KK, r = kk - c * KK, off = (c - c0) * S.plane + r / F.kw * S.wp + r % F.kw;
    const int64_t s0 = blockIdx.z * per_group, s1 = min(F.b, s0 + per_group);
    double acc[ZP];
#pragma unroll
    for (int u = 0; u < ZP; ++u) acc[u] = 0.0;
    for (int64_t s = s0; s < s1; ++s)
        for (int p0 = 0; p0 < P; p0 += kPositions)
        {
            __syncthreads();
            if (p0 == 0) stage_input(s_in, F, S, s, c0, nc);
            compact(list, count, F, S, s, z0, nz, p0);
            __syncthreads();
            const float *in = s_in + off;
#pragma unroll
            for (int u = 0; u < ZP; ++u)
            {
                const int z = zw * ZP + u;
                if (z >= nz) break;
                const Entry *e = list + z * kPositions;
                const int n = count[z];
                double a = acc[u];
#pragma unroll 4
                for (int i = 0; i < n; ++i)
                {
                    const Entry v = e[i];
                    if (in[v.base] < v.to) a += v.go;
                }
                acc[u] = a;
            }
        }
    if (k >= k1) return;
#pragma unroll
    for (int u = 0; u < ZP; ++u)
        if (zw * ZP + u < nz) part[(blockIdx.z * int64_t(F.cout) + z0 + zw * ZP + u) * K + k] = acc[u];
}

// The terms of a block's zero gradients (output row `row`, positions p0 .. p0 +
// np - 1), for weights that are not finite: the others add nothing there.
template <int TP>
__device__ __noinline__ void zero_terms(const FstGrad &F, const Stage &S, const float *s_in, float *mine,
                                        const int (&off)[TP], const bool (&on)[TP], const float (&wv)[TP], int64_t row,
                                        int p0, int np)
{
    for (int p = p0; p < p0 + np; ++p)
    {
        const float go = F.grad_out[row + p], to = F.t_out[row + p];
        if (go != 0.f) continue;  // (in the list)
        const int oy = p / F.ow, base = oy * F.sy * S.wp + (p - oy * F.ow) * F.sx;
#pragma unroll
        for (int u = 0; u < TP; ++u)
            if (on[u] && !(fabsf(wv[u]) <= FLT_MAX) && s_in[base + off[u]] < to)
                mine[base + off[u]] = __fmaf_rn(wv[u], go, mine[base + off[u]]);
        __syncwarp();
    }
}

// grid (channel blocks, samples); TP taps per lane (KK <= 32 * TP)
template <int TP>
__global__ void __launch_bounds__(512) fst_grad_in_kernel(FstGrad F, Stage S, float *__restrict__ gi, int cb,
                                                          int copies)
{
    extern __shared__ __align__(16) unsigned char gsm[];
    EntryF *list = reinterpret_cast<EntryF *>(gsm);
    int *count = reinterpret_cast<int *>(list + kMaps * kPositions);
    float *s_in = reinterpret_cast<float *>(count + kMaps);  // [cb][plane]
    float *s_gi = s_in + cb * S.plane;  // [copies][cb][plane]
    const int KK = F.kh * F.kw, P = F.oh * F.ow;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
    const int c0 = blockIdx.x * cb, nc = min(cb, F.cin - c0);
    const int64_t s = blockIdx.y;
    const int cpw = TP == 1 ? 32 / KK : 1;  // channels per warp
    stage_input(s_in, F, S, s, c0, nc);
    for (int i = threadIdx.x; i < copies * cb * S.plane; i += blockDim.x) s_gi[i] = 0.f;
    // warps of a copy take every copies-th map
    const int wpc = nw / copies, copy = warp / wpc;
    float *mine = s_gi + copy * cb * S.plane;
    for (int z0 = 0; z0 < F.cout; z0 += kMaps)
    {
        const int nz = min(kMaps, F.cout - z0);
        for (int p0 = 0; p0 < P; p0 += kPositions)
        {
            __syncthreads();
            compact(list, count, F, S, s, z0, nz, p0);
            __syncthreads();
            for (int g = warp - copy * wpc; copy < copies && g * cpw < nc; g += wpc)
            {
                int off[TP];
                bool on[TP];
                const float *kp[TP];
#pragma unroll
                for (int u = 0; u < TP; ++u)
                {
                    const int i = lane + 32 * u, c = g * cpw + (TP == 1 ? i / KK : 0), r = TP == 1 ? i % KK : i;
                    on[u] = (TP == 1 ? i < cpw * KK : i < KK) && c < nc;
                    off[u] = on[u] ? c * S.plane + r / F.kw * S.wp + r % F.kw : 0;
                    kp[u] = F.kernel + (int64_t(z0) * F.cin + c0 + c) * KK + r;
                }
                for (int z = copy; z < nz; z += copies)
                {
                    const EntryF *e = list + z * kPositions;
                    const int n = count[z];
                    float wv[TP];
#pragma unroll
                    for (int u = 0; u < TP; ++u) wv[u] = on[u] ? kp[u][int64_t(z) * F.cin * KK] : 0.f;
                    for (int i = 0; i < n; ++i)
                    {
                        const EntryF v = e[i];
#pragma unroll
                        for (int u = 0; u < TP; ++u)
                            if (on[u] && s_in[v.base + off[u]] < v.to)
                                mine[v.base + off[u]] = __fmaf_rn(wv[u], v.go, mine[v.base + off[u]]);
                        __syncwarp();  // the next entry's pixels overlap this one's
                    }
                    // Infinite and NaN weights meet the zero gradients too (NaN).  The
                    // vote waits for a map's weights, 11 us of an fc layer's 44; one
                    // vote a block behind its lists took 50, the block's weights in
                    // registers twice the time of a whole call.
                    bool odd = false;
#pragma unroll
                    for (int u = 0; u < TP; ++u) odd |= !(fabsf(wv[u]) <= FLT_MAX);
                    if (__any_sync(0xffffffffu, odd))
                        zero_terms<TP>(F, S, s_in, mine, off, on, wv, (s * F.cout + z0 + z) * int64_t(P), p0,
                                       min(kPositions, P - p0));
                }
            }
        }
    }
    __syncthreads();
    const int HW = F.h * F.w;
    for (int i = threadIdx.x; i < nc * HW; i += blockDim.x)
    {
        const int c = i / HW, q = i - c * HW, y = q / F.w;
        const float *g = s_gi + c * S.plane + (y + F.top) * S.wp + q - y * F.w + F.left;
        float sum = g[0];
        for (int k = 1; k < copies; ++k) sum += g[k * cb * S.plane];
        gi[(s * F.cin + c0) * HW + i] = sum;
    }
}

constexpr size_t kListBytes = size_t(kMaps) * kPositions * sizeof(Entry) + kMaps * 4;

bool fits(const FstGrad &F)
{
    // (indexes into the staged planes stay far below 2^31)
    return int64_t(F.oh) * F.sy + F.kh < 4096 && int64_t(F.ow) * F.sx + F.kw < 4096 && F.h + F.top < 4096 &&
           F.w + F.left < 4096;
}
}  // namespace

int64_t fst_grad_w_groups(int64_t b, int64_t weights, int64_t least)
{
    const int64_t room = (int64_t(64) << 20) / (weights * 8);
    return std::max(least, std::min({b, room, int64_t(3) * sm_count()}));
}

int64_t fst_grad_w(const FstGrad &F, double *part, int64_t groups, cudaStream_t s)
{
    if (!fits(F)) return 0;
    const Stage S = stage_of(F);
    const int KK = F.kh * F.kw;
    const int64_t K = int64_t(F.cin) * KK;
    // tap groups per CTA: as many as the staged channels leave room for
    int tg = int(std::min<int64_t>(kMaxTapGroups, ceil_div(K, 32)));
    auto channels = [&](int g) { return std::min<int64_t>(F.cin, (int64_t(g) * 32 + KK - 2) / KK + 1); };
    while (tg > 1 && channels(tg) * S.plane * 4 > 80 * 1024) --tg;
    const int64_t nc = channels(tg);
    if (nc * S.plane * 4 > 180 * 1024) return 0;
    const int zp = tg >= 5 ? 8 : tg >= 3 ? 4 : tg == 2 ? 2 : 1;
    const int64_t tb = ceil_div(K, int64_t(tg) * 32), zb = ceil_div(F.cout, kMaps);
    // samples per group: enough CTAs for three per SM, within the groups given
    const int64_t want = std::min({groups, F.b, std::max<int64_t>(1, ceil_div(int64_t(sm_count()) * 3, tb * zb))});
    const int64_t per = ceil_div(F.b, want), used = ceil_div(F.b, per);
    if (zb > 65535 || used > 65535) return 0;
    const size_t smem = kListBytes + size_t(nc) * S.plane * 4;
    const auto k = zp == 8 ? fst_grad_w_kernel<8> : zp == 4 ? fst_grad_w_kernel<4> : zp == 2 ? fst_grad_w_kernel<2> : fst_grad_w_kernel<1>;
    allow_smem(k, smem);
    k<<<dim3(unsigned(tb), unsigned(zb), unsigned(used)), tg * (kMaps / zp) * 32, smem, s>>>(F, S, part, tg, per, int(nc));
    SPK_LAUNCHED();
    return used;
}

bool fst_grad_in(const FstGrad &F, float *grad_in, double general_us, cudaStream_t s)
{
    if (!fits(F) || F.b > 65535) return false;
    const Stage S = stage_of(F);
    const int KK = F.kh * F.kw;
    if (KK > 128) return false;
    const int cpw = std::max(1, 32 / KK);
    // A warp waits for each step's sums before the next (0.1 us a step and group
    // of channels), so the steps are shared: `copies` sets of warps take turns at
    // the maps, each with sums of its own, and a CTA takes as few channels as
    // leave no SM without one.  Every CTA compacts all of its sample's gradients.
    // The costs are for a third of the gradients non-zero, the kernel of
    // temporal.cu, which takes every position, the cheaper one for dense gradients
    // of few maps.  us, a third of the gradients / all of them / that kernel: 1 -> 32
    // 5 x 5 on 28 x 28, 256 images 167 / 361 / 375 (two CTAs an SM with one warp at
    // work each: 855 / 2370); 32 -> 64 3 x 3 on 14 x 14, 16 images 92 / 188 / 278, 37
    // 112 / 232 / 289, 256 485 / 1400 / 1045; 128 -> 128, 8 images 199 / 444 / 557; 16 ->
    // 16 on 32 x 32, 4 images 150 / 410 / 79 (not taken).
    const double step = KK <= 32 ? 0.1 : KK <= 64 ? 0.18 : 0.36, nz = double(F.cout) * F.oh * F.ow / 3;
    const int64_t groups = ceil_div(F.cin, cpw), blocks = ceil_div(F.cout, kMaps) * ceil_div(F.oh * F.ow, kPositions);
    int copies = 0;
    int64_t cb = 0, warps = 0;
    size_t smem = 0;
    double best = general_us;
    for (int n = 1; n <= std::min(F.cout, kMaps); n *= 2)
    {
        const int64_t sets = std::min<int64_t>(16 / n, groups);
        for (int64_t each = 1;; each *= 2)  // groups of channels of a warp
        {
            const int64_t c = std::min<int64_t>(cpw * sets * each, F.cin);
            const int64_t w = std::max<int64_t>(n * sets, ceil_div(4, n) * n);
            const size_t bytes = kListBytes + size_t(c) * S.plane * 4 * (1 + n);
            if (bytes > 220 * 1024) break;
            const int64_t resident = std::min<int64_t>(220 * 1024 / int64_t(bytes + 1024), 64 / w);
            const int64_t ctas = F.b * ceil_div(F.cin, c);
            const double walk = nz / n * double(ceil_div(ceil_div(c, cpw), sets)) * step;
            const double us = double(ceil_div(ctas, std::max<int64_t>(resident, 1) * sm_count())) *
                              (walk + double(blocks) * (1.0 + 5.0 / w));
            // (more sets of sums cost their clearing and adding: for a clear gain only)
            const double gain = copies > 0 && copies < n ? 0.8 : 1.0;
            if (us < gain * best) best = us, copies = n, cb = c, warps = w, smem = bytes;
            if (c == F.cin) break;
        }
    }
    if (copies == 0) return false;
    const auto k = KK <= 32 ? fst_grad_in_kernel<1> : KK <= 64 ? fst_grad_in_kernel<2> : fst_grad_in_kernel<4>;
    allow_smem(k, smem);
    k<<<dim3(unsigned(ceil_div(F.cin, cb)), unsigned(F.b)), unsigned(warps * 32), smem, s>>>(F, S, grad_in, int(cb), copies);
    SPK_LAUNCHED();
    return true;
}
}  // namespace spk
