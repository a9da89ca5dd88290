// First-spike layer forward: t_out = first step whose potential exceeds the
// threshold, T when none.
//
// An input adds its weight once, at its own first spike, so the potentials of
// one output pixel at all steps are the running sums of its K = Cin*KH*KW
// weights taken in the order of their inputs' times: K additions per channel
// instead of the T x K products of the dense contraction, and none after the
// step at which every channel has fired (a quarter to a half of them in a
// trained range of thresholds).  256 images of 28 x 28 at T = 64 (32 x 5 x 5,
// 64 x 3 x 3, fc 10): 454 us for the three layers; the dense tensor-core kernel
// took 4377 us.
//
// A warp per output pixel: its K input times (bytes) are put in time order by
// a stable counting sort in shared memory (equal times in (channel, ky, kx)
// order, so the sums do not depend on scheduling), then the lanes, one channel
// each (NG groups of 32), walk the list and compare at the last input of each
// step.  Bound by the weight reads (8 bytes per channel and input) and the
// sort's issue slots.  The weights, FP64 [k][channel], are read through L1; small
// ones are copied to shared memory where a CTA has many pixels.  (Up to 150 KB
// of them there took as long for many pixels, 128 images of 14 x 14, 32 -> 64 3 x 3:
// 120 us against 113, and for few the copy by a CTA's few warps bounded the call,
// 6 images: 117 against 24.)
//
// Arithmetic: the BF16 split terms (h + m, or h + m + l = the F32 weight) of a
// weight are one exact FP64 number and the sums are FP64, the values that the
// dense kernel's per-term sums add up to; F32(sum) > threshold is tested as
// sum > bound with the FP64 bound of that rounding.
#include <algorithm>

#include <cuda_bf16.h>

#include "fst_walk.cuh"
#include "rounding.cuh"

namespace spk
{
namespace
{
constexpr int kMaxInputs = 4096;           // K: the list of a warp in shared memory
constexpr size_t kSmemWeights = 16 * 1024;
constexpr int64_t kMaxWeights = 64 * 1024;  // K x channels: read through L1
constexpr int kTile = 128;
constexpr int kBatch = 4;  // rounds of input times in flight
// warps per CTA (registers: 64, 80 or 128 a thread)
__host__ __device__ constexpr int max_warps(int ng) { return ng == 1 ? 32 : ng == 2 ? 24 : 16; }

inline size_t align256(size_t v) { return (v + 255) & ~size_t(255); }

struct WalkArgs
{
    const uint8_t *map;  // [b, cin, h, w] first steps, `time` = never
    const double *wt;    // [K][cout]
    float *t_out;
    int64_t npix;
    int cin, h, w, cout, kh, kw, sy, sx, top, left, ow, P, time, K;
    int tile, smem_weights;
    double bound;
};

__global__ void walk_times_kernel(const float *__restrict__ t_in, uint8_t *__restrict__ map, int64_t n, int time)
{
    for (int64_t i = int64_t(blockIdx.x) * blockDim.x + threadIdx.x; i < n; i += int64_t(gridDim.x) * blockDim.x)
    {
        const float t = t_in[i];
        map[i] = uint8_t((t >= 0.f && t < float(time)) ? int(t) : time);
    }
}

// [cout][K] F32 -> [K][cout] FP64 of the weight's BF16 terms
__global__ void walk_weights_kernel(const float *__restrict__ kernel, double *__restrict__ wt, int cout, int K,
                                    int terms)
{
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < cout * K; i += gridDim.x * blockDim.x)
    {
        const int k = i / cout, z = i - k * cout;
        const float v = kernel[int64_t(z) * K + k];
        const float h = __bfloat162float(__float2bfloat16_rn(v));
        const float m = __bfloat162float(__float2bfloat16_rn(v - h));
        double s = double(h) + double(m);
        if (terms == 3) s += double(__bfloat162float(__float2bfloat16_rn((v - h) - m)));
        wt[i] = s;
    }
}

template <int NG>
__global__ void __launch_bounds__(max_warps(NG) * 32) fst_walk_kernel(WalkArgs A)
{
    extern __shared__ __align__(16) unsigned char sm[];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
    const int z0 = blockIdx.y * 32 * NG, nz = min(32 * NG, A.cout - z0);
    // [K][nz] weights, [K] input offsets and taps, per warp: list [K], bins
    // [128], times [K]; the tile's output times [nz][tile]
    double *s_w = reinterpret_cast<double *>(sm);
    int2 *s_tap = reinterpret_cast<int2 *>(s_w + (A.smem_weights ? size_t(A.K) * nz : 0));
    unsigned *s_warp = reinterpret_cast<unsigned *>(s_tap + A.K);
    const int per = A.K + 128 + (A.K + 3) / 4;  // words of a warp
    unsigned *list = s_warp + warp * per, *bins = list + A.K;
    uint8_t *tl = reinterpret_cast<uint8_t *>(bins + 128);
    uint8_t *s_out = reinterpret_cast<uint8_t *>(s_warp + nw * per);
    const int KK = A.kh * A.kw;
    for (int k = threadIdx.x; k < A.K; k += blockDim.x)
    {
        const int c = k / KK, r = k - c * KK, ky = r / A.kw, kx = r - ky * A.kw;
        s_tap[k] = make_int2((c * A.h + ky) * A.w + kx, ky | (kx << 16));
    }
    if (A.smem_weights)
        for (int i = threadIdx.x; i < A.K * nz; i += blockDim.x)
        {
            const int k = i / nz;
            s_w[i] = A.wt[int64_t(k) * A.cout + z0 + (i - k * nz)];
        }
    // (loads through a pointer of either space: with global loads in their place
    // the compiler's order of the walk is 3 to 15 % slower)
    const double *wbase = A.smem_weights ? s_w : A.wt + z0;
    const int wstride = A.smem_weights ? nz : A.cout;
    int zi[NG];
#pragma unroll
    for (int g = 0; g < NG; ++g) zi[g] = min(lane + 32 * g, nz - 1);
    const unsigned lt = (1u << lane) - 1u;
    const int rounds = (A.K + 31) / 32;
    __syncthreads();
    for (int64_t p0 = int64_t(blockIdx.x) * A.tile; p0 < A.npix; p0 += int64_t(gridDim.x) * A.tile)
    {
        for (int j = warp; j < A.tile; j += nw)
        {
            const int64_t pix = p0 + j;
            if (pix >= A.npix) break;
            const int64_t smp = pix / A.P;
            const int q = int(pix - smp * A.P), oy = q / A.ow, ox = q - oy * A.ow;
            const int iy0 = oy * A.sy - A.top, ix0 = ox * A.sx - A.left;
            const uint8_t *src = A.map + smp * (int64_t(A.cin) * A.h * A.w) + iy0 * A.w + ix0;
            // counting sort of the inputs by time
#pragma unroll
            for (int u = 0; u < 4; ++u) bins[lane + 32 * u] = 0;
            __syncwarp();
            for (int r0 = 0; r0 < rounds; r0 += kBatch)
            {
                int t[kBatch];
#pragma unroll
                for (int u = 0; u < kBatch; ++u)
                {
                    const int k = 32 * (r0 + u) + lane;
                    t[u] = A.time;
                    if (k < A.K)
                    {
                        const int2 tap = s_tap[k];
                        const unsigned iy = unsigned(iy0 + (tap.y & 0xFFFF)), ix = unsigned(ix0 + (tap.y >> 16));
                        if (iy < unsigned(A.h) && ix < unsigned(A.w)) t[u] = __ldg(src + tap.x);
                    }
                }
#pragma unroll
                for (int u = 0; u < kBatch; ++u)
                {
                    const int k = 32 * (r0 + u) + lane;
                    if (k < A.K) tl[k] = uint8_t(t[u]);
                    if (t[u] < A.time) atomicAdd(&bins[t[u]], 1u);
                }
            }
            __syncwarp();
            // exclusive prefix over the steps, 4 per lane
            unsigned cnt[4], run = 0;
#pragma unroll
            for (int u = 0; u < 4; ++u) cnt[u] = bins[4 * lane + u], run += cnt[u];
            unsigned inc = run;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1)
            {
                const unsigned v = __shfl_up_sync(0xffffffffu, inc, o);
                if (lane >= o) inc += v;
            }
            const int n = int(__shfl_sync(0xffffffffu, inc, 31));
            run = inc - run;
            __syncwarp();
#pragma unroll
            for (int u = 0; u < 4; ++u) bins[4 * lane + u] = run, run += cnt[u];
            __syncwarp();
            for (int r = 0; r < rounds; ++r)
            {
                const int k = 32 * r + lane;
                const unsigned t = k < A.K ? tl[k] : unsigned(A.time);
                const unsigned peers = __match_any_sync(0xffffffffu, t);
                const bool on = t < unsigned(A.time);
                const unsigned pos = on ? bins[t] + __popc(peers & lt) : 0u;
                __syncwarp();
                if (on)
                {
                    list[pos] = (t << 16) | unsigned(k);
                    if ((peers >> lane) == 1u) bins[t] = pos + 1;  // the last of its step in this round
                }
                __syncwarp();
            }
            // the walk
            double acc[NG];
            int at[NG];
#pragma unroll
            for (int g = 0; g < NG; ++g) acc[g] = 0.0, at[g] = A.time;
            if (0.0 > A.bound && (n == 0 || (list[0] >> 16) > 0))
            {
                // fires before any input
#pragma unroll
                for (int g = 0; g < NG; ++g) at[g] = 0;
            }
            else
                for (int base = 0; base < n; base += 32)
                {
                    const int i = base + lane;
                    const unsigned e = i < n ? list[i] : 0u;
                    const bool last = i >= n - 1 || (list[i + 1] >> 16) != (e >> 16);
                    const unsigned ends = __ballot_sync(0xffffffffu, last);
                    bool done = false;
                    for (int i0 = 0; i0 < 32 && base + i0 < n; i0 += 8)
                    {
                        double wv[8][NG];
                        unsigned ev[8];
#pragma unroll
                        for (int u = 0; u < 8; ++u)
                        {
                            ev[u] = __shfl_sync(0xffffffffu, e, i0 + u);
                            const double *wk = wbase + (ev[u] & 0xFFFFu) * wstride;
#pragma unroll
                            for (int g = 0; g < NG; ++g) wv[u][g] = base + i0 + u < n ? wk[zi[g]] : 0.0;
                        }
#pragma unroll
                        for (int u = 0; u < 8; ++u)
                        {
#pragma unroll
                            for (int g = 0; g < NG; ++g) acc[g] += wv[u][g];
                            if (base + i0 + u < n && ((ends >> (i0 + u)) & 1u))
                            {
#pragma unroll
                                for (int g = 0; g < NG; ++g)
                                    if (at[g] == A.time && acc[g] > A.bound) at[g] = int(ev[u] >> 16);
                            }
                        }
                        bool fired = true;
#pragma unroll
                        for (int g = 0; g < NG; ++g) fired = fired && at[g] != A.time;
                        if (__all_sync(0xffffffffu, fired))
                        {
                            done = true;
                            break;
                        }
                    }
                    if (done) break;
                }
#pragma unroll
            for (int g = 0; g < NG; ++g)
                if (lane + 32 * g < nz) s_out[(lane + 32 * g) * A.tile + j] = uint8_t(at[g]);
            __syncwarp();
        }
        __syncthreads();
        for (int i = threadIdx.x; i < nz * A.tile; i += blockDim.x)
        {
            const int z = i / A.tile, j = i - z * A.tile;
            const int64_t pix = p0 + j;
            if (pix >= A.npix) continue;
            const int64_t smp = pix / A.P;
            A.t_out[(smp * A.cout + z0 + z) * A.P + (pix - smp * A.P)] = float(s_out[i]);
        }
        __syncthreads();
    }
}

// Layers with few output pixels (fc layers: one per sample) leave most SMs with
// a single warp in the walk.  Here a CTA takes one pixel and kStepMaps maps: its
// warps add their slices of the weights into per-step sums (shared memory,
// every warp its own, so the order is fixed), which are then run through in
// step order.  All K additions are made, by kStepWarps times the warps.
constexpr int kStepWarps = 16, kStepMaps = 32;

__global__ void __launch_bounds__(kStepWarps * 32) fst_steps_kernel(WalkArgs A)
{
    extern __shared__ __align__(16) unsigned char sm[];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
    const int64_t pix = blockIdx.x;
    const int z0 = blockIdx.y * kStepMaps, nz = min(kStepMaps, A.cout - z0), T = A.time;
    double *sums = reinterpret_cast<double *>(sm);  // [warps][T][nz]
    for (int i = threadIdx.x; i < nw * T * nz; i += blockDim.x) sums[i] = 0.0;
    __syncthreads();
    const int64_t smp = pix / A.P;
    const int q = int(pix - smp * A.P), oy = q / A.ow, ox = q - oy * A.ow;
    const int iy0 = oy * A.sy - A.top, ix0 = ox * A.sx - A.left, KK = A.kh * A.kw;
    const uint8_t *src = A.map + smp * (int64_t(A.cin) * A.h * A.w) + iy0 * A.w + ix0;
    double *mine = sums + warp * T * nz;
    // 32 inputs' times at a time, one per lane; then each input's weights,
    // one map per lane, 8 inputs in flight
    for (int k0 = warp * 32; k0 < A.K; k0 += nw * 32)
    {
        const int k = k0 + lane;
        int t = T;
        if (k < A.K)
        {
            const int c = k / KK, r = k - c * KK, ky = r / A.kw, kx = r - ky * A.kw;
            const unsigned iy = unsigned(iy0 + ky), ix = unsigned(ix0 + kx);
            if (iy < unsigned(A.h) && ix < unsigned(A.w)) t = __ldg(src + (c * A.h + ky) * A.w + kx);
        }
        unsigned on = __ballot_sync(0xffffffffu, t < T);
        while (on)
        {
            double w[8];
            int ts[8];
#pragma unroll
            for (int u = 0; u < 8; ++u)
            {
                const int l = on ? __ffs(on) - 1 : 0;
                ts[u] = on ? __shfl_sync(0xffffffffu, t, l) : T;
                w[u] = on && lane < nz ? __ldg(A.wt + int64_t(k0 + l) * A.cout + z0 + lane) : 0.0;
                on &= on - 1;
            }
#pragma unroll
            for (int u = 0; u < 8; ++u)
                if (ts[u] < T && lane < nz) mine[ts[u] * nz + lane] += w[u];
        }
    }
    __syncthreads();
    if (threadIdx.x >= nz) return;
    double v = 0.0;
    int at = T;
    for (int t = 0; t < T && at == T; ++t)
    {
        for (int w = 0; w < nw; ++w) v += sums[(w * T + t) * nz + threadIdx.x];
        if (v > A.bound) at = t;
    }
    A.t_out[(smp * A.cout + z0 + threadIdx.x) * A.P + q] = float(at);
}

struct WalkPlan
{
    int ng, tile, warps, smem_weights;
    size_t smem;
};

WalkPlan walk_plan(int64_t npix, int64_t K, int64_t cout)
{
    WalkPlan pl{};
    pl.ng = cout <= 32 ? 1 : cout <= 64 ? 2 : 4;
    const int64_t nz = std::min<int64_t>(cout, 32 * pl.ng);
    // tiles of up to 128 pixels, smaller while they leave SMs without one
    pl.tile = kTile;
    while (pl.tile > 1 && ceil_div(npix, pl.tile) < 2 * sm_count()) pl.tile /= 2;
    pl.smem_weights = pl.tile >= 32 && size_t(K) * nz * 8 <= kSmemWeights;
    const size_t word = size_t(K + 128 + (K + 3) / 4) * 4;
    const size_t fixed = (pl.smem_weights ? size_t(K) * nz * 8 : 0) + size_t(K) * 8 + size_t(nz) * pl.tile;
    pl.warps = std::min(max_warps(pl.ng), pl.tile);
    if (pl.ng == 1 && fixed + 32 * word < 100 * 1024) pl.warps = std::min(pl.warps, 16);  // two CTAs per SM
    while (pl.warps > 1 && fixed + pl.warps * word > 220 * 1024) --pl.warps;
    pl.smem = fixed + pl.warps * word + 16;
    return pl;
}
// Warps per CTA of the per-step sums, 0 where a warp per pixel takes the layer:
// few CTAs (three an SM, all resident), up to 64 steps to sum over, and no more
// weight reads than the L2 brings in the time of one pixel's walk.  us, sums /
// warp per pixel / dense kernel: fc 3136 -> 10, T = 64, 37 samples 43-53 / 86-211 /
// 57, 256 54-63 / 86-216 / 61, 590 92-112 / 87-216 / 96; T = 126, 256 80-119 / 86-213 /
// 92; 32 -> 64 3 x 3 on one 14 x 14, T = 16 21-23 / 27-45 / 33, T = 64 38-67 / 25-44 / 32.
int step_warps(int64_t npix, int64_t K, int64_t cout, int64_t time)
{
    if (K < 256 || time > 64 || npix * K * cout > (int64_t(1) << 24)) return 0;
    const int64_t nz = std::min<int64_t>(cout, kStepMaps);
    const int64_t warps = std::min({int64_t(kStepWarps), ceil_div(K, 32), 160 * 1024 / (time * nz * 8)});
    const int64_t resident = std::min<int64_t>(3, 225 * 1024 / (warps * time * nz * 8 + 1024)) * sm_count();
    return npix * ceil_div(cout, kStepMaps) <= resident ? int(warps) : 0;
}
}  // namespace

// The walk's time grows with the pixels, inputs and channels a lane, the dense
// kernel's with the pixels and steps (rounded up to a power of two), its K
// blocks or its columns; both start from the latency of one pixel, or of one
// tile.  The line is where both take the same for a threshold that the pixels
// reach after about a third of their inputs.  us, walk at 10 / 50 % of the summed
// weights, dense, 256 images of 14 x 14: 32 -> 64 3 x 3, T = 8 217 / 446 / 212, 16
// 212 / 441 / 384, 64 230 / 468 / 1440; 64 -> 64, T = 16 378 / 906 / 437, 64 407 /
// 931 / 1615; 128 -> 32, T = 16 552 / 1300 / 577, 64 618 / 1373 / 2125; 8 -> 128 5 x 5,
// T = 8 247 / 486 / 360; 28 x 28, 1 -> 32 5 x 5, T = 4 170 / 225 / 193, 8 161 / 233 / 360.
// 12 images of 14 x 14, T = 16: 32 -> 64 26 / 40 / 39, 128 -> 16 47 / 89 / 48.
bool fst_walk_pays(int64_t npix, int64_t cin, int64_t taps, int64_t cout, int64_t time)
{
    const int64_t K = cin * taps;
    if (step_warps(npix, K, cout, time)) return true;
    const int64_t kblocks = ceil_div(taps * ceil_div(cin, 8) * 8, 64), columns = ceil_div(cout, 16) * 16;
    int64_t steps = 1;
    while (steps < time) steps *= 2;
    // ns
    const double input = cout <= 32 ? 0.019 : cout <= 64 ? 0.023 : 0.034;
    const int64_t pixels = std::max<int64_t>(npix * ceil_div(cout, 128), 16 * sm_count());
    const double walk = 12e3 + double(pixels) * (0.6 + input * K);
    const double row = 0.04 + std::max(0.034 * kblocks, 0.0062 * columns);
    const double dense = 22e3 + 650.0 * kblocks + 100.0 * columns +
                         double(std::max<int64_t>(npix * steps - 128 * sm_count(), 0)) * row;
    return walk <= dense;
}

size_t fst_walk_workspace(int64_t b, int64_t cin, int64_t h, int64_t w, int64_t cout, int64_t kh, int64_t kw)
{
    const int64_t K = cin * kh * kw;
    if (K > kMaxInputs || kh > 255 || kw > 255 || cin * h * w >= (int64_t(1) << 30)) return 0;
    if (K * cout > kMaxWeights) return 0;
    return align256(size_t(K) * cout * 8) + align256(size_t(b) * cin * h * w);
}

void fst_walk(const FstWalk &F, void *ws, cudaStream_t s)
{
    const int K = F.cin * F.kh * F.kw;
    double *wt = static_cast<double *>(ws);
    uint8_t *map = static_cast<uint8_t *>(ws) + align256(size_t(K) * F.cout * 8);
    const int64_t n = F.b * F.cin * F.h * F.w;
    walk_times_kernel<<<grid_for(n, 256), 256, 0, s>>>(F.t_in, map, n, F.time);
    SPK_LAUNCHED();
    walk_weights_kernel<<<grid_for(int64_t(K) * F.cout, 256), 256, 0, s>>>(F.kernel, wt, F.cout, K, F.terms);
    SPK_LAUNCHED();
    const int64_t npix = F.b * F.oh * F.ow;
    const WalkPlan pl = walk_plan(npix, K, F.cout);
    WalkArgs A{map,  wt,     F.t_out, npix,   F.cin, F.h,           F.w,    F.cout, F.kh,    F.kw,
               F.sy, F.sx,   F.top,   F.left, F.ow,  F.oh * F.ow,   F.time, K,      pl.tile, pl.smem_weights,
               rounding_bound(F.threshold)};
    if (const int warps = step_warps(npix, K, F.cout, F.time))
    {
        const size_t smem = size_t(warps) * F.time * std::min(F.cout, kStepMaps) * 8;
        allow_smem(fst_steps_kernel, smem);
        fst_steps_kernel<<<dim3(unsigned(npix), unsigned(ceil_div(F.cout, kStepMaps))), warps * 32, smem, s>>>(A);
        SPK_LAUNCHED();
        return;
    }
    const auto k = pl.ng == 1 ? fst_walk_kernel<1> : pl.ng == 2 ? fst_walk_kernel<2> : fst_walk_kernel<4>;
    allow_smem(k, pl.smem);
    int occ = 0;
    SPK_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, k, pl.warps * 32, pl.smem));
    SPK_REQUIRE(occ > 0, "the layer does not fit one CTA");
    const dim3 grid(unsigned(std::min<int64_t>(ceil_div(npix, pl.tile), int64_t(sm_count()) * occ)),
                    unsigned(ceil_div(F.cout, 32 * pl.ng)));
    k<<<grid, pl.warps * 32, pl.smem, s>>>(A);
    SPK_LAUNCHED();
}
}  // namespace spk
