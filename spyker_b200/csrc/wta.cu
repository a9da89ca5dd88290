// Winner-take-all selection (convwta / fcwta), GPU resident: one CTA per
// sample computes the keys, then runs `count` rounds of block-wide argmax and
// suppression without any host round trip.
//
// src/spyker/cpu/wta.cpp:40-152.  For floating-point input, per sample:
//   min, max over all [T, X] values; diff = (max - min) * 2;
//   key(j) = (T - 1 - t0) + (x[t0, j] - min) / diff, t0 = first t with
//   x[t, j] > threshold, else -FLT_MAX (all in F32).
// For integer input: key(j) = T - t0 with t0 the first non-zero step, else 0.
// Each round takes the first index of the maximum key (std::max_element),
// stops on the sentinel, records the winner and suppresses the
// (2ry+1) x (2rx+1) box over all channels plus (convwta) the whole channel.
#include <type_traits>

#include "common.cuh"

namespace spk
{
namespace
{
constexpr int kWtaThreads = 1024;
constexpr int64_t kWtaSmemKeys = 40 * 1024;  // keys kept in shared memory up to 160 KB

// A key as an order-preserving word (0: none) and its position k * blockDim +
// tid (k: the thread's k-th position), so that positions compare as (k, tid).
struct Best
{
    unsigned e, k;
};

__device__ __forceinline__ unsigned order_enc(float v)
{
    const unsigned u = __float_as_uint(v + 0.0f);  // (-0 counts as 0)
    return (u & 0x80000000u) ? ~u : (u | 0x80000000u);
}

// A thread's first largest key among its positions (tid, tid + blockDim, ...).
__device__ __forceinline__ Best own_best(const float *keys, int64_t n)
{
    float v = -INFINITY;
    unsigned best = 0, k = 0;
    bool any = false;
#pragma unroll 4
    for (int64_t i = threadIdx.x; i < n; i += blockDim.x, ++k)
    {
        const float f = keys[i];
        if (f != f) continue;  // NaN never replaces the running maximum
        if (!any || v < f) v = f, best = k, any = true;
    }
    return Best{any ? order_enc(v) : 0u, best};
}

// Block-wide first-index argmax with std::max_element semantics, from the
// threads' own bests: per warp the largest word, its smallest k, its first
// lane (two redux instructions and a ballot), then the same over the warps.
__device__ __forceinline__ int64_t block_argmax(Best best, const float *keys, uint3 *s_best)
{
    const unsigned all = 0xffffffffu;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    unsigned e = __reduce_max_sync(all, best.e);
    unsigned k = __reduce_min_sync(all, best.e == e ? best.k : all);
    const unsigned who = __ballot_sync(all, best.e == e && best.k == k);
    if (lane == 0) s_best[warp] = make_uint3(e, k, unsigned(warp * 32 + __ffs(who) - 1));
    __syncthreads();
    const uint3 w = lane < int(blockDim.x >> 5) ? s_best[lane] : make_uint3(0, all, all);
    e = __reduce_max_sync(all, w.x);
    k = __reduce_min_sync(all, w.x == e ? w.y : all);
    const unsigned tid = __reduce_min_sync(all, w.x == e && w.y == k ? w.z : all);
    const float k0 = keys[0];
    return k0 != k0 || e == 0 ? 0 : int64_t(k) * blockDim.x + tid;
}

template <typename T>
__device__ __forceinline__ void minmax_update(T v, T &mn, T &mx)
{
    mn = (v < mn) ? v : mn;  // std::min(mn, v)
    mx = (mx < v) ? v : mx;  // std::max(mx, v)
}

// F32 input, read once by the whole chip: per position the first step above
// the threshold and its value, per block the smallest and largest value.
// Bound by the read (T x X values a sample).  One CTA per sample read its
// potentials twice and left SMs idle: 128 samples of 15 x 23520 took 228 us,
// this scan and the rounds below 36 and 42 us.  V: 4 neighbouring positions per thread
// where alignment allows, else 1.
constexpr int kScanThreads = 256;
constexpr uint16_t kNever = 0xFFFF;

struct WtaCandidates
{
    float *value;     // [b][x], where step is not kNever
    uint16_t *step;   // [b][x]
    float2 *extreme;  // [b][blocks]
    int blocks;
};

template <int V>
__global__ void __launch_bounds__(kScanThreads)
    wta_scan_kernel(const float *__restrict__ in, int t, int64_t x, float thr, WtaCandidates C)
{
    using Vec = typename std::conditional<V == 4, float4, float>::type;
    __shared__ float s_mn[kScanThreads / 32], s_mx[kScanThreads / 32];
    const int64_t b = blockIdx.y;
    const float *sample = in + b * int64_t(t) * x;
    float mn = sample[0], mx = mn;
    const int64_t j = (int64_t(blockIdx.x) * kScanThreads + threadIdx.x) * V;
    if (j < x)
    {
        float val[V];
        int at[V];
#pragma unroll
        for (int l = 0; l < V; ++l) at[l] = kNever, val[l] = 0.f;
        for (int q0 = 0; q0 < t; q0 += 8)
        {
            Vec r[8];
#pragma unroll
            for (int u = 0; u < 8; ++u)  // (a step past the last reads the last again)
                r[u] = __ldcs(reinterpret_cast<const Vec *>(sample + int64_t(min(q0 + u, t - 1)) * x + j));
#pragma unroll
            for (int u = 0; u < 8; ++u)
            {
                const float *v = reinterpret_cast<const float *>(&r[u]);
#pragma unroll
                for (int l = 0; l < V; ++l)
                {
                    minmax_update(v[l], mn, mx);
                    if (at[l] == kNever && v[l] > thr) at[l] = min(q0 + u, t - 1), val[l] = v[l];
                }
            }
        }
#pragma unroll
        for (int l = 0; l < V; ++l)
        {
            C.step[b * x + j + l] = uint16_t(at[l]);
            if (at[l] != kNever) C.value[b * x + j + l] = val[l];
        }
    }
    for (int o = 16; o > 0; o >>= 1)
    {
        const float a = __shfl_xor_sync(0xffffffffu, mn, o), z = __shfl_xor_sync(0xffffffffu, mx, o);
        minmax_update(a, mn, mx);
        minmax_update(z, mn, mx);
    }
    if ((threadIdx.x & 31) == 0) s_mn[threadIdx.x >> 5] = mn, s_mx[threadIdx.x >> 5] = mx;
    __syncthreads();
    if (threadIdx.x == 0)
    {
        for (int q = 1; q < kScanThreads / 32; ++q) minmax_update(s_mn[q], mn, mx), minmax_update(s_mx[q], mn, mx);
        C.extreme[b * C.blocks + blockIdx.x] = make_float2(mn, mx);
    }
}

template <typename T, bool kFloat>
__global__ void __launch_bounds__(kWtaThreads)
    wta_kernel(const T *__restrict__ in, int t, int64_t x, int c, int h, int w, int ry, int rx, int count, bool whole,
               T thr, int32_t *__restrict__ winners, int32_t *__restrict__ counts, float *__restrict__ gkeys,
               WtaCandidates C)
{
    extern __shared__ __align__(16) float smem_keys[];
    __shared__ uint3 s_best[32];
    __shared__ T s_mn[32], s_mx[32];
    const int64_t b = blockIdx.x;
    float *keys = gkeys ? gkeys + b * x : smem_keys;
    const T *sample = in + b * int64_t(t) * x;

    float low;
    if constexpr (kFloat)
    {
        T mn = sample[0], mx = sample[0];
        const int64_t tot = int64_t(t) * x;
        if (C.step)
            for (int i = threadIdx.x; i < C.blocks; i += blockDim.x)
            {
                const float2 e = C.extreme[b * C.blocks + i];
                minmax_update(T(e.x), mn, mx), minmax_update(T(e.y), mn, mx);
            }
        else
            for (int64_t i = threadIdx.x; i < tot; i += blockDim.x) minmax_update(sample[i], mn, mx);
        for (int o = 16; o > 0; o >>= 1)
        {
            T a = __shfl_xor_sync(0xffffffffu, mn, o), bb = __shfl_xor_sync(0xffffffffu, mx, o);
            minmax_update(a, mn, mx);
            minmax_update(bb, mn, mx);
        }
        if ((threadIdx.x & 31) == 0) s_mn[threadIdx.x >> 5] = mn, s_mx[threadIdx.x >> 5] = mx;
        __syncthreads();
        mn = s_mn[0], mx = s_mx[0];
        for (int q = 1; q < int(blockDim.x >> 5); ++q) minmax_update(s_mn[q], mn, mx), minmax_update(s_mx[q], mn, mx);
        const float fmn = float(mn);
        const float diff = __fmul_rn(__fsub_rn(float(mx), fmn), 2.0f);
        if (C.step)
            for (int64_t j0 = threadIdx.x; j0 < x; j0 += 8 * int64_t(blockDim.x))
            {
                int at[8];
                float val[8];
#pragma unroll
                for (int u = 0; u < 8; ++u)
                {
                    const int64_t j = j0 + u * int64_t(blockDim.x);
                    at[u] = j < x ? C.step[b * x + j] : kNever;
                }
#pragma unroll
                for (int u = 0; u < 8; ++u)
                    val[u] = at[u] != kNever ? C.value[b * x + j0 + u * int64_t(blockDim.x)] : 0.f;
#pragma unroll
                for (int u = 0; u < 8; ++u)
                {
                    const int64_t j = j0 + u * int64_t(blockDim.x);
                    if (j < x)
                        keys[j] = at[u] == kNever ? -FLT_MAX
                                                  : __fadd_rn(float(t - at[u] - 1), __fdiv_rn(__fsub_rn(val[u], fmn), diff));
                }
            }
        else
        for (int64_t j = threadIdx.x; j < x; j += blockDim.x)
        {
            float key = -FLT_MAX;
            for (int q = 0; q < t; ++q)
            {
                T v = sample[int64_t(q) * x + j];
                if (v > thr)
                {
                    key = __fadd_rn(float(t - q - 1), __fdiv_rn(__fsub_rn(float(v), fmn), diff));
                    break;
                }
            }
            keys[j] = key;
        }
        low = -FLT_MAX;
    }
    else
    {
        for (int64_t j = threadIdx.x; j < x; j += blockDim.x)
        {
            float key = 0.f;
            for (int q = 0; q < t; ++q)
                if (sample[int64_t(q) * x + j])
                {
                    key = float(t - q);
                    break;
                }
            keys[j] = key;
        }
        low = 0.f;
    }
    __syncthreads();

    // Keys only ever fall to `low`: a thread scans its positions again only
    // when its own best was suppressed.
    const int64_t len = int64_t(h) * w;
    Best best = own_best(keys, x);
    int found = 0;
    for (int r = 0; r < count; ++r)
    {
        if (r > 0 && best.e != 0 && order_enc(keys[int64_t(best.k) * blockDim.x + threadIdx.x]) != best.e)
            best = own_best(keys, x);
        int64_t idx = block_argmax(best, keys, s_best);
        float kv = keys[idx];
        __syncthreads();  // every thread has read the key and the warps' bests
        bool stop = kFloat ? (fabsf(__fsub_rn(kv, -FLT_MAX)) < 1e-5f) : (fabsf(kv) < 1e-5f);
        if (stop) break;
        const int z = int(idx / len), y = int((idx % len) / w), xx = int((idx % len) % w);
        if (threadIdx.x == 0)
        {
            int32_t *e = winners + (b * count + r) * 5;
            e[0] = 0, e[1] = 0, e[2] = z, e[3] = y, e[4] = xx;
        }
        const int sj = max(0, y - ry), ej = min(h, y + ry + 1);
        const int sk = max(0, xx - rx), ek = min(w, xx + rx + 1);
        // a row of the box in one channel per thread
        const unsigned bh = unsigned(ej - sj), rows = unsigned(c) * bh;
        for (unsigned i = threadIdx.x; i < rows; i += blockDim.x)
        {
            const unsigned ch = i / bh;
            float *row = keys + (int64_t(ch) * h + sj + (i - ch * bh)) * w;
            for (int k = sk; k < ek; ++k) row[k] = low;
        }
        if (whole)
            for (int64_t i = threadIdx.x; i < len; i += blockDim.x) keys[int64_t(z) * len + i] = low;
        __syncthreads();
        ++found;
    }
    if (threadIdx.x == 0) counts[b] = found;
    for (int i = found * 5 + threadIdx.x; i < count * 5; i += blockDim.x) winners[b * count * 5 + i] = 0;
}

size_t keys_bytes(int64_t b, int64_t x) { return x <= kWtaSmemKeys ? 0 : (size_t(b) * size_t(x) * 4 + 7) / 8 * 8; }

// the scan's candidates: block extremes, values, steps
size_t candidate_bytes(int64_t b, int64_t x) { return size_t(b) * (size_t(ceil_div(x, kScanThreads)) * 8 + size_t(x) * 6); }

// The scan pays where one CTA's two readings of a sample (some 80 ps a value)
// take longer than the second launch (some 8 us) and the scan's T steps (0.1 us
// each); sooner where the samples are several waves of CTAs.  us, scan and rounds
// / one CTA, 1 winner: 1 sample of 1000 steps x 100 positions 128 / 23, 100 x 800 33 /
// 23, 100 x 2000 33 / 29, 15 x 1890 30 / 22, 15 x 7000 23 / 25, 15 x 10000 25 / 29; 64 of
// 100 x 1400 43 / 26, 100 x 2200 49 / 31; 512 of 60 x 400 57 / 39, 15 x 1890 60 / 45, 15 x 4000 68 / 82, 15 x
// 7000 86 / 114.
bool scan_applies(int64_t b, int64_t t, int64_t x)
{
    return t * (x - 1250) > (b > sm_count() ? 25000 : 120000) && t < kNever && x < (int64_t(1) << 31);
}

size_t wta_workspace(int64_t b, int64_t t, int64_t x)
{
    return keys_bytes(b, x) + (scan_applies(b, t, x) ? candidate_bytes(b, x) : 0);
}

template <typename T, bool kFloat>
void launch_wta(const void *in, int64_t b, int64_t t, int64_t c, int64_t h, int64_t w, int64_t ry, int64_t rx,
                int64_t count, bool whole, double thr, int32_t *winners, int32_t *counts, void *ws, size_t ws_bytes,
                cudaStream_t s)
{
    const int64_t x = c * h * w;
    float *gkeys = nullptr;
    size_t smem = 0, used = 0;
    if (x <= kWtaSmemKeys)
        smem = size_t(x) * 4;
    else
    {
        used = keys_bytes(b, x);
        SPK_REQUIRE(ws != nullptr && ws_bytes >= used, "workspace is too small");
        gkeys = reinterpret_cast<float *>(ws);
    }
    // F32 input goes through the scan where the caller's workspace has room
    // for its candidates (else, and for samples that one CTA reads in a
    // microsecond or two, the selection reads the input itself)
    WtaCandidates C{};
    if constexpr (std::is_same<T, float>::value)
    {
        const size_t all = used + candidate_bytes(b, x);
        if (scan_applies(b, t, x) && b <= 65535 && ws != nullptr && ws_bytes >= all &&
            reinterpret_cast<uintptr_t>(ws) % 8 == 0)
        {
            char *base = static_cast<char *>(ws) + used;
            const bool vec = x % 4 == 0 && reinterpret_cast<uintptr_t>(in) % 16 == 0;
            C.blocks = int(ceil_div(x, kScanThreads * (vec ? 4 : 1)));
            C.extreme = reinterpret_cast<float2 *>(base);
            C.value = reinterpret_cast<float *>(base + size_t(b) * ceil_div(x, kScanThreads) * 8);
            C.step = reinterpret_cast<uint16_t *>(C.value + b * x);
            const dim3 grid(unsigned(C.blocks), unsigned(b));
            const auto scan = vec ? wta_scan_kernel<4> : wta_scan_kernel<1>;
            scan<<<grid, kScanThreads, 0, s>>>((const float *)in, int(t), x, scalar_to<float>(thr), C);
            SPK_LAUNCHED();
        }
    }
    auto k = wta_kernel<T, kFloat>;
    allow_smem(k, smem);
    k<<<unsigned(b), kWtaThreads, smem, s>>>((const T *)in, int(t), x, int(c), int(h), int(w), int(ry), int(rx),
                                             int(count), whole, scalar_to<T>(thr), winners, counts, gkeys, C);
    SPK_LAUNCHED();
}

void wta_dispatch(const void *in, spk_dtype type, int64_t b, int64_t t, int64_t c, int64_t h, int64_t w, int64_t ry,
                  int64_t rx, int64_t count, bool whole, double thr, int32_t *winners, int32_t *counts, void *ws,
                  size_t ws_bytes, cudaStream_t s)
{
    SPK_REQUIRE(count > 0, "winners count can't be less than 1");
    SPK_REQUIRE(ry >= 0 && rx >= 0, "radius can't be less than 0");
    SPK_REQUIRE(b >= 0 && t >= 1 && c >= 1 && h >= 1 && w >= 1, "invalid dims");
    SPK_REQUIRE(winners != nullptr && counts != nullptr, "null winners buffer");
    if (b == 0) return;
    switch (type)
    {
    case SPK_F32: launch_wta<float, true>(in, b, t, c, h, w, ry, rx, count, whole, thr, winners, counts, ws, ws_bytes, s); break;
    case SPK_U8: launch_wta<uint8_t, false>(in, b, t, c, h, w, ry, rx, count, whole, thr, winners, counts, ws, ws_bytes, s); break;
    case SPK_I32: launch_wta<int32_t, false>(in, b, t, c, h, w, ry, rx, count, whole, thr, winners, counts, ws, ws_bytes, s); break;
    default: throw Error(SPK_ERR_UNSUPPORTED, "WTA supports U8/I32/F32/F64 input");
    }
}
}  // namespace
}  // namespace spk

using namespace spk;

extern "C" {

size_t spk_rank_convwta_workspace(int64_t b, int64_t t, int64_t c, int64_t h, int64_t w)
{
    return wta_workspace(b, t, c * h * w);
}

spk_status spk_rank_convwta(const void *in, spk_dtype type, int64_t b, int64_t t, int64_t c, int64_t h, int64_t w,
                            int64_t ry, int64_t rx, int64_t count, double threshold, int32_t *winners, int32_t *counts,
                            void *ws, size_t ws_bytes, spk_stream stream)
{
    return guarded([&] {
        wta_dispatch(in, type, b, t, c, h, w, ry, rx, count, true, threshold, winners, counts, ws, ws_bytes,
                     stream_of(stream));
    });
}

size_t spk_rank_fcwta_workspace(int64_t b, int64_t t, int64_t n) { return wta_workspace(b, t, n); }

spk_status spk_rank_fcwta(const void *in, spk_dtype type, int64_t b, int64_t t, int64_t n, int64_t radius,
                          int64_t count, double threshold, int32_t *winners, int32_t *counts, void *ws, size_t ws_bytes,
                          spk_stream stream)
{
    return guarded([&] {
        wta_dispatch(in, type, b, t, 1, 1, n, 0, radius, count, false, threshold, winners, counts, ws, ws_bytes,
                     stream_of(stream));
    });
}

}  // extern "C"
