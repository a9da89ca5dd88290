// Output writer of the first-crossing search: cumulative spikes
// [B, T, C, OH, OW] and pooled spikes [B, T, C, POH, POW] from the per-pixel
// records (winner w, first step t0): channel w fires from t0 on, nothing else
// does.  Off the search path (negative weights or other input) it writes
// zeros, which the dense kernel then fills.
//
// Bound by the bytes written (T x C per pixel).  A CTA writes a range of
// channels of one sample, at every step; the ranges are cut so that a few
// samples still fill the chip (a grid of one CTA per sample took 75.6 ms for
// 8 maps of 128 x 128 x 256 at T = 30 and 12.8 us for one map of 28 x 28) and
// so that the range's pooled table fits shared memory (that call: 79.96 ->
// 4.72 ms).  Per pixel the winner
// and first-step bytes sit in shared memory (in global memory, behind one
// more launch, above 16384 pixels); pooled spikes come from a byte table of
// the first firing step per (channel, cell), a shared-memory minimum over the
// pixels won by the range's channels.
//
// Every store is 16 bytes at a 16-byte boundary; only the ragged ends of a
// (step, channel range) run go byte by byte.  Where the runs of all steps
// start aligned, a chunk's compares are made once and masked per step; other
// shapes (odd maps) rebuild the chunk at each step (a byte a thread before:
// a training step of 333 images of 33 x 33 1.51 -> 1.03 ms).  Chunks are read as
// unaligned words of the byte arrays, which are extended past the plane's end
// by its first 16 pixels so that a chunk may run into the next channel's
// plane.
#include <algorithm>

#include "search_write.cuh"

namespace spk
{
namespace
{
constexpr int kThreads = 256;
constexpr int kSmemPixels = 16384;    // larger maps keep their bytes in global memory
constexpr int kTableBytes = 48 * 1024;  // pooled table of a CTA's channel range
constexpr int64_t kRangeBytes = int64_t(1) << 30;  // a range's bytes of a step
constexpr int kTableMax = 160 * 1024;   // of one channel; above it cells are read from their windows

// bytes of one sample's extended array: the map, 16 bytes more, and what
// unaligned word loads read past those
__host__ __device__ inline int64_t ext_bytes(int64_t ohw) { return (ohw + 32 + 15) & ~int64_t(15); }

// Byte-parallel tests on four pixels at once (first steps below 0x80): the
// bytes of w that equal those of c4, and the bytes of t0 at or below t, as
// 0x80 flags.
__device__ __forceinline__ uint32_t bytes_eq(uint32_t w, uint32_t c4)
{
    const uint32_t x = w ^ c4;
    return ~(((x & 0x7F7F7F7Fu) + 0x7F7F7F7Fu) | x | 0x7F7F7F7Fu);
}
__device__ __forceinline__ uint32_t bytes_le(uint32_t t0, uint32_t t4) { return ((t4 | 0x80808080u) - t0) & 0x80808080u; }

// 16 bytes from any address of a 4-byte aligned array (reads up to 3 bytes
// on either side, inside the array's padding).
__device__ __forceinline__ void load16u(const uint8_t *p, uint32_t (&v)[4])
{
    const uintptr_t a = reinterpret_cast<uintptr_t>(p);
    const uint32_t *q = reinterpret_cast<const uint32_t *>(a & ~uintptr_t(3));
    const int sh = int(a & 3) * 8;
    uint32_t x = q[0];
    if (sh == 0)
    {
        v[0] = x, v[1] = q[1], v[2] = q[2], v[3] = q[3];
        return;
    }
#pragma unroll
    for (int j = 0; j < 4; ++j)
    {
        const uint32_t y = q[j + 1];
        v[j] = __funnelshift_r(x, y, sh);
        x = y;
    }
}

// Per-pixel bytes of maps too large to stage in shared memory, extended
// arrays: winners [b][ext], then first steps [b][ext].
__global__ void search_codes_kernel(const int4 *__restrict__ records, uint8_t *__restrict__ codes, int64_t b, int ohw,
                                    int T, const int *negw, const int *flag)
{
    if (*negw || *flag) return;
    const int64_t ext = ext_bytes(ohw), n = b * ext;
    for (int64_t i = int64_t(blockIdx.x) * blockDim.x + threadIdx.x; i < n; i += int64_t(gridDim.x) * blockDim.x)
    {
        const int64_t smp = i / ext;
        int p = int(i - smp * ext);
        p = p < ohw ? p : p - ohw;  // (these maps are far larger than the extension)
        const int4 r = records[smp * ohw + p];
        codes[i] = uint8_t(r.x);
        codes[n + i] = uint8_t(min(r.y, T));
    }
}

struct WriteArgs
{
    const int4 *records;
    const uint8_t *codes;
    const int *negw, *flag;
    uint8_t *spikes, *pooled;
    int64_t b;
    int T, C, ohw, ow, pky, pkx, poh, pow_;
    int nc;    // channels per CTA
    int ptab;  // pooled cells from a table in shared memory
};

// The chunk of 16 bytes of (channel, pixel) positions f .. f + 15 of a step's run
// (from the range's first channel on): as 0x80 flags of the pixels won by their
// channel, and first steps.
struct SpikeSource
{
    const uint8_t *w, *t;
    int hw, c0;
    __device__ __forceinline__ void get(int f, uint32_t (&eq)[4], uint32_t (&tw)[4]) const
    {
        const int k = f / hw, px = f - k * hw, c = c0 + k;
        load16u(w + px, eq);
        load16u(t + px, tw);
        const uint32_t c4 = uint32_t(c) * 0x01010101u, d4 = uint32_t(c + 1) * 0x01010101u;
#pragma unroll
        for (int j = 0; j < 4; ++j)
        {
            const int left = hw - px - 4 * j;  // pixels of the word still in plane c
            const uint32_t m = left >= 4 ? 0xFFFFFFFFu : left <= 0 ? 0u : (1u << (8 * left)) - 1u;
            eq[j] = bytes_eq(eq[j], (c4 & m) | (d4 & ~m));
        }
    }
    __device__ __forceinline__ uint8_t one(int f, int step) const
    {
        const int k = f / hw, px = f - k * hw;
        return int(w[px]) == c0 + k && int(t[px]) <= step;
    }
};

struct TableSource
{
    const uint8_t *first;  // [channel][cell] from the range's first channel
    __device__ __forceinline__ void get(int f, uint32_t (&eq)[4], uint32_t (&tw)[4]) const
    {
        load16u(first + f, tw);
#pragma unroll
        for (int j = 0; j < 4; ++j) eq[j] = 0x80808080u;
    }
    __device__ __forceinline__ uint8_t one(int f, int step) const { return int(first[f]) <= step; }
};

// The n bytes from dst on of every step's slab (slab bytes apart).  Off the
// search path (!lean) they are zero and the source is not read: its arrays are
// then unwritten, and the table of a large pooled map has no bytes.
template <typename Source>
__device__ __forceinline__ void write_range(uint8_t *dst, int T, int64_t slab, int n, bool lean, bool wide,
                                            const Source &src)
{
    if (wide && (reinterpret_cast<uintptr_t>(dst) & 15) == 0 && slab % 16 == 0 && n % 16 == 0)
    {
        for (int f = 16 * threadIdx.x; f < n; f += 16 * kThreads)
        {
            uint32_t eq[4] = {}, tw[4] = {};
            if (lean) src.get(f, eq, tw);
            for (int t = 0; t < T; ++t)
            {
                const uint32_t t4 = uint32_t(t) * 0x01010101u;
                *reinterpret_cast<uint4 *>(dst + t * slab + f) =
                    make_uint4((eq[0] & bytes_le(tw[0], t4)) >> 7, (eq[1] & bytes_le(tw[1], t4)) >> 7,
                               (eq[2] & bytes_le(tw[2], t4)) >> 7, (eq[3] & bytes_le(tw[3], t4)) >> 7);
            }
        }
        return;
    }
    if (!wide || n < 64)
    {
        // (planes of fewer than 16 pixels, or few bytes)
        for (int i = threadIdx.x; i < T * n; i += kThreads)
        {
            const int t = i / n, f = i - t * n;
            dst[t * slab + f] = lean ? src.one(f, t) : uint8_t(0);
        }
        return;
    }
    // per step, the 16-byte chunks of the run's address range
    const int per = n / 16 + 2, tn = max(1, min(T, (1 << 30) / per));
    for (int tb = 0; tb < T; tb += tn)
        for (int i = threadIdx.x; i < min(tn, T - tb) * per; i += kThreads)
        {
            const int dt = i / per, k = i - dt * per, t = tb + dt;
            uint8_t *run = dst + t * slab;
            const int f = 16 * k - int(reinterpret_cast<uintptr_t>(run) & 15);
            if (f >= n) continue;
            if (f < 0 || f + 16 > n)
            {
                for (int g = max(f, 0); g < min(f + 16, n); ++g) run[g] = lean ? src.one(g, t) : uint8_t(0);
                continue;
            }
            uint32_t eq[4] = {}, tw[4] = {};
            if (lean) src.get(f, eq, tw);
            const uint32_t t4 = uint32_t(t) * 0x01010101u;
            *reinterpret_cast<uint4 *>(run + f) =
                make_uint4((eq[0] & bytes_le(tw[0], t4)) >> 7, (eq[1] & bytes_le(tw[1], t4)) >> 7,
                           (eq[2] & bytes_le(tw[2], t4)) >> 7, (eq[3] & bytes_le(tw[3], t4)) >> 7);
        }
}

__global__ void __launch_bounds__(kThreads) search_write_kernel(WriteArgs A)
{
    // [ext] winner bytes, [ext] first-step bytes (maps up to kSmemPixels),
    // then the range's pooled first steps [nc][cells], 16 bytes of slack
    extern __shared__ __align__(16) uint8_t wsm_[];
    const bool lean = !*A.negw && !*A.flag;
    const int ohw = A.ohw, phw = A.poh * A.pow_;
    const int ext = int(ext_bytes(ohw));
    const int c0 = blockIdx.x * A.nc, c1 = min(c0 + A.nc, A.C);
    uint8_t *sw = wsm_, *st = wsm_ + ext, *first = wsm_ + (A.codes ? 0 : 2 * ext);
    for (int64_t smp = blockIdx.y; smp < A.b; smp += gridDim.y)
    {
        const uint8_t *wsrc = A.codes ? A.codes + smp * ext : sw;
        const uint8_t *tsrc = A.codes ? A.codes + (A.b + smp) * ext : st;
        if (lean)
        {
            if (!A.codes)
                for (int p = threadIdx.x; p < ohw; p += kThreads)
                {
                    const int4 r = A.records[smp * ohw + p];
                    const uint8_t w = uint8_t(r.x), t = uint8_t(min(r.y, A.T));
                    sw[p] = w, st[p] = t;
                    if (p < 16) sw[ohw + p] = w, st[ohw + p] = t;
                }
            if (A.ptab)
                for (int i = threadIdx.x; i < ((c1 - c0) * phw + 3) / 4; i += kThreads)
                    reinterpret_cast<uint32_t *>(first)[i] = uint32_t(A.T) * 0x01010101u;
            __syncthreads();
            if (A.ptab)
            {
                // earliest t0 per (channel, cell): bytes updated through their word
                for (int p = threadIdx.x; p < ohw; p += kThreads)
                {
                    const int t0 = int(tsrc[p]), c = int(wsrc[p]);
                    if (t0 >= A.T || c < c0 || c >= c1) continue;
                    const int y = p / A.ow, x = p - y * A.ow, py = y / A.pky, px = x / A.pkx;
                    if (py >= A.poh || px >= A.pow_) continue;
                    const int idx = (c - c0) * phw + py * A.pow_ + px;
                    unsigned *word = reinterpret_cast<unsigned *>(first + (idx & ~3));
                    const int sh = 8 * (idx & 3);
                    unsigned old = *word;
                    while (int((old >> sh) & 0xFF) > t0)
                    {
                        const unsigned nw = (old & ~(0xFFu << sh)) | (unsigned(t0) << sh);
                        const unsigned seen = atomicCAS(word, old, nw);
                        if (seen == old) break;
                        old = seen;
                    }
                }
                __syncthreads();
            }
        }
        const int64_t slab = int64_t(A.C) * ohw, pslab = int64_t(A.C) * phw;
        write_range(A.spikes + smp * A.T * slab + int64_t(c0) * ohw, A.T, slab, (c1 - c0) * ohw, lean, ohw >= 16,
                    SpikeSource{wsrc, tsrc, ohw, c0});
        if (A.pooled)
        {
            uint8_t *dst = A.pooled + smp * A.T * pslab + int64_t(c0) * phw;
            if (A.ptab || !lean)
                write_range(dst, A.T, pslab, (c1 - c0) * phw, lean, true, TableSource{first});
            else
                for (int64_t i = threadIdx.x; i < int64_t(c1 - c0) * phw; i += kThreads)
                {
                    const int c = c0 + int(i / phw), cell = int(i % phw), py = cell / A.pow_, px = cell - py * A.pow_;
                    int m = A.T;
                    for (int dy = 0; dy < A.pky; ++dy)
                        for (int dx = 0; dx < A.pkx; ++dx)
                        {
                            const int q = (py * A.pky + dy) * A.ow + px * A.pkx + dx;
                            if (int(wsrc[q]) == c) m = min(m, int(tsrc[q]));
                        }
                    for (int t = 0; t < A.T; ++t) dst[t * pslab + i] = m <= t;
                }
        }
        __syncthreads();
    }
}
}  // namespace

void search_write(const SearchWrite &W, cudaStream_t s)
{
    const int64_t ohw = int64_t(W.oh) * W.ow, phw = W.pooled ? int64_t(W.poh) * W.pow_ : 0;
    WriteArgs A{W.records, nullptr, W.negw, W.flag, W.spikes, W.pooled, W.b, W.T, W.C, int(ohw), W.ow, W.pky, W.pkx,
                W.poh, W.pow_, W.C, 0};
    if (ohw > kSmemPixels)
    {
        A.codes = W.codes;
        search_codes_kernel<<<grid_for(W.b * ext_bytes(ohw), 256), 256, 0, s>>>(W.records, W.codes, W.b, int(ohw), W.T,
                                                                             W.negw, W.flag);
        SPK_LAUNCHED();
    }
    A.ptab = W.pooled && phw <= kTableMax ? 1 : 0;
    // Channel ranges: enough CTAs for a few per SM when there are few samples
    // (each CTA reads the whole map's records once more), as many as keep
    // the pooled table small and a range's bytes of a step below 2^31 (its
    // positions are 32-bit), in steps that keep the runs 16-byte aligned.
    int64_t g = 16, r = ohw;
    while (r) { const int64_t q = g % r; g = r, r = q; }  // gcd(16, ohw)
    const int64_t unit = 16 / g;
    const int64_t want = ceil_div(int64_t(sm_count()) * 6, W.b);
    int64_t nc = ceil_div(W.C, std::min<int64_t>(want, W.C));
    if (A.ptab && phw > 0) nc = std::min<int64_t>(nc, std::max<int64_t>(1, kTableBytes / phw));
    nc = std::min(nc, std::max<int64_t>(1, kRangeBytes / ohw));
    if (nc >= unit) nc = nc / unit * unit;
    else if (phw * unit <= kTableBytes && ohw * unit <= kRangeBytes) nc = std::min<int64_t>(unit, W.C);
    A.nc = int(nc);
    const size_t smem = (A.codes ? 0 : size_t(2 * ext_bytes(ohw))) + (A.ptab ? size_t(nc * phw + 32) & ~size_t(15) : 0);
    allow_smem(search_write_kernel, smem);
    const dim3 grid(unsigned(ceil_div(W.C, nc)), unsigned(std::min<int64_t>(W.b, 65535)));
    search_write_kernel<<<grid, kThreads, smem, s>>>(A);
    SPK_LAUNCHED();
}
}  // namespace spk
