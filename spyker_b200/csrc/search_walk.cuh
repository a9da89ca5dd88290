// The search of a lean layer (kSearch) by walking each pixel's inputs in spike
// order; included by conv_tc.cu.
//
// With no negative weight a channel's potential only grows with the inputs
// that have fired, so the first crossing of a pixel is found by adding its
// inputs' weights in the order of their first spikes until some channel is
// above the threshold: one launch instead of the bisection's rounds (about 20
// launches a layer, each waiting for the one before it), and no work after the
// crossing.  A warp takes a pixel: its inputs' first-spike bytes (8 channels of
// a tap per lane and load) are counted, a pixel whose inputs cannot reach the
// threshold even at the layer's largest weight leaves at once, the others'
// inputs are put in time order by a counting sort in shared memory (listing
// them step by step with a warp scan each took 122 us against 74 for 64 images
// of 28 x 28), and the lanes, one channel each (NG groups of 32), add the
// inputs' weights, U inputs in flight, comparing at the last input of each step.
//
// Bound by issue slots (the sort and the additions, some 1000 instructions a
// pixel) and, for few pixels, by the latency of one pixel: 2 -> 30 channels 5 x
// 5 on one image of 28 x 28 6.2 us, on 64 images 46 us; 30 -> 100 channels on
// one image of 14 x 14 13.5 us.  The rounds took about 115 us for each of them
// (64 images: 140 us) and win above some 100,000 pixels (walk_pays).
//
// Arithmetic: a channel's weights are the 32-bit integers floor(w 2^(32-e)),
// 2^e the smallest power of two above the largest (remainder bound and
// certification as for the tensor-core rounds' 31-bit ones), so a running sum
// is the exact term total R, in 64-bit integers and in any order.  A winner's
// value that the remainders leave open comes from an FP64 sum whose error bound
// rounds to one float; pixels with a decision (or such a sum) left open go to a
// list, and walk_exact_kernel bisects them with the oracle's ordered FP64 sums
// (with that bisection inside the walk the kernel kept a stack and spilled: 60
// us instead of 46).

// Bytes 1 where the first-spike byte f <= t, else 0; tt = (t + 1) * 0x01010101
// ((f | 0x80) - (t + 1) keeps bit 7 iff f > t, no borrow between bytes).
__device__ __forceinline__ uint32_t spike_bytes(uint32_t f, uint32_t tt)
{
    return (~((f | 0x80808080u) - tt) >> 7) & 0x01010101u;
}

// wd[k][cz]: the integers of input k (channels-last order, `kreal` of them)
// and channel n, echan / cscale as fixed_split_kernel's, the layer's largest
// weight to *wmax.  A CTA per channel.
__global__ void __launch_bounds__(256) walk_split_kernel(const float *__restrict__ kernel, uint32_t *__restrict__ wd,
                                                         int cout, int cin, int taps, int cpad, int cz,
                                                         float *__restrict__ echan, float *__restrict__ cscale,
                                                         int *__restrict__ negw, unsigned *__restrict__ wmax)
{
    __shared__ float s_mx[8];
    __shared__ double s_err[8];
    __shared__ int s_lsb[8];
    const int n = blockIdx.x, tid = threadIdx.x, K = cin * taps, kreal = taps * cpad;
    const float *row = kernel + int64_t(n) * K;
    float mx = 0.f;
    bool neg = false;
    int lsb = INT_MAX;  // exponent of the lowest set bit of any weight
    for (int k = tid; n < cout && k < K; k += blockDim.x)
    {
        const float w = row[k];
        mx = fmaxf(mx, fabsf(w));
        neg |= !(w >= 0.f && w < 1e30f);  // (also NaN, infinities: the dense kernel's)
        const uint32_t bits = __float_as_uint(w) & 0x7FFFFFFFu;
        if (bits != 0u && bits < 0x7F800000u)
        {
            const int ex = int(bits >> 23);
            const uint32_t sig = ex ? ((bits & 0x7FFFFFu) | 0x800000u) : bits;
            lsb = min(lsb, __ffs(int(sig)) - 1 + (ex ? ex : 1) - 150);
        }
    }
    for (int o = 16; o > 0; o >>= 1)
    {
        mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
        lsb = min(lsb, __shfl_xor_sync(0xffffffffu, lsb, o));
    }
    if ((tid & 31) == 0) s_mx[tid >> 5] = mx, s_lsb[tid >> 5] = lsb;
    if (neg) atomicOr(negw, 1);
    __syncthreads();
    mx = s_mx[0], lsb = s_lsb[0];
    for (int i = 1; i < 8; ++i) mx = fmaxf(mx, s_mx[i]), lsb = min(lsb, s_lsb[i]);
    int e = 0;
    if (mx > 0.f) frexpf(mx, &e);  // mx < 2^e
    e = max(-94, min(100, e));
    double err = 0.0;
    for (int k = tid; k < kreal; k += blockDim.x)
    {
        const int tap = k / cpad, c = k - tap * cpad;
        uint32_t d = 0;
        if (n < cout && c < cin)
        {
            const double w = fmax(double(row[c * taps + tap]), 0.0), r = ldexp(w, 32 - e), f = floor(r);
            d = f < 4294967296.0 ? uint32_t(f) : 0xFFFFFFFFu;
            err += ldexp(r - f, e - 32);
        }
        wd[int64_t(k) * cz + n] = d;
    }
    for (int o = 16; o > 0; o >>= 1) err += __shfl_xor_sync(0xffffffffu, err, o);
    if ((tid & 31) == 0) s_err[tid >> 5] = err;
    __syncthreads();
    if (tid != 0) return;
    err = s_err[0];
    for (int i = 1; i < 8; ++i) err += s_err[i];
    // the oracle's ordered FP64 sum is exact when every partial sum (a
    // multiple of 2^lsb, at most kreal 2^e) fits in 53 bits
    int lk = 0;
    while ((1 << lk) < kreal) ++lk;
    const bool exact64 = lsb == INT_MAX || e + lk - lsb <= 53;
    echan[n] = __double2float_ru(err + (exact64 ? 0.0 : double(kreal) * double(kreal) * ldexp(1.0, e - 52)));
    cscale[n] = ldexpf(1.f, e - 32);
    atomicMax(wmax, __float_as_uint(mx));
}

struct WalkSearch
{
    const uint32_t *wd;
    const float *kernel;
    const unsigned *wmax;
    int cz, groups;  // channel stride of wd; 8-channel groups of a receptive field
    double bound;    // F32(S) > thr as S > bound
    int *redo, *redo_count;  // pixels left to walk_exact_kernel
};

__device__ __forceinline__ float warp_max(float v)
{
    return order_dec(__reduce_max_sync(0xffffffffu, order_enc(v + 0.0f)));
}

// What a pixel's crossing step settles: the first channel of the largest
// potential, and its value when `need` (WTA keys).  Returns 0: not certain,
// 1: no channel above the threshold, 2: winner w; exact: v is the oracle's.
template <int NG>
__device__ __forceinline__ int walk_decide(const uint64_t (&acc)[NG], const float (&scale)[NG], const float (&err)[NG],
                                           float thr, int lane, int cout, int &w, float &v, bool &exact)
{
    float p[NG], lo[NG], hi[NG];
    float top = -INFINITY, himax = -INFINITY;
#pragma unroll
    for (int g = 0; g < NG; ++g)
    {
        s_round(double(acc[g]) * double(scale[g]), err[g], p[g], lo[g], hi[g]);
        if (lane + 32 * g >= cout) p[g] = lo[g] = hi[g] = -INFINITY;
        top = fmaxf(top, p[g]), himax = fmaxf(himax, hi[g]);
    }
    top = warp_max(top);
    himax = warp_max(himax);
    if (himax <= thr) return 1;
    // the first channel of the largest P
    unsigned at = 0xFFFFFFFFu;
#pragma unroll
    for (int g = NG - 1; g >= 0; --g)
        if (p[g] == top) at = unsigned(lane + 32 * g);
    at = __reduce_min_sync(0xffffffffu, at);
    float wlo = 0.f, whi = 0.f;
#pragma unroll
    for (int g = 0; g < NG; ++g)
        if (int(at >> 5) == g) wlo = lo[g], whi = hi[g];
    wlo = __shfl_sync(0xffffffffu, wlo, at & 31);
    whi = __shfl_sync(0xffffffffu, whi, at & 31);
    exact = wlo == whi;
    if (!(wlo > thr)) return 0;
    // another channel that can reach the winner, unless both are exact (then
    // P's order, first index on ties, is the oracle's)
    bool open = false;
#pragma unroll
    for (int g = 0; g < NG; ++g)
        open |= unsigned(lane + 32 * g) != at && hi[g] >= wlo && !(exact && lo[g] == hi[g]);
    if (__any_sync(0xffffffffu, open)) return 0;
    w = int(at), v = top;
    return 2;
}

template <int R, int NG>
__global__ void __launch_bounds__(256, NG <= 4 ? 2 : 1)
    search_walk_kernel(const __grid_constant__ TcParams P, const __grid_constant__ WalkSearch A)
{
    constexpr int U = NG <= 4 && R * NG < 16 ? 8 : 4;  // inputs in flight
    extern __shared__ __align__(16) uint16_t walk_smem[];
    if (*P.negw || *P.flag) return;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int T = P.T, cap = A.groups * 8;
    // per warp: 4 x 32 bins, a word per lane, then the list (bit 15: last input of its step)
    unsigned *bins = reinterpret_cast<unsigned *>(walk_smem) + warp * (160 + cap / 2);
    uint16_t *list = reinterpret_cast<uint16_t *>(bins + 160);
    const int qmax = min(8, P.cin);  // real bytes of a group (the others never fire)
    const float thr = P.thr;
    // this lane's groups: offset in the map, tap
    int goff[R], gyx[R];
    const int g8 = P.cpad / 8;
#pragma unroll
    for (int r = 0; r < R; ++r)
    {
        const int g = 32 * r + lane, tap = g / g8, c = (g - tap * g8) * 8, ky = tap / P.kw, kx = tap - ky * P.kw;
        goff[r] = (ky * P.w + kx) * P.cpad + c;
        gyx[r] = g < A.groups ? (ky | (kx << 16)) : -1;
    }
    // this lane's channels
    float scale[NG], err[NG];
    uint64_t above[NG];  // a total that may be above the threshold
    bool col[NG];
#pragma unroll
    for (int g = 0; g < NG; ++g)
    {
        const int c = lane + 32 * g;
        col[g] = c < A.cz;
        scale[g] = c < P.cout ? P.cscale[c] : 0.f;
        err[g] = c < P.cout ? P.echan[c] : 0.f;
        above[g] = ~uint64_t(0);
        if (c < P.cout)
        {
            // S >= R scale - (rounding of the bound): R at or below floor(x)
            // stays at or below the threshold for certain when E = 0; else
            // two units less
            const double x = (A.bound - double(err[g])) / double(scale[g]);
            if (x < 0.0)
                above[g] = 0;
            else if (x < 9e18)
            {
                const uint64_t f = uint64_t(floor(x));
                above[g] = err[g] == 0.f ? f + 1 : (f > 2 ? f - 2 - (f >> 48) : 0);
            }
        }
    }
    const float wmax = __uint_as_float(*A.wmax);
    const uint32_t fired = uint32_t(T) * 0x01010101u;  // spike_bytes at T - 1
    const int64_t step = int64_t(gridDim.x) * (blockDim.x >> 5);
    for (int64_t pix = int64_t(blockIdx.x) * (blockDim.x >> 5) + warp; pix < P.npix; pix += step)
    {
        const uint32_t smp = div_by(uint32_t(pix), P.ohw_m, P.ohw_sh), pp = uint32_t(pix) - smp * uint32_t(P.ohw);
        const int oy = int(div_by(pp, P.ow_m, P.ow_sh)), ox = int(pp) - oy * P.ow;
        const int iy0 = oy * P.sy - P.top, ix0 = ox * P.sx - P.left;
        const uint8_t *fm = P.in + int64_t(smp) * P.img_stride;
        const int org = (iy0 * P.w + ix0) * P.cpad;
        uint2 f[R];
        int n = 0;
#pragma unroll
        for (int r = 0; r < R; ++r)
        {
            const int iy = iy0 + (gyx[r] & 0xFFFF), ix = ix0 + (gyx[r] >> 16);
            f[r] = make_uint2(~0u, ~0u);
            if (gyx[r] >= 0 && iy >= 0 && iy < P.h && ix >= 0 && ix < P.w)
                f[r] = __ldg(reinterpret_cast<const uint2 *>(fm + org + goff[r]));
        }
#pragma unroll
        for (int r = 0; r < R; ++r) n += __popc(spike_bytes(f[r].x, fired)) + __popc(spike_bytes(f[r].y, fired));
        const int total = __reduce_add_sync(0xffffffffu, n);
        int t0 = T, w = 0;
        bool redo = false;  // left to walk_exact_kernel
        float v = P.thv;
        // (the widening covers the sum's roundings: K < 2^13 terms)
        if (float(total) * wmax * 1.001f > thr)
        {
            // counting sort by step: 4 bins per step (by lane), so that lanes
            // meet in fewer shared-memory atomics
#pragma unroll
            for (int i = 0; i < 5; ++i) bins[32 * i + lane] = 0;
            __syncwarp();
            unsigned *sub = bins + 32 * (lane & 3);
            // each input's rank in its bin (inputs that never fire count in a
            // word of the lane's own: no branches, so the atomics overlap)
            unsigned rank[R][4];
#pragma unroll
            for (int r = 0; r < R; ++r)
#pragma unroll
                for (int q = 0; q < 8; q += 2)
                {
                    if (q >= qmax) break;
                    const uint32_t word = q < 4 ? f[r].x : f[r].y;
                    const unsigned ta = (word >> (8 * (q & 3))) & 0xFFu, tb = (word >> (8 * (q & 3) + 8)) & 0xFFu;
                    const unsigned ra = atomicAdd(ta < unsigned(T) ? &sub[ta] : &bins[128 + lane], 1u);
                    const unsigned rb = atomicAdd(tb < unsigned(T) ? &sub[tb] : &bins[128 + lane], 1u);
                    rank[r][q / 2] = ra | (rb << 16);
                }
            __syncwarp();
            unsigned c4[4], cnt = 0;
#pragma unroll
            for (int i = 0; i < 4; ++i) c4[i] = bins[32 * i + lane], cnt += c4[i];
            unsigned incl = cnt;  // lane t: inputs up to step t
#pragma unroll
            for (int o = 1; o < 32; o <<= 1)
            {
                const unsigned x = __shfl_up_sync(0xffffffffu, incl, o);
                if (lane >= o) incl += x;
            }
            unsigned run = incl - cnt;
#pragma unroll
            for (int i = 0; i < 4; ++i) bins[32 * i + lane] = run, run += c4[i];
            __syncwarp();
#pragma unroll
            for (int r = 0; r < R; ++r)
#pragma unroll
                for (int q = 0; q < 8; ++q)
                {
                    if (q >= qmax) break;
                    const unsigned t = ((q < 4 ? f[r].x : f[r].y) >> (8 * (q & 3))) & 0xFFu;
                    const unsigned pos = sub[t & 31u] + ((rank[r][q / 2] >> (16 * (q & 1))) & 0xFFFFu);
                    if (t < unsigned(T)) list[pos] = uint16_t((32 * r + lane) * 8 + q);
                }
            __syncwarp();
            if (cnt) list[incl - 1] |= 0x8000u;
            __syncwarp();
            uint64_t acc[NG];
#pragma unroll
            for (int g = 0; g < NG; ++g) acc[g] = 0;
            bool exact = true;
            for (int base = 0; base < total && t0 == T && !redo; base += 32)
            {
                const unsigned mine = base + lane < total ? list[base + lane] : 0u;
                const unsigned ends = __ballot_sync(0xffffffffu, mine & 0x8000u);
                for (int i0 = 0; i0 < 32 && base + i0 < total && t0 == T && !redo; i0 += U)
                {
                    const unsigned batch = ends >> i0;
                    uint32_t d[U][NG];
#pragma unroll
                    for (int u = 0; u < U; ++u)
                    {
                        const uint32_t *row =
                            A.wd + (__shfl_sync(0xffffffffu, mine, i0 + u) & 0x7FFFu) * unsigned(A.cz) + lane;
#pragma unroll
                        for (int g = 0; g < NG; ++g) d[u][g] = col[g] && base + i0 + u < total ? __ldg(row + 32 * g) : 0u;
                    }
                    // add until the last input of a step that may be above the
                    // threshold
                    for (int u0 = 0; u0 < U;)
                    {
                        int ub = U;
#pragma unroll
                        for (int u = 0; u < U; ++u)
                        {
                            if (u < u0 || ub < U) continue;  // (uniform)
#pragma unroll
                            for (int g = 0; g < NG; ++g) acc[g] += d[u][g];
                            if ((batch >> u) & 1u)
                            {
                                bool maybe = false;
#pragma unroll
                                for (int g = 0; g < NG; ++g) maybe |= acc[g] >= above[g];
                                if (__any_sync(0xffffffffu, maybe)) ub = u;
                            }
                        }
                        if (ub == U) break;
                        u0 = ub + 1;
                        // the step whose last input this is
                        const int t = __popc(__ballot_sync(0xffffffffu, incl <= unsigned(base + i0 + ub) && lane < T));
                        int dec = walk_decide<NG>(acc, scale, err, thr, lane, P.cout, w, v, exact);
                        if (dec == 0)
                        {
                            redo = true;
                            break;
                        }
                        if (dec == 2)
                        {
                            t0 = t;
                            break;
                        }
                    }
                }
            }
            if (t0 < T && P.wta && !redo)
            {
                // the winner's total at T - 1: the lanes add the inputs left
                float vt = v;
                bool texact = exact;
                if (t0 < T - 1)
                {
                    uint64_t rest = 0, sum = 0;
                    // (the inputs listed after the crossing step's)
                    const int from = int(__shfl_sync(0xffffffffu, incl, t0));
                    for (int i0 = from + lane; i0 < total; i0 += 32 * 8)
                    {
                        uint32_t x[8];
#pragma unroll
                        for (int u = 0; u < 8; ++u)
                            x[u] = i0 + 32 * u < total
                                       ? __ldg(A.wd + (list[i0 + 32 * u] & 0x7FFFu) * unsigned(A.cz) + unsigned(w))
                                       : 0u;
#pragma unroll
                        for (int u = 0; u < 8; ++u) rest += x[u];
                    }
                    __syncwarp();
                    float sc = 0.f, er = 0.f;
#pragma unroll
                    for (int g = 0; g < NG; ++g)
                        if (w >> 5 == g) sum = acc[g], sc = scale[g], er = err[g];
                    sum = __shfl_sync(0xffffffffu, sum, w & 31);
                    sc = __shfl_sync(0xffffffffu, sc, w & 31), er = __shfl_sync(0xffffffffu, er, w & 31);
                    for (int o = 16; o > 0; o >>= 1) rest += __shfl_xor_sync(0xffffffffu, rest, o);
                    float lo, hi;
                    s_round(double(sum + rest) * double(sc), er, vt, lo, hi);
                    texact = lo == hi;
                }
                // Values left open: FP64 sums of the winner's weights by all
                // lanes.  Their error is below (K / 32 + 6) 2^-53 S, the
                // ordered sum's below K 2^-53 S.
                for (int pass = 0; pass < 2; ++pass)
                {
                    if (pass == 0 ? exact : texact) continue;
                    const int t = pass == 0 ? t0 : T - 1;
                    const uint32_t tt = uint32_t(t + 1) * 0x01010101u;
                    const float *wk = A.kernel + int64_t(w) * P.cin * P.kh * P.kw;
                    double s = 0.0;
#pragma unroll
                    for (int r = 0; r < R; ++r)
                    {
                        const uint32_t a = spike_bytes(f[r].x, tt), b = spike_bytes(f[r].y, tt);
                        const int g = 32 * r + lane, tap = g / g8, c = (g - tap * g8) * 8;
#pragma unroll 1
                        for (int q = 0; q < 8; ++q)
                            if (((q < 4 ? a : b) >> (8 * (q & 3))) & 1u) s += double(__ldg(wk + (c + q) * P.kh * P.kw + tap));
                    }
                    __syncwarp();
                    for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
                    float pv, lo, hi;
                    s_round(s, __double2float_ru(s * 0x1p-39), pv, lo, hi);
                    redo |= lo != hi;
                    if (lane == 0) atomicAdd(&g_recomputes, 1ull);
                    (pass == 0 ? v : vt) = pv;
                    if (pass == 0 && t0 == T - 1) vt = pv, texact = true;
                }
                if (lane == 0 && !redo) atomicMax(P.maxs + smp, order_enc(vt));
            }
            __syncwarp();
        }
        if (lane == 0 && redo)
            A.redo[atomicAdd(A.redo_count, 1)] = int(pix);
        else if (lane == 0)
        {
            P.records[pix] = t0 < T ? make_int4(w, t0, __float_as_int(v), 0) : make_int4(0, T, __float_as_int(P.thv), 0);
            // a step below the threshold leaves its value in the sample
            if (P.wta && t0 > 0 && P.thv != 0.f)
            {
                atomicMin(P.mins + smp, order_enc(P.thv));
                atomicMax(P.maxs + smp, order_enc(P.thv));
            }
        }
    }
}

// The pixels the walk left open, a warp each, from the oracle's sums: the first
// step at which some channel is above the threshold by bisection (potentials
// only grow), the first channel of the largest potential there, and with WTA
// its potential at T - 1.
__global__ void __launch_bounds__(128) walk_exact_kernel(TcParams P, WalkSearch A)
{
    if (*P.negw || *P.flag) return;
    const int lane = threadIdx.x & 31, T = P.T, n = *A.redo_count;
    for (int i = blockIdx.x * 4 + (threadIdx.x >> 5); i < n; i += gridDim.x * 4)
    {
        const int pix = A.redo[i], smp = pix / int(P.ohw), pp = pix - smp * int(P.ohw);
        const int oy = pp / P.ow, ox = pp - oy * P.ow, iy0 = oy * P.sy - P.top, ix0 = ox * P.sx - P.left;
        const uint8_t *fm = P.in + int64_t(smp) * P.img_stride;
        int lo = -1, hi = T - 1, t = T - 1, w = 0;
        float v = P.thv, vt = 0.f;
        bool fires = true, last = false;
        while (true)
        {
            // all channels at step t (the last round: the winner at T - 1)
            float best = -INFINITY;
            unsigned bi = 0xFFFFFFFFu;
            for (int o = lane; o < P.cout; o += 32)
            {
                if (last && o != w) continue;
                const float pv = float(oracle_sum(P, fm, A.kernel + int64_t(o) * P.cin * P.kh * P.kw, iy0, ix0, P.cpad, t));
                if (pv > best) best = pv, bi = unsigned(o);
            }
            __syncwarp();
            const float top = warp_max(best);
            bi = __reduce_min_sync(0xffffffffu, best == top ? bi : 0xFFFFFFFFu);
            if (last)
            {
                vt = top;
                break;
            }
            if (top > P.thr)
                hi = t, w = int(bi), v = top;
            else if (t == T - 1)
            {
                fires = false;
                break;
            }
            else
                lo = t;
            if (hi - lo > 1)
                t = (lo + hi) >> 1;
            else if (P.wta)
                last = true, t = T - 1;
            else
                break;
        }
        if (lane != 0) continue;
        atomicAdd(&g_recomputes, 1ull);
        P.records[pix] = fires ? make_int4(w, hi, __float_as_int(v), 0) : make_int4(0, T, __float_as_int(P.thv), 0);
        if (!P.wta) continue;
        if (fires) atomicMax(P.maxs + smp, order_enc(vt));
        if ((!fires || hi > 0) && P.thv != 0.f)
        {
            atomicMin(P.mins + smp, order_enc(P.thv));
            atomicMax(P.maxs + smp, order_enc(P.thv));
        }
    }
}

// The walk's launch for a layer of `groups` 8-channel groups per receptive
// field (at most 256) and up to 256 channels.
void launch_search_walk(const TcParams &P, const WalkSearch &A, cudaStream_t s)
{
    auto go = [&](auto kernel) {
        const size_t smem = size_t(8) * (160 + size_t(A.groups) * 4) * 4;
        int occ = 1;
        SPK_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, kernel, 256, smem));
        const int64_t grid = std::min<int64_t>(ceil_div(P.npix, 8), int64_t(sm_count()) * std::max(occ, 1));
        kernel<<<unsigned(grid), 256, smem, s>>>(P, A);
        SPK_LAUNCHED();
    };
    auto by_groups = [&](auto ng) {
        constexpr int NG = decltype(ng)::value;
        if (A.groups <= 32) go(search_walk_kernel<1, NG>);
        else if (A.groups <= 64) go(search_walk_kernel<2, NG>);
        else if (A.groups <= 128) go(search_walk_kernel<4, NG>);
        else go(search_walk_kernel<8, NG>);
    };
    if (P.cout <= 32) by_groups(std::integral_constant<int, 1>());
    else if (P.cout <= 64) by_groups(std::integral_constant<int, 2>());
    else if (P.cout <= 128) by_groups(std::integral_constant<int, 4>());
    else by_groups(std::integral_constant<int, 8>());
    // (the list of open pixels is almost always empty: a small grid)
    walk_exact_kernel<<<unsigned(std::min<int64_t>(ceil_div(P.npix, 4), 2 * sm_count())), 128, 0, s>>>(P, A);
    SPK_LAUNCHED();
}
