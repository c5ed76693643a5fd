// Forward kernel: out[b,q,g,:] = sum_{l,k} a[l,k] * bilinear(value_l, loc[l,k]).
//
// Replaces the reference's forward path
//   sources/deformops/backends/cuda/include/msda_forward.cuh:13-123 (kernel)
//   sources/deformops/backends/cuda/include/interpolate.cuh:14-72   (bilinear gather)
// with a design of its own.  A warp owns a group of 32/LPH (query, head) pairs - for
// bf16 heads of 32 channels, the 8 heads of one query.  Per group:
//   1. pre-pass: the lanes read the group's sampling locations and weights straight from
//      global memory (contiguous, streaming, each byte exactly once), and ONE lane per
//      point turns them into a 32-byte descriptor in shared memory: the four corner
//      offsets and the four corner weights already multiplied by the
//      attention weight (softmax-normalised on the fly when asked);
//   2. gather: each slot's lanes read their point's descriptor as two broadcast 16-byte
//      shared loads, issue the four corner loads (16 bytes per lane along the head
//      dimension; a corner outside the level has weight zero and its load is redirected to
//      the nearest pixel inside, so no value is ever blended in from a clamped position)
//      and accumulate in float32 with packed f32x2 FMAs;
//   3. one 16-byte streaming store per lane: a warp writes a query's G*D row contiguously.
// That is forward_kernel, which takes every call it is given.  Dense calls of 16-bit values take
// forward_wide_kernel, 32 bytes per lane and shuffles instead of descriptors, where forward_is_wide() says so.
#include "msda_common.cuh"

// tuning knobs (compile-time): points whose corner loads are in flight together, and the
// CTAs per SM the register allocation is held to
#ifndef MSDA_FWD_UNROLL
#define MSDA_FWD_UNROLL 2
#endif
#ifndef MSDA_FWD_MIN_CTAS
#define MSDA_FWD_MIN_CTAS 4
#endif
// the same for calls that do not fill the GPU: their time is one warp's chain of round trips
#ifndef MSDA_FWD_SMALL_UNROLL
#define MSDA_FWD_SMALL_UNROLL 4
#endif

namespace msda_b200 {

namespace {

// Index: what a (query, head) pair is numbered in.  Two 64-bit divisions per group were 2 % of the
// kernel; calls of 2^31 pairs and more keep them.
template <typename T, bool SOFTMAX, bool REF, bool SMALL, typename Index>
__global__ void __launch_bounds__(256, SMALL ? 2 : MSDA_FWD_MIN_CTAS) forward_kernel(const Params p) {
    using VT = VecTraits<T>;
    constexpr int V = VT::kVec;
    constexpr int NV2 = V / 2;
    constexpr int kUnroll = SMALL ? MSDA_FWD_SMALL_UNROLL : MSDA_FWD_UNROLL;
    extern __shared__ uint4 smem[];
    __shared__ LevelTable lt;

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int nwarps = blockDim.x >> 5;
    const int lph = 1 << p.lph_log2;
    const int ppw = 32 >> p.lph_log2;          // pairs per warp (group size)
    const int PC = p.point_chunk;
    const int DS = 2 * PC + 1;                 // uint4 stride between slots (odd: no bank conflicts)
    const int G = p.G, D = p.D, K = p.K;
    const int P = p.L * K;
    const int GD = G * D;
    const float inv_K = 1.f / (float)K;

    uint4 *desc = smem + (size_t)warp * desc_warp_vec(ppw, PC);                 // [slot][PC][2]
    float2 *stats = reinterpret_cast<float2 *>(smem + (size_t)nwarps * desc_warp_vec(ppw, PC)) +
                    warp * 32;                                              // softmax only

    load_level_table(lt, p);
    __syncthreads();

    const int64_t total_pairs = p.B * p.Q * G;
    const int slot = lane >> p.lph_log2;
    const int sub = lane & (lph - 1);
    const T *value = reinterpret_cast<const T *>(p.value);
    const T *attn = reinterpret_cast<const T *>(p.attn);
    T *out = reinterpret_cast<T *>(p.out);

    for (int64_t group = (int64_t)blockIdx.x * nwarps + warp; group < p.num_groups;
         group += (int64_t)gridDim.x * nwarps) {
        const int64_t pair0 = group * ppw;
        const int nlive = (int)min((int64_t)ppw, total_pairs - pair0);
        if constexpr (SOFTMAX) {
            const float2 st = slot_softmax_stats(attn + (pair0 + slot) * P, P, lph, sub, slot < nlive);
            if (sub == 0) stats[slot] = st;
            __syncwarp();
        }
        const bool live = slot < nlive;
        const int64_t my_pair = pair0 + (live ? slot : 0);
        const Index bq = (Index)my_pair / (Index)G;
        const int g = (int)((Index)my_pair - bq * (Index)G);
        const int64_t b = (int64_t)(bq / (Index)p.Q);
        const T *vb = value + (b * p.S * G + g) * (int64_t)D;

        float2 acc[NV2];
        for (int c0 = 0; c0 < P; c0 += PC) {
            const int pc = min(PC, P - c0);
            const float inv_pc = 1.f / (float)pc;
            // ---- pre-pass: one lane per (pair, point) builds the descriptor --------------
            for (int it = lane; it < ppw * pc; it += 32) {
                const int sl = (int)(((float)it + 0.5f) * inv_pc);   // it / pc
                const int j = it - sl * pc;
                const int pt = c0 + j;
                uint4 A = make_uint4(0u, 0u, 0u, 0u), Wt = make_uint4(0u, 0u, 0u, 0u);
                if (sl < nlive) {
                    const int64_t e = (pair0 + sl) * P + pt;
                    const int l = (int)(((float)pt + 0.5f) * inv_K);  // pt / K
                    const float2 xy = forward_location<T, REF, Index>(p, e, (Index)(pair0 + sl), l,
                                                                      (float)lt.W[l], (float)lt.H[l]);
                    float a = VT::to_float(attn[e]);
                    if constexpr (SOFTMAX) {
                        const float2 st = stats[sl];
                        a = expf(a - st.x) * st.y;
                    }
                    const PointGeom geo = locate(xy.x, xy.y, lt.H[l], lt.W[l], lt.start[l], GD);
                    // A corner outside the level keeps weight 0 and is pointed at the nearest
                    // pixel inside it, so the gather needs no predicates; a skipped point
                    // (geo.r0 = geo.c0 = 0, all weights 0) reads pixel (0, 0) of its level.
                    const int H = lt.H[l], W = lt.W[l];
                    // (an empty level has H = W = 0 and start 0: everything lands on pixel 0)
                    const int ra = max(geo.r0, 0), rb = max(min(geo.r0 + 1, H - 1), 0);
                    const int ca = max(geo.c0, 0), cb = max(min(geo.c0 + 1, W - 1), 0);
                    const int row_a = (lt.start[l] + ra * W) * GD, row_b = (lt.start[l] + rb * W) * GD;
                    A = make_uint4((unsigned)(row_a + ca * GD), (unsigned)(row_a + cb * GD),
                                   (unsigned)(row_b + ca * GD), (unsigned)(row_b + cb * GD));
                    const float wr0 = 1.f - geo.fr, wc0 = 1.f - geo.fc;
                    const unsigned f = geo.flags;
                    Wt = make_uint4(__float_as_uint(f & kCorner00 ? a * (wr0 * wc0) : 0.f),
                                    __float_as_uint(f & kCorner01 ? a * (wr0 * geo.fc) : 0.f),
                                    __float_as_uint(f & kCorner10 ? a * (geo.fr * wc0) : 0.f),
                                    __float_as_uint(f & kCorner11 ? a * (geo.fr * geo.fc) : 0.f));
                }
                desc[sl * DS + 2 * j] = A;
                desc[sl * DS + 2 * j + 1] = Wt;
            }
            __syncwarp();
            // ---- gather ------------------------------------------------------------------
            const uint4 *dp = desc + slot * DS;
            for (int ch = sub * V; ch < D; ch += lph * V) {
                if (c0 == 0) {
#pragma unroll
                    for (int i = 0; i < NV2; ++i) acc[i] = make_float2(0.f, 0.f);
                }
                const T *vc = vb + ch;
#pragma unroll kUnroll
                for (int j = 0; j < pc; ++j) {
                    const uint4 A = dp[2 * j];
                    const uint4 Wt = dp[2 * j + 1];
                    const uint4 r0 = ldg16(vc + (int)A.x);
                    const uint4 r1 = ldg16(vc + (int)A.y);
                    const uint4 r2 = ldg16(vc + (int)A.z);
                    const uint4 r3 = ldg16(vc + (int)A.w);
                    const uint4 raw[4] = {r0, r1, r2, r3};
                    const float w[4] = {__uint_as_float(Wt.x), __uint_as_float(Wt.y),
                                        __uint_as_float(Wt.z), __uint_as_float(Wt.w)};
#pragma unroll
                    for (int c = 0; c < 4; ++c) {
                        float2 f[NV2];
                        VT::unpack(raw[c], f);
                        const float2 w2 = make_float2(w[c], w[c]);
#pragma unroll
                        for (int i = 0; i < NV2; ++i) ffma2(acc[i], f[i], w2);
                    }
                }
                if (c0 + PC >= P && live) st_stream16(out + my_pair * D + ch, VT::pack(acc));
            }
            __syncwarp();
        }
    }
}

// ---- dense calls of 16-bit values: 32 bytes per lane --------------------------------------------
// The same sum with 32-byte loads: a slot is LPH = D / 16 lanes, a warp covers twice the pairs per
// instruction, and a point's numbers go from the lane that placed it to its slot by shuffles, so that
// all of the SM's memory that is not the level table stays L1.  It adds the same products in the same
// order: which of the two kernels a call takes does not show in its results.  What bounds it is what bounds
// forward_kernel, one wavefront of the L1 data pipe per 64-byte corner row (79 % busy at the headline
// shape, 4 x 21 504 queries of 12 points, 8 x 32 channels); of the rest a third of the wavefronts and a
// seventh of the instructions are gone, and L1 hits 40 % of the sectors instead of 29 %.
// Forward, B200, us, forward_kernel -> this: headline shape 164 -> 160, its 512-pixel pyramid 8 samples
// 86 -> 82, four odd levels in float16 185.5 -> 182, softmax and offsets 109 -> 96; 6 x 64 channels,
// 9 points, softmax and offsets 98 -> 82; 8 x 16 channels 129 -> 111; 2 x 128 149 -> 138.
// Three CTAs of 80 registers: four of 64 spill (175), seven of four warps at 72 164; two points in
// flight instead of one 160; one CTA per eight or sixteen groups instead of persistent ones 165, 168;
// the next points' locations loaded a turn early, no difference.  With adjacent points in one load,
// added in another order than forward_kernel's, 158 (float16 174.5).
constexpr int kWideWarps = 8;

template <typename T>
__device__ __forceinline__ void gather32(float2 (&acc)[8], const char *at, float w) {
    uint4 lo, hi;
    asm("ld.global.nc.v8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
        : "=r"(lo.x), "=r"(lo.y), "=r"(lo.z), "=r"(lo.w), "=r"(hi.x), "=r"(hi.y), "=r"(hi.z), "=r"(hi.w)
        : "l"(at));
    float2 f[4], g[4];
    VecTraits<T>::unpack(lo, f);
    VecTraits<T>::unpack(hi, g);
    const float2 w2 = make_float2(w, w);
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        ffma2(acc[i], f[i], w2);
        ffma2(acc[4 + i], g[i], w2);
    }
}

// The offsets or locations and the weights of PTS adjacent points (two: an even one first), in one load each.
template <typename T, bool REF, int PTS>
__device__ __forceinline__ void load_points(const Params &p, int64_t e, float2 (&spot)[PTS], float (&weight)[PTS]) {
    using VT = VecTraits<T>;
    const T *attn = reinterpret_cast<const T *>(p.attn) + e;
    if constexpr (PTS == 1) {
        spot[0] = REF ? load_offset<T>(p, e) : ld_stream_f2(reinterpret_cast<const float2 *>(p.loc) + e);
        weight[0] = VT::to_float(*attn);
    } else {
        if (REF && p.offsets16) {
            const uint2 v = __ldg(reinterpret_cast<const uint2 *>(reinterpret_cast<const uint32_t *>(p.loc) + e));
            spot[0] = VT::unpack2(v.x), spot[1] = VT::unpack2(v.y);
        } else {
            const uint4 v = ld_stream16(reinterpret_cast<const float2 *>(p.loc) + e);
            spot[0] = make_float2(__uint_as_float(v.x), __uint_as_float(v.y));
            spot[1] = make_float2(__uint_as_float(v.z), __uint_as_float(v.w));
        }
        const float2 w = VT::unpack2(__ldg(reinterpret_cast<const uint32_t *>(attn)));
        weight[0] = w.x, weight[1] = w.y;
    }
}

// slot_softmax_stats() of a slot of twice as many lanes, a lane doing the work of two: the same additions in
// the same order.
template <int LPH, typename T>
__device__ __forceinline__ float2 wide_softmax_stats(const T *logits, int P, int sub) {
    float m = -INFINITY;
    for (int i = sub; i < P; i += LPH) m = fmaxf(m, VecTraits<T>::to_float(logits[i]));
#pragma unroll
    for (int o = LPH >> 1; o > 0; o >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, o));
    float sum = 0.f, other = 0.f;
    for (int i = sub; i < P; i += 2 * LPH) sum += expf(VecTraits<T>::to_float(logits[i]) - m);
    for (int i = sub + LPH; i < P; i += 2 * LPH) other += expf(VecTraits<T>::to_float(logits[i]) - m);
    sum += other;
#pragma unroll
    for (int o = LPH >> 1; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
    return make_float2(m, 1.f / sum);
}

template <typename T, bool SOFTMAX, bool REF, int LPH, int PTS>
__global__ void __launch_bounds__(kWideWarps * 32, 3) forward_wide_kernel(const __grid_constant__ Params p) {
    using VT = VecTraits<T>;
    constexpr int kPairs = 32 / LPH;
    __shared__ LevelTable lt;
    load_level_table<REF>(lt, p);
    __syncthreads();
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int slot = lane / LPH, sub = lane % LPH;
    const int G = p.G, P = p.L * p.K;
    const unsigned row_bytes = (unsigned)G * (LPH * 32u);
    const float inv_K = 1.f / (float)p.K;
    const int64_t total_pairs = p.B * p.Q * G;
    const T *attn = reinterpret_cast<const T *>(p.attn);

    for (int64_t group = (int64_t)blockIdx.x * kWideWarps + warp; group < p.num_groups;
         group += (int64_t)gridDim.x * kWideWarps) {
        const int64_t pair0 = group * kPairs;
        const bool live = pair0 + slot < total_pairs;
        const int64_t pair = live ? pair0 + slot : total_pairs - 1;
        const unsigned bq = (unsigned)pair / (unsigned)G;
        const int g = (int)((unsigned)pair - bq * (unsigned)G);
        const int64_t b = bq / (unsigned)p.Q;
        const char *vb = reinterpret_cast<const char *>(p.value) + (b * p.S * (int64_t)row_bytes + g * (LPH * 32) + sub * 32);
        const int64_t e0 = pair * P;
        float2 stats = make_float2(0.f, 0.f);
        if constexpr (SOFTMAX) stats = wide_softmax_stats<LPH>(attn + e0, P, sub);
        float2 acc[8];
#pragma unroll
        for (int i = 0; i < 8; ++i) acc[i] = make_float2(0.f, 0.f);
#pragma unroll 1
        for (int r = 0; r < P; r += LPH * PTS) {
            // ---- each lane of the slot takes PTS points: adjacent ones where the slot is one lane, else
            // one of every LPH
            const int mine = r + sub * (LPH == 1 ? PTS : 1);
            float2 spot[PTS];
            float weight[PTS];
            if constexpr (LPH == 1) {
                if (mine < P) load_points<T, REF, PTS>(p, e0 + mine, spot, weight);
            } else {
#pragma unroll
                for (int i = 0; i < PTS; ++i) {
                    float2 one_spot[1];
                    float one_weight[1];
                    if (mine + i * LPH < P) load_points<T, REF, 1>(p, e0 + mine + i * LPH, one_spot, one_weight);
                    spot[i] = one_spot[0], weight[i] = one_weight[0];
                }
            }
#pragma unroll
            for (int i = 0; i < PTS; ++i) {
                const int pt = mine + i * (LPH == 1 ? 1 : LPH);
                int place = 0, down = 0;
                float w00 = 0.f, w01 = 0.f, w10 = 0.f, w11 = 0.f;
                if (pt < P) {
                    const int l = (int)(((float)pt + 0.5f) * inv_K);  // pt / K
                    const int H = lt.H[l], W = lt.W[l];
                    float2 xy = spot[i];
                    if constexpr (REF)
                        xy = location_from_offset(p, xy, (int64_t)bq, l, (float)W, (float)H, lt.rcp_w[l], lt.rcp_h[l]);
                    float a = weight[i];
                    if constexpr (SOFTMAX) a = expf(a - stats.x) * stats.y;
                    const PointGeom geo = locate(xy.x, xy.y, H, W, 0, 0);
                    const int ra = max(geo.r0, 0), rb = max(min(geo.r0 + 1, H - 1), 0);
                    const int ca = max(geo.c0, 0), cb = max(min(geo.c0 + 1, W - 1), 0);
                    // (a sample has fewer than 2^31 / 16 positions: one word holds the step right too)
                    place = (lt.start[l] + ra * W + ca) * 2 + (cb - ca);
                    down = (rb - ra) * W;
                    const float wr0 = 1.f - geo.fr, wc0 = 1.f - geo.fc;
                    const unsigned f = geo.flags;
                    w00 = f & kCorner00 ? a * (wr0 * wc0) : 0.f;
                    w01 = f & kCorner01 ? a * (wr0 * geo.fc) : 0.f;
                    w10 = f & kCorner10 ? a * (geo.fr * wc0) : 0.f;
                    w11 = f & kCorner11 ? a * (geo.fr * geo.fc) : 0.f;
                }
                // ---- and the slot gathers them, in the order of the points
#pragma unroll 1
                for (int j = 0; j < LPH; ++j) {
                    if (r + i * LPH + j >= P) break;
                    const int from = LPH == 1 ? 0 : (lane & ~(LPH - 1)) + j;
                    auto get = [&](auto v) { return LPH == 1 ? v : __shfl_sync(0xffffffffu, v, from); };
                    const int pl = get(place), dy = get(down);
                    const float a0 = get(w00), a1 = get(w01), a2 = get(w10), a3 = get(w11);
                    const char *top = vb + (uint64_t)((unsigned)(pl >> 1) * row_bytes);
                    const char *bot = top + (uint64_t)((unsigned)dy * row_bytes);
                    const unsigned right = pl & 1 ? row_bytes : 0u;
                    gather32<T>(acc, top, a0);
                    gather32<T>(acc, top + right, a1);
                    gather32<T>(acc, bot, a2);
                    gather32<T>(acc, bot + right, a3);
                }
            }
        }
        if (live) {
            char *o = reinterpret_cast<char *>(p.out) + pair * (LPH * 32) + sub * 32;
            st_stream16(o, VT::pack(reinterpret_cast<const float2(&)[4]>(acc[0])));
            st_stream16(o + 16, VT::pack(reinterpret_cast<const float2(&)[4]>(acc[4])));
        }
    }
}

template <typename T, bool SOFTMAX, bool REF, int LPH, int PTS>
cudaError_t launch_wide_as(const Params &p, cudaStream_t stream) {
    auto kernel = forward_wide_kernel<T, SOFTMAX, REF, LPH, PTS>;
    static Residency residency;
    Params q = p;
    q.num_groups = (p.B * p.Q * p.G + 32 / LPH - 1) / (32 / LPH);
    q.grid = (unsigned)((q.num_groups + kWideWarps - 1) / kWideWarps);
    const unsigned resident = residency.ctas(kernel, kWideWarps * 32, 0);
    if (resident > 0 && q.grid > resident) q.grid = resident;
    kernel<<<q.grid, kWideWarps * 32, 0, stream>>>(q);
    return cudaGetLastError();
}
template <typename T, bool SOFTMAX, bool REF, int LPH>
cudaError_t launch_wide(const Params &p, cudaStream_t stream) {
    // (two points a lane: their loads go out together.  Slots of four lanes are better off without, 84
    // us against 82 of the ragged pyramid)
    if constexpr (LPH < 4)
        if (LPH > 1 || p.L * p.K % 2 == 0) return launch_wide_as<T, SOFTMAX, REF, LPH, 2>(p, stream);
    return launch_wide_as<T, SOFTMAX, REF, LPH, 1>(p, stream);
}

template <typename T, bool SOFTMAX, bool REF, bool SMALL, typename Index>
cudaError_t launch_as(const Params &p, cudaStream_t stream) {
    const size_t smem = forward_smem_bytes(p, SOFTMAX);
    auto kernel = forward_kernel<T, SOFTMAX, REF, SMALL, Index>;
    if (smem > kPlainSmem) {  // opt in to large dynamic shared memory only when needed
        cudaError_t e = allow_most_smem(kernel);
        if (e != cudaSuccess) return e;
    }
    // Persistent CTAs: launch no more CTAs than the GPU holds at once and let each walk the
    // groups with the grid stride.  Measured on B200 at the headline shape: 0.175 ms against
    // 0.193 ms for one CTA per eight groups (the level table is loaded once per CTA instead of
    // eighteen times, and the resident CTAs sweep the queries as one compact front).
    static Residency residency;
    Params q = p;
    unsigned resident = residency.ctas(kernel, p.threads, smem);
#ifdef MSDA_FWD_CTAS_PER_SM
    resident = 148 * MSDA_FWD_CTAS_PER_SM;
#endif
    if (resident > 0 && q.grid > resident) q.grid = resident;
    kernel<<<q.grid, q.threads, smem, stream>>>(q);
    return cudaGetLastError();
}

// Up to four groups per SM a call lasts as long as one warp's chain of loads (launch_sized).
constexpr int kSms = 148;
bool small_call(const Params &p) { return p.num_groups <= 4 * kSms; }

}  // namespace

// 32-byte loads halve the warps of a call.  Where neighbouring queries sample neighbouring pixels, or
// all pixels are sampled often, L1 makes up for it; few queries far apart wait for L2 instead (us,
// forward_kernel -> forward_wide_kernel: 900 queries on 17 821 positions, 8 samples 32 -> 39; 1 800, 16
// samples 84 -> 87; 7 000 on 21 504, 8 samples 111 -> 109, 10 752 166 -> 158).  Of the dense calls the last
// round of the persistent warps decides, 24 per SM here and 32 there (what their launch bounds hold the
// registers to): a round of this kernel takes 1.38 times one of the other (12.2 against 8.8 us, 12 points of
// 32 channels), with offsets or a softmax 1.25 times.  Rounds of either, us: 2 and 3, 26.8 -> 24.7; 3 and 4,
// 37 -> 37, offsets of 64 channels 32.9 -> 30.9; 4 and 5, 46.2 -> 47.4, offsets 55.4 -> 53.9; 4 and 6, 57.9 ->
// 53.5.  Of many rounds the last counts for little: 7 and 10, 86 -> 82; 8 and 11 (64 channels) 75.7 -> 69.8; 13
// and 19, 164 -> 160.  16 channels gain throughout (22.7 -> 18.6 .. 129 -> 111).  float32 gains nothing (262 ->
// 273): its rows are whole lines of L1 either way.
// Over 32, 64 and 128 channels, 3 to 24 points and 2 to 8 samples of 5 376 queries, what the rule picks is
// never slower than forward_kernel by more than 2 % but once (128 channels, offsets, 3 and 4 rounds: 33.0 ->
// 34.9); calls of 3 points that it keeps from this kernel would gain up to a quarter (18.5 -> 14.6).
bool forward_is_wide(const Params &p, bool softmax) {
    if (small_call(p) || (p.D != 16 && p.D != 32 && p.D != 64 && p.D != 128)) return false;
    const int64_t pairs = p.B * p.Q * p.G;
    if ((reinterpret_cast<uintptr_t>(p.value) & 31u) != 0 || 2 * p.Q < p.S || pairs >= (int64_t)1 << 31) return false;
    if (p.D == 16) return true;
    const int64_t wide = kSms * 24 * (512 / p.D), other = kSms * 32 * (256 / p.D);     // pairs of a round
    const int64_t rounds = (pairs + wide - 1) / wide, other_rounds = (pairs + other - 1) / other;
    if (rounds > 6) return true;
    return softmax || p.ref != nullptr ? 5 * rounds <= 4 * other_rounds : 18 * rounds <= 13 * other_rounds;
}

namespace {

template <typename T, bool SOFTMAX, bool REF>
cudaError_t launch_sized(const Params &p, cudaStream_t stream) {
    // Small calls: more points in flight per warp, and as few warps per CTA as still reach every SM.
    // Measured on B200, a decoder's 300 queries of 16 points, kernel: 8.1 us against 6.3 (8 points in
    // flight 6.1, 6 6.6; of 12 points 6.9 against 6.0, 6.4, 5.9); nine groups per SM, 7.4 us, gain nothing.
    if constexpr (sizeof(T) == 2) {
        if (forward_is_wide(p, SOFTMAX)) {
            switch (p.D) {
                case 16: return launch_wide<T, SOFTMAX, REF, 1>(p, stream);
                case 32: return launch_wide<T, SOFTMAX, REF, 2>(p, stream);
                case 64: return launch_wide<T, SOFTMAX, REF, 4>(p, stream);
                case 128: return launch_wide<T, SOFTMAX, REF, 8>(p, stream);
            }
        }
    }
    if (!small_call(p))
        return p.B * p.Q * p.G < (int64_t)1 << 31 ? launch_as<T, SOFTMAX, REF, false, unsigned>(p, stream)
                                                  : launch_as<T, SOFTMAX, REF, false, int64_t>(p, stream);
    Params q = p;
    int warps = 1;
    while (warps < p.threads / 32 && warps * kSms < p.num_groups) warps *= 2;
    q.threads = warps * 32;
    q.grid = (unsigned)((p.num_groups + warps - 1) / warps);
    return launch_as<T, SOFTMAX, REF, true, unsigned>(q, stream);
}

template <typename T, bool SOFTMAX>
cudaError_t launch_typed(const Params &p, cudaStream_t stream) {
    return p.ref != nullptr ? launch_sized<T, SOFTMAX, true>(p, stream) : launch_sized<T, SOFTMAX, false>(p, stream);
}

}  // namespace

size_t forward_smem_bytes(const Params &p, bool softmax) {
    const size_t nwarps = p.threads / 32;
    return nwarps * desc_warp_vec(32 >> p.lph_log2, p.point_chunk) * 16 +
           (softmax ? nwarps * 32 * sizeof(float2) : 0);
}

cudaError_t launch_forward(const Params &p, int dtype, bool softmax, cudaStream_t stream) {
    switch (dtype) {
        case 0:
            return softmax ? launch_typed<float, true>(p, stream) : launch_typed<float, false>(p, stream);
        case 1:
            return softmax ? launch_typed<__half, true>(p, stream)
                           : launch_typed<__half, false>(p, stream);
        case 2:
            return softmax ? launch_typed<__nv_bfloat16, true>(p, stream)
                           : launch_typed<__nv_bfloat16, false>(p, stream);
        default: return cudaErrorInvalidValue;
    }
}

}  // namespace msda_b200
