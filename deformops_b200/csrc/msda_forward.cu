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

template <typename T, bool SOFTMAX, bool REF, bool SMALL, typename Index>
cudaError_t launch_as(const Params &p, cudaStream_t stream) {
    const size_t smem = forward_smem_bytes(p, SOFTMAX);
    auto kernel = forward_kernel<T, SOFTMAX, REF, SMALL, Index>;
    if (smem > kPlainSmem) {  // opt in to large dynamic shared memory only when needed
        cudaError_t e =
            cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
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

template <typename T, bool SOFTMAX, bool REF>
cudaError_t launch_sized(const Params &p, cudaStream_t stream) {
    // Up to four groups per SM the call lasts as long as one warp's chain of loads: more points in
    // flight per warp, and as few warps per CTA as still reach every SM.  Measured on B200, a
    // decoder's 300 queries of 16 points, kernel: 8.1 us against 6.3 (8 points in flight 6.1, 6 6.6;
    // of 12 points 6.9 against 6.0, 6.4, 5.9); nine groups per SM, 7.4 us, gain nothing.
    constexpr int kSms = 148;
    if (p.num_groups > 4 * kSms)
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
