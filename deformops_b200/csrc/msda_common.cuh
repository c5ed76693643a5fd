// Shared device helpers for the sm_100a multi-scale deformable attention kernels.
//
// Layouts (all contiguous, row-major):
//   value / grad_value   (B, S, G, D)            element type T (f32, f16, bf16)
//   spatial_shapes       (L, 2) int64, rows (H, W)      level_start_index (L) int64
//   loc / grad_loc       (B, Q, G, L, K, 2) float32, (x, y) = (width, height) axis
//   attn / grad_attn     (B, Q, G, L*K)         element type T
//   out / grad_out       (B, Q, G*D)            element type T
//
// Vocabulary
//   pair    one (batch*query, head) row: P = L*K sample points, D channels.
//   slot    the LPH lanes of a warp that own a pair; each lane owns one 16-byte vector of
//           channels (8 for 16-bit types, 4 for float).  A bf16 head of 32 channels is a
//           4-lane slot, so a warp covers the 8 heads of one query.
//   group   the 32/LPH pairs a warp processes together.
//   point descriptor   32 bytes in shared memory per (pair, point): element offset of the
//           top-left corner, row stride, validity flags and the interpolation weights.
//           Descriptors are computed once per point by one lane (a warp-wide pre-pass over
//           coalesced loc/attn loads) and then broadcast to the slot's lanes, so the
//           gather loop itself is loads, unpacks and FMAs only.
#pragma once

#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include <atomic>

namespace msda_b200 {

constexpr int kMaxLevels = 16;           // level table kept in shared memory
constexpr int kScratchHeaderBytes = 256;  // backward scratch: header (magnitude cells), then the image
constexpr int kDescPerWarp = 128;        // descriptors (32 B each) a warp holds at a time
// tuning knob (compile-time): most descriptors per pair a warp holds at a time; 0 = no cap
#ifndef MSDA_POINT_CHUNK_CAP
#define MSDA_POINT_CHUNK_CAP 0
#endif
// uint4 words of descriptor storage per warp: a row of 2 * point_chunk words per slot, padded by
// one word so that the 8 (or fewer) slots of a warp read their 16-byte descriptor halves from
// distinct banks.  Sized to what the call needs: shared memory a CTA does not take stays L1,
// and L1 hits are what the gather lacks.
__host__ __device__ inline int desc_warp_vec(int pairs_per_warp, int point_chunk) {
    return pairs_per_warp * (2 * point_chunk + 1);
}

struct Params {
    const void *value;
    const int64_t *spatial_shapes;
    const int64_t *level_start_index;
    const float *loc;
    const void *attn;
    void *out;              // forward only
    const void *grad_out;   // backward only
    void *grad_value;       // backward only
    float *grad_loc;        // backward only
    void *grad_attn;        // backward only
    void *scratch;          // backward only, 16-bit dtypes: header + scaled f16 image of grad_value, or null
    int64_t B, S, Q;
    int G, D, L, K;
    int lph_log2;           // log2(lanes per slot)
    int threads;            // threads per CTA (multiple of 32)
    int point_chunk;        // descriptors per pair held in shared memory at a time
    int64_t num_groups;     // ceil(B*Q*G / pairs per warp)
    unsigned grid;
    unsigned *fused_header;  // one-launch backward: FusedCell cells, zero at the start
    int passes;             // backward: adjacent sets of groups one CTA walks (0 or 1: one)
    // Fused location arithmetic.  When `ref` is set, `loc` / `grad_loc` hold the predicted
    // offsets (B,Q,G,L,K,2) and their gradient, and a point samples at
    //   ref_coords == 2:  ref.xy + offset / (W_l, H_l)
    //   ref_coords == 4:  ref.xy + offset / K * ref.wh * 0.5      (ref = cx, cy, w, h)
    const float *ref;       // (B,Q,L,ref_coords) float32, or null: `loc` holds locations
    int ref_coords;
    int offsets16;          // offsets and their gradient are stored in the 16-bit value dtype
};

// ---------------------------------------------------------------------------------
// 16-byte channel vectors, handled as float2 pairs for the packed f32x2 pipe
// ---------------------------------------------------------------------------------
template <typename T> struct VecTraits;

template <> struct VecTraits<float> {
    static constexpr int kVec = 4;
    __device__ static __forceinline__ void unpack(const uint4 &raw, float2 (&f)[2]) {
        f[0] = make_float2(__uint_as_float(raw.x), __uint_as_float(raw.y));
        f[1] = make_float2(__uint_as_float(raw.z), __uint_as_float(raw.w));
    }
    __device__ static __forceinline__ uint4 pack(const float2 (&f)[2]) {
        return make_uint4(__float_as_uint(f[0].x), __float_as_uint(f[0].y),
                          __float_as_uint(f[1].x), __float_as_uint(f[1].y));
    }
    __device__ static __forceinline__ float to_float(float v) { return v; }
    __device__ static __forceinline__ float from_float(float v) { return v; }
    // 16-byte reduction into global memory, no return value.  Reductions carry no "memory"
    // clobber: their targets are never read by the kernels, so gather loads of later
    // points may be scheduled above them.
    __device__ static __forceinline__ void red_add(void *addr, const float2 (&f)[2]) {
        asm volatile("red.relaxed.gpu.global.add.v4.f32 [%0], {%1, %2, %3, %4};" ::"l"(addr),
                     "f"(f[0].x), "f"(f[0].y), "f"(f[1].x), "f"(f[1].y));
    }
};

template <> struct VecTraits<__nv_bfloat16> {
    static constexpr int kVec = 8;
    __device__ static __forceinline__ void unpack(const uint4 &raw, float2 (&f)[4]) {
        // bf16 -> f32 is a 16-bit shift: low half by shl, high half by mask
        const uint32_t w[4] = {raw.x, raw.y, raw.z, raw.w};
#pragma unroll
        for (int i = 0; i < 4; ++i)
            f[i] = make_float2(__uint_as_float(w[i] << 16), __uint_as_float(w[i] & 0xffff0000u));
    }
    __device__ static __forceinline__ float2 unpack2(uint32_t w) {
        return make_float2(__uint_as_float(w << 16), __uint_as_float(w & 0xffff0000u));
    }
    __device__ static __forceinline__ uint32_t pack2(float2 v) {
        uint32_t r;  // cvt packs {upper, lower} with round-to-nearest-even
        asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(r) : "f"(v.y), "f"(v.x));
        return r;
    }
    __device__ static __forceinline__ uint4 pack(const float2 (&f)[4]) {
        return make_uint4(pack2(f[0]), pack2(f[1]), pack2(f[2]), pack2(f[3]));
    }
    __device__ static __forceinline__ float to_float(__nv_bfloat16 v) { return __bfloat162float(v); }
    __device__ static __forceinline__ __nv_bfloat16 from_float(float v) {
        return __float2bfloat16_rn(v);
    }
    // one 16-byte packed reduction (eight bf16 adds) instead of four bf16x2 atomics
    __device__ static __forceinline__ void red_add(void *addr, const float2 (&f)[4]) {
        const uint4 p = pack(f);
        asm volatile("red.relaxed.gpu.global.add.noftz.v4.bf16x2 [%0], {%1, %2, %3, %4};" ::"l"(
                         addr),
                     "r"(p.x), "r"(p.y), "r"(p.z), "r"(p.w));
    }
};

template <> struct VecTraits<__half> {
    static constexpr int kVec = 8;
    __device__ static __forceinline__ void unpack(const uint4 &raw, float2 (&f)[4]) {
        const uint32_t w[4] = {raw.x, raw.y, raw.z, raw.w};
#pragma unroll
        for (int i = 0; i < 4; ++i) f[i] = __half22float2(*reinterpret_cast<const __half2 *>(&w[i]));
    }
    __device__ static __forceinline__ float2 unpack2(uint32_t w) {
        return __half22float2(*reinterpret_cast<const __half2 *>(&w));
    }
    __device__ static __forceinline__ uint32_t pack2(float2 v) {
        const __half2 h = __float22half2_rn(v);
        return *reinterpret_cast<const uint32_t *>(&h);
    }
    __device__ static __forceinline__ uint4 pack(const float2 (&f)[4]) {
        return make_uint4(pack2(f[0]), pack2(f[1]), pack2(f[2]), pack2(f[3]));
    }
    __device__ static __forceinline__ float to_float(__half v) { return __half2float(v); }
    __device__ static __forceinline__ __half from_float(float v) { return __float2half_rn(v); }
    __device__ static __forceinline__ void red_add(void *addr, const float2 (&f)[4]) {
        const uint4 p = pack(f);
        asm volatile("red.relaxed.gpu.global.add.noftz.v4.f16x2 [%0], {%1, %2, %3, %4};" ::"l"(
                         addr),
                     "r"(p.x), "r"(p.y), "r"(p.z), "r"(p.w));
    }
};

// predicated packed reductions: one instruction, no branch
template <typename T>
__device__ __forceinline__ void red_if(T *addr, const float2 (&g)[VecTraits<T>::kVec / 2], bool pred);

template <>
__device__ __forceinline__ void red_if<float>(float *addr, const float2 (&g)[2], bool pred) {
    asm volatile("{\n\t.reg .pred q;\n\tsetp.ne.u32 q, %5, 0;\n\t"
                 "@q red.relaxed.gpu.global.add.v4.f32 [%0], {%1, %2, %3, %4};\n\t}" ::"l"(addr),
                 "f"(g[0].x), "f"(g[0].y), "f"(g[1].x), "f"(g[1].y), "r"((unsigned)pred));
}
template <>
__device__ __forceinline__ void red_if<__nv_bfloat16>(__nv_bfloat16 *addr, const float2 (&g)[4],
                                                      bool pred) {
    const uint4 v = VecTraits<__nv_bfloat16>::pack(g);
    asm volatile("{\n\t.reg .pred q;\n\tsetp.ne.u32 q, %5, 0;\n\t"
                 "@q red.relaxed.gpu.global.add.noftz.v4.bf16x2 [%0], {%1, %2, %3, %4};\n\t}" ::"l"(
                     addr),
                 "r"(v.x), "r"(v.y), "r"(v.z), "r"(v.w), "r"((unsigned)pred));
}
template <>
__device__ __forceinline__ void red_if<__half>(__half *addr, const float2 (&g)[4], bool pred) {
    const uint4 v = VecTraits<__half>::pack(g);
    asm volatile("{\n\t.reg .pred q;\n\tsetp.ne.u32 q, %5, 0;\n\t"
                 "@q red.relaxed.gpu.global.add.noftz.v4.f16x2 [%0], {%1, %2, %3, %4};\n\t}" ::"l"(
                     addr),
                 "r"(v.x), "r"(v.y), "r"(v.z), "r"(v.w), "r"((unsigned)pred));
}

// packed two-wide float32 arithmetic (sm_100): one issue slot for two lanes of work
__device__ __forceinline__ void ffma2(float2 &acc, const float2 a, const float2 b) {
    asm("fma.rn.f32x2 %0, %1, %2, %0;"
        : "+l"(reinterpret_cast<unsigned long long &>(acc))
        : "l"(reinterpret_cast<const unsigned long long &>(a)),
          "l"(reinterpret_cast<const unsigned long long &>(b)));
}
__device__ __forceinline__ float2 fmul2(const float2 a, const float2 b) {
    float2 r;
    asm("mul.rn.f32x2 %0, %1, %2;"
        : "=l"(reinterpret_cast<unsigned long long &>(r))
        : "l"(reinterpret_cast<const unsigned long long &>(a)),
          "l"(reinterpret_cast<const unsigned long long &>(b)));
    return r;
}

// read-only 16-byte gather load
__device__ __forceinline__ uint4 ldg16(const void *p) {
    return __ldg(reinterpret_cast<const uint4 *>(p));
}

// load instruction of the backward's corner gather (a tuning knob: cache operators and
// eviction hints can be swapped in at compile time)
#ifndef MSDA_BWD_GATHER_LD
#define MSDA_BWD_GATHER_LD "ld.global.nc.v4.u32"
#endif

// Read-only 16-byte gather load, predicated: returns zeros and touches no memory when
// `pred` is false.  Not volatile, so the compiler may batch the loads of several points.
__device__ __forceinline__ uint4 ldg16_if(const void *p, bool pred) {
    uint4 r;
    asm("{\n\t.reg .pred q;\n\tsetp.ne.u32 q, %5, 0;\n\tmov.u32 %0, 0;\n\tmov.u32 %1, 0;\n\t"
        "mov.u32 %2, 0;\n\tmov.u32 %3, 0;\n\t@q " MSDA_BWD_GATHER_LD " {%0, %1, %2, %3}, [%4];\n\t}"
        : "=&r"(r.x), "=&r"(r.y), "=&r"(r.z), "=&r"(r.w)
        : "l"(p), "r"((unsigned)pred));
    return r;
}

// streaming loads/stores for operands touched exactly once (loc, attn, out, grads): keeps
// them from displacing the value tensor in L1/L2
__device__ __forceinline__ float2 ld_stream_f2(const float2 *p) {
    float2 r;
    asm volatile("ld.global.cs.v2.f32 {%0, %1}, [%2];" : "=f"(r.x), "=f"(r.y) : "l"(p));
    return r;
}
// Programmatic dependent launch.  A kernel launched with launch_after_predecessor() may become
// resident while the kernel before it in the stream is still draining; it must pass
// grid_dependency_wait() before it touches anything that kernel writes (the wait returns once
// the predecessor has completed and its writes are visible).  grid_launch_dependents() lets the
// next such kernel in: it takes effect once every CTA of this grid has issued it or exited.
// In a kernel launched the ordinary way both are no-ops.
__device__ __forceinline__ void grid_dependency_wait() {
    asm volatile("griddepcontrol.wait;" ::: "memory");
}
__device__ __forceinline__ void grid_launch_dependents() {
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}

// For calls of a million points and more (backward of the headline shape in three kernels 0.530 -> 0.525 ms).
// Smaller ones gain or lose by what the kernel before leaves them of the SMs, the host being no worse off
// either way (backward, us a call, ordinary launches -> dependent ones: 4 samples of 32x32, 16x16, 8x8 57.5 ->
// 52.4; on 17 821 positions of four levels 4 samples of 900 queries 68.2 -> 63.9, one of 3 000 48.9 -> 52.8, 8 of
// 300 78.6 -> 82.8).
inline bool worth_dependent_launch(const Params &p) {
    return p.B * p.Q * p.G * (int64_t)(p.L * p.K) >= ((int64_t)1 << 20);
}

template <typename Kernel, typename... More>
inline cudaError_t launch_after_predecessor(Kernel kernel, unsigned grid, unsigned threads, size_t smem,
                                            cudaStream_t stream, const Params &p, const More &...more) {
    if (!worth_dependent_launch(p)) {
        kernel<<<grid, threads, smem, stream>>>(p, more...);
        return cudaGetLastError();
    }
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(grid, 1, 1);
    cfg.blockDim = dim3(threads, 1, 1);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, kernel, p, more...);
}

// Shared memory a kernel may ask for without opting in, beside the level table and the like that
// these kernels hold statically.
constexpr size_t kPlainSmem = 46 * 1024;
// The most any call asks for (more than this is refused).  A kernel that may need more than kPlainSmem is
// always allowed all of it: with the size of the call at hand, two host threads whose calls differ
// would lower each other's limit between setting it and launching, and the launch would be refused.
constexpr size_t kMostSmem = 200 * 1024;
template <typename Kernel>
inline cudaError_t allow_most_smem(Kernel kernel) {
    return cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kMostSmem);
}

// CTAs of a kernel the GPU holds at once for a block size and a shared memory size.  The runtime is
// asked once per combination (a query costs the host about as much as a launch).  Every GPU this
// is built for answers alike; where fewer SMs can be had, grids sized by it run in more waves.
class Residency {
  public:
    template <typename Kernel>
    unsigned ctas(Kernel kernel, int threads, size_t smem) {
        const uint64_t key = (uint64_t)smem << 12 | (uint64_t)threads;
        const uint64_t known = last_.load(std::memory_order_relaxed);
        if (known >> 24 == key) return (unsigned)(known & 0xffffffu);
        int device = 0, sms = 0, per_sm = 0;
        if (cudaGetDevice(&device) != cudaSuccess ||
            cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device) != cudaSuccess ||
            cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, threads, smem) != cudaSuccess)
            return 0;
        const unsigned resident = (unsigned)sms * (unsigned)per_sm;
        last_.store(key << 24 | resident, std::memory_order_relaxed);
        return resident;
    }

  private:
    std::atomic<uint64_t> last_{0};
};

__device__ __forceinline__ uint4 ld_stream16(const void *p) {
    uint4 r;
    asm volatile("ld.global.cs.v4.u32 {%0, %1, %2, %3}, [%4];"
                 : "=r"(r.x), "=r"(r.y), "=r"(r.z), "=r"(r.w)
                 : "l"(p));
    return r;
}
__device__ __forceinline__ void st_stream16(void *p, const uint4 &v) {
    asm volatile("st.global.cs.v4.u32 [%0], {%1, %2, %3, %4};" ::"l"(p), "r"(v.x), "r"(v.y),
                 "r"(v.z), "r"(v.w));
}
__device__ __forceinline__ void st_stream_f2(float2 *p, float2 v) {
    asm volatile("st.global.cs.v2.f32 [%0], {%1, %2};" ::"l"(p), "f"(v.x), "f"(v.y));
}

// ---------------------------------------------------------------------------------
// Scaled float16 accumulation of a 16-bit grad_value
// ---------------------------------------------------------------------------------
// With a scratch buffer the 16-bit backward does not add into grad_value itself.  Every
// contribution is multiplied by one power of two, 2^e, rounded to float16 and added (packed
// red.global.add.f16x2) into a float16 image of grad_value that lives in the scratch; a last
// pass multiplies by 2^-e and writes grad_value in its own type.  float16 keeps 11 significant
// bits per addition where bfloat16 keeps 8, and the scale puts the sums where float16 can hold
// them: e is chosen from the largest |grad_out| and |attn| element of the call (found on the
// device, no host read) so that even Q*K contributions of the largest possible magnitude -
// the most one element can receive - stay below the float16 maximum.
//
// A float16 sum of n terms still loses about sqrt(n) * 2^-12 of its value, and the coarsest
// level of a pyramid can receive more than a thousand additions per element.  A level whose
// elements receive n = 4*K*Q / (H*W) > kAddsPerAccumulator additions on average is therefore
// given R = ceil(n / kAddsPerAccumulator) accumulators per element: the image itself plus R-1
// replicas of the level in a per-sample block of "extras"; a point adds into replica
// (query + point) mod R and the last pass sums them in float32.  Such levels are small by
// construction: all extras of a sample take at most L * K*Q*G*D / 64 elements.
//
// Scratch layout: kScratchHeaderBytes of header, then the image, B*S*G*D float16, then B blocks
// of extra_elems_per_sample() float16.  Header cell 0 / 1: the 15 magnitude bits of the largest
// |grad_out| / |attn| element (16-bit patterns order like their magnitudes; a NaN sorts above
// everything and switches the scaling off).
constexpr int kAddsPerAccumulator = 256;
constexpr int kMaxReplicas = 64;

__host__ __device__ inline int64_t extra_elems_per_sample(int64_t Q, int64_t G, int64_t D,
                                                         int64_t L, int64_t K) {
    return L * ((((K * Q * G * D + 63) / 64) + 7) & ~(int64_t)7);   // whole 16-byte vectors
}
template <typename T>
__device__ __forceinline__ float magnitude_from_bits(unsigned bits);
template <>
__device__ __forceinline__ float magnitude_from_bits<__nv_bfloat16>(unsigned bits) {
    return __uint_as_float(bits << 16);
}
template <>
__device__ __forceinline__ float magnitude_from_bits<__half>(unsigned bits) {
    return __half2float(__ushort_as_half((unsigned short)bits));
}

template <typename T>
__device__ __forceinline__ int grad_scale_exponent(const unsigned *header, int64_t Q, int K,
                                                   bool softmax) {
    const float mg = magnitude_from_bits<T>(header[0]);
    const float ma = softmax ? 1.f : magnitude_from_bits<T>(header[1]);   // probabilities are <= 1
    const float bound = mg * ma * (float)Q * (float)K;
    if (!(bound > 0.f) || !(bound < INFINITY)) return 0;   // all zero, or inf / NaN in the inputs
    const int e = 14 - ilogbf(bound);                      // bound * 2^e in [2^14, 2^15)
    return e < -100 ? -100 : (e > 100 ? 100 : e);
}

// largest magnitude pattern among the eight 16-bit elements of a vector
__device__ __forceinline__ unsigned max_magnitude_bits(const uint4 &v) {
    const unsigned a = __vmaxu2(v.x & 0x7fff7fffu, v.y & 0x7fff7fffu);
    const unsigned b = __vmaxu2(v.z & 0x7fff7fffu, v.w & 0x7fff7fffu);
    const unsigned m = __vmaxu2(a, b);
    return max(m & 0xffffu, m >> 16);
}

// largest magnitude pattern over vectors first, first + stride, ... of `p`: four loads in flight
__device__ __forceinline__ unsigned scan_max_magnitude(const uint4 *__restrict__ p, int64_t n,
                                                       int64_t first, int64_t stride) {
    unsigned m = 0;
    int64_t v = first;
    for (; v + 3 * stride < n; v += 4 * stride) {
        const uint4 a = p[v], b = p[v + stride], c = p[v + 2 * stride], d = p[v + 3 * stride];
        m = max(max(m, max(max_magnitude_bits(a), max_magnitude_bits(b))),
                max(max_magnitude_bits(c), max_magnitude_bits(d)));
    }
    for (; v < n; v += stride) m = max(m, max_magnitude_bits(p[v]));
    return m;
}

// ---------------------------------------------------------------------------------
// Level table -> shared memory (read from device memory: no host synchronisation)
// ---------------------------------------------------------------------------------
struct LevelTable {
    int H[kMaxLevels];
    int W[kMaxLevels];
    int start[kMaxLevels];          // first position of the level on the S axis
    int rowstride[kMaxLevels];      // elements between image rows: W * G * D
    float rcp_w[kMaxLevels], rcp_h[kMaxLevels];   // 1 / W, 1 / H, for location_from_offset()
    // scaled float16 backward: accumulators per element of the level (1 = the image only) and
    // where the level's additional replicas start in a sample's block of extras
    int rep[kMaxLevels];
    unsigned rep_base[kMaxLevels];
    unsigned level_elems[kMaxLevels];   // H * W * G * D
};

// Accumulators per level for the scaled float16 backward (see above); every kernel of a call
// derives the same plan from the same level table.  (R-1) * H*W*G*D <= K*Q*G*D / 64 per level,
// so the extras always fit the block extra_elems_per_sample() reserves.
__device__ inline void plan_replicas(LevelTable &t, const Params &p) {
    const long long n4 = 4ll * p.K * p.Q;
    unsigned base = 0;
    for (int l = 0; l < p.L; ++l) {
        const long long hw = (long long)t.H[l] * t.W[l];
        long long r = hw > 0 ? (n4 + kAddsPerAccumulator * hw - 1) / (kAddsPerAccumulator * hw) : 1;
        r = r < 1 ? 1 : (r > kMaxReplicas ? kMaxReplicas : r);
        t.rep[l] = (int)r;
        t.rep_base[l] = base;
        base += (unsigned)(r - 1) * t.level_elems[l];
    }
}

// Loads the level table from device memory.  A level that does not lie inside the value tensor
// (non-positive size, negative start, or start + H*W beyond S) becomes an empty level at
// position 0: every point on it is skipped, so a malformed table produces zeros for that level
// instead of an access outside `value` / `grad_value`.
// RECIPROCALS: rcp_w, rcp_h too (a small call lasts as long as one warp's chain, and feels two divisions).
template <bool RECIPROCALS = false>
__device__ __forceinline__ void load_level_table(LevelTable &t, const Params &p) {
    if (threadIdx.x < p.L) {
        const int64_t h = p.spatial_shapes[2 * threadIdx.x];
        const int64_t w = p.spatial_shapes[2 * threadIdx.x + 1];
        const int64_t first = p.level_start_index[threadIdx.x];
        const bool fits = h > 0 && w > 0 && first >= 0 && h <= p.S && w <= p.S &&
                          h * w <= p.S && first <= p.S - h * w;
        const int H = fits ? (int)h : 0, W = fits ? (int)w : 0;
        t.H[threadIdx.x] = H;
        t.W[threadIdx.x] = W;
        t.start[threadIdx.x] = fits ? (int)first : 0;
        t.rowstride[threadIdx.x] = W * p.G * p.D;
        if constexpr (RECIPROCALS) {
            t.rcp_w[threadIdx.x] = 1.f / (float)W;
            t.rcp_h[threadIdx.x] = 1.f / (float)H;
        }
        t.level_elems[threadIdx.x] = (unsigned)H * (unsigned)W * (unsigned)(p.G * p.D);
    }
}

// ---------------------------------------------------------------------------------
// Point geometry -> descriptor
// ---------------------------------------------------------------------------------
enum : unsigned {
    kCorner00 = 1u, kCorner01 = 2u, kCorner10 = 4u, kCorner11 = 8u,  // corner inside the level
    kInside = 16u,       // point passes -1 <= pixel < size on both axes (NaN / inf fail)
    kUseExtra = 32u,     // backward: this point adds into a replica in the extras, not the image
    kLevelShift = 8,     // bits 8.. of the flags word carry the level index (backward)
};

struct PointGeom {
    int off00;       // element offset of corner (r0, c0) from the sample's first element
    int rowstride;   // elements between image rows of this level: W * G * D
    unsigned flags;
    int r0, c0;      // integer pixel of corner (r0, c0); -1 is possible on either axis
    float fr, fc;    // fractional parts along height / width
    float Hf, Wf;
};

// pixel = loc * size - 0.5 in float32; corners outside the level are flagged off, never
// clamped; a point outside [-1, size) on either axis is skipped altogether.
__device__ __forceinline__ PointGeom locate(float x, float y, int H, int W, int start, int GD) {
    PointGeom g;
    g.Hf = (float)H;
    g.Wf = (float)W;
    const float px = fmaf(x, g.Wf, -0.5f);
    const float py = fmaf(y, g.Hf, -0.5f);
    // (an empty level, H == 0, skips everything: see load_level_table)
    const bool inside = (py >= -1.f) && (px >= -1.f) && (py < g.Hf) && (px < g.Wf) && H > 0;
    // keep the arithmetic finite for skipped points (their loads are predicated off)
    const float sx = inside ? px : 0.f;
    const float sy = inside ? py : 0.f;
    const float r0f = floorf(sy), c0f = floorf(sx);
    const int r0 = (int)r0f, c0 = (int)c0f;
    g.fr = sy - r0f;
    g.fc = sx - c0f;
    const bool r_ok0 = inside && r0 >= 0, r_ok1 = inside && r0 + 1 < H;
    const bool c_ok0 = c0 >= 0, c_ok1 = c0 + 1 < W;
    g.flags = (r_ok0 && c_ok0 ? kCorner00 : 0u) | (r_ok0 && c_ok1 ? kCorner01 : 0u) |
              (r_ok1 && c_ok0 ? kCorner10 : 0u) | (r_ok1 && c_ok1 ? kCorner11 : 0u) |
              (inside ? kInside : 0u);
    g.r0 = r0;
    g.c0 = c0;
    g.off00 = (start + r0 * W + c0) * GD;
    g.rowstride = W * GD;
    return g;
}

// Location of a predicted offset, in the float32 arithmetic of the torch expressions of the
// layers it replaces: `ref + offset / (W, H)` and `ref.xy + offset / K * ref.wh * 0.5`.
__device__ __forceinline__ float2 location_from_offset(const Params &p, float2 off, int64_t bq, int l,
                                                       float Wf, float Hf) {
    if (p.ref_coords == 2) {
        const float2 r = __ldg(reinterpret_cast<const float2 *>(p.ref) + bq * p.L + l);
        return make_float2(r.x + off.x / Wf, r.y + off.y / Hf);
    }
    const float4 r = __ldg(reinterpret_cast<const float4 *>(p.ref) + bq * p.L + l);
    const float Kf = (float)p.K;
    return make_float2(r.x + off.x / Kf * r.z * 0.5f, r.y + off.y / Kf * r.w * 0.5f);
}
// x / n for a whole number n and rcp = 1 / n, in three instructions: Markstein's correction of an
// approximate quotient by its remainder ("Computation of elementary functions on the IBM RISC System/6000",
// 1990).  For n below 2^20, q is at most two units in its last place off and the remainder, a multiple of
// that unit below 2^22 of them, exact; a quotient by such an n lies at least 2^-21 units from a rounding
// boundary, what the correction loses is 2^-23.  So the result is the quotient rounded to nearest, as
// the division gives it; where q leaves the normal range, or x is no number, a location so far off or so
// near its reference point that the pixel coordinate is the same.  For larger n, which only the wide forward
// meets, that is no proof, but 10^8 quotients within a few 2^-24 units of a boundary, or by an n whose
// reciprocal is furthest off, are all rounded right.
__device__ __forceinline__ float quotient(float x, float n, float rcp) {
    const float q = x * rcp;
    return fmaf(fmaf(-q, n, x), rcp, q);
}
// The same location without divisions (offsets at the headline shape, us: forward 186.1 -> 183.9,
// backward, whose sort kernels use it, 492.5 -> 487.2; ragged pyramid 194.8 -> 192.4).
__device__ __forceinline__ float2 location_from_offset(const Params &p, float2 off, int64_t bq, int l,
                                                       float Wf, float Hf, float rcp_w, float rcp_h) {
    if (p.ref_coords != 2) return location_from_offset(p, off, bq, l, Wf, Hf);
    const float2 r = __ldg(reinterpret_cast<const float2 *>(p.ref) + bq * p.L + l);
    return make_float2(r.x + quotient(off.x, Wf, rcp_w), r.y + quotient(off.y, Hf, rcp_h));
}
// Derivative of the pixel coordinate with respect to that offset.
__device__ __forceinline__ float2 offset_derivative(const Params &p, int64_t bq, int l, float Wf, float Hf) {
    if (p.ref_coords == 2) return make_float2(1.f, 1.f);
    const float4 r = __ldg(reinterpret_cast<const float4 *>(p.ref) + bq * p.L + l);
    const float Kf = (float)p.K;
    // d(location)/d(offset) = wh * 0.5 / K, evaluated as the forward expression at offset 1
    return make_float2(Wf * (1.f / Kf * r.z * 0.5f), Hf * (1.f / Kf * r.w * 0.5f));
}

// A predicted offset, stored in float32 or the 16-bit value type.
template <typename T>
__device__ __forceinline__ float2 load_offset(const Params &p, int64_t e) {
    const float2 *loc2 = reinterpret_cast<const float2 *>(p.loc);
    if constexpr (sizeof(T) == 2) {
        if (p.offsets16) return VecTraits<T>::unpack2(__ldg(reinterpret_cast<const uint32_t *>(p.loc) + e));
    }
    return ld_stream_f2(loc2 + e);
}

// The forward's location: REF says at compile time whether there are reference points.
template <typename T, bool REF, typename Index>
__device__ __forceinline__ float2 forward_location(const Params &p, int64_t e, Index pair, int l,
                                                   float Wf, float Hf) {
    if constexpr (REF) {
        return location_from_offset(p, load_offset<T>(p, e), (int64_t)(pair / (Index)p.G), l, Wf, Hf);
    } else {
        return ld_stream_f2(reinterpret_cast<const float2 *>(p.loc) + e);
    }
}

// Sample location of element `e` = (pair, point) of level `l`, and in `dpix` the derivative of
// the pixel coordinate with respect to what the caller differentiates: the location itself
// (W, H), or the predicted offset when the call carries reference points.
template <typename T>
__device__ __forceinline__ float2 sample_location(const Params &p, int64_t e, int64_t pair, int l,
                                                  float Wf, float Hf, float2 &dpix) {
    const float2 *loc2 = reinterpret_cast<const float2 *>(p.loc);
    if (p.ref == nullptr) {
        dpix = make_float2(Wf, Hf);
        return ld_stream_f2(loc2 + e);
    }
    const float2 off = load_offset<T>(p, e);
    // (a 64-bit division costs as much as the rest of the point)
    const int64_t bq = pair <= 0x7fffffffll ? (int64_t)((unsigned)pair / (unsigned)p.G) : pair / p.G;
    dpix = offset_derivative(p, bq, l, Wf, Hf);
    return location_from_offset(p, off, bq, l, Wf, Hf);
}

// Softmax statistics (max, 1 / sum of exp(logit - max)) of a group's pairs: the lanes of a slot
// share the P logits of its pair.  The whole warp takes part; `live` says whether the slot has a
// pair.  (One lane per pair reading all P, the others idle, took 25 us more of a forward call of
// 43 008 queries.)
template <typename T>
__device__ __forceinline__ float2 slot_softmax_stats(const T *logits, int P, int lph, int sub, bool live) {
    float m = -INFINITY;
    if (live)
        for (int i = sub; i < P; i += lph) m = fmaxf(m, VecTraits<T>::to_float(logits[i]));
    for (int o = lph >> 1; o > 0; o >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, o));
    float sum = 0.f;
    if (live)
        for (int i = sub; i < P; i += lph) sum += expf(VecTraits<T>::to_float(logits[i]) - m);
    for (int o = lph >> 1; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
    return make_float2(m, 1.f / sum);
}

// floats of per-warp staging in the backward kernel: softmax stats (32 float2), then per
// (pair, point) a float2 location gradient, a weight gradient and (softmax) a probability;
// a multiple of 4 so every warp's region stays 16-byte aligned
__host__ __device__ inline int backward_stage_floats(int pairs_per_warp, int P, bool softmax) {
    const int n = 64 + pairs_per_warp * P * (softmax ? 4 : 3);
    return (n + 3) & ~3;
}

// ---------------------------------------------------------------------------------
// Scaled float16 accumulation: the last pass
// ---------------------------------------------------------------------------------
// tuning knob (compile-time): vectors a thread has in flight
#ifndef MSDA_FIN_VECS
#define MSDA_FIN_VECS 4
#endif
// grad_value = (image + the replicas of the position's level) * 2^-e, rounded to T.
// Positions of levels that have replicas form a small range of every sample (the coarse levels:
// 1 024 of 21 504 positions at the headline shape); everything outside it takes the short path.
// `lt` has its replicas planned; `extra_range` is the CTA's.  `image` may be grad_value itself.
// The part of one of `shares` CTAs.
__device__ __forceinline__ void find_extra_range(const LevelTable &lt, int L, int (&extra_range)[2]) {
    int lo = 0x7fffffff, hi = 0;
    for (int l = 0; l < L; ++l)
        if (lt.rep[l] > 1) {
            lo = min(lo, lt.start[l]);
            hi = max(hi, lt.start[l] + lt.H[l] * lt.W[l]);
        }
    extra_range[0] = lo;
    extra_range[1] = hi;
}

template <typename T>
__device__ __forceinline__ void finalize_image(const Params &p, const LevelTable &lt,
                                               const int (&extra_range)[2], int exponent,
                                               const uint4 *image, const __half *extras, int share,
                                               int shares) {
    using VT = VecTraits<T>;
    const int extra_lo = extra_range[0], extra_hi = extra_range[1];
    const bool any_extra = extra_lo < extra_hi;
    const int GD = p.G * p.D;
    const int vec_per_row = GD / 8;
    const int S = (int)p.S;
    const int64_t extra_sample = extra_elems_per_sample(p.Q, p.G, p.D, p.L, p.K);
    const float inv = ldexpf(1.f, -exponent);
    const float2 inv2 = make_float2(inv, inv);
    uint4 *gv = reinterpret_cast<uint4 *>(p.grad_value);
    const int64_t total = p.B * p.S * (int64_t)vec_per_row;
    const int64_t stride = (int64_t)shares * blockDim.x;
    const int64_t first = (int64_t)share * blockDim.x + threadIdx.x;
    // where the thread's current vector lies - sample b, position s of the sample, vector col of
    // the position's row - kept up to date by additions: one division per thread, none per vector
    // (first and stride are below 2^31: the grid is capped at a few thousand CTAs of 256 threads)
    const unsigned first_row = (unsigned)first / (unsigned)vec_per_row;
    int col = (int)((unsigned)first - first_row * (unsigned)vec_per_row);
    int64_t b = first_row / (unsigned)S;
    int s = (int)(first_row - (unsigned)b * (unsigned)S);
    const unsigned step_rows_all = (unsigned)stride / (unsigned)vec_per_row;
    const int step_cols = (int)((unsigned)stride - step_rows_all * (unsigned)vec_per_row);
    const int step_samples = (int)(step_rows_all / (unsigned)S);          // whole samples per stride
    const int step_rows = (int)(step_rows_all - (unsigned)step_samples * (unsigned)S);
    constexpr int kTurn = MSDA_FIN_VECS;
    for (int64_t v0 = first; v0 < total; v0 += kTurn * stride) {
        // several vectors per turn, their image loads issued together
        uint4 raw[kTurn];
#pragma unroll
        for (int u = 0; u < kTurn; ++u)
            raw[u] = v0 + u * stride < total ? ld_stream16(image + v0 + u * stride)
                                             : make_uint4(0u, 0u, 0u, 0u);
#pragma unroll
        for (int u = 0; u < kTurn; ++u) {
            const int64_t v = v0 + u * stride;
            if (v >= total) break;
            float2 f[4];
            VecTraits<__half>::unpack(raw[u], f);
            if (any_extra) {
                if (s >= extra_lo && s < extra_hi) {
                    const __half *sample_extras = extras + b * extra_sample + col * 8;
                    // every level whose range holds this position (one, for a well-formed table)
                    for (int l = 0; l < p.L; ++l) {
                        const int at = s - lt.start[l];
                        if (lt.rep[l] <= 1 || at < 0 || at >= lt.H[l] * lt.W[l]) continue;
                        const __half *src = sample_extras + lt.rep_base[l] + (int64_t)at * GD;
                        for (int r = 1; r < lt.rep[l]; ++r) {
                            float2 x[4];
                            VecTraits<__half>::unpack(
                                ld_stream16(src + (int64_t)(r - 1) * lt.level_elems[l]), x);
#pragma unroll
                            for (int i = 0; i < 4; ++i) {
                                f[i].x += x[i].x;
                                f[i].y += x[i].y;
                            }
                        }
                    }
                }
                // on to the vector one stride further
                col += step_cols;
                s += step_rows;
                b += step_samples;
                if (col >= vec_per_row) {
                    col -= vec_per_row;
                    ++s;
                }
                if (s >= S) {
                    s -= S;
                    ++b;
                }
            }
#pragma unroll
            for (int i = 0; i < 4; ++i) f[i] = fmul2(f[i], inv2);
            gv[v] = VT::pack(f);
        }
    }
}

// launchers implemented in msda_forward.cu / msda_backward.cu; dtype: 0 f32, 1 f16, 2 bf16
cudaError_t launch_forward(const Params &p, int dtype, bool softmax, cudaStream_t stream);
// Whether a call of 16-bit values takes the forward kernel of 32-byte loads.
bool forward_is_wide(const Params &p, bool softmax);
cudaError_t launch_backward(const Params &p, int dtype, bool softmax, cudaStream_t stream);
// The scaled backward in one launch, for calls that are bound by the host: what its scratch needs
// beyond the usual is a header of its own.  (Forward + backward of a decoder layer, host bound, B200:
// 79.7 us with the three launches, 73.7 so.  On the GPU 51.2 us against 53.2 with 154 000 points, 77.9
// against 75.8 with 262 000.)
enum FusedCell : unsigned {                // a line of memory each
    kFusedGradOut = 0, kFusedAttn = 32,    // largest magnitudes
    kFusedSweep = 64, kFusedSwept = 96,    // shares of the first sweep: handed out, done
    kFusedGroup = 128, kFusedGroups = 160, // groups of pairs: handed out, done
    kFusedLast = 192,                      // shares of the last sweep handed out
    kFusedGaveUp = 224,                    // not zero: a wait ran into its limit
};
constexpr int64_t kFusedBytes = 1024;
inline bool fused_backward_pays(const Params &p) {
    return p.B * p.Q * p.G * (int64_t)(p.L * p.K) <= ((int64_t)1 << 18);
}
cudaError_t launch_backward_fused(const Params &p, int dtype, bool softmax, cudaStream_t stream);
cudaError_t launch_prepare_grad_value(const Params &p, int dtype, bool softmax, cudaStream_t stream);
cudaError_t launch_finalize_grad_value(const Params &p, int dtype, bool softmax, cudaStream_t stream);
// float64 kernels (msda_f64.cu): loc / grad_loc point at doubles
cudaError_t launch_forward_f64(const Params &p, bool softmax, cudaStream_t stream);
cudaError_t launch_backward_f64(const Params &p, bool softmax, cudaStream_t stream);
size_t forward_smem_bytes(const Params &p, bool softmax);
size_t backward_smem_bytes(const Params &p, bool softmax);
// records `message` as the calling thread's last error (what msda_b200_last_error returns)
// and hands `status` back; defined in msda_abi.cu next to the buffer it writes
int set_last_error(int status, const char *message);
// adds to what msda_b200_launches() reports; defined there too
void count_launches(int kernels, int memsets);

}  // namespace msda_b200
