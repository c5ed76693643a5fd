// Backward on sorted points (16-bit values, dense sampling): grad_value as a product on the
// tensor cores instead of one reduction per bilinear corner.
//
// What bounds the direct backward (msda_backward.cu) is each SM's path to L2: four 64-byte
// reductions per sample point, 16 bytes of payload a clock.  Where a level receives several
// points per pixel those reductions hit the same few rows over and over.  Here the points of a
// (sample, head) plane are first sorted by the cell they fall in - a counting sort, two passes
// over the locations - and a warp then walks the sorted points with the pixels of its cell held
// on the tensor cores:
//
//   cell        one pixel row r0 and kCols = 7 adjacent pixel columns c0 of the top left corner;
//               all four corners of its points lie in a window of 2 rows x 8 columns = the 16
//               rows of an m16n8k16 tile
//   scatter     acc[16 pixels][D] += W[16 pixels][16 points] * grad_out[16 points][D], W holding
//               the points' corner weights (zero elsewhere), float32 accumulation
//   dots        dot[16 pixels][8 points] = value[16 pixels][D] * grad_out[8 points][D]^T, of which
//               a point's four corners are picked out
//
// Cells are numbered down a column strip, so the window's lower row is the next cell's upper
// row: an accumulated pixel row leaves the warp once per strip, as one 16-byte reduction per
// eight channels, instead of once per corner and point (at 21 504 queries and 12 points per query
// 33 million rows of reductions become about 1 million).
//
// Measured at the headline shape (4 x 21 504 queries, 8.3 M points, bf16): backward call 398 us
// against 512 us, of which counting 42, writing records 92, the walk 243, the last pass 22, each by itself;
// grad_value 1.72e-3 off the float64 result, most of it bfloat16's own rounding (float16: 3.7e-4).
//
// Accumulation is float32 inside a warp's run of points; the few sums that meet in memory (two
// strips share a column, two runs share a row) meet in float16, scaled as in the direct backward
// (msda_common.cuh), in grad_value itself, which the last kernel rewrites in its own type.
#include "msda_sorted.cuh"

namespace msda_b200 {

namespace {

constexpr int kSortThreads = 512;
constexpr int kSortPoints = 8;         // points per thread of the sort kernels,
constexpr int kSortBatch = 4;          // loaded this many at a time
constexpr int kSharedCells = 8192;     // most cells of a plane that are counted in shared memory
static_assert(kSharedCells % 8 == 0, "scan_cells");
constexpr int kSortCtaPoints = kSortThreads * kSortPoints;
constexpr int kWalkWarps = 4;          // warps per CTA of the walk, each on its own run

// header cells beside the two magnitudes
constexpr int kNextItem = 2;           // runs of the walk handed out so far
constexpr int kNoCells = 3;            // not zero: the levels' cells do not fit
constexpr unsigned kNonFinite = 0x7fffu;   // magnitude bits of a NaN in either type

// ---- cells ---------------------------------------------------------------------------------------
struct CellTable {
    int first[kMaxLevels + 1];   // first cell of the level; [L]: number of cells
    int rows[kMaxLevels];        // cells per strip: H + 1 (r0 = -1 .. H - 1)
    bool fits;                   // the cells of all levels fit the room there is
};

// A table whose levels overlap can ask for more cells than there is room for (levels that tile
// `value` cannot): such a call is not sorted.
__device__ inline void plan_cells(CellTable &c, const LevelTable &t, int L, int bound) {
    int n = 0;
    c.fits = true;
    for (int l = 0; l < L; ++l) {
        const long long cells =
            t.H[l] > 0 ? (t.H[l] + 1ll) * ((t.W[l] + kCols) / kCols) : 0;   // ceil((W + 1) / kCols)
        c.first[l] = n;
        c.rows[l] = t.H[l] + 1;
        if (n + cells <= bound)
            n += (int)cells;
        else
            c.fits = false;
    }
    c.first[L] = n;
}

// A sort CTA takes the points of a stretch of queries of one (sample, head) plane.  A thread
// keeps to one point index and steps over queries, so all that depends on the level is in
// registers, and a warp's loads run over consecutive points.  Heads vary fastest over CTAs (those
// that read one stretch of locations run side by side), samples slowest: the records being
// written at a time are one or two samples' and stay in L2 until their sectors are complete.
struct SortLane {
    int plane, b, g;
    int pt, l;              // point of the query and its level
    int H, W, cell0, rows;  // of the level
    float rcp_w, rcp_h;     // 1 / W, 1 / H
    int ql, nq, step;       // first query of the thread (chunk-relative), queries of the chunk, stride
    int64_t q0;             // first query of the chunk
    bool active;
};
// `points` of every query from `point0` on are the CTA's.
template <int THREADS>
__device__ __forceinline__ SortLane sort_lane(const Params &p, const LevelTable &lt, const CellTable &ct, unsigned cta,
                                              int chunks, int chunk_queries, int points, int point0) {
    SortLane s;
    const unsigned per_sample = (unsigned)chunks * (unsigned)p.G;
    s.b = (int)(cta / per_sample);
    const int chunk = (int)((cta - (unsigned)s.b * per_sample) / (unsigned)p.G);
    s.g = (int)(cta - (unsigned)s.b * per_sample) - chunk * p.G;
    s.plane = s.b * p.G + s.g;
    s.step = THREADS / points;
    s.ql = (int)threadIdx.x / points;
    s.pt = point0 + (int)threadIdx.x - s.ql * points;
    s.l = s.pt / p.K;
    s.active = s.ql < s.step;
    s.H = lt.H[s.l];
    s.W = lt.W[s.l];
    s.rcp_w = lt.rcp_w[s.l], s.rcp_h = lt.rcp_h[s.l];      // (set where there are offsets)
    s.cell0 = ct.first[s.l];
    s.rows = ct.rows[s.l];
    s.q0 = (int64_t)chunk * chunk_queries;
    s.nq = (int)min((int64_t)chunk_queries, p.Q - s.q0);
    return s;
}

// Where a point of the thread's level falls; false if it is skipped.  The same float32
// arithmetic as locate().
struct PointCell {
    int cell, col;
    float fr, fc;
};
__device__ __forceinline__ bool find_cell(const SortLane &s, float2 xy, PointCell &o) {
    const float Wf = (float)s.W, Hf = (float)s.H;
    const float px = fmaf(xy.x, Wf, -0.5f), py = fmaf(xy.y, Hf, -0.5f);
    if (!(py >= -1.f && px >= -1.f && py < Hf && px < Wf && s.H > 0)) return false;
    const float r0f = floorf(py), c0f = floorf(px);
    o.fr = py - r0f;
    o.fc = px - c0f;
    const unsigned c1 = (unsigned)((int)c0f + 1), strip = c1 / kCols;
    o.col = (int)(c1 - strip * kCols);
    o.cell = s.cell0 + (int)strip * s.rows + (int)r0f + 1;
    return true;
}

// Sample location of the thread's point of query `q` of the chunk: sample_location() without its
// 64-bit divisions.  `base` is the element index of the same point of the chunk's first query.
template <typename T, bool REF>
__device__ __forceinline__ float2 point_xy(const Params &p, const SortLane &s, int64_t base, int q) {
    const int64_t e = base + (int64_t)(q * (p.G * p.L * p.K));
    if constexpr (REF) {
        const float2 off = p.offsets16 ? VecTraits<T>::unpack2(__ldg(reinterpret_cast<const uint32_t *>(p.loc) + e))
                                       : __ldg(reinterpret_cast<const float2 *>(p.loc) + e);
        return location_from_offset(p, off, (int64_t)s.b * p.Q + s.q0 + q, s.l, (float)s.W, (float)s.H, s.rcp_w, s.rcp_h);
    } else {
        return __ldg(reinterpret_cast<const float2 *>(p.loc) + e);
    }
}

// Adds the counts the CTA made in shared memory to the plane's.
__device__ __forceinline__ void merge_counts(const unsigned *hist, unsigned *plane, int cells) {
    for (int c = threadIdx.x; c < cells; c += blockDim.x)
        if (hist[c] != 0) atomicAdd(plane + c, hist[c]);
}

// Takes the CTA's counts per cell to `begin`, where the cell's points begin in the CTA's order,
// and leaves in their place the difference to where they begin in the plane's.  Returns how
// many points there are.
template <int THREADS>
__device__ __forceinline__ unsigned scan_cells(unsigned *counts, unsigned short *begin, unsigned *cursor,
                                               unsigned *warp_sums, int cells) {
    constexpr int kEach = 8;      // adjacent cells a thread takes (the arrays are padded to this)
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    unsigned base = 0;
    for (int c0 = 0; c0 < cells; c0 += THREADS * kEach) {
        const int at = c0 + threadIdx.x * kEach;
        unsigned n[kEach], place[kEach], sum = 0;
#pragma unroll
        for (int i = 0; i < kEach; i += 4) {
            const uint4 v = at < cells ? *reinterpret_cast<const uint4 *>(counts + at + i) : make_uint4(0u, 0u, 0u, 0u);
            n[i] = v.x, n[i + 1] = v.y, n[i + 2] = v.z, n[i + 3] = v.w;
        }
        // (the round trips to L2 overlap, and the scan with them)
#pragma unroll
        for (int i = 0; i < kEach; ++i) {
            if (at + i >= cells) n[i] = 0u;
            place[i] = n[i] != 0 ? atomicAdd(cursor + at + i, n[i]) : 0u;
            sum += n[i];
        }
        unsigned incl = sum;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const unsigned up = __shfl_up_sync(0xffffffffu, incl, o);
            if (lane >= o) incl += up;
        }
        if (lane == 31) warp_sums[warp] = incl;
        __syncthreads();
        unsigned before = 0, total = 0;
#pragma unroll
        for (int w = 0; w < THREADS / 32; ++w) {
            const unsigned s = warp_sums[w];
            before += w < warp ? s : 0u;
            total += s;
        }
        unsigned first = base + before + incl - sum;
        if (at < cells) {
            unsigned b[kEach];
#pragma unroll
            for (int i = 0; i < kEach; ++i) {
                b[i] = first;
                place[i] -= first;
                first += n[i];
            }
#pragma unroll
            for (int i = 0; i < kEach; i += 4)
                *reinterpret_cast<uint4 *>(counts + at + i) = make_uint4(place[i], place[i + 1], place[i + 2], place[i + 3]);
            *reinterpret_cast<uint4 *>(begin + at) = make_uint4(b[0] | b[1] << 16, b[2] | b[3] << 16,
                                                                b[4] | b[5] << 16, b[6] | b[7] << 16);
        }
        base += total;
        __syncthreads();
    }
    return base;
}

// f(i, value) for the P 16-bit values of a pair, four at a time where that is aligned
template <typename T, typename F>
__device__ __forceinline__ void for_values(const T *x, int P, F f) {
    using VT = VecTraits<T>;
    if ((P & 3) == 0) {
#pragma unroll 4
        for (int i = 0; i < P; i += 4) {
            const uint2 v = __ldg(reinterpret_cast<const uint2 *>(x + i));
            const float2 a = VT::unpack2(v.x), b = VT::unpack2(v.y);
            f(i, a.x), f(i + 1, a.y), f(i + 2, b.x), f(i + 3, b.y);
        }
    } else {
        for (int i = 0; i < P; ++i) f(i, VT::to_float(x[i]));
    }
}

// What has to be known or done before anything is accumulated: largest magnitudes for the scale,
// zeros in grad_value, softmax statistics (max, 1 / sum) of every pair.  The share of one of
// `ctas` CTAs.
// Header cell 1 is the largest |attn| element's; of a softmax, whose probabilities are at most 1, it
// says whether a pair's are numbers at all (a NaN or +inf logit, or nothing but -inf, makes every
// one of them NaN).
template <typename T, bool SOFTMAX>
__device__ __forceinline__ void prepare_share(const Params &p, const SortPlan &sp, int cta, int ctas) {
    unsigned *header = sp.header;
    __shared__ unsigned cta_max[2];
    if (threadIdx.x < 2) cta_max[threadIdx.x] = 0u;
    __syncthreads();
    const int64_t stride = (int64_t)ctas * blockDim.x;
    const int64_t first = (int64_t)cta * blockDim.x + threadIdx.x;
    const int64_t go_vecs = p.B * p.Q * (p.G * p.D / 8);
    unsigned mg = scan_max_magnitude(reinterpret_cast<const uint4 *>(p.grad_out), go_vecs, first, stride);
    unsigned ma = 0;
    if constexpr (!SOFTMAX) {
        // (a later sample's weights need not begin on a 16-byte boundary: whole vectors in the
        // middle, single elements at both ends)
        const unsigned short *at = reinterpret_cast<const unsigned short *>(p.attn);
        const int64_t n = p.B * p.Q * p.G * p.L * p.K;
        const int64_t head = min((int64_t)((16u - (unsigned)(reinterpret_cast<uintptr_t>(at) & 15u)) & 15u) / 2, n);
        const int64_t body = (n - head) / 8;
        ma = scan_max_magnitude(reinterpret_cast<const uint4 *>(at + head), body, first, stride);
        for (int64_t i = first; i < head; i += stride) ma = max(ma, at[i] & 0x7fffu);
        for (int64_t i = head + body * 8 + first; i < n; i += stride) ma = max(ma, at[i] & 0x7fffu);
    }
    if constexpr (SOFTMAX) {
        const int P = p.L * p.K;
        for (int64_t i = first; i < p.B * p.Q * p.G; i += stride) {
            const T *x = reinterpret_cast<const T *>(p.attn) + i * P;
            float m = -INFINITY, sum = 0.f;
            for_values(x, P, [&](int, float v) { m = fmaxf(m, v); });
            for_values(x, P, [&](int, float v) { sum += expf(v - m); });
            sp.stats[i] = make_float2(m, 1.f / sum);
            if (!(sum < INFINITY)) ma = kNonFinite;
        }
    }
    uint4 *gv = reinterpret_cast<uint4 *>(p.grad_value);
    const int64_t vecs = p.B * p.S * (p.G * p.D / 8);
    for (int64_t v = first; v < vecs; v += stride) gv[v] = make_uint4(0u, 0u, 0u, 0u);
    mg = __reduce_max_sync(0xffffffffu, mg);
    ma = __reduce_max_sync(0xffffffffu, ma);
    if ((threadIdx.x & 31) == 0) {
        if (mg != 0) atomicMax(&cta_max[0], mg);
        if (ma != 0) atomicMax(&cta_max[1], ma);
    }
    __syncthreads();
    if (threadIdx.x < 2 && cta_max[threadIdx.x] != 0) atomicMax(header + threadIdx.x, cta_max[threadIdx.x]);
}

// Exclusive prefix sum of a plane's cell counts by one CTA, in chunks of its size: `counts`
// becomes the cursor the scatter kernel hands places out from, `offsets` the cells' first places
// (offsets[cells]: the plane's points), `item_cell` the cell in which each unit of
// sp.item_points places begins.
template <int THREADS>
__device__ __forceinline__ void scan_plane(unsigned *counts, unsigned *offsets, int *item_cell, int cells,
                                  int item_points) {
    __shared__ unsigned warp_sums[THREADS / 32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    unsigned base = 0;
    for (int c0 = 0; c0 < cells; c0 += THREADS * 4) {
        const int at = c0 + threadIdx.x * 4;
        unsigned n[4], sum = 0;
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            n[i] = at + i < cells ? __ldcg(counts + at + i) : 0u;
            sum += n[i];
        }
        unsigned incl = sum;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const unsigned up = __shfl_up_sync(0xffffffffu, incl, o);
            if (lane >= o) incl += up;
        }
        if (lane == 31) warp_sums[warp] = incl;
        __syncthreads();
        unsigned before = 0, total = 0;
#pragma unroll
        for (int w = 0; w < THREADS / 32; ++w) {
            const unsigned s = warp_sums[w];
            before += w < warp ? s : 0u;
            total += s;
        }
        unsigned at_place = base + before + incl - sum;
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            if (at + i < cells) {
                counts[at + i] = at_place;
                offsets[at + i] = at_place;
                for (unsigned m = (at_place + item_points - 1) / item_points;
                     m * (unsigned)item_points < at_place + n[i]; ++m)
                    item_cell[m] = at + i;
                at_place += n[i];
            }
        }
        base += total;
        __syncthreads();
    }
    if (threadIdx.x == 0) offsets[cells] = base;
}

// ---- pass 1: count the points of every cell -------------------------------------------------------
// Bound by latency: a CTA's life is a dozen round trips to memory, so more warps per SM count for
// more than registers (2 / 3 / 4 CTAs of 512 threads per SM: 64 / 55 / 50 us at the headline shape;
// reading its operands alone takes 28 us).
//
// BY_LEVEL: a CTA takes the points that a stretch of queries has on one level (levels vary after heads):
// its cells are a level's only, so that a stretch can be longer and the counts of a cell are merged less
// often.  Backward, B200, us, all levels -> this: headline shape 404 -> 398, 512 pixels 8 samples 224 -> 221,
// four odd levels in float16 422 -> 418, 59 104 positions (2 samples, 4 x 64 channels) 487 -> 416; 1, 2 and 8
// points a level of 14 196 positions 593 -> 591, 527 -> 522, 440 -> 428.  Offsets, half as long and evaluated
// at more expense, are better off with all levels of a query side by side (ragged pyramid, this kernel 29
// us against 38).
__host__ __device__ constexpr int count_threads(bool by_level) { return by_level ? 256 : kSortThreads; }
template <typename T, bool SOFTMAX, bool REF, bool BY_LEVEL>
__global__ void __launch_bounds__(count_threads(BY_LEVEL), 2048 / count_threads(BY_LEVEL))
    sort_count_kernel(const __grid_constant__ Params p, const __grid_constant__ SortPlan sp) {
    constexpr int kThreads = count_threads(BY_LEVEL);
    grid_launch_dependents();
    // the first CTAs look for the magnitudes and clear grad_value, beside those that count
    if (blockIdx.x < (unsigned)sp.prepare_ctas) {
        prepare_share<T, SOFTMAX>(p, sp, (int)blockIdx.x, sp.prepare_ctas);
        return;
    }
    extern __shared__ unsigned hist[];
    __shared__ LevelTable lt;
    __shared__ CellTable ct;
    __shared__ bool last;
    load_level_table<REF>(lt, p);
    __syncthreads();
    if (threadIdx.x == 0) plan_cells(ct, lt, p.L, sp.cell_bound);
    __syncthreads();
    if (!ct.fits) {
        if (threadIdx.x == 0) sp.header[kNoCells] = 1u;   // (every CTA says the same)
        return;
    }
    SortLane c;
    unsigned cta = blockIdx.x - (unsigned)sp.prepare_ctas;
    int cell0 = 0, cells = ct.first[p.L];
    if constexpr (BY_LEVEL) {
        const unsigned heads = cta / (unsigned)p.G, stretch = heads / (unsigned)p.L;
        const int level = (int)(heads - stretch * (unsigned)p.L);
        c = sort_lane<kThreads>(p, lt, ct, stretch * (unsigned)p.G + (cta - heads * (unsigned)p.G), sp.count_stretches,
                                sp.count_queries, p.K, level * p.K);
        cell0 = ct.first[level];
        cells = ct.first[level + 1] - cell0;
    } else {
        c = sort_lane<kThreads>(p, lt, ct, cta, sp.count_stretches, sp.count_queries, p.L * p.K, 0);
    }
    c.cell0 -= cell0;
    const bool in_shared = cells <= sp.count_cells;
    if (in_shared)
        for (int i = threadIdx.x; i < cells; i += kThreads) hist[i] = 0u;
    unsigned *counts = sp.counts + (int64_t)c.plane * sp.cell_stride;
    __syncthreads();
    if (c.active) {
        const int64_t base = (((int64_t)c.b * p.Q + c.q0) * p.G + c.g) * (p.L * p.K) + c.pt;
        for (int q0 = c.ql; q0 < c.nq; q0 += kSortBatch * c.step) {
            float2 xy[kSortBatch];
#pragma unroll
            for (int r = 0; r < kSortBatch; ++r) {
                const int q = q0 + r * c.step;
                xy[r] = q < c.nq ? point_xy<T, REF>(p, c, base, q) : make_float2(-1e9f, -1e9f);
            }
            PointCell at;
#pragma unroll
            for (int r = 0; r < kSortBatch; ++r) {
                if (!find_cell(c, xy[r], at)) continue;
                if (in_shared)
                    atomicAdd(hist + at.cell, 1u);
                else
                    atomicAdd(counts + cell0 + at.cell, 1u);
            }
        }
    }
    __syncthreads();
    if (in_shared) merge_counts(hist, counts + cell0, cells);
    // the plane's last CTA turns its counts into places
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0) last = atomicAdd(sp.tickets + c.plane, 1u) == (unsigned)(sp.count_ctas - 1);
    __syncthreads();
    if (last) {
        __threadfence();
        scan_plane<kThreads>(counts, sp.offsets + (int64_t)c.plane * sp.cell_stride,
                             sp.item_cell + (int64_t)c.plane * sp.items, ct.first[p.L], sp.item_points);
    }
}

// Gradients of one point, wherever they were formed.  The weight's goes out in float32: the last
// kernel rounds it, after the softmax Jacobian where there is one (and scattered two-byte
// stores take half as long again as four-byte ones: 2.3 cycles of an SM each against 1.5).
template <typename T>
__device__ __forceinline__ void store_point_gradients(const Params &p, const SortPlan &sp, int64_t e,
                                                      float2 grad_loc, float grad_weight) {
    if (p.ref != nullptr && p.offsets16)
        reinterpret_cast<uint32_t *>(p.grad_loc)[e] = VecTraits<T>::pack2(grad_loc);
    else
        reinterpret_cast<float2 *>(p.grad_loc)[e] = grad_loc;
    sp.grad_prob[e] = grad_weight;
}

// What cannot be sorted: an inf or NaN in grad_out or in a weight has to reach its own point's
// corners only, and a tile product would spread it to the zero entries beside them (0 * inf); and
// tables without room for their cells.  A float16 step whose loss scale overflowed is such a call.
// Its points take the walk kernel's place in the order they have, accumulate_unsorted(), with
// the replicas of coarse levels that the direct backward gives them where the records would be.
template <typename T>
__device__ __forceinline__ bool unsorted_call(const unsigned *header) {
    return max(header[0], header[1]) >= (std::is_same<T, __half>::value ? 0x7c00u : 0x7f80u) ||
           header[kNoCells] != 0u;
}
// (at most L * K*Q*G*D / 64 float16 a sample, D / 32 <= 2 bytes a point where a record is 16)
__device__ __forceinline__ __half *unsorted_extras(const SortPlan &sp) {
    return reinterpret_cast<__half *>(sp.records);
}

// Clears them, the share of one CTA of a sort kernel.
__device__ inline void clear_unsorted_extras(const Params &p, const SortPlan &sp) {
    uint4 *extras = reinterpret_cast<uint4 *>(unsorted_extras(sp));
    const int64_t vecs = p.B * (extra_elems_per_sample(p.Q, p.G, p.D, p.L, p.K) / 8);
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < vecs; i += (int64_t)gridDim.x * blockDim.x)
        extras[i] = make_uint4(0u, 0u, 0u, 0u);
}

// The points of a call without the sort.  A warp takes 32 adjacent points, each lane locates one;
// then the D / 8 lanes of a slot gather and add a point's corners at a time, as in the direct
// backward, the point's numbers coming and its gradients going by shuffles.  Such a call takes
// 690 us at the headline shape (direct backward 515; one thread per point took 1540): half the
// direct kernel's warps per SM, and twice its shuffles, four points in flight as quick as two.
// Launching the direct kernels instead would cost every other call their empty launches.
template <typename T, int D>
__device__ __noinline__ void accumulate_unsorted(const Params &p, const SortPlan &sp, LevelTable &lt,
                                                 bool softmax) {
    using VT = VecTraits<T>;
    constexpr int LPH = D / 8, kSlots = 32 / LPH;
    if (threadIdx.x == 0) plan_replicas(lt, p);
    __syncthreads();
    const int lane = threadIdx.x & 31, slot = lane / LPH, ch = lane % LPH * 8;
    const unsigned P = (unsigned)(p.L * p.K), G = (unsigned)p.G;
    const int GD = p.G * D;
    const float scale = ldexpf(1.f, grad_scale_exponent<T>(sp.header, p.Q, p.K, softmax));
    const unsigned points = (unsigned)p.Q * G * P, turns = (points + 31u) / 32u;   // of a sample
    const int64_t extra_sample = extra_elems_per_sample(p.Q, p.G, D, p.L, p.K);
    const T *attn = reinterpret_cast<const T *>(p.attn);
    for (int64_t turn = (int64_t)blockIdx.x * kWalkWarps + (threadIdx.x >> 5); turn < p.B * turns;
         turn += (int64_t)gridDim.x * kWalkWarps) {
        const int64_t b = turn / turns;
        const unsigned at = (unsigned)(turn - b * turns) * 32u + lane;
        // ---- one lane per point
        unsigned flags = 0, off = 0, red_off = 0, pair = 0;
        float a = 0.f, fr = 0.f, fc = 0.f;
        float2 dpix = make_float2(0.f, 0.f);
        const int64_t e = b * points + at;
        if (at < points) {
            pair = at / P;
            const unsigned pt = at - pair * P, q = pair / G;
            const int l = (int)pt / p.K, head = (int)(pair - q * G) * D;
            const int64_t whole_pair = b * (p.Q * p.G) + pair;
            const float2 xy = sample_location<T>(p, e, whole_pair, l, (float)lt.W[l], (float)lt.H[l], dpix);
            const PointGeom geo = locate(xy.x, xy.y, lt.H[l], lt.W[l], lt.start[l], GD);
            flags = geo.flags | ((unsigned)l << kLevelShift);
            fr = geo.fr, fc = geo.fc;
            off = red_off = (unsigned)(geo.off00 + head);
            if (lt.rep[l] > 1) {
                const unsigned r = (q + pt) % (unsigned)lt.rep[l];
                if (r > 0) {
                    red_off = lt.rep_base[l] + (r - 1) * lt.level_elems[l] +
                              (unsigned)((geo.r0 * lt.W[l] + geo.c0) * GD + head);
                    flags |= kUseExtra;
                }
            }
            if (flags & kInside) {
                a = VT::to_float(attn[e]);
                if (softmax) {
                    const float2 st = sp.stats[whole_pair];
                    a = expf(a - st.x) * st.y;
                }
            }
        }
        // ---- one slot per point
        const T *value = reinterpret_cast<const T *>(p.value) + b * p.S * GD + ch;
        const T *grad_out = reinterpret_cast<const T *>(p.grad_out) + b * p.Q * GD + ch;
        __half *image = reinterpret_cast<__half *>(p.grad_value) + b * p.S * GD + ch;
        __half *extras = unsorted_extras(sp) + b * extra_sample + ch;
        float gx = 0.f, gy = 0.f, ga = 0.f;      // of the lane's own point
#pragma unroll 2
        for (int i = 0; i < LPH; ++i) {
            const int from = i * kSlots + slot;
            const unsigned f = __shfl_sync(0xffffffffu, flags, from);
            const unsigned o00 = __shfl_sync(0xffffffffu, off, from), q00 = __shfl_sync(0xffffffffu, red_off, from);
            const float r = __shfl_sync(0xffffffffu, fr, from), c = __shfl_sync(0xffffffffu, fc, from);
            const float s0 = __shfl_sync(0xffffffffu, a, from) * scale;
            const unsigned row = __shfl_sync(0xffffffffu, pair, from);
            const unsigned down = (unsigned)lt.rowstride[f >> kLevelShift];
            const unsigned step[4] = {0u, (unsigned)GD, down, down + (unsigned)GD};
            const float w[4] = {(1.f - r) * (1.f - c), (1.f - r) * c, r * (1.f - c), r * c};
            float2 go[4];
            VT::unpack(ldg16(grad_out + (size_t)row * D), go);
            uint4 raw[4];
#pragma unroll
            for (int k = 0; k < 4; ++k) raw[k] = ldg16_if(value + (int)(o00 + step[k]), f & (1u << k));
            __half *to = f & kUseExtra ? extras : image;
            float dot[4];
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                float2 v[4], gv[4], d2 = make_float2(0.f, 0.f);
                VT::unpack(raw[k], v);
                const float s = s0 * w[k];
#pragma unroll
                for (int n = 0; n < 4; ++n) {
                    ffma2(d2, v[n], go[n]);
                    gv[n] = fmul2(go[n], make_float2(s, s));
                }
                dot[k] = d2.x + d2.y;
                red_if<__half>(to + (q00 + step[k]), gv, f & (1u << k));
            }
            float x = (1.f - r) * (dot[1] - dot[0]) + r * (dot[3] - dot[2]);
            float y = (1.f - c) * (dot[2] - dot[0]) + c * (dot[3] - dot[1]);
            float g = w[0] * dot[0] + w[1] * dot[1] + w[2] * dot[2] + w[3] * dot[3];
#pragma unroll
            for (int o = LPH >> 1; o > 0; o >>= 1) {
                x += __shfl_xor_sync(0xffffffffu, x, o);
                y += __shfl_xor_sync(0xffffffffu, y, o);
                g += __shfl_xor_sync(0xffffffffu, g, o);
            }
            const int mine = lane % kSlots * LPH;      // a lane of the slot that had this lane's point
            x = __shfl_sync(0xffffffffu, x, mine);
            y = __shfl_sync(0xffffffffu, y, mine);
            g = __shfl_sync(0xffffffffu, g, mine);
            if (lane / kSlots == i) gx = x, gy = y, ga = g;
        }
        if (at < points) {
            const bool inside = flags & kInside;       // a skipped point: exact zeros
            store_point_gradients<T>(p, sp, e,
                                     inside ? make_float2(a * dpix.x * gx, a * dpix.y * gy) : make_float2(0.f, 0.f),
                                     inside ? ga : 0.f);
        }
    }
}

// ---- pass 2: write the points' records in order of their cells ------------------------------------
// A record: fractions of the pixel coordinate (column, row), weight, and where the point came
// from: query << 12 | point << 3 | column of the cell.  The CTA orders its records by cell before
// they leave: a warp's stores then fall on a few stretches of memory instead of 32 places (with
// the locations kept from being evaluated twice: 105 us at the headline shape against 126).
template <typename T, bool SOFTMAX, bool REF>
__global__ void __launch_bounds__(kSortThreads, 2) sort_scatter_kernel(const __grid_constant__ Params p,
                                                                       const __grid_constant__ SortPlan sp) {
    using VT = VecTraits<T>;
    extern __shared__ uint4 smem[];
    __shared__ LevelTable lt;
    __shared__ CellTable ct;
    __shared__ unsigned warp_sums[kSortThreads / 32];
    // the CTA's records, by thread; in order of their cells: which record, which cell; and per
    // cell: its count, then what takes a place in the CTA's order to one in the plane's, and its
    // first place in the CTA's
    uint4 *local = smem;
    unsigned *shift = reinterpret_cast<unsigned *>(local + kSortCtaPoints);
    unsigned short *order = reinterpret_cast<unsigned short *>(shift + sp.shared_cells);
    unsigned short *cell_of = order + kSortCtaPoints;
    unsigned short *begin = cell_of + kSortCtaPoints;
    load_level_table<REF>(lt, p);
    __syncthreads();
    if (threadIdx.x == 0) plan_cells(ct, lt, p.L, sp.cell_bound);
    __syncthreads();
    const int cells = ct.first[p.L];
    const bool in_shared = cells <= sp.shared_cells;
    if (in_shared)
        for (int i = threadIdx.x; i < cells; i += kSortThreads) shift[i] = 0u;
    const SortLane c = sort_lane<kSortThreads>(p, lt, ct, blockIdx.x, sp.chunks, sp.chunk_queries, p.L * p.K, 0);
    grid_launch_dependents();
    grid_dependency_wait();     // everything above reads the caller's tables only
    unsigned *cursor = sp.counts + (int64_t)c.plane * sp.cell_stride;
    uint4 *records = sp.records + (int64_t)c.plane * sp.plane_points;
    const T *attn = reinterpret_cast<const T *>(p.attn);
    const int P = p.L * p.K;
    const int64_t pair0 = ((int64_t)c.b * p.Q + c.q0) * p.G + c.g;   // of the chunk's first query
    const int64_t base = pair0 * P + c.pt;
    const int nq = c.active ? c.nq : 0;
    if (!ct.fits) {      // (its points have no cells to be counted in)
        clear_unsorted_extras(p, sp);
        return;
    }
    // (asked here, needed only when records leave: the points' loads do not wait for the answer)
    const bool unsorted = unsorted_call<T>(sp.header);
    __syncthreads();
    unsigned at[kSortPoints];     // cell << 16 | rank among the CTA's points of the cell; ~0: skipped
#pragma unroll
    for (int r0 = 0; r0 < kSortPoints; r0 += kSortBatch) {
        float2 xy[kSortBatch], stats[SOFTMAX ? kSortBatch : 1];
        T weight[kSortBatch];
#pragma unroll
        for (int r = 0; r < kSortBatch; ++r) {
            const int q = c.ql + (r0 + r) * c.step;
            if (q < nq) {
                xy[r] = point_xy<T, REF>(p, c, base, q);
            }
        }
        // (behind all the locations, not beside each: with reference points and softmax 40.5 us
        // against 45.5 of the ragged pyramid, 74 against 85 of the 512-pixel one)
#pragma unroll
        for (int r = 0; r < kSortBatch; ++r) {
            const int q = c.ql + (r0 + r) * c.step;
            if (q < nq) {
                if constexpr (SOFTMAX) stats[r] = sp.stats[pair0 + (int64_t)(q * p.G)];
                weight[r] = attn[base + (int64_t)(q * (p.G * P))];
            }
        }
#pragma unroll
        for (int r = 0; r < kSortBatch; ++r) {
            at[r0 + r] = ~0u;
            const int q = c.ql + (r0 + r) * c.step;
            if (q >= nq) continue;
            PointCell pc;
            if (!find_cell(c, xy[r], pc)) {
                // a skipped point: exact zeros
                store_point_gradients<T>(p, sp, base + (int64_t)(q * (p.G * P)), make_float2(0.f, 0.f), 0.f);
            } else {
                float a = VT::to_float(weight[r]);
                if constexpr (SOFTMAX) a = expf(a - stats[r].x) * stats[r].y;
                const uint4 record =
                    make_uint4(__float_as_uint(pc.fc), __float_as_uint(pc.fr), __float_as_uint(a),
                               ((unsigned)(c.q0 + q) << 12) | ((unsigned)c.pt << 3) | (unsigned)pc.col);
                if (in_shared) {
                    local[(r0 + r) * kSortThreads + threadIdx.x] = record;
                    at[r0 + r] = ((unsigned)pc.cell << 16) | atomicAdd(shift + pc.cell, 1u);
                } else {
                    const unsigned place = atomicAdd(cursor + pc.cell, 1u);
                    if (place < (unsigned)sp.plane_points && !unsorted) records[place] = record;
                }
            }
        }
    }
    if (unsorted) {
        clear_unsorted_extras(p, sp);
        return;
    }
    if (in_shared) {
        __syncthreads();
        const unsigned points = scan_cells<kSortThreads>(shift, begin, cursor, warp_sums, cells);
        __syncthreads();
#pragma unroll
        for (int r = 0; r < kSortPoints; ++r) {
            if (at[r] == ~0u) continue;
            const unsigned i = begin[at[r] >> 16] + (at[r] & 0xffffu);
            order[i] = (unsigned short)(r * kSortThreads + threadIdx.x);
            cell_of[i] = (unsigned short)(at[r] >> 16);
        }
        __syncthreads();
        // neighbours in the CTA's order are neighbours in the plane's for as long as a cell lasts
#pragma unroll 4
        for (unsigned i = threadIdx.x; i < points; i += kSortThreads) {
            const unsigned place = i + shift[cell_of[i]];
            if (place < (unsigned)sp.plane_points) records[place] = local[order[i]];
        }
    }
}

// The same a level at a time, for larger planes: a level has a third of the cells to look
// through and merge per turn, and a cell's records leave in longer runs; the price is that a load
// touches a line of memory for every query (why short offsets and small planes keep the other).  The
// fractions and weights stay in registers until their place in the turn's order is known: few threads
// with many registers, and persistent CTAs.  Bound by the latency of its phases (load/store pipe 62 %
// busy, issue slots 43 %, DRAM 40 %).
// Backward, B200, us, all levels -> this (4 points a level of 8 x 32 channels unless said): headline shape
// 414 -> 398, queries anywhere 437 -> 419, four odd levels in float16 427 -> 418, 2 samples of 27 750 positions
// on five levels 440 -> 396, one of 42 500 on four 296 -> 274, 2 of 59 104 with 4 x 64 channels 496 -> 416;
// 14 196 positions with 1, 2 and 8 points a level 618 -> 590, 545 -> 522, 442 -> 428: one line of memory per
// query and load is no loss with few points either.  (320 threads of 96 registers; when it took 394 us: 256 x 3
// of 80: 428; 384 of 80 and six points 400; 512 of 64, which spill, 412; without registers, as above, 256 x 3
// 407.)
constexpr int kLevelThreads = 320;
constexpr int kLevelPoints = 8;        // points per thread and turn,
constexpr int kLevelBatch = 4;         // loaded this many at a time
constexpr int kLevelTurn = kLevelThreads * kLevelPoints;
constexpr int kLevelCells = 10752;     // most cells of a level, so that two CTAs fit an SM
constexpr int kCountRoom = 3760;       // cells that any level may have in the counting kernel (plan_sorted)
static_assert(3 * kLevelPoints <= 32, "the columns of a thread's points share a word");
template <typename T, bool SOFTMAX, bool REF>
__global__ void __launch_bounds__(kLevelThreads, 2) sort_scatter_level_kernel(const __grid_constant__ Params p,
                                                                             const __grid_constant__ SortPlan sp) {
    using VT = VecTraits<T>;
    extern __shared__ uint4 smem[];
    __shared__ LevelTable lt;
    __shared__ CellTable ct;
    __shared__ unsigned warp_sums[kLevelThreads / 32];
    // the turn's records in order of their cells, the cell of each; per cell: its count, then what takes
    // a place in the turn's order to one in the plane's, and its first place in the turn's
    uint4 *local = smem;
    unsigned *shift = reinterpret_cast<unsigned *>(local + kLevelTurn);
    unsigned short *cell_of = reinterpret_cast<unsigned short *>(shift + sp.level_cells);
    unsigned short *begin = cell_of + kLevelTurn;
    load_level_table<REF>(lt, p);
    for (int i = threadIdx.x; i < sp.level_cells; i += kLevelThreads) shift[i] = 0u;
    __syncthreads();
    if (threadIdx.x == 0) plan_cells(ct, lt, p.L, sp.cell_bound);
    __syncthreads();
    grid_launch_dependents();
    grid_dependency_wait();     // everything above reads the caller's tables only
    if (!ct.fits) {      // (its points have no cells to be counted in)
        clear_unsorted_extras(p, sp);
        return;
    }
    const T *attn = reinterpret_cast<const T *>(p.attn);
    const int P = p.L * p.K;
    // (asked here, needed only when records leave: the points' loads do not wait for the answer)
    const bool unsorted = unsorted_call<T>(sp.header);
    for (unsigned turn = blockIdx.x; turn < sp.level_turns; turn += gridDim.x) {
        const unsigned heads = turn / (unsigned)p.G, stretch = heads / (unsigned)p.L;
        const int level = (int)(heads - stretch * (unsigned)p.L);
        SortLane c = sort_lane<kLevelThreads>(p, lt, ct, stretch * (unsigned)p.G + (turn - heads * (unsigned)p.G),
                                              sp.level_stretches, sp.level_queries, p.K, level * p.K);
        const int cell0 = ct.first[level], cells = ct.first[level + 1] - cell0;
        c.cell0 -= cell0;
        const bool in_shared = cells <= sp.level_cells;
        unsigned *cursor = sp.counts + (int64_t)c.plane * sp.cell_stride + cell0;
        uint4 *records = sp.records + (int64_t)c.plane * sp.plane_points;
        const int64_t pair0 = ((int64_t)c.b * p.Q + c.q0) * p.G + c.g;   // of the stretch's first query
        const int64_t base = pair0 * P + c.pt;
        const int nq = c.active ? c.nq : 0;
        auto record_of = [&](int q, float fc, float fr, float a, unsigned col) {
            return make_uint4(__float_as_uint(fc), __float_as_uint(fr), __float_as_uint(a),
                              ((unsigned)(c.q0 + q) << 12) | ((unsigned)c.pt << 3) | col);
        };
        unsigned at[kLevelPoints];     // cell << 16 | rank among the turn's points of the cell; ~0: skipped
        float3 kept[kLevelPoints];     // fractions and weight
        unsigned cols = 0;             // columns in their cells, three bits each
#pragma unroll
        for (int r0 = 0; r0 < kLevelPoints; r0 += kLevelBatch) {
            float2 xy[kLevelBatch], stats[SOFTMAX ? kLevelBatch : 1];
            T weight[kLevelBatch];
#pragma unroll
            for (int r = 0; r < kLevelBatch; ++r) {
                const int q = c.ql + (r0 + r) * c.step;
                if (q < nq) xy[r] = point_xy<T, REF>(p, c, base, q);
            }
#pragma unroll
            for (int r = 0; r < kLevelBatch; ++r) {
                const int q = c.ql + (r0 + r) * c.step;
                if (q < nq) {
                    if constexpr (SOFTMAX) stats[r] = sp.stats[pair0 + (int64_t)(q * p.G)];
                    weight[r] = attn[base + (int64_t)(q * (p.G * P))];
                }
            }
#pragma unroll
            for (int r = 0; r < kLevelBatch; ++r) {
                at[r0 + r] = ~0u;
                const int q = c.ql + (r0 + r) * c.step;
                if (q >= nq) continue;
                PointCell pc;
                if (!find_cell(c, xy[r], pc)) {
                    // a skipped point: exact zeros
                    store_point_gradients<T>(p, sp, base + (int64_t)(q * (p.G * P)), make_float2(0.f, 0.f), 0.f);
                } else {
                    float a = VT::to_float(weight[r]);
                    if constexpr (SOFTMAX) a = expf(a - stats[r].x) * stats[r].y;
                    if (in_shared) {
                        kept[r0 + r] = make_float3(pc.fc, pc.fr, a);
                        cols |= (unsigned)pc.col << (3 * (r0 + r));
                        at[r0 + r] = ((unsigned)pc.cell << 16) | atomicAdd(shift + pc.cell, 1u);
                    } else {
                        const unsigned place = atomicAdd(cursor + pc.cell, 1u);
                        if (place < (unsigned)sp.plane_points && !unsorted)
                            records[place] = record_of(q, pc.fc, pc.fr, a, (unsigned)pc.col);
                    }
                }
            }
        }
        if (unsorted) break;      // (every point's gradients are the walk's then)
        if (!in_shared) continue;
        __syncthreads();
        const unsigned points = scan_cells<kLevelThreads>(shift, begin, cursor, warp_sums, cells);
#pragma unroll
        for (int r = 0; r < kLevelPoints; ++r) {
            if (at[r] == ~0u) continue;
            const unsigned i = begin[at[r] >> 16] + (at[r] & 0xffffu);
            local[i] = record_of(c.ql + r * c.step, kept[r].x, kept[r].y, kept[r].z, (cols >> (3 * r)) & 7u);
            cell_of[i] = (unsigned short)(at[r] >> 16);
        }
        __syncthreads();
        // neighbours in the turn's order are neighbours in the plane's for as long as a cell lasts
#pragma unroll 4
        for (unsigned i = threadIdx.x; i < points; i += kLevelThreads) {
            const unsigned place = i + shift[cell_of[i]];
            if (place < (unsigned)sp.plane_points) records[place] = local[i];
        }
        __syncthreads();
        // (scan_cells wrote cells of whole eights)
        for (int i = threadIdx.x; i < ((cells + 7) & ~7); i += kLevelThreads) shift[i] = 0u;
        __syncthreads();
    }
    if (unsorted) clear_unsorted_extras(p, sp);
}

// ---- the walk over sorted points ------------------------------------------------------------------
template <typename T> struct Mma;
template <> struct Mma<__nv_bfloat16> {
    __device__ static __forceinline__ void run(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
        asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, "
                     "{%8, %9}, {%0, %1, %2, %3};"
                     : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
                     : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
    }
};
template <> struct Mma<__half> {
    __device__ static __forceinline__ void run(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
        asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, "
                     "{%8, %9}, {%0, %1, %2, %3};"
                     : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
                     : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
    }
};

__device__ __forceinline__ void cp_async16(uint32_t dst, const void *src) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_async_wait() {
    asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}
// transposes an 8x8 matrix of 16-bit elements held one row of pairs per four lanes
__device__ __forceinline__ uint32_t transpose8x8(uint32_t x) {
    uint32_t r;
    asm volatile("movmatrix.sync.aligned.m8n8.trans.b16 %0, %1;" : "=r"(r) : "r"(x));
    return r;
}
__device__ __forceinline__ uint4 lds16(uint32_t addr) {
    uint4 r;
    asm volatile("ld.shared.v4.u32 {%0, %1, %2, %3}, [%4];"
                 : "=r"(r.x), "=r"(r.y), "=r"(r.z), "=r"(r.w)
                 : "r"(addr)
                 : "memory");
    return r;
}
__device__ __forceinline__ uint2 lds8(uint32_t addr) {
    uint2 r;
    asm volatile("ld.shared.v2.u32 {%0, %1}, [%2];" : "=r"(r.x), "=r"(r.y) : "r"(addr) : "memory");
    return r;
}
__device__ __forceinline__ float lds4(uint32_t addr) {
    float r;
    asm volatile("ld.shared.f32 %0, [%1];" : "=f"(r) : "r"(addr) : "memory");
    return r;
}

constexpr int kStep = 32;          // points a warp takes at a time, one per lane

// byte offset of 16-byte chunk `chunk` of row `row` of a step's grad_out rows (2*D bytes each):
// chunks permuted so that the row-wise reads (8 lanes: two to four rows) touch every bank once.
// Rows 8 apart have the same permutation.
template <int D>
__device__ __forceinline__ uint32_t row_offset(int row, int chunk) {
    if constexpr (D == 32) return row * 64 + ((chunk ^ ((row >> 1) & 3)) << 4);
    if constexpr (D == 64) return row * 128 + ((chunk ^ ((row & 1) << 2) ^ ((row >> 1) & 3)) << 4);
    return row * 32 + ((chunk ^ ((row >> 2) & 1)) << 4);
}

// What a lane holds of one row of a D-channel matrix whose k index runs over channels: register
// 2*s + h is the k = 2*(lane%4) + {0,1} + 8*h pair of k-step s.  The channels are dealt to k in
// the order a 16-byte load per lane delivers them (lane c of four: channels 8c .. 8c+7 of every
// 32; D = 16: 4c .. 4c+3).  Both operands of the dot products use it, so it does not matter
// there, and in the transposed registers it leaves each lane with adjacent channels.
template <int D>
__device__ __forceinline__ void row_from_shared(uint32_t (&w)[D / 8], uint32_t base,
                                                const uint32_t (&at)[D == 64 ? 2 : 1]) {
    if constexpr (D == 16) {
        const uint2 v = lds8(base + at[0]);
        w[0] = v.x, w[1] = v.y;
    } else {
#pragma unroll
        for (int h = 0; h < D / 32; ++h) {
            const uint4 v = lds16(base + at[h]);
            w[4 * h] = v.x, w[4 * h + 1] = v.y, w[4 * h + 2] = v.z, w[4 * h + 3] = v.w;
        }
    }
}
template <typename T, int D>
__device__ __forceinline__ void row_from_global(uint32_t (&w)[D / 8], const T *row, int c, bool inside) {
    if constexpr (D == 16) {
        uint2 v = make_uint2(0u, 0u);
        if (inside) v = __ldg(reinterpret_cast<const uint2 *>(row) + c);
        w[0] = v.x, w[1] = v.y;
    } else {
#pragma unroll
        for (int h = 0; h < D / 32; ++h) {
            uint4 v = make_uint4(0u, 0u, 0u, 0u);
            if (inside) v = ldg16(reinterpret_cast<const uint4 *>(row) + h * 4 + c);
            w[4 * h] = v.x, w[4 * h + 1] = v.y, w[4 * h + 2] = v.z, w[4 * h + 3] = v.w;
        }
    }
}

// Adds one accumulated pixel row (8 pixels x D channels; this lane: pixel lane/4, the channels
// of its loads) into the float16 image.
template <int D>
__device__ __forceinline__ void flush_row(float (&acc)[D / 8][4], int half, float scale, __half *pixel,
                                          bool inside, int c) {
    uint32_t v[D / 8];
#pragma unroll
    for (int t = 0; t < D / 8; ++t)
        v[t] = VecTraits<__half>::pack2(make_float2(acc[t][2 * half] * scale, acc[t][2 * half + 1] * scale));
    if (!inside) return;
    if constexpr (D == 16) {
        asm volatile("red.relaxed.gpu.global.add.noftz.v2.f16x2 [%0], {%1, %2};" ::"l"(pixel + 4 * c), "r"(v[0]),
                     "r"(v[1]));
    } else {
#pragma unroll
        for (int h = 0; h < D / 32; ++h)
            asm volatile("red.relaxed.gpu.global.add.noftz.v4.f16x2 [%0], {%1, %2, %3, %4};" ::"l"(
                             pixel + 32 * h + 8 * c),
                         "r"(v[4 * h]), "r"(v[4 * h + 1]), "r"(v[4 * h + 2]), "r"(v[4 * h + 3]));
    }
}

// What bounds the walk is the latency of a step's chain beside the SM's load/store pipe, about five of its
// cycles a point (ncu, the headline shape: 63 % busy while the SM works, issue slots 47 %, tensor cores
// 29 %): without the two stores per point to addresses of their own the call takes 364 us instead of 398,
// the rest goes through shared memory.  Hence the weights' way over the tensor cores below.  More warps do
// not help - 12, 16, 20, 24 per SM: 252, 246, 261, 312 us when this kernel took 246 - nor did having grad_out
// rows in registers instead of shared memory (300 us), or the next cell's value row early (257 us).
// (CTAs per SM the registers are held to: more than these spill)
constexpr int walk_ctas(int D) { return D == 64 ? 3 : 4; }
__host__ __device__ constexpr int walk_warp_bytes(int D) { return 2 * kStep * D * 2 + kStep * 16 + kStep / 8 * 512; }

template <typename T, int D, bool REF>
__global__ void __launch_bounds__(kWalkWarps * 32, walk_ctas(D))
    sorted_walk_kernel(const __grid_constant__ Params p, const __grid_constant__ SortPlan sp, bool softmax) {
    using VT = VecTraits<T>;
    constexpr int NT = D / 8;       // channel tiles of eight
    constexpr int KS = D / 16;      // k-steps of the dot products
    constexpr bool kSplit = std::is_same<T, __nv_bfloat16>::value;   // weights as two bf16 terms
    extern __shared__ uint4 smem[];
    __shared__ LevelTable lt;
    __shared__ CellTable ct;
    load_level_table(lt, p);
    __syncthreads();
    if (threadIdx.x == 0) plan_cells(ct, lt, p.L, sp.cell_bound);
    __syncthreads();

    grid_launch_dependents();
    // (what the kernels before wrote is read with plain loads: an invariant load may be moved
    // above the wait)
    grid_dependency_wait();
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int j = lane >> 2, c = lane & 3;
    if (unsorted_call<T>(sp.header)) {
        accumulate_unsorted<T, D>(p, sp, lt, softmax);
        return;
    }
    const int cells = ct.first[p.L];
    const int GD = p.G * D, GP = p.G * p.L * p.K;
    // float16 weights are kept near 1 whatever their largest magnitude
    float weight_scale = 1.f;
    if constexpr (!kSplit) {
        const float ma = softmax ? 1.f : magnitude_from_bits<T>(sp.header[1]);
        if (ma > 0.f && ma < INFINITY) weight_scale = ldexpf(1.f, -ilogbf(ma));
    }
    const float flush_scale =
        ldexpf(1.f, grad_scale_exponent<T>(sp.header, p.Q, p.K, softmax)) / weight_scale;

    // shared memory of the warp: grad_out rows of two steps, the step's weights, and the dot
    // products of the window's 16 pixels with its points, in blocks of eight points
    constexpr int kRows = kStep * D * 2;   // bytes
    constexpr int kWarpBytes = walk_warp_bytes(D);
    uint4 *mine = smem + warp * (kWarpBytes / 16);
    const uint32_t s_rows = (uint32_t)__cvta_generic_to_shared(mine);
    const uint32_t s_weights = s_rows + 2 * kRows;
    const uint32_t s_dots = s_weights + kStep * 16;
    // (rows that a short step leaves out are multiplied by zero: they have to be finite)
    for (int i = lane; i < 2 * kRows / 16; i += 32) mine[i] = make_uint4(0u, 0u, 0u, 0u);
    __syncwarp();
    uint32_t at_row[D == 64 ? 2 : 1];      // this lane's part of row j
    if constexpr (D == 16)
        at_row[0] = row_offset<D>(j, c >> 1) + (c & 1) * 8;
    else
#pragma unroll
        for (int h = 0; h < D / 32; ++h) at_row[h] = row_offset<D>(j, h * 4 + c);
    // the lane's share of the copies: row r0 of every kRowsPerTurn, one 16-byte chunk.  Rows of
    // D = 64's odd turns are four on, where the permutation differs in one bit
    constexpr int kRowsPerTurn = 32 / NT;
    const int r0 = lane / NT;
    const uint32_t at_copy = row_offset<D>(r0, lane % NT);
    // the identity as the A operand of an m16n8k16 product (upper left and lower right corner)
    const uint32_t one = VT::pack2(make_float2(j == 2 * c ? 1.f : 0.f, j == 2 * c + 1 ? 1.f : 0.f));

    // (short runs belong on the finest level)
    const bool coarse_first = lt.H[p.L - 1] * lt.W[p.L - 1] > lt.H[0] * lt.W[0];
    // ---- runs of places, handed out as the warps come for them
    for (;;) {
        unsigned run = 0;
        if (lane == 0) run = atomicAdd(sp.header + kNextItem, 1u);
        run = __shfl_sync(0xffffffffu, run, 0);
        if (run >= sp.all_runs) break;
        int k = 0;
#pragma unroll
        for (int i = 1; i < kRunKinds; ++i) k += run >= sp.runs[i].run0;
        const WalkRuns &kind = sp.runs[k];
        const unsigned nth = (run - kind.run0) / kind.each;
        const int plane = (int)(kind.plane0 + nth);
        unsigned unit = kind.unit0 + ((run - kind.run0 - nth * kind.each) << kind.log2_size);
        if (coarse_first) unit = (unsigned)sp.items - unit - (1u << kind.log2_size);
        int pos = (int)unit * sp.item_points;
        const uint4 *records = sp.records + (int64_t)plane * sp.plane_points;
        // (places beyond the plane's points hold no record: what is read there is not kept)
        uint4 rec = __ldcg(records + min((int64_t)(pos + lane), sp.plane_points - 1));
        int cell = sp.item_cell[(unsigned)plane * (unsigned)sp.items + unit];
        const int total = (int)sp.offsets[(int64_t)plane * sp.cell_stride + cells];
        const int stop = min(pos + (sp.item_points << kind.log2_size), total);
        if (pos >= stop) continue;
        if (pos + lane >= total) rec = make_uint4(0u, 0u, 0u, 0u);
        const unsigned *offsets = sp.offsets + (int64_t)plane * sp.cell_stride;
        const int b = plane / p.G, g = plane - b * p.G;
        const T *value = reinterpret_cast<const T *>(p.value) + ((int64_t)b * p.S * p.G + g) * D;
        const T *grad_out = reinterpret_cast<const T *>(p.grad_out) + ((int64_t)b * p.Q * p.G + g) * D;
        __half *image = reinterpret_cast<__half *>(p.grad_value) + ((int64_t)b * p.S * p.G + g) * D;
        // element of the per-point outputs that point 0 of query 0 of this plane has
        const int64_t plane_point = ((int64_t)b * p.Q * p.G + g) * (p.L * p.K);

        auto fetch_record = [&](int place) { return __ldcg(records + min(place + lane, total - 1)); };
        const T *chunk_of_row = grad_out + lane % NT * 8;
        auto fetch_rows = [&](const uint4 &rec, int n, uint32_t buffer) {
            const unsigned mine = rec.w >> 12;
#pragma unroll
            for (int i = 0; i < kStep / kRowsPerTurn; ++i) {
                const unsigned q = __shfl_sync(0xffffffffu, mine, i * kRowsPerTurn + r0);
                const uint32_t to = buffer + i * kRowsPerTurn * D * 2 + (D == 64 && (i & 1) ? at_copy ^ 32u : at_copy);
                if (i * kRowsPerTurn + r0 < n) cp_async16(to, chunk_of_row + (size_t)(q * (unsigned)GD));
            }
            cp_async_commit();
        };

        // ---- where the run begins
        int level = 0, strip_end = 0, row = 0, H = 0, W = 0, col0 = 0, start = 0;
        auto enter_strip = [&]() {
            while (level + 1 < p.L && cell >= ct.first[level + 1]) ++level;
            const int rows = ct.rows[level];
            const int strip = (cell - ct.first[level]) / rows;
            strip_end = ct.first[level] + (strip + 1) * rows;
            row = cell - (strip_end - rows) - 1;
            H = lt.H[level], W = lt.W[level], start = lt.start[level];
            col0 = strip * kCols - 1;
        };
        enter_strip();
        int window = cell;      // the lanes hold the ends of cells window .. window + 31
        int ends = (int)offsets[min(window + 1 + lane, cells)];
        // the first cell at or after `window` that ends beyond `place` (which is below total)
        auto cell_at = [&](int place, int &end) {
            unsigned more;
            while ((more = __ballot_sync(0xffffffffu, ends > place)) == 0) {
                window += 32;
                ends = (int)offsets[min(window + 1 + lane, cells)];
            }
            const int k = __ffs(more) - 1;
            end = __shfl_sync(0xffffffffu, ends, k);
            return window + k;
        };

        uint32_t vtop[NT], vbot[NT];     // the window's value rows, this lane's pixel
        auto load_row = [&](uint32_t (&w)[NT], int r) {
            const int x = col0 + j;
            row_from_global<T, D>(w, value + (int64_t)(start + r * W + x) * GD, c,
                                  (unsigned)r < (unsigned)H && (unsigned)x < (unsigned)W);
        };
        load_row(vtop, row);
        load_row(vbot, row + 1);
        float acc[NT][4];
#pragma unroll
        for (int t = 0; t < NT; ++t) acc[t][0] = acc[t][1] = acc[t][2] = acc[t][3] = 0.f;
        auto flush = [&](int half, int r) {
            const int x = col0 + j;
            flush_row<D>(acc, half, flush_scale, image + (int64_t)(start + r * W + x) * GD,
                         (unsigned)r < (unsigned)H && (unsigned)x < (unsigned)W, c);
        };

        // ---- first steps
        int cell_end;
        cell_at(pos, cell_end);
        int n = min(min(kStep, cell_end - pos), stop - pos);
        uint4 rec_next = fetch_record(pos + n);
        uint32_t buffer = s_rows;
        fetch_rows(rec, n, buffer);

        for (;;) {
            // ---- what comes next, and its rows on their way
            const int pos_next = pos + n;
            const bool more = pos_next < stop;
            int cell_next = cell, n_next = 0;
            if (more) {
                if (pos_next >= cell_end) cell_next = cell_at(pos_next, cell_end);
                n_next = min(min(kStep, cell_end - pos_next), stop - pos_next);
            }
            const uint4 rec_after = fetch_record(pos_next + n_next);
            const uint32_t other = buffer ^ s_rows ^ (s_rows + kRows);
            fetch_rows(rec_next, n_next, other);

            // ---- one lane per point: its four weights
            const float fc = __uint_as_float(rec.x), fr = __uint_as_float(rec.y), a = __uint_as_float(rec.z);
            {
                const float w = lane < n ? a * weight_scale : 0.f;
                const float top = w * (1.f - fr), bot = w * fr;
                const float2 tw = make_float2(top * (1.f - fc), top * fc), bw = make_float2(bot * (1.f - fc), bot * fc);
                uint4 s;
                s.x = VT::pack2(tw);
                s.y = VT::pack2(bw);
                if constexpr (kSplit) {
                    // what the first term leaves; three low bits of it hold the column in the cell
                    const float2 th = VT::unpack2(s.x), bh = VT::unpack2(s.y);
                    s.z = VT::pack2(make_float2(tw.x - th.x, tw.y - th.y));
                    s.w = (VT::pack2(make_float2(bw.x - bh.x, bw.y - bh.y)) & ~7u) | (rec.w & 7u);
                } else {
                    s.z = 0u;
                    s.w = rec.w & 7u;
                }
                asm volatile("st.shared.v4.u32 [%0], {%1, %2, %3, %4};" ::"r"(s_weights + lane * 16), "r"(s.x),
                             "r"(s.y), "r"(s.z), "r"(s.w)
                             : "memory");
            }
            cp_async_wait<1>();
            __syncwarp();
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                if (h == 1 && n <= 16) break;
                uint32_t go[2][NT];
                uint32_t hi[4], lo[4];     // weights of pixels x points: the A operand
#pragma unroll
                for (int e = 0; e < 2; ++e) {
                    const int block = h * 2 + e;
                    row_from_shared<D>(go[e], buffer + block * 8 * D * 2, at_row);
                    // dot products of the window's pixels with eight points
                    float dot[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
                    for (int s = 0; s < KS; ++s) {
                        const uint32_t av[4] = {vtop[2 * s], vbot[2 * s], vtop[2 * s + 1], vbot[2 * s + 1]};
                        Mma<T>::run(dot, av, go[e][2 * s], go[e][2 * s + 1]);
                    }
                    const uint32_t to = s_dots + block * 512 + lane * 8;   // pixel j: 32 bytes, points 2c and 2c+1
                    asm volatile("st.shared.v2.f32 [%0], {%1, %2};" ::"r"(to), "f"(dot[0]), "f"(dot[1]) : "memory");
                    asm volatile("st.shared.v2.f32 [%0], {%1, %2};" ::"r"(to + 256), "f"(dot[2]), "f"(dot[3]) : "memory");
                    // The weights with the pixels as k, the points as n: this lane has point j and
                    // pixel columns 2c, 2c + 1 of either row.  The point's words hold its columns col
                    // and col + 1; they go where 2c - col is -1, 0 or 1 (shift 0, 16, 32).
                    const uint4 w = lds16(s_weights + (block * 8 + j) * 16);
                    const uint32_t shift = 16u + 32u * c - 16u * (w.w & 7u);
                    uint32_t pick = __funnelshift_rc(0x32101044u, 0x44444432u, shift);
                    if (shift > 32u) pick = 0x4444u;
                    // a product with the identity turns that into pixels x points, which is what the
                    // accumulation below takes: the tensor cores have time for it, the shared memory
                    // that four words per lane and point would pass through has not
                    float t[4] = {0.f, 0.f, 0.f, 0.f};
                    const uint32_t unit[4] = {one, 0u, 0u, one};
                    Mma<T>::run(t, unit, __byte_perm(w.x, 0u, pick), __byte_perm(w.y, 0u, pick));
                    hi[2 * e] = VT::pack2(make_float2(t[0], t[1]));
                    hi[2 * e + 1] = VT::pack2(make_float2(t[2], t[3]));
                    if constexpr (kSplit) {
                        t[0] = t[1] = t[2] = t[3] = 0.f;
                        Mma<T>::run(t, unit, __byte_perm(w.z, 0u, pick), __byte_perm(w.w & ~7u, 0u, pick));
                        lo[2 * e] = VT::pack2(make_float2(t[0], t[1]));
                        lo[2 * e + 1] = VT::pack2(make_float2(t[2], t[3]));
                    }
                }
#pragma unroll
                for (int t = 0; t < NT; ++t) {
                    const uint32_t b0 = transpose8x8(go[0][t]), b1 = transpose8x8(go[1][t]);
                    Mma<T>::run(acc[t], hi, b0, b1);
                    if constexpr (kSplit) Mma<T>::run(acc[t], lo, b0, b1);
                }
            }
            __syncwarp();
            // ---- gradients of the points: one lane each
            if (lane < n) {
                const uint32_t at = s_dots + (lane >> 3) * 512 + (rec.w & 7u) * 32 + (lane & 7) * 4;
                const float d00 = lds4(at), d01 = lds4(at + 32), d10 = lds4(at + 256), d11 = lds4(at + 288);
                const float wr0 = 1.f - fr, wc0 = 1.f - fc;
                const float gx = wr0 * (d01 - d00) + fr * (d11 - d10);
                const float gy = wc0 * (d10 - d00) + fc * (d11 - d01);
                const float ga = wr0 * wc0 * d00 + wr0 * fc * d01 + fr * wc0 * d10 + fr * fc * d11;
                const unsigned q = rec.w >> 12;
                const int64_t e = plane_point + (size_t)(q * (unsigned)GP + ((rec.w >> 3) & 511u));
                float2 dpix = make_float2((float)W, (float)H);
                if constexpr (REF) {
                    dpix = offset_derivative(p, (int64_t)b * p.Q + q, level, dpix.x, dpix.y);
                    store_point_gradients<T>(p, sp, e, make_float2(a * dpix.x * gx, a * dpix.y * gy), ga);
                } else {
                    reinterpret_cast<float2 *>(p.grad_loc)[e] = make_float2(a * dpix.x * gx, a * dpix.y * gy);
                    sp.grad_prob[e] = ga;
                }
            }
            __syncwarp();
            if (!more) break;
            pos = pos_next;
            n = n_next;
            buffer = other;
            rec = rec_next;
            rec_next = rec_after;
            if (cell_next == cell) continue;
            // ---- into the next cell
            if (cell_next == cell + 1 && cell_next < strip_end) {
                // one row down: the upper row is complete, the lower one becomes the upper
                flush(0, row);
                ++row;
                cell = cell_next;
#pragma unroll
                for (int t = 0; t < NT; ++t) {
                    acc[t][0] = acc[t][2], acc[t][1] = acc[t][3];
                    acc[t][2] = acc[t][3] = 0.f;
                    vtop[t] = vbot[t];
                }
                load_row(vbot, row + 1);
            } else {
                flush(0, row);
                flush(1, row + 1);
                if (cell_next < strip_end) {
                    row += cell_next - cell;
                    cell = cell_next;
                } else {
                    cell = cell_next;
                    enter_strip();
                }
#pragma unroll
                for (int t = 0; t < NT; ++t) acc[t][0] = acc[t][1] = acc[t][2] = acc[t][3] = 0.f;
                load_row(vtop, row);
                load_row(vbot, row + 1);
            }
        }
        flush(0, row);
        flush(1, row + 1);
        cp_async_wait<0>();
    }
}

// ---- last pass: grad_value from the scaled float16 image, in place; softmax Jacobian --------------
template <typename T, bool SOFTMAX>
__global__ void __launch_bounds__(256, 4) sorted_finish_kernel(const __grid_constant__ Params p,
                                                              const __grid_constant__ SortPlan sp) {
    grid_dependency_wait();
    using VT = VecTraits<T>;
    const int64_t stride = (int64_t)gridDim.x * blockDim.x;
    const int64_t first = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    const int P = p.L * p.K;
    T *grad_attn = reinterpret_cast<T *>(p.grad_attn);
    if constexpr (SOFTMAX) {
        // gradient of the logits, p_i (g_i - sum_j p_j g_j): one thread per (query, head) pair,
        // whose P values are adjacent
        const T *attn = reinterpret_cast<const T *>(p.attn);
        const int64_t pairs = p.B * p.Q * p.G;
        for (int64_t pair = first; pair < pairs; pair += stride) {
            const float *g = sp.grad_prob + pair * P;
            const float2 st = sp.stats[pair];
            float inner = 0.f;
            if ((P & 3) == 0) {
#pragma unroll 4
                for (int i = 0; i < P; i += 4) {
                    const uint2 v = __ldg(reinterpret_cast<const uint2 *>(attn + pair * P + i));
                    const float2 x0 = VT::unpack2(v.x), x1 = VT::unpack2(v.y);
                    const float4 gv = *reinterpret_cast<const float4 *>(g + i);
                    inner += expf(x0.x - st.x) * gv.x + expf(x0.y - st.x) * gv.y + expf(x1.x - st.x) * gv.z +
                             expf(x1.y - st.x) * gv.w;
                }
                inner *= st.y;
#pragma unroll 4
                for (int i = 0; i < P; i += 4) {
                    const uint2 v = __ldg(reinterpret_cast<const uint2 *>(attn + pair * P + i));
                    const float2 x0 = VT::unpack2(v.x), x1 = VT::unpack2(v.y);
                    const float4 gv = *reinterpret_cast<const float4 *>(g + i);
                    const float2 a = make_float2(expf(x0.x - st.x) * st.y * (gv.x - inner),
                                                 expf(x0.y - st.x) * st.y * (gv.y - inner));
                    const float2 b = make_float2(expf(x1.x - st.x) * st.y * (gv.z - inner),
                                                 expf(x1.y - st.x) * st.y * (gv.w - inner));
                    *reinterpret_cast<uint2 *>(grad_attn + pair * P + i) = make_uint2(VT::pack2(a), VT::pack2(b));
                }
            } else {
                for (int i = 0; i < P; ++i) inner += expf(VT::to_float(attn[pair * P + i]) - st.x) * g[i];
                inner *= st.y;
                for (int i = 0; i < P; ++i)
                    grad_attn[pair * P + i] =
                        VT::from_float(expf(VT::to_float(attn[pair * P + i]) - st.x) * st.y * (g[i] - inner));
            }
        }
    } else {
        // four values a thread (the first element of a pass is 16-byte aligned only if the
        // samples before it are; grad_prob always is)
        const int64_t points = p.B * p.Q * p.G * P;
        const bool whole = (reinterpret_cast<uintptr_t>(grad_attn) & 7u) == 0;
        const int64_t body = whole ? points / 4 : 0;
        for (int64_t i = first; i < body; i += stride) {
            const float4 g = __ldcs(reinterpret_cast<const float4 *>(sp.grad_prob) + i);
            const uint2 v = make_uint2(VT::pack2(make_float2(g.x, g.y)), VT::pack2(make_float2(g.z, g.w)));
            __stcs(reinterpret_cast<uint2 *>(grad_attn) + i, v);
        }
        for (int64_t i = body * 4 + first; i < points; i += stride) grad_attn[i] = VT::from_float(sp.grad_prob[i]);
    }
    const int exponent = grad_scale_exponent<T>(sp.header, p.Q, p.K, SOFTMAX);
    if (unsorted_call<T>(sp.header)) {
        __shared__ LevelTable lt;
        __shared__ int extra_range[2];
        load_level_table(lt, p);
        __syncthreads();
        if (threadIdx.x == 0) {
            plan_replicas(lt, p);
            find_extra_range(lt, p.L, extra_range);
        }
        __syncthreads();
        finalize_image<T>(p, lt, extra_range, exponent, reinterpret_cast<const uint4 *>(p.grad_value),
                          unsorted_extras(sp), (int)blockIdx.x, (int)gridDim.x);
        return;
    }
    const float inv = ldexpf(1.f, -exponent);
    uint4 *gv = reinterpret_cast<uint4 *>(p.grad_value);
    const int64_t total = p.B * p.S * (p.G * p.D / 8);
    constexpr int kTurn = 4;
    for (int64_t v0 = first; v0 < total; v0 += kTurn * stride) {
        uint4 raw[kTurn];
#pragma unroll
        for (int u = 0; u < kTurn; ++u)
            raw[u] = v0 + u * stride < total ? gv[v0 + u * stride] : make_uint4(0u, 0u, 0u, 0u);
#pragma unroll
        for (int u = 0; u < kTurn; ++u) {
            if (v0 + u * stride >= total) break;
            if ((raw[u].x | raw[u].y | raw[u].z | raw[u].w) == 0u) continue;   // zero in either type
            float2 f[4];
            VecTraits<__half>::unpack(raw[u], f);
#pragma unroll
            for (int i = 0; i < 4; ++i) f[i] = fmul2(f[i], make_float2(inv, inv));
            gv[v0 + u * stride] = VT::pack(f);
        }
    }
}

template <typename T, int D, bool REF>
cudaError_t launch_walk(const Params &p, const SortPlan &sp, bool softmax, cudaStream_t stream) {
    constexpr size_t smem = (size_t)kWalkWarps * walk_warp_bytes(D);
    static_assert(smem <= kPlainSmem, "would have to be asked for on every device");
    auto walk = sorted_walk_kernel<T, D, REF>;
    // as many CTAs as the GPU holds at once; the warps fetch their runs, so that any number
    // serves (asked once: every GPU this is built for has the same limits)
    static const int resident = [walk] {
        int device = 0, sms = 0, per_sm = 0;
        if (cudaGetDevice(&device) != cudaSuccess ||
            cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device) != cudaSuccess ||
            cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, walk, kWalkWarps * 32, smem) != cudaSuccess)
            return 0;
        return sms * per_sm;
    }();
    if (resident <= 0) return cudaErrorInvalidConfiguration;
    const int64_t ctas = ((int64_t)sp.all_runs + kWalkWarps - 1) / kWalkWarps;
    return launch_after_predecessor(walk, (unsigned)std::min<int64_t>(ctas, resident), kWalkWarps * 32, smem, stream,
                                    p, sp, softmax);
}

template <typename T, int D, bool SOFTMAX>
cudaError_t launch_sorted_typed(const Params &p, const SortPlan &sp, cudaStream_t stream) {
    const unsigned planes = (unsigned)(p.B * p.G);
    const size_t hist = (size_t)sp.count_cells * sizeof(unsigned);
    const size_t scatter_smem = (size_t)kSortCtaPoints * 20 + (size_t)sp.shared_cells * 6;
    cudaError_t e = cudaMemsetAsync(sp.header, 0, sp.cleared_bytes, stream);
    if (e != cudaSuccess) return e;
    auto count = p.ref != nullptr     ? sort_count_kernel<T, SOFTMAX, true, false>
                 : sp.count_by_level ? sort_count_kernel<T, SOFTMAX, false, true>
                                     : sort_count_kernel<T, SOFTMAX, false, false>;
    auto scatter = p.ref != nullptr ? sort_scatter_kernel<T, SOFTMAX, true> : sort_scatter_kernel<T, SOFTMAX, false>;
    count<<<planes * (unsigned)sp.count_ctas + sp.prepare_ctas, count_threads(sp.count_by_level), hist, stream>>>(p, sp);
    if (sp.scatter_by_level) {
        auto by_level = p.ref != nullptr ? sort_scatter_level_kernel<T, SOFTMAX, true>
                                         : sort_scatter_level_kernel<T, SOFTMAX, false>;
        const size_t smem = (size_t)kLevelTurn * 18 + (size_t)sp.level_cells * 6;
        e = allow_most_smem(by_level);
        if (e != cudaSuccess) return e;
        static Residency residency[2];
        const unsigned resident = residency[p.ref != nullptr].ctas(by_level, kLevelThreads, smem);
        e = launch_after_predecessor(by_level, resident == 0 ? sp.level_turns : std::min(resident, sp.level_turns),
                                     kLevelThreads, smem, stream, p, sp);
    } else {
        e = allow_most_smem(scatter);
        if (e != cudaSuccess) return e;
        e = launch_after_predecessor(scatter, planes * (unsigned)sp.chunks, kSortThreads, scatter_smem, stream, p, sp);
    }
    if (e != cudaSuccess) return e;
    e = p.ref != nullptr ? launch_walk<T, D, true>(p, sp, SOFTMAX, stream)
                         : launch_walk<T, D, false>(p, sp, SOFTMAX, stream);
    if (e != cudaSuccess) return e;
    const int64_t vecs = p.B * p.S * (p.G * D / 8);
    const int64_t blocks = (vecs + 1023) / 1024;
    return launch_after_predecessor(sorted_finish_kernel<T, SOFTMAX>, (unsigned)std::min<int64_t>(blocks, 148 * 4),
                                    256, 0, stream, p, sp);
}

template <typename T, bool SOFTMAX>
cudaError_t launch_sorted_head(const Params &p, const SortPlan &sp, cudaStream_t stream) {
    switch (p.D) {
        case 16: return launch_sorted_typed<T, 16, SOFTMAX>(p, sp, stream);
        case 32: return launch_sorted_typed<T, 32, SOFTMAX>(p, sp, stream);
        case 64: return launch_sorted_typed<T, 64, SOFTMAX>(p, sp, stream);
        default: return cudaErrorInvalidValue;
    }
}

int64_t round_up(int64_t n, int64_t to) { return (n + to - 1) / to * to; }

}  // namespace

// Where sorting wins (B200, backward call, us, direct -> sorted; bf16, 8 heads, 4 points):
//   points per value position   12: everything below; 7, random positions: 116 -> 126; 4: 116 ->
//                               158 (cells of a few points leave the tile products half empty)
//   points in the call          0.5 M 60 -> 63, 1.0 M 86 -> 73 .. 89 -> 85, 2 M 147 -> 133, 4 M
//                               265 -> 231, 8 M 512 -> 435, 33 M 1973 -> 1654
//   channels per head           16: 430 -> 380, 32: 512 -> 435, 64 (half the heads): 441 -> 304
//   offsets instead of          the arithmetic of the locations is done once more: 16 channels
//   locations                   228 -> 251, 32: 157 -> 159 at 2 M points, 285 -> 275 at 4 M, 551
//                               -> 503 at 8 M; 64 (1.8 M points): 241 -> 202
//   positions                   12 points per position, 2 samples, 59 104 positions: 16 channels 590 -> 574,
//                               32: 696 -> 635; 73 549: 739 -> 775, 880 -> 866; 16 points on four levels
//                               1148 -> 1033.  From about 85 000 the finest level has more than kLevelCells
//                               cells and its records leave unordered, one sample: 102 900 552 -> 668, 620 ->
//                               757, 134 400 720 -> 840, 805 -> 900.  The line lies below, at 55 000, where
//                               what is left to gain, 2 to 10 %, is not worth three times the scratch, but for
//                               64 channels (4 heads, 12 points, 59 104: one sample 308 -> 224, two 599 ->
//                               416) and 24 points of 32 (73 549: one sample 912 -> 679, two 1805 -> 1359).
//                               Offsets: more than kSharedCells cells from there on
bool sorting_pays(const Params &p, int dtype, bool offsets) {
    const int64_t P = (int64_t)p.L * p.K, points = p.B * p.G * p.Q * P;
    if (dtype != 1 && dtype != 2) return false;
    if (p.D != 16 && p.D != 32 && p.D != 64) return false;
    // (fields of a record; 32-bit offsets inside a sample; cells in 16 bits beside a rank)
    if (P > 512 || p.Q > (1 << 20) || p.Q * P * p.G >= (1ll << 31) || p.Q * p.G * p.D >= (1ll << 31) ||
        p.S >= (1ll << 29))
        return false;
    if (p.Q * P < 8 * p.S) return false;
    if (p.S > 55000 &&
        (offsets || p.L > 4 || p.D == 16 || (p.D == 32 && p.Q * P < 24 * p.S)))
        return false;
    if (offsets && p.D < 64) return p.D == 32 && points >= 3000000;
    return points >= 1000000;
}

// With room for some samples only, they take turns; a turn of few points costs more in launches
// and partly filled waves than sorting saves (four turns of 2 M points: 546 us against 512).
int64_t sorted_samples_per_turn(const Params &p, bool softmax, int64_t bytes) {
    int64_t n = p.B;
    while (n > 0 && sorted_workspace_bytes(p, softmax, n) > bytes) n = n > 8 ? n - n / 8 : n - 1;
    if (n == 0 || n == p.B) return n;
    const int64_t turns = (p.B + n - 1) / n;
    n = (p.B + turns - 1) / turns;                       // turns of about the same size
    return n * p.G * p.Q * p.L * p.K >= 4000000 ? n : 0;
}

Params samples_of(const Params &p, int64_t b, int64_t n) {
    // (16-bit values; offsets may be of that type too)
    const int64_t GD = (int64_t)p.G * p.D, pairs = p.Q * p.G, points = pairs * p.L * p.K;
    const int64_t point_bytes = p.ref != nullptr && p.offsets16 ? 4 : 8;
    auto at = [b](const void *base, int64_t bytes) {
        return const_cast<char *>(static_cast<const char *>(base)) + b * bytes;
    };
    Params r = p;
    r.B = n;
    r.value = at(p.value, p.S * GD * 2);
    r.loc = reinterpret_cast<const float *>(at(p.loc, points * point_bytes));
    r.attn = at(p.attn, points * 2);
    r.grad_out = at(p.grad_out, p.Q * GD * 2);
    r.grad_value = at(p.grad_value, p.S * GD * 2);
    r.grad_loc = reinterpret_cast<float *>(at(p.grad_loc, points * point_bytes));
    r.grad_attn = at(p.grad_attn, points * 2);
    if (p.ref != nullptr) r.ref = p.ref + b * p.Q * p.L * p.ref_coords;
    return r;
}

int64_t sorted_workspace_bytes(const Params &p, bool softmax, int64_t samples) {
    SortPlan sp;
    return plan_sorted(sp, p, softmax, samples, nullptr);
}

// Runs of the walk.  Where a run ends, the sums of two pixel rows leave it unfinished and meet in float16
// once more.  So no plane is in more runs than if all had `length` points: 128 to 256, by what a warp's
// share leaves room for, and more where a pixel collects hundreds of points (all have it there, and where
// there are fewer than two for every warp).  Within that, a long run is flushed and started less often, but
// the last ones to end leave the other warps idle: runs have twice the length, and the last planes - all
// planes of a small call - have some of once and of half of it too, together one and two for every warp.
// Of these planes the long runs are handed out first; the short ones lie on their finest level, where the
// fewest points share a pixel.
// Backward, B200, us, all of `length` -> this: headline shape 408 -> 398, 16 samples 1618 -> 1571, four odd
// levels in float16 430 -> 415, 512-pixel pyramid 8 samples 224 -> 215, with offsets 271 -> 258, 4 samples 135
// -> 127; 64 channels: ragged pyramid with offsets 208 -> 194, 512 pixels 16 samples 298 -> 270.  Which planes:
// eight runs' worth of them for every warp (sixteen: 415 at the headline shape, all 431: what a plane's levels
// share is no longer in L2 when its short runs come), but sixteen at 64 channels (eight: 198, 277).  No short
// runs, four of `length` left for every warp: 402, 1586, 423, 223, 271.
// Runs of 512 points getting shorter to 64 in the order of the planes take 399, 1579, 413, 217, 258, 124,
// 196, 276, but the float16 grad_value of the last plane is 5.6e-4 off then and of the first 3.6e-4 (four
// odd levels 8.2e-4 and 4.2e-4), where they are 3.7e-4 and 3.6e-4 (4.3e-4, 4.2e-4) with these runs and 4.0e-4
// (5.0e-4) with all of `length`.
void plan_runs(SortPlan &sp, const Params &p, int64_t planes) {
    const int64_t warps = 148 * kWalkWarps * walk_ctas(p.D);
    const int64_t share = planes * sp.plane_points / (148 * 16 * 4);
    const int64_t density = sp.plane_points / std::max<int64_t>(p.S, 1);
    const int64_t length = std::min<int64_t>(256, std::max<int64_t>(128, share / 32 * 32)) *
                           std::min<int64_t>(16, 1 + density / 128);
    sp.item_points = (int)(length / 2);
    sp.items = (int)round_up((sp.plane_points + sp.item_points - 1) / sp.item_points, 4);   // (no run in two planes)
    unsigned runs = 0;
    int kind = 0;
    auto add = [&](int64_t plane, int64_t of_planes, int64_t unit, int64_t each, int log2_size) {
        sp.runs[kind++] = {runs, (unsigned)plane, (unsigned)std::max<int64_t>(each, 1), (unsigned)unit, log2_size};
        runs += (unsigned)(of_planes * each);
    };
    if (planes * sp.items >= 4 * warps && density < 128) {
        const int64_t mixed = std::min(planes, ((p.D == 64 ? 16 : 8) * warps + sp.items - 1) / sp.items);
        // (in each n runs of `length`, 2 * n of half and items / 4 - n of twice that: items / 2 - 1 at most)
        const int64_t n = std::min((warps + mixed - 1) / mixed, (int64_t)(sp.items - 4) / 8);
        add(0, planes - mixed, 0, sp.items / 4, 2);
        add(planes - mixed, mixed, 4 * n, sp.items / 4 - n, 2);
        add(planes - mixed, mixed, 2 * n, n, 1);
        add(planes - mixed, mixed, 0, 2 * n, 0);
    } else {
        add(0, planes, 0, sp.items / 2, 1);
        while (kind < kRunKinds) add(planes, 0, 0, 0, 0);
    }
    sp.all_runs = runs;
}

int64_t plan_sorted(SortPlan &sp, const Params &p, bool softmax, int64_t samples, void *workspace) {
    const int64_t P = (int64_t)p.L * p.K;
    const int64_t planes = samples * p.G;
    sp.plane_points = p.Q * P;
    sp.chunk_queries = (int)(kSortThreads / P * kSortPoints);
    sp.chunks = (int)((p.Q + sp.chunk_queries - 1) / sp.chunk_queries);
    // (by level: stretches that leave four CTAs per SM, but no counts of few points to merge)
    sp.count_by_level = p.ref == nullptr && p.K <= count_threads(true);
    sp.count_queries = sp.chunk_queries;
    if (sp.count_by_level) {
        const int64_t share = std::min<int64_t>(std::max<int64_t>(planes * sp.plane_points / (148 * 4), 2048), 16384);
        sp.count_queries = (int)round_up(share / p.K, count_threads(true) / p.K * kSortBatch);
    }
    sp.count_stretches = (int)((p.Q + sp.count_queries - 1) / sp.count_queries);
    sp.count_ctas = sp.count_stretches * (sp.count_by_level ? p.L : 1);
    // a strip is at most 7 pixels short of its width and a level one row high: H + 1 <= 2 H and
    // ceil((W + 1) / 7) <= W leave at most two cells per pixel
    sp.prepare_ctas = (int)std::min<int64_t>(148 * 2, 1 + samples * (p.S + p.Q) * p.G * p.D / (8 * kSortThreads * 4));
    sp.cell_bound = (int)(2 * p.S + 2 * p.L);
    // a pyramid of ordinary proportions has a cell per five to six pixels (whole eights: the scatter
    // takes cells by eights, in 16-byte accesses to arrays that follow one another)
    sp.shared_cells = (int)std::min<int64_t>(kSharedCells, round_up(std::min<int64_t>(sp.cell_bound, p.S / 5 + 256), 8));
    // (backward, us, all levels -> by level: 5 376 positions, 8 samples 221 -> 224, 8 400, 4 samples 167 -> 170,
    // 14 196 270 -> 264; offsets: 14 196 323 -> 335, 21 504 497 -> 499, 27 750, 2 samples, where the other
    // kernel has one CTA per SM only, 584 -> 519, 42 500, one sample 369 -> 332)
    sp.scatter_by_level = p.K <= kLevelThreads && p.S >= (p.ref != nullptr ? 26000 : 12000);
    sp.level_queries = (int)(kLevelThreads / p.K * kLevelPoints);
    sp.level_stretches = sp.scatter_by_level ? (int)((p.Q + sp.level_queries - 1) / sp.level_queries) : 0;
    sp.level_turns = (unsigned)(planes * p.L * sp.level_stretches);
    // A level has a cell per five to seven positions; the finest of several that halve has four fifths of the
    // positions, the one of two may have nine tenths.  Room for more than the former takes L1 from the loads
    // (S / 5 in both kernels: headline shape 398 -> 401, four levels of 42 500 positions 271 -> 307), but for
    // kCountRoom in the counting kernel: eight CTAs take 132 KB then, a step of what an SM can set aside, as
    // they do at the headline shape (128x128 + 32x32 of 16 points a position 220 -> 211, 150x150 + 38x38
    // 342 -> 332).  The scatter is no faster for it: a level beyond its room leaves unordered, 128x128 + 32x32
    // at 259 us, in order 260; 140x140 + 35x35 352, 357; 192x192 + 48x48 301, 308
    auto room = [&](int64_t least) {
        const int64_t cells = p.L > 1 ? std::max(p.S / 8 + 256, least) : p.S / 5 + 256;
        return (int)std::min<int64_t>(kLevelCells, round_up(std::min<int64_t>(sp.cell_bound, cells), 8));
    };
    sp.level_cells = room(0);
    sp.count_cells = sp.count_by_level ? room(std::min<int64_t>(kCountRoom, p.S / 5 + 256)) : sp.shared_cells;
    sp.cell_stride = round_up(sp.cell_bound + 1, 32);
    plan_runs(sp, p, planes);
    char *at = static_cast<char *>(workspace);
    int64_t used = 0;
    auto take = [&](int64_t bytes) {
        char *r = at + used;
        used += round_up(bytes, 256);
        return r;
    };
    sp.header = reinterpret_cast<unsigned *>(take(kScratchHeaderBytes));
    sp.tickets = reinterpret_cast<unsigned *>(take(planes * 4));
    sp.counts = reinterpret_cast<unsigned *>(take(planes * sp.cell_stride * 4));
    sp.cleared_bytes = (size_t)used;
    sp.offsets = reinterpret_cast<unsigned *>(take(planes * sp.cell_stride * 4));
    sp.item_cell = reinterpret_cast<int *>(take(planes * sp.items * 4));
    sp.records = reinterpret_cast<uint4 *>(take(planes * sp.plane_points * 16));
    sp.grad_prob = reinterpret_cast<float *>(take(planes * sp.plane_points * 4));
    sp.stats = softmax ? reinterpret_cast<float2 *>(take(planes * p.Q * 8)) : nullptr;
    return used;
}

cudaError_t launch_backward_sorted(const Params &p, const SortPlan &sp, int dtype, bool softmax,
                                   cudaStream_t stream) {
    if (dtype == 1)
        return softmax ? launch_sorted_head<__half, true>(p, sp, stream)
                       : launch_sorted_head<__half, false>(p, sp, stream);
    return softmax ? launch_sorted_head<__nv_bfloat16, true>(p, sp, stream)
                   : launch_sorted_head<__nv_bfloat16, false>(p, sp, stream);
}

}  // namespace msda_b200
