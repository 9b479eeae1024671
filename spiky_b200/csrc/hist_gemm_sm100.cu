// Contractions of the histogram path on the sm_100a tensor cores: fp32 results from fp16 operands.
//
// Row counts are small integers (below 2049), exact in fp16.  An fp32 operand x (a table, an output gradient) is scaled
// by a power of two that brings the largest element of its row - or of its column within 1024 rows - to [2^14, 2^15), and kept as
// two fp16 values: hi = x * s rounded, lo = (x * s - hi) * 2^12 rounded.  x * s = hi + lo * 2^-12 to 2^-23 of x, as with the two
// 11-bit halves of a TF32 split, for elements down to 2^-14 (scaled; 2^-28 to 2^-29 of the largest).  The scale belongs to a free index
// of the contraction (and to a slice of the contraction, see below), so it comes out of the sum as a factor.
// Smaller elements have no place in these halves.  They are rare (less than one of 10^8 normally distributed elements, and what exact sums
// leave of each other), so that what is ordinarily done for them is to look whether there are any.  Where there are, they are
// zero in the halves and have halves of their own, 2^28 larger (down to 2^-56 of the largest); a tile with such elements takes another
// turn of MMAs with these for each slice that has some, up to three where both operands do, which are added to the result once all
// tiles are written.  Elements below that ("deep") are zero in both, and are multiplied in
// fp32: add_deep_rows, add_single_products.
// The products hi.hi go into one accumulator in tensor memory, hi.lo and lo.hi into another (their sum counts 2^-12 times),
// lo.lo (below 2^-22) is dropped; kind::f16 runs at twice the rate of kind::tf32.
//
// One kernel, a pair of SMs per 256 x 256 tile of the result (tcgen05 cta_group::2), persistent, warp-specialised:
//   warps 0 - 7  read the accumulators back into registers, add the two parts, undo the scales, and send the tile out through
//                shared memory by TMA (store, or add in L2 where the result accumulates)
//   warp 8       TMA: operand tiles of 64 contraction elements into a ring of shared-memory stages; each SM of the pair loads
//                its own 128 rows of A and its own 128 columns of B (plain copies: nobody to multicast to)
//   warp 9       one thread of the pair's first SM issues the MMAs for both
// The tile is this wide because shared memory is what limits the rate: per MMA cycle an SM then reads 64 bytes of operands and
// receives 42 to 47; 256 x 128 tiles with two sets of accumulators took 96 and 64, of the 128 there are, and were slower although
// their epilogues ran under the next tile's MMAs.  Here both accumulators (2 x 256 columns) are all of tensor memory: the MMAs
// wait while they are read into registers, not for the rest of the epilogue.
// The tensor core truncates its fp32 accumulator after each step, an error that grows with the length of the chain: after
// kSliceBlocks * 64 elements the epilogue takes the sum over into registers (rounded fp32 additions, where a column has a scale per
// slice with its factor) and the MMAs start afresh.
// Few tiles and a long contraction (the forward pass of few tokens): work items are (part of the contraction, tile), each
// part's result goes to scratch and a second kernel adds the parts in order.
//
// Bound by the tensor cores; measured with their operand copies (before: TF32 halves as operands of CUTLASS GEMMs, the two halves of
// the result added by a kernel of their own): see the table at launch_contraction.
#include "hist_gemm_sm100.cuh"

#include "mbarrier.cuh"
#include "tensor_map.cuh"

namespace lutb {

__device__ int g_contract_wait_errors = 0;

int contract_wait_errors(int *count_out) {
    LUTB_CUDA(cudaMemcpyFromSymbol(count_out, g_contract_wait_errors, sizeof(int)));
    return LUTB_OK;
}

namespace {

constexpr int kTileM = 256, kTileN = 256, kBlockK = 64;   // of a pair of SMs
constexpr int kSliceBlocks = 16;
constexpr int kOperandBytes = 128 * kBlockK * 2;           // 128 rows of A, 128 columns of B
constexpr int kEpilogueWarps = 8, kEpilogueBytes = kEpilogueWarps * 4096;   // per epilogue warp two pieces of 32 x 16 floats
constexpr int kWarpCols = kTileN / 2;                      // columns of an epilogue warp (four warps cover 128 rows)
constexpr float kLoScale = 1.0f / 4096.0f;

template <int A_PARTS>
struct Ring {
    static constexpr int kStageBytes = (A_PARTS + 2) * kOperandBytes;
    static constexpr int kStages = A_PARTS == 1 ? 4 : 3;
    static constexpr size_t kSmem = (size_t)kStages * kStageBytes + kEpilogueBytes + 512 + 1024;
};

struct ContractArgs {
    int M, N, kblocks;            // result and contraction extents; blocks of kBlockK
    int m_tiles, n_tiles, splits, kb_per_split;
    int m_fast;                   // tiles of neighbouring work items differ in m (else in n)
    int m_padded;                 // rows of one part's result in scratch (splits > 1)
    int accumulate;               // add to what is there
    // bits of the largest magnitude of each row of A (or null) and of each column of the result: [N], or, A exact, [slice][N]
    const uint32_t *row_bits, *col_bits;
    // where there are second halves (where there are none their place holds anything).  A exact: b_second, a byte for every 16 columns of the
    // result, [slice][16 * n_tiles], a bit for each kCopyRows rows of the slice.  Else a byte for every row of A and of B (column of the
    // result), up to whole tiles: kHasSecond, and besides kHasDeep where there are deep elements, kHasMany where there are more than kFew
    const uint8_t *a_second, *b_second;
    float alpha;                  // of the result; of what second halves and deep elements add to c, the result itself (not a part of it)
    float second_alpha;
    int64_t a_flags, b_flags;     // bytes of a_second and b_second, multiples of 16
    float *c;
    const float *a, *b;           // two-sided: the operands themselves, [M x depth] and [N x depth]
    int depth;
};

// Exponent of the scale of a row whose largest magnitude has these bits: the largest becomes 2^14 to 2^15 (as far as the
// scale itself is a normal number).
constexpr uint32_t kInfinity = 0x7f800000u;
constexpr uint32_t kHasSecond = 1u, kHasDeep = 2u, kHasMany = 4u;
constexpr int kFew = 4;
__device__ __forceinline__ int scale_exponent(uint32_t bits) { return min(141 - (int)(bits >> 23), 126); }
__device__ __forceinline__ float scale_of(uint32_t bits) { return __uint_as_float((uint32_t)(scale_exponent(bits) + 127) << 23); }
__device__ __forceinline__ float inverse_scale(uint32_t bits) { return __uint_as_float((uint32_t)(127 - scale_exponent(bits)) << 23); }

// ------------------------------------------------------------------------------------------------ operand copies
struct Halves { uint2 hi, lo; };   // of four neighbouring elements
__device__ __forceinline__ Halves split4(float4 v, float sx, float sy, float sz, float sw) {
    v.x *= sx; v.y *= sy; v.z *= sz; v.w *= sw;
    const __half2 h0 = __floats2half2_rn(v.x, v.y), h1 = __floats2half2_rn(v.z, v.w);
    const float2 f0 = __half22float2(h0), f1 = __half22float2(h1);
    const __half2 l0 = __floats2half2_rn((v.x - f0.x) * 4096.f, (v.y - f0.y) * 4096.f);
    const __half2 l1 = __floats2half2_rn((v.z - f1.x) * 4096.f, (v.w - f1.y) * 4096.f);
    Halves r;
    r.hi = make_uint2(*reinterpret_cast<const uint32_t *>(&h0), *reinterpret_cast<const uint32_t *>(&h1));
    r.lo = make_uint2(*reinterpret_cast<const uint32_t *>(&l0), *reinterpret_cast<const uint32_t *>(&l1));
    return r;
}
// Bits of the least magnitude that the first halves of a scale hold, 2^-14 over the scale, and the second ones, 2^-42.
__device__ __forceinline__ uint32_t power_bits(int e) { return e >= 1 ? (uint32_t)e << 23 : e > -23 ? 1u << (22 + e) : 0u; }   // of 2^(e - 127)
__device__ __forceinline__ uint32_t first_least(uint32_t bits) { return power_bits(113 - scale_exponent(bits)); }
__device__ __forceinline__ uint32_t second_least(uint32_t bits) { return power_bits(85 - scale_exponent(bits)); }
constexpr float kSecondScale = 268435456.f;   // 2^28
__device__ __forceinline__ uint32_t magnitude(float x) { return __float_as_uint(x) & 0x7fffffffu; }
__device__ __forceinline__ bool is_below(float x, uint32_t least) { return magnitude(x) - 1u < least - 1u && least != 0u; }   // (and not zero)
// Twice the bits of the smallest of four magnitudes less one, so that a zero is the largest of all; and the limit that goes with it.
__device__ __forceinline__ uint32_t twice_less_one(float x) { return __float_as_uint(x) * 2u - 1u; }
__device__ __forceinline__ uint32_t least4(float4 v) { return min(min(twice_less_one(v.x), twice_less_one(v.y)), min(twice_less_one(v.z), twice_less_one(v.w))); }
__device__ __forceinline__ bool some_below(uint32_t least, uint32_t limit) { return least < limit * 2u - 1u; }
__device__ __forceinline__ float kept(float x, uint32_t least) { return magnitude(x) < least ? 0.f : x; }
// what the second halves hold of x, to be scaled as it is
__device__ __forceinline__ float kept_second(float x, uint32_t first, uint32_t second) { return magnitude(x) < first && magnitude(x) >= second ? x : 0.f; }
__device__ __forceinline__ float magnitude4(float4 v) { return fmaxf(fmaxf(fabsf(v.x), fabsf(v.y)), fmaxf(fabsf(v.z), fabsf(v.w))); }   // (without what is not a number)

// Where the halves of a matrix go: rows of `pitch`.  second: see ContractArgs.
struct Copy {
    __half *hi, *lo, *hi2, *lo2;
    uint32_t *bits;
    uint8_t *second;
    int pitch;
};

// One row with elements that the first halves do not hold: its first halves again, and its second ones.
// Returns its byte of flags.
__device__ __noinline__ uint32_t split_row_twice(const float4 *src, int c4, uint32_t bits, const Copy &to, int64_t r) {
    const uint32_t first = first_least(bits), second = second_least(bits);
    const float s = scale_of(bits);
    bool deep = false;
    int small = 0;
    for (int c = threadIdx.x & 31; c < c4; c += 32) {
        const float4 x = __ldg(src + c);
        deep = deep || is_below(x.x, second) || is_below(x.y, second) || is_below(x.z, second) || is_below(x.w, second);
        small += is_below(x.x, first) + is_below(x.y, first) + is_below(x.z, first) + is_below(x.w, first);
        const Halves p = split4(make_float4(kept(x.x, first), kept(x.y, first), kept(x.z, first), kept(x.w, first)), s, s, s, s);
        const float4 y = make_float4(kept_second(x.x, first, second) * s, kept_second(x.y, first, second) * s, kept_second(x.z, first, second) * s, kept_second(x.w, first, second) * s);
        const Halves q = split4(y, kSecondScale, kSecondScale, kSecondScale, kSecondScale);
        reinterpret_cast<uint2 *>(to.hi + r * to.pitch)[c] = p.hi;
        reinterpret_cast<uint2 *>(to.lo + r * to.pitch)[c] = p.lo;
        reinterpret_cast<uint2 *>(to.hi2 + r * to.pitch)[c] = q.hi;
        reinterpret_cast<uint2 *>(to.lo2 + r * to.pitch)[c] = q.lo;
    }
    return kHasSecond | (__any_sync(0xffffffffu, deep) ? kHasDeep : 0u) | (__reduce_add_sync(0xffffffffu, small) > kFew ? kHasMany : 0u);
}

// Scaled by row: a warp per row, which stays in registers up to 1024 columns (read twice beyond).  HBM bound.  Rows up to a whole tile say
// that they have no second halves.
__global__ void __launch_bounds__(256) split_rows_kernel(const float *__restrict__ x, int64_t rows, int cols, const __grid_constant__ Copy to) {
    constexpr int KEEP = 8;
    const int lane = threadIdx.x & 31, c4 = cols >> 2;
    int64_t r = (int64_t)blockIdx.x * 8 + (threadIdx.x >> 5);
    for (; r < rows; r += (int64_t)gridDim.x * 8) {
        const float4 *src = reinterpret_cast<const float4 *>(x + r * cols);
        float4 v[KEEP];
        float most = 0.f;
        uint32_t least = ~0u;
#pragma unroll
        for (int n = 0; n < KEEP; n++) {
            const int c = n * 32 + lane;
            v[n] = c < c4 ? __ldg(src + c) : make_float4(0.f, 0.f, 0.f, 0.f);
        }
#pragma unroll
        for (int n = 0; n < KEEP; n++)
            if (n * 32 < c4) { most = fmaxf(most, magnitude4(v[n])); least = min(least, least4(v[n])); }
        for (int c = KEEP * 32 + lane; c < c4; c += 32) {
            const float4 w = __ldg(src + c);
            most = fmaxf(most, magnitude4(w));
            least = min(least, least4(w));
        }
        const uint32_t m = __reduce_max_sync(0xffffffffu, __float_as_uint(most));
        const float s = scale_of(m);
        uint2 *h = reinterpret_cast<uint2 *>(to.hi + r * to.pitch), *l = reinterpret_cast<uint2 *>(to.lo + r * to.pitch);
#pragma unroll
        for (int n = 0; n < KEEP; n++) {
            const int c = n * 32 + lane;
            if (c < c4) {
                const Halves q = split4(v[n], s, s, s, s);
                h[c] = q.hi;
                l[c] = q.lo;
            }
        }
        for (int c = KEEP * 32 + lane; c < c4; c += 32) {
            const Halves q = split4(__ldg(src + c), s, s, s, s);
            h[c] = q.hi;
            l[c] = q.lo;
        }
        uint32_t has = 0u;
        // (what is not finite makes its whole row of the result so)
        if (__any_sync(0xffffffffu, m < kInfinity && some_below(least, first_least(m))))
            has = split_row_twice(src, c4, m, to, r);
        if (lane == 0) {
            to.bits[r] = m;
            to.second[r] = (uint8_t)has;
        }
    }
    for (; r < (rows + kTileM - 1) / kTileM * kTileM; r += (int64_t)gridDim.x * 8)
        if (lane == 0) to.second[r] = 0u;
}

// Scaled by column and slice of kSliceRows rows: a block takes 16 columns of a slice, which stay in its registers between the
// maximum and the copy, so that the matrix is read once (a pass for the maxima of whole columns took 41 of the 123 us for 65536 x
// 1024, and 7 + 5 us for 16384 x 256).  bits: [slice][cols].
constexpr int kSliceRows = kSliceBlocks * kBlockK, kCopyRows = 128, kCopyCols = 16, kCopyThreads = kCopyRows * kCopyCols / 4;

// What deep elements of a copy by column are added to: C [M x cols] += alpha * A . (deep elements of x), A(m, k) = H[m * kt + k], or
// H[k * kt + m] where A is H transposed.
struct DeepTarget {
    const __half *H;
    float *C;
    int64_t kt;
    int M;
    float alpha;
    bool transposed;
};

// The products of the deep elements of kCopyCols columns and a slice of x: `marks` has a bit for each of the slice's rows with such an
// element.  Half a warp's lanes have a column each and eight rows of the result at a time.  One block does this for all rows: where it has to, it
// takes tens of microseconds for a few rows of x and milliseconds for a slice of them.
__device__ __noinline__ void add_deep_rows(const float *__restrict__ x, int cols, int64_t r0, int col0, const uint32_t *column_bits, const uint32_t *marks,
                                           const DeepTarget &t) {
    constexpr int R = 8;
    const int lane = threadIdx.x % kCopyCols, n = col0 + lane;
    const uint32_t second = second_least(column_bits[lane]);
    const bool mine = n < cols && column_bits[lane] < kInfinity;
    for (int m0 = (int)(threadIdx.x / kCopyCols) * R; m0 < t.M; m0 += (int)(blockDim.x / kCopyCols) * R) {
        float acc[R] = {};
        for (int w = 0; w < kSliceRows / 32; w++) {
            for (uint32_t left = marks[w]; left != 0u; left &= left - 1u) {
                const int64_t k = r0 + w * 32 + __ffs(left) - 1;
                float v = mine ? __ldg(x + k * cols + n) : 0.f;
                if (!is_below(v, second)) v = 0.f;
#pragma unroll
                for (int i = 0; i < R; i++) {
                    const int64_t at = t.transposed ? k * t.kt + m0 + i : (m0 + i) * t.kt + k;
                    if (m0 + i < t.M) acc[i] = fmaf(__half2float(t.H[at]), v, acc[i]);
                }
            }
        }
#pragma unroll
        for (int i = 0; i < R; i++)
            if (acc[i] != 0.f) atomicAdd(t.C + (int64_t)(m0 + i) * cols + n, t.alpha * acc[i]);
    }
}

// A thread's columns of a slice, where they have elements that the first halves do not hold: takes these out of the first halves.  Returns
// a bit for each row k * kCopyRows + ty of the slice with such elements, and from 16 on with deep ones.
__device__ __noinline__ uint32_t take_small_out(const float *__restrict__ x, int64_t rows, int cols, int64_t r0, int c4, uint4 b, const Copy &to) {
    constexpr int ROWS = kSliceRows / kCopyRows;
    const uint32_t bits[4] = {b.x, b.y, b.z, b.w};
    uint32_t found = 0u;
    float4 v[ROWS];
#pragma unroll
    for (int k = 0; k < ROWS; k++) {
        const int64_t r = r0 + k * kCopyRows + threadIdx.x / (kCopyCols / 4);
        v[k] = r < rows ? __ldg(reinterpret_cast<const float4 *>(x + r * cols) + c4) : make_float4(0.f, 0.f, 0.f, 0.f);
    }
#pragma unroll
    for (int k = 0; k < ROWS; k++) {
        const int64_t r = r0 + k * kCopyRows + threadIdx.x / (kCopyCols / 4);
        const float q[4] = {v[k].x, v[k].y, v[k].z, v[k].w};
        float p[4];
        bool small = false, deep = false;
#pragma unroll
        for (int e = 0; e < 4; e++) {
            small = small || (bits[e] < kInfinity && is_below(q[e], first_least(bits[e])));
            deep = deep || (bits[e] < kInfinity && is_below(q[e], second_least(bits[e])));
            p[e] = kept(q[e], first_least(bits[e])) * scale_of(bits[e]);
        }
        if (!small) continue;
        found |= 1u << k | (deep ? 1u << (16 + k) : 0u);
        const Halves h = split4(make_float4(p[0], p[1], p[2], p[3]), 1.f, 1.f, 1.f, 1.f);
        reinterpret_cast<uint2 *>(to.hi + r * to.pitch)[c4] = h.hi;
        reinterpret_cast<uint2 *>(to.lo + r * to.pitch)[c4] = h.lo;
    }
    return found;
}

// The second halves: of the groups of kCopyRows rows that have some (a bit for each), and zeros in the others, which the tile's other columns
// may have some in.
__device__ __noinline__ void write_second(const float *__restrict__ x, int64_t rows, int cols, int64_t r0, int c4, uint4 b, uint32_t groups, const Copy &to) {
    const uint32_t bits[4] = {b.x, b.y, b.z, b.w};
#pragma unroll 1
    for (int k = 0; k < kSliceRows / kCopyRows; k++) {
        const int64_t r = r0 + k * kCopyRows + threadIdx.x / (kCopyCols / 4);
        if (r >= rows) break;
        Halves h = {make_uint2(0u, 0u), make_uint2(0u, 0u)};
        if ((groups >> k) & 1u) {
            const float4 v = __ldg(reinterpret_cast<const float4 *>(x + r * cols) + c4);
            const float q[4] = {v.x, v.y, v.z, v.w};
            float p[4];
#pragma unroll
            for (int e = 0; e < 4; e++) p[e] = kept_second(q[e], first_least(bits[e]), second_least(bits[e])) * scale_of(bits[e]);
            h = split4(make_float4(p[0], p[1], p[2], p[3]), kSecondScale, kSecondScale, kSecondScale, kSecondScale);
        }
        reinterpret_cast<uint2 *>(to.hi2 + r * to.pitch)[c4] = h.hi;
        reinterpret_cast<uint2 *>(to.lo2 + r * to.pitch)[c4] = h.lo;
    }
}

// (parameters in place: what is handed on by reference would be copied to local memory by every thread, 113 -> 130 us for 65536 x 1024)
__global__ void __launch_bounds__(kCopyThreads, 2) split_columns_kernel(const float *__restrict__ x, int64_t rows, int cols, const __grid_constant__ Copy to,
                                                                       const __grid_constant__ DeepTarget target) {
    constexpr int KEEP = kSliceRows / kCopyRows, QUADS = kCopyCols / 4, WARPS = kCopyThreads / 32;
    __shared__ uint32_t part[WARPS][kCopyCols], marks[kSliceRows / 32];
    const int tx = threadIdx.x % QUADS, ty = threadIdx.x / QUADS, c4 = blockIdx.y * QUADS + tx;
    uint8_t *second = to.second + (int64_t)blockIdx.x * gridDim.y + blockIdx.y;
    if ((int)blockIdx.y * kCopyCols >= cols) {   // (columns up to a whole tile)
        if (threadIdx.x == 0) *second = 0u;
        return;
    }
    const bool live = c4 < (cols >> 2);
    const int64_t r0 = (int64_t)blockIdx.x * kSliceRows;
    float4 v[KEEP];
    float4 most = make_float4(0.f, 0.f, 0.f, 0.f);
    uint4 least = make_uint4(~0u, ~0u, ~0u, ~0u);
#pragma unroll
    for (int k = 0; k < KEEP; k++) {
        const int64_t r = r0 + k * kCopyRows + ty;
        v[k] = live && r < rows ? __ldg(reinterpret_cast<const float4 *>(x + r * cols) + c4) : make_float4(0.f, 0.f, 0.f, 0.f);
    }
#pragma unroll
    for (int k = 0; k < KEEP; k++) {
        most.x = fmaxf(most.x, fabsf(v[k].x)); most.y = fmaxf(most.y, fabsf(v[k].y));
        most.z = fmaxf(most.z, fabsf(v[k].z)); most.w = fmaxf(most.w, fabsf(v[k].w));
        least.x = min(least.x, twice_less_one(v[k].x)); least.y = min(least.y, twice_less_one(v[k].y));
        least.z = min(least.z, twice_less_one(v[k].z)); least.w = min(least.w, twice_less_one(v[k].w));
    }
    uint4 m = make_uint4(__float_as_uint(most.x), __float_as_uint(most.y), __float_as_uint(most.z), __float_as_uint(most.w));
#pragma unroll
    for (int o = QUADS; o < 32; o <<= 1) {   // a warp has 32 / QUADS rows of the column quadruples
        m.x = max(m.x, __shfl_xor_sync(0xffffffffu, m.x, o));
        m.y = max(m.y, __shfl_xor_sync(0xffffffffu, m.y, o));
        m.z = max(m.z, __shfl_xor_sync(0xffffffffu, m.z, o));
        m.w = max(m.w, __shfl_xor_sync(0xffffffffu, m.w, o));
    }
    if ((threadIdx.x & 31) < QUADS) *reinterpret_cast<uint4 *>(&part[threadIdx.x >> 5][4 * tx]) = m;
    __syncthreads();
    if (threadIdx.x < kCopyCols) {
        uint32_t all = 0u;
#pragma unroll
        for (int k = 0; k < WARPS; k++) all = max(all, part[k][threadIdx.x]);
        part[0][threadIdx.x] = all;
        const int n = blockIdx.y * kCopyCols + threadIdx.x;
        if (n < cols) to.bits[(int64_t)blockIdx.x * cols + n] = all;
    }
    __syncthreads();
    const uint4 b = *reinterpret_cast<const uint4 *>(&part[0][4 * tx]);
    if (live) {
        const float sx = scale_of(b.x), sy = scale_of(b.y), sz = scale_of(b.z), sw = scale_of(b.w);
#pragma unroll
        for (int k = 0; k < KEEP; k++) {
            const int64_t r = r0 + k * kCopyRows + ty;
            if (r >= rows) break;
            const Halves q = split4(v[k], sx, sy, sz, sw);
            *(reinterpret_cast<uint2 *>(to.hi + r * to.pitch) + c4) = q.hi;
            *(reinterpret_cast<uint2 *>(to.lo + r * to.pitch) + c4) = q.lo;
        }
    }
    // (what is not finite makes its whole column of the result so)
    const bool small = (b.x < kInfinity && some_below(least.x, first_least(b.x))) || (b.y < kInfinity && some_below(least.y, first_least(b.y))) ||
                       (b.z < kInfinity && some_below(least.z, first_least(b.z))) || (b.w < kInfinity && some_below(least.w, first_least(b.w)));
    if (__syncthreads_or(small) == 0) {
        if (threadIdx.x == 0) *second = 0u;
        return;
    }
    __shared__ uint32_t groups;
    if (threadIdx.x == 0) groups = 0u;
    if (threadIdx.x < kSliceRows / 32) marks[threadIdx.x] = 0u;
    __syncthreads();
    const uint32_t found = small ? take_small_out(x, rows, cols, r0, c4, b, to) : 0u;
    if ((found & 0xffffu) != 0u) atomicOr(&groups, found & 0xffffu);
#pragma unroll
    for (int k = 0; k < KEEP; k++) {
        const int row = k * kCopyRows + ty;
        if ((found >> (16 + k)) & 1u) atomicOr(&marks[row >> 5], 1u << (row & 31));
    }
    const bool deep = __syncthreads_or((found >> 16) != 0u) != 0;
    if (live) write_second(x, rows, cols, r0, c4, b, groups, to);
    if (threadIdx.x == 0) *second = (uint8_t)groups;
    if (!deep) return;
    add_deep_rows(x, cols, r0, blockIdx.y * kCopyCols, part[0], marks, target);
}

// C += alpha * sum of the parts, in order and in double (up to 32 parts: fp32 additions were most of the result's error).
constexpr int kAddThreads = 64;
template <int AHEAD>   // parts whose loads are in flight (they are one latency each otherwise)
__global__ void __launch_bounds__(kAddThreads) add_parts_kernel(const float *__restrict__ P, float *__restrict__ C, int64_t M, int N, int parts,
                                                        int64_t part_stride, float alpha) {
    const int64_t n4 = M * (N / 4);
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n4; i += (int64_t)gridDim.x * blockDim.x) {
        double s[4] = {0., 0., 0., 0.};
        for (int k0 = 0; k0 < parts; k0 += AHEAD) {
            float4 t[AHEAD];
#pragma unroll
            for (int k = 0; k < AHEAD; k++)
                t[k] = k0 + k < parts ? __ldcs(reinterpret_cast<const float4 *>(P + (k0 + k) * part_stride) + i) : make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
            for (int k = 0; k < AHEAD; k++) { s[0] += t[k].x; s[1] += t[k].y; s[2] += t[k].z; s[3] += t[k].w; }
        }
        float4 *dst = reinterpret_cast<float4 *>(C) + i;
        float4 o = *dst;
        o.x += alpha * (float)s[0]; o.y += alpha * (float)s[1]; o.z += alpha * (float)s[2]; o.w += alpha * (float)s[3];
        *dst = o;
    }
}

// ------------------------------------------------------------------------------------------------ PTX
__device__ __forceinline__ uint32_t cluster_rank() {
    uint32_t r;
    asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
    return r;
}
__device__ __forceinline__ void cluster_sync() {
    asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
// the address of the pair's first SM's copy of a shared variable
__device__ __forceinline__ uint32_t in_first(uint32_t addr) {
    uint32_t r;
    asm volatile("mapa.shared::cluster.u32 %0, %1, 0;" : "=r"(r) : "r"(addr));
    return r;
}
__device__ __forceinline__ void arrive_in_cluster(uint32_t bar) {
    asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(bar) : "memory");
}
__device__ __forceinline__ bool try_wait_cluster(uint32_t bar, uint32_t parity) {
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok)
        : "r"(bar), "r"(parity)
        : "memory");
    return ok != 0;
}
__device__ __forceinline__ bool wait_cluster(uint32_t bar, uint32_t parity) {
    if (try_wait_cluster(bar, parity)) return true;
    const long long t0 = clock64();
    while (!try_wait_cluster(bar, parity)) {
        if (clock64() - t0 > kWaitLimitCycles) return false;
    }
    return true;
}
__device__ __forceinline__ void tma_load(uint32_t dst, const CUtensorMap *map, int x, int y, uint32_t bar) {
    asm volatile(
        "cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];" ::"r"(dst),
        "l"(map), "r"(bar), "r"(x), "r"(y)
        : "memory");
}
__device__ __forceinline__ void tma_store(const CUtensorMap *map, uint32_t src, int x, int y) {
    asm volatile("cp.async.bulk.tensor.2d.global.shared::cta.tile.bulk_group [%0, {%2, %3}], [%1];" ::"l"(map), "r"(src), "r"(x), "r"(y)
                 : "memory");
}
__device__ __forceinline__ void tma_add(const CUtensorMap *map, uint32_t src, int x, int y) {
    asm volatile("cp.reduce.async.bulk.tensor.2d.global.shared::cta.add.tile.bulk_group [%0, {%2, %3}], [%1];" ::"l"(map), "r"(src),
                 "r"(x), "r"(y)
                 : "memory");
}
__device__ __forceinline__ void mma_f16_pair(uint32_t d, uint64_t a, uint64_t b, uint32_t idesc, uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p;\n\t}" ::"r"(d), "l"(a), "l"(b), "r"(idesc), "r"(accumulate)
        : "memory");
}
// arrives on the barrier at this offset in both SMs once every MMA issued so far has finished
__device__ __forceinline__ void commit_pair(uint32_t bar) {
    asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;" ::"r"(bar),
                 "h"((uint16_t)3)
                 : "memory");
}
__device__ __forceinline__ void fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tmem_load16(uint32_t (&v)[16], uint32_t addr) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
        : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]), "=r"(v[8]), "=r"(v[9]),
          "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15])
        : "r"(addr));
}
__device__ __forceinline__ void tmem_load_wait() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }
// (the loaded registers pass through: nothing that reads them can move above the wait)
__device__ __forceinline__ void loaded(uint32_t (&v)[16]) {
#pragma unroll
    for (int n = 0; n < 16; n++) asm volatile("" : "+r"(v[n]));
}

// Shared-memory operand descriptors, 128-byte swizzle (8 rows of 128 bytes are a unit of 1024).  Contraction index contiguous:
// units follow each other along the free index.  Free index contiguous: units of 8 contraction steps follow each other, and the
// next 64 free elements start 64 steps on.
template <bool FREE_CONTIGUOUS>
__device__ __forceinline__ uint64_t operand_desc(uint32_t addr) {
    const uint64_t leading = FREE_CONTIGUOUS ? (64 * 128) >> 4 : 1, stride = 1024 >> 4;
    return (uint64_t)((addr & 0x3ffffu) >> 4) | leading << 16 | stride << 32 | 1ull << 46 | 2ull << 61;
}
// bytes from one 16-element contraction step to the next
template <bool FREE_CONTIGUOUS>
constexpr uint32_t kStepBytes = FREE_CONTIGUOUS ? 16 * 128 : 32;

struct Item { int m_tile, n_tile, split, kb0, kb1; };
__device__ __forceinline__ int slice_end(const Item &it, int kb) { return min(it.kb1, (kb / kSliceBlocks + 1) * kSliceBlocks); }
__device__ __forceinline__ Item item_of(const ContractArgs &g, int i) {
    Item it;
    const int tiles = g.m_tiles * g.n_tiles;
    it.split = i / tiles;
    const int t = i - it.split * tiles;
    if (g.m_fast) { it.n_tile = t / g.m_tiles; it.m_tile = t - it.n_tile * g.m_tiles; }
    else { it.m_tile = t / g.n_tiles; it.n_tile = t - it.m_tile * g.n_tiles; }
    it.kb0 = it.split * g.kb_per_split;
    it.kb1 = min(g.kblocks, it.kb0 + g.kb_per_split);
    return it;
}

// Tiles of rows and of columns with second halves, a bit for each by its number modulo the bits (two-sided contractions).
constexpr int kMarkWords = 32;
__device__ __forceinline__ bool is_marked(const volatile uint32_t *marked, int tile) { return (marked[(tile >> 5) % kMarkWords] >> (tile & 31)) & 1u; }

// Turns of MMAs that a slice of a tile takes, a bit for each: 0 the first halves of both, 1 A's second ones with B's first, 2 B's
// second ones with A's first, 3 the second ones of both (A exact: 0 and 2).  All of the pair's warps read the same.
__device__ __forceinline__ uint32_t turns_from(bool in_a, bool in_b) { return 1u | (in_a ? 2u : 0u) | (in_b ? 4u : 0u) | (in_a && in_b ? 8u : 0u); }
template <int N>
__device__ __forceinline__ uint32_t any_of(const uint8_t *bytes) {   // of N bytes, on 16
    uint32_t any = 0u;
#pragma unroll
    for (int n = 0; n < N / 16; n++) {
        const uint4 v = __ldg(reinterpret_cast<const uint4 *>(bytes) + n);
        any |= v.x | v.y | v.z | v.w;
    }
    return any;
}
__device__ __forceinline__ const uint8_t *second_columns(const ContractArgs &g, const Item &it, int slice) {
    return g.b_second + ((int64_t)slice * g.n_tiles + it.n_tile) * (kTileN / kCopyCols);
}
// What a two-sided tile does for the small elements of A's rows and of B's.  Few of them (a row or two with no more than kFew) are multiplied in
// fp32 as deep ones are, else there are turns of MMAs: 8192 x 16384 x 256 with one small element in A 215 us against 226, 188 with none.
struct Sides {
    bool a_turn, b_turn;         // turns
    bool a_single, b_single;     // elements by themselves: all small ones where there are no turns, else deep ones
};
__device__ __forceinline__ Sides sides_of(const ContractArgs &g, const Item &it, const volatile uint32_t *marked) {
    const int lane = threadIdx.x & 31;
    Sides t{};
    if (!is_marked(marked, it.m_tile) && !is_marked(marked + kMarkWords, it.n_tile)) return t;
    const uint4 v = __ldg(reinterpret_cast<const uint4 *>(lane < 16 ? g.a_second + it.m_tile * kTileM : g.b_second + it.n_tile * kTileN) + (lane & 15));
    const uint32_t any = v.x | v.y | v.z | v.w, with = kHasSecond * 0x01010101u;
    const int mine = __popc(v.x & with) + __popc(v.y & with) + __popc(v.z & with) + __popc(v.w & with);
    const uint32_t many = __ballot_sync(0xffffffffu, (any & (kHasMany * 0x01010101u)) != 0u), deep = __ballot_sync(0xffffffffu, (any & (kHasDeep * 0x01010101u)) != 0u);
    const int in_a = __reduce_add_sync(0xffffffffu, lane < 16 ? mine : 0), in_b = __reduce_add_sync(0xffffffffu, lane < 16 ? 0 : mine);
    t.a_turn = in_a > 2 || (many & 0xffffu) != 0u;
    t.b_turn = in_b > 2 || (many >> 16) != 0u;
    t.a_single = t.a_turn ? (deep & 0xffffu) != 0u : in_a > 0;
    t.b_single = t.b_turn ? (deep >> 16) != 0u : in_b > 0;
    return t;
}

// Calls f(kb, turn, groups) for a tile's second turns, slice by slice: kb the slice's first block, groups a bit for each kCopyRows rows of
// the contraction that it takes.  False: one of them was.  All of a warp's lanes.
template <int A_PARTS, class F>
__device__ __forceinline__ bool each_second_turn(const ContractArgs &g, const Item &it, const Sides &sides, F f) {
    const int lane = threadIdx.x & 31;
    if (A_PARTS == 2) {
        const uint32_t turns = turns_from(sides.a_turn, sides.b_turn);
        if (turns == 1u) return true;
        for (int kb = it.kb0; kb < it.kb1; kb = slice_end(it, kb))
            for (int turn = 1; turn < 4; turn++)
                if (((turns >> turn) & 1u) && !f(kb, turn, ~0u)) return false;
        return true;
    }
    const int first = it.kb0 / kSliceBlocks, last = (it.kb1 + kSliceBlocks - 1) / kSliceBlocks;
    for (int s0 = first; s0 < last; s0 += 32) {
        uint32_t mine = s0 + lane < last ? any_of<kTileN / kCopyCols>(second_columns(g, it, s0 + lane)) : 0u;
        mine |= mine >> 16;
        mine = (mine | mine >> 8) & 0xffu;
        for (uint32_t left = __ballot_sync(0xffffffffu, mine != 0u); left != 0u; left &= left - 1u) {
            const int from = __ffs(left) - 1, kb = max(it.kb0, (s0 + from) * kSliceBlocks);
            // (a part of the contraction may begin or end inside a slice)
            uint32_t groups = 0u;
            for (int n = kb; n < slice_end(it, kb); n++) groups |= 1u << (n % kSliceBlocks * kBlockK / kCopyRows);
            groups &= __shfl_sync(0xffffffffu, mine, from);
            if (groups != 0u && !f(kb, 2, groups)) return false;
        }
    }
    return true;
}

// Products of a two-sided contraction that its turns leave out, for 32 rows and kWarpCols columns of the result, which the warp has written
// (and waited for): single elements of B times all of A's, then single elements of A times the others of B.
__device__ __noinline__ void add_single_products(const ContractArgs &g, const Sides &t, int row0, int n0) {
    constexpr int AHEAD = 8;   // 256 elements of a row at a time
    const int lane = threadIdx.x & 31, m = row0 + lane;
    const int64_t K = g.depth;
    const int n1 = min(g.N, n0 + kWarpCols);
    auto limit = [](uint32_t bits, bool turn) { return turn ? second_least(bits) : first_least(bits); };
    // f(c, v) for the single elements of a row
    auto each = [&](const float *row, uint32_t least, auto f) {
        for (int c0 = 0; c0 < g.depth; c0 += 32 * AHEAD) {
            float v[AHEAD];
#pragma unroll
            for (int k = 0; k < AHEAD; k++) v[k] = c0 + k * 32 + lane < g.depth ? __ldg(row + c0 + k * 32 + lane) : 0.f;
#pragma unroll
            for (int k = 0; k < AHEAD; k++)
                for (uint32_t left = __ballot_sync(0xffffffffu, is_below(v[k], least)); left != 0u; left &= left - 1u)
                    f(c0 + k * 32 + __ffs(left) - 1, __shfl_sync(0xffffffffu, v[k], __ffs(left) - 1));
        }
    };
    for (int c = 0; c < kWarpCols && t.b_single; c += 32) {   // a lane has a row
        const uint32_t flags = n0 + c + lane < n1 ? __ldg(g.b_second + n0 + c + lane) : 0u;
        for (uint32_t left = __ballot_sync(0xffffffffu, (flags & (t.b_turn ? kHasDeep : kHasSecond)) != 0u); left != 0u; left &= left - 1u) {
            const int n = n0 + c + __ffs(left) - 1;
            float acc = 0.f;
            each(g.b + n * K, limit(__ldg(g.col_bits + n), t.b_turn), [&](int k, float v) {
                if (m < g.M) acc = fmaf(__ldg(g.a + m * K + k), v, acc);
            });
            if (acc != 0.f) atomicAdd(g.c + (int64_t)m * g.N + n, g.second_alpha * acc);
        }
    }
    const uint32_t flags = t.a_single && m < g.M ? __ldg(g.a_second + m) : 0u;
    for (uint32_t left = __ballot_sync(0xffffffffu, (flags & (t.a_turn ? kHasDeep : kHasSecond)) != 0u); left != 0u; left &= left - 1u) {
        const int r = row0 + __ffs(left) - 1;   // a lane has every 32nd column
        float acc[kWarpCols / 32] = {};
        uint32_t least_b[kWarpCols / 32];
#pragma unroll
        for (int e = 0; e < kWarpCols / 32; e++) least_b[e] = n0 + e * 32 + lane < n1 ? limit(__ldg(g.col_bits + n0 + e * 32 + lane), t.b_turn) : 0u;
        each(g.a + r * K, limit(__ldg(g.row_bits + r), t.a_turn), [&](int k, float v) {
            float b[kWarpCols / 32];
#pragma unroll
            for (int e = 0; e < kWarpCols / 32; e++) b[e] = n0 + e * 32 + lane < n1 ? __ldg(g.b + (n0 + e * 32 + lane) * K + k) : 0.f;
#pragma unroll
            for (int e = 0; e < kWarpCols / 32; e++) acc[e] = fmaf(v, is_below(b[e], least_b[e]) ? 0.f : b[e], acc[e]);
        });
#pragma unroll
        for (int e = 0; e < kWarpCols / 32; e++)
            if (acc[e] != 0.f) atomicAdd(g.c + (int64_t)r * g.N + n0 + e * 32 + lane, g.second_alpha * acc[e]);
    }
}

// Adds what the accumulators hold after a second turn to the result, for this warp's 32 rows and kWarpCols columns.  Few of them have second
// halves as a rule: the others are left out, 16 columns at a time.
template <int A_PARTS>
__device__ __forceinline__ void add_second_turn(const ContractArgs &g, const Item &it, uint32_t src, int cols0, int row0, int slice, int turn) {
    const int lane = threadIdx.x & 31, row = row0 + lane, n0 = it.n_tile * kTileN + cols0;
    const bool row_second = A_PARTS == 1 || (row < g.M && __ldg(g.a_second + row) != 0);
    if ((turn & 1) && !__any_sync(0xffffffffu, row_second)) return;
    const bool row_taken = row < g.M && (row_second || !(turn & 1));
    const float row_factor = A_PARTS == 2 && row < g.M ? inverse_scale(__ldg(g.row_bits + row)) : 1.f;
    const float scale = g.second_alpha * (turn == 3 ? 1.f / kSecondScale / kSecondScale : 1.f / kSecondScale);
    // of columns c * 32 + lane: the factor, whether it is taken
    float factor[kWarpCols / 32];
    uint32_t taken[kWarpCols / 32];
#pragma unroll
    for (int c = 0; c < kWarpCols / 32; c++) {
        const int n = n0 + c * 32 + lane;
        const uint8_t *second = A_PARTS == 1 ? second_columns(g, it, slice) + (cols0 + c * 32 + lane) / kCopyCols : g.b_second + n;
        factor[c] = n < g.N ? inverse_scale(__ldg(g.col_bits + (A_PARTS == 1 ? (int64_t)slice * g.N : 0) + n)) : 1.f;
        taken[c] = __ballot_sync(0xffffffffu, n < g.N && (!(turn & 2) || __ldg(second) != 0));
    }
#pragma unroll
    for (int c = 0; c < kWarpCols / 16; c++) {
        const uint32_t cols = (taken[c / 2] >> (c % 2 * 16)) & 0xffffu;
        if (cols == 0u) continue;   // (no second halves: anything)
        uint32_t big[16], small[16];
        tmem_load16(big, src + c * 16);
        tmem_load16(small, src + kTileN + c * 16);
        tmem_load_wait();
        loaded(big);
        loaded(small);
#pragma unroll
        for (int n4 = 0; n4 < 4; n4++) {
            float o[4];
#pragma unroll
            for (int e = 0; e < 4; e++) {
                const int n = n4 * 4 + e;
                const float f = __shfl_sync(0xffffffffu, factor[c / 2], c % 2 * 16 + n);
                const float v = scale * fmaf(__uint_as_float(small[n]), kLoScale, __uint_as_float(big[n]));
                o[e] = (cols >> n) & 1u ? v * fminf(row_factor, f) * fmaxf(row_factor, f) : 0.f;
            }
            // (columns come in fours, so that those beyond the last are all of one)
            if (row_taken && (o[0] != 0.f || o[1] != 0.f || o[2] != 0.f || o[3] != 0.f))
                asm volatile("red.global.add.v4.f32 [%0], {%1, %2, %3, %4};" ::"l"(g.c + (int64_t)row * g.N + n0 + c * 16 + n4 * 4), "f"(o[0]), "f"(o[1]),
                             "f"(o[2]), "f"(o[3])
                             : "memory");
        }
    }
}

// Says whether there are second halves anywhere, and in which tiles, by the epilogue's threads while they have nothing to do.
template <int A_PARTS>
__device__ __forceinline__ void look_for_second(const ContractArgs &g, volatile uint32_t *found, uint32_t *marked) {
    bool any = false;
    auto look = [&](const uint8_t *bytes, int64_t n_bytes, uint32_t *marks) {
#pragma unroll 4
        for (int64_t n = 16 * (int64_t)threadIdx.x; n < n_bytes; n += 16 * 32 * kEpilogueWarps)
            if (any_of<16>(bytes + n) != 0u) {
                any = true;
                if (A_PARTS == 2) atomicOr(marks + ((n / kTileM >> 5) % kMarkWords), 1u << (n / kTileM & 31));
            }
    };
    static_assert(kTileM == kTileN);
    if (A_PARTS == 2) look(g.a_second, g.a_flags, marked);
    look(g.b_second, g.b_flags, marked + kMarkWords);
    if (any) *found = 1u;
}

// A stage's operands; each SM of the pair loads its own, the first one's barrier counts both.
template <bool A_FREE, bool B_FREE, int A_PARTS>
__device__ __forceinline__ void load_stage(uint32_t dst, uint32_t own_bar, uint32_t bar, uint32_t rank, const CUtensorMap *a_hi, const CUtensorMap *a_lo,
                                           const CUtensorMap *b_hi, const CUtensorMap *b_lo, int m0, int n0, int k) {
    if (rank == 0) mbar_arrive_expect_tx(own_bar, 2 * Ring<A_PARTS>::kStageBytes);
#pragma unroll
    for (int part = 0; part < A_PARTS; part++) {
        const CUtensorMap *am = part == 0 ? a_hi : a_lo;
        const uint32_t d = dst + part * kOperandBytes;
        if (A_FREE) {
            tma_load(d, am, m0, k, bar);
            tma_load(d + kOperandBytes / 2, am, m0 + 64, k, bar);
        } else {
            tma_load(d, am, k, m0, bar);
        }
    }
#pragma unroll
    for (int part = 0; part < 2; part++) {
        const CUtensorMap *bm = part == 0 ? b_hi : b_lo;
        const uint32_t d = dst + (A_PARTS + part) * kOperandBytes;
        if (B_FREE) {
            tma_load(d, bm, n0, k, bar);
            tma_load(d + kOperandBytes / 2, bm, n0 + 64, k, bar);
        } else {
            tma_load(d, bm, k, n0, bar);
        }
    }
}

// Its MMAs.
template <bool A_FREE, bool B_FREE, int A_PARTS>
__device__ __forceinline__ void multiply_stage(uint32_t a0, uint32_t tmem, bool accumulate) {
    // fp32 accumulators, fp16 operands, 256 x 256
    constexpr uint32_t idesc = 1u << 4 | (A_FREE ? 1u << 15 : 0u) | (B_FREE ? 1u << 16 : 0u) | (uint32_t)(kTileN >> 3) << 17 | (uint32_t)(kTileM >> 4) << 24;
    const uint32_t d_main = tmem, d_small = tmem + kTileN, b0 = a0 + A_PARTS * kOperandBytes;
#pragma unroll
    for (int k = 0; k < kBlockK / 16; k++) {
        const uint32_t later = accumulate || k > 0;
        const uint64_t ah = operand_desc<A_FREE>(a0 + k * kStepBytes<A_FREE>);
        const uint64_t bh = operand_desc<B_FREE>(b0 + k * kStepBytes<B_FREE>);
        const uint64_t bl = operand_desc<B_FREE>(b0 + kOperandBytes + k * kStepBytes<B_FREE>);
        mma_f16_pair(d_small, ah, bl, idesc, later);
        if (A_PARTS == 2) mma_f16_pair(d_small, operand_desc<A_FREE>(a0 + kOperandBytes + k * kStepBytes<A_FREE>), bh, idesc, 1u);
        mma_f16_pair(d_main, ah, bh, idesc, later);
    }
}

// A wait ran out: tells the others, and leaves only after a time in which every copy and MMA in flight has landed.
__device__ __forceinline__ void give_up(volatile uint32_t *gave_up) {
    if (*gave_up == 0u) atomicAdd(&g_contract_wait_errors, 1);
    *gave_up = 1u;
    const long long t0 = clock64();
    while (clock64() - t0 < kWaitLimitCycles / 16) {
    }
}

// All tiles' second turns, behind their first ones (a function of its own: together they cost the first ones' epilogue its registers).  The
// roles go on where they were; every tile of this pair has been written.
template <bool A_FREE, bool B_FREE, int A_PARTS>
__device__ __noinline__ void second_phase(uint32_t base, uint32_t full0, uint32_t tmem, volatile uint32_t *gave_up, const CUtensorMap *a_hi, const CUtensorMap *a_lo,
                                          const CUtensorMap *b_hi, const CUtensorMap *b_lo, const CUtensorMap *a_hi2, const CUtensorMap *a_lo2,
                                          const CUtensorMap *b_hi2, const CUtensorMap *b_lo2, const ContractArgs &g) {
    using R = Ring<A_PARTS>;
    const uint32_t empty0 = full0 + 8 * R::kStages, done0 = empty0 + 8 * R::kStages, free0 = done0 + 8;
    const volatile uint32_t *states = gave_up + 1, *marked = states + 4;
    auto takes = [](uint32_t groups, int kb) { return (groups >> (kb % kSliceBlocks * kBlockK / kCopyRows)) & 1u; };
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const uint32_t rank = cluster_rank();
    const int cluster = blockIdx.x >> 1, clusters = gridDim.x >> 1, items = g.m_tiles * g.n_tiles * g.splits;
    bool ok = __all_sync(0xffffffffu, *gave_up == 0u);
    auto sides = [&](const Item &it) { return A_PARTS == 2 ? sides_of(g, it, marked) : Sides{}; };
    if (warp == kEpilogueWarps) {
        int s = (int)(states[0] >> 2);
        uint32_t phase = states[0] & 1u;
        const uint32_t full_first = in_first(full0);
        for (int i = cluster; i < items && ok; i += clusters) {
            const Item it = item_of(g, i);
            const int m0 = it.m_tile * kTileM + (int)rank * 128, n0 = it.n_tile * kTileN + (int)rank * 128;
            ok = each_second_turn<A_PARTS>(g, it, sides(it), [&](int kb0, int turn, uint32_t groups) {
                for (int kb = kb0; kb < slice_end(it, kb0) && lane == 0 && ok; kb++) {
                    if (!takes(groups, kb)) continue;
                    ok = wait_cluster(empty0 + 8 * s, phase) && *gave_up == 0u;
                    if (!ok) break;
                    load_stage<A_FREE, B_FREE, A_PARTS>(base + s * R::kStageBytes, full0 + 8 * s, full_first + 8 * s, rank, turn & 1 ? a_hi2 : a_hi,
                                                        turn & 1 ? a_lo2 : a_lo, turn & 2 ? b_hi2 : b_hi, turn & 2 ? b_lo2 : b_lo, m0, n0, kb * kBlockK);
                    if (++s == R::kStages) { s = 0; phase ^= 1u; }
                }
                return __all_sync(0xffffffffu, ok) != 0;
            });
        }
        for (int n = 0; n < R::kStages && lane == 0 && ok; n++) {
            ok = wait_cluster(empty0 + 8 * s, phase);
            if (++s == R::kStages) { s = 0; phase ^= 1u; }
        }
    } else if (warp == kEpilogueWarps + 1 && rank == 0) {
        int s = (int)(states[1] >> 2);
        uint32_t phase = states[1] & 1u, acc_phase = (states[1] >> 1) & 1u;
        for (int i = cluster; i < items && ok; i += clusters) {
            const Item it = item_of(g, i);
            ok = each_second_turn<A_PARTS>(g, it, sides(it), [&](int kb0, int, uint32_t groups) {
                if (lane == 0) {
                    ok = wait_cluster(free0, acc_phase) && *gave_up == 0u;
                    fence_after();
                    acc_phase ^= 1u;
                    bool first = true;
                    for (int kb = kb0; kb < slice_end(it, kb0) && ok; kb++) {
                        if (!takes(groups, kb)) continue;
                        ok = wait_cluster(full0 + 8 * s, phase);
                        if (!ok) break;
                        fence_after();
                        multiply_stage<A_FREE, B_FREE, A_PARTS>(base + s * R::kStageBytes, tmem, !first);
                        first = false;
                        commit_pair(empty0 + 8 * s);
                        if (++s == R::kStages) { s = 0; phase ^= 1u; }
                    }
                    if (ok) commit_pair(done0);
                }
                return __all_sync(0xffffffffu, ok) != 0;
            });
        }
    } else if (warp < kEpilogueWarps) {
        const int quarter = warp & 3, cols0 = (warp >> 2) * kWarpCols;
        uint32_t acc_phase = states[2];
        const uint32_t src = tmem + cols0 + ((uint32_t)(quarter * 32) << 16), free_first = in_first(free0);
        if (lane == 0) asm volatile("fence.proxy.async;" ::: "memory");   // (the tiles went out through the asynchronous proxy)
        __syncwarp();
        for (int i = cluster; i < items && ok; i += clusters) {
            const Item it = item_of(g, i);
            const int row0 = it.m_tile * kTileM + (int)rank * 128 + quarter * 32;
            ok = each_second_turn<A_PARTS>(g, it, sides(it), [&](int kb0, int turn, uint32_t) {
                if (!__all_sync(0xffffffffu, wait_cluster(done0, acc_phase) && *gave_up == 0u)) return false;
                fence_after();
                acc_phase ^= 1u;
                add_second_turn<A_PARTS>(g, it, src, cols0, row0, kb0 / kSliceBlocks, turn);
                fence_before();
                __syncwarp();
                if (lane == 0) arrive_in_cluster(free_first);
                return true;
            });
        }
        // (behind all turns: nobody waits for these, and they have no limit in time)
        for (int i = cluster; i < items && ok && A_PARTS == 2; i += clusters) {
            const Item it = item_of(g, i);
            const Sides t = sides(it);
            if (t.a_single || t.b_single) add_single_products(g, t, it.m_tile * kTileM + (int)rank * 128 + quarter * 32, it.n_tile * kTileN + cols0);
        }
    }
    if (!ok) give_up(gave_up);
}

// A_FREE / B_FREE: the operand's free index is the contiguous one.  A_PARTS: 1: A is exact, 2: A has hi and lo as well.
template <bool A_FREE, bool B_FREE, int A_PARTS>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(32 * (kEpilogueWarps + 2), 1)
    contract_kernel(const __grid_constant__ CUtensorMap a_hi, const __grid_constant__ CUtensorMap a_lo, const __grid_constant__ CUtensorMap b_hi,
                    const __grid_constant__ CUtensorMap b_lo, const __grid_constant__ CUtensorMap a_hi2, const __grid_constant__ CUtensorMap a_lo2,
                    const __grid_constant__ CUtensorMap b_hi2, const __grid_constant__ CUtensorMap b_lo2, const __grid_constant__ CUtensorMap c_map,
                    const __grid_constant__ ContractArgs g) {
    using R = Ring<A_PARTS>;
    extern __shared__ unsigned char smem_raw[];
    const uint32_t base = (smem_u32(smem_raw) + 1023u) & ~1023u;
    unsigned char *base_ptr = smem_raw + (base - smem_u32(smem_raw));
    const uint32_t out0 = base + R::kStages * R::kStageBytes;
    const uint32_t bars = out0 + kEpilogueBytes;
    const uint32_t full0 = bars, empty0 = full0 + 8 * R::kStages, done0 = empty0 + 8 * R::kStages, free0 = done0 + 8;
    const uint32_t tmem_slot = free0 + 8;
    volatile uint32_t *tmem_ptr = reinterpret_cast<volatile uint32_t *>(base_ptr + (tmem_slot - base));
    volatile uint32_t *gave_up = tmem_ptr + 1, *states = tmem_ptr + 2;   // of three roles at the end, whether there are second halves, where
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const uint32_t rank = cluster_rank();
    const int cluster = blockIdx.x >> 1, clusters = gridDim.x >> 1;
    const int items = g.m_tiles * g.n_tiles * g.splits;

    if (threadIdx.x == 0) {
        for (int s = 0; s < R::kStages; s++) {
            mbar_init(full0 + 8 * s, 1);
            mbar_init(empty0 + 8 * s, 1);
        }
        mbar_init(done0, 1);
        mbar_init(free0, 2 * kEpilogueWarps);   // those of both SMs
        *gave_up = 0u;
        states[3] = 0u;
        fence_barrier_init();
    }
    if (warp == 0)
        for (int n = lane; n < 2 * kMarkWords; n += 32) states[4 + n] = 0u;
    if (warp == kEpilogueWarps + 1) {
        asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], 512;" ::"r"(tmem_slot) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;");
    }
    fence_before();
    __syncthreads();
    cluster_sync();
    fence_after();
    const uint32_t tmem = *tmem_ptr;
    bool ok = true;

    if (warp == kEpilogueWarps && lane == 0) {
        int s = 0;
        uint32_t phase = 1u;   // the first round finds the stages empty
        const uint32_t full_first = in_first(full0);
        for (int i = cluster; i < items && ok; i += clusters) {
            const Item it = item_of(g, i);
            const int m0 = it.m_tile * kTileM + (int)rank * 128, n0 = it.n_tile * kTileN + (int)rank * 128;
            for (int kb = it.kb0; kb < it.kb1; kb++) {
                ok = wait_cluster(empty0 + 8 * s, phase) && *gave_up == 0u;
                if (!ok) break;
                load_stage<A_FREE, B_FREE, A_PARTS>(base + s * R::kStageBytes, full0 + 8 * s, full_first + 8 * s, rank, &a_hi, &a_lo, &b_hi, &b_lo, m0, n0, kb * kBlockK);
                if (++s == R::kStages) { s = 0; phase ^= 1u; }
            }
        }
        states[0] = (uint32_t)s << 2 | phase;   // (of the next load: it may wait for the same as here)
        // the last stages' MMAs have read them before the pair leaves
        for (int n = 0; n < R::kStages && ok; n++) {
            ok = wait_cluster(empty0 + 8 * s, phase);
            if (++s == R::kStages) { s = 0; phase ^= 1u; }
        }
    } else if (warp == kEpilogueWarps + 1 && lane == 0 && rank == 0) {
        int s = 0;
        uint32_t phase = 0u, acc_phase = 1u;
        for (int i = cluster; i < items && ok; i += clusters) {
            const Item it = item_of(g, i);
            for (int kb0 = it.kb0, kb1; kb0 < it.kb1 && ok; kb0 = kb1) {
                kb1 = slice_end(it, kb0);
                ok = wait_cluster(free0, acc_phase) && *gave_up == 0u;
                if (!ok) break;
                fence_after();
                acc_phase ^= 1u;
                for (int kb = kb0; kb < kb1; kb++) {
                    ok = wait_cluster(full0 + 8 * s, phase);
                    if (!ok) break;
                    fence_after();
                    multiply_stage<A_FREE, B_FREE, A_PARTS>(base + s * R::kStageBytes, tmem, kb > kb0);
                    commit_pair(empty0 + 8 * s);
                    if (++s == R::kStages) { s = 0; phase ^= 1u; }
                }
                commit_pair(done0);
            }
        }
        states[1] = (uint32_t)s << 2 | acc_phase << 1 | phase;
    } else if (warp < kEpilogueWarps) {
        const int quarter = warp & 3, cols0 = (warp >> 2) * kWarpCols;   // (a warp reaches the 32 lanes of tensor memory of its number mod 4)
        const uint32_t out = out0 + warp * 4096;
        float *out_ptr = reinterpret_cast<float *>(base_ptr + (out - base));
        const uint32_t free_first = in_first(free0);
        uint32_t acc_phase = 0u;
        look_for_second<A_PARTS>(g, states + 3, const_cast<uint32_t *>(states) + 4);
        for (int i = cluster; i < items && ok; i += clusters) {
            const Item it = item_of(g, i);
            const int n0 = it.n_tile * kTileN + cols0, row0 = it.m_tile * kTileM + (int)rank * 128 + quarter * 32;
            // factors of columns c * 32 + lane (of the slice, where a column has one for each)
            float factor[kWarpCols / 32];
            auto load_factors = [&](const uint32_t *bits) {
#pragma unroll
                for (int c = 0; c < kWarpCols / 32; c++) {
                    const int n = n0 + c * 32 + lane;
                    factor[c] = n < g.N ? inverse_scale(__ldg(bits + n)) : 1.f;
                }
            };
            if (A_PARTS == 2) load_factors(g.col_bits);
            const float row_factor = A_PARTS == 2 && row0 + lane < g.M ? inverse_scale(__ldg(g.row_bits + row0 + lane)) : 1.f;
            float sum[kWarpCols];
#pragma unroll
            for (int n = 0; n < kWarpCols; n++) sum[n] = 0.f;
            for (int kb0 = it.kb0; kb0 < it.kb1; kb0 = (kb0 / kSliceBlocks + 1) * kSliceBlocks) {
                if (A_PARTS == 1) {
                    // through this warp's piece of shared memory, from which every lane reads four at a time (the last tile's
                    // stores have left it)
                    load_factors(g.col_bits + (int64_t)(kb0 / kSliceBlocks) * g.N);
                    if (lane == 0) asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");
                    __syncwarp();
#pragma unroll
                    for (int c = 0; c < kWarpCols / 32; c++) out_ptr[c * 32 + lane] = factor[c];
                    __syncwarp();
                }
                ok = __all_sync(0xffffffffu, wait_cluster(done0, acc_phase) && *gave_up == 0u);
                if (!ok) break;
                fence_after();
                acc_phase ^= 1u;
                const uint32_t src = tmem + cols0 + ((uint32_t)(quarter * 32) << 16);
#pragma unroll
                for (int c = 0; c < kWarpCols / 16; c++) {
                    uint32_t big[16], small[16];
                    tmem_load16(big, src + c * 16);
                    tmem_load16(small, src + kTileN + c * 16);
                    tmem_load_wait();
                    loaded(big);
                    loaded(small);
#pragma unroll
                    for (int n4 = 0; n4 < 4; n4++) {
                        const float4 f4 = A_PARTS == 1 ? *reinterpret_cast<const float4 *>(out_ptr + c * 16 + n4 * 4) : make_float4(1.f, 1.f, 1.f, 1.f);
                        const float f[4] = {f4.x, f4.y, f4.z, f4.w};
#pragma unroll
                        for (int e = 0; e < 4; e++) {
                            const int n = n4 * 4 + e;
                            const float v = fmaf(__uint_as_float(small[n]), kLoScale, __uint_as_float(big[n]));
                            sum[c * 16 + n] = A_PARTS == 1 ? fmaf(v, f[e], sum[c * 16 + n]) : sum[c * 16 + n] + v;
                        }
                    }
                }
                fence_before();
                __syncwarp();
                if (lane == 0) arrive_in_cluster(free_first);
            }
            if (!ok) break;
            // both factors within 2^+-60: any order will do; else the smaller one first, no overflow on the way to a finite result
            bool near = true;
            if (A_PARTS == 2) {
                near = fabsf(__log2f(row_factor)) < 60.f;
#pragma unroll
                for (int c = 0; c < kWarpCols / 32; c++) near = near && fabsf(__log2f(factor[c])) < 60.f;
                near = __all_sync(0xffffffffu, near);
            } else {
                __syncwarp();   // (the piece held the factors)
            }
#pragma unroll
            for (int c = 0; c < kWarpCols / 16; c++) {
                float o[16];
#pragma unroll
                for (int n = 0; n < 16; n++) {
                    o[n] = sum[c * 16 + n];
                    if (A_PARTS == 1) {
                        o[n] *= g.alpha;
                        continue;
                    }
                    const float f = __shfl_sync(0xffffffffu, factor[c / 2], (c & 1) * 16 + n);
                    if (near) o[n] = g.alpha * (o[n] * row_factor * f);
                    else o[n] = g.alpha * (o[n] * fminf(row_factor, f) * fmaxf(row_factor, f));
                }
                // the piece's previous store has been read from shared memory
                if (lane == 0) asm volatile("cp.async.bulk.wait_group.read 1;" ::: "memory");
                __syncwarp();
                float4 *row = reinterpret_cast<float4 *>(out_ptr + (c & 1) * 512 + lane * 16);
#pragma unroll
                for (int q = 0; q < 4; q++) row[q ^ ((lane >> 1) & 3)] = make_float4(o[4 * q], o[4 * q + 1], o[4 * q + 2], o[4 * q + 3]);
                asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
                __syncwarp();
                if (lane == 0) {
                    const uint32_t piece = out + (c & 1) * 2048;
                    const int n = n0 + c * 16;
                    if (row0 < g.M && n < g.N) {
                        if (g.splits > 1) tma_store(&c_map, piece, n, it.split * g.m_padded + row0);
                        else if (g.accumulate) tma_add(&c_map, piece, n, row0);
                        else tma_store(&c_map, piece, n, row0);
                    }
                    asm volatile("cp.async.bulk.commit_group;" ::: "memory");
                }
            }
        }
        if (lane == 0) asm volatile("cp.async.bulk.wait_group 0;" ::: "memory");
        if (threadIdx.x == 0) states[2] = acc_phase;
    }
    if (!ok) give_up(gave_up);
    __syncwarp();
    fence_before();
    __syncthreads();
    if (states[3] != 0u) {
        second_phase<A_FREE, B_FREE, A_PARTS>(base, full0, tmem, gave_up, &a_hi, &a_lo, &b_hi, &b_lo, &a_hi2, &a_lo2, &b_hi2, &b_lo2, g);
        __syncwarp();
        fence_before();
        __syncthreads();
    }
    cluster_sync();
    if (warp == kEpilogueWarps + 1) asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, 512;" ::"r"(tmem));
}

// ------------------------------------------------------------------------------------------------ host side
// A row-major matrix [rows x cols] read in boxes of box_rows x 64 (fp16) or written in boxes of 32 x 16 (fp32), swizzled.
int tensor_map(CUtensorMap *map, bool half, const void *p, int64_t rows, int64_t cols, int64_t pitch_bytes, int box_rows) {
    return tensor_map_2d(map, half ? 2 : 4, p, rows, cols, pitch_bytes, box_rows, half ? 64 : 16, half ? 128 : 64);
}

size_t align256(size_t v) { return (v + 255) & ~(size_t)255; }
int half_pitch(int cols) { return (cols + 7) & ~7; }   // rows of the fp16 copies start on 16 bytes

// Parts of the contraction.  A part keeps at least 8 blocks; the scratch of all parts is bounded.
constexpr int kMostParts = 32, kPartRows = 32768;
int most_parts(int M, int kblocks) {
    const int padded = (M + kTileM - 1) / kTileM * kTileM;
    int most = kblocks / 8 < kMostParts ? kblocks / 8 : kMostParts;
    if (most > kPartRows / padded) most = kPartRows / padded;
    return most < 1 ? 1 : most;
}
size_t parts_bytes(int M, int N, int kblocks) {
    // (of the most parts any smaller M or kblocks could take: a pass over fewer rows finds room as well)
    const int64_t padded = (M + kTileM - 1) / kTileM * (int64_t)kTileM;
    int64_t most = kblocks / 8 < kMostParts ? kblocks / 8 : kMostParts;
    int64_t rows = most * padded;
    if (rows > kPartRows) rows = kPartRows;
    return most < 2 ? 0 : align256((size_t)rows * N * 4);
}

size_t copy_bytes(int64_t rows, int cols, int64_t n_bits, int64_t n_second) {
    return 4 * align256((size_t)rows * half_pitch(cols) * 2) + align256((size_t)n_bits * 4) + align256((size_t)n_second);
}
Copy take_copy(unsigned char *&p, int64_t rows, int cols, int64_t n_bits, int64_t n_second) {
    Copy c;
    c.pitch = half_pitch(cols);
    const size_t one = align256((size_t)rows * c.pitch * 2);
    c.hi = reinterpret_cast<__half *>(p);
    c.lo = reinterpret_cast<__half *>(p + one);
    c.hi2 = reinterpret_cast<__half *>(p + 2 * one);
    c.lo2 = reinterpret_cast<__half *>(p + 3 * one);
    c.bits = reinterpret_cast<uint32_t *>(p + 4 * one);
    c.second = p + 4 * one + align256((size_t)n_bits * 4);
    p += copy_bytes(rows, cols, n_bits, n_second);
    return c;
}
int64_t slices_of(int64_t rows) { return (rows + kSliceRows - 1) / kSliceRows; }
int64_t tiles_of(int64_t n) { return (n + kTileN - 1) / kTileN; }
size_t row_copy_bytes(int64_t rows, int cols) { return copy_bytes(rows, cols, rows, tiles_of(rows) * kTileN); }
Copy take_row_copy(unsigned char *&p, int64_t rows, int cols) { return take_copy(p, rows, cols, rows, tiles_of(rows) * kTileN); }
size_t column_copy_bytes(int64_t rows, int cols) { return copy_bytes(rows, cols, slices_of(rows) * cols, slices_of(rows) * tiles_of(cols) * (kTileN / kCopyCols)); }
Copy take_column_copy(unsigned char *&p, int64_t rows, int cols) {
    return take_copy(p, rows, cols, slices_of(rows) * cols, slices_of(rows) * tiles_of(cols) * (kTileN / kCopyCols));
}

int copy_by_row(const float *x, int64_t rows, int cols, const Copy &c, cudaStream_t stream) {
    const int64_t want = (rows + 7) / 8, cap = (int64_t)device_info().sm_count * 8;
    split_rows_kernel<<<(unsigned)(want < cap ? want : cap), 256, 0, stream>>>(x, rows, cols, c);
    LUTB_LAUNCH_CHECK();
    return LUTB_OK;
}

int copy_by_column(const float *x, int64_t rows, int cols, const Copy &c, const DeepTarget &target, cudaStream_t stream) {
    LUTB_REQUIRE(tiles_of(cols) * (kTileN / kCopyCols) <= 65535, LUTB_ERR_SHAPE, "tensor-core contraction: too many columns");
    const dim3 grid((unsigned)slices_of(rows), (unsigned)(tiles_of(cols) * (kTileN / kCopyCols)));
    split_columns_kernel<<<grid, kCopyThreads, 0, stream>>>(x, rows, cols, c, target);
    LUTB_LAUNCH_CHECK();
    return LUTB_OK;
}

// Parts of the contraction: the count with the shortest estimated time, in SM cycles.  A work item takes about 1024 cycles a
// block; the parts are written and read once at about 3000 bytes a cycle.
int choose_parts(int M, int N, int kblocks, int clusters) {
    const int64_t tiles = (int64_t)((M + kTileM - 1) / kTileM) * ((N + kTileN - 1) / kTileN);
    int best = 1;
    int64_t least = -1;
    for (int s = 1; s <= most_parts(M, kblocks); s++) {
        const int64_t per = (kblocks + s - 1) / s, waves = (tiles * s + clusters - 1) / clusters;
        if ((kblocks + per - 1) / per != s) continue;   // (an empty last part)
        const int64_t cost = waves * (per * 1024 + 2000) + (s > 1 ? (int64_t)s * M * N * 8 / 3000 + 4000 : 0);
        if (least < 0 || cost < least) { least = cost; best = s; }
    }
    return best;
}

// Measured on one B200, the contraction / its operand copies and sums of parts, us (before, TF32 halves -> now):
//   forward   8192 x 256, KT 16384   176 / 29 -> 101 / 24     1024 x 1024, KT 65536   345 / 174 -> 182 / 102
//   table gradient, same sizes       166 / 24 -> 101 / 8                              340 / 101 -> 213 / 8
//   row dots, same sizes             258 / 13 -> 184 / 13                             491 / 165 -> 273 / 92
// 1400 to 1500 TFLOP/s of fp16 in the long ones; 64 work items on 74 pairs of SMs in the first two of the left column.
template <bool A_FREE, bool B_FREE, int A_PARTS>
int launch_contraction(ContractArgs g, const CUtensorMap (&a)[4], const CUtensorMap (&b)[4], float *C, float *parts, cudaStream_t stream) {
    using R = Ring<A_PARTS>;
    const int clusters = device_info().sm_count / 2;
    g.m_tiles = (g.M + kTileM - 1) / kTileM;
    g.n_tiles = (g.N + kTileN - 1) / kTileN;
    g.m_padded = g.m_tiles * kTileM;
    g.splits = parts != nullptr ? choose_parts(g.M, g.N, g.kblocks, clusters) : 1;
    g.kb_per_split = (g.kblocks + g.splits - 1) / g.splits;
    g.m_fast = g.N > g.M;   // the larger operand is read once, the smaller one stays in L2
    const int64_t items = (int64_t)g.m_tiles * g.n_tiles * g.splits;
    LUTB_REQUIRE(items <= 0x7fffffff, LUTB_ERR_SHAPE, "tensor-core contraction: too many tiles");
    const float alpha = g.alpha;
    g.c = C;
    g.second_alpha = alpha;
    g.a_flags = A_PARTS == 2 ? (int64_t)g.m_tiles * kTileM : 0;
    g.b_flags = A_PARTS == 2 ? (int64_t)g.n_tiles * kTileN : slices_of((int64_t)g.kblocks * kBlockK) * g.n_tiles * (kTileN / kCopyCols);
    CUtensorMap c;
    int rc;
    if (g.splits > 1) {
        g.alpha = 1.f;
        rc = tensor_map(&c, false, parts, (int64_t)g.splits * g.m_padded, g.N, (int64_t)g.N * 4, 32);
    } else {
        rc = tensor_map(&c, false, C, g.M, g.N, (int64_t)g.N * 4, 32);
    }
    if (rc) return rc;
    auto kern = contract_kernel<A_FREE, B_FREE, A_PARTS>;
    LUTB_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)R::kSmem));
    const int grid = 2 * (int)(items < clusters ? items : clusters);
    kern<<<grid, 32 * (kEpilogueWarps + 2), R::kSmem, stream>>>(a[0], a[1], b[0], b[1], a[2], a[3], b[2], b[3], c, g);
    LUTB_LAUNCH_CHECK();
    if (g.splits > 1) {
        const int64_t want = ((int64_t)g.M * (g.N / 4) + kAddThreads - 1) / kAddThreads, cap = (int64_t)device_info().sm_count * 16;
        auto add = g.splits > 4 ? add_parts_kernel<16> : g.splits > 2 ? add_parts_kernel<4> : add_parts_kernel<2>;
        add<<<(unsigned)(want < cap ? want : cap), kAddThreads, 0, stream>>>(parts, C, g.M, g.N, g.splits, (int64_t)g.m_padded * g.N, alpha);
        LUTB_LAUNCH_CHECK();
    }
    return LUTB_OK;
}

unsigned char *aligned_base(void *workspace) {
    return reinterpret_cast<unsigned char *>((reinterpret_cast<uintptr_t>(workspace) + 255) & ~(uintptr_t)255);
}
int blocks_of(int k) { return (k + kBlockK - 1) / kBlockK; }

}  // namespace

size_t hist_gemm_workspace(HistGemmKind kind, int rows, int KT, int O) {
    if (kind == HG_FORWARD) return column_copy_bytes(KT, O) + parts_bytes(rows, O, blocks_of(KT)) + 256;
    if (kind == HG_TABLE_GRAD) return column_copy_bytes(rows, O) + parts_bytes(KT, O, blocks_of(rows)) + 256;
    return row_copy_bytes(rows, O) + row_copy_bytes(KT, O) + 256;
}

// Tensor maps of the first and second halves
static int operand_maps(CUtensorMap (&m)[4], const Copy &c, int64_t rows, int cols, int box_rows) {
    const __half *p[4] = {c.hi, c.lo, c.hi2, c.lo2};
    int rc = LUTB_OK;
    for (int i = 0; i < 4 && !rc; i++) rc = tensor_map(&m[i], true, p[i], rows, cols, (int64_t)c.pitch * 2, box_rows);
    return rc;
}
static int exact_maps(CUtensorMap (&m)[4], const __half *H, int64_t rows, int64_t cols, int box_rows) {
    const int rc = tensor_map(&m[0], true, H, rows, cols, cols * 2, box_rows);
    m[1] = m[2] = m[3] = m[0];
    return rc;
}

#define LUTB_CONTRACT_WORKSPACE(KIND)                                                                                \
    LUTB_REQUIRE(workspace != nullptr && workspace_bytes >= hist_gemm_workspace(KIND, rows, KT, O), LUTB_ERR_WORKSPACE, \
                 "tensor-core contraction needs %zu bytes of workspace", hist_gemm_workspace(KIND, rows, KT, O))

int hist_gemm_forward(int rows, int KT, int O, const __half *H, const float *W, float *y, void *workspace, size_t workspace_bytes,
                      cudaStream_t stream) {
    LUTB_CONTRACT_WORKSPACE(HG_FORWARD);
    unsigned char *p = aligned_base(workspace);
    const Copy w = take_column_copy(p, KT, O);
    float *parts = parts_bytes(rows, O, blocks_of(KT)) ? reinterpret_cast<float *>(p) : nullptr;
    int rc = copy_by_column(W, KT, O, w, DeepTarget{H, y, KT, rows, 1.f, false}, stream);
    CUtensorMap a[4], b[4];
    if (!rc) rc = exact_maps(a, H, rows, KT, 128);
    if (!rc) rc = operand_maps(b, w, KT, O, kBlockK);
    if (rc) return rc;
    ContractArgs g{};
    g.M = rows; g.N = O; g.kblocks = blocks_of(KT);
    g.accumulate = 1; g.col_bits = w.bits; g.b_second = w.second; g.alpha = 1.f;
    return launch_contraction<false, true, 1>(g, a, b, y, parts, stream);
}

int hist_gemm_table_grad(int rows, int KT, int O, const __half *H, const float *dY, float *target, float lr, void *workspace,
                         size_t workspace_bytes, cudaStream_t stream) {
    LUTB_CONTRACT_WORKSPACE(HG_TABLE_GRAD);
    unsigned char *p = aligned_base(workspace);
    const Copy d = take_column_copy(p, rows, O);
    float *parts = parts_bytes(KT, O, blocks_of(rows)) ? reinterpret_cast<float *>(p) : nullptr;
    int rc = copy_by_column(dY, rows, O, d, DeepTarget{H, target, KT, KT, lr, true}, stream);
    CUtensorMap a[4], b[4];
    if (!rc) rc = exact_maps(a, H, rows, KT, kBlockK);
    if (!rc) rc = operand_maps(b, d, rows, O, kBlockK);
    if (rc) return rc;
    ContractArgs g{};
    g.M = KT; g.N = O; g.kblocks = blocks_of(rows);
    g.accumulate = 1; g.col_bits = d.bits; g.b_second = d.second; g.alpha = lr;
    return launch_contraction<true, true, 1>(g, a, b, target, parts, stream);
}

int hist_gemm_row_dots(int rows, int KT, int O, const float *dY, const float *W, float *Q, void *workspace, size_t workspace_bytes,
                       cudaStream_t stream) {
    LUTB_CONTRACT_WORKSPACE(HG_ROW_DOTS);
    unsigned char *p = aligned_base(workspace);
    const Copy d = take_row_copy(p, rows, O), w = take_row_copy(p, KT, O);
    int rc = copy_by_row(dY, rows, O, d, stream);
    if (!rc) rc = copy_by_row(W, KT, O, w, stream);
    CUtensorMap a[4], b[4];
    if (!rc) rc = operand_maps(a, d, rows, O, 128);
    if (!rc) rc = operand_maps(b, w, KT, O, 128);
    if (rc) return rc;
    ContractArgs g{};
    g.M = rows; g.N = KT; g.kblocks = blocks_of(O);
    g.row_bits = d.bits; g.col_bits = w.bits; g.a_second = d.second; g.b_second = w.second; g.alpha = 1.f;
    g.a = dY; g.b = W; g.depth = O;
    return launch_contraction<false, false, 2>(g, a, b, Q, nullptr, stream);
}

}  // namespace lutb
