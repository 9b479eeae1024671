// Contractions of the histogram path on the sm_100a tensor cores: fp32 results from fp16 operands.
//
// Row counts are small integers (below 2049), exact in fp16.  An fp32 operand x (a table, an output gradient) is scaled
// by a power of two that brings the largest element of its row - or of its column within 1024 rows - to [2^14, 2^15), and kept as
// two fp16 values: hi = x * s rounded, lo = (x * s - hi) * 2^11 rounded.  x * s = hi + lo * 2^-11 to 2^-22 of x, as with the two
// 11-bit halves of a TF32 split, for elements down to 2^-29 of the largest, and to 2^-51 of the largest below that.  The scale
// belongs to a free index of the contraction (and to a slice of the contraction, see below), so it comes out of the sum as a factor.
// The products hi.hi go into one accumulator in tensor memory, hi.lo and lo.hi into another (their sum counts 2^-11 times),
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
constexpr float kLoScale = 1.0f / 2048.0f;

template <int A_PARTS>
struct Ring {
    static constexpr int kStageBytes = (A_PARTS + 2) * kOperandBytes;
    static constexpr int kStages = A_PARTS == 1 ? 4 : 3;
    static constexpr size_t kSmem = (size_t)kStages * kStageBytes + kEpilogueBytes + 256 + 1024;
};

struct ContractArgs {
    int M, N, kblocks;            // result and contraction extents; blocks of kBlockK
    int m_tiles, n_tiles, splits, kb_per_split;
    int m_fast;                   // tiles of neighbouring work items differ in m (else in n)
    int m_padded;                 // rows of one part's result in scratch (splits > 1)
    int accumulate;               // add to what is there
    // bits of the largest magnitude of each row of A (or null) and of each column of the result: [N], or, A exact, [slice][N]
    const uint32_t *row_bits, *col_bits;
    float alpha;
};

// Exponent of the scale of a row whose largest magnitude has these bits: the largest becomes 2^14 to 2^15 (as far as the
// scale itself is a normal number).
__device__ __forceinline__ int scale_exponent(uint32_t bits) { return min(141 - (int)(bits >> 23), 126); }
__device__ __forceinline__ float scale_of(uint32_t bits) { return __uint_as_float((uint32_t)(scale_exponent(bits) + 127) << 23); }
__device__ __forceinline__ float inverse_scale(uint32_t bits) { return __uint_as_float((uint32_t)(127 - scale_exponent(bits)) << 23); }

// ------------------------------------------------------------------------------------------------ operand copies
struct Halves { uint2 hi, lo; };   // of four neighbouring elements
__device__ __forceinline__ Halves split4(float4 v, float sx, float sy, float sz, float sw) {
    v.x *= sx; v.y *= sy; v.z *= sz; v.w *= sw;
    const __half2 h0 = __floats2half2_rn(v.x, v.y), h1 = __floats2half2_rn(v.z, v.w);
    const float2 f0 = __half22float2(h0), f1 = __half22float2(h1);
    const __half2 l0 = __floats2half2_rn((v.x - f0.x) * 2048.f, (v.y - f0.y) * 2048.f);
    const __half2 l1 = __floats2half2_rn((v.z - f1.x) * 2048.f, (v.w - f1.y) * 2048.f);
    Halves r;
    r.hi = make_uint2(*reinterpret_cast<const uint32_t *>(&h0), *reinterpret_cast<const uint32_t *>(&h1));
    r.lo = make_uint2(*reinterpret_cast<const uint32_t *>(&l0), *reinterpret_cast<const uint32_t *>(&l1));
    return r;
}
__device__ __forceinline__ uint32_t magnitude4(float4 v) {
    const uint32_t a = max(__float_as_uint(v.x) & 0x7fffffffu, __float_as_uint(v.y) & 0x7fffffffu);
    const uint32_t b = max(__float_as_uint(v.z) & 0x7fffffffu, __float_as_uint(v.w) & 0x7fffffffu);
    return max(a, b);
}

// Scaled by row: a warp per row, which stays in registers up to 1024 columns (read twice beyond).  HBM bound.
__global__ void __launch_bounds__(256) split_rows_kernel(const float *__restrict__ x, int64_t rows, int cols, __half *__restrict__ hi,
                                                         __half *__restrict__ lo, int pitch, uint32_t *__restrict__ bits) {
    constexpr int KEEP = 8;
    const int lane = threadIdx.x & 31, c4 = cols >> 2;
    for (int64_t r = (int64_t)blockIdx.x * 8 + (threadIdx.x >> 5); r < rows; r += (int64_t)gridDim.x * 8) {
        const float4 *src = reinterpret_cast<const float4 *>(x + r * cols);
        float4 v[KEEP];
        uint32_t m = 0u;
#pragma unroll
        for (int n = 0; n < KEEP; n++) {
            const int c = n * 32 + lane;
            v[n] = c < c4 ? __ldg(src + c) : make_float4(0.f, 0.f, 0.f, 0.f);
        }
#pragma unroll
        for (int n = 0; n < KEEP; n++) m = max(m, magnitude4(v[n]));
        for (int c = KEEP * 32 + lane; c < c4; c += 32) m = max(m, magnitude4(__ldg(src + c)));
        m = __reduce_max_sync(0xffffffffu, m);
        if (lane == 0) bits[r] = m;
        const float s = scale_of(m);
        uint2 *h = reinterpret_cast<uint2 *>(hi + r * pitch), *l = reinterpret_cast<uint2 *>(lo + r * pitch);
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
    }
}

// Scaled by column and slice of kSliceRows rows: a block takes 32 columns of a slice, which stay in its registers between the
// maximum and the copy, so that the matrix is read once (a pass for the maxima of whole columns took 41 of the 123 us for 65536 x
// 1024, and 7 + 5 us for 16384 x 256).  bits: [slice][cols].
constexpr int kSliceRows = kSliceBlocks * kBlockK, kCopyRows = 128;
__global__ void __launch_bounds__(8 * kCopyRows) split_columns_kernel(const float *__restrict__ x, int64_t rows, int cols, __half *__restrict__ hi,
                                                                      __half *__restrict__ lo, int pitch, uint32_t *__restrict__ bits) {
    __shared__ uint32_t part[kCopyRows / 4][32];
    constexpr int KEEP = kSliceRows / kCopyRows;
    const int tx = threadIdx.x & 7, ty = threadIdx.x >> 3, c4 = blockIdx.y * 8 + tx;
    const bool live = c4 < (cols >> 2);
    const int64_t r0 = (int64_t)blockIdx.x * kSliceRows;
    float4 v[KEEP];
    uint4 m = make_uint4(0u, 0u, 0u, 0u);
#pragma unroll
    for (int k = 0; k < KEEP; k++) {
        const int64_t r = r0 + k * kCopyRows + ty;
        v[k] = live && r < rows ? __ldg(reinterpret_cast<const float4 *>(x + r * cols) + c4) : make_float4(0.f, 0.f, 0.f, 0.f);
    }
#pragma unroll
    for (int k = 0; k < KEEP; k++) {
        m.x = max(m.x, __float_as_uint(v[k].x) & 0x7fffffffu);
        m.y = max(m.y, __float_as_uint(v[k].y) & 0x7fffffffu);
        m.z = max(m.z, __float_as_uint(v[k].z) & 0x7fffffffu);
        m.w = max(m.w, __float_as_uint(v[k].w) & 0x7fffffffu);
    }
#pragma unroll
    for (int o = 8; o < 32; o <<= 1) {   // a warp has four rows of the eight column quadruples
        m.x = max(m.x, __shfl_xor_sync(0xffffffffu, m.x, o));
        m.y = max(m.y, __shfl_xor_sync(0xffffffffu, m.y, o));
        m.z = max(m.z, __shfl_xor_sync(0xffffffffu, m.z, o));
        m.w = max(m.w, __shfl_xor_sync(0xffffffffu, m.w, o));
    }
    if ((threadIdx.x & 31) < 8) *reinterpret_cast<uint4 *>(&part[threadIdx.x >> 5][4 * tx]) = m;
    __syncthreads();
    if (threadIdx.x < 32) {
        uint32_t most = 0u;
#pragma unroll
        for (int k = 0; k < kCopyRows / 4; k++) most = max(most, part[k][threadIdx.x]);
        part[0][threadIdx.x] = most;
        if (blockIdx.y * 32 + threadIdx.x < cols) bits[(int64_t)blockIdx.x * cols + blockIdx.y * 32 + threadIdx.x] = most;
    }
    __syncthreads();
    if (!live) return;
    const uint4 b = *reinterpret_cast<const uint4 *>(&part[0][4 * tx]);
    const float sx = scale_of(b.x), sy = scale_of(b.y), sz = scale_of(b.z), sw = scale_of(b.w);
#pragma unroll
    for (int k = 0; k < KEEP; k++) {
        const int64_t r = r0 + k * kCopyRows + ty;
        if (r >= rows) break;
        const Halves q = split4(v[k], sx, sy, sz, sw);
        *(reinterpret_cast<uint2 *>(hi + r * pitch) + c4) = q.hi;
        *(reinterpret_cast<uint2 *>(lo + r * pitch) + c4) = q.lo;
    }
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

// A_FREE / B_FREE: the operand's free index is the contiguous one.  A_PARTS: 1: A is exact, 2: A has hi and lo as well.
template <bool A_FREE, bool B_FREE, int A_PARTS>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(32 * (kEpilogueWarps + 2), 1)
    contract_kernel(const __grid_constant__ CUtensorMap a_hi, const __grid_constant__ CUtensorMap a_lo, const __grid_constant__ CUtensorMap b_hi,
                    const __grid_constant__ CUtensorMap b_lo, const __grid_constant__ CUtensorMap c_map, const ContractArgs g) {
    using R = Ring<A_PARTS>;
    extern __shared__ unsigned char smem_raw[];
    const uint32_t base = (smem_u32(smem_raw) + 1023u) & ~1023u;
    unsigned char *base_ptr = smem_raw + (base - smem_u32(smem_raw));
    const uint32_t out0 = base + R::kStages * R::kStageBytes;
    const uint32_t bars = out0 + kEpilogueBytes;
    const uint32_t full0 = bars, empty0 = full0 + 8 * R::kStages, done0 = empty0 + 8 * R::kStages, free0 = done0 + 8;
    const uint32_t tmem_slot = free0 + 8;
    volatile uint32_t *tmem_ptr = reinterpret_cast<volatile uint32_t *>(base_ptr + (tmem_slot - base));
    volatile uint32_t *gave_up = tmem_ptr + 1;
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
        fence_barrier_init();
    }
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
                if (rank == 0) mbar_arrive_expect_tx(full0 + 8 * s, 2 * R::kStageBytes);
                const uint32_t dst = base + s * R::kStageBytes, bar = full_first + 8 * s;
                const int k = kb * kBlockK;
#pragma unroll
                for (int part = 0; part < A_PARTS; part++) {
                    const CUtensorMap *am = part == 0 ? &a_hi : &a_lo;
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
                    const CUtensorMap *bm = part == 0 ? &b_hi : &b_lo;
                    const uint32_t d = dst + (A_PARTS + part) * kOperandBytes;
                    if (B_FREE) {
                        tma_load(d, bm, n0, k, bar);
                        tma_load(d + kOperandBytes / 2, bm, n0 + 64, k, bar);
                    } else {
                        tma_load(d, bm, k, n0, bar);
                    }
                }
                if (++s == R::kStages) { s = 0; phase ^= 1u; }
            }
        }
        // the last stages' MMAs have read them before the pair leaves
        for (int n = 0; n < R::kStages && ok; n++) {
            ok = wait_cluster(empty0 + 8 * s, phase);
            if (++s == R::kStages) { s = 0; phase ^= 1u; }
        }
    } else if (warp == kEpilogueWarps + 1 && lane == 0 && rank == 0) {
        // fp32 accumulators, fp16 operands, 256 x 256
        const uint32_t idesc = 1u << 4 | (A_FREE ? 1u << 15 : 0u) | (B_FREE ? 1u << 16 : 0u) | (uint32_t)(kTileN >> 3) << 17 | (uint32_t)(kTileM >> 4) << 24;
        int s = 0;
        uint32_t phase = 0u, acc_phase = 1u;
        for (int i = cluster; i < items && ok; i += clusters) {
            const Item it = item_of(g, i);
            for (int kb0 = it.kb0, kb1; kb0 < it.kb1 && ok; kb0 = kb1) {
                kb1 = min(it.kb1, (kb0 / kSliceBlocks + 1) * kSliceBlocks);
                ok = wait_cluster(free0, acc_phase) && *gave_up == 0u;
                if (!ok) break;
                fence_after();
                acc_phase ^= 1u;
                const uint32_t d_main = tmem, d_small = tmem + kTileN;
                for (int kb = kb0; kb < kb1; kb++) {
                    ok = wait_cluster(full0 + 8 * s, phase);
                    if (!ok) break;
                    fence_after();
                    const uint32_t a0 = base + s * R::kStageBytes, b0 = a0 + A_PARTS * kOperandBytes;
#pragma unroll
                    for (int k = 0; k < kBlockK / 16; k++) {
                        const uint32_t later = kb > kb0 || k > 0;
                        const uint64_t ah = operand_desc<A_FREE>(a0 + k * kStepBytes<A_FREE>);
                        const uint64_t bh = operand_desc<B_FREE>(b0 + k * kStepBytes<B_FREE>);
                        const uint64_t bl = operand_desc<B_FREE>(b0 + kOperandBytes + k * kStepBytes<B_FREE>);
                        mma_f16_pair(d_small, ah, bl, idesc, later);
                        if (A_PARTS == 2) mma_f16_pair(d_small, operand_desc<A_FREE>(a0 + kOperandBytes + k * kStepBytes<A_FREE>), bh, idesc, 1u);
                        mma_f16_pair(d_main, ah, bh, idesc, later);
                    }
                    commit_pair(empty0 + 8 * s);
                    if (++s == R::kStages) { s = 0; phase ^= 1u; }
                }
                commit_pair(done0);
            }
        }
    } else if (warp < kEpilogueWarps) {
        const int quarter = warp & 3, cols0 = (warp >> 2) * kWarpCols;   // (a warp reaches the 32 lanes of tensor memory of its number mod 4)
        const uint32_t out = out0 + warp * 4096;
        float *out_ptr = reinterpret_cast<float *>(base_ptr + (out - base));
        const uint32_t free_first = in_first(free0);
        uint32_t acc_phase = 0u;
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
    }
    if (!ok) {
        // a wait ran out: tell the others, and leave only after a time in which every copy and MMA in flight has landed
        if (*gave_up == 0u) atomicAdd(&g_contract_wait_errors, 1);
        *gave_up = 1u;
        const long long t0 = clock64();
        while (clock64() - t0 < kWaitLimitCycles / 16) {
        }
    }
    __syncwarp();
    fence_before();
    __syncthreads();
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

struct Copy { __half *hi, *lo; uint32_t *bits; int pitch; };
size_t copy_bytes(int64_t rows, int cols, int64_t n_bits) { return 2 * align256((size_t)rows * half_pitch(cols) * 2) + align256((size_t)n_bits * 4); }
Copy take_copy(unsigned char *&p, int64_t rows, int cols, int64_t n_bits) {
    Copy c;
    c.pitch = half_pitch(cols);
    const size_t one = align256((size_t)rows * c.pitch * 2);
    c.hi = reinterpret_cast<__half *>(p);
    c.lo = reinterpret_cast<__half *>(p + one);
    c.bits = reinterpret_cast<uint32_t *>(p + 2 * one);
    p += 2 * one + align256((size_t)n_bits * 4);
    return c;
}

int copy_by_row(const float *x, int64_t rows, int cols, const Copy &c, cudaStream_t stream) {
    const int64_t want = (rows + 7) / 8, cap = (int64_t)device_info().sm_count * 8;
    split_rows_kernel<<<(unsigned)(want < cap ? want : cap), 256, 0, stream>>>(x, rows, cols, c.hi, c.lo, c.pitch, c.bits);
    LUTB_LAUNCH_CHECK();
    return LUTB_OK;
}

int64_t slices_of(int64_t rows) { return (rows + kSliceRows - 1) / kSliceRows; }

int copy_by_column(const float *x, int64_t rows, int cols, const Copy &c, cudaStream_t stream) {
    LUTB_REQUIRE((cols + 31) / 32 <= 65535, LUTB_ERR_SHAPE, "tensor-core contraction: too many columns");
    const dim3 grid((unsigned)slices_of(rows), (unsigned)((cols + 31) / 32));
    split_columns_kernel<<<grid, 8 * kCopyRows, 0, stream>>>(x, rows, cols, c.hi, c.lo, c.pitch, c.bits);
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
int launch_contraction(ContractArgs g, const CUtensorMap (&a)[2], const CUtensorMap (&b)[2], float *C, float *parts, cudaStream_t stream) {
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
    kern<<<grid, 32 * (kEpilogueWarps + 2), R::kSmem, stream>>>(a[0], a[1], b[0], b[1], c, g);
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
    if (kind == HG_FORWARD) return copy_bytes(KT, O, slices_of(KT) * O) + parts_bytes(rows, O, blocks_of(KT)) + 256;
    if (kind == HG_TABLE_GRAD) return copy_bytes(rows, O, slices_of(rows) * O) + parts_bytes(KT, O, blocks_of(rows)) + 256;
    return copy_bytes(rows, O, rows) + copy_bytes(KT, O, KT) + 256;
}

#define LUTB_CONTRACT_WORKSPACE(KIND)                                                                                \
    LUTB_REQUIRE(workspace != nullptr && workspace_bytes >= hist_gemm_workspace(KIND, rows, KT, O), LUTB_ERR_WORKSPACE, \
                 "tensor-core contraction needs %zu bytes of workspace", hist_gemm_workspace(KIND, rows, KT, O))

int hist_gemm_forward(int rows, int KT, int O, const __half *H, const float *W, float *y, void *workspace, size_t workspace_bytes,
                      cudaStream_t stream) {
    LUTB_CONTRACT_WORKSPACE(HG_FORWARD);
    unsigned char *p = aligned_base(workspace);
    const Copy w = take_copy(p, KT, O, slices_of(KT) * O);
    float *parts = parts_bytes(rows, O, blocks_of(KT)) ? reinterpret_cast<float *>(p) : nullptr;
    int rc = copy_by_column(W, KT, O, w, stream);
    if (rc) return rc;
    CUtensorMap a[2], b[2];
    rc = tensor_map(&a[0], true, H, rows, KT, (int64_t)KT * 2, 128);
    if (!rc) rc = tensor_map(&b[0], true, w.hi, KT, O, (int64_t)w.pitch * 2, kBlockK);
    if (!rc) rc = tensor_map(&b[1], true, w.lo, KT, O, (int64_t)w.pitch * 2, kBlockK);
    if (rc) return rc;
    a[1] = a[0];
    ContractArgs g{};
    g.M = rows; g.N = O; g.kblocks = blocks_of(KT);
    g.accumulate = 1; g.col_bits = w.bits; g.alpha = 1.f;
    return launch_contraction<false, true, 1>(g, a, b, y, parts, stream);
}

int hist_gemm_table_grad(int rows, int KT, int O, const __half *H, const float *dY, float *target, float lr, void *workspace,
                         size_t workspace_bytes, cudaStream_t stream) {
    LUTB_CONTRACT_WORKSPACE(HG_TABLE_GRAD);
    unsigned char *p = aligned_base(workspace);
    const Copy d = take_copy(p, rows, O, slices_of(rows) * O);
    float *parts = parts_bytes(KT, O, blocks_of(rows)) ? reinterpret_cast<float *>(p) : nullptr;
    int rc = copy_by_column(dY, rows, O, d, stream);
    if (rc) return rc;
    CUtensorMap a[2], b[2];
    rc = tensor_map(&a[0], true, H, rows, KT, (int64_t)KT * 2, kBlockK);
    if (!rc) rc = tensor_map(&b[0], true, d.hi, rows, O, (int64_t)d.pitch * 2, kBlockK);
    if (!rc) rc = tensor_map(&b[1], true, d.lo, rows, O, (int64_t)d.pitch * 2, kBlockK);
    if (rc) return rc;
    a[1] = a[0];
    ContractArgs g{};
    g.M = KT; g.N = O; g.kblocks = blocks_of(rows);
    g.accumulate = 1; g.col_bits = d.bits; g.alpha = lr;
    return launch_contraction<true, true, 1>(g, a, b, target, parts, stream);
}

int hist_gemm_row_dots(int rows, int KT, int O, const float *dY, const float *W, float *Q, void *workspace, size_t workspace_bytes,
                       cudaStream_t stream) {
    LUTB_CONTRACT_WORKSPACE(HG_ROW_DOTS);
    unsigned char *p = aligned_base(workspace);
    const Copy d = take_copy(p, rows, O, rows), w = take_copy(p, KT, O, KT);
    int rc = copy_by_row(dY, rows, O, d, stream);
    if (!rc) rc = copy_by_row(W, KT, O, w, stream);
    if (rc) return rc;
    CUtensorMap a[2], b[2];
    rc = tensor_map(&a[0], true, d.hi, rows, O, (int64_t)d.pitch * 2, 128);
    if (!rc) rc = tensor_map(&a[1], true, d.lo, rows, O, (int64_t)d.pitch * 2, 128);
    if (!rc) rc = tensor_map(&b[0], true, w.hi, KT, O, (int64_t)w.pitch * 2, 128);
    if (!rc) rc = tensor_map(&b[1], true, w.lo, KT, O, (int64_t)w.pitch * 2, 128);
    if (rc) return rc;
    ContractArgs g{};
    g.M = rows; g.N = KT; g.kblocks = blocks_of(O);
    g.row_bits = d.bits; g.col_bits = w.bits; g.alpha = 1.f;
    return launch_contraction<false, false, 2>(g, a, b, Q, nullptr, stream);
}

}  // namespace lutb
