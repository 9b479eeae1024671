// Non-sequence, fully connected LUT layer: anchor comparison + bit packing, table-row gather and
// accumulate, surrogate input gradient and table-gradient scatter.  sm_100a, no tensor cores: the
// path is gather/scatter bound.
#include "lutb_common.cuh"
#include "nonseq_fc.cuh"
#include "fc_dw_sorted.cuh"
#include "infer_staged.cuh"

#include <type_traits>

namespace lutb {

// --------------------------------------------------------------------------------------------
// Kernel 1: anchor-pair comparison and bit packing.
//
// A block stages `GROUPS * R` input rows in shared memory, transposed to [input][row] so that one
// 128-bit shared load returns the same input of four rows.  Each thread owns one detector, walks its
// anchor pairs once and evaluates all R rows of its group from registers.  Per (row, detector) it
// emits the packed table index and, for training, the first anchor pair of minimal |delta| with its
// signed delta (reference: check_detectors[_eval]_logic, lut_runtime_kernels_logic.proto:1050-1158).
// --------------------------------------------------------------------------------------------
// 16-byte slots of the transposed staging area are XOR-swizzled with the 8-slot row they lie in: neighbouring
// lanes stage inputs 4 apart (slots 4 * R / 4 apart), which without the swizzle all fall into the same banks.
__device__ __forceinline__ int swizzle_slot(int slot) { return slot ^ ((slot >> 3) & 7); }
// floats of one row group's staging area (whole 8-slot rows, so a swizzled slot never leaves the area)
template <int R>
__host__ __device__ constexpr size_t staged_floats(int n_inputs) {
    return R % 4 == 0 ? ((((size_t)n_inputs * (R / 4)) + 7) & ~(size_t)7) * 4 : (size_t)R * n_inputs;
}

static size_t staged_bytes(int R, int n_inputs) {
    return 4 * (R == 8 ? staged_floats<8>(n_inputs) : R == 4 ? staged_floats<4>(n_inputs) : (size_t)R * n_inputs);
}

// Stages the R rows [row0, row0 + nrows) of one row group: coalesced global reads, transposed shared writes.
template <int R>
__device__ __forceinline__ void stage_rows(float *xs, const float *__restrict__ x, int64_t row0, int nrows, int n_inputs,
                                           int lt, int threads_per_group, bool vec_ok) {
    if (vec_ok) {
        const int n4 = n_inputs >> 2;
        auto four_inputs = [&](int i4) {
            float v[R][4];
#pragma unroll
            for (int r = 0; r < R; r++) {
                float4 q = make_float4(0.f, 0.f, 0.f, 0.f);
                if (r < nrows) q = __ldcs(reinterpret_cast<const float4 *>(x + (row0 + r) * n_inputs) + i4);
                v[r][0] = q.x; v[r][1] = q.y; v[r][2] = q.z; v[r][3] = q.w;
            }
#pragma unroll
            for (int j = 0; j < 4; j++) {
                float *dst = xs + (size_t)(4 * i4 + j) * R;
                if constexpr (R % 4 == 0) {
#pragma unroll
                    for (int r4 = 0; r4 < R / 4; r4++)
                        reinterpret_cast<float4 *>(xs)[swizzle_slot((4 * i4 + j) * (R / 4) + r4)] =
                            make_float4(v[4 * r4][j], v[4 * r4 + 1][j], v[4 * r4 + 2][j], v[4 * r4 + 3][j]);
                } else {
#pragma unroll
                    for (int r = 0; r < R; r++) dst[r] = v[r][j];
                }
            }
        };
        if constexpr (R == 4) {   // (eight loads in flight, as with eight rows; the other counts are as fast as they come)
#pragma unroll 2
            for (int i4 = lt; i4 < n4; i4 += threads_per_group) four_inputs(i4);
        } else {
            for (int i4 = lt; i4 < n4; i4 += threads_per_group) four_inputs(i4);
        }
    } else {
        for (int i = lt; i < n_inputs; i += threads_per_group) {
#pragma unroll
            for (int r = 0; r < R; r++) {
                const float v = (r < nrows) ? __ldcs(x + (row0 + r) * n_inputs + i) : 0.f;
                if constexpr (R % 4 == 0) xs[swizzle_slot(i * (R / 4) + (r >> 2)) * 4 + (r & 3)] = v;
                else xs[(size_t)i * R + r] = v;
            }
        }
    }
}

// One word of a plan: the swizzled 16-byte slots of the two inputs (of the first four rows; the other four's differ in the lowest
// bit) in the order in which they are read, the anchor's bit, and whether that order is the reverse of the anchor's.  (14 bits a slot
// hold 8192 inputs; eight rows of more than 7232 do not fit shared memory, so that lists are made up to there, see two_lanes().)
constexpr int kPlanInputs = 8192, kPlanAnchors = 8;
__device__ __forceinline__ uint32_t plan_word(int first, int second, int k, int swapped) {
    return (uint32_t)swizzle_slot(2 * first) | (uint32_t)swizzle_slot(2 * second) << 14 | (uint32_t)k << 28 | (uint32_t)swapped << 31;
}

// Orders the anchors of four detectors at a time (those that share a wavefront in check_detectors_kernel<8, 2>): step by step
// each detector in turn takes the anchor, either way round, that makes the step's two reads the shortest.  A warp per four
// detectors, a lane per (anchor, way round); an input's banks are its pair of 16-byte slots after the swizzle.
// plan: [detector][kPlanAnchors].
__global__ void __launch_bounds__(128) anchor_plan_kernel(const int2 *__restrict__ anchors, int n_detectors, int n_anchors, uint32_t *__restrict__ plan) {
    const int lane = threadIdx.x & 31, i = lane >> 1, swapped = lane & 1;
    const int t0 = (blockIdx.x * 4 + (threadIdx.x >> 5)) * 4;
    if (t0 >= n_detectors) return;
    uint32_t word[4], left[4];
    int first[4], second[4];   // bank groups
    auto banks = [](int p) { return (p & 3) ^ ((p >> 3) & 3); };
#pragma unroll
    for (int d = 0; d < 4; d++) {
        int2 a = make_int2(0, 0);   // (an unused anchor compares an input with itself)
        if (i < n_anchors && t0 + d < n_detectors) a = __ldg(anchors + (size_t)(t0 + d) * n_anchors + i);
        if (a.x == kNoAnchor || a.y == kNoAnchor) a = make_int2(0, 0);
        if (swapped) a = make_int2(a.y, a.x);
        word[d] = plan_word(a.x, a.y, i, swapped);
        first[d] = banks(a.x);
        second[d] = banks(a.y);
        left[d] = (1u << n_anchors) - 1u;
    }
    for (int s = 0; s < n_anchors; s++) {
        uint32_t count_a = 0u, count_b = 0u;   // reads of each bank group in this step, a byte each
        int most_a = 0, most_b = 0;
#pragma unroll
        for (int d = 0; d < 4; d++) {
            const int a = max(most_a, (int)((count_a >> (8 * first[d])) & 255u) + 1), b = max(most_b, (int)((count_b >> (8 * second[d])) & 255u) + 1);
            const bool open = i < n_anchors && ((left[d] >> i) & 1u);
            const uint32_t best = __reduce_min_sync(0xffffffffu, open ? (uint32_t)(a + b) << 5 | (uint32_t)lane : 0xffffffffu);
            const int from = (int)(best & 31u);
            most_a = __shfl_sync(0xffffffffu, a, from);
            most_b = __shfl_sync(0xffffffffu, b, from);
            count_a += 1u << (8 * __shfl_sync(0xffffffffu, first[d], from));
            count_b += 1u << (8 * __shfl_sync(0xffffffffu, second[d], from));
            left[d] &= ~(1u << (from >> 1));
            if (lane == from && t0 + d < n_detectors) plan[(size_t)(t0 + d) * kPlanAnchors + s] = word[d];
        }
    }
}

// Work items: (row tile of GROUPS * R rows, chunk of threads_per_group / D detectors), row tile major.  Block b takes the
// items [n * b / grid, n * (b + 1) / grid): with a grid of one block per row tile that is the tile's own chunks; small
// batches launch a multiple of the SM count instead and a block's range may cross into the next tile, which it then
// stages as well.  (Splitting the detectors into a fixed number of slices per tile left 320 blocks on 148 SMs: the SMs
// with three blocks set the kernel's time, max / avg active cycles 1.3.)
//
// Bound by the wavefronts of the load/store unit where anchors are many: their inputs are random, so the 8 lanes that share a
// wavefront of 16-byte reads fall into the same banks 2.65 times over, and an anchor list read 8 bytes at a time touches 16
// lines per load.  D = 2: of 8 rows, two neighbouring lanes share a detector (4 rows each): a wavefront then holds 4 random
// 32-byte pieces, which collide 2.1 times; lists are read two anchors at a time.  Where anchors are few the stores count instead
// (D = 2 writes 64-byte pieces) and blocks of 256 threads overlap staging better; two_lanes() draws the line.
//
// PLAN (evaluation only): the anchors come from a list of one word each that anchor_plan_kernel has put in an order in which the
// four detectors of a wavefront collide less (1.5 times instead of 2.1 with random anchors), four anchors a load instead of
// two, and with the addresses worked out.  The order of the comparisons does not matter to the indices.  EPS: there is a dead band;
// without one the sign bit of minus the difference, which is never -0, is the answer.  16384 rows x 4096 inputs, 4096 detectors of 8 anchors:
// 445 -> 319 us (list and collisions 445 -> 367, addresses and signs 367 -> 319).
template <int R, int D, bool TRAIN, bool PLAN, bool EPS = true>
__global__ void __launch_bounds__(D == 2 ? 1024 : 256) check_detectors_kernel(const float *__restrict__ x, int64_t rows, int n_inputs,
                                                             const int2 *__restrict__ anchors, int n_detectors,
                                                             int n_anchors, float cmp_eps, int threads_per_group,
                                                             int32_t *__restrict__ idx,
                                                             float *__restrict__ min_delta,
                                                             int32_t *__restrict__ min_k,
                                                             uint8_t *__restrict__ packed, size_t packed_pitch,
                                                             const uint4 *__restrict__ plan) {
    static_assert(!PLAN || (R == 8 && D == 2 && !TRAIN), "plans are made for eight rows and two lanes");
    extern __shared__ __align__(16) float xs_all[];
    constexpr int RT = R / D;   // rows of a thread (D threads per detector)
    const int groups = blockDim.x / threads_per_group;
    const int g = threadIdx.x / threads_per_group;
    const int lt = threadIdx.x - g * threads_per_group;
    const int half = lt % D, per_chunk = threads_per_group / D;
    float *xs = xs_all + (size_t)g * staged_floats<R>(n_inputs);
    const bool vec_ok = (n_inputs % 4 == 0) && ((reinterpret_cast<uintptr_t>(x) & 15) == 0);
    const bool pairs_ok = (n_anchors % 2 == 0) && ((reinterpret_cast<uintptr_t>(anchors) & 15) == 0);
    const int chunks = (n_detectors + per_chunk - 1) / per_chunk;
    const int64_t rows_per_tile = (int64_t)groups * R;
    const int64_t n_items = ((rows + rows_per_tile - 1) / rows_per_tile) * chunks;
    const int64_t item0 = n_items * blockIdx.x / gridDim.x, item1 = n_items * (blockIdx.x + 1) / gridDim.x;
    int64_t staged = -1;
    for (int64_t item = item0; item < item1; ++item) {
        const int64_t tile = item / chunks;
        const int chunk = (int)(item - tile * chunks);
        const int64_t row0 = (tile * groups + g) * R;
        const int nrows = (int)min((int64_t)R, max((int64_t)0, rows - row0));
        if (tile != staged) {
            if (staged >= 0) __syncthreads();   // everyone is done reading the previous tile
            stage_rows<R>(xs, x, row0, nrows, n_inputs, lt, threads_per_group, vec_ok);
            __syncthreads();
            staged = tile;
        }
        const int t = chunk * per_chunk + lt / D;
        if (nrows <= 0 || t >= n_detectors) continue;
        int32_t li[RT];
        float md[RT];
        int32_t mk[RT];
#pragma unroll
        for (int r = 0; r < RT; r++) { li[r] = 0; md[r] = 0.f; mk[r] = -1; }
        auto one_anchor = [&](int k, int px, int py) {
            if (px == kNoAnchor || py == kNoAnchor) return;
            float a[RT], b[RT];
            if constexpr (R % 4 == 0) {
#pragma unroll
                for (int r4 = 0; r4 < RT / 4; r4++) {
                    const float4 qa = reinterpret_cast<const float4 *>(xs)[swizzle_slot(px * (R / 4) + half * (RT / 4) + r4)];
                    const float4 qb = reinterpret_cast<const float4 *>(xs)[swizzle_slot(py * (R / 4) + half * (RT / 4) + r4)];
                    a[4 * r4] = qa.x; a[4 * r4 + 1] = qa.y; a[4 * r4 + 2] = qa.z; a[4 * r4 + 3] = qa.w;
                    b[4 * r4] = qb.x; b[4 * r4 + 1] = qb.y; b[4 * r4 + 2] = qb.z; b[4 * r4 + 3] = qb.w;
                }
            } else {
#pragma unroll
                for (int r = 0; r < RT; r++) { a[r] = xs[(size_t)px * R + r]; b[r] = xs[(size_t)py * R + r]; }
            }
#pragma unroll
            for (int r = 0; r < RT; r++) {
                const float d = __fsub_rn(a[r], b[r]);
                if (greater_than_zero(d, cmp_eps)) li[r] |= (1 << k);
                if (TRAIN) {
                    if (mk[r] == -1 || fabsf(d) < fabsf(md[r])) { md[r] = d; mk[r] = k; }
                }
            }
        };
        const int2 *ap = anchors + (size_t)t * n_anchors;
        if constexpr (PLAN) {
            const char *rows4 = reinterpret_cast<const char *>(xs);
            const uint32_t which = (uint32_t)half << 4;
#pragma unroll
            for (int half_list = 0; half_list < 2; half_list++) {
                if (4 * half_list >= n_anchors) break;
                const uint4 q = __ldg(plan + 2 * t + half_list);
                const uint32_t e4[4] = {q.x, q.y, q.z, q.w};
#pragma unroll
                for (int n = 0; n < 4; n++) {
                    if (4 * half_list + n >= n_anchors) break;
                    const uint32_t e = e4[n];
                    const float4 a = *reinterpret_cast<const float4 *>(rows4 + (((e << 4) & 0x3fff0u) ^ which));
                    const float4 b = *reinterpret_cast<const float4 *>(rows4 + (((e >> 10) & 0x3fff0u) ^ which));
                    const uint32_t bit = 1u << ((e >> 28) & 7u);
                    // minus the anchor's difference: second input less first, or the reverse where they are swapped (one rounding, as
                    // a subtraction; a sum that is not a number has a clear sign bit).  The zero turns -0 into +0, so that a
                    // difference of two zeros is +0 whatever their signs.
                    const float f = __uint_as_float((e & 0x80000000u) | 0x3f800000u);
                    const float d[4] = {__fmaf_rn(-f, a.x, __fmaf_rn(f, b.x, 0.f)), __fmaf_rn(-f, a.y, __fmaf_rn(f, b.y, 0.f)),
                                        __fmaf_rn(-f, a.z, __fmaf_rn(f, b.z, 0.f)), __fmaf_rn(-f, a.w, __fmaf_rn(f, b.w, 0.f))};
#pragma unroll
                    for (int r = 0; r < 4; r++) {
                        if constexpr (EPS) {
                            if (greater_than_zero(-d[r], cmp_eps)) li[r] |= bit;
                        } else {
                            li[r] |= (uint32_t)((int32_t)__float_as_uint(d[r]) >> 31) & bit;
                        }
                    }
                }
            }
        } else if (pairs_ok) {
#pragma unroll 2
            for (int k = 0; k < n_anchors; k += 2) {
                const int4 p = __ldg(reinterpret_cast<const int4 *>(ap + k));
                one_anchor(k, p.x, p.y);
                one_anchor(k + 1, p.z, p.w);
            }
        } else {
#pragma unroll 4
            for (int k = 0; k < n_anchors; k++) {
                const int2 p = __ldg(ap + k);
                one_anchor(k, p.x, p.y);
            }
        }
#pragma unroll
        for (int r = 0; r < RT; r++) {
            const int row = half * RT + r;
            if (row < nrows) {
                const int64_t o = (row0 + row) * n_detectors + t;
                idx[o] = li[r];
                if (TRAIN) { min_delta[o] = md[r]; min_k[o] = mk[r]; }
            }
        }
        if (!TRAIN && packed != nullptr) {
            // (the bytes of rows past the end lie in the row's padding)
            uint8_t *dst = packed + (size_t)t * packed_pitch + row0 + half * RT;
            if constexpr (RT % 4 == 0) {
                uint32_t four[RT / 4];
#pragma unroll
                for (int r = 0; r < RT; r += 4)
                    four[r / 4] = (uint32_t)li[r] | (uint32_t)li[r + 1] << 8 | (uint32_t)li[r + 2] << 16 | (uint32_t)li[r + 3] << 24;
                if constexpr (RT == 8) *reinterpret_cast<uint2 *>(dst) = make_uint2(four[0], four[1]);
                else *reinterpret_cast<uint32_t *>(dst) = four[0];
            } else {
#pragma unroll
                for (int r = 0; r < RT; r++) dst[r] = (uint8_t)li[r];
            }
        }
    }
}

// Fallback for input rows that do not fit in shared memory: gathers straight from global memory.
template <bool TRAIN>
__global__ void check_detectors_global_kernel(const float *__restrict__ x, int64_t rows, int n_inputs,
                                              const int2 *__restrict__ anchors, int n_detectors, int n_anchors,
                                              float cmp_eps, int32_t *__restrict__ idx, float *__restrict__ min_delta,
                                              int32_t *__restrict__ min_k, uint8_t *__restrict__ packed, size_t packed_pitch) {
    const int64_t total = rows * n_detectors;
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < total; i += (int64_t)gridDim.x * blockDim.x) {
        const int64_t r = i / n_detectors;
        const int t = (int)(i - r * n_detectors);
        const float *xr = x + r * n_inputs;
        int32_t li = 0, mk = -1;
        float md = 0.f;
        for (int k = 0; k < n_anchors; k++) {
            const int2 p = __ldg(anchors + (size_t)t * n_anchors + k);
            if (p.x == kNoAnchor || p.y == kNoAnchor) continue;
            const float d = __fsub_rn(__ldg(xr + p.x), __ldg(xr + p.y));
            if (greater_than_zero(d, cmp_eps)) li |= (1 << k);
            if (TRAIN) {
                if (mk == -1 || fabsf(d) < fabsf(md)) { md = d; mk = k; }
            }
        }
        idx[i] = li;
        if (TRAIN) { min_delta[i] = md; min_k[i] = mk; }
        else if (packed != nullptr) packed[(size_t)t * packed_pitch + r] = (uint8_t)li;
    }
}

template <int R, int D>
static int launch_check_detectors_r(const float *x, int64_t rows, int n_inputs, const int32_t *anchors,
                                    int n_detectors, int n_anchors, float cmp_eps, int32_t *idx, float *min_delta,
                                    int32_t *min_k, int tpg, int groups, int64_t blocks, cudaStream_t stream,
                                    uint8_t *packed, size_t packed_pitch, uint32_t *plan = nullptr) {
    const size_t smem = (size_t)groups * staged_floats<R>(n_inputs) * sizeof(float);
    LUTB_REQUIRE(blocks <= 0x7FFFFFFF, LUTB_ERR_SHAPE, "batch too large for one launch");
    const bool train = min_delta != nullptr;
    auto kern = train ? check_detectors_kernel<R, D, true, false, true> : check_detectors_kernel<R, D, false, false, true>;
    if constexpr (R == 8 && D == 2) {
        if (plan != nullptr && !train) {
            KernelScope scope(K_CHECK_DETECTORS, stream);
            anchor_plan_kernel<<<(unsigned)((n_detectors + 15) / 16), 128, 0, stream>>>(reinterpret_cast<const int2 *>(anchors), n_detectors, n_anchors, plan);
            LUTB_LAUNCH_CHECK();
            kern = cmp_eps == 0.f ? check_detectors_kernel<8, 2, false, true, false> : check_detectors_kernel<8, 2, false, true, true>;
        }
    }
    if (smem > kPlainSmem) LUTB_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    KernelScope scope(K_CHECK_DETECTORS, stream);
    kern<<<(unsigned)blocks, tpg * groups, smem, stream>>>(x, rows, n_inputs, reinterpret_cast<const int2 *>(anchors),
                                                          n_detectors, n_anchors, cmp_eps, tpg, idx, min_delta, min_k, packed, packed_pitch,
                                                          reinterpret_cast<const uint4 *>(plan));
    LUTB_LAUNCH_CHECK();
    return LUTB_OK;
}

constexpr size_t kCheckBudget = 100 * 1024;   // staged rows of a block: two resident blocks per SM

// Whether two lanes share a detector (8 rows a group).  Measured over 8 to 32768 rows, 32 to 6000 inputs, 16 to 4096
// detectors, 2 to 13 anchors, training and evaluation; figures in us, two lanes / one lane a detector:
//  - rows that leave room for one block of 1024 threads (the other side: 4 rows): many anchors and detectors, and row tiles for
//    most of the SMs: 4096 rows x 4096 inputs, 4096 detectors of 8 anchors 0.78 of the time; 8192 x 4000, 16 detectors 291 / 109,
//    1000 detectors of 2 anchors 60 / 56, 64 rows, 1000 of 8 10.4 / 6.3; 100 x 6000, 4096 of 8 10.8 / 15.0; 20000 x 7000, 500 of 8 0.8
//  - few detectors: one lane each leaves an SM short of threads, the sooner the more shared memory their rows take: 32768 x 784,
//    64 detectors 0.87, 32768 x 3000, 64 detectors 0.6, 128 detectors 0.74; 100000 x 32, 64 detectors of 4 47 / 39
//  - long rows: 32768 x 3000, 256 detectors of 6 0.9; x 1500 to 2048 0.93 to 0.97, of 2 anchors in evaluation 1.1
//  - a few row tiles per SM, which are all there is to fill it: 4096 x 300, 1024 detectors of 7 29 / 39; 32768 rows 1.1 to 1.2
//  - indices that also leave as bytes (`packed`: 8 or 4 bytes a thread, `pitch` apart): 4096 x 512, 2048 detectors of 4 38 / 48
//  - many anchors and detectors: 32768 x 784, 768 detectors of 8 anchors 0.95; 100000 x 32, 300 of 3 222 / 149
static bool two_lanes(int64_t rows, int n_inputs, int n_detectors, int n_anchors, bool packed) {
    const size_t staged = staged_bytes(8, n_inputs);
    const int64_t tiles = (rows + 7) / 8;
    const int sm = device_info().sm_count;
    if (rows < 8 || staged > (size_t)kMaxSmemPerBlock - 1024) return false;
    if (staged > kCheckBudget) {
        const int64_t items = tiles * ((n_detectors + 511) / 512);
        if (n_anchors < 6) return false;
        if (staged_bytes(4, n_inputs) > kCheckBudget) return n_detectors >= 448 && items >= sm / 3;   // (the other side: 2 rows)
        return n_detectors >= 768 && items >= 2 * sm / 3 && (rows <= 16384 || n_detectors >= 2048 || n_anchors >= 8);
    }
    if (packed && tiles >= sm) return true;
    if (n_detectors <= 32) return staged < 22 * 1024;
    if (n_detectors <= 128 && staged >= 22 * 1024) return true;
    if (n_detectors <= 64 && rows <= 8192) return true;
    if (staged >= 80 * 1024) return n_detectors <= 192 || n_anchors >= 4;
    if (staged >= 44 * 1024) return n_anchors >= 6 && n_detectors >= 256;
    if (n_anchors >= 6 && n_detectors >= (n_anchors >= 10 ? 256 : 384) && tiles >= 2 * sm && tiles <= 5 * sm) return true;
    return n_anchors >= 8 && n_detectors >= 768 && staged >= 6 * 1024;
}

int launch_check_detectors(const float *x, int64_t rows, int n_inputs, const int32_t *anchors, int n_detectors,
                           int n_anchors, float cmp_eps, int32_t *idx, float *min_delta, int32_t *min_k,
                           cudaStream_t stream, uint8_t *packed, size_t packed_pitch, uint32_t *plan) {
    const int sm = device_info().sm_count;
    // rows per group: 8 while two blocks fit an SM (each anchor pair is fetched once per 8 rows), or one block of twice the threads
    // where that pays; fewer for few or longer rows
    const size_t row_bytes = (size_t)n_inputs * sizeof(float);
    const int D = two_lanes(rows, n_inputs, n_detectors, n_anchors, packed != nullptr) ? 2 : 1;
    int R = 8;
    while (R > 1 && (rows < R || (D == 1 && staged_bytes(R, n_inputs) > kCheckBudget))) R >>= 1;
    // threads per row group: D per detector, rounded to warps; at most 256 detectors, or 512 where the rows leave room for one block
    const int widest = D == 1 ? 256 : staged_bytes(R, n_inputs) > kCheckBudget ? 1024 : 512;
    int tpg = ((min(n_detectors * D, widest) + 31) / 32) * 32;
    if ((size_t)R * row_bytes > (size_t)kMaxSmemPerBlock - 1024) {
        const bool train = min_delta != nullptr;
        const int64_t total = rows * n_detectors;
        int64_t blocks = min((total + 255) / 256, (int64_t)sm * 32);
        KernelScope scope(K_CHECK_DETECTORS, stream);
        if (train)
            check_detectors_global_kernel<true><<<(unsigned)blocks, 256, 0, stream>>>(
                x, rows, n_inputs, reinterpret_cast<const int2 *>(anchors), n_detectors, n_anchors, cmp_eps, idx,
                min_delta, min_k, packed, packed_pitch);
        else
            check_detectors_global_kernel<false><<<(unsigned)blocks, 256, 0, stream>>>(
                x, rows, n_inputs, reinterpret_cast<const int2 *>(anchors), n_detectors, n_anchors, cmp_eps, idx,
                min_delta, min_k, packed, packed_pitch);
        LUTB_LAUNCH_CHECK();
        return LUTB_OK;
    }
    int groups = tpg >= 256 ? 1 : 256 / tpg;
    while (groups > 1 && ((size_t)groups * R * row_bytes > kCheckBudget || rows < (int64_t)groups * R * 2 * sm)) groups >>= 1;
    // one block per row tile; small batches: as many blocks as are resident (two per SM, one where the rows take more than
    // half of it), each with an equal share of the (tile, detector chunk) work items
    const int64_t resident = (int64_t)sm * (groups * staged_bytes(R, n_inputs) > kCheckBudget ? 1 : 2);
    const int64_t row_tiles = (rows + (int64_t)groups * R - 1) / ((int64_t)groups * R);
    const int64_t items = row_tiles * ((n_detectors + tpg / D - 1) / (tpg / D));
    const int64_t blocks = row_tiles >= resident ? row_tiles : min(items, resident);
    // the plan costs a launch of 3 us and pays from a row tile per SM on
    const bool planned = plan != nullptr && n_inputs <= kPlanInputs && n_anchors <= kPlanAnchors && row_tiles >= sm;
    switch (R) {
        case 8:
            if (D == 2) return launch_check_detectors_r<8, 2>(x, rows, n_inputs, anchors, n_detectors, n_anchors, cmp_eps, idx, min_delta, min_k, tpg, groups, blocks, stream, packed, packed_pitch, planned ? plan : nullptr);
            return launch_check_detectors_r<8, 1>(x, rows, n_inputs, anchors, n_detectors, n_anchors, cmp_eps, idx, min_delta, min_k, tpg, groups, blocks, stream, packed, packed_pitch);
        case 4: return launch_check_detectors_r<4, 1>(x, rows, n_inputs, anchors, n_detectors, n_anchors, cmp_eps, idx, min_delta, min_k, tpg, groups, blocks, stream, packed, packed_pitch);
        case 2: return launch_check_detectors_r<2, 1>(x, rows, n_inputs, anchors, n_detectors, n_anchors, cmp_eps, idx, min_delta, min_k, tpg, groups, blocks, stream, packed, packed_pitch);
        default: return launch_check_detectors_r<1, 1>(x, rows, n_inputs, anchors, n_detectors, n_anchors, cmp_eps, idx, min_delta, min_k, tpg, groups, blocks, stream, packed, packed_pitch);
    }
}

// --------------------------------------------------------------------------------------------
// Kernel 2: table-row gather and accumulate, y[b, :] += sum_t W[t, idx[b, t], :]
// (reference: fill_outputs_non_seq_fc_logic, proto:1214-1299).
//
// One warp per (sample, output chunk).  The warp is split into NG lane groups of LG lanes; a group
// owns every NG-th detector and its lanes cover the chunk's columns VEC floats at a time, so a row
// read is one coalesced 16*LG byte segment.  Table indices are fetched 32 at a time (coalesced)
// and broadcast with shuffles, so the row loads do not wait on a dependent index load.  Partial
// sums are fp32 inside a block of 32 detectors and double across blocks.
//
// Fixed-point mode reproduces the reference bit for bit: detectors are summed in double in order,
// in blocks of `det_block` (backward_group_size), each block sum is truncated to int32 and added.
// --------------------------------------------------------------------------------------------
constexpr int kFwdJ = 4;  // vectors per lane and chunk

template <int VEC>
struct Vec;
template <>
struct Vec<4> {
    using T = float4;
    static __device__ __forceinline__ void load(const float *p, float (&v)[4]) {
        const float4 q = __ldg(reinterpret_cast<const float4 *>(p));
        v[0] = q.x; v[1] = q.y; v[2] = q.z; v[3] = q.w;
    }
};
template <>
struct Vec<1> {
    using T = float;
    static __device__ __forceinline__ void load(const float *p, float (&v)[1]) { v[0] = __ldg(p); }
};

template <int VEC>
__global__ void __launch_bounds__(256) fc_gather_forward_fixed_kernel(const float *__restrict__ W, const int32_t *__restrict__ idx,
                                                                     float *__restrict__ y, int64_t batch, int n_outputs,
                                                                     int n_detectors, int table_rows, int t0, int t1,
                                                                     int det_block, int chunk, double fixed_scale) {
    constexpr int LG = 32;
    const int j = threadIdx.x & 31;
    const int64_t b = (int64_t)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
    if (b >= batch) return;
    const int c0 = blockIdx.y * chunk;
    const int clen = min(chunk, n_outputs - c0);
    const int32_t *idx_b = idx + b * n_detectors;
    const size_t row_stride = (size_t)n_outputs;

    int32_t iacc[kFwdJ][VEC];
#pragma unroll
    for (int q = 0; q < kFwdJ; q++)
#pragma unroll
        for (int e = 0; e < VEC; e++) iacc[q][e] = 0;
    for (int tb = t0; tb < t1; tb += det_block) {
        const int tend = min(tb + det_block, t1);
        double s[kFwdJ][VEC];
#pragma unroll
        for (int q = 0; q < kFwdJ; q++)
#pragma unroll
            for (int e = 0; e < VEC; e++) s[q][e] = 0.0;
        for (int t = tb; t < tend; t++) {
            const int32_t li = __ldg(idx_b + t);
            const float *row = W + ((size_t)t * table_rows + li) * row_stride + c0;
#pragma unroll
            for (int q = 0; q < kFwdJ; q++) {
                const int col = (j + q * LG) * VEC;
                if (col < clen) {
                    float v[VEC];
                    Vec<VEC>::load(row + col, v);
#pragma unroll
                    for (int e = 0; e < VEC; e++) s[q][e] += (double)v[e];
                }
            }
        }
#pragma unroll
        for (int q = 0; q < kFwdJ; q++)
#pragma unroll
            for (int e = 0; e < VEC; e++) iacc[q][e] += to_fixed(s[q][e], fixed_scale);
    }
    int32_t *yb = reinterpret_cast<int32_t *>(y) + b * n_outputs + c0;
#pragma unroll
    for (int q = 0; q < kFwdJ; q++) {
        const int col = (j + q * LG) * VEC;
        if (col < clen) {
#pragma unroll
            for (int e = 0; e < VEC; e++) yb[col + e] += iacc[q][e];
        }
    }
}

// Forward gather for fp32 accumulators and 16-byte aligned rows: one warp per (sample, chunk of LG float4 columns); the row
// loads of up to 16 detectors per lane are all issued before the first one is consumed, which is what hides the latency of the
// (random) row reads.
// Blocks an SM named for the groups of 4, 16 and 32 lanes: without it the compiler does not issue all row loads first (20000 samples, 50
// detectors x 64 outputs 30 -> 19 us, x 16 11.5 -> 10.1; 16384 samples, 32 detectors x 128 outputs 17.8 -> 15.9; 256 samples, 64 detectors x 64 outputs
// 7.6 -> 3.9; four or six instead of five are within 5 % there); the others are best left alone (65536 samples, 64 detectors x 32 outputs 41.3
// against 42.2 to 46.8).
template <int LG>
__global__ void __launch_bounds__(256, LG == 4 || LG >= 16 ? 5 : 0) fc_gather_forward_vec_kernel(const float *__restrict__ W,
                                                                   const int32_t *__restrict__ idx,
                                                                   float *__restrict__ y, int64_t batch, int n_outputs,
                                                                   int n_detectors, int table_rows, int t0, int t1) {
    constexpr int NG = 32 / LG;
    constexpr int IT = 32 / NG;                  // row loads per lane and 32 detectors
    constexpr int BATCH = IT > 16 ? 16 : IT;     // loads in flight per lane
    const int lane = threadIdx.x & 31;
    const int64_t b = (int64_t)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
    if (b >= batch) return;
    const int g = lane / LG, j = lane - g * LG;
    const int col = (blockIdx.y * LG + j) * 4;
    const bool active = col < n_outputs;
    const int32_t *idx_b = idx + b * n_detectors;
    // addresses: this lane's columns of a table, tables NG apart, plus 32-bit row numbers times the row's bytes (a 64-bit product per
    // row less: 65536 samples, 64 detectors of 64 rows x 32 outputs 46.8 -> 42.9 us; 8192 samples, 16 detectors, 256 outputs 17.3 -> 14.8)
    const char *table = reinterpret_cast<const char *>(W + ((size_t)(t0 + g) * table_rows) * n_outputs + col);
    const size_t group_bytes = (size_t)NG * table_rows * n_outputs * 4;
    const uint32_t row_bytes = (uint32_t)n_outputs * 4u;
    double acc[4] = {0.0, 0.0, 0.0, 0.0};
    for (int tb = t0; tb < t1; tb += 32) {
        const int nvalid = min(32, t1 - tb);
        const int32_t mine = (lane < nvalid) ? __ldg(idx_b + tb + lane) : 0;
        float part[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
        for (int i0 = 0; i0 < IT; i0 += BATCH) {
            float4 w[BATCH];
#pragma unroll
            for (int i = 0; i < BATCH; i++) {
                const int d = (i0 + i) * NG + g;
                const int32_t li = __shfl_sync(0xffffffffu, mine, d);
                w[i] = (active && d < nvalid) ? __ldg(reinterpret_cast<const float4 *>(table + (uint64_t)(uint32_t)li * row_bytes))
                                              : make_float4(0.f, 0.f, 0.f, 0.f);
                table += group_bytes;
            }
#pragma unroll
            for (int i = 0; i < BATCH; i++) { part[0] += w[i].x; part[1] += w[i].y; part[2] += w[i].z; part[3] += w[i].w; }
        }
#pragma unroll
        for (int e = 0; e < 4; e++) acc[e] += (double)part[e];
    }
#pragma unroll
    for (int m = LG; m < 32; m <<= 1) {
#pragma unroll
        for (int e = 0; e < 4; e++) acc[e] += __shfl_xor_sync(0xffffffffu, acc[e], m);
    }
    if (active && g == 0) {
        float4 *out = reinterpret_cast<float4 *>(y + b * n_outputs + col);
        float4 cur = *out;
        cur.x += (float)acc[0]; cur.y += (float)acc[1]; cur.z += (float)acc[2]; cur.w += (float)acc[3];
        *out = cur;
    }
}

// The same for rows that are not 16-byte aligned: chunks of LG * J columns, J columns a lane (LG apart), the row loads of up to
// 16 / J detectors in flight.  J = 2 where a row is a little wider than a warp, J = 4 for wide rows (a chunk per 32 columns reads
// the indices again for each of them).  (One template for both kernels cost the aligned rows 5 %: 60000 samples, 40 detectors,
// 256 outputs 223 -> 235 us.)
// Measured (a loop with a load per detector and lane in flight before): 1111 samples, 50 detectors, 33 outputs 18.4 -> 6.3 us;
// 512 samples, 64 detectors, 10 outputs 17.7 -> 5.7 us.  J = 1 / 4, with the index comparison: 8192 samples, 16 detectors, 129
// outputs 29 / 21, 1001 outputs 132 / 56; 60000 x 40, 65 outputs 227 / 106; few warps (32 samples, 65 outputs) 10.5 / 12.6.
template <int LG, int J>
__global__ void __launch_bounds__(256) fc_gather_forward_scalar_kernel(const float *__restrict__ W,
                                                                      const int32_t *__restrict__ idx,
                                                                      float *__restrict__ y, int64_t batch, int n_outputs,
                                                                      int n_detectors, int table_rows, int t0, int t1) {
    constexpr int NG = 32 / LG;
    constexpr int IT = 32 / NG;                          // row loads per lane and 32 detectors
    constexpr int BATCH = IT > 16 / J ? 16 / J : IT;     // detectors in flight per lane
    const int lane = threadIdx.x & 31;
    const int64_t b = (int64_t)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
    if (b >= batch) return;
    const int g = lane / LG, j = lane - g * LG;
    const int col = blockIdx.y * (LG * J) + j;   // further columns of the lane LG apart
    bool active[J];
#pragma unroll
    for (int q = 0; q < J; q++) active[q] = col + q * LG < n_outputs;
    const int32_t *idx_b = idx + b * n_detectors;
    const float *Wc = W + col;
    double acc[J];
#pragma unroll
    for (int q = 0; q < J; q++) acc[q] = 0.0;
    for (int tb = t0; tb < t1; tb += 32) {
        const int nvalid = min(32, t1 - tb);
        const int32_t mine = (lane < nvalid) ? __ldg(idx_b + tb + lane) : 0;
        float part[J];
#pragma unroll
        for (int q = 0; q < J; q++) part[q] = 0.f;
#pragma unroll
        for (int i0 = 0; i0 < IT; i0 += BATCH) {
            if (J > 1 && i0 * NG >= nvalid) break;   // (warp uniform; J = 1 keeps the next batch's loads ahead of this one's sums)
            float w[BATCH][J];
#pragma unroll
            for (int i = 0; i < BATCH; i++) {
                const int d = (i0 + i) * NG + g;
                const int32_t li = __shfl_sync(0xffffffffu, mine, d);
#pragma unroll
                for (int q = 0; q < J; q++)
                    w[i][q] = (active[q] && d < nvalid) ? __ldg(Wc + ((size_t)(tb + d) * table_rows + li) * n_outputs + q * LG) : 0.f;
            }
#pragma unroll
            for (int i = 0; i < BATCH; i++)
#pragma unroll
                for (int q = 0; q < J; q++) part[q] += w[i][q];
        }
#pragma unroll
        for (int q = 0; q < J; q++) acc[q] += (double)part[q];
    }
#pragma unroll
    for (int m = LG; m < 32; m <<= 1) {
#pragma unroll
        for (int q = 0; q < J; q++) acc[q] += __shfl_xor_sync(0xffffffffu, acc[q], m);
    }
    if (g != 0) return;
#pragma unroll
    for (int q = 0; q < J; q++)
        if (active[q]) y[b * n_outputs + col + q * LG] += (float)acc[q];
}

static int pow2_ceil(int v) {
    int p = 1;
    while (p < v) p <<= 1;
    return p;
}

int launch_fc_gather_forward(const float *W, const int32_t *idx, float *y, int64_t batch, int n_outputs,
                             int n_detectors, int table_rows, int det_block, bool int_mode, double fixed_scale,
                             cudaStream_t stream) {
    const bool vec4 = (n_outputs % 4 == 0) && ((reinterpret_cast<uintptr_t>(W) & 15) == 0) &&
                      ((reinterpret_cast<uintptr_t>(y) & 15) == 0);
    const int vec = vec4 ? 4 : 1;
    const int vpr = (n_outputs + vec - 1) / vec;  // vectors per row
    const int lanes = int_mode ? 32 : min(32, pow2_ceil(vpr));
    const int chunk = min(n_outputs, lanes * kFwdJ * vec);
    const int n_chunks = (n_outputs + chunk - 1) / chunk;
    const int warps = 8;
    const int64_t blocks = (batch + warps - 1) / warps;
    LUTB_REQUIRE(blocks <= 0x7FFFFFFF && n_chunks <= 65535, LUTB_ERR_SHAPE, "grid too large");
    // Detector ranges are sized so that one range's tables stay resident in L2 while the whole batch
    // streams through them; fixed-point blocks must not straddle a range.
    const size_t table_bytes = (size_t)table_rows * n_outputs * sizeof(float);
    int64_t per_range = (int64_t)((size_t)(48u << 20) / (table_bytes ? table_bytes : 1));
    const int align = int_mode ? det_block : 32;
    per_range = max((int64_t)align, per_range / align * align);
    dim3 grid((unsigned)blocks, (unsigned)n_chunks);
    for (int64_t t0 = 0; t0 < n_detectors; t0 += per_range) {
        const int t1 = (int)min((int64_t)n_detectors, t0 + per_range);
        KernelScope scope(K_FC_GATHER_FORWARD, stream);
        if (!int_mode) {
            // columns of a lane: two where one pass of the warp leaves a remainder (scalar rows of 33 to 64 outputs), four for
            // wider scalar rows once that gives every SM six warps (and where a grid has no room for a chunk per 32 columns)
            const bool wide = !vec4 && vpr > 64 && (batch * ((vpr + 127) / 128) >= 6 * (int64_t)device_info().sm_count || vpr > 65535 * 32);
            const int cols = wide ? 4 : !vec4 && vpr > 32 && vpr <= 64 ? 2 : 1;
            const dim3 vgrid((unsigned)blocks, (unsigned)((vpr + lanes * cols - 1) / (lanes * cols)));
            LUTB_REQUIRE(vgrid.y <= 65535, LUTB_ERR_SHAPE, "grid too large");
            auto launch = [&](auto kern) {
                kern<<<vgrid, warps * 32, 0, stream>>>(W, idx, y, batch, n_outputs, n_detectors, table_rows, (int)t0, t1);
            };
            if (vec4) {
                switch (lanes) {
                    case 32: launch(fc_gather_forward_vec_kernel<32>); break;
                    case 16: launch(fc_gather_forward_vec_kernel<16>); break;
                    case 8: launch(fc_gather_forward_vec_kernel<8>); break;
                    case 4: launch(fc_gather_forward_vec_kernel<4>); break;
                    case 2: launch(fc_gather_forward_vec_kernel<2>); break;
                    default: launch(fc_gather_forward_vec_kernel<1>); break;
                }
            } else if (cols == 4) {
                launch(fc_gather_forward_scalar_kernel<32, 4>);
            } else if (cols == 2) {
                launch(fc_gather_forward_scalar_kernel<32, 2>);
            } else {
                switch (lanes) {
                    case 32: launch(fc_gather_forward_scalar_kernel<32, 1>); break;
                    case 16: launch(fc_gather_forward_scalar_kernel<16, 1>); break;
                    case 8: launch(fc_gather_forward_scalar_kernel<8, 1>); break;
                    case 4: launch(fc_gather_forward_scalar_kernel<4, 1>); break;
                    case 2: launch(fc_gather_forward_scalar_kernel<2, 1>); break;
                    default: launch(fc_gather_forward_scalar_kernel<1, 1>); break;
                }
            }
        } else if (vec4) {
            fc_gather_forward_fixed_kernel<4><<<grid, warps * 32, 0, stream>>>(W, idx, y, batch, n_outputs, n_detectors, table_rows, (int)t0, t1, det_block, chunk, fixed_scale);
        } else {
            fc_gather_forward_fixed_kernel<1><<<grid, warps * 32, 0, stream>>>(W, idx, y, batch, n_outputs, n_detectors, table_rows, (int)t0, t1, det_block, chunk, fixed_scale);
        }
        LUTB_LAUNCH_CHECK();
    }
    return LUTB_OK;
}

// --------------------------------------------------------------------------------------------
// Kernel 3: surrogate input gradient (reference: propagate_through_detectors_non_seq_fc_logic,
// proto:1421-1499).  Per (sample, detector): g = sum_o dY[o] * (W[t, j, o] - W[t, j ^ 2^k, o]),
// du = up(min_delta) * g, then +du / -du on the two inputs of the flipped anchor pair.
// A warp owns a sample; its lane groups of LG lanes read the two rows of a detector with coalesced vector loads, two or four
// detectors a group in flight, up to eight before they are reduced.  The products of one vector are summed in fp32 and added
// to a double per lane; the lanes of a group transpose-reduce their detectors' sums in double (one shuffle step per halving
// of the detectors instead of a full reduction each), so that every lane ends with one detector's dot product and the
// surrogate derivative (a double division) and the two reductions into dX run on 32 lanes.
// Bound: the latency of the row reads and load/store wavefronts (half of their peak at 65536 samples x 64 detectors of 64 rows x 32
// outputs).  Measured (one detector a group in flight, a full reduction per detector before), with the clearing of dX:
// 256 samples 10.9 -> 8.6 us; 1111 samples, 50 detectors, 33 outputs 32.0 -> 14.8 us; 512 samples, 64 detectors, 10 outputs
// 18.8 -> 8.7 us; 8192 samples, 16 detectors, 256 outputs 33.4 -> 28.5 us; 65536 samples 187 -> 167 us, and 109 as said at ONE below.
// (Walking groups of detectors whose tables fit L1 measured 220 us there: the groups leave lanes idle.)
// --------------------------------------------------------------------------------------------
// WRITE: dX is written instead of added to (and need not be cleared): the warp sums its sample's row in shared memory and
// writes it out once.
// Blocks an SM: rows of one step four, from 16 lanes a group on three (115 us with three for the layer of 65536 samples above, 109 with
// four, 5000 samples 12.8 and 13.2; 20000 samples, 50 detectors of 128 rows x 64 outputs 58 with two, 47 with three; 16384 samples x 128 outputs
// 44 and 38), others two (8192 samples x 256 outputs 28 with two, 34 with three: spills).
// ONE: rows of one step (n_outputs <= LG * VEC).  A lane then has one fp32 product sum per detector, which the first exchange
// takes as it is; lanes without a column and detectors without an anchor to flip read the first column and one row twice (nobody
// takes what comes out), so that the loads need no predicates and four detectors are in flight; addresses are row numbers times the
// row's bytes.  65536 samples 167 -> 109 us, 256 samples 7.4 -> 5.3.  (The same for rows of several steps spilled registers and
// gained nothing.)
template <int LG, int VEC, bool WRITE, bool ONE>
__global__ void __launch_bounds__(256, !ONE ? 2 : LG >= 16 ? 3 : 4) fc_input_grad_kernel(const float *__restrict__ W, const float *__restrict__ dY,
                                                           const int2 *__restrict__ anchors,
                                                           const int32_t *__restrict__ idx,
                                                           const float *__restrict__ min_delta,
                                                           const int32_t *__restrict__ min_k, float *__restrict__ dX,
                                                           int64_t batch, int n_inputs, int n_outputs, int n_detectors,
                                                           int n_anchors, int table_rows, int group_dets, int block_samples) {
    constexpr int NG = 32 / LG, CH = LG < 8 ? LG : 8, UM = LG >= 16 || ONE ? 4 : 2, U = CH < UM ? CH : UM;   // CH detectors a group at a time
    const int lane = threadIdx.x & 31, g = lane / LG, j = lane - g * LG;
    const int my_s = j * NG + g;   // this lane's detector of every 32: iteration i of group g takes detector i * NG + g
    const int t_begin = blockIdx.y * group_dets, t_end = min(n_detectors, t_begin + group_dets);
    const int64_t b_end = min(batch, ((int64_t)blockIdx.x + 1) * block_samples);
    extern __shared__ __align__(16) float dx_rows[];
    const uint32_t row_bytes = (uint32_t)n_outputs * 4u;
    const size_t table_bytes = (size_t)table_rows * row_bytes;
    const int row_floats = (n_inputs + 3) & ~3;
    float *dx_s = dx_rows + (threadIdx.x >> 5) * row_floats;
    if (WRITE) {
        for (int i = lane; i < row_floats; i += 32) dx_s[i] = 0.f;
        __syncwarp();
    }
    for (int64_t b = (int64_t)blockIdx.x * block_samples + (threadIdx.x >> 5); b < b_end; b += blockDim.x >> 5) {
        const float *dy = dY + b * n_outputs;
        float *dx = dX + b * n_inputs;
        const int64_t base = b * n_detectors;
        float d0[VEC];   // this lane's columns of dY where a row is one step
        if (j * VEC < n_outputs) Vec<VEC>::load(dy + j * VEC, d0);
        else {
#pragma unroll
            for (int e = 0; e < VEC; e++) d0[e] = 0.f;
        }
        for (int tb = t_begin; tb < t_end; tb += 32) {
            const int nvalid = min(32, t_end - tb);
            int32_t my_idx = 0, my_k = -1;
            float my_m = 0.f;
            if (my_s < nvalid) {
                my_idx = __ldg(idx + base + tb + my_s);
                my_k = __ldg(min_k + base + tb + my_s);
                my_m = __ldg(min_delta + base + tb + my_s);
            }
            double dot = 0.0;
            const int32_t own_row = my_k >= 0 ? my_idx : 0, own_alt = my_k >= 0 ? my_idx ^ (1 << my_k) : 0;
            const bool in_row = j * VEC < n_outputs;
            const char *tables = reinterpret_cast<const char *>(W + (size_t)tb * table_rows * n_outputs + (in_row ? j * VEC : 0));
#pragma unroll 1
            for (int ch = 0; ch < LG && ch * NG < nvalid; ch += CH) {
                using Part = std::conditional_t<ONE, float, double>;
                Part v[CH];
#pragma unroll
                for (int i0 = 0; i0 < CH; i0 += U) {
#pragma unroll
                    for (int u = 0; u < U; u++) v[i0 + u] = 0;
                    if ((ch + i0) * NG >= nvalid) continue;   // warp uniform
                    if constexpr (ONE) {
                        const char *row[U], *alt[U];
#pragma unroll
                        for (int u = 0; u < U; u++) {
                            const int i = ch + i0 + u, s = i * NG + g;
                            const uint32_t li = (uint32_t)__shfl_sync(0xffffffffu, own_row, g * LG + i);
                            const uint32_t la = (uint32_t)__shfl_sync(0xffffffffu, own_alt, g * LG + i);
                            const char *tab = tables + (size_t)(uint32_t)(s < nvalid ? s : 0) * table_bytes;
                            row[u] = tab + (uint64_t)li * row_bytes;
                            alt[u] = tab + (uint64_t)la * row_bytes;
                        }
                        float a[U][VEC], c[U][VEC];
#pragma unroll
                        for (int u = 0; u < U; u++) {
                            Vec<VEC>::load(reinterpret_cast<const float *>(row[u]), a[u]);
                            Vec<VEC>::load(reinterpret_cast<const float *>(alt[u]), c[u]);
                        }
#pragma unroll
                        for (int u = 0; u < U; u++) {
                            float part = 0.f;
#pragma unroll
                            for (int e = 0; e < VEC; e++) part = fmaf(d0[e], a[u][e] - c[u][e], part);
                            v[i0 + u] = in_row ? part : 0.f;
                        }
                        continue;
                    }
                    const float *row[U], *alt[U];
                    bool on[U];
#pragma unroll
                    for (int u = 0; u < U; u++) {
                        const int i = ch + i0 + u, s = i * NG + g;
                        const int32_t li = __shfl_sync(0xffffffffu, my_idx, g * LG + i);
                        const int32_t k = __shfl_sync(0xffffffffu, my_k, g * LG + i);
                        on[u] = s < nvalid && k >= 0;
                        const float *tab = W + (size_t)(tb + (on[u] ? s : 0)) * table_rows * n_outputs;
                        row[u] = tab + (size_t)li * n_outputs;
                        alt[u] = tab + (size_t)(on[u] ? li ^ (1 << k) : 0) * n_outputs;
                    }
                    for (int c0 = 0; c0 < n_outputs; c0 += LG * VEC) {
                        const int col = c0 + j * VEC;
                        float d[VEC], a[U][VEC], c[U][VEC];
                        if (c0 == 0) {
#pragma unroll
                            for (int e = 0; e < VEC; e++) d[e] = d0[e];
                        } else if (col < n_outputs) {
                            Vec<VEC>::load(dy + col, d);
                        }
#pragma unroll
                        for (int u = 0; u < U; u++) {
#pragma unroll
                            for (int e = 0; e < VEC; e++) a[u][e] = c[u][e] = 0.f;
                            if (on[u] && col < n_outputs) {
                                Vec<VEC>::load(row[u] + col, a[u]);
                                Vec<VEC>::load(alt[u] + col, c[u]);
                            }
                        }
                        if (col < n_outputs) {
#pragma unroll
                            for (int u = 0; u < U; u++) {
                                float part = 0.f;
#pragma unroll
                                for (int e = 0; e < VEC; e++) part = fmaf(d[e], a[u][e] - c[u][e], part);
                                v[i0 + u] += (double)part;
                            }
                        }
                    }
                }
                // lane j ends with the chunk's detector j % CH: halving steps over the detectors, then plain ones
                double w[CH];
#pragma unroll
                for (int i = 0; i < CH; i++) w[i] = (double)v[i];
                if constexpr (ONE && CH > 1) {   // (the first step exchanges the fp32 sums as they are)
                    const bool upper = (j & (CH / 2)) != 0;
#pragma unroll
                    for (int i = 0; i < CH / 2; i++) {
                        const Part send = upper ? v[i] : v[i + CH / 2], keep = upper ? v[i + CH / 2] : v[i];
                        w[i] = (double)keep + (double)__shfl_xor_sync(0xffffffffu, send, CH / 2);
                    }
                }
#pragma unroll
                for (int o = ONE ? CH / 4 : CH / 2; o >= 1; o >>= 1) {
                    const bool upper = (j & o) != 0;
#pragma unroll
                    for (int i = 0; i < o; i++) {
                        const double send = upper ? w[i] : w[i + o];
                        const double keep = upper ? w[i + o] : w[i];
                        w[i] = keep + __shfl_xor_sync(0xffffffffu, send, o);
                    }
                }
#pragma unroll
                for (int o = CH; o < LG; o <<= 1) w[0] += __shfl_xor_sync(0xffffffffu, w[0], o);
                if (j / CH == ch / CH) dot = w[0];
            }
            if (my_s < nvalid && my_k >= 0) {
                const double du = surrogate_up(my_m) * dot;
                if (fabs(du) > kEps) {
                    const int2 p = __ldg(anchors + (size_t)(tb + my_s) * n_anchors + my_k);
                    float *cells = WRITE ? dx_s : dx;
                    atomicAdd(cells + p.x, (float)du);
                    atomicAdd(cells + p.y, -(float)du);
                }
            }
        }
        if (WRITE) {
            __syncwarp();
            if (row_floats == n_inputs && (reinterpret_cast<uintptr_t>(dX) & 15) == 0) {
                for (int i = lane * 4; i < n_inputs; i += 128) {
                    __stcs(reinterpret_cast<float4 *>(dx + i), *reinterpret_cast<const float4 *>(dx_s + i));
                    *reinterpret_cast<float4 *>(dx_s + i) = make_float4(0.f, 0.f, 0.f, 0.f);
                }
            } else {
                for (int i = lane; i < n_inputs; i += 32) {
                    dx[i] = dx_s[i];
                    dx_s[i] = 0.f;
                }
            }
            __syncwarp();
        }
    }
}

// Fixed-point variant: one thread per (sample, detector), outputs walked in order in blocks of
// `out_block` (forward_group_size); each block's du is truncated to int32 on its own, exactly as
// the reference does, and added with integer atomics (order independent).
__global__ void fc_input_grad_fixed_kernel(const float *__restrict__ W, const float *__restrict__ dY,
                                           const int2 *__restrict__ anchors, const int32_t *__restrict__ idx,
                                           const float *__restrict__ min_delta, const int32_t *__restrict__ min_k,
                                           float *__restrict__ dX, int64_t batch, int n_inputs, int n_outputs,
                                           int n_detectors, int n_anchors, int table_rows, int out_block,
                                           double fixed_scale) {
    const int64_t total = batch * n_detectors;
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < total; i += (int64_t)gridDim.x * blockDim.x) {
        const int64_t b = i / n_detectors;
        const int t = (int)(i - b * n_detectors);
        const int32_t li = idx[i];
        const int32_t k = min_k[i];
        const double up = surrogate_up(min_delta[i]);
        const float *row = W + ((size_t)t * table_rows + li) * n_outputs;
        const float *alt = W + ((size_t)t * table_rows + (li ^ (1 << k))) * n_outputs;
        const float *dy = dY + b * n_outputs;
        const int2 p = __ldg(anchors + (size_t)t * n_anchors + k);
        int32_t *dx = reinterpret_cast<int32_t *>(dX) + b * n_inputs;
        for (int o0 = 0; o0 < n_outputs; o0 += out_block) {
            const int o1 = min(o0 + out_block, n_outputs);
            double ms = 0.0, as = 0.0;
            for (int o = o0; o < o1; o++) {
                const double gdy = (double)__ldg(dy + o);
                ms += (double)__ldg(row + o) * gdy;
                as += (double)__ldg(alt + o) * gdy;
            }
            const double du = up * (ms - as);
            if (fabs(du) > kEps) {
                const int32_t d = to_fixed(du, fixed_scale);
                atomicAdd(dx + p.x, d);
                atomicAdd(dx + p.y, -d);
            }
        }
    }
}

// --------------------------------------------------------------------------------------------
// Kernel 4a: table-gradient scatter with row-coalesced global reductions
// (reference: gather_w_gradients_non_seq_fc_logic, proto:1547-1585, helper :716-819):
// target[t, idx[b, t], :] += lr * dY[b, :] for |dY| > EPS.  `target` is dW, or W itself for the
// internal (in-place SGD) policy with lr = -external_lr * lr_meta.
// --------------------------------------------------------------------------------------------
__device__ __forceinline__ void red_add_v4(float *addr, float a, float b, float c, float d) {
    asm volatile("red.global.add.v4.f32 [%0], {%1, %2, %3, %4};" ::"l"(addr), "f"(a), "f"(b), "f"(c), "f"(d) : "memory");
}

template <int VEC, bool INT_MODE>
__global__ void __launch_bounds__(256) fc_weight_grad_atomic_kernel(const float *__restrict__ dY, const int32_t *__restrict__ idx,
                                                                   float *__restrict__ target, int64_t batch,
                                                                   int n_outputs, int n_detectors, int table_rows,
                                                                   int lanes_per_row, int chunk, double lr,
                                                                   double fixed_scale) {
    const int lane = threadIdx.x & 31;
    const int64_t b = (int64_t)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
    if (b >= batch) return;
    const int c0 = blockIdx.y * chunk;
    const int clen = min(chunk, n_outputs - c0);
    const int LG = lanes_per_row;
    const int NG = 32 / LG;
    const int g = lane / LG;
    const int j = lane - g * LG;
    const float *dy = dY + b * n_outputs + c0;
    const int32_t *idx_b = idx + b * n_detectors;

    float val[kFwdJ][VEC];
    int32_t ival[kFwdJ][VEC];
#pragma unroll
    for (int q = 0; q < kFwdJ; q++) {
        const int col = (j + q * LG) * VEC;
#pragma unroll
        for (int e = 0; e < VEC; e++) { val[q][e] = 0.f; ival[q][e] = 0; }
        if (col < clen) {
            float d[VEC];
            Vec<VEC>::load(dy + col, d);
#pragma unroll
            for (int e = 0; e < VEC; e++) {
                const double gd = (double)d[e];
                if (fabs(gd) > kEps) {
                    if (INT_MODE) ival[q][e] = to_fixed(gd * lr, fixed_scale);
                    else val[q][e] = (float)(gd * lr);
                }
            }
        }
    }
    for (int tb = 0; tb < n_detectors; tb += 32) {
        const int nvalid = min(32, n_detectors - tb);
        const int32_t mine = (lane < nvalid) ? __ldg(idx_b + tb + lane) : 0;
        for (int sb = 0; sb < nvalid; sb += NG) {
            const int s = sb + g;
            const int32_t li = __shfl_sync(0xffffffffu, mine, s & 31);
            if (s < nvalid) {
                float *row = target + ((size_t)(tb + s) * table_rows + li) * n_outputs + c0;
#pragma unroll
                for (int q = 0; q < kFwdJ; q++) {
                    const int col = (j + q * LG) * VEC;
                    if (col < clen) {
                        if constexpr (INT_MODE) {
#pragma unroll
                            for (int e = 0; e < VEC; e++)
                                if (ival[q][e] != 0) atomicAdd(reinterpret_cast<int32_t *>(row + col + e), ival[q][e]);
                        } else if constexpr (VEC == 4) {
                            red_add_v4(row + col, val[q][0], val[q][1], val[q][2], val[q][3]);
                        } else {
                            if (val[q][0] != 0.f) atomicAdd(row + col, val[q][0]);
                        }
                    }
                }
            }
        }
    }
}

int launch_fc_backward(const lutb_layer_cfg *cfg, int64_t batch, float *W, const float *dY, const int32_t *anchors,
                       const int32_t *idx, const float *min_delta, const int32_t *min_k, float *dX, float *target,
                       double lr, cudaStream_t stream, bool skip_table_gradient = false, bool write_dx = false) {
    const int O = cfg->n_outputs, Nt = cfg->n_detectors, T = 1 << cfg->n_anchors;
    const bool int_mode = cfg->int_mode != 0;
    const bool vec4 = (O % 4 == 0) && ((reinterpret_cast<uintptr_t>(W) & 15) == 0) &&
                      ((reinterpret_cast<uintptr_t>(dY) & 15) == 0) && ((reinterpret_cast<uintptr_t>(target) & 15) == 0);
    const int vec = vec4 ? 4 : 1;
    const int vpr = (O + vec - 1) / vec;
    const int lanes = min(32, pow2_ceil(vpr));
    const int warps = 8;
    const int64_t blocks = (batch + warps - 1) / warps;
    LUTB_REQUIRE(blocks <= 0x7FFFFFFF, LUTB_ERR_SHAPE, "batch too large for one launch");
    const int sm = device_info().sm_count;

    // rows of dX in shared memory: while at least three blocks of eight warps fit an SM
    const size_t row_bytes = (size_t)((cfg->n_inputs + 3) & ~3) * 4;
    const bool rows = write_dx && dX != nullptr && !int_mode && 8 * row_bytes <= 64 * 1024;
    // few samples: small blocks, or (a sample's row has one owner where it is written) 32 detectors a block, so that more SMs
    // share the work
    const bool few = blocks < 2 * sm;
    // (32 at a time; more where a grid would have no room for the groups)
    const int group_dets = few && !rows ? min(Nt, max(32, (int)(((int64_t)Nt + 65534) / 65535))) : Nt, dx_warps = few && rows ? 2 : warps;
    if (write_dx && dX != nullptr && !rows) {
        const int rc = lutb_zero_buffers(dX, batch * (int64_t)cfg->n_inputs * 4, nullptr, 0, nullptr, 0, stream);
        if (rc) return rc;
    }

    // input gradient (dX == nullptr: the caller does not want it)
    if (dX != nullptr) {
    KernelScope scope(K_FC_INPUT_GRAD, stream);
    if (int_mode) {
        const int64_t total = batch * Nt;
        const int64_t gblocks = min((total + 127) / 128, (int64_t)sm * 64);
        fc_input_grad_fixed_kernel<<<(unsigned)gblocks, 128, 0, stream>>>(
            W, dY, reinterpret_cast<const int2 *>(anchors), idx, min_delta, min_k, dX, batch, cfg->n_inputs, O, Nt,
            cfg->n_anchors, T, cfg->forward_group, cfg->int_rescaler);
    } else {
        const int groups = (Nt + group_dets - 1) / group_dets;
        // (many short blocks: the last wave of 16 blocks an SM was a fifth empty, 60000 samples x 4000 inputs 216 -> 195 us)
        int64_t per_block = (batch * groups / ((int64_t)sm * 32) + dx_warps - 1) / dx_warps * dx_warps;
        if (per_block < dx_warps) per_block = dx_warps;
        if (per_block > 4096) per_block = 4096;
        const dim3 grid((unsigned)((batch + per_block - 1) / per_block), (unsigned)groups);
        LUTB_REQUIRE(groups <= 65535, LUTB_ERR_SHAPE, "too many detectors for one launch");
        int launch_rc = LUTB_OK;
        auto launch = [&](auto add, auto write) -> int {
            const size_t smem = rows ? dx_warps * row_bytes : 0;
            auto kern = rows ? write : add;
            if (smem > kPlainSmem) LUTB_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
            kern<<<grid, dx_warps * 32, smem, stream>>>(W, dY, reinterpret_cast<const int2 *>(anchors), idx, min_delta, min_k, dX, batch,
                                                  cfg->n_inputs, O, Nt, cfg->n_anchors, T, group_dets, (int)per_block);
            return LUTB_OK;
        };
        auto pick = [&](auto lg, auto v) -> int {
            constexpr int LG = decltype(lg)::value, V = decltype(v)::value;
            if constexpr (LG == 32) {   // (the only groups whose rows can have more steps than one)
                if (O > LG * V) return launch(fc_input_grad_kernel<LG, V, false, false>, fc_input_grad_kernel<LG, V, true, false>);
            }
            return launch(fc_input_grad_kernel<LG, V, false, true>, fc_input_grad_kernel<LG, V, true, true>);
        };
        auto pick_lanes = [&](auto v) -> int {
            switch (lanes) {
                case 32: return pick(std::integral_constant<int, 32>{}, v);
                case 16: return pick(std::integral_constant<int, 16>{}, v);
                case 8: return pick(std::integral_constant<int, 8>{}, v);
                case 4: return pick(std::integral_constant<int, 4>{}, v);
                case 2: return pick(std::integral_constant<int, 2>{}, v);
                default: return pick(std::integral_constant<int, 1>{}, v);
            }
        };
        launch_rc = vec4 ? pick_lanes(std::integral_constant<int, 4>{}) : pick_lanes(std::integral_constant<int, 1>{});
        if (launch_rc) return launch_rc;
    }
    }
    LUTB_LAUNCH_CHECK();

    if (skip_table_gradient) return LUTB_OK;
    // table gradient (or in-place update)
    const int chunk = min(O, lanes * kFwdJ * vec);
    const int n_chunks = (O + chunk - 1) / chunk;
    LUTB_REQUIRE(n_chunks <= 65535, LUTB_ERR_SHAPE, "too many output chunks");
    dim3 grid((unsigned)blocks, (unsigned)n_chunks);
    KernelScope scope(K_FC_WEIGHT_GRAD, stream);
    if (vec4) {
        if (int_mode)
            fc_weight_grad_atomic_kernel<4, true><<<grid, warps * 32, 0, stream>>>(dY, idx, target, batch, O, Nt, T, lanes, chunk, lr, cfg->int_rescaler);
        else
            fc_weight_grad_atomic_kernel<4, false><<<grid, warps * 32, 0, stream>>>(dY, idx, target, batch, O, Nt, T, lanes, chunk, lr, cfg->int_rescaler);
    } else {
        if (int_mode)
            fc_weight_grad_atomic_kernel<1, true><<<grid, warps * 32, 0, stream>>>(dY, idx, target, batch, O, Nt, T, lanes, chunk, lr, cfg->int_rescaler);
        else
            fc_weight_grad_atomic_kernel<1, false><<<grid, warps * 32, 0, stream>>>(dY, idx, target, batch, O, Nt, T, lanes, chunk, lr, cfg->int_rescaler);
    }
    LUTB_LAUNCH_CHECK();
    return LUTB_OK;
}

}  // namespace lutb

// ------------------------------------------------------------------------------------------ C ABI
using namespace lutb;

extern "C" int lutb_nonseq_fc_forward(const lutb_layer_cfg *cfg, int64_t batch, const float *weights, const float *x,
                                      const int32_t *anchors, float *y, int32_t *idx, float *min_delta,
                                      int32_t *min_k, void *stream) {
    int rc = validate_cfg(cfg);
    if (rc) return rc;
    LUTB_REQUIRE(cfg->seq_len == 1, LUTB_ERR_MODE, "forward_step should only be called when sequence_length == 1");
    LUTB_REQUIRE(batch > 0, LUTB_ERR_SHAPE, "batch_size == 0");
    LUTB_REQUIRE(weights && x && anchors && y && idx, LUTB_ERR_NULL, "a required tensor pointer is NULL");
    LUTB_REQUIRE((min_delta == nullptr) == (min_k == nullptr), LUTB_ERR_MODE,
                 "min_anchor_deltas and min_anchor_delta_indices must be given together");
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    rc = launch_check_detectors(x, batch, cfg->n_inputs, anchors, cfg->n_detectors, cfg->n_anchors, cfg->cmp_eps, idx,
                                min_delta, min_k, st);
    if (rc) return rc;
    rc = launch_fc_gather_forward(weights, idx, y, batch, cfg->n_outputs, cfg->n_detectors, 1 << cfg->n_anchors,
                                  cfg->backward_group, cfg->int_mode != 0, cfg->int_rescaler, st);
    if (rc) return rc;
    if (cfg->int_mode) return launch_fixed_to_float(y, batch * (int64_t)cfg->n_outputs, cfg->int_rescaler, st);
    return LUTB_OK;
}

extern "C" size_t lutb_infer_fp32_workspace(const lutb_layer_cfg *cfg, int64_t batch) {
    const void *aligned = reinterpret_cast<const void *>((uintptr_t)256);
    if (validate_cfg(cfg) != LUTB_OK || batch <= 0 || !infer_staged_fp32_applies(cfg, batch, aligned, aligned)) return 0;
    return infer_staged_fp32_workspace(cfg, batch);
}

extern "C" int lutb_infer_fp32_accumulate(const lutb_layer_cfg *cfg, int64_t batch, const float *weights, const float *x,
                                          const int32_t *anchors, float *y, int32_t *idx, void *workspace,
                                          size_t workspace_bytes, void *stream) {
    int rc = validate_cfg(cfg);
    if (rc) return rc;
    const bool staged = workspace != nullptr && batch > 0 && infer_staged_fp32_applies(cfg, batch, weights, y) &&
                        infer_staged_pass(cfg, batch, false) > 0;
    if (!staged) return lutb_nonseq_fc_forward(cfg, batch, weights, x, anchors, y, idx, nullptr, nullptr, stream);
    LUTB_REQUIRE(cfg->seq_len == 1, LUTB_ERR_MODE, "inference is defined for non-sequence layers");
    LUTB_REQUIRE(weights && x && anchors && y && idx, LUTB_ERR_NULL, "a required tensor pointer is NULL");
    const size_t need = infer_staged_fp32_workspace(cfg, batch);
    LUTB_REQUIRE(workspace_bytes >= need, LUTB_ERR_WORKSPACE, "the staged gather needs %zu bytes of workspace", need);
    LUTB_REQUIRE((reinterpret_cast<uintptr_t>(workspace) & 255) == 0, LUTB_ERR_ALIGN, "workspace must be 256-byte aligned");
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    const int64_t pass = infer_staged_pass(cfg, batch, false);
    uint8_t *packed = static_cast<uint8_t *>(workspace);
    float *partial = reinterpret_cast<float *>(packed + packed_index_bytes(cfg, pass));
    uint32_t *plan = reinterpret_cast<uint32_t *>(static_cast<uint8_t *>(workspace) + need - anchor_plan_bytes(cfg));
    for (int64_t b0 = 0; b0 < batch; b0 += pass) {
        const int64_t n = batch - b0 < pass ? batch - b0 : pass;
        rc = launch_check_detectors(x + b0 * cfg->n_inputs, n, cfg->n_inputs, anchors, cfg->n_detectors, cfg->n_anchors, cfg->cmp_eps,
                                    idx + b0 * cfg->n_detectors, nullptr, nullptr, st, packed, packed_index_pitch(n), plan);
        if (rc) return rc;
        rc = launch_infer_staged_fp32(cfg, n, weights, packed, partial, y + b0 * cfg->n_outputs, st);
        if (rc) return rc;
    }
    return LUTB_OK;
}

extern "C" size_t lutb_nonseq_fc_backward_workspace(const lutb_layer_cfg *cfg, int64_t batch, int dw_variant) {
    dw_variant &= ~LUTB_DX_WRITE;
    if (cfg == nullptr || batch <= 0 || dw_variant != LUTB_DW_SORTED || cfg->int_mode) return 0;
    return fc_dw_sorted_workspace(batch, cfg->n_detectors, 1 << cfg->n_anchors);
}

extern "C" int lutb_nonseq_fc_backward(const lutb_layer_cfg *cfg, int64_t batch, float *weights, const float *dY,
                                       const int32_t *anchors, const int32_t *idx, const float *min_delta,
                                       const int32_t *min_k, float *dX, float *dW, double external_lr, int dw_variant,
                                       void *workspace, size_t workspace_bytes, void *stream) {
    int rc = validate_cfg(cfg);
    if (rc) return rc;
    LUTB_REQUIRE(cfg->seq_len == 1, LUTB_ERR_MODE, "backward_backprop should only be called when sequence_length == 1");
    const bool write_dx = (dw_variant & LUTB_DX_WRITE) != 0;
    dw_variant &= ~LUTB_DX_WRITE;
    LUTB_REQUIRE(dw_variant == LUTB_DW_AUTO || dw_variant == LUTB_DW_ATOMIC || dw_variant == LUTB_DW_SORTED, LUTB_ERR_MODE,
                 "unknown dw_variant %d", dw_variant);
    // fixed-point sums are order independent already: the sorted variant only applies to fp32 accumulators
    const bool sorted = dw_variant == LUTB_DW_SORTED && !cfg->int_mode;
    if (sorted) {
        const size_t need = fc_dw_sorted_workspace(batch, cfg->n_detectors, 1 << cfg->n_anchors);
        LUTB_REQUIRE(workspace != nullptr && workspace_bytes >= need, LUTB_ERR_WORKSPACE,
                     "the sorted table-gradient variant needs %zu bytes of workspace", need);
        LUTB_REQUIRE((reinterpret_cast<uintptr_t>(workspace) & 255) == 0, LUTB_ERR_ALIGN, "workspace must be 256-byte aligned");
    }
    LUTB_REQUIRE(batch > 0, LUTB_ERR_SHAPE, "batch_size == 0");
    LUTB_REQUIRE(weights && dY && anchors && idx && min_delta && min_k, LUTB_ERR_NULL,
                 "a required tensor pointer is NULL");
    LUTB_REQUIRE(!(external_lr >= 0.0 && dW != nullptr), LUTB_ERR_MODE,
                 "in internal weight gradients mode w_weights_gradients should be nullptr");
    const bool skip_table = external_lr == LUTB_SKIP_TABLE_GRADIENT;
    LUTB_REQUIRE(!(skip_table && dW != nullptr), LUTB_ERR_MODE, "no table gradient asked for, w_weights_gradients should be nullptr");
    LUTB_REQUIRE(!(external_lr < 0.0 && dW == nullptr && !skip_table), LUTB_ERR_NULL, "w_weights_gradients is NULL");
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    double lr = cfg->lr_meta;
    // the reference narrows external_lr to fp32 before use (lut.cu:1076)
    if (external_lr >= 0.0) lr *= -(double)(float)external_lr;
    float *target = external_lr >= 0.0 ? weights : dW;
    rc = launch_fc_backward(cfg, batch, weights, dY, anchors, idx, min_delta, min_k, dX, target, lr, st, sorted || skip_table, write_dx);
    if (rc) return rc;
    if (sorted && !skip_table) {
        rc = launch_fc_dw_sorted(dY, idx, target, batch, cfg->n_outputs, cfg->n_detectors, 1 << cfg->n_anchors, lr,
                                 workspace, st);
        if (rc) return rc;
    }
    if (cfg->int_mode) {
        if (dX) rc = launch_fixed_to_float(dX, batch * (int64_t)cfg->n_inputs, cfg->int_rescaler, st);
        if (rc) return rc;
        if (dW) rc = launch_fixed_to_float(dW, (int64_t)cfg->n_detectors * (1 << cfg->n_anchors) * cfg->n_outputs, cfg->int_rescaler, st);
    }
    return rc;
}

extern "C" size_t lutb_nonseq_fc_table_grad_rows_workspace(const lutb_layer_cfg *cfg, int64_t batch) {
    if (cfg == nullptr || batch <= 0 || cfg->int_mode) return 0;
    return fc_dw_rows_workspace(batch, cfg->n_detectors, 1 << cfg->n_anchors);
}

extern "C" int lutb_nonseq_fc_table_grad_rows(const lutb_layer_cfg *cfg, int64_t batch, const float *dY,
                                              const int32_t *idx, int64_t *row_ids, float *values, int64_t capacity,
                                              int64_t *count_out, void *workspace, size_t workspace_bytes, void *stream) {
    int rc = validate_cfg(cfg);
    if (rc) return rc;
    LUTB_REQUIRE(cfg->seq_len == 1, LUTB_ERR_MODE, "the row-list table gradient is for sequence_length == 1");
    LUTB_REQUIRE(cfg->int_mode == 0, LUTB_ERR_MODE, "the row-list table gradient needs fp32 accumulators");
    LUTB_REQUIRE(batch > 0, LUTB_ERR_SHAPE, "batch_size == 0");
    LUTB_REQUIRE(dY && idx && row_ids && values && count_out, LUTB_ERR_NULL, "a required tensor pointer is NULL");
    LUTB_REQUIRE(capacity > 0, LUTB_ERR_SHAPE, "capacity == 0");
    const size_t need = fc_dw_rows_workspace(batch, cfg->n_detectors, 1 << cfg->n_anchors);
    LUTB_REQUIRE(workspace != nullptr && workspace_bytes >= need, LUTB_ERR_WORKSPACE,
                 "the row-list table gradient needs %zu bytes of workspace", need);
    LUTB_REQUIRE((reinterpret_cast<uintptr_t>(workspace) & 255) == 0, LUTB_ERR_ALIGN, "workspace must be 256-byte aligned");
    return launch_fc_dw_rows(dY, idx, batch, cfg->n_outputs, cfg->n_detectors, 1 << cfg->n_anchors, cfg->lr_meta, row_ids,
                             values, capacity, count_out, workspace, static_cast<cudaStream_t>(stream));
}

extern "C" int lutb_nonseq_fc_backward_noalloc(const lutb_layer_cfg *cfg, int64_t batch, float *weights,
                                               const float *dY, const int32_t *anchors, const int32_t *idx,
                                               const float *min_delta, const int32_t *min_k, float *dX, float *dW,
                                               double external_lr, void *stream) {
    NoEventsGuard no_events;  // event creation allocates
    int rc = validate_cfg(cfg);
    if (rc) return rc;
    LUTB_REQUIRE(cfg->int_mode == 0, LUTB_ERR_MODE,
                 "the no-allocation backward supports fp32 accumulators only (int_mode must be 0)");
    LUTB_REQUIRE(batch > 0, LUTB_ERR_SHAPE, "batch_size == 0");
    const size_t need = fc_dw_sorted_workspace(batch, cfg->n_detectors, 1 << cfg->n_anchors);
    LUTB_REQUIRE(need <= (size_t)LUTB_STATIC_SCRATCH_BYTES, LUTB_ERR_WORKSPACE,
                 "problem needs %zu bytes of scratch, the built-in array holds %u: reduce the batch or use "
                 "lutb_nonseq_fc_backward with a caller workspace", need, (unsigned)LUTB_STATIC_SCRATCH_BYTES);
    void *scratch = nullptr;
    rc = static_scratch(&scratch);
    if (rc) return rc;
    return lutb_nonseq_fc_backward(cfg, batch, weights, dY, anchors, idx, min_delta, min_k, dX, dW, external_lr,
                                   LUTB_DW_SORTED, scratch, (size_t)LUTB_STATIC_SCRATCH_BYTES, stream);
}
