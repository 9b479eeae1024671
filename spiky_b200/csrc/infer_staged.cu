// Forward gathers of large layers: y[b, :] += sum_t table_t[idx[b, t], :] with the tables in shared memory.
//
// Gathering rows from L2 is limited by the number of row requests (about 37 G rows a second whether a row is 64 or 256
// bytes), and a large batch asks for every row many times.  Here a block owns a tile of samples, keeps its sums in
// registers and streams the tables of a run of detectors through a three-slot shared-memory ring (two
// or four detectors a slot), so that a row costs one conflict-free shared-memory wavefront: the 8 lanes that add a row read its
// 128 bytes side by side.  What a block loads is the whole table once per tile, so tiles are as large as the register
// file allows; a small batch reads the tables once, in order, instead of by random rows.
#include "infer_staged.cuh"

#include "mbarrier.cuh"
#include "tensor_map.cuh"

namespace lutb {

constexpr int kStagedThreads = 512;
constexpr int kStages = 3;          // ring slots

__device__ __forceinline__ uint32_t smem_addr(const void *p) { return (uint32_t)__cvta_generic_to_shared(p); }
template <int BYTES>
__device__ __forceinline__ void async_copy(uint32_t dst, const void *src) {
    if constexpr (BYTES == 16) asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(src) : "memory");
    else asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(dst), "l"(src) : "memory");
}
__device__ __forceinline__ void async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void async_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }

// --------------------------------------------------------------------------------------------
// fp32 tables.  Tile: 1024 samples x 32 columns, kSlots samples per group of 8 lanes (4 columns a lane): 64 accumulators
// per thread.  A work item is (block of kDetBlock detectors, tile, column slice); the detectors' block sums go to a partial
// buffer and are added up in double by a second kernel.  Precision: two detectors are added before they meet the
// accumulator, and a chain is kDetBlock / 2 = 12 long: the distance from 64-bit sums is 7.6e-8 (2-norm, relative), against
// 8.1e-8 (512 detectors) to 9.5e-8 (4096) for the L2 gather of rows of 33 to 64 outputs, whose chains are 16 single rows.
// --------------------------------------------------------------------------------------------
constexpr int kLanes = 8, kSlots = 16, kDetBlock = 24;
constexpr int kGroups = kStagedThreads / kLanes, kTile = kGroups * kSlots, kRow = kLanes * 4;   // kRow: floats per staged row

struct StagedFp32 {
    const float *W;
    const uint8_t *packed;
    float *out;            // [n_blocks][batch][O] partial sums
    int64_t batch;
    size_t pitch;
    int O, Nt, T, n_tiles, n_slices, n_items;
};

// A warp of its own brings the tables in by TMA (a column slice of a whole table is one box) and the samples' indices by bulk
// copies, and waits for a slot's readers one by one; the 16 warps that add wait for a slot to fill and say when they have read it, so
// that none of them waits for the slowest (with cp.async and a block barrier per two detectors, 1024 samples a step: 834 -> 600 us
// for 16384 samples, 4096 detectors of 256 rows x 64 outputs, the rate of the shared-memory wavefronts: 480 us of row reads and
// 120 of tables coming in).
__device__ int g_staged_wait_errors = 0;

int staged_wait_errors(int *count_out) {
    LUTB_CUDA(cudaMemcpyFromSymbol(count_out, g_staged_wait_errors, sizeof(int)));
    return LUTB_OK;
}

// After a wait that ran out: tell the block's others, and leave only after a time in which every copy in flight has landed.
__device__ __noinline__ void leave_late(volatile int *gave_up) {
    if (*gave_up == 0) atomicAdd(&g_staged_wait_errors, 1);
    *gave_up = 1;
    const long long t0 = clock64();
    while (clock64() - t0 < kWaitLimitCycles / 16) {
    }
}

__device__ __forceinline__ void tma_load_box(uint32_t dst, const CUtensorMap *map, int x, int y, uint32_t bar) {
    asm volatile("cp.async.bulk.tensor.2d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];" ::"r"(dst),
                 "l"(map), "r"(bar), "r"(x), "r"(y)
                 : "memory");
}

__global__ void __launch_bounds__(kStagedThreads + 32, 1) infer_staged_fp32_kernel(const __grid_constant__ CUtensorMap tables, const StagedFp32 p) {
    extern __shared__ __align__(128) unsigned char sbuf[];
    const int stage_floats = 2 * p.T * kRow;
    float *ring = reinterpret_cast<float *>(sbuf);                             // [kStages][2][T][kRow]
    uint8_t *ibuf = sbuf + (size_t)kStages * stage_floats * 4;                 // [kStages][2][kTile]
    const uint32_t full0 = smem_addr(ibuf + (size_t)kStages * 2 * kTile), empty0 = full0 + 8 * kStages;
    volatile int *gave_up = reinterpret_cast<volatile int *>(ibuf + (size_t)kStages * 2 * kTile + 16 * kStages);
    const int tid = threadIdx.x, g = tid / kLanes, l = tid % kLanes;
    const uint32_t mask = (uint32_t)p.T - 1u;   // (samples past the batch hold any byte)
    if (tid == 0) {
        for (int s = 0; s < kStages; s++) {
            mbar_init(full0 + 8 * s, 1);
            mbar_init(empty0 + 8 * s, kStagedThreads / 32);
        }
        *gave_up = 0;
        fence_barrier_init();
    }
    __syncthreads();
    // detector blocks outermost: the blocks that run together read the same tables
    const int per = p.n_tiles * p.n_slices;
    int slot = 0;
    uint32_t phase = 0u;
    bool ok = true;
    if (tid >= kStagedThreads) {
        if (tid == kStagedThreads) {
            for (int item = blockIdx.x; item < p.n_items && ok; item += gridDim.x) {
                const int db = item / per, ts = item - db * per;
                const int tile = ts / p.n_slices, slice = ts - tile * p.n_slices;
                const int t0 = db * kDetBlock, nd = min(kDetBlock, p.Nt - t0);
                for (int t = t0; t < t0 + nd; t += 2) {
                    ok = mbar_wait(empty0 + 8 * slot, phase ^ 1u) && *gave_up == 0;
                    if (!ok) break;
                    const int dets = min(2, t0 + nd - t);
                    const uint32_t bar = full0 + 8 * slot, dst = smem_addr(ring + (size_t)slot * stage_floats), idst = smem_addr(ibuf + (size_t)slot * 2 * kTile);
                    mbar_arrive_expect_tx(bar, (uint32_t)dets * (uint32_t)(p.T * kRow * 4 + kTile));
                    for (int d = 0; d < dets; d++) {
                        tma_load_box(dst + (uint32_t)(d * p.T * kRow * 4), &tables, slice * kRow, (t + d) * p.T, bar);
                        bulk_copy_g2s(idst + (uint32_t)(d * kTile), p.packed + (size_t)(t + d) * p.pitch + (size_t)tile * kTile, kTile, bar);
                    }
                    if (++slot == kStages) { slot = 0; phase ^= 1u; }
                }
            }
        }
    } else {
        for (int item = blockIdx.x; item < p.n_items && ok; item += gridDim.x) {
            const int db = item / per, ts = item - db * per;
            const int tile = ts / p.n_slices, slice = ts - tile * p.n_slices;
            const int t0 = db * kDetBlock, nd = min(kDetBlock, p.Nt - t0), np = (nd + 1) / 2;
            const int64_t b0 = (int64_t)tile * kTile;
            const int c0 = slice * kRow, width = min(kRow, p.O - c0);
            float2 acc[kSlots][2];
#pragma unroll
            for (int s = 0; s < kSlots; s++) acc[s][0] = acc[s][1] = make_float2(0.f, 0.f);
            for (int pr = 0; pr < np; pr++) {
                ok = __all_sync(0xffffffffu, mbar_wait(full0 + 8 * slot, phase) && *gave_up == 0);
                if (!ok) break;
                const char *tab = reinterpret_cast<const char *>(ring + (size_t)slot * stage_floats) + l * 16;
                const uint8_t *ib = ibuf + (size_t)slot * 2 * kTile + g * kSlots;
                const uint4 ia = *reinterpret_cast<const uint4 *>(ib);
                const uint32_t wa[4] = {ia.x, ia.y, ia.z, ia.w};
                if (2 * pr + 1 < nd) {
                    const uint4 ic = *reinterpret_cast<const uint4 *>(ib + kTile);
                    const uint32_t wb[4] = {ic.x, ic.y, ic.z, ic.w};
                    const char *tab2 = tab + (size_t)p.T * kRow * 4;
#pragma unroll
                    for (int s = 0; s < kSlots; s++) {
                        const uint32_t ra = (wa[s / 4] >> (8 * (s % 4))) & mask, rb = (wb[s / 4] >> (8 * (s % 4))) & mask;
                        const float4 a = *reinterpret_cast<const float4 *>(tab + ra * (kRow * 4));
                        const float4 b = *reinterpret_cast<const float4 *>(tab2 + rb * (kRow * 4));
                        acc[s][0] = __fadd2_rn(acc[s][0], __fadd2_rn(make_float2(a.x, a.y), make_float2(b.x, b.y)));
                        acc[s][1] = __fadd2_rn(acc[s][1], __fadd2_rn(make_float2(a.z, a.w), make_float2(b.z, b.w)));
                    }
                } else {
#pragma unroll
                    for (int s = 0; s < kSlots; s++) {
                        const uint32_t ra = (wa[s / 4] >> (8 * (s % 4))) & mask;
                        const float4 a = *reinterpret_cast<const float4 *>(tab + ra * (kRow * 4));
                        acc[s][0] = __fadd2_rn(acc[s][0], make_float2(a.x, a.y));
                        acc[s][1] = __fadd2_rn(acc[s][1], make_float2(a.z, a.w));
                    }
                }
                __syncwarp();
                if ((tid & 31) == 0) mbar_arrive(empty0 + 8 * slot);
                if (++slot == kStages) { slot = 0; phase ^= 1u; }
            }
            if (ok && l * 4 < width) {
                float *out = p.out + (size_t)db * p.batch * p.O + c0 + l * 4;
#pragma unroll
                for (int s = 0; s < kSlots; s++) {
                    const int64_t b = b0 + g * kSlots + s;
                    if (b < p.batch)
                        *reinterpret_cast<float4 *>(out + (size_t)b * p.O) = make_float4(acc[s][0].x, acc[s][0].y, acc[s][1].x, acc[s][1].y);
                }
            }
        }
    }
    if (!ok) leave_late(gave_up);
}

// y[i] += sum over the detector blocks, in double
__global__ void __launch_bounds__(256) add_partials_kernel(const float *__restrict__ partial, float *__restrict__ y, int64_t n4, int blocks) {
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n4; i += (int64_t)gridDim.x * blockDim.x) {
        double s[4] = {0.0, 0.0, 0.0, 0.0};
        const float4 *src = reinterpret_cast<const float4 *>(partial) + i;
#pragma unroll 8
        for (int k = 0; k < blocks; k++) {
            const float4 v = __ldcs(src + (size_t)k * n4);
            s[0] += (double)v.x; s[1] += (double)v.y; s[2] += (double)v.z; s[3] += (double)v.w;
        }
        float4 *dst = reinterpret_cast<float4 *>(y) + i;
        float4 o = *dst;
        o.x = (float)(s[0] + (double)o.x); o.y = (float)(s[1] + (double)o.y);
        o.z = (float)(s[2] + (double)o.z); o.w = (float)(s[3] + (double)o.w);
        *dst = o;
    }
}

// --------------------------------------------------------------------------------------------
// int8 tables, exact de-quantisation.  The sum of a truncation block, sum_t scale_t * q_t as an exact real, is formed in
// integers where the block's scales allow it: scale_t = m_t * 2^e with one e per block and |m_t| < 2^31, m_t = h_t * 2^16 +
// l_t, so that two int32 sums of h_t * q_t and l_t * q_t (at most 255 detectors) hold it exactly and one conversion per
// block gives the same double as fp64 multiply-adds (the fp64 unit takes a sixteenth of a warp a cycle: a conversion and a
// multiply-add per entry bound the kernel).  Blocks whose scales spread over more than 2^7, or are not finite, take the
// fp64 route; its sums use the same registers.
// Two detectors' entries are taken at a time (dp2a: two products of a 16-bit and an 8-bit number), which is 10 instructions for four
// columns of both against 24 with a sign extension and a multiply-add for each; with that, no spilled registers and whole sectors in the
// final additions: 4096 samples, 4096 detectors x 64 outputs 328 -> 203 us.
// 8 lanes x 8 columns per row (rows of 64 bytes; wider rows in column slices), four samples per lane group.  A work item is
// (run of whole truncation blocks, tile, column slice); its int32 sums are added to the result with integer reductions.
// --------------------------------------------------------------------------------------------
constexpr int kSlots8 = 4, kCols8 = 64, kTile8 = kGroups * kSlots8, kDets8 = 4;   // kDets8: detectors per ring slot

struct ScalePlan {
    int2 *planes;    // [Nt] (h, l)
    double *unit;    // [truncation blocks] 2^e, 0: fp64 route
};
__host__ __device__ inline size_t scale_plan_bytes(int Nt, int trunc_blocks) { return (size_t)Nt * 8 + (size_t)trunc_blocks * 8; }
__host__ __device__ inline ScalePlan scale_plan_at(void *base, int Nt) {
    return ScalePlan{static_cast<int2 *>(base), reinterpret_cast<double *>(static_cast<int2 *>(base) + Nt)};
}

// one warp per truncation block
__global__ void int8_scale_plan_kernel(const float *__restrict__ scales, int Nt, int det_block, int trunc_blocks, void *plan) {
    const ScalePlan sp = scale_plan_at(plan, Nt);
    const int blk = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5), lane = threadIdx.x & 31;
    if (blk >= trunc_blocks) return;
    const int t0 = blk * det_block, t1 = min(Nt, t0 + det_block);
    int lo = 1 << 20, hi = -(1 << 20);   // smallest exponent of a last mantissa bit, largest exponent of a value
    for (int t = t0 + lane; t < t1; t += 32) {
        const uint32_t b = __float_as_uint(scales[t]) & 0x7fffffffu;
        if (b == 0u) continue;
        const int e = (int)(b >> 23);
        const int ulp = (e == 0 ? 1 : e) - 150;
        lo = min(lo, ulp);
        hi = max(hi, e == 255 ? 1 << 20 : ulp + 24);
    }
    for (int m = 16; m >= 1; m >>= 1) {
        lo = min(lo, __shfl_xor_sync(0xffffffffu, lo, m));
        hi = max(hi, __shfl_xor_sync(0xffffffffu, hi, m));
    }
    const bool none = hi < lo;   // all scales are zero
    const bool ok = none || (hi - lo <= 31 && t1 - t0 <= 255);
    const int e = none ? 0 : lo;
    for (int t = t0 + lane; t < t1; t += 32) {
        const int m = ok ? (int)scalbn((double)scales[t], -e) : 0;
        sp.planes[t] = make_int2(m >> 16, m & 0xffff);
    }
    if (lane == 0) sp.unit[blk] = ok ? scalbn(1.0, e) : 0.0;
}

struct StagedInt8 {
    const int8_t *Q;
    const float *scales;
    const uint8_t *packed;
    int32_t *acc;
    ScalePlan plan;
    int64_t batch;
    size_t pitch;
    int O, Nt, T, n_tiles, n_slices, n_items, det_block, dets_per_item;
    int wide;      // rows allow 16-byte copies
    double fixed_scale;
};

// c plus the products of a's two 16-bit halves with bytes 0 and 1 (lo) or 2 and 3 (hi) of b, b's bytes signed; a's halves signed
// (h) or unsigned (l)
__device__ __forceinline__ int dot_h_lo(uint32_t a, uint32_t b, int c) { asm("dp2a.lo.s32.s32 %0, %1, %2, %0;" : "+r"(c) : "r"(a), "r"(b)); return c; }
__device__ __forceinline__ int dot_h_hi(uint32_t a, uint32_t b, int c) { asm("dp2a.hi.s32.s32 %0, %1, %2, %0;" : "+r"(c) : "r"(a), "r"(b)); return c; }
__device__ __forceinline__ int dot_l_lo(uint32_t a, uint32_t b, int c) { asm("dp2a.lo.u32.s32 %0, %1, %2, %0;" : "+r"(c) : "r"(a), "r"(b)); return c; }
__device__ __forceinline__ int dot_l_hi(uint32_t a, uint32_t b, int c) { asm("dp2a.hi.u32.s32 %0, %1, %2, %0;" : "+r"(c) : "r"(a), "r"(b)); return c; }

// FP64: the items with a truncation block whose scales do not share an exponent range, which the other instantiation leaves
// (together they spilled registers); each passes over the other's items.
// (The fp32 kernel's ring of bulk copies was slower here, 234 us against 203: its registers are the scarce ones.)
template <bool FP64>
__global__ void __launch_bounds__(kStagedThreads, 1) infer_staged_int8_kernel(const StagedInt8 p) {
    extern __shared__ __align__(128) unsigned char sbuf[];
    const int stage_bytes = kDets8 * p.T * kCols8;
    unsigned char *ring = sbuf;                                     // [kStages][kDets8][T][kCols8]
    uint8_t *ibuf = sbuf + (size_t)kStages * stage_bytes;           // [kStages][kDets8][kTile8]
    int2 *mbuf = reinterpret_cast<int2 *>(ibuf + kStages * kDets8 * kTile8);   // [kStages][kDets8] integer scales
    const int tid = threadIdx.x, g = tid / kLanes, l = tid % kLanes;
    const uint32_t mask = (uint32_t)p.T - 1u, mask4 = mask * 0x01010101u;   // (samples past the batch hold any byte)
    for (int item = blockIdx.x; item < p.n_items; item += gridDim.x) {
        const int per = p.n_tiles * p.n_slices;
        const int db = item / per, ts = item - db * per;
        const int tile = ts / p.n_slices, slice = ts - tile * p.n_slices;
        const int t0 = db * p.dets_per_item, nd = min(p.dets_per_item, p.Nt - t0), np = (nd + kDets8 - 1) / kDets8;
        bool spread = false;
        for (int k = t0 / p.det_block; k * p.det_block < t0 + nd; k++) spread |= __ldg(p.plan.unit + k) == 0.0;
        if (spread != FP64) continue;
        const int64_t b0 = (int64_t)tile * kTile8;
        const int c0 = slice * kCols8, width = min(kCols8, p.O - c0);
        auto load_stage = [&](int pr) {
            if (pr < np) {
                const int slot = pr % kStages;
                const uint32_t dst = smem_addr(ring + (size_t)slot * stage_bytes);
                const int dets = min(kDets8, nd - kDets8 * pr), t = t0 + kDets8 * pr;
                const int8_t *src = p.Q + (size_t)t * p.T * p.O + c0;
                if (p.wide) {
                    const int c = (tid & 3) * 16;
                    if (c < width)
                        for (int r = tid >> 2; r < dets * p.T; r += kStagedThreads / 4)
                            async_copy<16>(dst + (uint32_t)(r * kCols8 + c), src + (size_t)r * p.O + c);
                } else if (l * 8 < width) {
                    for (int r = g; r < dets * p.T; r += kGroups)
                        async_copy<8>(dst + (uint32_t)(r * kCols8 + l * 8), src + (size_t)r * p.O + l * 8);
                }
                const uint32_t idst = smem_addr(ibuf + (size_t)slot * kDets8 * kTile8);
                if (tid < dets * (kTile8 / 16)) {
                    const int d = tid / (kTile8 / 16), q = tid % (kTile8 / 16);
                    async_copy<16>(idst + (uint32_t)(d * kTile8 + q * 16), p.packed + (size_t)(t + d) * p.pitch + b0 + q * 16);
                } else if (tid >= kStagedThreads - dets) {
                    const int d = kStagedThreads - 1 - tid;
                    async_copy<8>(smem_addr(mbuf + slot * kDets8 + d), p.plan.planes + t + d);
                }
            }
            async_commit();
        };
        // (h, l): the two integer sums of a block, or the halves of its fp64 sum
        int h[kSlots8][8], lw[kSlots8][8], iacc[kSlots8][8];
#pragma unroll
        for (int k = 0; k < kSlots8; k++)
#pragma unroll
            for (int e = 0; e < 8; e++) h[k][e] = lw[k][e] = iacc[k][e] = 0;
        load_stage(0);
        load_stage(1);
        int blk = t0 / p.det_block, left = p.det_block;   // detectors until the block sum is truncated (items start on a block)
        double unit = __ldg(p.plan.unit + blk);
        for (int pr = 0; pr < np; pr++) {
            async_wait<1>();
            __syncthreads();
            load_stage(pr + 2);
            const int slot = pr % kStages;
            const int here = min(kDets8, nd - kDets8 * pr);
            const unsigned char *stage_tab = ring + (size_t)slot * stage_bytes + l * 8;
            const uint8_t *stage_ib = ibuf + (size_t)slot * kDets8 * kTile8 + g * kSlots8;
            // Four columns of two detectors' rows at a time.  (masked: samples past the batch hold any byte)
            auto add_pair = [&](const unsigned char *tab, const unsigned char *tab2, uint32_t rows, uint32_t rows2, int2 m, int2 m2) {
                const uint32_t mh = __byte_perm((uint32_t)m.x, (uint32_t)m2.x, 0x5410), ml = __byte_perm((uint32_t)m.y, (uint32_t)m2.y, 0x5410);
                rows &= mask4;
                rows2 &= mask4;
#pragma unroll
                for (int k = 0; k < kSlots8; k++) {
                    const uint2 u = *reinterpret_cast<const uint2 *>(tab + __byte_perm(rows, 0u, 0x4440 | k) * kCols8);
                    const uint2 v = *reinterpret_cast<const uint2 *>(tab2 + __byte_perm(rows2, 0u, 0x4440 | k) * kCols8);
                    // (entry e of the first, entry e of the second) in neighbouring bytes
                    const uint32_t q[4] = {__byte_perm(u.x, v.x, 0x5140), __byte_perm(u.x, v.x, 0x7362), __byte_perm(u.y, v.y, 0x5140),
                                           __byte_perm(u.y, v.y, 0x7362)};
#pragma unroll
                    for (int e = 0; e < 4; e++) {
                        h[k][2 * e] = dot_h_lo(mh, q[e], h[k][2 * e]);
                        h[k][2 * e + 1] = dot_h_hi(mh, q[e], h[k][2 * e + 1]);
                        lw[k][2 * e] = dot_l_lo(ml, q[e], lw[k][2 * e]);
                        lw[k][2 * e + 1] = dot_l_hi(ml, q[e], lw[k][2 * e + 1]);
                    }
                }
            };
            for (int d = 0, step; d < here; d += step) {
                const int t = t0 + kDets8 * pr + d;
                const unsigned char *tab = stage_tab + (size_t)d * p.T * kCols8;
                const uint8_t *ib = stage_ib + d * kTile8;
                const uint32_t rows = *reinterpret_cast<const uint32_t *>(ib);
                if (!FP64 || unit != 0.0) {
                    const int2 *ms = mbuf + slot * kDets8 + d;
                    if (d + 1 < here && left > 1) {
                        step = 2;
                        add_pair(tab, tab + (size_t)p.T * kCols8, rows, *reinterpret_cast<const uint32_t *>(ib + kTile8), ms[0], ms[1]);
                    } else {   // (the second with a scale of zero)
                        step = 1;
                        add_pair(tab, tab, rows, rows, ms[0], make_int2(0, 0));
                    }
                } else if constexpr (FP64) {
                    step = 1;
                    const double sd = (double)__ldg(p.scales + t);
#pragma unroll
                    for (int k = 0; k < kSlots8; k++) {
                        const uint2 w = *reinterpret_cast<const uint2 *>(tab + ((rows >> (8 * k)) & mask) * kCols8);
#pragma unroll
                        for (int e = 0; e < 8; e++) {
                            const int q = (int)(int8_t)(((e < 4 ? w.x : w.y) >> (8 * (e & 3))) & 0xffu);
                            const double s = fma(sd, (double)q, __hiloint2double(h[k][e], lw[k][e]));
                            h[k][e] = __double2hiint(s);
                            lw[k][e] = __double2loint(s);
                        }
                    }
                }
                left -= step;
                if (left == 0 || t + step == t0 + nd) {
#pragma unroll
                    for (int k = 0; k < kSlots8; k++)
#pragma unroll
                        for (int e = 0; e < 8; e++) {
                            const double v = !FP64 || unit != 0.0 ? (double)((long long)h[k][e] * 65536ll + (long long)lw[k][e]) * unit
                                                         : __hiloint2double(h[k][e], lw[k][e]);
                            iacc[k][e] += to_fixed(v, p.fixed_scale);
                            h[k][e] = lw[k][e] = 0;
                        }
                    left = p.det_block;
                    if (t + step < t0 + nd) unit = __ldg(p.plan.unit + ++blk);
                }
            }
        }
        // A lane has eight neighbouring columns of four samples: the eight lanes of a group change places (three halving steps) so
        // that they add to neighbouring columns, whole sectors, at a time.  (One column in eight a time took eight times the requests
        // to L2, 16 M additions for 4096 samples.)
#pragma unroll
        for (int k = 0; k < kSlots8; k++) {
#pragma unroll
            for (int o = 4; o >= 1; o >>= 1)
#pragma unroll
                for (int e = 0; e < 8; e++)
                    if ((e & o) == 0) {
                        const bool upper = (l & o) != 0;
                        const int other = __shfl_xor_sync(0xffffffffu, upper ? iacc[k][e] : iacc[k][e + o], o);
                        if (upper) iacc[k][e] = other;
                        else iacc[k][e + o] = other;
                    }
            const int64_t b = b0 + g * kSlots8 + k;
            if (b < p.batch) {
                int32_t *dst = p.acc + (size_t)b * p.O + c0;
#pragma unroll
                for (int e = 0; e < 8; e++)   // (entry e is now column 8 e + l)
                    if (8 * e + l < width) atomicAdd(dst + 8 * e + l, iacc[k][e]);
            }
        }
        async_wait<0>();
        __syncthreads();
    }
}

// ------------------------------------------------------------------------------------------ rules and launches
static size_t align256(size_t v) { return (v + 255) & ~(size_t)255; }

// A pass takes as many samples as a workspace of kPassBytes (packed indices and partial sums) and kPassSamples allow, in whole
// tiles; every pass reads the tables once more.  Where not even one tile fits, the plain gather runs.  The bound lets
// the 16384 samples of 4096 detectors x 64 outputs (784 MB) through in one pass.
constexpr int64_t kPassSamples = 16384, kPassBytes = 800ll << 20;

// Where the staged gather is the better one (indices included; staged / plain, us).  A staged tile costs the same whether it
// is full or holds one sample, and grows with detectors x outputs; the plain gather pays for each sample's rows, in more blocks
// at once the wider they are, and for tables beyond L2.
// fp32, from 512 detectors on: 4096 detectors x 256 rows x 64 outputs 132 / 396 at 16 samples, 181 / 857 at 1024, 503 / 949 at
// 4096, 1650 / 2395 at 16384; 512 detectors 42 / 56, 46 / 63, 89 / 87, 216 / 245.  Rows of 32 outputs or fewer leave lanes idle
// here while the plain gather's chains get short, and more exact: they stay there; 36 outputs (two slices, the second nearly
// empty) 46 / 93 at 1 sample, 134 / 146 at 4096 with 1024 detectors.  Wide rows, few samples: 1024 detectors x 256 rows x 1024
// outputs, 1 sample 245 / 204, 64 samples 254 / 338; 512 detectors x 4096 outputs 435 / 107 at 1 sample, 452 / 370 at 256;
// 256 outputs 64 / 58 and 64 / 97 at 1 and 256 samples with 512 detectors, 93 / 107 at 1 sample with 1024; 4096 detectors x 64 rows x
// 512 outputs, 8 samples 431 / 594.  Tables in L2: 512
// detectors x 16 rows x 512 outputs 71 / 58 at 256 samples.  A little more than one wave of work items is as slow as two: 512
// detectors x 36 outputs x 4096 samples 91 / 81.
// int8, from 1024 detectors on: 4096 detectors x 64 outputs 56 / 245, 183 / 318, 540 / 812, 1857 / 2440; 1024 detectors 50 / 68,
// 67 / 81, 175 / 194, 499 / 585; 512 detectors 48 / 40, 60 / 44, 95 / 103, 300 / 298.  1024 detectors x 1024 outputs 101 / 87 at
// 1 sample, 108 / 114 at 8; x 4096 outputs 253 / 87 and 265 / 181 at 1 and 64.
constexpr int kMinOutputs = 33, kMinDetectorsFp32 = 512, kMinDetectorsInt8 = 1024;

static bool staged_fp32_pays(int64_t batch, int Nt, int T, int O) {
    const int64_t sm = device_info().sm_count;
    const int64_t items = (int64_t)((Nt + kDetBlock - 1) / kDetBlock) * ((batch + kTile - 1) / kTile) * ((O + kRow - 1) / kRow);
    if (Nt < 1024 && batch > kTile && items > sm && 2 * items < 3 * sm) return false;
    if (batch >= 512 || O <= (Nt < 1024 ? 128 : 256)) return true;
    return O <= 1024 && batch * Nt >= (Nt < 1024 && O <= 512 ? 65536 : 32768) && (int64_t)Nt * T >= 65536;
}
static bool staged_int8_pays(int64_t batch, int O) { return O <= 512 || batch >= 256 || (O <= 1024 && batch >= 8); }

size_t packed_index_pitch(int64_t batch) { return (size_t)((batch + kTile - 1) / kTile * kTile); }

static int det_blocks(int Nt) { return (Nt + kDetBlock - 1) / kDetBlock; }
static int trunc_blocks(const lutb_layer_cfg *cfg) { return (cfg->n_detectors + cfg->backward_group - 1) / cfg->backward_group; }

// bytes of the partial sums of one sample
static int64_t partial_bytes(const lutb_layer_cfg *cfg, bool int8) { return int8 ? 0 : (int64_t)det_blocks(cfg->n_detectors) * cfg->n_outputs * 4; }

// samples of one pass (batch or a multiple of kTile, the passes of one call nearly equal); 0: one tile is too much
int64_t infer_staged_pass(const lutb_layer_cfg *cfg, int64_t batch, bool int8) {
    int64_t most = kPassBytes / (cfg->n_detectors + partial_bytes(cfg, int8)) / kTile * kTile;
    if (most > kPassSamples) most = kPassSamples;
    if (most == 0 || batch <= most) return most == 0 ? 0 : batch;
    const int64_t passes = (batch + most - 1) / most, each = (batch + passes - 1) / passes;
    return (each + kTile - 1) / kTile * kTile;
}
size_t packed_index_bytes(const lutb_layer_cfg *cfg, int64_t pass) { return align256(packed_index_pitch(pass) * cfg->n_detectors); }

static size_t smem_fp32(int T) { return (size_t)kStages * 2 * ((size_t)T * kRow * 4 + kTile) + 16 * kStages + 16; }
static size_t smem_int8(int T) { return (size_t)kStages * kDets8 * ((size_t)T * kCols8 + kTile8 + 8); }

bool infer_staged_fp32_applies(const lutb_layer_cfg *cfg, int64_t batch, const void *weights, const void *y) {
    const int O = cfg->n_outputs;
    if (cfg->int_mode || cfg->n_anchors > 8 || O % 4 != 0 || O < kMinOutputs) return false;
    if (((reinterpret_cast<uintptr_t>(weights) | reinterpret_cast<uintptr_t>(y)) & 15) != 0) return false;
    return cfg->n_detectors >= kMinDetectorsFp32 && staged_fp32_pays(batch, cfg->n_detectors, 1 << cfg->n_anchors, O);
}

bool infer_staged_int8_applies(const lutb_layer_cfg *cfg, int64_t batch, const void *q_tables) {
    if (cfg->n_anchors > 8 || cfg->n_outputs % 8 != 0 || cfg->n_outputs < kMinOutputs || (reinterpret_cast<uintptr_t>(q_tables) & 7) != 0) return false;
    return cfg->n_detectors >= kMinDetectorsInt8 && staged_int8_pays(batch, cfg->n_outputs);
}

size_t anchor_plan_bytes(const lutb_layer_cfg *cfg) { return align256((size_t)cfg->n_detectors * 8 * sizeof(uint32_t)); }

size_t infer_staged_fp32_workspace(const lutb_layer_cfg *cfg, int64_t batch) {
    const int64_t pass = infer_staged_pass(cfg, batch, false);
    return pass == 0 ? 0 : packed_index_bytes(cfg, pass) + align256((size_t)(pass * partial_bytes(cfg, false))) + 256 + anchor_plan_bytes(cfg);
}
size_t infer_staged_int8_workspace(const lutb_layer_cfg *cfg, int64_t batch) {
    const int64_t pass = infer_staged_pass(cfg, batch, true);
    return pass == 0 ? 0 : packed_index_bytes(cfg, pass) + align256(scale_plan_bytes(cfg->n_detectors, trunc_blocks(cfg))) + 256 + anchor_plan_bytes(cfg);
}

int launch_infer_staged_fp32(const lutb_layer_cfg *cfg, int64_t batch, const float *weights, const uint8_t *packed, float *partial,
                             float *y, cudaStream_t stream) {
    const int O = cfg->n_outputs, T = 1 << cfg->n_anchors, nb = det_blocks(cfg->n_detectors);
    StagedFp32 p;
    p.W = weights; p.packed = packed; p.out = partial;
    p.batch = batch; p.pitch = packed_index_pitch(batch);
    p.O = O; p.Nt = cfg->n_detectors; p.T = T;
    p.n_tiles = (int)((batch + kTile - 1) / kTile);
    p.n_slices = (O + kRow - 1) / kRow;
    const int64_t items = (int64_t)nb * p.n_tiles * p.n_slices;
    LUTB_REQUIRE(items <= 0x3FFFFFFF, LUTB_ERR_SHAPE, "staged gather: too many work items");
    p.n_items = (int)items;
    const size_t smem = smem_fp32(T);
    const int blocks = p.n_items < device_info().sm_count ? p.n_items : device_info().sm_count;
    CUtensorMap tables;
    const int rc = tensor_map_2d(&tables, 4, weights, (int64_t)p.Nt * T, O, (int64_t)O * 4, T, kRow, 0);
    if (rc) return rc;
    LUTB_CUDA(cudaFuncSetAttribute(infer_staged_fp32_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    {
        KernelScope scope(K_FC_GATHER_FORWARD, stream);
        infer_staged_fp32_kernel<<<(unsigned)blocks, kStagedThreads + 32, smem, stream>>>(tables, p);
        LUTB_LAUNCH_CHECK();
    }
    const int64_t n4 = batch * O / 4;
    const int64_t want = (n4 + 255) / 256, cap = (int64_t)device_info().sm_count * 8;
    KernelScope scope(K_FC_GATHER_FORWARD, stream);
    add_partials_kernel<<<(unsigned)(want < cap ? want : cap), 256, 0, stream>>>(partial, y, n4, nb);
    LUTB_LAUNCH_CHECK();
    return LUTB_OK;
}

int launch_int8_scale_plan(const lutb_layer_cfg *cfg, const float *scales, void *scale_plan, cudaStream_t stream) {
    const int n = trunc_blocks(cfg);
    KernelScope scope(K_INT8_GATHER, stream);
    int8_scale_plan_kernel<<<(unsigned)((n + 3) / 4), 128, 0, stream>>>(scales, cfg->n_detectors, cfg->backward_group, n, scale_plan);
    LUTB_LAUNCH_CHECK();
    return LUTB_OK;
}

int launch_infer_staged_int8(const lutb_layer_cfg *cfg, int64_t batch, const int8_t *q_tables, const float *scales,
                             const void *scale_plan, const uint8_t *packed, int32_t *acc, cudaStream_t stream) {
    StagedInt8 p;
    p.Q = q_tables; p.scales = scales; p.packed = packed; p.acc = acc;
    p.plan = scale_plan_at(const_cast<void *>(scale_plan), cfg->n_detectors);
    p.batch = batch; p.pitch = packed_index_pitch(batch);
    p.O = cfg->n_outputs; p.Nt = cfg->n_detectors; p.T = 1 << cfg->n_anchors;
    p.n_tiles = (int)((batch + kTile8 - 1) / kTile8);
    p.n_slices = (p.O + kCols8 - 1) / kCols8;
    p.det_block = cfg->backward_group;
    p.fixed_scale = cfg->int_rescaler;
    p.wide = p.O % 16 == 0 && (reinterpret_cast<uintptr_t>(q_tables) & 15) == 0;
    // runs of whole truncation blocks, short enough that the last wave of items is a small part of the work
    const int blocks_all = trunc_blocks(cfg);
    const int64_t per = (int64_t)p.n_tiles * p.n_slices;
    int64_t runs = (8 * (int64_t)device_info().sm_count + per - 1) / per;
    if (runs > blocks_all) runs = blocks_all;
    const int64_t run = (int64_t)((blocks_all + runs - 1) / runs) * p.det_block;
    p.dets_per_item = (int)(run < p.Nt ? run : p.Nt);
    const int64_t items = per * ((p.Nt + p.dets_per_item - 1) / p.dets_per_item);
    LUTB_REQUIRE(items <= 0x3FFFFFFF, LUTB_ERR_SHAPE, "staged gather: too many work items");
    p.n_items = (int)items;
    const size_t smem = smem_int8(p.T);
    const int blocks = p.n_items < device_info().sm_count ? p.n_items : device_info().sm_count;
    for (auto kern : {infer_staged_int8_kernel<false>, infer_staged_int8_kernel<true>}) {
        LUTB_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
        KernelScope scope(K_INT8_GATHER, stream);
        kern<<<(unsigned)blocks, kStagedThreads, smem, stream>>>(p);
        LUTB_LAUNCH_CHECK();
    }
    return LUTB_OK;
}

}  // namespace lutb
