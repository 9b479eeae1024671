// Histogram formulation of the product-mode sequence layer (see product_hist.cuh).
//
// Reference semantics: fill_outputs_product_cpu_logic (lut_runtime_kernels_logic.proto:2148-2264),
// propagate_backward_product_cpu_logic (:2396-2628), gather_w_gradients_internal_product_cpu_logic (:2630-2744).
#include <type_traits>

#include "product_hist.cuh"
#include "hist_gemm_sm100.cuh"
#include "product_pairs.cuh"

namespace lutb {

// --------------------------------------------------------------------------------------------
// What the histogram and the routing kernel share: the detector's anchors sorted by what they compare.  An anchor pair
// reads two elements of [x_i | x_j | pe(j - i - 1)], key token i and query token j.
// --------------------------------------------------------------------------------------------
constexpr int kHistAnchors = 12;   // anchors per detector on the histogram path (tables of at most 4096 rows)

struct AnchorLists {
    int comp[2 * kHistAnchors], elem[2 * kHistAnchors];
    int kq_pos[kHistAnchors];      // slot of a key-query anchor, -1: another kind
    int pe_k[kHistAnchors];        // anchors with a positional end
    int n_kq, n_pe;
    uint32_t query_only, key_only, pe_mask;   // bit k set: anchor k is of that kind
    // staged operands of the positional anchors: end e of anchor m is smem[at.x + i * at.y + q * at.z] for key i and query
    // q as the kernel counts them, or (at.w) the query's staged end at.x
    int4 pe_at[2 * kHistAnchors];
};

__device__ __forceinline__ void list_anchors(AnchorLists &al, const int32_t *__restrict__ anchors_t, int n_anchors, bool sliced,
                                             int e1, int e2) {
    if (threadIdx.x < 32) {   // lane k: anchor k
        const int k = threadIdx.x;
        int c[2] = {3, 3}, e[2] = {0, 0};
        if (k < n_anchors) {
            decode_anchor(__ldg(anchors_t + 2 * k), sliced, e1, e2, c[0], e[0]);
            decode_anchor(__ldg(anchors_t + 2 * k + 1), sliced, e1, e2, c[1], e[1]);
        }
        const bool used = c[0] != 3 && c[1] != 3, pe = used && (c[0] == 2 || c[1] == 2);
        const bool kq = used && !pe && c[0] != c[1];
        const unsigned pe_m = __ballot_sync(0xffffffffu, pe), kq_m = __ballot_sync(0xffffffffu, kq);
        const unsigned ko_m = __ballot_sync(0xffffffffu, used && !pe && !kq && c[0] == 0);
        const unsigned qo_m = __ballot_sync(0xffffffffu, used && !pe && !kq && c[0] == 1);
        const unsigned below = (1u << k) - 1u;
        if (k < kHistAnchors) {
            al.comp[2 * k] = c[0]; al.comp[2 * k + 1] = c[1];
            al.elem[2 * k] = e[0]; al.elem[2 * k + 1] = e[1];
            al.kq_pos[k] = kq ? __popc(kq_m & below) : -1;
            if (pe) al.pe_k[__popc(pe_m & below)] = k;
        }
        if (k == 0) {
            al.n_kq = __popc(kq_m);
            al.n_pe = __popc(pe_m);
            al.pe_mask = pe_m; al.key_only = ko_m; al.query_only = qo_m;
        }
    }
    __syncthreads();
}

// key > query with the dead band.  Without one the comparison of the operands is the comparison of their difference with
// zero (subnormals are kept; equal infinities and NaN give false both ways).
template <bool EPS>
__device__ __forceinline__ bool above(float a, float b, float cmp_eps) {
    return EPS ? greater_than_zero(__fsub_rn(a, b), cmp_eps) : a > b;
}

// Operands of query j0 + q, anchor k (each thread takes some (q, k)): the query end of key-query anchors (negated where
// it comes first: every delta is then key minus query) with the anchor's bit, the whole delta of query-only ones, the
// query end of positional ones.
__device__ __forceinline__ void stage_query(const AnchorLists &al, float2 *qv, float *qd, const float *__restrict__ xq, int q, int k) {
    const int slot = al.kq_pos[k];
    const int c0 = al.comp[2 * k], c1 = al.comp[2 * k + 1];
    if (c0 != 1 && c1 != 1) return;
    const float v0 = c0 == 1 ? __ldg(xq + al.elem[2 * k]) : 0.f, v1 = c1 == 1 ? __ldg(xq + al.elem[2 * k + 1]) : 0.f;
    if (slot >= 0) qv[q * kHistAnchors + slot] = make_float2(c0 == 1 ? -v0 : v1, __uint_as_float(1u << k));
    else if ((al.query_only >> k) & 1u) qd[q * kHistAnchors + k] = __fsub_rn(v0, v1);
    else qd[q * kHistAnchors + k] = c0 == 1 ? v0 : v1;
}

// The two ends of positional anchor m: staged, or (anchors past the staged ones) from global memory.  i, q: key and query
// as the kernel counts them for its staged operands; qd_row: the query's staged ends.
__device__ __forceinline__ void positional_ends(const AnchorLists &al, const float *smem, const float *qd_row, int m, bool staged,
                                                int i, int q, const float *__restrict__ xk, const float *__restrict__ xq,
                                                const float *__restrict__ pe_d, float &v0, float &v1) {
    if (staged) {
        const int4 a = al.pe_at[2 * m], b = al.pe_at[2 * m + 1];
        v0 = (a.w ? qd_row : smem)[a.x + i * a.y + q * a.z];
        v1 = (b.w ? qd_row : smem)[b.x + i * b.y + q * b.z];
        return;
    }
    const int k = al.pe_k[m];
    const int c0 = al.comp[2 * k], c1 = al.comp[2 * k + 1];
    v0 = __ldg((c0 == 0 ? xk : c0 == 1 ? xq : pe_d) + al.elem[2 * k]);
    v1 = __ldg((c1 == 0 ? xk : c1 == 1 ? xq : pe_d) + al.elem[2 * k + 1]);
}

// --------------------------------------------------------------------------------------------
// Row-selection histogram: for every query (b, j) and detector t, how many of the j keys select each of the T rows.
// Block = (detector, 32 to 128 queries, sequence); what the pairs need of the keys is staged once, then the warps work on their
// own: a warp takes four queries at a time, counts in a private shared-memory array and writes it out.  LANE = KEY: the
// key ends of 32 keys are in registers while the warp walks its queries, whose operands (two anchors' query ends and
// bits per 16-byte load) are the same for all lanes; a key-query anchor then costs a compare and a predicated OR.  The
// loop over the anchors is unrolled for their number (NKQ), so that the four queries overlap.
// HALF_ROWS: the counters are written as fp16 (exact: counts are below 2048 there) in the layout [row of the chunk = local
// sequence * S + j][detector][T], the operand layout of the tensor-core contractions (one plain GEMM over all detectors per
// pass); otherwise as uint16 in the layout [detector][row of the chunk][T].
// PER: counters per 32-bit word, four for sequences of at most 256 tokens (a count is at most S - 1), else two.
// Bound: load/store wavefronts and issue, and at 256-row tables the 537 MB of counters it writes.  Measured (before: lanes over the
// keys of one query, the anchors' operands read from shared memory for every pair): 64 sequences x 128 tokens, 64 detectors of
// 256 rows 271 -> 195 us; 1 x 1024 tokens, 64 detectors of 1024 rows 844 -> 173 us.  Then, with bytes or pairs of counters instead of
// words, fp16 without conversion instructions, blocks of one detector together (as in product_route_kernel) and more blocks of fewer
// warps: 195 -> 174 us; 4 x 256 tokens, 64 detectors of 1024 rows 100 -> 65; 4 x 200, 40 of 512 rows 51 -> 30; 2 x 512, 64 of 256
// rows 90 -> 79; 1 x 1024 172.
// --------------------------------------------------------------------------------------------
constexpr int kHistTile = 4;

struct HistArgs {
    int sequences;   // of the chunk
    const float *x1, *x2, *pe;
    const int32_t *anchors;
    void *H;
    int64_t b0, chunk_rows;
    int S, e1, e2, npe, n_detectors, n_anchors, sliced;
    float cmp_eps;
    int pe_cap;      // anchors with a positional end whose operands are staged in shared memory
    int queries;     // of one block
};

// dynamic shared memory of one block, in floats: per warp counters and query operands | key ends | key bits | positional operands
__host__ __device__ inline size_t hist_warp_floats(int T, int per_word) {
    return (size_t)kHistTile * T / per_word + kHistTile * kHistAnchors * 3;
}
__host__ __device__ inline size_t hist_floats(int T, int per_word, int warps, int n_anchors, int pe_cap, int S) {
    const int Sp = (S + 31) & ~31;
    return warps * hist_warp_floats(T, per_word) + (size_t)(n_anchors + 1 + 3 * pe_cap) * Sp;
}

template <int PER>
__device__ __forceinline__ void count_row(uint32_t *hist, uint32_t li) {
    if (PER == 4) atomicAdd(hist + (li >> 2), 1u << ((li & 3u) * 8u));
    else atomicAdd(hist + (li >> 1), 1u << ((li & 1u) * 16u));
}

// Two counts below 2048 in the halves of c, as fp16: 1024 + the lower ten bits is 0x6400 with these bits behind it, bit 10 is worth
// 1024 = 0x6400 = 25 * 0x400 itself; exact.  (A conversion instruction takes eight times as long as these.)
template <bool TEN_BITS>
__device__ __forceinline__ uint32_t half_counts(uint32_t c) {
    const uint32_t lower = TEN_BITS ? c | 0x64006400u : (c & 0x03ff03ffu) | 0x64006400u, upper = (c & 0x04000400u) * 25u;
    __half2 h = __hsub2(*reinterpret_cast<const __half2 *>(&lower), __half2half2(__ushort_as_half((unsigned short)0x6400)));
    if (!TEN_BITS) h = __hadd2(h, *reinterpret_cast<const __half2 *>(&upper));
    return *reinterpret_cast<const uint32_t *>(&h);
}

struct HistTile {
    const float *smem, *ks, *qd, *x1b, *x2b, *pe_t;   // pe_t: embeddings of the block's detector
    const uint32_t *kb_s;
    uint32_t *hist;
    const float2 *qv;
    int Sp, j0, nq, n_kq, n_pe, pe_stride;
};

// counts the keys of queries j0 .. j0 + nq - 1
template <int NKQ, bool PE, bool EPS, int PER>
__device__ __forceinline__ void count_tile(const HistArgs &p, const AnchorLists &al, const HistTile &h, uint32_t qbits) {
    const int lane = threadIdx.x & 31;
    const int T = 1 << p.n_anchors, words = T / PER;
    for (int i0 = 0; i0 < h.j0 + h.nq - 1; i0 += 32) {
        const int i = i0 + lane;
        float kv[NKQ > 0 ? NKQ : 1];
#pragma unroll
        for (int m = 0; m < NKQ; m++) kv[m] = m < h.n_kq ? h.ks[m * h.Sp + i] : 0.f;
        const uint32_t kbits = h.kb_s[i];
#pragma unroll
        for (int q = 0; q < kHistTile; q++) {
            const int j = h.j0 + q;
            uint32_t li = kbits | __shfl_sync(0xffffffffu, qbits, q);
            const float4 *qv4 = reinterpret_cast<const float4 *>(h.qv + q * kHistAnchors);
#pragma unroll
            for (int m = 0; m < NKQ; m += 2) {
                const float4 f = qv4[m / 2];
                if (above<EPS>(kv[m], f.x, p.cmp_eps)) li |= __float_as_uint(f.y);
                if (above<EPS>(kv[m + 1], f.z, p.cmp_eps)) li |= __float_as_uint(f.w);
            }
            if (i < j && q < h.nq) {
                if (PE) {
                    for (int m = 0; m < h.n_pe; m++) {
                        float v0, v1;
                        positional_ends(al, h.smem, h.qd + q * kHistAnchors, m, m < p.pe_cap, i, j, h.x1b + (size_t)i * p.e1, h.x2b + (size_t)j * p.e2,
                                        h.pe_t + (size_t)(j - i - 1) * h.pe_stride, v0, v1);
                        if (above<EPS>(v0, v1, p.cmp_eps)) li |= 1u << al.pe_k[m];
                    }
                }
                count_row<PER>(h.hist + q * words, li);
            }
        }
    }
}

template <int MAXKQ, bool EPS, bool HALF_ROWS, int PER>
__global__ void __launch_bounds__(512, 2) product_hist_kernel(const HistArgs p) {
    extern __shared__ __align__(16) float smem[];
    __shared__ AnchorLists al;
    // blocks of one detector run together, see product_route_kernel
    const int t = blockIdx.x / p.sequences;
    const int j_begin = (gridDim.y - 1 - blockIdx.y) * p.queries;   // the ranges with the most keys first
    const int64_t bl = blockIdx.x - t * p.sequences, b = p.b0 + bl;
    const int S = p.S, Nc = p.n_anchors, T = 1 << Nc, Sp = (S + 31) & ~31;
    const int j_end = min(S, j_begin + p.queries);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, nwarps = blockDim.x >> 5;
    const int words = T / PER;
    const size_t per_warp = hist_warp_floats(T, PER);
    uint32_t *hist = reinterpret_cast<uint32_t *>(smem + warp * per_warp);          // [kHistTile][words]
    float2 *qv = reinterpret_cast<float2 *>(hist + kHistTile * words);             // [kHistTile][kHistAnchors] (query end, bit)
    float *qd = reinterpret_cast<float *>(qv + kHistTile * kHistAnchors);          // [kHistTile][kHistAnchors]
    float *ks = smem + nwarps * per_warp;                                          // [Nc][Sp] key ends of the key-query anchors
    uint32_t *kb_s = reinterpret_cast<uint32_t *>(ks + Nc * Sp);                   // [Sp] bits of the key-only anchors
    float *kpe = reinterpret_cast<float *>(kb_s + Sp);                             // [pe_cap][Sp] key ends of the positional anchors
    float *pes = kpe + p.pe_cap * Sp;                                              // [2 * pe_cap][Sp] positional ends by distance
    list_anchors(al, p.anchors + (size_t)t * Nc * 2, Nc, p.sliced != 0, p.e1, p.e2);
    const int n_kq = al.n_kq, n_pe = al.n_pe;

    for (int w = lane; w < kHistTile * words; w += 32) hist[w] = 0u;
    // slots past the last key-query anchor: a NaN compares false everywhere
    for (int w = lane; w < kHistTile * kHistAnchors; w += 32) qv[w] = make_float2(__int_as_float(0x7fffffff), 0.f);
    const float *x1b = p.x1 + (size_t)b * S * p.e1, *x2b = p.x2 + (size_t)b * S * p.e2;
    for (int k = warp; k <= Nc; k += nwarps) {   // one warp per anchor; the key bits last
        if (k == Nc) {
            for (int i = lane; i < j_end; i += 32) {
                uint32_t bits = 0u;
                for (uint32_t left = al.key_only; left; left &= left - 1) {
                    const int a = __ffs(left) - 1;
                    if (above<EPS>(__ldg(x1b + (size_t)i * p.e1 + al.elem[2 * a]), __ldg(x1b + (size_t)i * p.e1 + al.elem[2 * a + 1]), p.cmp_eps)) bits |= 1u << a;
                }
                kb_s[i] = bits;
            }
            continue;
        }
        const int slot = al.kq_pos[k], c0 = al.comp[2 * k];
        if (slot < 0) continue;
        const float *src = x1b + al.elem[2 * k + (c0 == 0 ? 0 : 1)];
#pragma unroll 4
        for (int i = lane; i < j_end; i += 32) {
            const float v = __ldg(src + (size_t)i * p.e1);
            ks[slot * Sp + i] = c0 == 0 ? v : -v;
        }
    }
    for (int m = 0; m < min(n_pe, p.pe_cap); m++) {
        const int k = al.pe_k[m];
        for (int e = 0; e < 2; e++) {
            const int c = al.comp[2 * k + e], el = al.elem[2 * k + e];
            if (c == 0)
                for (int i = threadIdx.x; i < j_end; i += blockDim.x) kpe[m * Sp + i] = __ldg(x1b + (size_t)i * p.e1 + el);
            else if (c == 2)
                for (int d = threadIdx.x; d < j_end - 1; d += blockDim.x)
                    pes[(2 * m + e) * Sp + d] = __ldg(p.pe + ((size_t)d * p.n_detectors + t) * p.npe + el);
            // (keys and queries are counted from the start of the sequence here: distance j - i - 1)
            if (threadIdx.x == 0)
                al.pe_at[2 * m + e] = c == 0 ? make_int4((int)(kpe + m * Sp - smem), 1, 0, 0)
                                    : c == 2 ? make_int4((int)(pes + (2 * m + e) * Sp - smem) - 1, -1, 1, 0)
                                             : make_int4(k, 0, 0, 1);
        }
    }
    __syncthreads();

    HistTile h;
    h.smem = smem; h.ks = ks; h.kb_s = kb_s; h.x1b = x1b; h.x2b = x2b;
    h.pe_t = p.pe + (size_t)t * p.npe;
    h.pe_stride = p.n_detectors * p.npe;
    h.hist = hist; h.qv = qv; h.qd = qd; h.Sp = Sp; h.n_kq = n_kq; h.n_pe = n_pe;
    const int tiles = (j_end - j_begin + kHistTile - 1) / kHistTile;
    for (int n = 0; n * nwarps < tiles; n++) {
        // back and forth over the warps: later tiles have more keys
        const int tile = n * nwarps + ((n & 1) ? nwarps - 1 - warp : warp);
        if (tile >= tiles) continue;
        const int j0 = j_begin + tile * kHistTile, nq = min(kHistTile, j_end - j0);
        {
            const int q = lane & (kHistTile - 1);
            if (q < nq)
                for (int k = lane / kHistTile; k < Nc; k += 32 / kHistTile) stage_query(al, qv, qd, x2b + (size_t)(j0 + q) * p.e2, q, k);
        }
        __syncwarp();
        uint32_t qbits = 0u;   // lane q: the query-only anchors of query j0 + q
        if (lane < kHistTile) {
            for (uint32_t left = al.query_only; left; left &= left - 1) {
                const int k = __ffs(left) - 1;
                if (above<EPS>(qd[lane * kHistAnchors + k], 0.f, p.cmp_eps)) qbits |= 1u << k;
            }
        }
        h.j0 = j0; h.nq = nq;
        if (EPS || n_pe > 0) count_tile<MAXKQ, true, EPS, PER>(p, al, h, qbits);
        else if (n_kq <= 2) count_tile<2, false, EPS, PER>(p, al, h, qbits);
        else if (n_kq <= 4) count_tile<4, false, EPS, PER>(p, al, h, qbits);
        else if (n_kq <= 6) count_tile<6, false, EPS, PER>(p, al, h, qbits);
        else if (MAXKQ == 8 || n_kq <= 8) count_tile<8, false, EPS, PER>(p, al, h, qbits);
        else count_tile<MAXKQ, false, EPS, PER>(p, al, h, qbits);
        __syncwarp();
        // write out and clear
        __half *out_f = static_cast<__half *>(p.H) + ((size_t)(bl * S + j0) * p.n_detectors + t) * T;
        uint16_t *out_h = static_cast<uint16_t *>(p.H) + ((size_t)t * p.chunk_rows + bl * S + j0) * T;
        for (int w = lane; w < nq * (T / 8); w += 32) {
            const int q = w >> (Nc - 3), r = w & (T / 8 - 1);
            uint4 c;   // eight 16-bit counts
            if (PER == 4) {
                uint2 *cell = reinterpret_cast<uint2 *>(hist) + w;
                const uint2 u = *cell;
                *cell = make_uint2(0u, 0u);
                c = make_uint4(__byte_perm(u.x, 0u, 0x4140), __byte_perm(u.x, 0u, 0x4342), __byte_perm(u.y, 0u, 0x4140), __byte_perm(u.y, 0u, 0x4342));
            } else {
                uint4 *cell = reinterpret_cast<uint4 *>(hist) + w;
                c = *cell;
                *cell = make_uint4(0u, 0u, 0u, 0u);
            }
            constexpr bool kTen = PER == 4;
            if (HALF_ROWS) *reinterpret_cast<uint4 *>(out_f + (size_t)q * p.n_detectors * T + r * 8) = make_uint4(half_counts<kTen>(c.x), half_counts<kTen>(c.y), half_counts<kTen>(c.z), half_counts<kTen>(c.w));
            else *reinterpret_cast<uint4 *>(out_h + (size_t)w * 8) = c;
        }
        __syncwarp();
    }
}

// --------------------------------------------------------------------------------------------
// Input-gradient routing: every pair (i, j) reads two entries of Q_t[(b,j), :] (the dot products of dY[b,j,:] with the
// rows of table t): g = Q[idx] - Q[idx ^ 2^kmin], du = up(min_delta) * g, +du / -du to the sources of the flipped
// anchor's two ends.
//
// Bound by instruction issue, so the pairs are laid out for the fewest instructions per pair.  Block = (detector, 128
// keys, sequence), four warps; LANE = KEY: a lane keeps what a pair needs of its key in registers for the whole block
// (the key ends of the anchors that compare a key with a query, the bits and smallest delta of the anchors that read
// the key alone), and the warps walk the queries above it, eight at a time.  What a pair needs of the query is the same
// for all lanes: one 16-byte shared load brings two anchors' query ends and their bits.  Values whose query end comes
// first are negated on both sides, so that every delta is key minus query.  Key-range blocks also give a single long
// sequence S / 128 times the blocks (64 detectors alone leave more than half of the SMs idle).
//
// Sums: the key's cells are a private shared-memory column per lane (plain read-modify-write), flushed once per block.
// The query's cells would collide (32 lanes, a few anchors), so a pair's (du, anchor) is parked in an 8 x 32 tile that
// the warp reads back with the lanes over queries, again into private columns; the block adds the columns up once per
// eight queries.
// Measured (before: a warp per query, about 600 instructions per 32 pairs): 64 sequences x 128 tokens, 64 detectors of 256
// rows 862 -> 490 us; 1 x 1024 tokens, 64 detectors of 1024 rows 1910 -> 435 us (851 before a block's queries were limited).
// Since then the pairs of two queries are interleaved (475 -> 438 us and 446 -> 409; four at a time 540 and 416) and the blocks
// numbered detector by detector instead of sequence by sequence (438 -> 396 and 409 -> 361: fewer blocks add to the dX of one
// sequence at a time, and fewer of the loops for different numbers of anchors run side by side; which weighs more was not
// isolated).  Slower: asking for the next tile's rows before the query cells are added up (447 -> 457), a loop for every number
// of anchors instead of every other one (438 -> 480), blocks of one detector on one SM (396 -> 421).  The rounded reciprocal of the
// surrogate takes 8 %.  Two barriers per eight queries instead of four
// gave 8 % at 128 tokens; a per-warp window of distances for dPE instead of an add per pair cost 20 % there.
// --------------------------------------------------------------------------------------------
constexpr int kRouteWarps = 4, kRouteKeys = 32 * kRouteWarps, kTileQ = 8, kRouteWindow = kRouteKeys + kTileQ;
constexpr int kExLd = 33;          // leading dimension of the (query, key) exchange tile

struct RouteArgs {
    int sequences, parts;   // sequences of the chunk; blocks per (detector, sequence)
    const float *x1, *x2, *pe;
    const int32_t *anchors;
    const float *Q;
    float *dX1, *dX2, *dPE;
    int64_t b0, q_row_stride, q_det_stride;
    int S, e1, e2, npe, n_detectors, n_anchors, sliced;
    float cmp_eps;
    int pe_cap;      // anchors with a positional end whose operands are staged in shared memory
    int pe_cells;    // 1: the block sums dPE in shared memory
    int queries;     // of one block
};

// dynamic shared memory of one block, in floats: Q rows | query operands | per-warp columns and exchange tile | staged
// positional operands | dPE cells
__host__ __device__ inline size_t route_floats(int T, int n_anchors, int pe_cap, int pe_cells, int S, int npe) {
    return (size_t)kTileQ * T + kTileQ * kHistAnchors * 3 + (size_t)kRouteWarps * (64 * n_anchors + 2 * kTileQ * kExLd) +
           (size_t)pe_cap * (kRouteKeys + 2 * kRouteWindow) + (pe_cells ? (size_t)(S - 1) * npe : 0);
}

// The running first minimum of |delta| as one ordered integer: |delta| above, the anchor below, so that "smaller, or equal
// with a smaller anchor number" is a 64-bit comparison.  It starts at FLT_MAX without an anchor; a delta that is no smaller
// (or NaN) never replaces it.  low: the anchor's bit; with a dead band, twice that plus "delta > 0" (without one, that is
// what the anchor's bit of the table index says).
__device__ __forceinline__ unsigned long long margin_key(float abs_d, uint32_t low) {
    return ((unsigned long long)__float_as_uint(abs_d) << 32) | low;
}
template <bool EPS>
__device__ __forceinline__ uint32_t margin_low(uint32_t bit, float d) {
    return EPS ? 2u * bit + (d > 0.f ? 1u : 0u) : bit;
}

struct RouteTile {
    const float *smem, *Qs, *qd, *xk, *x2b, *pe_t;
    const float2 *qv;
    float *kcol, *pacc;
    float2 *ex;
    int j0, j_end, i, ikey, n_pe, pe_stride, t;
    uint32_t pe_mask, kbits;
    unsigned long long kmin;
    // lane q < kTileQ: the query-only anchors of query j0 + q
    uint32_t qbits;
    float qmd;
    uint32_t qlow;
};

__device__ __forceinline__ void add_positional(const RouteArgs &p, float *pacc, int dist, int t, int elem, float v) {
    if (p.pe_cells) atomicAdd(pacc + dist * p.npe + elem, v);
    else atomicAdd(p.dPE + ((size_t)dist * p.n_detectors + t) * p.npe + elem, v);
}

template <int NKQ, bool PE, bool EPS, int MAXKQ>
__device__ __forceinline__ void route_tile(const RouteArgs &p, const AnchorLists &al, const RouteTile &r, const float (&kv)[MAXKQ]) {
    const int lane = threadIdx.x & 31, T = 1 << p.n_anchors;
    // the first positional anchor's operands as two addresses and steps per query (it is always staged)
    const float *end0 = nullptr, *end1 = nullptr;
    int step0 = 0, step1 = 0;
    uint32_t pe_bit = 0u;
    if (PE && r.n_pe > 0) {
        const int4 a = al.pe_at[0], b = al.pe_at[1];
        end0 = a.w ? r.qd + a.x : r.smem + a.x + r.ikey * a.y;
        end1 = b.w ? r.qd + b.x : r.smem + b.x + r.ikey * b.y;
        step0 = a.w ? kHistAnchors : a.z;
        step1 = b.w ? kHistAnchors : b.z;
        pe_bit = 1u << al.pe_k[0];
    }
    // Two queries at a time, in three phases: both table rows' entries are asked for before the first reciprocal, and both key
    // cells are read before either is written (the compiler may not move a load across a store of shared memory itself).
    constexpr int U = 2;
#pragma unroll 1
    for (int q0 = 0; q0 < kTileQ; q0 += U) {
        float dus[U], slopes[U], halves[U];
        int offs[U];
#pragma unroll
        for (int u = 0; u < U; u++) {
            const int q = q0 + u, j = r.j0 + q;
            uint32_t li = r.kbits | __shfl_sync(0xffffffffu, r.qbits, q);
            unsigned long long best = margin_key(__shfl_sync(0xffffffffu, r.qmd, q), __shfl_sync(0xffffffffu, r.qlow, q));
            best = r.kmin < best ? r.kmin : best;
            if (NKQ > 0) {
                // anchor numbers ascend: strictly smaller is enough inside this group
                float md = kFltMax;
                uint32_t low = 0u;
                const float4 *qv4 = reinterpret_cast<const float4 *>(r.qv + q * kHistAnchors);
#pragma unroll
                for (int m = 0; m < NKQ; m += 2) {
                    const float4 f = qv4[m / 2];
                    const float da = __fsub_rn(kv[m], f.x), db = __fsub_rn(kv[m + 1], f.z);
                    const uint32_t ba = __float_as_uint(f.y), bb = __float_as_uint(f.w);
                    if (EPS ? greater_than_zero(da, p.cmp_eps) : da > 0.f) li |= ba;
                    if (fabsf(da) < md) { md = fabsf(da); low = margin_low<EPS>(ba, da); }
                    if (EPS ? greater_than_zero(db, p.cmp_eps) : db > 0.f) li |= bb;
                    if (fabsf(db) < md) { md = fabsf(db); low = margin_low<EPS>(bb, db); }
                }
                const unsigned long long mixed = margin_key(md, low);
                best = mixed < best ? mixed : best;
            }
            const bool pair = r.i < j && j < r.j_end;
            const int dist = max(0, min(j, p.S - 1) - r.i - 1);
            if (PE && r.n_pe > 0) {
                {
                    const float d = __fsub_rn(end0[q * step0], end1[q * step1]);
                    if (EPS ? greater_than_zero(d, p.cmp_eps) : d > 0.f) li |= pe_bit;
                    const unsigned long long c = margin_key(fabsf(d), margin_low<EPS>(pe_bit, d));
                    best = c < best ? c : best;
                }
                for (int m = 1; m < r.n_pe; m++) {
                    float v0, v1;
                    positional_ends(al, r.smem, r.qd + q * kHistAnchors, m, m < p.pe_cap, r.ikey, q, r.xk,
                                    r.x2b + (size_t)min(j, p.S - 1) * p.e2, r.pe_t + (size_t)dist * r.pe_stride, v0, v1);
                    const uint32_t bit = 1u << al.pe_k[m];
                    const float d = __fsub_rn(v0, v1);
                    if (EPS ? greater_than_zero(d, p.cmp_eps) : d > 0.f) li |= bit;
                    const unsigned long long c = margin_key(fabsf(d), margin_low<EPS>(bit, d));
                    best = c < best ? c : best;
                }
            }
            const float md = __uint_as_float((uint32_t)(best >> 32));
            const uint32_t low = (uint32_t)best, bit = EPS ? low >> 1 : low;
            const bool positive = EPS ? (low & 1u) != 0u : (li & bit) != 0u;
            // up(d) * (Q[row] - Q[flipped row]) in fp32: Q is an fp32 contraction already (the direct kernels and the
            // fixed-point mode keep the double-precision reciprocal of the reference's formula)
            const float *qrow = r.Qs + q * T;
            slopes[u] = 1.0f + md;
            dus[u] = qrow[li] - qrow[li ^ bit];
            halves[u] = pair && bit != 0u ? (positive ? 0.5f : -0.5f) : 0.f;
            offs[u] = bit ? (31 - __clz(bit)) * 32 : 0;
        }
#pragma unroll
        for (int u = 0; u < U; u++) {
            const float rc = __frcp_rn(slopes[u]);
            const float du = halves[u] * rc * rc * dus[u];
            dus[u] = halves[u] != 0.f && fabsf(du) > kEpsF ? du : 0.f;
        }
        static_assert(U == 2);
        {   // both cells are read before either is written
            float c0 = r.kcol[offs[0] + lane], c1 = r.kcol[offs[1] + lane];
            c0 += dus[0];
            c1 = (offs[1] == offs[0] ? c0 : c1) + dus[1];
            r.kcol[offs[0] + lane] = c0;
            r.kcol[offs[1] + lane] = c1;
        }
#pragma unroll
        for (int u = 0; u < U; u++) {
            const int q = q0 + u, off = offs[u];
            const float du = dus[u];
            r.ex[q * kExLd + lane] = make_float2(du, __int_as_float(off));
            if (PE && r.n_pe > 0) {
                // (du is zero where there is no pair or no anchor)
                const int k = off / 32;
                if (((r.pe_mask >> k) & 1u) && du != 0.f) {
                    const int dist = max(0, min(r.j0 + q, p.S - 1) - r.i - 1);
#pragma unroll
                    for (int e = 0; e < 2; e++) {
                        if (al.comp[2 * k + e] == 2)
                            add_positional(p, r.pacc, dist, r.t, al.elem[2 * k + e], e == 0 ? du : -du);
                    }
                }
            }
        }
    }
}

template <int MAXKQ, bool EPS>
__global__ void __launch_bounds__(32 * kRouteWarps, MAXKQ <= 8 ? 8 : 7) product_route_kernel(const RouteArgs p) {
    extern __shared__ __align__(16) float smem[];
    __shared__ AnchorLists al;
    const int place = blockIdx.x / p.sequences, t = place / p.parts, part = place - t * p.parts;
    // a part: (segment of p.queries queries, key range); the later key ranges have fewer segments
    const int n_ranges = (p.S - 1 + kRouteKeys - 1) / kRouteKeys;
    const int seg = part / n_ranges, k0 = (part - seg * n_ranges) * kRouteKeys;
    const int j_begin = k0 + 1 + seg * p.queries, j_end = min(p.S, j_begin + p.queries);
    if (j_begin >= p.S) return;
    const int64_t bl = blockIdx.x - place * p.sequences, b = p.b0 + bl;
    const int S = p.S, Nc = p.n_anchors, T = 1 << Nc;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    float *Qs = smem;                                             // [kTileQ][T]
    float2 *qv = reinterpret_cast<float2 *>(Qs + kTileQ * T);     // [kTileQ][kHistAnchors] (query end, anchor bit)
    float *qd = reinterpret_cast<float *>(qv + kTileQ * kHistAnchors);   // [kTileQ][kHistAnchors] see stage_query
    float *cols = qd + kTileQ * kHistAnchors;                     // per warp: [Nc][32] key cells, [Nc][32] query cells
    float *kcol = cols + warp * 64 * Nc, *qcol = kcol + 32 * Nc;
    float *rest = cols + kRouteWarps * 64 * Nc;
    float2 *ex = reinterpret_cast<float2 *>(rest) + warp * kTileQ * kExLd;   // [kTileQ][kExLd] (du, column offset)
    float *kpe = rest + kRouteWarps * 2 * kTileQ * kExLd;         // [pe_cap][kRouteKeys] key ends of the positional anchors
    float *pew = kpe + p.pe_cap * kRouteKeys;                     // [2 * pe_cap][kRouteWindow] their positional ends
    float *pacc = pew + 2 * p.pe_cap * kRouteWindow;              // [S-1][npe]
    list_anchors(al, p.anchors + (size_t)t * Nc * 2, Nc, p.sliced != 0, p.e1, p.e2);
    const int n_kq = al.n_kq, n_pe = al.n_pe, n_staged = min(n_pe, p.pe_cap);

    for (int w = lane; w < 64 * Nc; w += 32) kcol[w] = 0.f;
    if (p.pe_cells)
        for (int w = threadIdx.x; w < (S - 1) * p.npe; w += blockDim.x) pacc[w] = 0.f;
    // query slots past the last key-query anchor: a NaN compares false everywhere
    for (int w = threadIdx.x; w < kTileQ * kHistAnchors; w += blockDim.x) qv[w] = make_float2(__int_as_float(0x7fffffff), 0.f);

    // this lane's key
    const int ikey = threadIdx.x, i = k0 + ikey;
    const float *xk = p.x1 + ((size_t)b * S + min(i, S - 1)) * p.e1;
    float kv[MAXKQ];
#pragma unroll
    for (int m = 0; m < MAXKQ; m++) kv[m] = 0.f;
    uint32_t kbits = 0u;
    unsigned long long kmin = margin_key(kFltMax, 0u);
    for (int k = 0; k < Nc; k++) {
        const int c0 = al.comp[2 * k];
        const int slot = al.kq_pos[k];
        if (slot >= 0) {
            const float v = c0 == 0 ? __ldg(xk + al.elem[2 * k]) : -__ldg(xk + al.elem[2 * k + 1]);
#pragma unroll
            for (int m = 0; m < MAXKQ; m++)
                if (m == slot) kv[m] = v;
        } else if ((al.key_only >> k) & 1u) {
            const float d = __fsub_rn(__ldg(xk + al.elem[2 * k]), __ldg(xk + al.elem[2 * k + 1]));
            if (greater_than_zero(d, p.cmp_eps)) kbits |= 1u << k;
            const unsigned long long c = margin_key(fabsf(d), margin_low<EPS>(1u << k, d));
            kmin = c < kmin ? c : kmin;
        }
    }
    for (int m = 0; m < n_staged; m++) {
        const int k = al.pe_k[m];
        for (int e = 0; e < 2; e++) {
            const int c = al.comp[2 * k + e];
            if (c == 0) kpe[m * kRouteKeys + ikey] = __ldg(xk + al.elem[2 * k + e]);
            // (keys are counted from the block's first, queries from the tile's: window entry q - i + kRouteKeys - 1)
            if (threadIdx.x == 0)
                al.pe_at[2 * m + e] = c == 0 ? make_int4((int)(kpe + m * kRouteKeys - smem), 1, 0, 0)
                                    : c == 2 ? make_int4((int)(pew + (2 * m + e) * kRouteWindow - smem) + kRouteKeys - 1, -1, 1, 0)
                                             : make_int4(k, 0, 0, 1);
        }
    }

    RouteTile r;
    r.smem = smem; r.Qs = Qs; r.qd = qd; r.xk = xk; r.qv = qv;
    r.x2b = p.x2 + (size_t)b * S * p.e2;
    r.pe_t = p.pe + (size_t)t * p.npe;
    r.pe_stride = p.n_detectors * p.npe;
    r.kcol = kcol; r.pacc = pacc; r.ex = ex;
    r.j_end = j_end;
    r.i = i; r.ikey = ikey; r.n_pe = n_pe; r.t = t;
    r.pe_mask = al.pe_mask;
    r.kbits = kbits; r.kmin = kmin;
    const float *Qt = p.Q + (size_t)t * p.q_det_stride + (size_t)bl * S * p.q_row_stride;
    __syncthreads();
    for (int j0 = j_begin; j0 < j_end; j0 += kTileQ) {
        const int nq = min(kTileQ, j_end - j0);
        // (every warp has passed the barrier behind the previous tile's pairs: its operands are free)
        for (int w = threadIdx.x; w < nq * (T / 4); w += blockDim.x) {
            const int q = w >> (Nc - 2), c = w & (T / 4 - 1);
            const uint32_t dst = (uint32_t)__cvta_generic_to_shared(Qs + w * 4);
            asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(Qt + (size_t)(j0 + q) * p.q_row_stride + c * 4) : "memory");
        }
        {
            const int q = threadIdx.x & (kTileQ - 1), k = threadIdx.x / kTileQ;
            if (k < Nc && q < nq) stage_query(al, qv, qd, r.x2b + (size_t)(j0 + q) * p.e2, q, k);
        }
        // positional ends of the distances between the tile's queries and the block's keys: entry w holds distance
        // j0 - k0 - kRouteKeys + w
        for (int m = 0; m < 2 * n_staged; m++) {
            const int end = 2 * al.pe_k[m >> 1] + (m & 1);
            if (al.comp[end] != 2) continue;
            for (int w = threadIdx.x; w < kRouteWindow; w += blockDim.x) {
                const int dist = j0 - k0 - kRouteKeys + w;
                if (dist >= 0 && dist < S - 1) pew[m * kRouteWindow + w] = __ldg(r.pe_t + (size_t)dist * r.pe_stride + al.elem[end]);
            }
        }
        asm volatile("cp.async.wait_all;" ::: "memory");
        __syncthreads();
        if (k0 + warp * 32 < j0 + nq - 1) {   // (otherwise no key of this warp lies below any of the queries)
            r.j0 = j0;
            r.qbits = 0u;
            unsigned long long best = margin_key(kFltMax, 0u);
            if (lane < kTileQ) {
                for (uint32_t left = al.query_only; left; left &= left - 1) {
                    const int k = __ffs(left) - 1;
                    const float d = qd[lane * kHistAnchors + k];
                    if (greater_than_zero(d, p.cmp_eps)) r.qbits |= 1u << k;
                    const unsigned long long c = margin_key(fabsf(d), margin_low<EPS>(1u << k, d));
                    best = c < best ? c : best;
                }
            }
            r.qmd = __uint_as_float((uint32_t)(best >> 32));
            r.qlow = (uint32_t)best;
            if (EPS || n_pe > 0) {
                if (MAXKQ > 8 && !EPS && n_kq <= 6) route_tile<6, true, EPS, MAXKQ>(p, al, r, kv);
                else route_tile<MAXKQ, true, EPS, MAXKQ>(p, al, r, kv);
            } else if (n_kq <= 4) route_tile<4, false, EPS, MAXKQ>(p, al, r, kv);
            else if (n_kq <= 6) route_tile<6, false, EPS, MAXKQ>(p, al, r, kv);
            else route_tile<MAXKQ, false, EPS, MAXKQ>(p, al, r, kv);
            __syncwarp();
            // lanes over (query, quarter of the keys)
            const float2 *mine = ex + (lane & (kTileQ - 1)) * kExLd + (lane / kTileQ) * kTileQ;
#pragma unroll
            for (int n = 0; n < 8; n += 2) {
                const float2 v = mine[n], w = mine[n + 1];
                const int o0 = __float_as_int(v.y) + lane, o1 = __float_as_int(w.y) + lane;
                float c0 = qcol[o0], c1 = qcol[o1];
                c0 += v.x;
                c1 = (o1 == o0 ? c0 : c1) + w.x;
                qcol[o0] = c0;
                qcol[o1] = c1;
            }
        }
        __syncthreads();
        // add up the query cells: 4 warps x 4 quarters per (query, anchor)
        const int q = threadIdx.x & (kTileQ - 1);
        for (int k = threadIdx.x / kTileQ; k < Nc; k += 4 * kRouteWarps) {
            float s = 0.f;
#pragma unroll
            for (int w = 0; w < kRouteWarps; w++)
#pragma unroll
                for (int h = 0; h < 4; h++) {
                    float *c = cols + w * 64 * Nc + 32 * Nc + k * 32 + q + 8 * ((h + k) & 3);
                    s += *c;
                    *c = 0.f;
                }
            if (j0 + q < S && s != 0.f) {
#pragma unroll
                for (int e = 0; e < 2; e++)
                    if (al.comp[2 * k + e] == 1) atomicAdd(p.dX2 + ((size_t)b * S + j0 + q) * p.e2 + al.elem[2 * k + e], e == 0 ? s : -s);
            }
        }
    }
    if (i < S) {
        for (int k = 0; k < Nc; k++) {
            const float s = kcol[k * 32 + lane];
            if (s == 0.f) continue;
#pragma unroll
            for (int e = 0; e < 2; e++)
                if (al.comp[2 * k + e] == 0) atomicAdd(p.dX1 + ((size_t)b * S + i) * p.e1 + al.elem[2 * k + e], e == 0 ? s : -s);
        }
    }
    if (p.pe_cells) {
        __syncthreads();
        for (int w = threadIdx.x; w < (S - 1) * p.npe; w += blockDim.x) {
            const float v = pacc[w];
            if (v == 0.f) continue;
            const int d = w / p.npe, c = w - d * p.npe;
            atomicAdd(p.dPE + ((size_t)d * p.n_detectors + t) * p.npe + c, v);
        }
    }
}

// --------------------------------------------------------------------------------------------
// Register-tiled fp32 contraction  C[z] (+)= alpha * A[z] . B[z]  on 128 x 128 x 16 tiles: 256 threads, an
// 8 x 8 accumulator block per thread (updated with packed two-wide fp32 FMAs), operands staged k-major in shared
// memory ([k][m] and [k][n]) so the inner loop reads them with 16-byte loads, the next tile prefetched into registers while the current one is
// consumed.  Operand sources come in two layouts: "k contiguous" (element (m, k) at m * ld + k) and "row of k"
// (element (m, k) at k * ld + m); A may hold uint16 counters.
// --------------------------------------------------------------------------------------------
constexpr int GM = 128, GK = 16, GLD = GM + 4;

enum OperandKind { KC_F32, KC_U16, RK_F32, RK_U16 };

struct Frag { uint4 r[2]; };

// Loads this thread's part of the tile rows [m0, m0+128) x k [k0, k0+16); out-of-range parts read as zero.
template <int KIND>
__device__ __forceinline__ void fetch_tile(Frag &f, const void *base, int64_t ld, int m0, int M, int k0, int K) {
    const int tid = threadIdx.x;
    f.r[0] = make_uint4(0u, 0u, 0u, 0u);
    f.r[1] = make_uint4(0u, 0u, 0u, 0u);
    if (KIND == KC_F32) {
        const float *p = static_cast<const float *>(base);
        const int k = k0 + (tid & 3) * 4;
#pragma unroll
        for (int h = 0; h < 2; h++) {
            const int m = m0 + (tid >> 2) + h * 64;
            if (m < M && k < K) f.r[h] = __ldg(reinterpret_cast<const uint4 *>(p + (int64_t)m * ld + k));
        }
    } else if (KIND == KC_U16) {
        const uint16_t *p = static_cast<const uint16_t *>(base);
        // a warp takes 32 consecutive rows of one k-half: its transposed stores then fall into 32 different banks
        const int m = m0 + (tid & 127), k = k0 + (tid >> 7) * 8;
        if (m < M && k < K) f.r[0] = __ldg(reinterpret_cast<const uint4 *>(p + (int64_t)m * ld + k));
    } else if (KIND == RK_F32) {
        const float *p = static_cast<const float *>(base);
        const int m = m0 + (tid & 31) * 4;
#pragma unroll
        for (int h = 0; h < 2; h++) {
            const int k = k0 + (tid >> 5) + h * 8;
            if (m < M && k < K) f.r[h] = __ldg(reinterpret_cast<const uint4 *>(p + (int64_t)k * ld + m));
        }
    } else {
        const uint16_t *p = static_cast<const uint16_t *>(base);
        const int m = m0 + (tid & 15) * 8, k = k0 + (tid >> 4);
        if (m < M && k < K) f.r[0] = __ldg(reinterpret_cast<const uint4 *>(p + (int64_t)k * ld + m));
    }
}

__device__ __forceinline__ float lo16(uint32_t v) { return (float)(v & 0xffffu); }
__device__ __forceinline__ float hi16(uint32_t v) { return (float)(v >> 16); }

template <int KIND>
__device__ __forceinline__ void stash_tile(const Frag &f, float (*tile)[GLD]) {
    const int tid = threadIdx.x;
    if (KIND == KC_F32) {
        const int k = (tid & 3) * 4;
#pragma unroll
        for (int h = 0; h < 2; h++) {
            const int m = (tid >> 2) + h * 64;
            tile[k + 0][m] = __uint_as_float(f.r[h].x);
            tile[k + 1][m] = __uint_as_float(f.r[h].y);
            tile[k + 2][m] = __uint_as_float(f.r[h].z);
            tile[k + 3][m] = __uint_as_float(f.r[h].w);
        }
    } else if (KIND == KC_U16) {
        const int m = tid & 127, k = (tid >> 7) * 8;
        tile[k + 0][m] = lo16(f.r[0].x); tile[k + 1][m] = hi16(f.r[0].x);
        tile[k + 2][m] = lo16(f.r[0].y); tile[k + 3][m] = hi16(f.r[0].y);
        tile[k + 4][m] = lo16(f.r[0].z); tile[k + 5][m] = hi16(f.r[0].z);
        tile[k + 6][m] = lo16(f.r[0].w); tile[k + 7][m] = hi16(f.r[0].w);
    } else if (KIND == RK_F32) {
        const int m = (tid & 31) * 4;
#pragma unroll
        for (int h = 0; h < 2; h++) *reinterpret_cast<uint4 *>(&tile[(tid >> 5) + h * 8][m]) = f.r[h];
    } else {
        const int m = (tid & 15) * 8, k = tid >> 4;
        *reinterpret_cast<float4 *>(&tile[k][m]) = make_float4(lo16(f.r[0].x), hi16(f.r[0].x), lo16(f.r[0].y), hi16(f.r[0].y));
        *reinterpret_cast<float4 *>(&tile[k][m + 4]) = make_float4(lo16(f.r[0].z), hi16(f.r[0].z), lo16(f.r[0].w), hi16(f.r[0].w));
    }
}

struct GemmArgs {
    const void *A;
    const float *B;
    float *C;
    int M, N, K;
    int64_t lda, ldb, ldc;
    int64_t za, zb, zc;  // per blockIdx.z strides, in elements
    int kblock;          // A only: k = q * kblock + r is found at k-offset q * kblock_stride + r (k contiguous kinds)
    int64_t kblock_stride;
    float alpha;
    int accumulate;      // 0: C = alpha * acc, 1: C += alpha * acc
    int ksplit;          // > 1: blockIdx.z also splits K; partial sums are added atomically (accumulate only)
};

template <int KIND_A, int KIND_B>
__global__ void __launch_bounds__(256, 2) tile_contract_kernel(const GemmArgs g) {
    __shared__ __align__(16) float As[2][GK][GLD];
    __shared__ __align__(16) float Bs[2][GK][GLD];
    const int tid = threadIdx.x, tx = tid & 15, ty = tid >> 4;
    const int m0 = blockIdx.y * GM, n0 = blockIdx.x * GM;
    const int64_t z = blockIdx.z / g.ksplit;
    const int split = blockIdx.z - (int)z * g.ksplit;
    const size_t a_elem = (KIND_A == KC_U16 || KIND_A == RK_U16) ? 2 : 4;
    const char *A = static_cast<const char *>(g.A) + (size_t)(z * g.za) * a_elem;
    const float *B = g.B + z * g.zb;
    float *C = g.C + z * g.zc;

    float2 acc[8][4];   // acc[i][j] = columns 2j, 2j+1 of accumulator row i (register pairs for the packed FMA)
#pragma unroll
    for (int i = 0; i < 8; i++)
#pragma unroll
        for (int j = 0; j < 4; j++) acc[i][j] = make_float2(0.f, 0.f);

    const int all_tiles = (g.K + GK - 1) / GK, per_split = (all_tiles + g.ksplit - 1) / g.ksplit;
    const int kt0 = split * per_split, nkt = min(all_tiles, kt0 + per_split);
    Frag fa, fb;
    auto fetch = [&](int kt) {
        const int k0 = kt * GK;
        if (KIND_A == KC_F32 || KIND_A == KC_U16) {
            const int q = k0 / g.kblock, r = k0 - q * g.kblock;
            fetch_tile<KIND_A>(fa, A + (size_t)(q * g.kblock_stride) * a_elem, g.lda, m0, g.M, r, g.kblock < g.K ? g.kblock : g.K);
        } else {
            fetch_tile<KIND_A>(fa, A, g.lda, m0, g.M, k0, g.K);
        }
        fetch_tile<KIND_B>(fb, B, g.ldb, n0, g.N, k0, g.K);
    };
    if (kt0 >= nkt) return;
    fetch(kt0);
    stash_tile<KIND_A>(fa, As[kt0 & 1]);
    stash_tile<KIND_B>(fb, Bs[kt0 & 1]);
    __syncthreads();
    for (int kt = kt0; kt < nkt; kt++) {
        const int buf = kt & 1;
        if (kt + 1 < nkt) fetch(kt + 1);
#pragma unroll 2
        for (int k = 0; k < GK; k++) {
            const float4 a0 = *reinterpret_cast<const float4 *>(&As[buf][k][ty * 4]);
            const float4 a1 = *reinterpret_cast<const float4 *>(&As[buf][k][64 + ty * 4]);
            const float4 b0 = *reinterpret_cast<const float4 *>(&Bs[buf][k][tx * 4]);
            const float4 b1 = *reinterpret_cast<const float4 *>(&Bs[buf][k][64 + tx * 4]);
            const float a[8] = {a0.x, a0.y, a0.z, a0.w, a1.x, a1.y, a1.z, a1.w};
            const float2 b[4] = {make_float2(b0.x, b0.y), make_float2(b0.z, b0.w), make_float2(b1.x, b1.y),
                                 make_float2(b1.z, b1.w)};
            // packed fp32 FMA (two independent round-to-nearest FMAs per instruction on sm_100): the loop is bound by
            // instruction issue, and halving the FMA instructions measured +15-18 %
#pragma unroll
            for (int i = 0; i < 8; i++) {
                const float2 aa = make_float2(a[i], a[i]);
#pragma unroll
                for (int j = 0; j < 4; j++) acc[i][j] = __ffma2_rn(aa, b[j], acc[i][j]);
            }
        }
        if (kt + 1 < nkt) {
            stash_tile<KIND_A>(fa, As[buf ^ 1]);
            stash_tile<KIND_B>(fb, Bs[buf ^ 1]);
        }
        __syncthreads();
    }
#pragma unroll
    for (int i = 0; i < 8; i++) {
        const int m = m0 + (i < 4 ? ty * 4 + i : 64 + ty * 4 + (i - 4));
        if (m >= g.M) continue;
#pragma unroll
        for (int h = 0; h < 2; h++) {
            const int n = n0 + h * 64 + tx * 4;
            if (n >= g.N) continue;
            float4 *dst = reinterpret_cast<float4 *>(C + (int64_t)m * g.ldc + n);
            float4 v = make_float4(g.alpha * acc[i][h * 2].x, g.alpha * acc[i][h * 2].y, g.alpha * acc[i][h * 2 + 1].x,
                                   g.alpha * acc[i][h * 2 + 1].y);
            if (g.ksplit > 1) {
                asm volatile("red.global.add.v4.f32 [%0], {%1, %2, %3, %4};" ::"l"(dst), "f"(v.x), "f"(v.y), "f"(v.z), "f"(v.w)
                             : "memory");
                continue;
            }
            if (g.accumulate) {
                const float4 old = *dst;
                v.x += old.x; v.y += old.y; v.z += old.z; v.w += old.w;
            }
            *dst = v;
        }
    }
}

template <int KIND_A, int KIND_B>
static int launch_contract(KernelId id, GemmArgs g, int batches, cudaStream_t stream) {
    if (g.ksplit < 1) g.ksplit = 1;
    dim3 grid((unsigned)((g.N + GM - 1) / GM), (unsigned)((g.M + GM - 1) / GM), (unsigned)(batches * g.ksplit));
    LUTB_REQUIRE(grid.y <= 65535 && grid.z <= 65535, LUTB_ERR_SHAPE, "product histogram path: chunk too large");
    KernelScope scope(id, stream);
    tile_contract_kernel<KIND_A, KIND_B><<<grid, 256, 0, stream>>>(g);
    LUTB_LAUNCH_CHECK();
    return LUTB_OK;
}

static size_t align256(size_t v) { return (v + 255) & ~(size_t)255; }

// The bound on the sequence length of this path: the shared memory that a routing kernel staging whole sequences as the direct
// kernels do (product_pairs.cuh) would take.  What is launched takes less: the histogram kernel without staged positional operands
// (n_anchors + 1) floats a token, the routing kernel at most 181 KB whatever the length.
static size_t stage_bytes(const ProductCall &c, size_t per_warp_floats) {
    return (pair_stage_floats(c.S, c.cfg->n_anchors, c.cfg->pos_dim) + (size_t)8 * per_warp_floats) * 4;
}

// Anchors with a positional end whose operands the kernels stage: all of them in sliced mode (a third of the anchor ends
// are positional there), two otherwise.
static int staged_pe_anchors(const lutb_layer_cfg *cfg) {
    if (cfg->pos_dim == 0) return 0;
    return cfg->sliced_product || cfg->n_anchors < 2 ? cfg->n_anchors : 2;
}

bool product_hist_supported(const ProductCall &c, const void *weights, const void *io_rows, const void *dW) {
    const lutb_layer_cfg *cfg = c.cfg;
    if (cfg->int_mode || c.S < 2 || c.S > 65535) return false;
    if (cfg->n_anchors < 4 || cfg->n_anchors > 12 || cfg->n_outputs % 4 != 0) return false;
    const uintptr_t bits = reinterpret_cast<uintptr_t>(weights) | reinterpret_cast<uintptr_t>(io_rows) |
                           reinterpret_cast<uintptr_t>(dW);
    if (bits & 15) return false;
    const size_t T = (size_t)1 << cfg->n_anchors;
    return stage_bytes(c, T + 64 * cfg->n_anchors) <= (size_t)kMaxSmemPerBlock - 1024;
}

static size_t bytes_per_sequence(const lutb_layer_cfg *cfg, int S, bool backward) {
    const size_t cells = (size_t)cfg->n_detectors * S * ((size_t)1 << cfg->n_anchors);
    return align256(cells * 2) + (backward ? align256(cells * 4) : 0) + 512;
}

// Scratch of the tensor-core contractions of one pass over `rows` query rows (operand copies: the tables, and the output
// gradients in the backward pass); the largest of the calls the pass makes.
static size_t tc_scratch_bytes(const lutb_layer_cfg *cfg, int64_t rows, bool backward) {
    const int KT = cfg->n_detectors << cfg->n_anchors, O = cfg->n_outputs;
    const size_t fwd = hist_gemm_workspace(HG_FORWARD, (int)rows, KT, O);
    if (!backward) return align256(fwd);
    // (the forward contraction's scratch counts here too: a forward pass that leaves its histogram for the backward
    // pass lays the workspace out as the backward pass does)
    const size_t dw = hist_gemm_workspace(HG_TABLE_GRAD, (int)rows, KT, O), q = hist_gemm_workspace(HG_ROW_DOTS, (int)rows, KT, O);
    const size_t m = dw > q ? dw : q;
    return align256(m > fwd ? m : fwd);
}

size_t product_hist_workspace_bytes(const lutb_layer_cfg *cfg, int64_t batch, int S, bool backward) {
    // what lets `batch` sequences through in one pass with either contraction
    return tc_scratch_bytes(cfg, batch * S, backward) + (size_t)batch * bytes_per_sequence(cfg, S, backward) + 256;
}

struct HistPlan {
    int64_t chunk;  // sequences per pass
    bool tc;        // tensor-core contractions: H is fp16 [row][detector][T], Q fp32 [row][detector][T]
    void *H;
    float *Q;
    void *gemm_ws;
    size_t gemm_ws_bytes;
};

static int plan(const ProductCall &c, bool backward, bool allow_tc, void *workspace, size_t bytes, HistPlan &p) {
    LUTB_REQUIRE(workspace != nullptr, LUTB_ERR_WORKSPACE, "product histogram path needs a workspace");
    const uintptr_t base0 = (reinterpret_cast<uintptr_t>(workspace) + 255) & ~(uintptr_t)255;
    const size_t slack = base0 - reinterpret_cast<uintptr_t>(workspace);
    const size_t T = (size_t)1 << c.cfg->n_anchors;
    // tensor cores when the workspace holds at least one sequence and the operand copies, the extents fit 32-bit sizes and
    // the row counts (at most S - 1) are exact in fp16
    const size_t per_seq = bytes_per_sequence(c.cfg, c.S, backward);
    p.tc = allow_tc && c.S <= 2048 && (size_t)c.cfg->n_detectors * T < ((size_t)1 << 30) &&
           bytes >= slack + tc_scratch_bytes(c.cfg, c.S, backward) + per_seq;
    LUTB_REQUIRE(bytes >= slack + per_seq, LUTB_ERR_WORKSPACE,
                 "product histogram path: workspace of %zu bytes is smaller than the %zu bytes one sequence needs", bytes,
                 per_seq + 256);
    p.chunk = (int64_t)((bytes - slack) / per_seq);
    if (p.chunk > c.batch) p.chunk = c.batch;
    // grid.y of the FMA contraction covers chunk * S / 128 row tiles; the GEMM extents are 32-bit
    const int64_t max_rows = p.tc ? (int64_t)1 << 30 : (int64_t)65535 * GM;
    if (p.chunk * c.S > max_rows) p.chunk = max_rows / c.S;
    size_t head = 0;
    if (p.tc) {
        // the GEMM scratch grows with the rows of a pass: shrink the pass until both fit
        while (p.chunk > 1 && slack + tc_scratch_bytes(c.cfg, p.chunk * c.S, backward) + (size_t)p.chunk * per_seq > bytes) p.chunk--;
        head = tc_scratch_bytes(c.cfg, p.chunk * c.S, backward);
    }
    LUTB_REQUIRE(p.chunk >= 1, LUTB_ERR_SHAPE, "product histogram path: sequence too long");
    const size_t cells = (size_t)c.cfg->n_detectors * (size_t)p.chunk * c.S * T;
    uintptr_t base = base0;
    p.gemm_ws = p.tc ? reinterpret_cast<void *>(base) : nullptr;
    p.gemm_ws_bytes = head;
    base += head;
    p.H = reinterpret_cast<void *>(base);
    p.Q = backward ? reinterpret_cast<float *>(base + align256(cells * 2)) : nullptr;
    return LUTB_OK;
}

// Queries of one block of the pair kernels: the most, up to 128, that still give every SM a dozen blocks.
// Routing (`resident`: blocks an SM holds): below 32, down to 8, only while all blocks are resident at once: a block walks its
// queries eight at a time, each step waits for the one before, so that short or few sequences take as long as their longest
// block.  With positional anchors, 8 / 16 / 32 / 64 / 128 queries, us: 1 x 33 tokens, 16 detectors of 128 rows 19 / 27 / 39 (with a
// warp per query 21); 64 detectors of 256 rows: 1 x 64 tokens 19 / 27 / 43, 1 x 128 27 / 31 / 46 / 63 / 117, 4 x 128 65 / 64 / 59,
// 8 x 128 - / - / 86 / 91 / 136, 4 x 256 - / - / 117 / 121 / 139, 64 x 128 - / - / 529 / 467 / 458; 1 x 1024 tokens, 1024 rows
// - / - / 453 / 413 / 410 (with every query of a key range in one block 851).
// key_range: keys of one block (a block has the queries above its first key); 0: all of them, as the histogram kernel has it: its
// blocks stage every key below their queries first, so that long sequences keep 128 queries (1 x 1024 tokens 187 us with 128
// queries, 352 with 32; 1 x 500 tokens 64 and 42 us; 1 x 128 tokens 26 and 14 us).
static int queries_per_block(int S, int64_t detectors_times_sequences, int key_range, int resident) {
    const int64_t sm = device_info().sm_count;
    auto blocks = [&](int q) {
        int64_t n = 0;
        if (key_range == 0) n = (S + q - 1) / q;
        else
            for (int k0 = 0; k0 < S - 1; k0 += key_range) n += (S - 1 - k0 + q - 1) / q;
        return n * detectors_times_sequences;
    };
    const int least = key_range == 0 && S > 512 ? 128 : 32;
    for (int q = 128; q > least; q /= 2)
        if (blocks(q) >= 12 * sm) return q;
    int q = least;
    if (key_range != 0)
        while (q > kTileQ && blocks(q / 2) <= resident * sm) q /= 2;
    return q;
}

static int launch_hist(const ProductCall &c, const HistPlan &p, int64_t b0, int64_t n, cudaStream_t stream) {
    const lutb_layer_cfg *cfg = c.cfg;
    const size_t T = (size_t)1 << cfg->n_anchors;
    HistArgs h;
    h.x1 = c.x1; h.x2 = c.x2; h.pe = c.pe; h.anchors = c.anchors; h.H = p.H;
    h.b0 = b0; h.chunk_rows = n * c.S;
    h.S = c.S; h.e1 = c.e1; h.e2 = c.e2; h.npe = cfg->pos_dim;
    h.n_detectors = cfg->n_detectors; h.n_anchors = cfg->n_anchors; h.sliced = cfg->sliced_product; h.cmp_eps = cfg->cmp_eps;
    const int per_word = c.S <= 256 ? 4 : 2;
    // warps per block: what puts the most warps on an SM, of 32 at most (a wide table's counters leave room for one block only, which
    // then has to bring them all), and with many blocks rather four of 8 warps than two of 16, whose starts overlap less (64
    // sequences x 128 tokens, 64 detectors of 256 rows 196 -> 174 us; one of 700 tokens, 512 rows, the other way round 164 / 107);
    // very long sequences leave the positional operands in global memory
    h.queries = queries_per_block(c.S, (int64_t)cfg->n_detectors * n, 0, 0);
    const bool many = (int64_t)cfg->n_detectors * n * ((c.S + h.queries - 1) / h.queries) * 8 >= 64ll * device_info().sm_count;
    const int tiles = ((c.S < h.queries ? c.S : h.queries) + kHistTile - 1) / kHistTile;
    int warps = 0;
    for (int cap = staged_pe_anchors(cfg);; cap = 0) {
        int most = 0;
        for (int w = 16; w >= 1; w /= 2) {
            const size_t need = hist_floats(T, per_word, w, cfg->n_anchors, cap, c.S) * 4 + 1024;
            const int resident = min(32, w * (int)((size_t)kMaxSmemPerBlock / need));
            if ((resident > most || (resident == most && many && w == 8)) && (w <= tiles || w == 1)) { most = resident; warps = w; }
        }
        h.pe_cap = cap;
        if (most >= 4 || cap == 0) break;
    }
    LUTB_REQUIRE(warps > 0, LUTB_ERR_SHAPE, "product histogram path: sequence too long");
    const size_t smem = hist_floats(T, per_word, warps, cfg->n_anchors, h.pe_cap, c.S) * 4;
    h.sequences = (int)n;
    LUTB_REQUIRE(cfg->n_detectors * n <= 0x7FFFFFFF, LUTB_ERR_SHAPE, "product histogram path: too many blocks for one launch");
    const dim3 grid((unsigned)(cfg->n_detectors * n), (unsigned)((c.S + h.queries - 1) / h.queries));
    KernelScope scope(K_PRODUCT_HIST, stream);
    auto launch = [&](auto kern) -> int {
        if (smem > kPlainSmem) LUTB_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
        kern<<<grid, warps * 32, smem, stream>>>(h);
        return LUTB_OK;
    };
    const bool eps = cfg->cmp_eps != 0.f;
    auto pick = [&](auto f32) -> int {
        constexpr bool F = decltype(f32)::value;
        auto width = [&](auto per) -> int {
            constexpr int P = decltype(per)::value;
            if (cfg->n_anchors <= 8) return eps ? launch(product_hist_kernel<8, true, F, P>) : launch(product_hist_kernel<8, false, F, P>);
            return eps ? launch(product_hist_kernel<12, true, F, P>) : launch(product_hist_kernel<12, false, F, P>);
        };
        return per_word == 4 ? width(std::integral_constant<int, 4>{}) : width(std::integral_constant<int, 2>{});
    };
    const int rc = p.tc ? pick(std::true_type{}) : pick(std::false_type{});
    if (rc) return rc;
    LUTB_LAUNCH_CHECK();
    return LUTB_OK;
}

bool product_hist_keeps(const ProductCall &c, bool allow_tc, void *workspace, size_t workspace_bytes) {
    HistPlan p;
    if (workspace == nullptr || workspace_bytes < product_hist_workspace_bytes(c.cfg, 1, c.S, true)) return false;
    if (plan(c, true, allow_tc, workspace, workspace_bytes, p) != LUTB_OK) return false;
    return p.chunk == c.batch;
}

int launch_product_hist_forward(const ProductCall &c, const float *weights, float *y, bool allow_tc, void *workspace,
                                size_t workspace_bytes, cudaStream_t stream, bool keep) {
    HistPlan p;
    // keep: the workspace is laid out as the backward pass lays it out, so that the histogram stays where that pass
    // looks for it (only when the whole batch goes through in one pass; otherwise the forward pass's own layout)
    const bool as_backward = keep && product_hist_keeps(c, allow_tc, workspace, workspace_bytes);
    int rc = plan(c, as_backward, allow_tc, workspace, workspace_bytes, p);
    if (rc) return rc;
    const lutb_layer_cfg *cfg = c.cfg;
    const int T = 1 << cfg->n_anchors, O = cfg->n_outputs, Nt = cfg->n_detectors;
    for (int64_t b0 = 0; b0 < c.batch; b0 += p.chunk) {
        const int64_t n = (c.batch - b0 < p.chunk) ? c.batch - b0 : p.chunk;
        const int64_t rows = n * c.S;
        rc = launch_hist(c, p, b0, n, stream);
        if (rc) return rc;
        if (p.tc) {
            // y[rows, O] += H[rows, Nt*T] . W[Nt*T, O]
            KernelScope scope(K_PRODUCT_HIST_FORWARD, stream);
            rc = hist_gemm_forward((int)rows, Nt * T, O, static_cast<const __half *>(p.H), weights, y + b0 * c.S * O, p.gemm_ws, p.gemm_ws_bytes, stream);
            if (rc) return rc;
            continue;
        }
        GemmArgs g{};
        g.A = p.H; g.B = weights; g.C = y + b0 * c.S * O;
        g.M = (int)rows; g.N = O; g.K = Nt * T;
        g.lda = T; g.ldb = O; g.ldc = O;
        g.kblock = T; g.kblock_stride = rows * T;
        g.alpha = 1.f; g.accumulate = 1;
        rc = launch_contract<KC_U16, RK_F32>(K_PRODUCT_HIST_FORWARD, g, 1, stream);
        if (rc) return rc;
    }
    return LUTB_OK;
}

int launch_product_hist_backward(const ProductCall &c, const float *weights, const float *dY, float *dX1, float *dX2,
                                 float *dPE, float *target, double lr, bool in_place, bool allow_tc, void *workspace,
                                 size_t workspace_bytes, cudaStream_t stream, bool reuse) {
    HistPlan p;
    int rc = plan(c, true, allow_tc, workspace, workspace_bytes, p);
    if (rc) return rc;
    // reuse: the caller vouches that the workspace still holds the histogram a forward pass over the same inputs left
    // there; it is complete only when the whole batch is one pass
    const bool have_hist = reuse && p.chunk == c.batch;
    const lutb_layer_cfg *cfg = c.cfg;
    const int T = 1 << cfg->n_anchors, O = cfg->n_outputs, Nt = cfg->n_detectors;
    const int pe_cap = staged_pe_anchors(cfg);
    // dPE cells in shared memory while they are few
    const int pe_cells = cfg->pos_dim > 0 && (size_t)(c.S - 1) * cfg->pos_dim * 4 <= 8 * 1024;
    const size_t route_smem = route_floats(T, cfg->n_anchors, pe_cap, pe_cells, c.S, cfg->pos_dim) * 4;
    // In-place SGD reads unmodified tables for every input gradient: with more than one chunk the table update
    // runs as a second sweep over the chunks.
    const bool second_sweep = in_place && p.chunk < c.batch;
    auto table_gradient = [&](int64_t b0, int64_t rows) -> int {
        if (p.tc) {
            // target[Nt*T, O] += lr * H^T . dY  (H stored [rows, Nt*T])
            KernelScope scope(K_PRODUCT_HIST_WEIGHT_GRAD, stream);
            return hist_gemm_table_grad((int)rows, Nt * T, O, static_cast<const __half *>(p.H), dY + b0 * c.S * O, target, (float)lr, p.gemm_ws, p.gemm_ws_bytes, stream);
        }
        GemmArgs g{};
        g.A = p.H; g.B = dY + b0 * c.S * O; g.C = target;
        g.M = T; g.N = O; g.K = (int)rows;
        g.lda = T; g.ldb = O; g.ldc = O;
        g.za = rows * T; g.zb = 0; g.zc = (int64_t)T * O;
        g.kblock = g.K; g.kblock_stride = 0;
        g.alpha = (float)lr; g.accumulate = 1;
        // few output tiles and a long reduction: split K so that every SM gets several blocks
        const int64_t tiles = (int64_t)((T + GM - 1) / GM) * ((O + GM - 1) / GM) * Nt;
        const int64_t want = (8 * (int64_t)device_info().sm_count + tiles - 1) / tiles;
        const int64_t most = (rows / GK + 31) / 32;  // at least 32 k-tiles per block
        g.ksplit = (int)(want < 1 ? 1 : (want > most ? (most < 1 ? 1 : most) : want));
        return launch_contract<RK_U16, RK_F32>(K_PRODUCT_HIST_WEIGHT_GRAD, g, Nt, stream);
    };
    for (int64_t b0 = 0; b0 < c.batch; b0 += p.chunk) {
        const int64_t n = (c.batch - b0 < p.chunk) ? c.batch - b0 : p.chunk;
        const int64_t rows = n * c.S;
        if (!have_hist) {
            rc = launch_hist(c, p, b0, n, stream);
            if (rc) return rc;
        }
        if (p.tc) {
            // Q[rows, Nt*T] = dY[rows, O] . W^T  (W stored [Nt*T, O])
            KernelScope scope(K_PRODUCT_ROW_DOTS, stream);
            rc = hist_gemm_row_dots((int)rows, Nt * T, O, dY + b0 * c.S * O, weights, p.Q, p.gemm_ws, p.gemm_ws_bytes, stream);
            if (rc) return rc;
        } else {
            GemmArgs g{};
            g.A = dY + b0 * c.S * O; g.B = weights; g.C = p.Q;
            g.M = (int)rows; g.N = T; g.K = O;
            g.lda = O; g.ldb = O; g.ldc = T;
            g.za = 0; g.zb = (int64_t)T * O; g.zc = rows * T;
            g.kblock = O; g.kblock_stride = 0;
            g.alpha = 1.f; g.accumulate = 0;
            rc = launch_contract<KC_F32, KC_F32>(K_PRODUCT_ROW_DOTS, g, Nt, stream);
            if (rc) return rc;
        }
        {
            RouteArgs ra;
            ra.x1 = c.x1; ra.x2 = c.x2; ra.pe = c.pe; ra.anchors = c.anchors; ra.Q = p.Q;
            ra.dX1 = dX1; ra.dX2 = dX2; ra.dPE = dPE;
            ra.b0 = b0;
            ra.q_row_stride = p.tc ? (int64_t)Nt * T : T;
            ra.q_det_stride = p.tc ? T : rows * T;
            ra.S = c.S; ra.e1 = c.e1; ra.e2 = c.e2; ra.npe = cfg->pos_dim;
            ra.n_detectors = Nt; ra.n_anchors = cfg->n_anchors; ra.sliced = cfg->sliced_product; ra.cmp_eps = cfg->cmp_eps;
            ra.pe_cap = pe_cap; ra.pe_cells = pe_cells;
            // (no block for the last key range when its first key is the last token: it has no query)
            const int most = cfg->n_anchors <= 8 ? 8 : 7;   // (the launch bounds of the kernel)
            const int resident = (int)((size_t)kMaxSmemPerBlock / (route_smem + 2048));
            ra.queries = queries_per_block(c.S, (int64_t)Nt * n, kRouteKeys, resident < most ? resident : most);
            const int ranges = (c.S - 1 + kRouteKeys - 1) / kRouteKeys, segs = (c.S - 1 + ra.queries - 1) / ra.queries;
            LUTB_REQUIRE((int64_t)ranges * segs <= 65535, LUTB_ERR_SHAPE, "product histogram path: sequence too long");
            ra.sequences = (int)n;
            ra.parts = ranges * segs;
            const int64_t grid = (int64_t)Nt * ra.parts * n;
            LUTB_REQUIRE(grid <= 0x7FFFFFFF, LUTB_ERR_SHAPE, "product histogram path: too many blocks for one launch");
            KernelScope scope(K_PRODUCT_ROUTE, stream);
            auto launch = [&](auto kern) -> int {
                if (route_smem > kPlainSmem)
                    LUTB_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)route_smem));
                kern<<<(unsigned)grid, 32 * kRouteWarps, route_smem, stream>>>(ra);
                return LUTB_OK;
            };
            const bool eps = cfg->cmp_eps != 0.f;
            if (cfg->n_anchors <= 8) rc = eps ? launch(product_route_kernel<8, true>) : launch(product_route_kernel<8, false>);
            else rc = eps ? launch(product_route_kernel<12, true>) : launch(product_route_kernel<12, false>);
            if (rc) return rc;
            LUTB_LAUNCH_CHECK();
        }
        if (!second_sweep) {
            rc = table_gradient(b0, rows);
            if (rc) return rc;
        }
    }
    if (second_sweep) {
        for (int64_t b0 = 0; b0 < c.batch; b0 += p.chunk) {
            const int64_t n = (c.batch - b0 < p.chunk) ? c.batch - b0 : p.chunk;
            rc = launch_hist(c, p, b0, n, stream);
            if (rc) return rc;
            rc = table_gradient(b0, n * c.S);
            if (rc) return rc;
        }
    }
    return LUTB_OK;
}

}  // namespace lutb
