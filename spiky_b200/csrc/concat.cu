// Concatenation-mode sequence (attention) layer.  Every token has its own table index (anchor
// comparison over the B*S token rows, the non-sequence kernel), every (distance, detector) a positional
// index; a causal pair (i < j) selects row (Q_j << (Nc + Npe)) | (K_i << Npe) | PE_{j-i-1} of a table
// with 2^(2Nc+Npe) rows.
//
// Reference: check_positional_embeddings[_eval]_logic (lut_runtime_kernels_logic.proto:1709-1805),
// fill_outputs_fully_connected_seq_logic (:1807-1904), propagate_through_detectors_seq_fc_logic
// (:3629-3835), gather_w_gradients_seq_fc_cpu_logic (:3944-4044).
#include <type_traits>

#include "lutb_common.cuh"
#include "nonseq_fc.cuh"

namespace lutb {

// sign bits of pe[d][t][:], first minimal |value| and its dimension
template <bool TRAIN>
__global__ void check_positional_kernel(const float *__restrict__ pe, int64_t n_items, int npe, float cmp_eps,
                                        int32_t *__restrict__ pidx, float *__restrict__ pmin,
                                        int32_t *__restrict__ pmin_k) {
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n_items) return;
    const float *p = pe + i * npe;
    int32_t li = 0, mk = -1;
    float md = 0.f;
    for (int d = 0; d < npe; d++) {
        const float v = __ldg(p + d);
        if (greater_than_zero(v, cmp_eps)) li |= (1 << d);
        if (TRAIN && (mk == -1 || fabsf(v) < fabsf(md))) { md = v; mk = d; }
    }
    pidx[i] = li;
    if (TRAIN) { pmin[i] = md; pmin_k[i] = mk; }
}

__device__ __forceinline__ size_t concat_row(int32_t Q, int32_t K, int32_t PE, int nc, int npe) {
    return (size_t)(((uint32_t)Q << (nc + npe)) | ((uint32_t)K << npe) | (uint32_t)PE);
}

// --------------------------------------------------------------------------------------------
// Pair order of the fp32 kernels.  Block = (detector, sample); a warp owns a "folded" query pair: of the queries [j_begin,
// j_end) (the whole sequence, or one rank's share when the queries are sharded) the r-th from the end and the r-th from the
// start have j_begin + j_end - 1 keys together, so every unit of work has the same number of pairs, S - 1 for a whole
// sequence, and 32 of them fill a warp (walking one query at a time leaves half of the lanes without a key at 32 tokens;
// folding a share of the queries about the middle of the sequence leaves most units of a small share empty: 32 of 256 queries
// of 4 sequences cost 117 us forward and 465 us backward).  A lane works out one pair's table row; then the warp's lane groups of LG lanes (LG * VEC columns, a whole row where it fits) take the
// pairs of the 32 that belong to them, NG = 32 / LG pairs at a time, with the row loads of U pairs per group issued
// before the first is used: the rows are random, so what bounds the kernel is how many of these reads are in flight.
// Measured (32 sequences x 32 tokens, 64 detectors of 65536 rows x 32 outputs, 1.0 M pairs; lanes over the outputs of
// one pair before, which left 24 of 32 idle): forward 44.5 -> 33.7 us (3.9 TB/s of rows), input gradient 780 -> 97 us
// (4.6 TB/s), table update 124 -> 39 us.
// --------------------------------------------------------------------------------------------
struct FoldedPair {
    int i, j;
    bool first;   // belongs to the longer query of the two
};
__device__ __forceinline__ FoldedPair folded_pair(int ja, int jb, int p) {
    FoldedPair f;
    f.first = p < ja;
    f.j = f.first ? ja : jb;
    f.i = f.first ? p : p - ja;
    return f;
}

template <int VEC>
__device__ __forceinline__ void load_row(const float *p, bool on, float (&v)[VEC]) {
    if constexpr (VEC == 4) {
        const float4 q = on ? __ldg(reinterpret_cast<const float4 *>(p)) : make_float4(0.f, 0.f, 0.f, 0.f);
        v[0] = q.x; v[1] = q.y; v[2] = q.z; v[3] = q.w;
    } else {
        v[0] = on ? __ldg(p) : 0.f;
    }
}

template <int VEC>
__device__ __forceinline__ void red_row(float *p, const float (&v)[VEC]) {
    if constexpr (VEC == 4)
        asm volatile("red.global.add.v4.f32 [%0], {%1, %2, %3, %4};" ::"l"(p), "f"(v[0]), "f"(v[1]), "f"(v[2]), "f"(v[3]) : "memory");
    else
        atomicAdd(p, v[0]);
}

// Forward, fp32 accumulators: y[b, j, :] += sum over keys of the selected rows.
template <int LG, int VEC>
__global__ void __launch_bounds__(256) concat_forward_kernel(const float *__restrict__ W, const int32_t *__restrict__ idx,
                                                            const int32_t *__restrict__ pidx, float *__restrict__ y,
                                                            int batch, int S, int n_outputs, int n_detectors, int nc,
                                                            int npe, int j_begin, int j_end) {
    extern __shared__ __align__(16) int32_t ismem[];
    constexpr int NG = 32 / LG;
    constexpr int U = LG < 8 ? LG : 8;
    const int t = blockIdx.x / batch;
    const int64_t b = blockIdx.x - (int64_t)t * batch;
    int32_t *Ks = ismem;          // [S]
    int32_t *Ps = ismem + S;      // [S-1]
    for (int s = threadIdx.x; s < S; s += blockDim.x) Ks[s] = __ldg(idx + ((size_t)b * S + s) * n_detectors + t);
    for (int d = threadIdx.x; d < S - 1; d += blockDim.x) Ps[d] = npe > 0 ? __ldg(pidx + (size_t)d * n_detectors + t) : 0;
    __syncthreads();
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, nwarps = blockDim.x >> 5;
    const int g = lane / LG, q = lane - g * LG;
    const size_t rows = (size_t)1 << (2 * nc + npe);
    const float *Wt = W + (size_t)t * rows * n_outputs;
    for (int r = warp; 2 * r < j_end - j_begin; r += nwarps) {
        const int ja = j_end - 1 - r, jb = j_begin + r;
        const int count = ja + (jb != ja ? jb : 0);   // (the middle query of an odd number is alone)
        for (int c0 = 0; c0 < n_outputs; c0 += LG * VEC) {
            const int col = c0 + q * VEC;
            const bool active = col < n_outputs;
            float acc_a[VEC], acc_b[VEC];
#pragma unroll
            for (int e = 0; e < VEC; e++) acc_a[e] = acc_b[e] = 0.f;
            for (int p0 = 0; p0 < count; p0 += 32) {
                // bit 31: the pair belongs to the shorter query; bit 30: no pair
                uint32_t mine = 0x40000000u;
                if (p0 + lane < count) {
                    const FoldedPair f = folded_pair(ja, jb, p0 + lane);
                    mine = (uint32_t)concat_row(Ks[f.j], Ks[f.i], Ps[f.j - f.i - 1], nc, npe) | (f.first ? 0u : 0x80000000u);
                }
#pragma unroll 1
                for (int i0 = 0; i0 < LG && p0 + i0 < count; i0 += U) {
                    float w[U][VEC];
                    uint32_t row[U];
#pragma unroll
                    for (int u = 0; u < U; u++) {
                        row[u] = __shfl_sync(0xffffffffu, mine, g * LG + i0 + u);
                        load_row<VEC>(Wt + (size_t)(row[u] & 0x3fffffffu) * n_outputs + col, active && !(row[u] & 0x40000000u), w[u]);
                    }
#pragma unroll
                    for (int u = 0; u < U; u++) {
                        const bool second = (row[u] & 0x80000000u) != 0;
#pragma unroll
                        for (int e = 0; e < VEC; e++) {
                            acc_a[e] += second ? 0.f : w[u][e];
                            acc_b[e] += second ? w[u][e] : 0.f;
                        }
                    }
                }
            }
#pragma unroll
            for (int m = LG; m < 32; m <<= 1) {
#pragma unroll
                for (int e = 0; e < VEC; e++) {
                    acc_a[e] += __shfl_xor_sync(0xffffffffu, acc_a[e], m);
                    acc_b[e] += __shfl_xor_sync(0xffffffffu, acc_b[e], m);
                }
            }
            float *yb = y + (size_t)b * S * n_outputs + col;
            // one group adds the longer query's sum, the next (where there is one) the shorter's
            if (active && g == 0 && ja > 0) red_row<VEC>(yb + (size_t)ja * n_outputs, acc_a);
            if (active && g == (NG > 1 ? 1 : 0) && jb > 0 && jb != ja) red_row<VEC>(yb + (size_t)jb * n_outputs, acc_b);
        }
    }
}

// Forward, fixed-point accumulators: each (query, detector, output) is summed in double in key order and truncated
// once, exactly as the reference does.  A warp owns a query, the lanes cover the outputs.
__global__ void __launch_bounds__(256) concat_forward_fixed_kernel(const float *__restrict__ W, const int32_t *__restrict__ idx,
                                                                  const int32_t *__restrict__ pidx, float *__restrict__ y,
                                                                  int S, int n_outputs, int n_detectors, int nc, int npe,
                                                                  double fixed_scale, int j_begin, int j_end) {
    extern __shared__ __align__(16) int32_t ismem[];
    const int t = blockIdx.x;
    const int64_t b = blockIdx.y;
    int32_t *Ks = ismem;          // [S]
    int32_t *Ps = ismem + S;      // [S-1]
    for (int s = threadIdx.x; s < S; s += blockDim.x) Ks[s] = __ldg(idx + ((size_t)b * S + s) * n_detectors + t);
    for (int d = threadIdx.x; d < S - 1; d += blockDim.x) Ps[d] = npe > 0 ? __ldg(pidx + (size_t)d * n_detectors + t) : 0;
    __syncthreads();
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, nwarps = blockDim.x >> 5;
    const size_t rows = (size_t)1 << (2 * nc + npe);
    const float *Wt = W + (size_t)t * rows * n_outputs;
    // queries [j_begin, j_end): the whole sequence, or one rank's share when the queries are sharded
    for (int j = max(1, j_begin) + warp; j < j_end; j += nwarps) {
        const int32_t Q = Ks[j];
        int32_t *yj = reinterpret_cast<int32_t *>(y) + ((size_t)b * S + j) * n_outputs;
        for (int o = lane; o < n_outputs; o += 32) {
            double dacc = 0.0;
#pragma unroll 4
            for (int i = 0; i < j; i++) dacc += (double)__ldg(Wt + concat_row(Q, Ks[i], Ps[j - i - 1], nc, npe) * n_outputs + o);
            atomicAdd(yj + o, to_fixed(dacc, fixed_scale));
        }
    }
}

// --------------------------------------------------------------------------------------------
// Backward, fp32 accumulators.  Pairs and lane groups as above.  Per pair the side (query or key) with the smaller
// |min delta| is flipped; g = sum_o dY[b,j,o] * (W[row,o] - W[alt,o]), every lane summing its columns of the group's
// pairs and the group transpose-reducing them so that lane l ends with pair l of the 32, and du = up(delta) * g goes to
// the flipped token's two anchor inputs.  When the positional margin is the strictly smallest of the three, the
// positional embedding receives its own gradient from the row with the positional bit flipped.  The table gradient
// adds lr * dY[b,j,:] to the pair's row.
// smem_dx: the block sums its contributions per (token, anchor pair) in shared memory and issues two global
// reductions per touched cell at the end instead of two per pair (S * nc cells against S * (S - 1) / 2 pairs); without
// it (sequences whose cells do not fit) every pair issues its own.
// --------------------------------------------------------------------------------------------
// ONE: rows of one step (n_outputs <= LG * VEC).  The two queries' rows of dY are then loaded once per pair of queries and chosen by
// a bit, and the pairs whose positional margin is the smallest (about a quarter) have a loop of their own behind the others', which
// leaves registers for three blocks an SM instead of two.  Bound: the latency and rate of random rows from HBM.  Measured with and
// without: 32 x 32 tokens, 64 detectors of 65536 rows x 32 outputs, input gradient 97 -> 87 us, with the table gradient 149 -> 109;
// 16 x 32 tokens, 32 detectors of 16384 rows x 64 outputs 67 -> 55; 8 x 33 tokens x 10 outputs 46 -> 31.
template <int LG, int VEC, bool DO_DX, bool DO_DW, bool ONE>
__global__ void __launch_bounds__(256, !ONE || LG == 32 ? 1 : LG == 16 ? 2 : 3) concat_backward_kernel(const float *__restrict__ W, const float *__restrict__ dY,
                                                             const int2 *__restrict__ anchors,
                                                             const int32_t *__restrict__ idx,
                                                             const float *__restrict__ min_delta,
                                                             const int32_t *__restrict__ min_k,
                                                             const int32_t *__restrict__ pidx,
                                                             const float *__restrict__ pmin,
                                                             const int32_t *__restrict__ pmin_k, float *__restrict__ dX,
                                                             float *__restrict__ dPE, float *__restrict__ target, int batch,
                                                             int S, int n_inputs, int n_outputs, int n_detectors, int nc,
                                                             int npe, double lr, int j_begin, int j_end, int smem_dx) {
    extern __shared__ __align__(16) int32_t ismem[];
    constexpr int U = LG < 4 ? LG : 4;
    const int t = blockIdx.x / batch;
    const int64_t b = blockIdx.x - (int64_t)t * batch;
    int32_t *Ks = ismem;                                         // [S] token index
    int32_t *Kk = Ks + S;                                        // [S] token min-margin pair
    float *Km = reinterpret_cast<float *>(Kk + S);               // [S] token min margin
    int32_t *Ps = reinterpret_cast<int32_t *>(Km + S);           // [S] positional index (S-1 used)
    int32_t *Pk = Ps + S;                                        // [S]
    float *Pm = reinterpret_cast<float *>(Pk + S);               // [S]
    float *dxs = Pm + S;                                         // [S][nc] when smem_dx
    for (int s = threadIdx.x; s < S; s += blockDim.x) {
        const size_t o = ((size_t)b * S + s) * n_detectors + t;
        Ks[s] = __ldg(idx + o); Kk[s] = __ldg(min_k + o); Km[s] = __ldg(min_delta + o);
    }
    for (int d = threadIdx.x; d < S - 1; d += blockDim.x) {
        const size_t o = (size_t)d * n_detectors + t;
        Ps[d] = npe > 0 ? __ldg(pidx + o) : 0;
        Pk[d] = npe > 0 ? __ldg(pmin_k + o) : -1;
        Pm[d] = npe > 0 ? __ldg(pmin + o) : 0.f;
    }
    if (DO_DX && smem_dx)
        for (int w = threadIdx.x; w < S * nc; w += blockDim.x) dxs[w] = 0.f;
    __syncthreads();
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, nwarps = blockDim.x >> 5;
    const int g = lane / LG, q = lane - g * LG;
    const size_t rows = (size_t)1 << (2 * nc + npe);
    const float *Wt = W + (size_t)t * rows * n_outputs;
    float *Tt = DO_DW ? target + (size_t)t * rows * n_outputs : nullptr;
    const float *dYb = dY + (size_t)b * S * n_outputs;
    for (int r = warp; 2 * r < j_end - j_begin; r += nwarps) {
        const int ja = j_end - 1 - r, jb = j_begin + r;
        const int count = ja + (jb != ja ? jb : 0);   // (the middle query of an odd number is alone)
        float da[VEC], db[VEC], ua[VEC], ub[VEC];     // ONE: this lane's columns of dY of both queries; as the table gradient takes them
        bool add_a = false, add_b = false;
        if constexpr (ONE) {
            load_row<VEC>(dYb + (size_t)ja * n_outputs + q * VEC, q * VEC < n_outputs, da);
            load_row<VEC>(dYb + (size_t)jb * n_outputs + q * VEC, q * VEC < n_outputs, db);
            if (DO_DW) {
                auto scaled = [&](const float (&d)[VEC], float (&up)[VEC], bool &add) {
#pragma unroll
                    for (int e = 0; e < VEC; e++) {
                        up[e] = lr != 1.0 ? (float)((double)d[e] * lr) : d[e];   // lr == 1: dY itself
                        up[e] = fabsf(d[e]) > kEpsF ? up[e] : 0.f;
                    }
                    add = q * VEC < n_outputs && (VEC == 4 || fabsf(d[0]) > kEpsF);
                };
                scaled(da, ua, add_a);
                scaled(db, ub, add_b);
            }
        }
        for (int p0 = 0; p0 < count; p0 += 32) {
            // this lane's pair; my_j < 0: none
            int my_j = -1, my_i = 0, my_flip = 0, my_pos = 0;
            uint32_t my_row = 0, my_alt = 0, my_palt = 0;
            float my_m = 0.f;
            bool my_pe = false;
            if (p0 + lane < count) {
                const FoldedPair f = folded_pair(ja, jb, p0 + lane);
                my_j = f.j; my_i = f.i;
                const int32_t Q = Ks[f.j], K = Ks[f.i], PEi = Ps[f.j - f.i - 1];
                const float qm = Km[f.j], km = Km[f.i], pm = Pm[f.j - f.i - 1];
                const int qk = Kk[f.j], kk = Kk[f.i];
                my_row = (uint32_t)concat_row(Q, K, PEi, nc, npe);
                const bool flip_query = fabsf(qm) < fabsf(km);
                my_flip = flip_query ? qk : kk;
                my_m = flip_query ? qm : km;
                my_pos = flip_query ? f.j : f.i;
                // (a detector without a usable anchor pair has no bit to flip)
                my_alt = my_flip < 0 ? my_row : my_row ^ (1u << (my_flip + npe + (flip_query ? nc : 0)));
                if (npe > 0 && fabsf(pm) < fabsf(qm) && fabsf(pm) < fabsf(km)) {
                    my_pe = true;
                    my_palt = my_row ^ (1u << Pk[f.j - f.i - 1]);
                }
            }
            const unsigned pe_mask = DO_DX ? __ballot_sync(0xffffffffu, my_pe) : 0u;
            float v[LG], vp[LG];
            if constexpr (ONE) {
                // pairs of the longer query come first, so that one number tells the query, and one whether there is a pair
                const bool in_row = q * VEC < n_outputs;
                const int col = q * VEC;
#pragma unroll
                for (int i0 = 0; i0 < LG; i0 += U) {
#pragma unroll
                    for (int u = 0; u < U; u++) v[i0 + u] = 0.f;
                    if (p0 + i0 >= count) continue;   // (warp uniform; group 0 holds the first pairs)
                    uint32_t r0[U];
                    float a[U][VEC], c[U][VEC];
#pragma unroll
                    for (int u = 0; u < U; u++) {
                        const int src = g * LG + i0 + u;
                        r0[u] = __shfl_sync(0xffffffffu, my_row, src);
                        if (DO_DX) {
                            const uint32_t r1 = __shfl_sync(0xffffffffu, my_alt, src);
                            const bool on = in_row && p0 + src < count;
                            load_row<VEC>(Wt + (size_t)r0[u] * n_outputs + col, on, a[u]);
                            load_row<VEC>(Wt + (size_t)r1 * n_outputs + col, on, c[u]);
                        }
                    }
#pragma unroll
                    for (int u = 0; u < U; u++) {
                        const int pair = p0 + g * LG + i0 + u;
                        const bool first = pair < ja;
                        if (DO_DX) {
                            float s0 = 0.f;
#pragma unroll
                            for (int e = 0; e < VEC; e++) s0 = fmaf(first ? da[e] : db[e], a[u][e] - c[u][e], s0);
                            v[i0 + u] = s0;
                        }
                        if (DO_DW && pair < count && (first ? add_a : add_b)) {
                            float up[VEC];
#pragma unroll
                            for (int e = 0; e < VEC; e++) up[e] = first ? ua[e] : ub[e];
                            red_row<VEC>(Tt + (size_t)r0[u] * n_outputs + col, up);
                        }
                    }
                }
            } else {
#pragma unroll
                for (int i0 = 0; i0 < LG; i0 += U) {
#pragma unroll
                    for (int u = 0; u < U; u++) { v[i0 + u] = 0.f; vp[i0 + u] = 0.f; }
                    if (p0 + i0 >= count) continue;   // (warp uniform; group 0 holds the first pairs)
                    uint32_t r0[U], r1[U], r2[U];
                    int jj[U];
                    bool pe[U];
#pragma unroll
                    for (int u = 0; u < U; u++) {
                        const int src = g * LG + i0 + u;
                        r0[u] = __shfl_sync(0xffffffffu, my_row, src);
                        jj[u] = __shfl_sync(0xffffffffu, my_j, src);
                        pe[u] = (pe_mask >> src) & 1u;
                        if (DO_DX) {
                            r1[u] = __shfl_sync(0xffffffffu, my_alt, src);
                            r2[u] = pe_mask ? __shfl_sync(0xffffffffu, my_palt, src) : 0u;
                        }
                    }
                    for (int c0 = 0; c0 < n_outputs; c0 += LG * VEC) {
                        const int col = c0 + q * VEC;
                        float d[U][VEC], a[U][VEC], c[U][VEC], e2[U][VEC];
#pragma unroll
                        for (int u = 0; u < U; u++) {
                            const bool on = jj[u] >= 0 && col < n_outputs;
                            load_row<VEC>(dYb + (size_t)max(jj[u], 0) * n_outputs + col, on, d[u]);
                            if (DO_DX) {
                                load_row<VEC>(Wt + (size_t)r0[u] * n_outputs + col, on, a[u]);
                                load_row<VEC>(Wt + (size_t)r1[u] * n_outputs + col, on, c[u]);
                                load_row<VEC>(Wt + (size_t)r2[u] * n_outputs + col, on && pe[u], e2[u]);
                            }
                        }
#pragma unroll
                        for (int u = 0; u < U; u++) {
                            if (DO_DX) {
                                float s0 = 0.f, s1 = 0.f;
#pragma unroll
                                for (int e = 0; e < VEC; e++) {
                                    s0 = fmaf(d[u][e], a[u][e] - c[u][e], s0);
                                    s1 = fmaf(d[u][e], a[u][e] - e2[u][e], s1);
                                }
                                v[i0 + u] += s0;
                                vp[i0 + u] += s1;
                            }
                            if (DO_DW && jj[u] >= 0 && col < n_outputs) {
                                float up[VEC];
#pragma unroll
                                for (int e = 0; e < VEC; e++) {
                                    up[e] = lr != 1.0 ? (float)((double)d[u][e] * lr) : d[u][e];   // lr == 1: dY itself
                                    up[e] = fabsf(d[u][e]) > kEpsF ? up[e] : 0.f;
                                }
                                if (VEC == 4 || fabsf(d[u][0]) > kEpsF) red_row<VEC>(Tt + (size_t)r0[u] * n_outputs + col, up);
                            }
                        }
                    }
                }
            }
            if (!DO_DX) continue;
#pragma unroll
            for (int o = LG / 2; o >= 1; o >>= 1) {
                const bool upper = (q & o) != 0;
#pragma unroll
                for (int p = 0; p < o; p++) {
                    const float send = upper ? v[p] : v[p + o];
                    const float keep = upper ? v[p + o] : v[p];
                    v[p] = keep + __shfl_xor_sync(0xffffffffu, send, o);
                }
            }
            if (pe_mask) {
                if constexpr (ONE) {
#pragma unroll
                    for (int i0 = 0; i0 < LG; i0 += U) {
#pragma unroll
                        for (int u = 0; u < U; u++) vp[i0 + u] = 0.f;
                        if (p0 + i0 >= count) continue;
                        float a[U][VEC], c[U][VEC];
#pragma unroll
                        for (int u = 0; u < U; u++) {
                            const int src = g * LG + i0 + u;
                            const uint32_t r0 = __shfl_sync(0xffffffffu, my_row, src), r2 = __shfl_sync(0xffffffffu, my_palt, src);
                            const bool on = q * VEC < n_outputs && ((pe_mask >> src) & 1u);
                            load_row<VEC>(Wt + (size_t)r0 * n_outputs + q * VEC, on, a[u]);
                            load_row<VEC>(Wt + (size_t)r2 * n_outputs + q * VEC, on, c[u]);
                        }
#pragma unroll
                        for (int u = 0; u < U; u++) {
                            const bool first = p0 + g * LG + i0 + u < ja;
#pragma unroll
                            for (int e = 0; e < VEC; e++) vp[i0 + u] = fmaf(first ? da[e] : db[e], a[u][e] - c[u][e], vp[i0 + u]);
                        }
                    }
                }
#pragma unroll
                for (int o = LG / 2; o >= 1; o >>= 1) {
                    const bool upper = (q & o) != 0;
#pragma unroll
                    for (int p = 0; p < o; p++) {
                        const float send = upper ? vp[p] : vp[p + o];
                        const float keep = upper ? vp[p + o] : vp[p];
                        vp[p] = keep + __shfl_xor_sync(0xffffffffu, send, o);
                    }
                }
            }
            if (my_j >= 0) {
                const double du = surrogate_up(my_m) * (double)v[0];
                if (fabs(du) > kEps && my_flip >= 0) {
                    if (smem_dx) {
                        atomicAdd(dxs + my_pos * nc + my_flip, (float)du);
                    } else {
                        const int2 an = __ldg(anchors + (size_t)t * nc + my_flip);
                        float *dx = dX + ((size_t)b * S + my_pos) * n_inputs;
                        atomicAdd(dx + an.x, (float)du);
                        atomicAdd(dx + an.y, -(float)du);
                    }
                }
                if (my_pe) {
                    const int d = my_j - my_i - 1;
                    const double dp = surrogate_up(Pm[d]) * (double)vp[0];
                    atomicAdd(dPE + ((size_t)d * n_detectors + t) * npe + Pk[d], (float)dp);
                }
            }
        }
    }
    if (DO_DX && smem_dx) {
        __syncthreads();
        for (int w = threadIdx.x; w < S * nc; w += blockDim.x) {
            const float s = dxs[w];
            if (s == 0.f) continue;
            const int pos = w / nc, k = w - pos * nc;
            const int2 an = __ldg(anchors + (size_t)t * nc + k);
            float *dx = dX + ((size_t)b * S + pos) * n_inputs;
            atomicAdd(dx + an.x, s);
            atomicAdd(dx + an.y, -s);
        }
    }
}

// Fixed-point backward: one thread per (sample, query, detector, key, output block) walks the block's
// outputs in order in double like the reference's host loop; contributions are truncated to int32 and
// added with integer atomics (order independent).
__global__ void concat_backward_fixed_kernel(const float *__restrict__ W, const float *__restrict__ dY,
                                             const int2 *__restrict__ anchors, const int32_t *__restrict__ idx,
                                             const float *__restrict__ min_delta, const int32_t *__restrict__ min_k,
                                             const int32_t *__restrict__ pidx, const float *__restrict__ pmin,
                                             const int32_t *__restrict__ pmin_k, float *__restrict__ dX,
                                             float *__restrict__ dPE, float *__restrict__ dW, int64_t batch, int S,
                                             int n_inputs, int n_outputs, int n_detectors, int nc, int npe, int out_block,
                                             double lr, double fixed_scale) {
    const int n_ob = (n_outputs + out_block - 1) / out_block;
    const int64_t total = batch * S * (int64_t)n_detectors * S * n_ob;
    for (int64_t w = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; w < total; w += (int64_t)gridDim.x * blockDim.x) {
        const int ob = (int)(w % n_ob);
        int64_t r = w / n_ob;
        const int i = (int)(r % S); r /= S;
        const int t = (int)(r % n_detectors); r /= n_detectors;
        const int j = (int)(r % S);
        const int64_t b = r / S;
        if (i >= j) continue;
        const int o0 = ob * out_block, o1 = min(n_outputs, o0 + out_block);
        const size_t ko = ((size_t)b * S + i) * n_detectors + t, qo = ((size_t)b * S + j) * n_detectors + t;
        const int32_t K = idx[ko], Q = idx[qo];
        const float km = min_delta[ko], qm = min_delta[qo];
        const size_t po = (size_t)(j - i - 1) * n_detectors + t;
        int32_t PE = 0, pk = -1;
        float pm = 0.f;
        if (npe > 0) { PE = pidx[po]; pk = pmin_k[po]; pm = pmin[po]; }
        const size_t rows = (size_t)1 << (2 * nc + npe);
        const float *Wt = W + (size_t)t * rows * n_outputs;
        const size_t row = concat_row(Q, K, PE, nc, npe);
        size_t alt;
        float m;
        int flip, pos;
        if (fabsf(qm) < fabsf(km)) { alt = concat_row(Q ^ (1 << min_k[qo]), K, PE, nc, npe); m = qm; flip = min_k[qo]; pos = j; }
        else { alt = concat_row(Q, K ^ (1 << min_k[ko]), PE, nc, npe); m = km; flip = min_k[ko]; pos = i; }
        const float *dy = dY + ((size_t)b * S + j) * n_outputs;
        double ms = 0.0, as = 0.0;
        for (int o = o0; o < o1; o++) {
            const double g = (double)__ldg(dy + o);
            ms += (double)__ldg(Wt + row * n_outputs + o) * g;
            as += (double)__ldg(Wt + alt * n_outputs + o) * g;
        }
        const double du = surrogate_up(m) * (ms - as);
        if (fabs(du) > kEps) {
            const int2 a = __ldg(anchors + (size_t)t * nc + flip);
            int32_t *dx = reinterpret_cast<int32_t *>(dX) + ((size_t)b * S + pos) * n_inputs;
            const int32_t d = to_fixed(du, fixed_scale);
            atomicAdd(dx + a.x, d);
            atomicAdd(dx + a.y, -d);
        }
        if (npe > 0 && fabsf(pm) < fabsf(qm) && fabsf(pm) < fabsf(km)) {
            const size_t palt = concat_row(Q, K, PE ^ (1 << pk), nc, npe);
            double ps = 0.0;
            for (int o = o0; o < o1; o++) ps += (double)__ldg(Wt + palt * n_outputs + o) * (double)__ldg(dy + o);
            const double dp = surrogate_up(pm) * (ms - ps);
            atomicAdd(reinterpret_cast<int32_t *>(dPE) + po * npe + pk, to_fixed(dp, fixed_scale));
        }
        if (dW) {
            int32_t *drow = reinterpret_cast<int32_t *>(dW) + ((size_t)t * rows + row) * n_outputs;
            for (int o = o0; o < o1; o++) {
                const double g = (double)__ldg(dy + o);
                if (fabs(g) > kEps) atomicAdd(drow + o, to_fixed(g * lr, fixed_scale));
            }
        }
    }
}

// --------------------------------------------------------------------------------------------
// Concatenation-mode layers with sparse lookup -> output connectivity (reference: fill_outputs_sparse_seq_logic,
// proto:1906-2013; propagate_through_detectors_seq_sparse_logic, :3371-3627; gather_w_gradients_seq_sparse_logic,
// :3837-3942).  A causal pair selects lookup neuron (t, row(i, j)) as in the fully connected case; that neuron's
// synapses (slot p + 2 * (p / G) behind the row base, targets shared by all rows of the detector) are walked as in
// the non-sequence sparse layer.  One thread per (sample, query, detector, key): sums in double per synapse group
// (every group issues its own contribution, as the reference does with one block per group), fp32 or int32
// fixed-point atomics.  No layer of the benchmark configurations takes this path; it is written for exactness.
// --------------------------------------------------------------------------------------------
struct SparseRows {
    const int64_t *wbase;
    const int32_t *stride, *count, *sstart, *target;
    int group;
};

__device__ __forceinline__ int64_t sparse_slot(int64_t row_base, int p, int G) { return row_base + p + 2 * (p / G); }

template <bool INT_MODE>
__global__ void concat_sparse_forward_kernel(const float *__restrict__ W, const int32_t *__restrict__ idx,
                                             const int32_t *__restrict__ pidx, float *__restrict__ y, SparseRows sp,
                                             int64_t batch, int S, int n_outputs, int n_detectors, int nc, int npe,
                                             double fixed_scale) {
    const int64_t total = batch * S * (int64_t)n_detectors * S;
    for (int64_t w = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; w < total; w += (int64_t)gridDim.x * blockDim.x) {
        const int i = (int)(w % S);
        int64_t r = w / S;
        const int t = (int)(r % n_detectors);
        r /= n_detectors;
        const int j = (int)(r % S);
        const int64_t b = r / S;
        if (i >= j) continue;
        const int32_t K = idx[(b * S + i) * n_detectors + t], Q = idx[(b * S + j) * n_detectors + t];
        const int32_t PE = npe > 0 ? pidx[(int64_t)(j - i - 1) * n_detectors + t] : 0;
        const int64_t row = sp.wbase[t] + (int64_t)concat_row(Q, K, PE, nc, npe) * sp.stride[t];
        const int32_t *tg = sp.target + sp.sstart[t];
        float *yb = y + (b * S + j) * n_outputs;
        const int P = sp.count[t];
        for (int p = 0; p < P; p++) {
            const float wv = __ldg(W + sparse_slot(row, p, sp.group));
            if (INT_MODE) atomicAdd(reinterpret_cast<int32_t *>(yb) + tg[p], to_fixed((double)wv, fixed_scale));
            else atomicAdd(yb + tg[p], wv);
        }
    }
}

template <bool INT_MODE>
__global__ void concat_sparse_backward_kernel(const float *__restrict__ W, const float *__restrict__ dY,
                                              const int2 *__restrict__ anchors, const int32_t *__restrict__ idx,
                                              const float *__restrict__ min_delta, const int32_t *__restrict__ min_k,
                                              const int32_t *__restrict__ pidx, const float *__restrict__ pmin,
                                              const int32_t *__restrict__ pmin_k, float *__restrict__ dX,
                                              float *__restrict__ dPE, float *__restrict__ target, SparseRows sp,
                                              int64_t batch, int S, int n_inputs, int n_outputs, int n_detectors, int nc,
                                              int npe, int do_dx, double lr, double fixed_scale) {
    const int64_t total = batch * S * (int64_t)n_detectors * S;
    for (int64_t w = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; w < total; w += (int64_t)gridDim.x * blockDim.x) {
        const int i = (int)(w % S);
        int64_t r = w / S;
        const int t = (int)(r % n_detectors);
        r /= n_detectors;
        const int j = (int)(r % S);
        const int64_t b = r / S;
        if (i >= j) continue;
        const int64_t ko = (b * S + i) * n_detectors + t, qo = (b * S + j) * n_detectors + t;
        const int32_t K = idx[ko], Q = idx[qo];
        const int64_t po = (int64_t)(j - i - 1) * n_detectors + t;
        int32_t PE = 0, pk = -1;
        float pm = 0.f;
        if (npe > 0) { PE = pidx[po]; pk = pmin_k[po]; pm = pmin[po]; }
        const int64_t base = sp.wbase[t];
        const int64_t stride = sp.stride[t];
        const int64_t row = base + (int64_t)concat_row(Q, K, PE, nc, npe) * stride;
        const int32_t *tg = sp.target + sp.sstart[t];
        const float *dy = dY + (b * S + j) * n_outputs;
        const int P = sp.count[t], G = sp.group;
        if (do_dx) {
            const float qm = min_delta[qo], km = min_delta[ko];
            int64_t alt;
            double up;
            int flip, pos;
            if (fabsf(qm) < fabsf(km)) {
                alt = base + (int64_t)concat_row(Q ^ (1 << min_k[qo]), K, PE, nc, npe) * stride;
                up = surrogate_up(qm); flip = min_k[qo]; pos = j;
            } else {
                alt = base + (int64_t)concat_row(Q, K ^ (1 << min_k[ko]), PE, nc, npe) * stride;
                up = surrogate_up(km); flip = min_k[ko]; pos = i;
            }
            const bool pe_flip = npe > 0 && fabsf(pm) < fabsf(qm) && fabsf(pm) < fabsf(km);
            const int64_t palt = pe_flip ? base + (int64_t)concat_row(Q, K, PE ^ (1 << pk), nc, npe) * stride : 0;
            const int2 a = __ldg(anchors + (size_t)t * nc + flip);
            float *dx = dX + (b * S + pos) * (int64_t)n_inputs;
            for (int p0 = 0; p0 < P; p0 += G) {
                const int p1 = min(P, p0 + G);
                double ms = 0.0, as = 0.0, ps = 0.0;
                for (int p = p0; p < p1; p++) ms += (double)__ldg(W + sparse_slot(row, p, G)) * (double)__ldg(dy + tg[p]);
                for (int p = p0; p < p1; p++) as += (double)__ldg(W + sparse_slot(alt, p, G)) * (double)__ldg(dy + tg[p]);
                const double du = up * (ms - as);
                if (fabs(du) > kEps) {
                    if (INT_MODE) {
                        const int32_t d = to_fixed(du, fixed_scale);
                        atomicAdd(reinterpret_cast<int32_t *>(dx) + a.x, d);
                        atomicAdd(reinterpret_cast<int32_t *>(dx) + a.y, -d);
                    } else {
                        atomicAdd(dx + a.x, (float)du);
                        atomicAdd(dx + a.y, -(float)du);
                    }
                }
                if (pe_flip) {
                    for (int p = p0; p < p1; p++) ps += (double)__ldg(W + sparse_slot(palt, p, G)) * (double)__ldg(dy + tg[p]);
                    const double dp = surrogate_up(pm) * (ms - ps);
                    if (INT_MODE) atomicAdd(reinterpret_cast<int32_t *>(dPE) + po * npe + pk, to_fixed(dp, fixed_scale));
                    else atomicAdd(dPE + po * npe + pk, (float)dp);
                }
            }
        }
        if (target) {
            for (int p = 0; p < P; p++) {
                const double g = (double)__ldg(dy + tg[p]);
                if (fabs(g) > kEps) {
                    const int64_t slot = sparse_slot(row, p, G);
                    if (INT_MODE) atomicAdd(reinterpret_cast<int32_t *>(target) + slot, to_fixed(g * lr, fixed_scale));
                    else atomicAdd(target + slot, (float)(g * lr));
                }
            }
        }
    }
}

static int validate_sparse_rows(const lutb_sparse_index *sp, SparseRows *out) {
    LUTB_REQUIRE(sp != nullptr, LUTB_ERR_NULL, "sparse index is NULL");
    LUTB_REQUIRE(sp->det_wbase && sp->det_stride && sp->det_count && sp->det_sstart && sp->syn_target, LUTB_ERR_NULL,
                 "a sparse index array is NULL");
    LUTB_REQUIRE(sp->group_size > 0 && sp->n_weights > 0, LUTB_ERR_SHAPE, "empty sparse index");
    out->wbase = sp->det_wbase; out->stride = sp->det_stride; out->count = sp->det_count;
    out->sstart = sp->det_sstart; out->target = sp->syn_target; out->group = sp->group_size;
    return LUTB_OK;
}

static int validate_concat(const lutb_layer_cfg *cfg, int64_t batch) {
    int rc = validate_cfg(cfg);
    if (rc) return rc;
    LUTB_REQUIRE(batch > 0, LUTB_ERR_SHAPE, "batch_size == 0");
    LUTB_REQUIRE(batch <= 65535, LUTB_ERR_SHAPE, "batch_size > 65535 is not supported by the sequence kernels");
    LUTB_REQUIRE(cfg->seq_len > 1, LUTB_ERR_MODE, "forward_step_concat should only be called when sequence_length > 1");
    LUTB_REQUIRE(2 * cfg->n_anchors + cfg->pos_dim <= 30, LUTB_ERR_SHAPE, "more than 2^30 rows per detector");
    return LUTB_OK;
}

}  // namespace lutb

using namespace lutb;

static int launch_check_positional(const lutb_layer_cfg *cfg, const float *pos_embeddings, int32_t *pos_idx,
                                   float *pos_min_delta, int32_t *pos_min_k, cudaStream_t st) {
    const int64_t n = (int64_t)(cfg->seq_len - 1) * cfg->n_detectors;
    const bool train = pos_min_delta != nullptr;
    KernelScope scope(K_CHECK_POSITIONAL, st);
    if (train) check_positional_kernel<true><<<(unsigned)((n + 127) / 128), 128, 0, st>>>(pos_embeddings, n, cfg->pos_dim, cfg->cmp_eps, pos_idx, pos_min_delta, pos_min_k);
    else check_positional_kernel<false><<<(unsigned)((n + 127) / 128), 128, 0, st>>>(pos_embeddings, n, cfg->pos_dim, cfg->cmp_eps, pos_idx, nullptr, nullptr);
    LUTB_LAUNCH_CHECK();
    return LUTB_OK;
}

// Lane groups and vector width of the fp32 pair kernels: VEC = 4 where rows and tensors allow 16-byte accesses; LG lanes
// cover a row of up to LG * VEC columns (narrower rows: several pairs side by side in a warp), wider rows are walked in steps.
template <class F>
static int dispatch_pair_kernel(bool vec4, int n_outputs, F &&f) {
    const int v = vec4 ? (n_outputs + 3) / 4 : n_outputs;
    if (vec4) {
        if (v > 16) return f(std::integral_constant<int, 32>{}, std::integral_constant<int, 4>{});
        if (v > 8) return f(std::integral_constant<int, 16>{}, std::integral_constant<int, 4>{});
        if (v > 4) return f(std::integral_constant<int, 8>{}, std::integral_constant<int, 4>{});
        if (v > 2) return f(std::integral_constant<int, 4>{}, std::integral_constant<int, 4>{});
        return f(std::integral_constant<int, 2>{}, std::integral_constant<int, 4>{});
    }
    if (v > 8) return f(std::integral_constant<int, 32>{}, std::integral_constant<int, 1>{});
    return f(std::integral_constant<int, 8>{}, std::integral_constant<int, 1>{});
}

static bool aligned16(const void *p) { return (reinterpret_cast<uintptr_t>(p) & 15) == 0; }

// Blocks of one launch are (detector, sample) with the samples of a detector next to one another; more than 2^31 of them
// are launched a range of samples at a time.
static int64_t samples_per_launch(int n_detectors) { return max((int64_t)1, (int64_t)0x7FFFFFFF / n_detectors); }

static int launch_concat_pairs_forward(const lutb_layer_cfg *cfg, int64_t batch, const float *weights, const int32_t *idx,
                                       const int32_t *pos_idx, float *y, int j_begin, int j_end, cudaStream_t st) {
    const int S = cfg->seq_len, npe = cfg->pos_dim, Nt = cfg->n_detectors, O = cfg->n_outputs, Nc = cfg->n_anchors;
    const size_t smem = (size_t)(2 * S) * 4;
    LUTB_REQUIRE(smem <= (size_t)kMaxSmemPerBlock - 1024, LUTB_ERR_SHAPE, "sequence too long for the sequence kernels");
    KernelScope scope(K_CONCAT_FORWARD, st);
    if (cfg->int_mode) {
        dim3 grid((unsigned)Nt, (unsigned)batch);
        if (smem > kPlainSmem) LUTB_CUDA(cudaFuncSetAttribute(concat_forward_fixed_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
        concat_forward_fixed_kernel<<<grid, 256, smem, st>>>(weights, idx, pos_idx, y, S, O, Nt, Nc, npe, cfg->int_rescaler, j_begin, j_end);
        LUTB_LAUNCH_CHECK();
        return LUTB_OK;
    }
    const bool vec4 = O % 4 == 0 && aligned16(weights) && aligned16(y);
    const int threads = 32 * min(8, (j_end - j_begin + 1) / 2);
    const int64_t per = samples_per_launch(Nt);
    for (int64_t b0 = 0; b0 < batch; b0 += per) {
        const int n = (int)min(per, batch - b0);
        const int rc = dispatch_pair_kernel(vec4, O, [&](auto lg, auto vec) -> int {
            auto kern = concat_forward_kernel<lg.value, vec.value>;
            if (smem > kPlainSmem) LUTB_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
            kern<<<(unsigned)((int64_t)Nt * n), threads, smem, st>>>(weights, idx + b0 * S * Nt, pos_idx, y + b0 * S * O, n, S, O, Nt, Nc,
                                                                   npe, j_begin, j_end);
            return LUTB_OK;
        });
        if (rc) return rc;
        LUTB_LAUNCH_CHECK();
    }
    return LUTB_OK;
}

// fp32 accumulators only
static int launch_concat_pairs_backward(const lutb_layer_cfg *cfg, int64_t batch, float *weights, const float *dY,
                                        const int32_t *anchors, const int32_t *idx, const float *min_delta,
                                        const int32_t *min_k, const int32_t *pos_idx, const float *pos_min_delta,
                                        const int32_t *pos_min_k, float *dX, float *dPE, float *dW, double external_lr,
                                        int j_begin, int j_end, cudaStream_t st) {
    const int S = cfg->seq_len, npe = cfg->pos_dim, Nt = cfg->n_detectors, O = cfg->n_outputs, Nc = cfg->n_anchors;
    double lr = cfg->lr_meta;
    if (external_lr >= 0.0) lr *= -(double)(float)external_lr;
    const int2 *an = reinterpret_cast<const int2 *>(anchors);
    // the bound of the entry point, token state plus eight rows of dY, is an older kernel's and more than the launches below take:
    // what was refused stays refused
    LUTB_REQUIRE(((size_t)((6 * S + 3) & ~3) + (size_t)8 * ((O + 3) & ~3)) * 4 <= (size_t)kMaxSmemPerBlock - 1024, LUTB_ERR_SHAPE,
                 "sequence too long for the sequence kernels");
    const int64_t per = samples_per_launch(Nt);
    // the (token, anchor pair) cells of dX join the token state while four blocks still fit an SM
    const size_t state = (size_t)6 * S * 4, cells = (size_t)S * Nc * 4;
    const int smem_dx = state + cells <= 48 * 1024;
    const int threads = 32 * min(8, (j_end - j_begin + 1) / 2);
    auto pass = [&](auto dx_c, auto dw_c, float *target) -> int {
        constexpr bool DX = decltype(dx_c)::value, DWF = decltype(dw_c)::value;
        const bool vec4 = O % 4 == 0 && aligned16(weights) && aligned16(dY) && aligned16(target);
        const size_t smem = state + (DX && smem_dx ? cells : 0);
        for (int64_t b0 = 0; b0 < batch; b0 += per) {
            const int n = (int)min(per, batch - b0);
            const int64_t tok = b0 * S;
            const int rc = dispatch_pair_kernel(vec4, O, [&](auto lg, auto vec) -> int {
                constexpr int L = decltype(lg)::value, V = decltype(vec)::value;
                auto kern = concat_backward_kernel<L, V, DX, DWF, false>;
                // (rows of one step; 32 lanes with vectors would spill: 128 outputs 74 us against 54.  Fewer blocks than SMs: the
                // second loop's latency counts instead, 1 x 32 tokens 18 us against 13)
                if constexpr (L <= 16 || V == 1) {
                    if (O <= L * V && (int64_t)Nt * n >= device_info().sm_count) kern = concat_backward_kernel<L, V, DX, DWF, true>;
                }
                if (smem > kPlainSmem) LUTB_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
                kern<<<(unsigned)((int64_t)Nt * n), threads, smem, st>>>(
                    weights, dY + tok * O, an, idx + tok * Nt, min_delta + tok * Nt, min_k + tok * Nt, pos_idx, pos_min_delta, pos_min_k,
                    dX + tok * cfg->n_inputs, dPE, target, n, S, cfg->n_inputs, O, Nt, Nc, npe, lr, j_begin, j_end, smem_dx);
                return LUTB_OK;
            });
            if (rc) return rc;
            LUTB_LAUNCH_CHECK();
        }
        return LUTB_OK;
    };
    if (external_lr >= 0.0) {
        {
            // in-place SGD: every input gradient is computed from the unmodified tables first
            KernelScope scope(K_CONCAT_BACKWARD, st);
            const int rc = pass(std::true_type{}, std::false_type{}, nullptr);
            if (rc) return rc;
        }
        KernelScope scope(K_CONCAT_WEIGHT_UPDATE, st);
        return pass(std::false_type{}, std::true_type{}, weights);
    }
    KernelScope scope(K_CONCAT_BACKWARD, st);
    return pass(std::true_type{}, std::true_type{}, dW);
}

extern "C" int lutb_check_detectors(const lutb_layer_cfg *cfg, int64_t rows, const float *x, const int32_t *anchors,
                                    int32_t *idx, float *min_delta, int32_t *min_k, void *stream) {
    int rc = validate_cfg(cfg);
    if (rc) return rc;
    LUTB_REQUIRE(rows > 0, LUTB_ERR_SHAPE, "no input rows");
    LUTB_REQUIRE(x && anchors && idx, LUTB_ERR_NULL, "a required tensor pointer is NULL");
    LUTB_REQUIRE((min_delta == nullptr) == (min_k == nullptr), LUTB_ERR_MODE,
                 "min_anchor_deltas and min_anchor_delta_indices must be given together");
    return launch_check_detectors(x, rows, cfg->n_inputs, anchors, cfg->n_detectors, cfg->n_anchors, cfg->cmp_eps, idx,
                                  min_delta, min_k, static_cast<cudaStream_t>(stream));
}

extern "C" int lutb_check_positional(const lutb_layer_cfg *cfg, const float *pos_embeddings, int32_t *pos_idx,
                                     float *pos_min_delta, int32_t *pos_min_k, void *stream) {
    int rc = validate_cfg(cfg);
    if (rc) return rc;
    LUTB_REQUIRE(cfg->seq_len > 1 && cfg->pos_dim > 0, LUTB_ERR_MODE, "the layer has no positional embeddings");
    LUTB_REQUIRE(pos_embeddings && pos_idx, LUTB_ERR_NULL, "positional embeddings / indices are NULL");
    LUTB_REQUIRE((pos_min_delta == nullptr) == (pos_min_k == nullptr), LUTB_ERR_MODE,
                 "positional min deltas and their indices must be given together");
    return launch_check_positional(cfg, pos_embeddings, pos_idx, pos_min_delta, pos_min_k, static_cast<cudaStream_t>(stream));
}

static int validate_query_range(const lutb_layer_cfg *cfg, int j_begin, int j_end) {
    LUTB_REQUIRE(j_begin >= 0 && j_begin <= j_end && j_end <= cfg->seq_len, LUTB_ERR_SHAPE,
                 "query range [%d, %d) outside [0, %d)", j_begin, j_end, cfg->seq_len);
    return LUTB_OK;
}

extern "C" int lutb_concat_pairs_forward(const lutb_layer_cfg *cfg, int64_t batch, const float *weights,
                                         const int32_t *idx, const int32_t *pos_idx, float *y, int32_t j_begin,
                                         int32_t j_end, void *stream) {
    int rc = validate_concat(cfg, batch);
    if (rc) return rc;
    rc = validate_query_range(cfg, j_begin, j_end);
    if (rc) return rc;
    LUTB_REQUIRE(weights && idx && y, LUTB_ERR_NULL, "a required tensor pointer is NULL");
    LUTB_REQUIRE(cfg->pos_dim == 0 || pos_idx, LUTB_ERR_NULL, "positional indices are NULL");
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    if (j_begin == j_end) return LUTB_OK;
    rc = launch_concat_pairs_forward(cfg, batch, weights, idx, pos_idx, y, j_begin, j_end, st);
    if (rc) return rc;
    if (cfg->int_mode) {
        // only the rows of the range hold fixed-point accumulators
        for (int64_t b = 0; b < batch; b++) {
            rc = launch_fixed_to_float(y + (b * cfg->seq_len + j_begin) * (int64_t)cfg->n_outputs,
                                       (int64_t)(j_end - j_begin) * cfg->n_outputs, cfg->int_rescaler, st);
            if (rc) return rc;
        }
    }
    return LUTB_OK;
}

extern "C" int lutb_concat_pairs_backward(const lutb_layer_cfg *cfg, int64_t batch, float *weights, const float *dY,
                                          const int32_t *anchors, const int32_t *idx, const float *min_delta,
                                          const int32_t *min_k, const int32_t *pos_idx, const float *pos_min_delta,
                                          const int32_t *pos_min_k, float *dX, float *dPE, float *dW, double external_lr,
                                          int32_t j_begin, int32_t j_end, void *stream) {
    int rc = validate_concat(cfg, batch);
    if (rc) return rc;
    rc = validate_query_range(cfg, j_begin, j_end);
    if (rc) return rc;
    LUTB_REQUIRE(cfg->int_mode == 0, LUTB_ERR_MODE, "the query-range backward needs fp32 accumulators");
    LUTB_REQUIRE(weights && dY && anchors && idx && min_delta && min_k && dX, LUTB_ERR_NULL, "a required tensor pointer is NULL");
    LUTB_REQUIRE(cfg->pos_dim == 0 || (pos_idx && pos_min_delta && pos_min_k && dPE), LUTB_ERR_NULL, "positional tensors are NULL");
    LUTB_REQUIRE(!(external_lr >= 0.0 && dW != nullptr), LUTB_ERR_MODE,
                 "in internal weight gradients mode w_weights_gradients should be nullptr");
    LUTB_REQUIRE(!(external_lr < 0.0 && dW == nullptr), LUTB_ERR_NULL, "w_weights_gradients is NULL");
    if (j_begin == j_end) return LUTB_OK;
    return launch_concat_pairs_backward(cfg, batch, weights, dY, anchors, idx, min_delta, min_k, pos_idx, pos_min_delta,
                                        pos_min_k, dX, dPE, dW, external_lr, j_begin, j_end, static_cast<cudaStream_t>(stream));
}

extern "C" int lutb_concat_forward(const lutb_layer_cfg *cfg, int64_t batch, const float *weights, const float *x,
                                   const int32_t *anchors, const float *pos_embeddings, float *y, int32_t *idx,
                                   float *min_delta, int32_t *min_k, int32_t *pos_idx, float *pos_min_delta,
                                   int32_t *pos_min_k, void *stream) {
    int rc = validate_concat(cfg, batch);
    if (rc) return rc;
    LUTB_REQUIRE(weights && x && anchors && y && idx, LUTB_ERR_NULL, "a required tensor pointer is NULL");
    LUTB_REQUIRE((min_delta == nullptr) == (min_k == nullptr), LUTB_ERR_MODE,
                 "min_anchor_deltas and min_anchor_delta_indices must be given together");
    const int S = cfg->seq_len, npe = cfg->pos_dim, Nt = cfg->n_detectors;
    const bool train = min_delta != nullptr;
    if (npe > 0) {
        LUTB_REQUIRE(pos_embeddings && pos_idx, LUTB_ERR_NULL, "positional embeddings / indices are NULL");
        LUTB_REQUIRE(!train || (pos_min_delta && pos_min_k), LUTB_ERR_NULL, "positional min-delta outputs are NULL");
    }
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    rc = launch_check_detectors(x, batch * S, cfg->n_inputs, anchors, Nt, cfg->n_anchors, cfg->cmp_eps, idx, min_delta,
                                min_k, st);
    if (rc) return rc;
    if (npe > 0) {
        rc = launch_check_positional(cfg, pos_embeddings, pos_idx, train ? pos_min_delta : nullptr,
                                     train ? pos_min_k : nullptr, st);
        if (rc) return rc;
    }
    rc = launch_concat_pairs_forward(cfg, batch, weights, idx, pos_idx, y, 0, S, st);
    if (rc) return rc;
    if (cfg->int_mode) return launch_fixed_to_float(y, batch * S * (int64_t)cfg->n_outputs, cfg->int_rescaler, st);
    return LUTB_OK;
}

extern "C" int lutb_concat_backward(const lutb_layer_cfg *cfg, int64_t batch, float *weights, const float *dY,
                                    const int32_t *anchors, const int32_t *idx, const float *min_delta,
                                    const int32_t *min_k, const int32_t *pos_idx, const float *pos_min_delta,
                                    const int32_t *pos_min_k, float *dX, float *dPE, float *dW, double external_lr,
                                    void *stream) {
    int rc = validate_concat(cfg, batch);
    if (rc) return rc;
    LUTB_REQUIRE(weights && dY && anchors && idx && min_delta && min_k && dX, LUTB_ERR_NULL, "a required tensor pointer is NULL");
    const int S = cfg->seq_len, npe = cfg->pos_dim, Nt = cfg->n_detectors, O = cfg->n_outputs, Nc = cfg->n_anchors;
    LUTB_REQUIRE(npe == 0 || (pos_idx && pos_min_delta && pos_min_k && dPE), LUTB_ERR_NULL, "positional tensors are NULL");
    LUTB_REQUIRE(!(external_lr >= 0.0 && dW != nullptr), LUTB_ERR_MODE,
                 "in internal weight gradients mode w_weights_gradients should be nullptr");
    LUTB_REQUIRE(!(external_lr < 0.0 && dW == nullptr), LUTB_ERR_NULL, "w_weights_gradients is NULL");
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    if (cfg->int_mode) {
        double lr = cfg->lr_meta;
        if (external_lr >= 0.0) lr *= -(double)(float)external_lr;
        const int2 *an = reinterpret_cast<const int2 *>(anchors);
        const int n_ob = (O + cfg->forward_group - 1) / cfg->forward_group;
        const int64_t total = batch * S * (int64_t)Nt * S * n_ob;
        const int64_t blocks = min((total + 127) / 128, (int64_t)device_info().sm_count * 64);
        KernelScope scope(K_CONCAT_BACKWARD, st);
        concat_backward_fixed_kernel<<<(unsigned)blocks, 128, 0, st>>>(weights, dY, an, idx, min_delta, min_k, pos_idx, pos_min_delta, pos_min_k, dX, dPE, dW, batch, S, cfg->n_inputs, O, Nt, Nc, npe, cfg->forward_group, lr, cfg->int_rescaler);
        LUTB_LAUNCH_CHECK();
    } else {
        rc = launch_concat_pairs_backward(cfg, batch, weights, dY, anchors, idx, min_delta, min_k, pos_idx, pos_min_delta,
                                          pos_min_k, dX, dPE, dW, external_lr, 0, S, st);
        if (rc) return rc;
    }
    if (cfg->int_mode) {
        rc = launch_fixed_to_float(dX, batch * S * (int64_t)cfg->n_inputs, cfg->int_rescaler, st);
        if (rc) return rc;
        if (dW) {
            rc = launch_fixed_to_float(dW, (int64_t)Nt * ((int64_t)1 << (2 * Nc + npe)) * O, cfg->int_rescaler, st);
            if (rc) return rc;
        }
        if (npe > 0) rc = launch_fixed_to_float(dPE, (int64_t)(S - 1) * Nt * npe, cfg->int_rescaler, st);
    }
    return rc;
}

extern "C" int lutb_concat_sparse_forward(const lutb_layer_cfg *cfg, const lutb_sparse_index *sparse, int64_t batch,
                                          const float *weights, const float *x, const int32_t *anchors,
                                          const float *pos_embeddings, float *y, int32_t *idx, float *min_delta,
                                          int32_t *min_k, int32_t *pos_idx, float *pos_min_delta, int32_t *pos_min_k,
                                          void *stream) {
    int rc = validate_concat(cfg, batch);
    if (rc) return rc;
    SparseRows rows;
    rc = validate_sparse_rows(sparse, &rows);
    if (rc) return rc;
    LUTB_REQUIRE(weights && x && anchors && y && idx, LUTB_ERR_NULL, "a required tensor pointer is NULL");
    LUTB_REQUIRE((min_delta == nullptr) == (min_k == nullptr), LUTB_ERR_MODE,
                 "min_anchor_deltas and min_anchor_delta_indices must be given together");
    const int S = cfg->seq_len, npe = cfg->pos_dim, Nt = cfg->n_detectors;
    const bool train = min_delta != nullptr;
    if (npe > 0) {
        LUTB_REQUIRE(pos_embeddings && pos_idx, LUTB_ERR_NULL, "positional embeddings / indices are NULL");
        LUTB_REQUIRE(!train || (pos_min_delta && pos_min_k), LUTB_ERR_NULL, "positional min-delta outputs are NULL");
    }
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    rc = launch_check_detectors(x, batch * S, cfg->n_inputs, anchors, Nt, cfg->n_anchors, cfg->cmp_eps, idx, min_delta,
                                min_k, st);
    if (rc) return rc;
    if (npe > 0) {
        const int64_t n = (int64_t)(S - 1) * Nt;
        KernelScope scope(K_CHECK_POSITIONAL, st);
        if (train) check_positional_kernel<true><<<(unsigned)((n + 127) / 128), 128, 0, st>>>(pos_embeddings, n, npe, cfg->cmp_eps, pos_idx, pos_min_delta, pos_min_k);
        else check_positional_kernel<false><<<(unsigned)((n + 127) / 128), 128, 0, st>>>(pos_embeddings, n, npe, cfg->cmp_eps, pos_idx, nullptr, nullptr);
        LUTB_LAUNCH_CHECK();
    }
    {
        const int64_t total = batch * S * (int64_t)Nt * S;
        const int64_t blocks = min((total + 127) / 128, (int64_t)device_info().sm_count * 64);
        KernelScope scope(K_CONCAT_FORWARD, st);
        if (cfg->int_mode)
            concat_sparse_forward_kernel<true><<<(unsigned)blocks, 128, 0, st>>>(weights, idx, pos_idx, y, rows, batch, S, cfg->n_outputs, Nt, cfg->n_anchors, npe, cfg->int_rescaler);
        else
            concat_sparse_forward_kernel<false><<<(unsigned)blocks, 128, 0, st>>>(weights, idx, pos_idx, y, rows, batch, S, cfg->n_outputs, Nt, cfg->n_anchors, npe, cfg->int_rescaler);
        LUTB_LAUNCH_CHECK();
    }
    if (cfg->int_mode) return launch_fixed_to_float(y, batch * S * (int64_t)cfg->n_outputs, cfg->int_rescaler, st);
    return LUTB_OK;
}

extern "C" int lutb_concat_sparse_backward(const lutb_layer_cfg *cfg, const lutb_sparse_index *sparse, int64_t batch,
                                           float *weights, const float *dY, const int32_t *anchors, const int32_t *idx,
                                           const float *min_delta, const int32_t *min_k, const int32_t *pos_idx,
                                           const float *pos_min_delta, const int32_t *pos_min_k, float *dX, float *dPE,
                                           float *dW, double external_lr, void *stream) {
    int rc = validate_concat(cfg, batch);
    if (rc) return rc;
    SparseRows rows;
    rc = validate_sparse_rows(sparse, &rows);
    if (rc) return rc;
    LUTB_REQUIRE(weights && dY && anchors && idx && min_delta && min_k && dX, LUTB_ERR_NULL, "a required tensor pointer is NULL");
    const int S = cfg->seq_len, npe = cfg->pos_dim, Nt = cfg->n_detectors, O = cfg->n_outputs, Nc = cfg->n_anchors;
    LUTB_REQUIRE(npe == 0 || (pos_idx && pos_min_delta && pos_min_k && dPE), LUTB_ERR_NULL, "positional tensors are NULL");
    LUTB_REQUIRE(!(external_lr >= 0.0 && dW != nullptr), LUTB_ERR_MODE,
                 "in internal weight gradients mode w_weights_gradients should be nullptr");
    LUTB_REQUIRE(!(external_lr < 0.0 && dW == nullptr), LUTB_ERR_NULL, "w_weights_gradients is NULL");
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    double lr = cfg->lr_meta;
    if (external_lr >= 0.0) lr *= -(double)(float)external_lr;
    const int2 *an = reinterpret_cast<const int2 *>(anchors);
    const int64_t total = batch * S * (int64_t)Nt * S;
    const int64_t blocks = min((total + 127) / 128, (int64_t)device_info().sm_count * 64);
#define LUTB_CS_BWD(DO_DX, TARGET)                                                                                          \
    do {                                                                                                                    \
        if (cfg->int_mode)                                                                                                  \
            concat_sparse_backward_kernel<true><<<(unsigned)blocks, 128, 0, st>>>(weights, dY, an, idx, min_delta, min_k, pos_idx, pos_min_delta, pos_min_k, dX, dPE, TARGET, rows, batch, S, cfg->n_inputs, O, Nt, Nc, npe, DO_DX, lr, cfg->int_rescaler); \
        else                                                                                                                \
            concat_sparse_backward_kernel<false><<<(unsigned)blocks, 128, 0, st>>>(weights, dY, an, idx, min_delta, min_k, pos_idx, pos_min_delta, pos_min_k, dX, dPE, TARGET, rows, batch, S, cfg->n_inputs, O, Nt, Nc, npe, DO_DX, lr, cfg->int_rescaler); \
    } while (0)
    if (external_lr >= 0.0) {
        // in-place SGD: every input gradient is computed from the unmodified tables first
        {
            KernelScope scope(K_CONCAT_BACKWARD, st);
            LUTB_CS_BWD(1, nullptr);
        }
        LUTB_LAUNCH_CHECK();
        KernelScope scope(K_CONCAT_WEIGHT_UPDATE, st);
        LUTB_CS_BWD(0, weights);
    } else {
        KernelScope scope(K_CONCAT_BACKWARD, st);
        LUTB_CS_BWD(1, dW);
    }
#undef LUTB_CS_BWD
    LUTB_LAUNCH_CHECK();
    if (cfg->int_mode) {
        rc = launch_fixed_to_float(dX, batch * S * (int64_t)cfg->n_inputs, cfg->int_rescaler, st);
        if (rc) return rc;
        if (dW) {
            rc = launch_fixed_to_float(dW, sparse->n_weights, cfg->int_rescaler, st);
            if (rc) return rc;
        }
        if (npe > 0) rc = launch_fixed_to_float(dPE, (int64_t)(S - 1) * Nt * npe, cfg->int_rescaler, st);
    }
    return rc;
}
