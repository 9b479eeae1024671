// General fp32 GEMMs on the sm_100a tensor cores (lutb_fp32_gemm; the histogram path of the product-mode layer has kernels of
// its own, hist_gemm_sm100.cu).
//
// Results keep fp32 accuracy (1e-5), so plain TF32 or BF16 inputs are not an option.  Two routes, both CUTLASS 3
// collectives instantiated for sm_100a (operands arrive in shared memory by TMA - a cluster of one block or one pair: plain copies of this
// GPU's own memory -, tcgen05.mma accumulates in fp32 in tensor memory, the epilogue reads the accumulators back with
// tcgen05.ld and applies alpha / beta):
//
//   split TF32 (default)  every fp32 operand x is written once as hi = x rounded to TF32 and lo = x - hi (exact)
//                         rounded to TF32, and the product is formed as hi.hi + hi.lo + lo.hi; concatenated copies
//                         make that ONE TF32 GEMM where the layouts allow.  The dropped lo.lo term and the rounding of lo are each
//                         below 2^-22 relative.
//   fast fp32             one GEMM whose mainloop splits the operands into three BF16 terms on the fly (CUTLASS'
//                         "FastF32" schedule); simpler, no scratch, but bound by the conversion work: 80-90 TFLOP/s on
//                         the contraction shapes against 2-3 times that for the split TF32 route.
//
// Results agree with an fp32 FMA contraction to about 1e-6 relative; the summation order differs.
// All matrices are fp32 with 16-byte aligned base pointers and leading dimensions that are multiples of 4.
#include "fp32_gemm_sm100.cuh"

#ifdef LUTB_NO_CUTLASS
// built without a CUTLASS header tree
namespace lutb {
bool tc_gemm_available() { return false; }
size_t tc_gemm_workspace(TcGemmKind, int, int, int) { return 0; }
size_t tc_gemm_fast_workspace(int, int, int) { return 0; }
int tc_gemm(TcGemmKind, int, int, int, const float *, int64_t, const float *, int64_t, float *, int64_t, float, float, void *, size_t,
            cudaStream_t) {
    set_error("the library was built without the tensor-core contractions (no CUTLASS headers at build time)");
    return LUTB_ERR_MODE;
}
int tc_gemm_fast(TcGemmKind, int, int, int, const float *, int64_t, const float *, int64_t, float *, int64_t, float, float,
                 void *, size_t, cudaStream_t) {
    set_error("the library was built without the tensor-core contractions (no CUTLASS headers at build time)");
    return LUTB_ERR_MODE;
}
}  // namespace lutb
#else

#include "cutlass/cutlass.h"
#include "cutlass/epilogue/collective/collective_builder.hpp"
#include "cutlass/gemm/collective/collective_builder.hpp"
#include "cutlass/gemm/device/gemm_universal_adapter.h"
#include "cutlass/gemm/kernel/gemm_universal.hpp"
#include "cutlass/util/packed_stride.hpp"

namespace lutb {

using namespace cute;

template <class LayoutA, class LayoutB>
struct FastF32Gemm {
    using Element = float;
    using LayoutC = cutlass::layout::RowMajor;
    static constexpr int kAlign = 4;   // 16 bytes
    using MmaTile = Shape<_128, _128, _16>;
    using Cluster = Shape<_1, _1, _1>;
    using Epilogue = typename cutlass::epilogue::collective::CollectiveBuilder<
        cutlass::arch::Sm100, cutlass::arch::OpClassTensorOp, MmaTile, Cluster,
        cutlass::epilogue::collective::EpilogueTileAuto, float, float, Element, LayoutC, kAlign, Element, LayoutC, kAlign,
        cutlass::epilogue::collective::EpilogueScheduleAuto>::CollectiveOp;
    using Mainloop = typename cutlass::gemm::collective::CollectiveBuilder<
        cutlass::arch::Sm100, cutlass::arch::OpClassTensorOp, Element, LayoutA, kAlign, Element, LayoutB, kAlign, float, MmaTile,
        Cluster, cutlass::gemm::collective::StageCountAutoCarveout<static_cast<int>(sizeof(typename Epilogue::SharedStorage))>,
        cutlass::gemm::KernelTmaWarpSpecialized1SmFastFP32Sm100>::CollectiveOp;
    using Kernel = cutlass::gemm::kernel::GemmUniversal<Shape<int, int, int, int>, Mainloop, Epilogue>;
    using Gemm = cutlass::gemm::device::GemmUniversalAdapter<Kernel>;
    using StrideA = typename Kernel::StrideA;
    using StrideB = typename Kernel::StrideB;
    using StrideC = typename Kernel::StrideC;
    using StrideD = typename Kernel::StrideD;
};

// PAIR: two SMs share a 256 x 256 tile (cta_group::2): each loads its half of both operands, so that an operand byte from
// shared memory feeds twice the multiply-adds.  The loads are plain (a cluster of exactly one pair has nobody to multicast to).
template <class LayoutA, class LayoutB, bool PAIR = false>
struct Tf32Gemm {
    using Element = cutlass::tfloat32_t;   // fp32 storage; the MMA reads sign, exponent and the top 10 mantissa bits
    using LayoutC = cutlass::layout::RowMajor;
    static constexpr int kAlign = 4;
    using MmaTile = cute::conditional_t<PAIR, Shape<_256, _256, _32>, Shape<_128, _128, _32>>;
    using Cluster = cute::conditional_t<PAIR, Shape<_2, _1, _1>, Shape<_1, _1, _1>>;
    using Epilogue = typename cutlass::epilogue::collective::CollectiveBuilder<
        cutlass::arch::Sm100, cutlass::arch::OpClassTensorOp, MmaTile, Cluster,
        cutlass::epilogue::collective::EpilogueTileAuto, float, float, float, LayoutC, kAlign, float, LayoutC, kAlign,
        cutlass::epilogue::collective::EpilogueScheduleAuto>::CollectiveOp;
    using Mainloop = typename cutlass::gemm::collective::CollectiveBuilder<
        cutlass::arch::Sm100, cutlass::arch::OpClassTensorOp, Element, LayoutA, kAlign, Element, LayoutB, kAlign, float, MmaTile,
        Cluster, cutlass::gemm::collective::StageCountAutoCarveout<static_cast<int>(sizeof(typename Epilogue::SharedStorage))>,
        cutlass::gemm::collective::KernelScheduleAuto>::CollectiveOp;
    using Kernel = cutlass::gemm::kernel::GemmUniversal<Shape<int, int, int, int>, Mainloop, Epilogue>;
    using Gemm = cutlass::gemm::device::GemmUniversalAdapter<Kernel>;
    using StrideA = typename Kernel::StrideA;
    using StrideB = typename Kernel::StrideB;
    using StrideC = typename Kernel::StrideC;
    using StrideD = typename Kernel::StrideD;
};

template <class Cfg>
static size_t workspace_of(int M, int N, int K) {
    typename Cfg::Gemm::Arguments args{cutlass::gemm::GemmUniversalMode::kGemm, {M, N, K, 1}};
    return Cfg::Gemm::get_workspace_size(args);
}

template <class Cfg>
static int run(int M, int N, int K, const float *A, int64_t lda, const float *B, int64_t ldb, float *C, int64_t ldc,
               float alpha, float beta, void *workspace, size_t workspace_bytes, cudaStream_t stream) {
    typename Cfg::StrideA sa;
    typename Cfg::StrideB sb;
    typename Cfg::StrideC sc;
    // the dynamic (non unit) mode of every stride is the leading dimension
    if constexpr (cute::is_same_v<decltype(get<1>(sa)), cute::Int<1>>) sa = make_stride(lda, Int<1>{}, int64_t(0));
    else sa = make_stride(Int<1>{}, lda, int64_t(0));
    if constexpr (cute::is_same_v<decltype(get<1>(sb)), cute::Int<1>>) sb = make_stride(ldb, Int<1>{}, int64_t(0));
    else sb = make_stride(Int<1>{}, ldb, int64_t(0));
    sc = make_stride(ldc, Int<1>{}, int64_t(0));
    using ElementAB = typename Cfg::Element;
    typename Cfg::Gemm::Arguments args{cutlass::gemm::GemmUniversalMode::kGemm,
                                       {M, N, K, 1},
                                       {reinterpret_cast<const ElementAB *>(A), sa, reinterpret_cast<const ElementAB *>(B), sb},
                                       {{alpha, beta}, C, sc, C, sc}};
    typename Cfg::Gemm gemm;
    LUTB_REQUIRE(gemm.can_implement(args) == cutlass::Status::kSuccess, LUTB_ERR_SHAPE,
                 "tensor-core contraction: shapes or alignments not supported (M=%d N=%d K=%d)", M, N, K);
    const size_t need = Cfg::Gemm::get_workspace_size(args);
    LUTB_REQUIRE(need <= workspace_bytes, LUTB_ERR_WORKSPACE, "tensor-core contraction needs %zu bytes of workspace", need);
    cutlass::Status st = gemm.initialize(args, workspace, stream);
    LUTB_REQUIRE(st == cutlass::Status::kSuccess, LUTB_ERR_MODE, "tensor-core contraction: initialisation failed (%d)", (int)st);
    st = gemm.run(stream);
    LUTB_REQUIRE(st == cutlass::Status::kSuccess, LUTB_ERR_MODE, "tensor-core contraction: launch failed (%d)", (int)st);
    return LUTB_OK;
}

// operand layouts: TN = A [M x K] row-major, B stored as [N x K] row-major; NN = A [M x K], B [K x N] row-major;
// TT = A stored as [K x M] row-major, B [K x N] row-major
using FastTN = FastF32Gemm<cutlass::layout::RowMajor, cutlass::layout::ColumnMajor>;
using FastNN = FastF32Gemm<cutlass::layout::RowMajor, cutlass::layout::RowMajor>;
using FastTT = FastF32Gemm<cutlass::layout::ColumnMajor, cutlass::layout::RowMajor>;
using Tf32TN = Tf32Gemm<cutlass::layout::RowMajor, cutlass::layout::ColumnMajor>;
using Tf32NN = Tf32Gemm<cutlass::layout::RowMajor, cutlass::layout::RowMajor>;
using Tf32TT = Tf32Gemm<cutlass::layout::ColumnMajor, cutlass::layout::RowMajor>;
template <class Cfg>
struct PairOf;
template <class LayoutA, class LayoutB>
struct PairOf<Tf32Gemm<LayoutA, LayoutB, false>> {
    using type = Tf32Gemm<LayoutA, LayoutB, true>;
};

bool tc_gemm_available() { return true; }

// Nearest value with a 10-bit mantissa (what a TF32 operand keeps; the MMA itself would truncate).
__device__ __forceinline__ float round_tf32(float x) {
    return __uint_as_float((__float_as_uint(x) + 0x00001000u) & 0xFFFFE000u);
}

// hi = x rounded to TF32 (|x - hi| <= 2^-11 |x|), lo = x - hi (exact in fp32) rounded to TF32 (error <= 2^-22 |x|).
// The two parts of a [rows x cols] matrix are written into a [rows x parts * cols] matrix, part p at columns
// [p * cols, (p + 1) * cols); `pattern` says which part goes where (bit p set: lo, clear: hi).  Concatenating along
// the contraction index turns hi.hi + hi.lo + lo.hi into ONE GEMM with three times the depth (A parts hi|hi|lo, B
// parts hi|lo|hi); concatenating B along its free index turns A.hi + A.lo into one GEMM with twice the width.
__global__ void split_tf32_kernel(const float *__restrict__ x, int64_t rows, int64_t cols, int64_t ld, float *__restrict__ out,
                                  int parts, unsigned pattern) {
    const int64_t n4 = rows * (cols / 4);
    const int64_t ldo = (int64_t)parts * cols;
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n4; i += (int64_t)gridDim.x * blockDim.x) {
        const int64_t r = i / (cols / 4), c = (i - r * (cols / 4)) * 4;
        const float4 v = *reinterpret_cast<const float4 *>(x + r * ld + c);
        float4 h, l;
        h.x = round_tf32(v.x); l.x = round_tf32(v.x - h.x);
        h.y = round_tf32(v.y); l.y = round_tf32(v.y - h.y);
        h.z = round_tf32(v.z); l.z = round_tf32(v.z - h.z);
        h.w = round_tf32(v.w); l.w = round_tf32(v.w - h.w);
        for (int p = 0; p < parts; p++)
            *reinterpret_cast<float4 *>(out + r * ldo + p * cols + c) = ((pattern >> p) & 1u) ? l : h;
    }
}

static int split(const float *x, int64_t rows, int64_t cols, int64_t ld, float *out, int parts, unsigned pattern,
                 cudaStream_t stream) {
    const int64_t n4 = rows * (cols / 4);
    int64_t blocks = (n4 + 255) / 256;
    const int64_t cap = (int64_t)device_info().sm_count * 16;
    if (blocks > cap) blocks = cap;
    split_tf32_kernel<<<(unsigned)blocks, 256, 0, stream>>>(x, rows, cols, ld, out, parts, pattern);
    LUTB_LAUNCH_CHECK();
    return LUTB_OK;
}

static size_t align256(size_t v) { return (v + 255) & ~(size_t)255; }

// A pair of SMs per 256 x 256 tile or one SM per 128 x 128 tile: whichever takes less time by waves of tiles.  A wave is what
// the SMs hold at once; a pair's tile is four times the work on twice the SMs and takes 1.6 times as long (a byte from shared
// memory feeds twice the multiply-adds).  Padding counts: a half empty 256-row tile takes as long as a full one.  Measured on the
// shapes of one deep GEMM with its operand copies, one SM / pair, us:
// pair: 8192 x 16384 x 768 318 / 258, 1024 x 65536 x 3072 592 / 488, 512 x 16384 x 768 50 / 46
// one SM: 128 x 16384 x 768 34 / 39, 384 x 16384 x 768 45 / 48
// even: 160 to 256 x 16384 x 768 38 / 38, 640 x 16384 x 768 55 / 55; 1024 x 4096 x 768 takes the pair at 30 / 33
static bool pair_tiles(int M, int N) {
    const int64_t sm = device_info().sm_count > 1 ? device_info().sm_count : 2;
    const int64_t pairs = (int64_t)((M + 255) / 256) * ((N + 255) / 256), singles = (int64_t)((M + 127) / 128) * ((N + 127) / 128);
    const int64_t pair_waves = (pairs + sm / 2 - 1) / (sm / 2), single_waves = (singles + sm - 1) / sm;
    return 8 * pair_waves < 5 * single_waves;
}
template <class Cfg>
static int run_tiles(int M, int N, int K, const float *A, int64_t lda, const float *B, int64_t ldb, float *C, int64_t ldc,
                     float alpha, float beta, void *workspace, size_t workspace_bytes, cudaStream_t stream) {
    if (pair_tiles(M, N))
        return run<typename PairOf<Cfg>::type>(M, N, K, A, lda, B, ldb, C, ldc, alpha, beta, workspace, workspace_bytes, stream);
    return run<Cfg>(M, N, K, A, lda, B, ldb, C, ldc, alpha, beta, workspace, workspace_bytes, stream);
}
template <class Cfg>
static size_t workspace_of_tiles(int M, int N, int K) {
    const size_t a = workspace_of<Cfg>(M, N, K), b = workspace_of<typename PairOf<Cfg>::type>(M, N, K);
    return a > b ? a : b;
}

// Plan of one call.  TN (both operands contraction-major): one GEMM of depth 3K on concatenated copies.  Anything else: three
// GEMMs on separate hi / lo copies.
struct SplitPlan {
    bool deep;
    size_t gemm_ws, a_bytes, b_bytes;
};

static SplitPlan split_plan(TcGemmKind kind, int M, int N, int K) {
    SplitPlan p{};
    p.deep = kind == TC_A_ROWS_B_ROWS_OF_N;
    if (p.deep) {
        p.gemm_ws = align256(workspace_of_tiles<Tf32TN>(M, N, 3 * K));
        p.a_bytes = align256((size_t)M * 3 * K * 4);
        p.b_bytes = align256((size_t)N * 3 * K * 4);
    } else {
        const size_t w2 = workspace_of<Tf32NN>(M, N, K), w3 = workspace_of<Tf32TT>(M, N, K);
        p.gemm_ws = align256(w2 > w3 ? w2 : w3);
        p.a_bytes = align256((size_t)M * K * 4 * 2);
        p.b_bytes = align256((size_t)N * K * 4 * 2);
    }
    return p;
}

size_t tc_gemm_workspace(TcGemmKind kind, int M, int N, int K) {
    const SplitPlan p = split_plan(kind, M, N, K);
    return p.gemm_ws + p.a_bytes + p.b_bytes + 512;
}

template <class Cfg>
static int run3(int M, int N, int K, const float *Ah, const float *Al, int64_t lda, const float *Bh, const float *Bl, int64_t ldb,
                float *C, int64_t ldc, float alpha, float beta, void *ws, size_t ws_bytes, cudaStream_t stream) {
    // small terms first, so that they are added to each other before they meet the large one
    int rc = run<Cfg>(M, N, K, Ah, lda, Bl, ldb, C, ldc, alpha, beta, ws, ws_bytes, stream);
    if (rc) return rc;
    rc = run<Cfg>(M, N, K, Al, lda, Bh, ldb, C, ldc, alpha, 1.f, ws, ws_bytes, stream);
    if (rc) return rc;
    return run<Cfg>(M, N, K, Ah, lda, Bh, ldb, C, ldc, alpha, 1.f, ws, ws_bytes, stream);
}

int tc_gemm(TcGemmKind kind, int M, int N, int K, const float *A, int64_t lda, const float *B, int64_t ldb, float *C,
            int64_t ldc, float alpha, float beta, void *workspace, size_t workspace_bytes, cudaStream_t stream) {
    const size_t need = tc_gemm_workspace(kind, M, N, K);
    LUTB_REQUIRE(workspace_bytes >= need, LUTB_ERR_WORKSPACE, "tensor-core contraction needs %zu bytes of workspace", need);
    // stored extents of the operands: A is [ar x ac], B is [br x bc] (row-major, contiguous in the second)
    const int64_t ar = kind == TC_A_COLS_B_ROWS_OF_K ? K : M, ac = kind == TC_A_COLS_B_ROWS_OF_K ? M : K;
    const int64_t br = kind == TC_A_ROWS_B_ROWS_OF_N ? N : K, bc = kind == TC_A_ROWS_B_ROWS_OF_N ? K : N;
    LUTB_REQUIRE(ac % 4 == 0 && bc % 4 == 0, LUTB_ERR_ALIGN, "tensor-core contraction: row lengths must be multiples of 4");
    const SplitPlan plan = split_plan(kind, M, N, K);
    unsigned char *p = reinterpret_cast<unsigned char *>((reinterpret_cast<uintptr_t>(workspace) + 255) & ~(uintptr_t)255);
    void *gw = p;
    p += plan.gemm_ws;
    float *Bs = reinterpret_cast<float *>(p);
    p += plan.b_bytes;
    float *As = reinterpret_cast<float *>(p);
    int rc;
    if (plan.deep) {
        // A' = [hi | lo | hi], B' = [lo | hi | hi] along the contraction index: one GEMM of depth 3K.  The mainloop
        // walks the contraction index upwards and the tensor core truncates its fp32 accumulator after every step, an
        // error proportional to the accumulator's size: the two small products go first, while it is small.
        rc = split(A, M, K, lda, As, 3, 0b010u, stream);
        if (rc) return rc;
        rc = split(B, N, K, ldb, Bs, 3, 0b001u, stream);
        if (rc) return rc;
        return run_tiles<Tf32TN>(M, N, 3 * K, As, 3 * (int64_t)K, Bs, 3 * (int64_t)K, C, ldc, alpha, beta, gw, plan.gemm_ws, stream);
    }
    // separate hi / lo copies (one matrix with two parts each)
    rc = split(B, br, bc, ldb, Bs, 2, 0b10u, stream);
    if (!rc) rc = split(A, ar, ac, lda, As, 2, 0b10u, stream);
    if (rc) return rc;
    const float *Al = As + ac, *Bl = Bs + bc;
    if (kind == TC_A_ROWS_B_ROWS_OF_K) return run3<Tf32NN>(M, N, K, As, Al, 2 * ac, Bs, Bl, 2 * bc, C, ldc, alpha, beta, gw, plan.gemm_ws, stream);
    return run3<Tf32TT>(M, N, K, As, Al, 2 * ac, Bs, Bl, 2 * bc, C, ldc, alpha, beta, gw, plan.gemm_ws, stream);
}

size_t tc_gemm_fast_workspace(int M, int N, int K) {
    size_t w = workspace_of<FastTN>(M, N, K);
    const size_t w2 = workspace_of<FastNN>(M, N, K), w3 = workspace_of<FastTT>(M, N, K);
    w = w > w2 ? w : w2;
    return (w > w3 ? w : w3) + 256;
}

int tc_gemm_fast(TcGemmKind kind, int M, int N, int K, const float *A, int64_t lda, const float *B, int64_t ldb, float *C,
                 int64_t ldc, float alpha, float beta, void *workspace, size_t workspace_bytes, cudaStream_t stream) {
    switch (kind) {
        case TC_A_ROWS_B_ROWS_OF_N: return run<FastTN>(M, N, K, A, lda, B, ldb, C, ldc, alpha, beta, workspace, workspace_bytes, stream);
        case TC_A_ROWS_B_ROWS_OF_K: return run<FastNN>(M, N, K, A, lda, B, ldb, C, ldc, alpha, beta, workspace, workspace_bytes, stream);
        default: return run<FastTT>(M, N, K, A, lda, B, ldb, C, ldc, alpha, beta, workspace, workspace_bytes, stream);
    }
}

}  // namespace lutb
#endif  // LUTB_NO_CUTLASS

// C-ABI face, for callers that want an fp32-accurate tensor-core GEMM; nothing else in the library uses it.
extern "C" int lutb_fp32_gemm_available(void) { return lutb::tc_gemm_available() ? 1 : 0; }

extern "C" size_t lutb_fp32_gemm_workspace(int32_t m, int32_t n, int32_t k) {
    if (!(m > 0 && n > 0 && k > 0)) return 0;
    size_t a = 0;
    for (int kind = 0; kind < 3; kind++) {
        const size_t w = lutb::tc_gemm_workspace(static_cast<lutb::TcGemmKind>(kind), m, n, k);
        a = w > a ? w : a;
    }
    const size_t b = lutb::tc_gemm_fast_workspace(m, n, k);
    return a > b ? a : b;
}

extern "C" int lutb_fp32_gemm(int kind, int32_t m, int32_t n, int32_t k, const float *a, int64_t lda, const float *b,
                              int64_t ldb, float *c, int64_t ldc, float alpha, float beta, void *workspace,
                              size_t workspace_bytes, void *stream) {
    using namespace lutb;
    const bool fast = (kind & LUTB_GEMM_FAST_FP32) != 0;
    kind &= ~LUTB_GEMM_FAST_FP32;
    LUTB_REQUIRE(kind >= LUTB_GEMM_A_ROWS_B_ROWS_OF_N && kind <= LUTB_GEMM_A_COLS_B_ROWS_OF_K, LUTB_ERR_MODE, "unknown GEMM kind %d", kind);
    LUTB_REQUIRE(m > 0 && n > 0 && k > 0, LUTB_ERR_SHAPE, "empty GEMM");
    LUTB_REQUIRE(a && b && c, LUTB_ERR_NULL, "a matrix pointer is NULL");
    LUTB_REQUIRE(((reinterpret_cast<uintptr_t>(a) | reinterpret_cast<uintptr_t>(b) | reinterpret_cast<uintptr_t>(c)) & 15) == 0,
                 LUTB_ERR_ALIGN, "matrices must be 16-byte aligned");
    LUTB_REQUIRE(((lda | ldb | ldc) & 3) == 0, LUTB_ERR_ALIGN, "leading dimensions must be multiples of 4");
    KernelScope scope(K_FP32_GEMM, static_cast<cudaStream_t>(stream));
    if (fast)
        return tc_gemm_fast(static_cast<TcGemmKind>(kind), m, n, k, a, lda, b, ldb, c, ldc, alpha, beta, workspace,
                            workspace_bytes, static_cast<cudaStream_t>(stream));
    return tc_gemm(static_cast<TcGemmKind>(kind), m, n, k, a, lda, b, ldb, c, ldc, alpha, beta, workspace, workspace_bytes,
                   static_cast<cudaStream_t>(stream));
}

