// gl_mdft.cu — tensor-core matrix products for the matrix-DFT starburst.
//
// This unit holds the tcgen05 machinery shared by the MDFT forms: TMA tensor
// maps built on the host, a warp-specialised CTA (one TMA producer thread,
// one MMA-issuing thread, four epilogue warps reading TMEM) and the plain
// BF16 GEMM C = A * B^T that pins the descriptors against torch.
#include "gl_internal.h"
#include "gl_launch.cuh"
#include "gl_tc.cuh"

#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <vector>
#include <cstring>
#include <mutex>
#include <string>

namespace gl {

// ---- host: tensor maps --------------------------------------------------------
typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                  const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                  CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

static EncodeTiledFn encode_fn()
{
    static std::once_flag once;
    static EncodeTiledFn fn = nullptr;
    std::call_once(once, [] {
        void* p = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &p, 12000, cudaEnableDefault, &q) ==
                cudaSuccess &&
            q == cudaDriverEntryPointSuccess)
            fn = reinterpret_cast<EncodeTiledFn>(p);
    });
    return fn;
}

// 2-D row-major matrix of `rows` x `cols` elements (cols contiguous) with a
// box of box_rows x box_cols, 128-byte swizzle (box_cols * elem = 128 B).
int make_tmap_2d(CUtensorMap* map, const void* base, CUtensorMapDataType dtype, int elem_bytes, uint64_t rows,
                 uint64_t cols, uint32_t box_rows, uint32_t box_cols)
{
    EncodeTiledFn fn = encode_fn();
    if (!fn) return fail(GL_ERR_CUDA, "cuTensorMapEncodeTiled is not available from the driver");
    if (((uintptr_t)base & 15) != 0) return fail(GL_ERR_INVALID, "tensor base must be 16-byte aligned");
    if ((cols * elem_bytes) % 16 != 0) return fail(GL_ERR_INVALID, "tensor row pitch must be a multiple of 16 bytes");
    cuuint64_t gdim[2] = {cols, rows};
    cuuint64_t gstride[1] = {cols * (uint64_t)elem_bytes};
    cuuint32_t box[2] = {box_cols, box_rows};
    cuuint32_t estr[2] = {1, 1};
    CUresult r = fn(map, dtype, 2, const_cast<void*>(base), gdim, gstride, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                    CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) return fail(GL_ERR_INVALID, "cuTensorMapEncodeTiled failed (" + std::to_string((int)r) + ")");
    return GL_OK;
}

namespace {

constexpr int kBM = 128, kBN = 128, kBK = 64, kStages = 4;
constexpr int kTileBytes = kBM * kBK * 2;   // 16 KB per operand tile

__device__ __forceinline__ uint8_t* align1024(uint8_t* p)
{
    return reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(p) + 1023) & ~uintptr_t(1023));
}

// C[M x N] (fp32, row-major) = A[M x K] * B[N x K]^T, BF16 operands, FP32
// accumulation in TMEM.  One 128x128 tile per CTA; 128 threads.
__global__ void __launch_bounds__(128, 1) tc_gemm_bf16_kernel(const __grid_constant__ CUtensorMap ta,
                                                              const __grid_constant__ CUtensorMap tb, float* C,
                                                              int M, int N, int K, int* err)
{
    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = align1024(smem_raw);
    uint8_t* sa = smem;
    uint8_t* sb = smem + kStages * kTileBytes;
    __shared__ uint64_t full[kStages], empty[kStages], accbar;
    __shared__ uint32_t tmem_base;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int m0 = blockIdx.y * kBM, n0 = blockIdx.x * kBN;
    const int nk = K / kBK;

    if (warp == 0) tc::tmem_alloc(&tmem_base, 128);
    if (threadIdx.x == 32)
    {
        for (int s = 0; s < kStages; ++s) { tc::mbar_init(&full[s], 1); tc::mbar_init(&empty[s], 1); }
        tc::mbar_init(&accbar, 1);
        tc::fence_mbar_init();
        tc::tma_prefetch(&ta);
        tc::tma_prefetch(&tb);
    }
    tc::tc_fence_before();
    __syncthreads();
    tc::tc_fence_after();
    const uint32_t tmem = tmem_base;

    if (warp == 0 && lane == 0)
    {
        // TMA producer
        int issued = 0;
        for (int kb = 0; kb < nk; ++kb)
        {
            const int s = kb % kStages;
            if (kb >= kStages && !tc::mbar_wait(&empty[s], ((kb / kStages) - 1) & 1, err, tc::TC_TIMEOUT_EMPTY)) break;
            tc::mbar_expect_tx(&full[s], 2 * kTileBytes);
            tc::tma_load_2d(sa + s * kTileBytes, &ta, kb * kBK, m0, &full[s]);
            tc::tma_load_2d(sb + s * kTileBytes, &tb, kb * kBK, n0, &full[s]);
            ++issued;
        }
        // our own copies must have landed before the CTA can retire
        for (int kb = (issued > kStages ? issued - kStages : 0); kb < issued; ++kb)
            tc::mbar_wait(&full[kb % kStages], (kb / kStages) & 1, err, tc::TC_TIMEOUT_FULL);
    }
    else if (warp == 1 && lane == 0)
    {
        // MMA issuer
        const uint32_t idesc = tc::idesc_bf16(kBM, kBN, false);
        for (int kb = 0; kb < nk; ++kb)
        {
            const int s = kb % kStages;
            if (!tc::mbar_wait(&full[s], (kb / kStages) & 1, err, tc::TC_TIMEOUT_FULL)) break;
            tc::tc_fence_after();
            const uint64_t da = tc::sw128_desc(tc::smem_u32(sa + s * kTileBytes));
            const uint64_t db = tc::sw128_desc(tc::smem_u32(sb + s * kTileBytes));
            #pragma unroll
            for (int kk = 0; kk < kBK / 16; ++kk)
                tc::mma_f16(tmem, da + 2 * kk, db + 2 * kk, idesc, (kb | kk) != 0);
            tc::mma_commit(&empty[s]);
        }
        tc::mma_commit(&accbar);   // also on the error path: no MMA may outlive TMEM
    }
    __syncwarp();

    // Epilogue: TMEM lane = tile row; 8 chunks of 16 columns.
    const bool ok = tc::mbar_wait(&accbar, 0, err, tc::TC_TIMEOUT_ACC);
    tc::tc_fence_after();
    const int row = warp * 32 + lane;
    #pragma unroll 1
    for (int c = 0; c < kBN / 16; ++c)
    {
        float v[16];
        tc::tmem_ld16(tmem + ((uint32_t)(warp * 32) << 16) + (uint32_t)(c * 16), v);
        if (ok && m0 + row < M)
        {
            float* dst = C + (size_t)(m0 + row) * N + n0 + c * 16;
            #pragma unroll
            for (int i = 0; i < 16; i += 4) *reinterpret_cast<float4*>(dst + i) = make_float4(v[i], v[i + 1], v[i + 2], v[i + 3]);
        }
    }
    tc::tc_fence_before();
    __syncthreads();
    if (warp == 0) tc::tmem_dealloc(tmem, 128);
}

}  // namespace
}  // namespace gl

using namespace gl;

extern "C" int gl_gemm_bf16_tc(const void* d_a, const void* d_b, float* d_c, int M, int N, int K, void* stream)
{
    if (!d_a || !d_b || !d_c) return fail(GL_ERR_INVALID, "gemm_bf16_tc: null pointer");
    if (M <= 0 || N <= 0 || K <= 0 || M % 128 || N % 128 || K % 64)
        return fail(GL_ERR_INVALID, "gemm_bf16_tc: M and N must be multiples of 128, K of 64");
    CUtensorMap ta, tb;
    int rc = make_tmap_2d(&ta, d_a, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, (uint64_t)M, (uint64_t)K, 128, 64);
    if (rc) return rc;
    rc = make_tmap_2d(&tb, d_b, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, (uint64_t)N, (uint64_t)K, 128, 64);
    if (rc) return rc;
    cudaStream_t st = (cudaStream_t)stream;
    int* d_err = nullptr;
    GL_CUDA_TRY(cudaMallocAsync(&d_err, sizeof(int), st));
    GL_CUDA_TRY(cudaMemsetAsync(d_err, 0, sizeof(int), st));
    const size_t smem = 2 * kStages * kTileBytes + 1024;
    GL_CUDA_TRY(cudaFuncSetAttribute(tc_gemm_bf16_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    dim3 grid(N / 128, M / 128);
    tc_gemm_bf16_kernel<<<grid, 128, smem, st>>>(ta, tb, d_c, M, N, K, d_err);
    GL_CUDA_TRY(cudaGetLastError());
    int h_err = 0;
    GL_CUDA_TRY(cudaMemcpyAsync(&h_err, d_err, sizeof(int), cudaMemcpyDeviceToHost, st));
    GL_CUDA_TRY(cudaStreamSynchronize(st));
    cudaFreeAsync(d_err, st);
    g_last_launches = 1;
    if (h_err) return fail(GL_ERR_TIMEOUT, "gemm_bf16_tc: a pipeline wait timed out (code " + std::to_string(h_err) + ")");
    return GL_OK;
}

// ===========================================================================
// Matrix-DFT starburst, field form:  E_l = W_y(l) A W_x(l)^T,  I_l = |E_l|^2,
// out_c = sum_l w_c(l) I_l   (the field form of mdft_render.cu's
// per-wavelength triple product, evaluated on the tensor cores).
//
//   W_x[k][j] = exp(-2 pi i s_x(l) (j - c_j)(k - c_x)),  same for y.
//
// The operand A is real and the phase is odd in d = j - c_j, so the sums run
// over |d| only, on A's even and odd parts about the centre:
//   A_ee, A_oe, A_eo, A_oo   (first letter: row parity, second: column parity;
//                             even = A[+d] + A[-d], odd = A[+d] - A[-d])
// with C = cos, S = sin of the phase at d >= 0 (nh of them, half of n):
//   step 1   Te_r = C A_ee, To_r = C A_oe, Te_i = -S A_eo, To_i = -S A_oo
//   step 2   Re E = C_y Te_r + S_y To_i,   Im E = C_y Te_i - S_y To_r
// (Te / To the even and odd parts of T over the pupil rows).  Both steps take
// half the products of the unfolded form, the matrices half the memory, and
// Re E and Im E accumulate directly.  The pixel-integrated (box) form needs
// Re E only, Te_r and To_i; it is not folded in any storage (below).
//
// FORM 0 (split BF16): every operand X is stored as X_hi = bf16(X) and
// X_lo = bf16(X - X_hi), rows [hi | lo]; each 128-byte step of the reduction
// loads the four tiles once and accumulates A_hi B_hi + A_hi B_lo + A_lo B_hi.
// FORM 1 (TF32): FP32 operands, kind::tf32 MMAs, not folded: sums of two
// operand entries round differently in 11 bits, and this form's results are
// its roundings.  Step 1 makes [Tr | Ti] = [Wr | Wi] A, step 2 accumulates
// D1 = Wr [Tr | Ti], D2 = Wi [Tr | Ti] and combines them (Re E = D1[Tr] -
// D2[Ti], Im E = D1[Ti] + D2[Tr]); the box form makes D1[Tr] and D2[Ti] only.
// The pixel-integrated form in split BF16 is not folded either: its images are a
// small window of dim pixels around a peak, where the order of the additions
// shows.  Nor is the field form about another centre than the pupil's middle: the
// halves do not match there, so less is saved and the error grows (256^2 disc,
// centre at 0.4 of it: 2.1e-6 unfolded, 2.9e-6 folded; in the middle 2.1 and 1.3e-6).
// Both run like TF32, with the reduction in three passes (hi hi, hi lo, lo hi) over
// the same [hi | lo] rows.
// FORM 2 (FP32 on the CUDA cores) is folded in the field form; its
// pixel-integrated form makes the folded products over all signed distances, with
// the operand in both parts (Te_r = C A, To_i = -S A).  Accumulation is FP32 in TMEM (or
// registers) throughout.
//
// 512^2 pupil to 2048^2, 31 wavelengths, split BF16: step 1 233 -> 109 us, step
// 2 1093 -> 460 us (in pairs of CTAs; 91% of the measured dense BF16 rate).
//
// Storage (Kp = 2 nh bf16, or nh floats; rows of Kp; unfolded: nh = n):
//   W'  [lam][C | S][k]                                  TF32: [Wr | Wi]
//   A'  [ee | oe | eo | oo][row d]   FP32 box: A twice   (nhr rows each; TF32: A)
//   T'  [lam][k / 128][Te_r | Te_i | To_i | -To_r][k % 128]   FP32 box: [Te_r | To_i]
//                                              TF32, unfolded split BF16: [Tr | Ti]
// ===========================================================================
namespace gl {
namespace {

constexpr int kMdftThreads = 192;     // warps 0-3 epilogue, warp 4 TMA, warp 5 MMA
constexpr int kTf32 = 1;              // not folded
constexpr int kSplitWhole = 3;        // split BF16, not folded, three passes (a plan's form 0 with box, or off the middle)
__host__ __device__ constexpr bool is_bf16(int form) { return form == 0 || form == kSplitWhole; }
__host__ __device__ constexpr bool is_folded(int form) { return form == 0 || form == 2; }
constexpr int kOpTile = 128 * 128;    // bytes of one 128-row x 128-byte operand tile

struct MdftArgs {
    int KA;       // rows of the A operand per (wavelength, C / S part): Kx in step 1, Ky in step 2
    int NBm;      // 128-row blocks of the A operand (step 1: Kx / 128, step 2: Ky / 128)
    int nh, nhr;                      // folded reduction length (multiple of 16), rows per parity block of A'
    int nkb;                          // 128-byte steps of one folded reduction
    int NB, NI, n_units;              // T' blocks per wavelength (Kx / 128), step-1 tiles across nh
    void* tprime;                     // step 1 output / step 2 B operand
    float* out_r;
    float* out_g;
    float* out_b;
    const float4* weights;            // per wavelength (w_r, w_g, w_b, 0)
    int* err;
    // step-2 output placement: plan pixel (l, k) -> frame (y0 + l, x0 + k) of
    // planes out_w wide, kept when l < win_h and k < win_w
    int out_w, x0, y0, win_w, win_h;
    float* parts;                     // FP32 step 2 in several wavelength ranges: each wavelength's own Re E or |E|^2, Ky x Kx
    int vec;                          // 1: every row piece of a tile starts on a 16-byte boundary in all three planes
    float4 tint;                      // per-launch colour factor on the weights
    int lam_base;                     // first wavelength of this launch's range
    int NBt;                          // step 2: output tiles per row of the frame (Kx / tile width)
};

template <int FORM>
__device__ __forceinline__ void mma_any(uint32_t d, uint64_t a, uint64_t b, uint32_t idesc, uint32_t acc)
{
    if (is_bf16(FORM)) tc::mma_f16(d, a, b, idesc, acc);
    else tc::mma_tf32(d, a, b, idesc, acc);
}

template <int FORM>
__host__ __device__ constexpr uint32_t idesc_any(int M, int N)
{
    return is_bf16(FORM) ? tc::idesc_bf16(M, N, false) : tc::idesc_tf32(M, N, false);
}

__device__ __forceinline__ void store_split16(__nv_bfloat16* row, int nh, int i0, const float (&v)[16], float sign)
{
    // [hi | lo] at columns i0, nh + i0
    __align__(16) __nv_bfloat16 hi[16], lo[16];
    #pragma unroll
    for (int j = 0; j < 16; ++j)
    {
        const float x = sign * v[j];
        hi[j] = __float2bfloat16_rn(x);
        lo[j] = __float2bfloat16_rn(x - __bfloat162float(hi[j]));
    }
    const uint4* h4 = reinterpret_cast<const uint4*>(hi);
    const uint4* l4 = reinterpret_cast<const uint4*>(lo);
    uint4* d0 = reinterpret_cast<uint4*>(row + i0);
    uint4* d1 = reinterpret_cast<uint4*>(row + nh + i0);
    d0[0] = h4[0]; d0[1] = h4[1];
    d1[0] = l4[0]; d1[1] = l4[1];
}

// Shared-memory stages of one CTA and its accumulators.  A stage holds two A
// tiles of 128 rows (folded: hi and lo; TF32: Wr and Wi) and the row blocks of
// B (folded: hi and lo of each), as many stages as fit, four at most.
template <int FORM, int STEP, int TN, bool BOX, int CL>
struct MdftShape {
    static constexpr bool kFold = is_folded(FORM);
    static constexpr int kBSets = kFold ? 2 : 1;
    static_assert(!(kFold && BOX), "the pixel form is not folded on the tensor cores");
    static constexpr int kBlocks = kFold ? 2 : STEP;                // row blocks of B per unit and set
    static constexpr int kRows = STEP == 2 ? TN : 128;              // rows of one block
    static constexpr int kN = (STEP == 2 && BOX) ? TN : kBlocks * kRows;   // MMA N
    static constexpr int kOwn = kBlocks / CL;                       // of them this CTA loads (a pair: one each)
    static constexpr int kBBytes = kOwn * kRows * 128;
    static constexpr int kStageBytes = 2 * kOpTile + kBSets * kBBytes;
    static constexpr int kStages = 212992 / kStageBytes < 4 ? 212992 / kStageBytes : 4;
    static constexpr int kAccCols = kFold ? kN : 2 * kN;            // TMEM columns of a unit (TF32: D1 and D2)
    static constexpr int kAccBufs = kAccCols <= 256 ? 2 : 1;
    static constexpr int kParts = (kFold && STEP == 1) ? 2 : 1;     // units per tile: C and S apart
    // reductions per unit: C and S, step by step in turn (the two cancel far
    // from the centre: one after the other the sum would grow in between)
    static constexpr int kPhases = (kFold && STEP == 2) ? 2 : 1;
    // step 2's epilogue turns 32 x 32 blocks of the tile per warp
    static constexpr int kTurn = STEP == 2 ? 4 * 32 * 33 * 4 : 0;
    static constexpr int kSmem = kStages * kStageBytes + kTurn + 1024;
};

// TN (step 2): complex output columns per unit, 128 or 64 (the autotuner's
// tile-shape knob); twice the units spread a small frame over more SMs.
// CL = 2 (split BF16, field form): a pair of CTAs takes two neighbouring row blocks
// of one column block as one product of 256 rows (cta_group::2): each loads its
// own rows of A and one of the two row blocks of B, the first one issues, and each
// finds its 128 rows in its own TMEM.  Half of B per CTA is 64 KB a stage instead
// of 96, so three stages fit, and half the shared-memory reads for B, which with
// one CTA are the bound (36 KB of operands and 24 KB of fill per 384 cycles of MMA,
// at 128 bytes a cycle).  512^2 -> 2048^2 x 31: step 2 550 -> 460 us.  (Two CTAs that
// only shared B's tiles by multicast: 540.)
template <int FORM, int STEP, int TN, bool BOX, int CL>
__global__ void __launch_bounds__(kMdftThreads, 1) mdft_kernel(const __grid_constant__ CUtensorMap tA,
                                                              const __grid_constant__ CUtensorMap tB, MdftArgs args)
{
    static_assert(TN == 128 || TN == 64, "tile width");
    static_assert(CL == 1 || (CL == 2 && FORM == 0 && !BOX && TN == 128), "pairs");
    const int rank = CL == 2 ? (int)(blockIdx.x & 1) : 0;
    using Sh = MdftShape<FORM, STEP, TN, BOX, CL>;
    constexpr int kStagesM = Sh::kStages;
    constexpr int kbe = is_bf16(FORM) ? 64 : 32;                   // reduction elements per 128-byte row
    constexpr int kStep = is_bf16(FORM) ? 16 : 8;                  // and per MMA
    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = align1024(smem_raw);
    __shared__ uint64_t full[kStagesM], empty[kStagesM], acc_full[2], acc_empty[2], mma_done;
    __shared__ uint32_t tmem_base;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    int* err = args.err;

    if (warp == 5)
    {
        if (CL == 2) tc::tmem_alloc_pair(&tmem_base, 512);
        else tc::tmem_alloc(&tmem_base, 512);
    }
    if (threadIdx.x == 128)
    {
        // a pair's full and acc_empty are the first CTA's; empty and acc_full are
        // signalled in both
        for (int s = 0; s < kStagesM; ++s) { tc::mbar_init(&full[s], 1); tc::mbar_init(&empty[s], 1); }
        for (int b = 0; b < 2; ++b) { tc::mbar_init(&acc_full[b], 1); tc::mbar_init(&acc_empty[b], 128 * CL); }
        tc::mbar_init(&mma_done, 1);
        tc::fence_mbar_init();
        tc::tma_prefetch(&tA);
        tc::tma_prefetch(&tB);
    }
    tc::tc_fence_before();
    __syncthreads();
    tc::tc_fence_after();
    const uint32_t tmem = tmem_base;
    if (CL == 2) tc::cluster_sync();           // the other's barriers are set up

    // Units are dealt round-robin (unit u to CTA u mod G), so the units in
    // flight at any moment are consecutive: with wavelength-major unit order
    // they share one wavelength's operands, which then stay in L2.
    const int G = gridDim.x / CL;
    const int u0 = blockIdx.x / CL, u1 = args.n_units / CL;       // CL = 2: pairs of units

    auto decode = [&](int u, int& lam, int& mb, int& xb, int& part) {
        part = 0;
        if (STEP == 2)
        {
            // wavelength-major: all output tiles of one wavelength, then the next
            const int tiles = args.NBm / CL * args.NBt;
            const int lr = u / tiles;               // wavelength within this launch's range
            lam = args.lam_base + lr;
            const int tile = u - lr * tiles;
            mb = tile / args.NBt * CL + rank;
            xb = tile % args.NBt;
        }
        else
        {
            const int per = args.NBm / CL * args.NI * Sh::kParts;
            lam = args.lam_base + u / per;
            const int r = u % per;
            part = r % Sh::kParts;                  // C, then S
            mb = (r / Sh::kParts) / args.NI * CL + rank;
            xb = (r / Sh::kParts) % args.NI;
        }
    };

    if (warp == 4)
    {
        if (lane == 0)
        {
            int it = 0, issued = 0;
            bool stop = false;
            for (int u = u0; u < u1 && !stop; u += G)
            {
                int lam, mb, xb, part;
                decode(u, lam, mb, xb, part);
                {
                    for (int kk0 = 0; kk0 < Sh::kPhases * args.nkb; ++kk0, ++it)
                    {
                        const int kb = kk0 / Sh::kPhases, cs = STEP == 2 ? kk0 % Sh::kPhases : part;
                        const int rowA = (lam * 2 + cs) * args.KA + mb * 128;
                        const int s = it % kStagesM, r = it / kStagesM;
                        if (it >= kStagesM && !tc::mbar_wait(&empty[s], (r - 1) & 1, err, tc::TC_TIMEOUT_EMPTY)) { stop = true; break; }
                        uint8_t* st = smem + s * Sh::kStageBytes;
                        if (rank == 0) tc::mbar_expect_tx(&full[s], CL * Sh::kStageBytes);
                        // three passes: hi hi, hi lo, lo hi
                        const int pass = FORM == kSplitWhole ? kb / (args.nkb / 3) : 0;
                        const int x = (FORM == kSplitWhole ? kb % (args.nkb / 3) : kb) * kbe + (pass == 2 ? args.nh : 0);
                        const int xB = FORM == kSplitWhole ? (kb % (args.nkb / 3)) * kbe + (pass == 1 ? args.nh : 0) : x;
                        const uint32_t bar = CL == 2 ? tc::leader_u32(&full[s]) : 0u;
                        auto load = [&](uint8_t* dst, const CUtensorMap* map, int c0, int c1) {
                            if (CL == 2) tc::tma_load_2d_pair(dst, map, c0, c1, bar);
                            else tc::tma_load_2d(dst, map, c0, c1, &full[s]);
                        };
                        load(st, &tA, x, rowA);
                        if (Sh::kFold) load(st + kOpTile, &tA, args.nh + x, rowA);
                        else load(st + kOpTile, &tA, x, rowA + args.KA);
                        #pragma unroll
                        for (int t = 0; t < Sh::kBSets; ++t)
                            #pragma unroll
                            for (int j = 0; j < Sh::kOwn; ++j)
                            {
                                const int q = cs * Sh::kBlocks + j + rank;
                                int rowB;
                                if (STEP == 2)
                                {
                                    // T' holds each part in blocks of 128 columns; a
                                    // 64-column tile takes one half of each
                                    const int xb128 = (TN == 128) ? xb : (xb >> 1);
                                    const int half = (TN == 128) ? 0 : (xb & 1) * 64;
                                    rowB = ((lam * args.NB + xb128) * (Sh::kPhases * Sh::kBlocks) + q) * 128 + half;
                                }
                                else
                                    rowB = q * args.nhr + xb * 128;
                                load(st + 2 * kOpTile + t * Sh::kBBytes + j * Sh::kRows * 128, &tB, t * args.nh + xB, rowB);
                            }
                        ++issued;
                    }
                }
            }
            // this thread's copies have landed (a pair: have been used, which both CTAs are told)
            for (int q = (issued > kStagesM ? issued - kStagesM : 0); q < issued; ++q)
                tc::mbar_wait(CL == 2 ? &empty[q % kStagesM] : &full[q % kStagesM], (q / kStagesM) & 1, err,
                              CL == 2 ? tc::TC_TIMEOUT_EMPTY : tc::TC_TIMEOUT_FULL);
        }
        __syncwarp();
    }
    else if (warp == 5)
    {
        if (lane == 0 && rank == 0)
        {
            const uint32_t id = idesc_any<FORM>(128 * CL, Sh::kN);
            auto mma = [&](uint32_t d, uint64_t a, uint64_t b, uint32_t acc) {
                if (CL == 2) tc::mma_f16_pair(d, a, b, id, acc);
                else mma_any<FORM>(d, a, b, id, acc);
            };
            auto commit = [&](uint64_t* bar) {
                if (CL == 2) tc::mma_commit_pair(bar);
                else tc::mma_commit(bar);
            };
            int it = 0, ui = 0;
            bool stop = false;
            for (int u = u0; u < u1 && !stop; u += G, ++ui)
            {
                const int b = ui % Sh::kAccBufs, ur = ui / Sh::kAccBufs;
                if (ui >= Sh::kAccBufs && !tc::mbar_wait(&acc_empty[b], (ur - 1) & 1, err, tc::TC_TIMEOUT_ACC_FREE)) break;
                tc::tc_fence_after();
                const uint32_t d = tmem + (uint32_t)(b * 256);
                for (int kk0 = 0; kk0 < Sh::kPhases * args.nkb; ++kk0, ++it)
                {
                    const int kb = kk0 / Sh::kPhases;
                    const int s = it % kStagesM, r = it / kStagesM;
                    if (!tc::mbar_wait(&full[s], r & 1, err, tc::TC_TIMEOUT_FULL)) { stop = true; break; }
                    tc::tc_fence_after();
                    uint8_t* st = smem + s * Sh::kStageBytes;
                    const uint64_t a0 = tc::sw128_desc(tc::smem_u32(st));
                    const uint64_t a1 = tc::sw128_desc(tc::smem_u32(st + kOpTile));
                    const uint64_t b0 = tc::sw128_desc(tc::smem_u32(st + 2 * kOpTile));
                    // folded: the lo set; TF32 box: the Ti block
                    const uint64_t b1 = tc::sw128_desc(tc::smem_u32(st + 2 * kOpTile + (Sh::kFold ? Sh::kBBytes : Sh::kRows * 128)));
                    // the last step of a reduction may be partly past nh (whatever lies there is not multiplied)
                    const int left = FORM == kSplitWhole ? 4 : (args.nh - kb * kbe) / kStep;
                    #pragma unroll
                    for (int kk = 0; kk < 4; ++kk)
                    {
                        if (kk >= left) break;
                        const uint32_t acc = (kk0 | kk) != 0;
                        mma(d, a0 + 2 * kk, b0 + 2 * kk, acc);
                        if (Sh::kFold)
                        {
                            mma(d, a0 + 2 * kk, b1 + 2 * kk, 1);
                            mma(d, a1 + 2 * kk, b0 + 2 * kk, 1);
                        }
                        else
                            mma(d + Sh::kN, a1 + 2 * kk, (STEP == 2 && BOX ? b1 : b0) + 2 * kk, acc);
                    }
                    commit(&empty[s]);
                }
                commit(&acc_full[b]);
            }
            // every MMA this thread issued must be complete before TMEM is freed
            commit(&mma_done);
            tc::mbar_wait(&mma_done, 0, err, tc::TC_TIMEOUT_ACC);
        }
        __syncwarp();
    }
    else
    {
        // Epilogue warps 0-3: TMEM lane = tile row.
        int ui = 0;
        const int row = warp * 32 + lane;
        for (int u = u0; u < u1; u += G, ++ui)
        {
            int lam, mb, xb, part;
            decode(u, lam, mb, xb, part);
            const int b = ui % Sh::kAccBufs, ur = ui / Sh::kAccBufs;
            const bool ok = tc::mbar_wait(&acc_full[b], ur & 1, err, tc::TC_TIMEOUT_ACC);
            tc::tc_fence_after();
            const uint32_t ta = tmem + ((uint32_t)(warp * 32) << 16) + (uint32_t)(b * 256);
            if (STEP == 2)
            {
                const float4 w0 = args.weights[lam];
                const float4 w = make_float4(w0.x * args.tint.x, w0.y * args.tint.y, w0.z * args.tint.z, 0.0f);
                // A TMEM lane is a row of the tile, so a thread holds 32 columns
                // of one row; turned through shared memory, a warp adds whole
                // 128-byte row pieces to the planes: 16-byte vector atomics
                // where every row starts on a 16-byte boundary, else scalar
                // ones.  Adding each thread's own row left the warp's 32 rows
                // in 32 sectors per instruction and bound the kernel: 512^2 ->
                // 2048^2 x 31 650 -> 550 us, a 389 x 301 window 118 -> 42 us.
                float* turn = reinterpret_cast<float*>(smem + kStagesM * Sh::kStageBytes) + warp * (32 * 33);
                const int lrow = mb * 128 + warp * 32;
                const size_t o0 = (size_t)(args.y0 + lrow) * (size_t)args.out_w + (size_t)args.x0 + (size_t)xb * TN;
                const int rows = min(32, args.win_h - lrow);
                #pragma unroll 1
                for (int c = 0; c < TN / 32; ++c)
                {
                    #pragma unroll
                    for (int h = 0; h < 2; ++h)
                    {
                        float re[16], im[16];
                        const uint32_t tc0 = ta + (uint32_t)(c * 32 + h * 16);
                        tc::tmem_ld16(tc0, re);
                        if (!BOX) tc::tmem_ld16(tc0 + TN, im);
                        if (!Sh::kFold)
                        {
                            // Re E = D1[Tr] - D2[Ti], Im E = D1[Ti] + D2[Tr]
                            float u[16];
                            tc::tmem_ld16(tc0 + (BOX ? TN : 3 * TN), u);
                            #pragma unroll
                            for (int j = 0; j < 16; ++j) re[j] -= u[j];
                            if (!BOX)
                            {
                                tc::tmem_ld16(tc0 + 2 * TN, u);
                                #pragma unroll
                                for (int j = 0; j < 16; ++j) im[j] += u[j];
                            }
                        }
                        #pragma unroll
                        for (int j = 0; j < 16; ++j)
                            turn[lane * 33 + h * 16 + j] = BOX ? re[j] : re[j] * re[j] + im[j] * im[j];
                    }
                    __syncwarp();
                    const int kc = xb * TN + c * 32;
                    if (ok && args.vec)
                    {
                        const int col = (lane & 7) * 4;
                        for (int r = lane >> 3; r < rows; r += 4)
                        {
                            const float* t = turn + r * 33 + col;
                            const size_t o = o0 + (size_t)r * args.out_w + c * 32 + col;
                            if (kc + col + 3 < args.win_w)
                            {
                                atomicAdd(reinterpret_cast<float4*>(args.out_r + o), make_float4(w.x * t[0], w.x * t[1], w.x * t[2], w.x * t[3]));
                                atomicAdd(reinterpret_cast<float4*>(args.out_g + o), make_float4(w.y * t[0], w.y * t[1], w.y * t[2], w.y * t[3]));
                                atomicAdd(reinterpret_cast<float4*>(args.out_b + o), make_float4(w.z * t[0], w.z * t[1], w.z * t[2], w.z * t[3]));
                            }
                            else
                            {
                                #pragma unroll
                                for (int q = 0; q < 4; ++q)
                                {
                                    if (kc + col + q >= args.win_w) break;
                                    atomicAdd(args.out_r + o + q, w.x * t[q]);
                                    atomicAdd(args.out_g + o + q, w.y * t[q]);
                                    atomicAdd(args.out_b + o + q, w.z * t[q]);
                                }
                            }
                        }
                    }
                    else if (ok && kc + lane < args.win_w)
                    {
                        for (int r = 0; r < rows; ++r)
                        {
                            const float v = turn[r * 33 + lane];
                            const size_t o = o0 + (size_t)r * args.out_w + c * 32 + lane;
                            atomicAdd(args.out_r + o, w.x * v);
                            atomicAdd(args.out_g + o, w.y * v);
                            atomicAdd(args.out_b + o, w.z * v);
                        }
                    }
                    __syncwarp();
                }
            }
            else
            {
                // T' rows of this k.  The C part gives (Te_r, To_r), the S part
                // (-Te_i, -To_i); step 2 wants [Te_r | Te_i | To_i | -To_r].  TF32:
                // (Tr, Ti) as they are.
                const size_t blk = (size_t)(lam * args.NB + mb) * (Sh::kParts * 2) * 128;
                #pragma unroll
                for (int j = 0; j < 2; ++j)
                {
                    const int dst = !Sh::kFold ? j : (part == 0 ? (j == 0 ? 0 : 3) : (j == 0 ? 1 : 2));
                    const float sign = (!Sh::kFold || (part == 0 && j == 0)) ? 1.0f : -1.0f;
                    #pragma unroll 1
                    for (int c = 0; c < 8; ++c)
                    {
                        float v[16];
                        tc::tmem_ld16(ta + (uint32_t)(j * 128 + c * 16), v);
                        const int i0 = xb * 128 + c * 16;
                        if (!ok || i0 >= args.nh) continue;
                        if (is_bf16(FORM))
                        {
                            __nv_bfloat16* T = static_cast<__nv_bfloat16*>(args.tprime);
                            store_split16(T + (blk + dst * 128 + row) * (size_t)(2 * args.nh), args.nh, i0, v, sign);
                        }
                        else
                        {
                            float* r0 = static_cast<float*>(args.tprime) + (blk + dst * 128 + row) * (size_t)args.nh + i0;
                            #pragma unroll
                            for (int q = 0; q < 16; q += 4)
                                *reinterpret_cast<float4*>(r0 + q) = make_float4(sign * v[q], sign * v[q + 1], sign * v[q + 2], sign * v[q + 3]);
                        }
                    }
                }
            }
            tc::tc_fence_before();
            if (CL == 2) tc::mbar_arrive_cluster(tc::leader_u32(&acc_empty[b]));
            else tc::mbar_arrive(&acc_empty[b]);
        }
        // the arrival that the first CTA's last commit makes here too
        if (CL == 2 && rank == 1 && threadIdx.x == 0) tc::mbar_wait(&mma_done, 0, err, tc::TC_TIMEOUT_ACC);
        __syncwarp();
    }
    tc::tc_fence_before();
    __syncthreads();
    // a pair's MMAs read and write both CTAs, and arrive in both: neither leaves
    // before the other is done (every wait above ends, so both get here)
    if (CL == 2) tc::cluster_sync();
    if (warp == 5)
    {
        if (CL == 2) tc::tmem_dealloc_pair(tmem, 512);
        else tc::tmem_dealloc(tmem, 512);
    }
}

// DFT matrices W'[lam][C | S][k][Kp]: cos and sin of 2 pi s(lam) d (k - ck) at
// the folded distances d = m (centre cj whole) or m + 1/2, zero from nf on
// (TF32: cos and -sin at every d = m - cj).
// The phase is formed in FP32 double-float arithmetic (Dekker /
// Ogita-Rump-Oishi error-free products with FMA): s = s_hi + s_lo and
// ck = ck_hi + ck_lo are split on the host, d is exact, b = k - ck is carried
// as a two-float sum, and the product's integer cycles are removed from the
// leading term exactly; the reduced phase is accurate to ~1e-9 cycles, then
// evaluated with sincospif.  (The FP64 units of this part are slow.)
// With box set each entry also carries the pixel-box factor sinc(s d) of the
// reference's pixel-integrated form (mdft_render.cu:109-135).
// The factor depends on (wavelength, d) alone: a plan's table, made once.  A
// thread makes two neighbouring entries of a row, so the stores are whole words
// and no index is divided in the inner loop.  Bound by the instructions of the
// phase and sincospif.  W_x' and W_y' of a 640^2 operand, 512 x 384 outputs, 31
// wavelengths: 141 us in the unfolded layout (with the factor made per entry),
// 33 us now.
struct DftRows {
    void* out;
    const float2* scale;
    const float* amp;                  // [lam][nh]
    float ck_hi, ck_lo;
    int K;
};

// amp[lam][m]: 1 (box: sinc(s d)) up to nf, 0 past it
__global__ void mdft_amp_kernel(float* __restrict__ amp, const float2* __restrict__ scale, int nh, int nf, float d0,
                                int box)
{
    const int lam = blockIdx.x;
    const float2 sc = scale[lam];
    for (int m = threadIdx.x; m < nh; m += blockDim.x)
    {
        float v = m < nf ? 1.0f : 0.0f;
        if (box && m < nf)
        {
            // pixel-box factor of the pixel-integrated form: d the lag, s =
            // pixel pitch / pattern period at this wavelength
            const float x = ((float)m + d0) * (sc.x + sc.y);
            v = fabsf(x) < 1e-7f ? 1.0f : sinpif(x) / (3.14159265358979323846f * x);
        }
        amp[(size_t)lam * nh + m] = v;
    }
}

template <int FORM>
__global__ void __launch_bounds__(256) mdft_dft_kernel(DftRows R, int n_lambda, int nh, float d0)
{
    const int row = blockIdx.x * blockDim.y + threadIdx.y;
    if (row >= n_lambda * R.K) return;
    const int lam = row / R.K, k = row - lam * R.K;
    const float* amps = R.amp + (size_t)lam * nh;
    const float2 sc = R.scale[lam];                // (s_hi, s_lo)
    // b = k - ck as bh + bl: Knuth's two-sum of k and -ck_hi, then -ck_lo
    const float kf = (float)k;
    const float bh = kf - R.ck_hi;
    const float bb = bh - kf;
    const float bl = ((kf - (bh - bb)) + (-R.ck_hi - bb)) - R.ck_lo;
    const int Kp = is_bf16(FORM) ? 2 * nh : nh;
    const size_t rc = ((size_t)(lam * 2 + 0) * R.K + k) * Kp, rs = ((size_t)(lam * 2 + 1) * R.K + k) * Kp;
    for (int m = 2 * threadIdx.x; m < nh; m += 2 * blockDim.x)
    {
        float cv[2], sv[2];
        #pragma unroll
        for (int q = 0; q < 2; ++q)
        {
            const float a = (float)(m + q) + d0;   // exact
            const float p1 = a * bh;
            const float e1 = fmaf(a, bh, -p1);             // a*bh = p1 + e1 exactly
            const float m_lo = e1 + a * bl;
            const float qq = sc.x * p1;
            const float eq = fmaf(sc.x, p1, -qq);          // s_hi*p1 = qq + eq exactly
            const float rest = eq + sc.x * m_lo + sc.y * p1;
            float fr = (qq - rintf(qq)) + rest;            // qq - rint(qq) is exact
            fr -= rintf(fr);
            sincospif(2.0f * fr, &sv[q], &cv[q]);
            const float amp = amps[m + q];
            cv[q] *= amp;
            sv[q] = is_folded(FORM) ? amp * sv[q] : -amp * sv[q];
        }
        if (is_bf16(FORM))
        {
            __nv_bfloat16* W = static_cast<__nv_bfloat16*>(R.out);
            __nv_bfloat162 ch, cl, sh, sl;
            ch.x = __float2bfloat16_rn(cv[0]); ch.y = __float2bfloat16_rn(cv[1]);
            sh.x = __float2bfloat16_rn(sv[0]); sh.y = __float2bfloat16_rn(sv[1]);
            cl.x = __float2bfloat16_rn(cv[0] - __bfloat162float(ch.x)); cl.y = __float2bfloat16_rn(cv[1] - __bfloat162float(ch.y));
            sl.x = __float2bfloat16_rn(sv[0] - __bfloat162float(sh.x)); sl.y = __float2bfloat16_rn(sv[1] - __bfloat162float(sh.y));
            *reinterpret_cast<__nv_bfloat162*>(W + rc + m) = ch;
            *reinterpret_cast<__nv_bfloat162*>(W + rc + nh + m) = cl;
            *reinterpret_cast<__nv_bfloat162*>(W + rs + m) = sh;
            *reinterpret_cast<__nv_bfloat162*>(W + rs + nh + m) = sl;
        }
        else
        {
            float* W = static_cast<float*>(R.out);
            *reinterpret_cast<float2*>(W + rc + m) = make_float2(cv[0], cv[1]);
            *reinterpret_cast<float2*>(W + rs + m) = make_float2(sv[0], sv[1]);
        }
    }
}

// Pupil amplitude of the lens's stop (build_pupil_kernel,
// starburst_render.cu:155-191, stop term): grid coordinate g in [-1, 1) maps
// to pupil coordinate g / pupil_fill; 4 x 4 supersamples per texel tested
// against the stop silhouette (PupilMask::contains, aperture_sampler.h:63-82:
// ellipse of the stop's aspect, then the regular n-gon or the authored blade
// profile).
struct PupilDev {
    float aspect, rot_rad, apothem, sector;
    int n_blades;
    BladeProfile blade;
};

__device__ __forceinline__ bool pupil_in(const PupilDev& m, float u, float v)
{
    const float ux = u / m.aspect;
    const float r2 = ux * ux + v * v;
    if (r2 > 1.0f) return false;
    if (m.n_blades >= 3)
    {
        if (m.blade.deformed) return sqrtf(r2) <= blade_radius_at(m.blade, atan2f(v, ux));
        const float angle = atan2f(v, ux) - m.rot_rad;
        float sector = fmodf(angle, m.sector);
        if (sector < 0.0f) sector += m.sector;
        if (sqrtf(r2) * cosf(sector - m.sector * 0.5f) > m.apothem) return false;
    }
    return true;
}

// bilinear sample of the cat's-eye envelope (ME x ME over pupil [-1, 1]^2,
// cell centres, clamped at the edges): sample_env, starburst_render.cu:136-149
__device__ __forceinline__ float pupil_env(const float* __restrict__ env, int ME, float u, float v)
{
    float fx = (u * 0.5f + 0.5f) * ME - 0.5f;
    float fy = (v * 0.5f + 0.5f) * ME - 0.5f;
    fx = fminf(fmaxf(fx, 0.0f), (float)(ME - 1));
    fy = fminf(fmaxf(fy, 0.0f), (float)(ME - 1));
    const int x0 = (int)floorf(fx), y0 = (int)floorf(fy);
    const int x1 = min(x0 + 1, ME - 1), y1 = min(y0 + 1, ME - 1);
    const float tx = fx - x0, ty = fy - y0;
    const float a = env[(size_t)y0 * ME + x0] * (1.0f - tx) + env[(size_t)y0 * ME + x1] * tx;
    const float b = env[(size_t)y1 * ME + x0] * (1.0f - tx) + env[(size_t)y1 * ME + x1] * tx;
    return a * (1.0f - ty) + b * ty;
}

// env == nullptr: the plain stop (coverage of the 16 supersamples); else
// each inside supersample weighs the envelope at its own position
__global__ void pupil_build_kernel(float* __restrict__ out, int N, float fill, PupilDev m,
                                   const float* __restrict__ env, int ME)
{
    const int idx = blockIdx.x * blockDim.x + threadIdx.x;
    if (idx >= N * N) return;
    const int i = idx % N, j = idx / N;
    int cnt = 0;
    float acc = 0.0f;
    #pragma unroll
    for (int sy = 0; sy < 4; ++sy)
        #pragma unroll
        for (int sx = 0; sx < 4; ++sx)
        {
            const float u = (((float)i + ((float)sx + 0.5f) * 0.25f) / (float)N * 2.0f - 1.0f) / fill;
            const float v = (((float)j + ((float)sy + 0.5f) * 0.25f) / (float)N * 2.0f - 1.0f) / fill;
            if (!pupil_in(m, u, v)) continue;
            ++cnt;
            if (env) acc += pupil_env(env, ME, u, v);
        }
    out[idx] = (env ? acc : (float)cnt) * (1.0f / 16.0f);
}

// Operand A[i][j] (float, n x n) -> its even and odd parts about the centre,
// A'[part][row d][col d'], split BF16 [hi | lo] or FP32.  i1 / i2 are the
// indices at +d and -d (outside the operand: zero); d = 0 of a whole centre
// counts once in the even part.
template <int FORM>
__device__ __forceinline__ void mdft_fold_one(const float* __restrict__ a, void* out, int n, int nh, int nhr, int nf,
                                              int h2, int box, int x, int y)
{
    const int Kp = is_bf16(FORM) ? 2 * nh : nh;
    if (!is_folded(FORM))                            // nh = n
    {
        const float w = a[(size_t)y * n + x];
        if (!is_bf16(FORM))
        {
            static_cast<float*>(out)[(size_t)y * Kp + x] = w;
            return;
        }
        __nv_bfloat16* M = static_cast<__nv_bfloat16*>(out) + (size_t)y * Kp + x;
        const __nv_bfloat16 h = __float2bfloat16_rn(w);
        M[0] = h;
        M[nh] = __float2bfloat16_rn(w - __bfloat162float(h));
        return;
    }
    if (FORM == 2 && box)                            // all signed distances: both parts are the operand
    {
        const float w = a[(size_t)y * n + x];
        for (int k = 0; k < 2; ++k) static_cast<float*>(out)[((size_t)k * nhr + y) * Kp + x] = w;
        return;
    }
    const int base = (h2 + 1) >> 1;                  // index at the smallest distance
    auto at = [&](int r, int c) {
        return (r >= 0 && r < n && c >= 0 && c < n) ? a[(size_t)r * n + c] : 0.0f;
    };
    const int r1 = base + y, r2 = h2 - r1, c1 = base + x, c2 = h2 - c1;
    float v[4] = {0.0f, 0.0f, 0.0f, 0.0f};           // ee, oe, eo, oo
    if (x < nf && y < nf)
    {
        const float p = at(r1, c1), q = c1 == c2 ? 0.0f : at(r1, c2);
        const float s = r1 == r2 ? 0.0f : at(r2, c1), t = (r1 == r2 || c1 == c2) ? 0.0f : at(r2, c2);
        const bool ro = r1 != r2, co = c1 != c2;     // no odd part at distance 0
        v[0] = (p + q) + (s + t);
        v[1] = ro ? (p + q) - (s + t) : 0.0f;
        v[2] = co ? (p - q) + (s - t) : 0.0f;
        v[3] = ro && co ? (p - q) - (s - t) : 0.0f;
    }
    #pragma unroll
    for (int k = 0; k < 4; ++k)
    {
        const float w = v[k];
        const size_t o = ((size_t)k * nhr + y) * Kp + x;
        if (FORM == 0)
        {
            __nv_bfloat16* M = static_cast<__nv_bfloat16*>(out);
            const __nv_bfloat16 h = __float2bfloat16_rn(w);
            M[o] = h;
            M[o + nh] = __float2bfloat16_rn(w - __bfloat162float(h));
        }
        else
        {
            static_cast<float*>(out)[o] = w;
        }
    }
}

// The blocks past the nh rows zero the output planes and the error word, in
// place of four memset nodes.
template <int FORM>
__global__ void __launch_bounds__(128) mdft_fold_kernel(const float* __restrict__ a, void* out, int n, int nh, int nhr,
                                                        int nf, int h2, int box, float* z0, float* z1, float* z2,
                                                        size_t npx, int* err)
{
    const int y = blockIdx.x;
    if (y >= nh)
    {
        const size_t at = (size_t)(y - nh) * blockDim.x + threadIdx.x, all = (size_t)(gridDim.x - nh) * blockDim.x;
        if (at == 0) *err = 0;
        float* planes[3] = {z0, z1, z2};
        #pragma unroll
        for (int c = 0; c < 3; ++c)
        {
            const bool vec = (reinterpret_cast<uintptr_t>(planes[c]) & 15) == 0;
            const size_t quads = vec ? npx / 4 : 0;
            for (size_t i = at; i < quads; i += all)
                reinterpret_cast<float4*>(planes[c])[i] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
            for (size_t i = 4 * quads + at; i < npx; i += all) planes[c][i] = 0.0f;
        }
        return;
    }
    for (int x = threadIdx.x; x < nh; x += blockDim.x) mdft_fold_one<FORM>(a, out, n, nh, nhr, nf, h2, box, x, y);
}


// ---- FP32 CUDA-core form -------------------------------------------------------
// The same folded products in FP32 FMAs over the TF32 form's storage.  A CTA
// makes a tile of 16 P x 64 of every row block of a unit (step 1: one parity of T;
// step 2: Re E and Im E over both), 256 threads of P x 4 per block, reduction
// chunks of 16 staged in shared memory one chunk ahead, sums in two levels (32
// terms, then their sums): one long sum rounded the pattern's peak 0.3 to 1.7e-6 off
// 64 bits, two levels 0.1 to 0.3e-6.  In step 2 the wavelengths are split over CTAs
// (n_ranges); each wavelength's result then goes to a plane of its own and
// mdft_simt_sum adds them up in order, so that a call repeats bit for bit (the
// ranges' additions into the output planes would come in any order).
// Bound by shared-memory reads and the FP32 pipes: P = 4 32 FMA per three 16-byte
// loads (box: 16 per two), P = 8 64 per four (32 per three).  256^2 pupil to 512^2,
// 8 wavelengths: both steps 1.75 -> 0.08 ms (the unfolded form looped over the
// wavelengths in 16 CTAs of 128 x 128 tiles).
constexpr int kSB = 64, kSK = 16;

template <int STEP, bool BOX, int P>
__global__ void __launch_bounds__(256, P == 8 ? 1 : 2) mdft_simt_kernel(const float* __restrict__ W, const float* __restrict__ B,
                                                           MdftArgs args, int lam1, int n_ranges)
{
    after_previous();
    static_assert(P == 4 || (P == 8 && STEP == 2), "rows per thread");
    constexpr int NBLK = BOX ? 1 : 2;
    constexpr int kRows = 16 * P, kLoads = P / 4;              // rows of the tile, staging loads of them per thread
    __shared__ __align__(16) float sA[kSK][kRows + 4];
    __shared__ __align__(16) float sB[NBLK][kSK][kSB + 4];
    const int tid = threadIdx.x, tx = tid & 15, ty = tid >> 4;
    const int lr = tid >> 2, lc = (tid & 3) * 4;               // row and first column of this thread's staging loads
    const int nh = args.nh, xb = blockIdx.x, mb = blockIdx.y;  // tiles of kRows x 64
    int l0, l1, part = 0;
    if (STEP == 1)
    {
        l0 = args.lam_base + (int)(blockIdx.z >> 1);
        l1 = l0 + 1;
        part = blockIdx.z & 1;
    }
    else
    {
        const int total = lam1 - args.lam_base, per = (total + n_ranges - 1) / n_ranges;
        l0 = args.lam_base + (int)blockIdx.z * per;
        l1 = min(lam1, l0 + per);
    }
    for (int lam = l0; lam < l1; ++lam)
    {
        // two levels: a long sum of one sign (the pattern's peak) would round at every step
        float total[NBLK][P][4] = {}, acc[NBLK][P][4] = {};
        {
            // chunks of C and S in turn (step 2), like the tensor-core forms
            constexpr int kPh = STEP == 2 ? 2 : 1;
            const float* Ar = W + ((size_t)(lam * 2 + part) * args.KA + mb * kRows + lr) * nh + lc;
            const size_t step_a = (size_t)args.KA * nh, step_b = (size_t)NBLK * (STEP == 2 ? 128 : args.nhr) * nh;
            const float* Br[NBLK];
            #pragma unroll
            for (int j = 0; j < NBLK; ++j)
            {
                // the last tile across nh may end past nh, not past A's padded rows (nhr is a multiple of 128)
                const size_t row = STEP == 2
                    ? ((size_t)(lam * args.NB + (xb >> 1)) * (2 * NBLK) + j) * 128 + (xb & 1) * kSB + lr
                    : (size_t)(part * NBLK + j) * args.nhr + xb * kSB + lr;
                Br[j] = B + row * nh + lc;
            }
            float4 pa[kLoads], pb[NBLK];
            #pragma unroll
            for (int h = 0; h < kLoads; ++h) pa[h] = *reinterpret_cast<const float4*>(Ar + (size_t)h * 64 * nh);
            #pragma unroll
            for (int j = 0; j < NBLK; ++j) pb[j] = *reinterpret_cast<const float4*>(Br[j]);
            const int chunks = kPh * (nh / kSK);
            for (int ch = 0; ch < chunks; ++ch)
            {
                __syncthreads();
                #pragma unroll
                for (int h = 0; h < kLoads; ++h)
                {
                    const int r = lr + h * 64;
                    sA[lc][r] = pa[h].x; sA[lc + 1][r] = pa[h].y; sA[lc + 2][r] = pa[h].z; sA[lc + 3][r] = pa[h].w;
                }
                #pragma unroll
                for (int j = 0; j < NBLK; ++j)
                {
                    sB[j][lc][lr] = pb[j].x; sB[j][lc + 1][lr] = pb[j].y;
                    sB[j][lc + 2][lr] = pb[j].z; sB[j][lc + 3][lr] = pb[j].w;
                }
                __syncthreads();
                if (ch + 1 < chunks)
                {
                    const int k0 = ((ch + 1) / kPh) * kSK, cs = (ch + 1) % kPh;
                    #pragma unroll
                    for (int h = 0; h < kLoads; ++h) pa[h] = *reinterpret_cast<const float4*>(Ar + cs * step_a + (size_t)h * 64 * nh + k0);
                    #pragma unroll
                    for (int j = 0; j < NBLK; ++j) pb[j] = *reinterpret_cast<const float4*>(Br[j] + cs * step_b + k0);
                }
                #pragma unroll
                for (int kk = 0; kk < kSK; ++kk)
                {
                    float av[P];
                    #pragma unroll
                    for (int h = 0; h < kLoads; ++h)
                    {
                        const float4 a4 = *reinterpret_cast<const float4*>(&sA[kk][h * 64 + ty * 4]);
                        av[4 * h] = a4.x; av[4 * h + 1] = a4.y; av[4 * h + 2] = a4.z; av[4 * h + 3] = a4.w;
                    }
                    #pragma unroll
                    for (int j = 0; j < NBLK; ++j)
                    {
                        const float4 b4 = *reinterpret_cast<const float4*>(&sB[j][kk][tx * 4]);
                        const float bv[4] = {b4.x, b4.y, b4.z, b4.w};
                        #pragma unroll
                        for (int p = 0; p < P; ++p)
                            #pragma unroll
                            for (int q = 0; q < 4; ++q) acc[j][p][q] = fmaf(av[p], bv[q], acc[j][p][q]);
                    }
                }
                if ((ch & 1) == 1 || ch + 1 == chunks)
                {
                    #pragma unroll
                    for (int j = 0; j < NBLK; ++j)
                        #pragma unroll
                        for (int p = 0; p < P; ++p)
                            #pragma unroll
                            for (int q = 0; q < 4; ++q)
                            {
                                total[j][p][q] += acc[j][p][q];
                                acc[j][p][q] = 0.0f;
                            }
                }
            }
        }
        if (STEP == 1)
        {
            // A rows are k, B rows the folded pupil rows: T'[block][k % 128][i]
            float* T = static_cast<float*>(args.tprime);
            const size_t blk = (size_t)(lam * args.NB + (mb >> 1)) * (2 * NBLK) * 128;
            const int i0 = xb * kSB + tx * 4;
            if (i0 >= nh) continue;
            #pragma unroll
            for (int j = 0; j < NBLK; ++j)
            {
                const int dst = BOX ? part : (part == 0 ? (j == 0 ? 0 : 3) : (j == 0 ? 1 : 2));
                const float sign = (part == 0 && j == 0) ? 1.0f : -1.0f;
                #pragma unroll
                for (int p = 0; p < P; ++p)
                    *reinterpret_cast<float4*>(T + (blk + dst * 128 + (mb & 1) * kSB + ty * 4 + p) * nh + i0) =
                        make_float4(sign * total[j][p][0], sign * total[j][p][1], sign * total[j][p][2], sign * total[j][p][3]);
            }
        }
        else
        {
            const float4 w = args.weights[lam];
            const float wr = w.x * args.tint.x, wg = w.y * args.tint.y, wb = w.z * args.tint.z;
            #pragma unroll
            for (int p = 0; p < P; ++p)
            {
                float I[4];
                #pragma unroll
                for (int q = 0; q < 4; ++q)
                {
                    const float re = total[0][p][q], im = BOX ? 0.0f : total[NBLK - 1][p][q];
                    I[q] = BOX ? re : re * re + im * im;
                }
                const int l = mb * kRows + (p >> 2) * 64 + ty * 4 + (p & 3), c0 = xb * kSB + tx * 4;
                if (l >= args.win_h) continue;
                if (n_ranges > 1)
                {
                    *reinterpret_cast<float4*>(args.parts + ((size_t)(lam - args.lam_base) * args.KA + l) * (args.NB * 128) + c0) =
                        make_float4(I[0], I[1], I[2], I[3]);
                    continue;
                }
                const size_t o = (size_t)(args.y0 + l) * args.out_w + args.x0 + c0;
                float* outs[3] = {args.out_r + o, args.out_g + o, args.out_b + o};
                const float wc[3] = {wr, wg, wb};
                #pragma unroll
                for (int c = 0; c < 3; ++c)
                {
                    if (c0 + 3 < args.win_w && ((uintptr_t)outs[c] & 15) == 0)
                        atomicAdd(reinterpret_cast<float4*>(outs[c]), make_float4(wc[c] * I[0], wc[c] * I[1], wc[c] * I[2], wc[c] * I[3]));
                    else
                    {
                        #pragma unroll
                        for (int q = 0; q < 4; ++q)
                            if (c0 + q < args.win_w) atomicAdd(outs[c] + q, wc[c] * I[q]);
                    }
                }
            }
        }
    }
}

// The weighted sum of the wavelengths' planes, in their order, added to the output
// window: a thread four columns of a row.
__global__ void __launch_bounds__(256) mdft_simt_sum(const MdftArgs args, int nl)
{
    after_previous();
    const int quads = args.NB * 32, idx = blockIdx.x * 256 + threadIdx.x;
    const int l = idx / quads, c0 = (idx - l * quads) * 4;
    if (l >= args.win_h || c0 >= args.win_w) return;
    const float4* part = reinterpret_cast<const float4*>(args.parts) + idx;
    const size_t plane = (size_t)args.KA * quads;
    float sum[3][4] = {};
    #pragma unroll 4
    for (int k = 0; k < nl; ++k)
    {
        const float4 w = args.weights[args.lam_base + k], I = part[k * plane];
        const float wc[3] = {w.x * args.tint.x, w.y * args.tint.y, w.z * args.tint.z}, v[4] = {I.x, I.y, I.z, I.w};
        #pragma unroll
        for (int c = 0; c < 3; ++c)
            #pragma unroll
            for (int q = 0; q < 4; ++q) sum[c][q] = fmaf(wc[c], v[q], sum[c][q]);
    }
    const size_t o = (size_t)(args.y0 + l) * args.out_w + args.x0 + c0;
    float* outs[3] = {args.out_r + o, args.out_g + o, args.out_b + o};
    #pragma unroll
    for (int c = 0; c < 3; ++c)          // one plane after the other: they may be the same memory
    {
        if (args.vec && c0 + 3 < args.win_w)
        {
            float4 v = *reinterpret_cast<const float4*>(outs[c]);
            v.x += sum[c][0]; v.y += sum[c][1]; v.z += sum[c][2]; v.w += sum[c][3];
            *reinterpret_cast<float4*>(outs[c]) = v;
        }
        else
        {
            #pragma unroll
            for (int q = 0; q < 4; ++q)
                if (c0 + q < args.win_w) outs[c][q] += sum[c][q];
        }
    }
}

}  // namespace

// ---- MDFT plan ----------------------------------------------------------------
constexpr double kMaxCentre = 12288.0;   // pattern centre range (pixels)

// The kernels' form of a plan.
static int mdft_kernel_form(int form, int box, int n, float red_center)
{
    return form == 0 && (box || red_center != 0.5f * (float)(n - 1)) ? kSplitWhole : form;
}

struct MdftPlan {
    int n = 0, Kx = 0, Ky = 0, n_lambda = 0, form = 0, Kp = 0, elem = 2;
    int kform = 0;          // the kernels' form
    // folded reduction: nf distances |j - cj|, padded to nh (16); nhr rows per
    // part of A' (128); h2 = 2 cj
    // (not folded: nf = nh = n); d0 = smallest distance (not folded: -cj)
    int nf = 0, nh = 0, nhr = 0, h2 = 0;
    float d0 = 0.0f;
    void* wx = nullptr;     // W_x' [lam][C | S][Kx][Kp]
    void* wy = nullptr;     // W_y' [lam][C | S][Ky][Kp]
    void* mask = nullptr;   // A'   [4 parts, box 2][nhr][Kp]
    void* tprime = nullptr; // T'   [lam][Kx/128][4 parts, box 2][128][Kp]
    float* parts = nullptr; // FP32 form: part_l wavelengths' Ky x Kx planes (where step 2 splits them over CTAs)
    int part_l = 0;
    float4* weights = nullptr;
    float2* scales = nullptr;   // [2][n_lambda] (s_hi, s_lo) device copy
    float* amp = nullptr;       // [x, y][n_lambda][nh] factors of the matrix entries
    double cx = 0.0, cy = 0.0;
    float cj = 0.0f;            // reduction-axis centre: (n - 1) / 2, or the zero lag mc of the box form
    int box = 0;                // pixel-integrated form (the reference's MDFT engine)
    int lam0 = 0, lam1 = -1;    // wavelength range of the next executes (lam1 < 0: all)
    int ctas = 0;               // GEMM grid (0 = one CTA per SM)
    int tile_n = 128;           // step-2 output tile width (complex columns): 128 or 64
    int* err = nullptr;
    CUtensorMap t_wx, t_wy, t_mask, t_tp, t_tp64;
    int sms = 0;
    int pairs = 0;              // clusters of two CTAs resident at once (split BF16)
};

static void mdft_free(MdftPlan* p)
{
    if (!p) return;
    cudaFree(p->wx); cudaFree(p->wy); cudaFree(p->mask); cudaFree(p->tprime); cudaFree(p->parts);
    cudaFree(p->weights); cudaFree(p->scales); cudaFree(p->amp); cudaFree(p->err);
    delete p;
}

}  // namespace gl

struct gl_mdft_plan { gl::MdftPlan* p; };

namespace gl {

// Enqueue the DFT matrices of the plan's current centre.
static cudaError_t mdft_build_matrices(MdftPlan* p, cudaStream_t st)
{
    const float cxh = (float)p->cx, cxl = (float)(p->cx - (double)cxh);
    const float cyh = (float)p->cy, cyl = (float)(p->cy - (double)cyh);
    const DftRows R[2] = {{p->wx, p->scales, p->amp, cxh, cxl, p->Kx},
                          {p->wy, p->scales + p->n_lambda, p->amp + (size_t)p->n_lambda * p->nh, cyh, cyl, p->Ky}};
    const int tx = p->nh >= 128 ? 64 : 32;             // two entries per thread and pass
    const dim3 block(tx, 256 / tx);
    for (const DftRows& r : R)
    {
        const int grid = (p->n_lambda * r.K + (int)block.y - 1) / (int)block.y;
        if (p->kform == kSplitWhole) mdft_dft_kernel<kSplitWhole><<<grid, block, 0, st>>>(r, p->n_lambda, p->nh, p->d0);
        else if (p->form == 0) mdft_dft_kernel<0><<<grid, block, 0, st>>>(r, p->n_lambda, p->nh, p->d0);
        else if (p->form == kTf32) mdft_dft_kernel<kTf32><<<grid, block, 0, st>>>(r, p->n_lambda, p->nh, p->d0);
        else mdft_dft_kernel<2><<<grid, block, 0, st>>>(r, p->n_lambda, p->nh, p->d0);
    }
    return cudaGetLastError();
}

// Opt one GEMM instance in to its shared memory.
template <int FORM, int STEP, int TN, bool BOX, int CL>
static cudaError_t mdft_prepare()
{
    return cudaFuncSetAttribute(mdft_kernel<FORM, STEP, TN, BOX, CL>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                MdftShape<FORM, STEP, TN, BOX, CL>::kSmem);
}

struct MdftLaunch {
    cudaLaunchConfig_t cfg{};
    cudaLaunchAttribute attr{};
    MdftLaunch(int grid, int cl, int smem, cudaStream_t st)
    {
        cfg.gridDim = dim3((unsigned)grid);
        cfg.blockDim = dim3(kMdftThreads);
        cfg.dynamicSmemBytes = (size_t)smem;
        cfg.stream = st;
        if (cl == 1) return;
        attr.id = cudaLaunchAttributeClusterDimension;
        attr.val.clusterDim.x = (unsigned)cl;
        attr.val.clusterDim.y = attr.val.clusterDim.z = 1;
        cfg.attrs = &attr;
        cfg.numAttrs = 1;
    }
};

// *pairs: pairs of CTAs that are resident at once (0: the form has none).
template <int FORM, bool BOX>
static cudaError_t mdft_prepare_all(int* pairs)
{
    cudaError_t e = mdft_prepare<FORM, 1, 128, BOX, 1>();
    if (e == cudaSuccess) e = mdft_prepare<FORM, 2, 128, BOX, 1>();
    if (e == cudaSuccess) e = mdft_prepare<FORM, 2, 64, BOX, 1>();
    *pairs = 0;
    if constexpr (FORM == 0 && !BOX)
    {
        if (e == cudaSuccess) e = mdft_prepare<0, 1, 128, false, 2>();
        if (e == cudaSuccess) e = mdft_prepare<0, 2, 128, false, 2>();
        int n1 = 0, n2 = 0;
        const MdftLaunch L1(2, 2, MdftShape<0, 1, 128, false, 2>::kSmem, nullptr);
        const MdftLaunch L2(2, 2, MdftShape<0, 2, 128, false, 2>::kSmem, nullptr);
        if (e == cudaSuccess) e = cudaOccupancyMaxActiveClusters(&n1, mdft_kernel<0, 1, 128, false, 2>, &L1.cfg);
        if (e == cudaSuccess) e = cudaOccupancyMaxActiveClusters(&n2, mdft_kernel<0, 2, 128, false, 2>, &L2.cfg);
        if (e == cudaSuccess) *pairs = std::min(n1, n2);
    }
    return e;
}

// One step over its units.  The field form in split BF16 runs in pairs where the
// row blocks come in pairs, a unit's reduction is long and there are many units: a
// cluster's launch costs 2 us more, and a short reduction is bound by its epilogue.
// Measured, whole plan, step in single CTAs -> in pairs: step 2 at 8 stages a unit
// 682 -> 621 us (7936 units), 95.5 -> 92.3 (496), 37.0 -> 38.9 (128), at 4 stages
// 148 -> 152; step 1 at 16 stages 137 -> 125 (512 units), at 8 stages 141 -> 137 and
// 355 -> 379, at 4 stages 219 -> 224.
template <int FORM, int STEP, int TN, bool BOX>
static int mdft_pairs(const MdftArgs& a, int gmax, int pairs)
{
    if constexpr (FORM == 0 && !BOX && TN == 128)
    {
        const int stages = MdftShape<FORM, STEP, TN, BOX, 2>::kPhases * a.nkb;
        const bool worth = stages >= (STEP == 1 ? 16 : 8) && (long long)stages * a.n_units >= 3000;
        if ((a.NBm & 1) == 0 && worth) return std::min(std::min(a.n_units, gmax) / 2, pairs);
    }
    return 0;
}

template <int FORM, int STEP, int TN, bool BOX>
static cudaError_t mdft_step(const CUtensorMap& tA, const CUtensorMap& tB, const MdftArgs& a, int gmax, int pairs, cudaStream_t st)
{
    if constexpr (FORM == 0 && !BOX && TN == 128)
    {
        const int two = mdft_pairs<FORM, STEP, TN, BOX>(a, gmax, pairs);
        if (two > 0)
        {
            const MdftLaunch L(2 * two, 2, MdftShape<FORM, STEP, TN, BOX, 2>::kSmem, st);
            return cudaLaunchKernelEx(&L.cfg, mdft_kernel<FORM, STEP, TN, BOX, 2>, tA, tB, a);
        }
    }
    const MdftLaunch L(std::min(a.n_units, gmax), 1, MdftShape<FORM, STEP, TN, BOX, 1>::kSmem, st);
    return cudaLaunchKernelEx(&L.cfg, mdft_kernel<FORM, STEP, TN, BOX, 1>, tA, tB, a);
}

template <int FORM, bool BOX>
static cudaError_t mdft_gemms(const MdftPlan* p, const MdftArgs& a1, const MdftArgs& a2, int gmax, cudaStream_t st)
{
    cudaError_t e = mdft_step<FORM, 1, 128, BOX>(p->t_wx, p->t_mask, a1, gmax, p->pairs, st);
    if (e != cudaSuccess) return e;
    return p->tile_n == 64 ? mdft_step<FORM, 2, 64, BOX>(p->t_wy, p->t_tp64, a2, gmax, p->pairs, st)
                           : mdft_step<FORM, 2, 128, BOX>(p->t_wy, p->t_tp, a2, gmax, p->pairs, st);
}

// Wavelengths of the FP32 form whose planes are kept at a time: 64 MB of them,
// which stay in L2 between step 2 and the sum.  0: the output has tiles enough
// for every SM without splitting the wavelengths.
static int mdft_part_lambdas(int Kx, int Ky, int n_lambda, int sms)
{
    if (n_lambda < 2 || (long long)(Kx / kSB) * (Ky / kSB) >= 4LL * sms) return 0;
    return (int)std::max<long long>(2, std::min<long long>(n_lambda, (16LL << 20) / ((long long)Kx * Ky)));
}

// Both steps; *launches grows by their launches (each set up while the one before
// drains, gl_launch.cuh).
template <bool BOX>
static cudaError_t mdft_simt(const MdftPlan* p, const MdftArgs& a1, const MdftArgs& a2, int l1, int* launches, cudaStream_t st)
{
    const int nl = l1 - a1.lam_base;
    const dim3 t1((p->nh + kSB - 1) / kSB, p->Kx / kSB, 2 * nl);
    cudaError_t e = launch_after(mdft_simt_kernel<1, BOX, 4>, t1, 256, 0, st, static_cast<const float*>(p->wx),
                                 static_cast<const float*>(p->mask), a1, l1, 1);
    ++*launches;
    const int tiles = (p->Kx / kSB) * (p->Ky / kSB);
    const int groups = p->part_l > 0 ? (nl + p->part_l - 1) / p->part_l : 1;
    MdftArgs a = a2;
    for (int g = 0; g < groups; ++g)
    {
        a.lam_base = a2.lam_base + (int)((long long)nl * g / groups);
        const int lg = a2.lam_base + (int)((long long)nl * (g + 1) / groups), n = lg - a.lam_base;
        // Tall tiles read a third less shared memory per FMA, but halve the CTAs.  256^2
        // to 512^2, whole call, 64 x 64 -> 128 x 64: 86 -> 78 us (256 tall CTAs), 47 -> 45
        // (96), 35 -> 43 (64), 35 -> 43 (32); pixel form, half the FMA per load: 117 -> 109,
        // 64 -> 60, 39 -> 50, 36 -> 49.
        const bool tall = (long long)tiles * n > p->sms;          // tiles / 2 tall ones: half of the SMs or more
        const int rows = tall ? 128 : kSB;
        // wavelength ranges until about three CTAs per SM are in flight (tall tiles,
        // twice the work each: two)
        const int ranges = p->part_l > 0 ? std::min(n, std::max(1, ((tall ? 2 : 3) * p->sms + tiles * kSB / rows - 1) / (tiles * kSB / rows))) : 1;
        const dim3 t2(p->Kx / kSB, p->Ky / rows, ranges);
        if (e == cudaSuccess)
            e = launch_after(tall ? mdft_simt_kernel<2, BOX, 8> : mdft_simt_kernel<2, BOX, 4>, t2, 256, 0, st,
                             static_cast<const float*>(p->wy), static_cast<const float*>(p->tprime), a, lg, ranges);
        ++*launches;
        const int quads = p->Kx / 4 * a2.win_h;
        if (ranges == 1 || quads == 0) continue;
        if (e == cudaSuccess) e = launch_after(mdft_simt_sum, (quads + 255) / 256, 256, 0, st, a, n);
        ++*launches;
    }
    return e;
}

}  // namespace gl

extern "C" int gl_mdft_plan_create3(int n, int Kx, int Ky, int n_lambda, const double* scale_x, const double* scale_y,
                                    double center_x, double center_y, const float* weights_rgb, int form, int box,
                                    float red_center, void* stream, gl_mdft_plan** out)
{
    using namespace gl;
    if (!out || !scale_x || !scale_y || !weights_rgb) return fail(GL_ERR_INVALID, "mdft_plan_create: null argument");
    if (box != 0 && box != 1) return fail(GL_ERR_INVALID, "mdft_plan_create: box must be 0 or 1");
    if (!(red_center >= 0.0f) || !(red_center <= (float)n) || red_center != std::floor(2.0f * red_center) * 0.5f)
        return fail(GL_ERR_INVALID, "mdft_plan_create: the reduction centre must be a whole or half index in [0, n]");
    if (n <= 0 || n % 128 || Kx <= 0 || Kx % 128 || Ky <= 0 || Ky % 128)
        return fail(GL_ERR_INVALID, "mdft_plan_create: the pupil side n and output sides Kx, Ky must be multiples of 128");
    if (Kx > 8192 || Ky > 8192 || n > 4096) return fail(GL_ERR_INVALID, "mdft_plan_create: sides above 8192 (4096 for n)");
    if (n_lambda < 1 || n_lambda > 1024) return fail(GL_ERR_INVALID, "mdft_plan_create: 1..1024 wavelengths");
    if (form < 0 || form > 2)
        return fail(GL_ERR_UNSUPPORTED, "mdft_plan_create: form must be 0 (split BF16), 1 (TF32) or 2 (FP32 CUDA cores)");
    // |k - c| < 8192 + 12288 and |j - cj| <= 2048 keep the phase product
    // a (k - c) below 2^26, whose float rounding error the FMA captures exactly
    if (!(std::fabs(center_x) < kMaxCentre) || !(std::fabs(center_y) < kMaxCentre))
        return fail(GL_ERR_INVALID, "mdft_plan_create: centre coordinates must lie within +-12288 pixels");
    cudaStream_t st = (cudaStream_t)stream;
    MdftPlan* p = new MdftPlan();
    p->n = n; p->Kx = Kx; p->Ky = Ky; p->n_lambda = n_lambda; p->form = form;
    p->cx = center_x; p->cy = center_y;
    p->box = box; p->cj = red_center;
    p->h2 = (int)(2.0f * red_center);
    p->kform = mdft_kernel_form(form, box, n, red_center);
    const bool folded = is_folded(p->kform), distances = folded && !box;
    p->nf = !distances ? n : (int)std::floor(std::max((double)red_center, (double)(n - 1) - (double)red_center)) + 1;
    p->d0 = !distances ? -red_center : ((p->h2 & 1) ? 0.5f : 0.0f);
    p->nh = (p->nf + 15) / 16 * 16;
    p->nhr = (p->nh + 127) / 128 * 128;
    p->Kp = form == 0 ? 2 * p->nh : p->nh;
    p->elem = form == 0 ? 2 : 4;
    const int NBx = Kx / 128, parts = (box || !folded) ? 2 : 4;            // of T'
    const int mparts = !folded ? 1 : parts;                          // of A'
    const size_t wxbytes = (size_t)n_lambda * 2 * Kx * p->Kp * p->elem;
    const size_t wybytes = (size_t)n_lambda * 2 * Ky * p->Kp * p->elem;
    const size_t mbytes = (size_t)mparts * p->nhr * p->Kp * p->elem;
    const size_t tbytes = (size_t)n_lambda * NBx * parts * 128 * p->Kp * p->elem;
    cudaError_t e = cudaSuccess;
    auto chk = [&](cudaError_t x) { if (e == cudaSuccess) e = x; };
    chk(cudaMalloc(&p->wx, wxbytes));
    chk(cudaMalloc(&p->wy, wybytes));
    chk(cudaMalloc(&p->mask, mbytes));
    chk(cudaMalloc(&p->tprime, tbytes));
    chk(cudaMalloc(&p->weights, sizeof(float4) * n_lambda));
    chk(cudaMalloc(&p->scales, sizeof(float2) * 2 * n_lambda));
    chk(cudaMalloc(&p->amp, sizeof(float) * 2 * n_lambda * p->nh));
    chk(cudaMalloc(&p->err, sizeof(int)));
    chk(cudaMemset(p->err, 0, sizeof(int)));          // a plan never executed reports no error
    chk(cudaMemset(p->mask, 0, mbytes));              // the rows between nh and nhr stay zero
    int dev = 0;
    chk(cudaGetDevice(&dev));
    chk(cudaDeviceGetAttribute(&p->sms, cudaDevAttrMultiProcessorCount, dev));
    if (e == cudaSuccess && form == 2) p->part_l = mdft_part_lambdas(Kx, Ky, n_lambda, p->sms);
    if (p->part_l > 0) chk(cudaMalloc(&p->parts, sizeof(float) * (size_t)p->part_l * Kx * Ky));
    if (e != cudaSuccess)
    {
        mdft_free(p);
        return fail(e == cudaErrorMemoryAllocation ? GL_ERR_OOM : GL_ERR_CUDA, std::string("mdft_plan_create: ") + cudaGetErrorString(e));
    }
    std::vector<float4> w((size_t)n_lambda);
    for (int l = 0; l < n_lambda; ++l) w[l] = make_float4(weights_rgb[3 * l], weights_rgb[3 * l + 1], weights_rgb[3 * l + 2], 0.0f);
    std::vector<float2> sc((size_t)2 * n_lambda);
    for (int l = 0; l < n_lambda; ++l)
    {
        const float xh = (float)scale_x[l], yh = (float)scale_y[l];
        sc[l] = make_float2(xh, (float)(scale_x[l] - (double)xh));
        sc[n_lambda + l] = make_float2(yh, (float)(scale_y[l] - (double)yh));
    }
    chk(cudaMemcpy(p->weights, w.data(), sizeof(float4) * n_lambda, cudaMemcpyHostToDevice));
    chk(cudaMemcpy(p->scales, sc.data(), sizeof(float2) * 2 * n_lambda, cudaMemcpyHostToDevice));
    if (e == cudaSuccess)
    {
        mdft_amp_kernel<<<2 * n_lambda, 256, 0, st>>>(p->amp, p->scales, p->nh, p->nf, p->d0, box);
        chk(mdft_build_matrices(p, st));
    }
    chk(cudaStreamSynchronize(st));
    // shared-memory opt-in once here, so execute enqueues kernels only (graph capture)
    if (p->kform == kSplitWhole) chk(box ? mdft_prepare_all<kSplitWhole, true>(&p->pairs) : mdft_prepare_all<kSplitWhole, false>(&p->pairs));
    else if (form == 0) chk(mdft_prepare_all<0, false>(&p->pairs));
    else if (form == 1) chk(box ? mdft_prepare_all<1, true>(&p->pairs) : mdft_prepare_all<1, false>(&p->pairs));
    const CUtensorMapDataType dt = form == 0 ? CU_TENSOR_MAP_DATA_TYPE_BFLOAT16 : CU_TENSOR_MAP_DATA_TYPE_FLOAT32;
    const uint32_t bc = form == 0 ? 64 : 32;
    int rc = GL_OK;
    if (e == cudaSuccess && form != 2)
    {
        rc = make_tmap_2d(&p->t_wx, p->wx, dt, p->elem, (uint64_t)n_lambda * 2 * Kx, (uint64_t)p->Kp, 128, bc);
        if (!rc) rc = make_tmap_2d(&p->t_wy, p->wy, dt, p->elem, (uint64_t)n_lambda * 2 * Ky, (uint64_t)p->Kp, 128, bc);
        if (!rc) rc = make_tmap_2d(&p->t_mask, p->mask, dt, p->elem, (uint64_t)mparts * p->nhr, (uint64_t)p->Kp, 128, bc);
        if (!rc) rc = make_tmap_2d(&p->t_tp, p->tprime, dt, p->elem, (uint64_t)n_lambda * NBx * parts * 128, (uint64_t)p->Kp, 128, bc);
        if (!rc) rc = make_tmap_2d(&p->t_tp64, p->tprime, dt, p->elem, (uint64_t)n_lambda * NBx * parts * 128, (uint64_t)p->Kp, 64, bc);
    }
    if (e != cudaSuccess || rc)
    {
        mdft_free(p);
        if (rc) return rc;
        return fail(GL_ERR_CUDA, std::string("mdft_plan_create: ") + cudaGetErrorString(e));
    }
    *out = new gl_mdft_plan{p};
    return GL_OK;
}

extern "C" int gl_mdft_plan_create2(int n, int Kx, int Ky, int n_lambda, const double* scale_x, const double* scale_y,
                                    double center_x, double center_y, const float* weights_rgb, int form, void* stream,
                                    gl_mdft_plan** out)
{
    return gl_mdft_plan_create3(n, Kx, Ky, n_lambda, scale_x, scale_y, center_x, center_y, weights_rgb, form, 0,
                                0.5f * (float)(n - 1), stream, out);
}

extern "C" int gl_mdft_plan_create(int n, int K_out, int n_lambda, const double* scale_x, const double* scale_y,
                                   double center_x, double center_y, const float* weights_rgb, int form,
                                   void* stream, gl_mdft_plan** out)
{
    return gl_mdft_plan_create2(n, K_out, K_out, n_lambda, scale_x, scale_y, center_x, center_y, weights_rgb, form,
                                stream, out);
}

extern "C" int gl_mdft_plan_set_center(gl_mdft_plan* plan, double center_x, double center_y, void* stream)
{
    using namespace gl;
    if (!plan) return fail(GL_ERR_INVALID, "mdft_plan_set_center: null plan");
    if (!(std::fabs(center_x) < kMaxCentre) || !(std::fabs(center_y) < kMaxCentre))
        return fail(GL_ERR_INVALID, "mdft_plan_set_center: centre coordinates must lie within +-12288 pixels");
    plan->p->cx = center_x;
    plan->p->cy = center_y;
    GL_CUDA_TRY(mdft_build_matrices(plan->p, (cudaStream_t)stream));
    g_last_launches = 2;
    return GL_OK;
}

// The sizes of both steps' reductions and units; a1 holds what they share.
static void mdft_units(const MdftPlan* p, MdftArgs& a1, MdftArgs& a2)
{
    const int kbe = p->form == 0 ? 64 : 32, nl = (p->lam1 < 0 ? p->n_lambda : p->lam1) - p->lam0;
    a1.KA = p->Kx;
    a1.NB = a1.NBm = a1.NBt = p->Kx / 128;
    a1.nh = p->nh; a1.nhr = p->nhr;
    a1.nkb = (p->nh + kbe - 1) / kbe * (p->kform == kSplitWhole ? 3 : 1);
    a1.NI = p->nhr / 128;
    a1.lam_base = p->lam0;
    // step 1: (lambda, k block, pupil-row block, C / S); step 2: (lambda, output tile)
    a1.n_units = nl * a1.NB * a1.NI * (is_folded(p->kform) ? 2 : 1);
    a2 = a1;
    a2.KA = p->Ky; a2.NBm = p->Ky / 128;
    a2.NBt = p->Kx / p->tile_n;
    a2.n_units = a2.NBm * a2.NBt * nl;
}

extern "C" int gl_mdft_plan_pairs(const gl_mdft_plan* plan, int* step1, int* step2)
{
    using namespace gl;
    if (!plan || !step1 || !step2) return fail(GL_ERR_INVALID, "mdft_plan_pairs: null argument");
    const MdftPlan* p = plan->p;
    MdftArgs a1{}, a2;
    mdft_units(p, a1, a2);
    const int gmax = p->ctas > 0 ? p->ctas : p->sms;
    const bool field = p->kform == 0;
    *step1 = field ? mdft_pairs<0, 1, 128, false>(a1, gmax, p->pairs) : 0;
    *step2 = field && p->tile_n == 128 ? mdft_pairs<0, 2, 128, false>(a2, gmax, p->pairs) : 0;
    return GL_OK;
}

extern "C" int gl_mdft_plan_execute3(gl_mdft_plan* plan, const float* d_pupil, float* d_out_r, float* d_out_g,
                                     float* d_out_b, int accumulate, int out_w, int out_h, int x0, int y0, int win_w,
                                     int win_h, const float* tint_rgb, void* stream)
{
    using namespace gl;
    if (!plan || !d_pupil || !d_out_r || !d_out_g || !d_out_b) return fail(GL_ERR_INVALID, "mdft_plan_execute: null argument");
    MdftPlan* p = plan->p;
    if (out_w <= 0 || out_h <= 0 || x0 < 0 || y0 < 0 || win_w < 0 || win_h < 0 || win_w > p->Kx || win_h > p->Ky ||
        x0 + win_w > out_w || y0 + win_h > out_h)
        return fail(GL_ERR_INVALID, "mdft_plan_execute: the output window must lie inside the planes and the plan");
    cudaStream_t st = (cudaStream_t)stream;
    const size_t npx = (size_t)out_w * out_h;
    int launches = 0;
    // zeroing blocks: one wave of the chip at most, one block at least (the error
    // word).  A pupil that shares memory with a plane is read before the plane is
    // zeroed, by memsets behind the fold.
    float* planes[3] = {d_out_r, d_out_g, d_out_b};
    const uintptr_t pupil0 = reinterpret_cast<uintptr_t>(d_pupil), pupil1 = pupil0 + sizeof(float) * (size_t)p->n * p->n;
    bool shared = false;
    for (float* c : planes)
    {
        const uintptr_t c0 = reinterpret_cast<uintptr_t>(c);
        shared = shared || (pupil0 < c0 + sizeof(float) * npx && c0 < pupil1);
    }
    const size_t zero = accumulate || shared ? 0 : npx;
    const int fold = p->nh + (int)std::max<size_t>(1, std::min<size_t>((3 * zero / 4 + 1023) / 1024, 16 * (size_t)p->sms));
    auto run_fold = [&](auto kernel) {
        kernel<<<fold, 128, 0, st>>>(d_pupil, p->mask, p->n, p->nh, p->nhr, p->nf, p->h2, p->box, d_out_r, d_out_g,
                                     d_out_b, zero, p->err);
    };
    if (p->kform == kSplitWhole) run_fold(mdft_fold_kernel<kSplitWhole>);
    else if (p->form == 0) run_fold(mdft_fold_kernel<0>);
    else if (p->form == kTf32) run_fold(mdft_fold_kernel<kTf32>);
    else run_fold(mdft_fold_kernel<2>);
    ++launches;
    if (shared && !accumulate)
        for (float* c : planes) GL_CUDA_TRY(cudaMemsetAsync(c, 0, sizeof(float) * npx, st));
    MdftArgs a{}, a2;
    a.tprime = p->tprime; a.out_r = d_out_r; a.out_g = d_out_g; a.out_b = d_out_b;
    a.weights = p->weights; a.err = p->err; a.parts = p->parts;
    a.out_w = out_w; a.x0 = x0; a.y0 = y0; a.win_w = win_w; a.win_h = win_h;
    // the planes may be views that start at any float
    a.vec = ((out_w | x0) & 3) == 0 && ((reinterpret_cast<uintptr_t>(d_out_r) | reinterpret_cast<uintptr_t>(d_out_g) |
                                         reinterpret_cast<uintptr_t>(d_out_b)) & 15) == 0;
    a.tint = tint_rgb ? make_float4(tint_rgb[0], tint_rgb[1], tint_rgb[2], 0.0f) : make_float4(1.0f, 1.0f, 1.0f, 0.0f);
    const int gmax = p->ctas > 0 ? p->ctas : p->sms, l1 = p->lam1 < 0 ? p->n_lambda : p->lam1;
    mdft_units(p, a, a2);
    if (p->form == 2)
    {
        GL_CUDA_TRY(p->box ? mdft_simt<true>(p, a, a2, l1, &launches, st) : mdft_simt<false>(p, a, a2, l1, &launches, st));
    }
    else if (p->form == 0)
    {
        if (p->kform == 0) GL_CUDA_TRY((mdft_gemms<0, false>(p, a, a2, gmax, st)));
        else GL_CUDA_TRY(p->box ? (mdft_gemms<kSplitWhole, true>(p, a, a2, gmax, st)) : (mdft_gemms<kSplitWhole, false>(p, a, a2, gmax, st)));
    }
    else
    {
        GL_CUDA_TRY(p->box ? (mdft_gemms<1, true>(p, a, a2, gmax, st)) : (mdft_gemms<1, false>(p, a, a2, gmax, st)));
    }
    GL_CUDA_TRY(cudaGetLastError());
    if (p->form != 2) launches += 2;
    g_last_launches = launches;
    return GL_OK;
}

extern "C" int gl_mdft_plan_execute2(gl_mdft_plan* plan, const float* d_pupil, float* d_out_r, float* d_out_g,
                                     float* d_out_b, int accumulate, void* stream)
{
    if (!plan) return gl::fail(GL_ERR_INVALID, "mdft_plan_execute: null argument");
    const gl::MdftPlan* p = plan->p;
    return gl_mdft_plan_execute3(plan, d_pupil, d_out_r, d_out_g, d_out_b, accumulate, p->Kx, p->Ky, 0, 0, p->Kx, p->Ky,
                                 nullptr, stream);
}

extern "C" int gl_mdft_plan_set_lambda_range(gl_mdft_plan* plan, int lam_begin, int lam_end)
{
    using namespace gl;
    if (!plan) return fail(GL_ERR_INVALID, "mdft_plan_set_lambda_range: null plan");
    MdftPlan* p = plan->p;
    if (lam_begin == 0 && lam_end < 0) { p->lam0 = 0; p->lam1 = -1; return GL_OK; }
    if (lam_begin < 0 || lam_end <= lam_begin || lam_end > p->n_lambda)
        return fail(GL_ERR_INVALID, "mdft_plan_set_lambda_range: need 0 <= begin < end <= n_lambda");
    p->lam0 = lam_begin;
    p->lam1 = lam_end;
    return GL_OK;
}

extern "C" int gl_mdft_plan_set_launch(gl_mdft_plan* plan, int ctas)
{
    using namespace gl;
    if (!plan || ctas < 0) return fail(GL_ERR_INVALID, "mdft_plan_set_launch: bad arguments");
    // one 192-thread CTA with up to 210 KB of shared memory fits per SM
    plan->p->ctas = ctas == 0 ? 0 : std::min(ctas, plan->p->sms);
    return GL_OK;
}

extern "C" int gl_mdft_plan_set_tile(gl_mdft_plan* plan, int tile_n)
{
    using namespace gl;
    if (!plan || (tile_n != 64 && tile_n != 128))
        return fail(GL_ERR_INVALID, "mdft_plan_set_tile: the tile width must be 64 or 128 output columns");
    plan->p->tile_n = tile_n;
    return GL_OK;
}

extern "C" int gl_mdft_plan_execute(gl_mdft_plan* plan, const float* d_pupil, float* d_out_r, float* d_out_g,
                                    float* d_out_b, void* stream)
{
    return gl_mdft_plan_execute2(plan, d_pupil, d_out_r, d_out_g, d_out_b, 0, stream);
}

extern "C" int gl_build_pupil2(const gl_surface* surfaces, int n_surfaces, int N, float pupil_fill,
                               int blades_override, float rotation_deg, int aspect_one, const float* d_env, int env_n,
                               float* d_out, void* stream)
{
    using namespace gl;
    if (!surfaces || n_surfaces <= 0 || !d_out) return fail(GL_ERR_INVALID, "build_pupil: bad arguments");
    if (N <= 0 || N > 8192) return fail(GL_ERR_INVALID, "build_pupil: N must be 1..8192");
    if (!(pupil_fill > 0.0f) || pupil_fill > 1.0f) return fail(GL_ERR_INVALID, "build_pupil: pupil_fill must lie in (0, 1]");
    if (d_env && (env_n < 1 || env_n > 4096)) return fail(GL_ERR_INVALID, "build_pupil: envelope side must be 1..4096");
    PupilMask m = resolve_pupil_mask(surfaces, n_surfaces, blades_override, rotation_deg);
    if (aspect_one) m.aspect = 1.0f;
    PupilDev d{m.aspect, m.rot_rad, m.apothem, m.sector, m.n_blades, m.blade};
    const int total = N * N;
    pupil_build_kernel<<<(total + 255) / 256, 256, 0, (cudaStream_t)stream>>>(d_out, N, pupil_fill, d, d_env, env_n);
    GL_CUDA_TRY(cudaGetLastError());
    g_last_launches = 1;
    return GL_OK;
}

extern "C" int gl_build_pupil(const gl_surface* surfaces, int n_surfaces, int N, float pupil_fill,
                              int blades_override, float rotation_deg, float* d_out, void* stream)
{
    return gl_build_pupil2(surfaces, n_surfaces, N, pupil_fill, blades_override, rotation_deg, 0, nullptr, 0, d_out,
                           stream);
}

extern "C" int gl_mdft_plan_status(gl_mdft_plan* plan, int* err_code)
{
    if (!plan || !err_code) return gl::fail(GL_ERR_INVALID, "mdft_plan_status: null argument");
    GL_CUDA_TRY(cudaMemcpy(err_code, plan->p->err, sizeof(int), cudaMemcpyDeviceToHost));
    return GL_OK;
}

extern "C" int gl_mdft_plan_destroy(gl_mdft_plan* plan)
{
    if (!plan) return GL_OK;
    gl::mdft_free(plan->p);
    delete plan;
    return GL_OK;
}
