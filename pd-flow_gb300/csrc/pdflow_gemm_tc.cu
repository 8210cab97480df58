// BF16 GEMM on the 5th-generation tensor cores (tcgen05, sm_103a).
//
//   C[M, N] (+)= A[M, K] * B[N, K]^T        A, B: bf16, K contiguous
//
// One CTA of 128 threads owns a 128 x BN tile of C (BN = 16..128, multiple of
// 16).  K advances in chunks of 64 through a 3-stage ring: all threads copy
// the A and B chunks into shared memory with asynchronous 16-byte copies
// (cp.async, two chunks ahead of the one being multiplied) in the canonical
// no-swizzle K-major layout (8-row x 16-byte core matrices; 128 B between core
// matrices along K, 1024 B between 8-row groups), one elected thread issues
// four tcgen05.mma (K = 16 each) into an FP32 accumulator in tensor memory and
// commits them to the stage's mbarrier, which frees the stage for the chunk
// three ahead.  The epilogue
// reads the accumulator with tcgen05.ld (warp w owns TMEM lanes 32w..32w+31 =
// rows of the tile), adds the bias, applies ReLU and stores FP32 or BF16, 16
// bytes at a time where rows are aligned (a value at a time, a 64-input
// gradient took 6.87 ms on a GB300 instead of 5.36).
// grid.z splits K (split-K partials go to C + z * split_stride).
//
// Every wait is bounded: a wait that gives up records kGemmTimeout in
// *status, the kernel still drains, frees its tensor memory and returns.
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include "pdflow_gemm_tc.cuh"

namespace pdflow {
namespace {

constexpr int kBM = 128, kBK = 64, kMaxBN = 128, kThreads = 128;
constexpr uint32_t kTmemCols = 128;
constexpr int kStageA = kBM * kBK * 2;         // 16 KB
constexpr int kStageB = kMaxBN * kBK * 2;      // 16 KB at the widest N tile
constexpr int kStages = 3;
constexpr int kSmemBytes = kStages * (kStageA + kStageB) + 64;   // the attribute: the largest launch
// A launch's B stages hold only its N tile (bn rows), so narrow GEMMs fit
// more CTAs per SM (bn = 16: 55 KB, four CTAs, 4 x 128 TMEM columns = 512).
constexpr int smem_bytes(int bn) { return kStages * (kStageA + bn * kBK * 2) + 64; }
constexpr uint32_t kWaitLimit = 1u << 20;

__device__ __forceinline__ uint32_t smem_u32(const void* p)
{
    return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}

// Shared-memory matrix descriptor (tcgen05 format): start address, leading
// byte offset (K direction), stride byte offset (M/N direction), all >> 4;
// bits 46-48 = 0b001; no swizzle.
__device__ __forceinline__ uint64_t smem_desc(uint32_t addr, uint32_t lbo, uint32_t sbo)
{
    uint64_t d = 0;
    d |= uint64_t((addr >> 4) & 0x3FFFu);
    d |= uint64_t((lbo >> 4) & 0x3FFFu) << 16;
    d |= uint64_t((sbo >> 4) & 0x3FFFu) << 32;
    d |= uint64_t(1) << 46;
    return d;
}

// Instruction descriptor of kind::f16: D = F32, A = B = BF16, both K-major.
__device__ __forceinline__ uint32_t instr_desc(int bn)
{
    return (1u << 4) | (1u << 7) | (1u << 10) | (uint32_t(bn >> 3) << 17) | (uint32_t(kBM >> 4) << 24);
}

__device__ __forceinline__ bool mbar_wait(uint32_t addr, uint32_t parity)
{
    for (uint32_t i = 0; i < kWaitLimit; ++i) {
        uint32_t ok;
        asm volatile(
            "{\n\t.reg .pred p;\n\t"
            "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
            "selp.u32 %0, 1, 0, p;\n\t}"
            : "=r"(ok)
            : "r"(addr), "r"(parity)
            : "memory");
        if (ok) return true;
    }
    return false;
}

__device__ __forceinline__ void fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }

// Starts the asynchronous copy of rows [row0, row0 + rows) x K chunk
// [k0, k0 + 64) of a K-major bf16 matrix into the core-matrix layout; rows >=
// nrows and k >= K are zero-filled (source size 0, the source address is then
// the matrix base and nothing is read).  K is a multiple of 8, so a 16-byte
// piece is wholly inside or wholly outside.
__device__ __forceinline__ void stage_tile(unsigned char* dst, const __nv_bfloat16* src, int ld, int row0,
                                           int rows, int nrows, int k0, int K)
{
    const int chunks = rows * 8;   // 16-byte pieces
    for (int c = threadIdx.x; c < chunks; c += kThreads) {
        const int r = c % rows, kc = c / rows;
        const int gr = row0 + r, gk = k0 + kc * 8;
        const bool in = gr < nrows && gk < K;
        const __nv_bfloat16* g = in ? src + (size_t)gr * ld + gk : src;
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(
                         smem_u32(dst + ((r >> 3) * 8 + kc) * 128 + (r & 7) * 16)),
                     "l"(g), "r"(in ? 16 : 0)
                     : "memory");
    }
}

// The pixel of an A row gathered by ConvGather: each thread stages the same
// row of every A tile (kThreads == kBM), so its (b, y, x) is found once.
struct ConvRow {
    int b, y, x;
    bool valid;
};

__device__ __forceinline__ ConvRow conv_row(const ConvGather& cv, int gr, int nrows)
{
    ConvRow cr;
    const int hw = cv.H * cv.W;
    cr.valid = gr < nrows;
    cr.b = gr / hw;
    const int rr = gr - cr.b * hw;
    cr.y = rr / cv.W;
    cr.x = rr - cr.y * cv.W;
    return cr;
}

// stage_tile for an A operand that is the im2col of a 3x3 convolution
// (ConvGather): each 16-byte piece is 8 channels of one tap of this thread's
// pixel, read from the NHWC source, or zero-filled outside the image, past
// row nrows or past K, exactly the values the materialised im2col holds.
__device__ __forceinline__ void stage_conv_tile(unsigned char* dst, const ConvGather& cv, const ConvRow& cr, int k0,
                                                int K)
{
    static_assert(kThreads == kBM, "one A row per thread");
    const __nv_bfloat16* s1 = static_cast<const __nv_bfloat16*>(cv.s1);
    const __nv_bfloat16* s2 = static_cast<const __nv_bfloat16*>(cv.s2);
    const int cin = cv.c1 + cv.c2;
    const int HH = cv.up1 ? cv.H1 : cv.H, WW = cv.up1 ? cv.W1 : cv.W;
    const int r = threadIdx.x;
    int tap = k0 / cin, ch = k0 - tap * cin;   // of piece 0; pieces step 8 channels
#pragma unroll
    for (int kc = 0; kc < kBK / 8; ++kc) {
        const int gk = k0 + kc * 8;
        const __nv_bfloat16* g = s1;   // read nothing (source size 0)
        bool in = cr.valid && gk < K;
        if (in) {
            const int h = cr.y + tap / 3 - 1, w = cr.x + tap % 3 - 1;
            in = h >= 0 && h < cv.H && w >= 0 && w < cv.W;
            if (in) {
                if (ch < cv.c1) {
                    const int hh = cv.up1 ? h / 2 : h, ww = cv.up1 ? w / 2 : w;
                    g = s1 + (((size_t)cr.b * HH + hh) * WW + ww) * cv.c1 + ch;
                } else {
                    g = s2 + (((size_t)cr.b * cv.H + h) * cv.W + w) * cv.c2 + (ch - cv.c1);
                }
            }
        }
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(
                         smem_u32(dst + ((r >> 3) * 8 + kc) * 128 + (r & 7) * 16)),
                     "l"(g), "r"(in ? 16 : 0)
                     : "memory");
        ch += 8;
        if (ch >= cin) {
            ch -= cin;
            ++tap;
        }
    }
}

// The weight gradient's operands: the reduction runs over pixels (K), and both
// operands lie in memory with their M / N index contiguous (im2col values of a
// pixel, output channels of a pixel), so they are staged as they lie, 8 M (N)
// values of a pixel as one 16-byte piece, 8 pixels x 16 bytes a core matrix,
// and multiplied as MN-major operands: no im2col matrix, no transposed copies
// in memory.  With both (1.4 ms of passes over up to 265 MB a layer) a 64-input
// gradient took 5.35 ms on a GB300, gathered 4.03.
// A: im2col values [m0, m0 + 128) of pixels [k0, k0 + 64), zero past `M`, past
// pixel K and outside the image.  Core matrices: pixel group j, value group i
// at (16 j + i) * 128 bytes.
__device__ __forceinline__ void stage_conv_tile_mn(unsigned char* dst, const ConvGather& cv, int m0, int M, int k0,
                                                   int K)
{
    const __nv_bfloat16* s1 = static_cast<const __nv_bfloat16*>(cv.s1);
    const __nv_bfloat16* s2 = static_cast<const __nv_bfloat16*>(cv.s2);
    const int cin = cv.c1 + cv.c2, hw = cv.H * cv.W;
    const int HH = cv.up1 ? cv.H1 : cv.H, WW = cv.up1 ? cv.W1 : cv.W;
    // eight consecutive threads take eight pixels of one piece (128 contiguous
    // shared bytes); the next eight the next piece of the same pixels
    const int pr = threadIdx.x & 7, i0 = threadIdx.x >> 3;   // 16 piece columns
    const int k = m0 + 8 * i0;                               // this thread's im2col value of every pixel group
    const int tap = k / cin, ch = k - tap * cin;
    const int dh = tap / 3 - 1, dw = tap % 3 - 1;
    const bool first = ch < cv.c1;
#pragma unroll
    for (int j = 0; j < kBK / 8; ++j) {
        const int p = k0 + 8 * j + pr;
        const int b = p / hw, rr = p - b * hw, y = rr / cv.W, h = y + dh, w = rr - y * cv.W + dw;
        const bool in = k < M && p < K && h >= 0 && h < cv.H && w >= 0 && w < cv.W;
        const __nv_bfloat16* g = s1;   // read nothing (source size 0)
        if (in)
            g = first ? s1 + (((size_t)b * HH + (cv.up1 ? h / 2 : h)) * WW + (cv.up1 ? w / 2 : w)) * cv.c1 + ch
                      : s2 + (((size_t)b * cv.H + h) * cv.W + w) * cv.c2 + (ch - cv.c1);
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(
                         smem_u32(dst + (16 * j + i0) * 128 + pr * 16)),
                     "l"(g), "r"(in ? 16 : 0)
                     : "memory");
    }
}
// B: columns [n0, n0 + bn) of rows [k0, k0 + 64) of a row-major matrix.
__device__ __forceinline__ void stage_tile_mn(unsigned char* dst, const __nv_bfloat16* src, int ld, int n0, int bn,
                                              int N, int k0, int K)
{
    const int groups = bn / 8, pieces = groups * kBK;
    for (int c = threadIdx.x; c < pieces; c += kThreads) {
        const int pr = c & 7, i = (c >> 3) % groups, j = (c >> 3) / groups;
        const int p = k0 + 8 * j + pr, n = n0 + 8 * i;
        const bool in = p < K && n < N;
        const __nv_bfloat16* g = in ? src + (size_t)p * ld + n : src;
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(
                         smem_u32(dst + (groups * j + i) * 128 + pr * 16)),
                     "l"(g), "r"(in ? 16 : 0)
                     : "memory");
    }
}

// kWeightGrad: A and B as above (A = conv's im2col, B = dY, both MN-major).
template <bool kWeightGrad>
__global__ void __launch_bounds__(kThreads, 1) k_gemm_tc(GemmArgs a)
{
    extern __shared__ __align__(1024) unsigned char smem[];
    // stage i: A at smem + i * kStageA, B after all A stages
    auto sA = [&](int i) { return smem + i * kStageA; };
    const int stage_b = a.bn * kBK * 2;
    auto sB = [&](int i) { return smem + kStages * kStageA + i * stage_b; };
    uint64_t* mbar = reinterpret_cast<uint64_t*>(smem + kStages * (kStageA + stage_b));
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(mbar + kStages);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int m0 = blockIdx.x * kBM, n0 = blockIdx.y * a.bn;
    const int kbeg = blockIdx.z * a.k_per_split;
    const int kend = min(a.K, kbeg + a.k_per_split);
    const int nk = kend > kbeg ? (kend - kbeg + kBK - 1) / kBK : 0;

    if (threadIdx.x == 0) {
#pragma unroll
        for (int i = 0; i < kStages; ++i)
            asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_u32(&mbar[i])));
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)),
                     "r"(kTmemCols));
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
    }
    fence_before();
    __syncthreads();
    fence_after();
    const uint32_t tmem = *tmem_slot;
    const uint32_t idesc = instr_desc(a.bn) | (kWeightGrad ? 3u << 15 : 0u);   // bits 15, 16: A, B MN-major
    // K-major: 16 K values = two core matrices 128 bytes apart, 8-row groups
    // 1024 apart.  MN-major: two pixel groups a tile row of core matrices apart.
    const uint32_t lbo_a = kWeightGrad ? 2048u : 128u, sbo_a = kWeightGrad ? 128u : 1024u;
    const uint32_t lbo_b = kWeightGrad ? uint32_t(a.bn) * 16u : 128u, sbo_b = sbo_a;
    bool ok = true;

    const __nv_bfloat16* A = static_cast<const __nv_bfloat16*>(a.A);
    const ConvRow crow = !kWeightGrad && a.conv_a ? conv_row(a.conv, m0 + (int)threadIdx.x, a.M) : ConvRow{0, 0, 0, false};
    const __nv_bfloat16* B = static_cast<const __nv_bfloat16*>(a.B);
    auto stage = [&](int i, int k0) {
        if constexpr (kWeightGrad) {
            stage_conv_tile_mn(sA(i), a.conv, m0, a.M, k0, kend);
            stage_tile_mn(sB(i), B, a.ldb, n0, a.bn, a.N, k0, kend);
        } else {
            if (a.conv_a) stage_conv_tile(sA(i), a.conv, crow, k0, kend);
            else stage_tile(sA(i), A, a.lda, m0, kBM, a.M, k0, kend);
            stage_tile(sB(i), B, a.ldb, n0, a.bn, a.N, k0, kend);
        }
    };
    // prologue: chunks 0 .. kStages-2, one commit group each (empty past the end)
#pragma unroll
    for (int i = 0; i < kStages - 1; ++i) {
        if (i < nk) stage(i, kbeg + i * kBK);
        asm volatile("cp.async.commit_group;" ::: "memory");
    }
    for (int kc = 0; kc < nk; ++kc) {
        const int s = kc % kStages;
        // groups committed so far: kStages - 1 + kc; chunk kc's is complete when
        // at most kStages - 2 younger ones are pending
        asm volatile("cp.async.wait_group %0;" ::"n"(kStages - 2) : "memory");
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        __syncthreads();
        if (threadIdx.x == 0) {
            fence_after();
            const uint32_t abase = smem_u32(sA(s)), bbase = smem_u32(sB(s));
#pragma unroll
            for (int ks = 0; ks < kBK / 16; ++ks) {
                const uint64_t ad = smem_desc(abase + ks * 2 * lbo_a, lbo_a, sbo_a);
                const uint64_t bd = smem_desc(bbase + ks * 2 * lbo_b, lbo_b, sbo_b);
                const uint32_t acc = (kc > 0 || ks > 0) ? 1u : 0u;
                asm volatile(
                    "{\n\t.reg .pred p;\n\t"
                    "setp.ne.b32 p, %4, 0;\n\t"
                    "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}" ::"r"(tmem),
                    "l"(ad), "l"(bd), "r"(idesc), "r"(acc));
            }
            asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(
                             smem_u32(&mbar[s]))
                         : "memory");
        }
        // refill: chunk kc + kStages - 1 goes into the stage chunk kc - 1 used,
        // once that chunk's multiplies have completed
        const int nc = kc + kStages - 1;
        if (nc < nk) {
            const int ns = nc % kStages;
            if (kc >= 1) ok &= mbar_wait(smem_u32(&mbar[ns]), uint32_t(((kc - 1) / kStages) & 1));
            stage(ns, kbeg + nc * kBK);
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    }
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    if (nk > 0) ok &= mbar_wait(smem_u32(&mbar[(nk - 1) % kStages]), uint32_t(((nk - 1) / kStages) & 1));
    fence_after();

    // ---- epilogue: warp w holds rows 32w..32w+31 of the tile ----
    const int row = m0 + warp * 32 + lane;
    for (int c0 = 0; c0 < a.bn; c0 += 16) {
        uint32_t r[16];
        const uint32_t taddr = tmem + (uint32_t(warp * 32) << 16) + uint32_t(c0);
        asm volatile(
            "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, "
            "%14, %15}, [%16];"
            : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
              "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
            : "r"(taddr));
        asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
        if (row < a.M && nk > 0) {
            const int col0 = n0 + c0;
            float v[16];
#pragma unroll
            for (int j = 0; j < 16; ++j) {
                float x = __uint_as_float(r[j]);
                if (a.bias && col0 + j < a.N) x += a.bias[col0 + j];
                if (a.relu) x = fmaxf(x, 0.f);
                v[j] = x;
            }
            const bool whole = a.vec && col0 + 16 <= a.N;   // 16-byte stores
            if (a.out_bf16) {
                __nv_bfloat16* C = static_cast<__nv_bfloat16*>(a.C) + (size_t)row * a.ldc + col0;
                if (whole) {
                    uint4 q[2];
                    __nv_bfloat162* h = reinterpret_cast<__nv_bfloat162*>(q);
#pragma unroll
                    for (int j = 0; j < 8; ++j) h[j] = __floats2bfloat162_rn(v[2 * j], v[2 * j + 1]);
                    reinterpret_cast<uint4*>(C)[0] = q[0];
                    reinterpret_cast<uint4*>(C)[1] = q[1];
                } else {
#pragma unroll
                    for (int j = 0; j < 16; ++j)
                        if (col0 + j < a.N) C[j] = __float2bfloat16_rn(v[j]);
                }
            } else {
                float* C =
                    static_cast<float*>(a.C) + (size_t)blockIdx.z * a.split_stride + (size_t)row * a.ldc + col0;
                if (whole) {
#pragma unroll
                    for (int j = 0; j < 4; ++j)
                        reinterpret_cast<float4*>(C)[j] = make_float4(v[4 * j], v[4 * j + 1], v[4 * j + 2], v[4 * j + 3]);
                } else {
#pragma unroll
                    for (int j = 0; j < 16; ++j)
                        if (col0 + j < a.N) C[j] = v[j];
                }
            }
        }
        __syncwarp();
    }
    if (!ok && lane == 0 && a.status) atomicExch(a.status, kGemmTimeout);

    fence_before();
    __syncthreads();
    if (warp == 0) {
        fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(kTmemCols));
    }
}

// The input gradient of a 3x3 "same" convolution: d_in[q][c] = sum over taps of
// dY[q - off(tap)] . W^T[tap * cin + c], FP32 [P][cin].  A CTA owns 128 pixels;
// per kernel row of three taps it stages the shifted dY rows (zero outside the
// image) and the taps' weights, multiplies each tap into an accumulator of its
// own, and adds the three to the pixel's running sums in registers, tap by tap:
// the products and sums of a GEMM over all taps followed by the adjoint of
// im2col (col2im), bit for bit, without the [P][9 cin] FP32 matrix between
// them (0.53 GB for the widest layer of 64 inputs, written and read).  While
// the sums are formed the next three taps are staged.  Memory-bound: reads dY
// nine times from L2, writes [P][cin] once, as one bulk copy from shared memory.
// The eleven layers of a 64-input gradient: GEMM 0.90 + col2im 0.71 ms before.
constexpr int kTapGroup = 3;
constexpr uint32_t tmem_cols(int cols)
{
    return cols <= 32 ? 32u : cols <= 64 ? 64u : cols <= 128 ? 128u : cols <= 256 ? 256u : 512u;
}
constexpr int dgrad_smem(int cin, int co)
{
    const int stage = kTapGroup * (kBM + cin) * co * 2, out = kBM * cin * 4;
    return (stage > out ? stage : out) + 32;
}

struct DgradArgs {
    const __nv_bfloat16 *dy, *wt;   // [P][co]; [9 cin][co]
    float* out;                     // [P][cin]
    int P, H, W, co;
    unsigned* status;
};

template <int kCin>
__global__ void __launch_bounds__(kThreads) k_conv_dgrad(DgradArgs a)
{
    constexpr uint32_t kCols = tmem_cols(kTapGroup * kCin);
    extern __shared__ __align__(1024) unsigned char smem[];
    __shared__ __align__(8) uint64_t mbar;
    __shared__ uint32_t tmem_slot;
    const int t = threadIdx.x, warp = t >> 5;
    const int pieces = a.co / 8, tile_a = kBM * a.co * 2, tile_b = kCin * a.co * 2;
    unsigned char* sB = smem + kTapGroup * tile_a;
    const int m0 = blockIdx.x * kBM, q = m0 + t;   // this thread's pixel
    const int hw = a.H * a.W, rr = q % hw, h = rr / a.W, w = rr - h * a.W;

    if (t == 0) {
        asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_u32(&mbar)));
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_slot)),
                     "r"(kCols));
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
    }
    fence_before();
    __syncthreads();
    fence_after();
    const uint32_t tmem = tmem_slot;
    const uint32_t idesc = instr_desc(kCin);
    const uint32_t sbo = uint32_t(pieces) * 128u;

    // taps 3g .. 3g + 2 (kernel row g): core matrices of 8 rows x 16 bytes, the
    // pieces of 8 rows side by side
    auto stage = [&](int g) {
        const int ph = h - (g - 1);
        for (int x = 0; x < kTapGroup; ++x) {
            const int pw = w - (x - 1);
            const bool in = q < a.P && ph >= 0 && ph < a.H && pw >= 0 && pw < a.W;
            const __nv_bfloat16* src = in ? a.dy + (size_t)(q - (g - 1) * a.W - (x - 1)) * a.co : a.dy;
            unsigned char* dst = smem + x * tile_a + (t >> 3) * pieces * 128 + (t & 7) * 16;
            for (int kc = 0; kc < pieces; ++kc)
                asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(smem_u32(dst + kc * 128)),
                             "l"(in ? src + kc * 8 : src), "r"(in ? 16 : 0)
                             : "memory");
        }
        const __nv_bfloat16* wg = a.wt + (size_t)g * kTapGroup * kCin * a.co;
        for (int e = t; e < kTapGroup * kCin * pieces; e += kThreads) {
            const int r = e / pieces, kc = e - r * pieces, x = r / kCin, c = r - x * kCin;
            asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(
                             smem_u32(sB + x * tile_b + ((c >> 3) * pieces + kc) * 128 + (c & 7) * 16)),
                         "l"(wg + (size_t)r * a.co + kc * 8)
                         : "memory");
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };

    float acc[kCin];
#pragma unroll
    for (int c = 0; c < kCin; ++c) acc[c] = 0.f;
    bool ok = true;
    stage(0);
    for (int g = 0; g < 3; ++g) {
        asm volatile("cp.async.wait_group 0;" ::: "memory");
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        fence_before();   // the previous group's accumulator reads before they are overwritten
        __syncthreads();
        if (t == 0) {
            fence_after();
            for (int x = 0; x < kTapGroup; ++x)
                for (int ks = 0; ks < a.co / 16; ++ks) {
                    const uint64_t ad = smem_desc(smem_u32(smem + x * tile_a) + ks * 256, 128, sbo);
                    const uint64_t bd = smem_desc(smem_u32(sB + x * tile_b) + ks * 256, 128, sbo);
                    asm volatile(
                        "{\n\t.reg .pred p;\n\t"
                        "setp.ne.b32 p, %4, 0;\n\t"
                        "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}" ::"r"(tmem + uint32_t(x * kCin)),
                        "l"(ad), "l"(bd), "r"(idesc), "r"(ks > 0 ? 1u : 0u));
                }
            asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(
                             smem_u32(&mbar))
                         : "memory");
        }
        ok &= mbar_wait(smem_u32(&mbar), uint32_t(g & 1));
        fence_after();
        if (g < 2) stage(g + 1);   // the multiplies have read this group's operands
#pragma unroll
        for (int c0 = 0; c0 < kCin; c0 += 16)
#pragma unroll
            for (int x = 0; x < kTapGroup; ++x) {
                uint32_t r[16];
                const uint32_t taddr = tmem + (uint32_t(warp * 32) << 16) + uint32_t(x * kCin + c0);
                asm volatile(
                    "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, "
                    "%13, %14, %15}, [%16];"
                    : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
                      "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]),
                      "=r"(r[15])
                    : "r"(taddr));
                asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
                for (int j = 0; j < 16; ++j) acc[c0 + j] = __fadd_rn(acc[c0 + j], __uint_as_float(r[j]));
            }
    }
    // the tile's rows are contiguous in out: one copy from shared memory (the
    // last multiplies have read the operands it overwrites)
    float* so = reinterpret_cast<float*>(smem) + (size_t)t * kCin;
#pragma unroll
    for (int c = 0; c < kCin; c += 4)
        *reinterpret_cast<float4*>(so + c) = make_float4(acc[c], acc[c + 1], acc[c + 2], acc[c + 3]);
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    fence_before();
    __syncthreads();
    if (t == 0) {
        const int rows = min(kBM, a.P - m0);
        asm volatile("cp.async.bulk.global.shared::cta.bulk_group [%0], [%1], %2;" ::"l"(a.out + (size_t)m0 * kCin),
                     "r"(smem_u32(smem)), "r"(rows * kCin * 4)
                     : "memory");
        asm volatile("cp.async.bulk.commit_group;" ::: "memory");
        asm volatile("cp.async.bulk.wait_group 0;" ::: "memory");
    }
    if (!ok && (t & 31) == 0 && a.status) atomicExch(a.status, kGemmTimeout);
    if (warp == 0) {
        fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(kCols));
    }
}

// Sums split-K partials [splits][M][ldc] into out: [M][ldc], or, with `ldt`,
// its transpose [N][ldt].  Bound by the partials' latency (a value has up to
// 608 of them): eight threads a value add an eighth each in order, with 16
// loads in flight, then the eighths are added in order.
// The blocks after the first `blocks` add the bias gradients' partials, a
// channel's by 16 interleaved sums (two a thread) and a fixed tree: as a launch of
// its own that took 6 us a layer (64 inputs' gradients 2.120 ms, as part of this one 2.065).
constexpr int kSumGroups = 8;
__global__ void __launch_bounds__(32 * kSumGroups) k_splitk_sum(const float* __restrict__ part, int splits,
                                                               size_t stride, int M, int N, int ldc,
                                                               float* __restrict__ out, int ldt, unsigned blocks,
                                                               BiasSum bias)
{
    __shared__ float red[2 * kSumGroups][33];
    if (blockIdx.x >= blocks) {
        const int c = (int)(blockIdx.x - blocks) * 32 + (int)threadIdx.x;
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            float s = 0.f;
            if (c < bias.C)
                for (int b = (int)threadIdx.y + h * kSumGroups; b < bias.nblocks; b += 2 * kSumGroups)
                    s += bias.part[(size_t)b * bias.C + c];
            red[threadIdx.y + h * kSumGroups][threadIdx.x] = s;
        }
        for (int w = kSumGroups; w > 0; w >>= 1) {
            __syncthreads();
            if ((int)threadIdx.y < w) red[threadIdx.y][threadIdx.x] += red[threadIdx.y + w][threadIdx.x];
        }
        if (threadIdx.y == 0 && c < bias.cout) bias.out[c] = red[0][threadIdx.x];
        return;
    }
    const size_t i = (size_t)blockIdx.x * 32 + threadIdx.x;
    const bool in = i < (size_t)M * N;
    const size_t r = in ? i / N : 0, c = in ? i % N : 0;
    const float* q = part + r * ldc + c;
    const int each = (splits + kSumGroups - 1) / kSumGroups;
    int z = threadIdx.y * each;
    const int end = min(splits, z + each);
    float s = 0.f;
    for (; z + 16 <= end; z += 16) {
        float v[16];
#pragma unroll
        for (int j = 0; j < 16; ++j) v[j] = q[(z + j) * stride];
#pragma unroll
        for (int j = 0; j < 16; ++j) s += v[j];
    }
    for (; z < end; ++z) s += q[z * stride];
    red[threadIdx.y][threadIdx.x] = s;
    __syncthreads();
    if (threadIdx.y != 0 || !in) return;
#pragma unroll
    for (int g = 1; g < kSumGroups; ++g) s += red[g][threadIdx.x];
    out[ldt ? c * ldt + r : r * ldc + c] = s;
}

}  // namespace

// The input channel counts of the network's convolutions.
#define PDFLOW_DGRAD_CINS(X) X(16) X(32) X(48) X(64) X(96) X(160)

static cudaError_t prepare_conv_dgrad()
{
    cudaError_t e = cudaSuccess;
#define X(c)                                                                                                   \
    if (e == cudaSuccess)                                                                                      \
        e = cudaFuncSetAttribute(k_conv_dgrad<c>, cudaFuncAttributeMaxDynamicSharedMemorySize, dgrad_smem(c, 96));
    PDFLOW_DGRAD_CINS(X)
#undef X
    return e;
}

cudaError_t prepare_gemm_tc()
{
    cudaError_t e = cudaFuncSetAttribute(k_gemm_tc<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmemBytes);
    if (e == cudaSuccess)
        e = cudaFuncSetAttribute(k_gemm_tc<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmemBytes);
    if (e == cudaSuccess) e = prepare_conv_dgrad();
    return e;
}

cudaError_t launch_conv_dgrad(const void* dy, const void* wt, int P, int H, int W, int cin, int co, float* out,
                              unsigned* status, cudaStream_t st)
{
    if (P <= 0 || co < 16 || co > 96 || co % 16 != 0 || reinterpret_cast<uintptr_t>(out) % 16u != 0)
        return cudaErrorInvalidValue;
    const DgradArgs a{static_cast<const __nv_bfloat16*>(dy), static_cast<const __nv_bfloat16*>(wt), out, P, H, W, co,
                      status};
    const unsigned grid = unsigned((P + kBM - 1) / kBM);
    switch (cin) {
#define X(c)                                                                   \
    case c:                                                                    \
        k_conv_dgrad<c><<<grid, kThreads, dgrad_smem(c, co), st>>>(a);         \
        break;
        PDFLOW_DGRAD_CINS(X)
#undef X
        default:
            return cudaErrorInvalidValue;
    }
    return cudaGetLastError();
}

cudaError_t launch_gemm_tc(const GemmArgs& args, cudaStream_t st)
{
    GemmArgs a = args;
    // the weight gradient's K (pixels) and leading dimensions have their own
    // rules: 16-byte pieces along M and N, any number of pixels
    if (a.bn < 16 || a.bn > kMaxBN || (a.bn & 15) || (a.ldb & 7) || a.M <= 0 || a.N <= 0 || a.K <= 0 ||
        (a.weight_grad ? !a.conv_a || (a.M & 7) || (a.N & 7) : (a.K & 7) || (a.lda & 7)))
        return cudaErrorInvalidValue;
    if (a.k_per_split <= 0) a.k_per_split = a.K;
    // the epilogue's 16-byte stores: every row and split starts on one
    const int unit = a.out_bf16 ? 8 : 4;
    a.vec = reinterpret_cast<uintptr_t>(a.C) % 16u == 0 && a.ldc % unit == 0 && a.split_stride % unit == 0;
    a.k_per_split = (a.k_per_split + kBK - 1) / kBK * kBK;
    const unsigned splits = (unsigned)((a.K + a.k_per_split - 1) / a.k_per_split);
    if (splits > 1 && a.out_bf16) return cudaErrorInvalidValue;
    dim3 grid((a.M + kBM - 1) / kBM, (a.N + a.bn - 1) / a.bn, splits);
    if (a.weight_grad) k_gemm_tc<true><<<grid, kThreads, smem_bytes(a.bn), st>>>(a);
    else k_gemm_tc<false><<<grid, kThreads, smem_bytes(a.bn), st>>>(a);
    return cudaGetLastError();
}

unsigned gemm_splits(int K, int k_per_split)
{
    const int kp = (k_per_split + kBK - 1) / kBK * kBK;
    return (unsigned)((K + kp - 1) / kp);
}

cudaError_t launch_splitk_sum(const float* part, int splits, size_t stride, int M, int N, int ldc, float* out,
                              cudaStream_t st, int ldt, BiasSum bias)
{
    const unsigned blocks = unsigned(((size_t)M * N + 31) / 32);
    const unsigned more = bias.part ? unsigned((bias.C + 31) / 32) : 0u;
    k_splitk_sum<<<blocks + more, dim3(32, kSumGroups), 0, st>>>(part, splits, stride, M, N, ldc, out, ldt, blocks, bias);
    return cudaGetLastError();
}

}  // namespace pdflow
