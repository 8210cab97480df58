// Stage kernels of the PD-Flow solver on sm_103a.
//
// One thread per pixel, column-major planes (idx = v + u*R, rows contiguous,
// so a warp reads 32 consecutive rows of one column: coalesced).  The image
// gradients of all levels are one kernel, a level's set-up two (starting point
// and connectivity; warping and step sizes), an iteration is two kernels
// (gradient+dual, divergence+primal; the reference uses four) and the last
// primal kernel of a level also saturates; the weighted median and the motion
// field are one kernel.  All per-pixel arithmetic lives in pdflow_math.cuh.
#include <algorithm>

#include "pdflow_kernels.cuh"
#include "pdflow_math.cuh"

namespace pdflow {

namespace {

constexpr unsigned kBlock = 256;

__host__ __device__ inline unsigned blocks_for(unsigned n) { return (n + kBlock - 1) / kBlock; }

// ---------------------------------------------------------------------------
// Pyramid (computePyramidLevel, pdflow_cudalib.cu:331-434)
// ---------------------------------------------------------------------------

// One pixel (v, u) of an R x C level from the level above it: the depth-weighted
// 5x5 mask; above(k, l) is (intensity, depth) of the level above at row 2v + k,
// column 2u + l.  sumc and sumd fuse their products; the depth weight is added after
// rounding (acu_weights_d += aux_w), as in the reference build.
template <class Above>
__device__ __forceinline__ float2 down_px(unsigned v, unsigned u, unsigned R, unsigned C, Above above)
{
    const float max_depth_dif = 0.1f;
    const float dcenter = above(0, 0).y;
    float sumd = 0.f, sumc = 0.f, acu_weights_d = 0.f, acu_weights_c = 0.f;
    auto depth_tap = [&](float gm, float d) {
        const float ad = fabsf(sub(d, dcenter));
        if ((d > 0.f) && (ad < max_depth_dif)) {
            const float aux_w = mul(gm, sub(max_depth_dif, ad));
            acu_weights_d = add(acu_weights_d, aux_w);
            sumd = fm(aux_w, d, sumd);
        }
    };
    float cres;
    if ((v > 0) && (v < R - 1) && (u > 0) && (u < C - 1)) {
#pragma unroll
        for (int k = -2; k < 3; k++)
#pragma unroll
            for (int l = -2; l < 3; l++) {
                const float gm = gmask(k, l);
                const float2 x = above(k, l);
                sumc = fm(gm, x.x, sumc);
                depth_tap(gm, x.y);
            }
        cres = sumc;
    } else {
        for (int k = -2; k < 3; k++)
            for (int l = -2; l < 3; l++) {
                const int indv = 2 * (int)v + k, indu = 2 * (int)u + l;
                if ((indv >= 0) && (indv < 2 * (int)R) && (indu >= 0) && (indu < 2 * (int)C)) {
                    const float gm = gmask(k, l);
                    const float2 x = above(k, l);
                    sumc = fm(gm, x.x, sumc);
                    acu_weights_c = add(acu_weights_c, gm);
                    depth_tap(gm, x.y);
                }
            }
        cres = qt(sumc, acu_weights_c);
    }
    return make_float2(cres, (sumd > 0.f) ? qt(sumd, acu_weights_d) : 0.f);
}

__device__ __forceinline__ void put_px(const PyrLevel& out, unsigned R, unsigned C, unsigned v, unsigned u, float2 cz,
                                       float inv_f_i)
{
    const unsigned idx = v + u * R;
    out.col[idx] = cz.x;
    out.dep[idx] = cz.y;
    out.xx[idx] = backproject(u, C, cz.y, inv_f_i);
    out.yy[idx] = backproject(v, R, cz.y, inv_f_i);
}

// Where a pyramid starts: (intensity, metres) of pixel (row v, column u).
// Row-major camera images ([pair][H][W]) are read along their rows, column-major
// planes along their columns.
struct SourceU16 {   // uint8 intensity, uint16 depth
    static constexpr bool kRowMajor = true;
    const uint8_t* img;
    const uint16_t* depth;
    unsigned W, H;
    __device__ __forceinline__ void pair(unsigned z, size_t)
    {
        img += (size_t)z * W * H;
        depth += (size_t)z * W * H;
    }
    __device__ __forceinline__ float2 at(unsigned v, unsigned u) const
    {
        const size_t i = (size_t)v * W + u;
        return make_float2(float(img[i]), decode_depth(depth[i]));
    }
};
// RGB888 + millimetre depth with the live application's conversion (gray_rgb,
// decode_depth_mm).  rotate180: its camera loop
// (scene_flow_visualization.cpp:313-323) stores camera pixel (y, x) at row
// H-1-y, column W-1-x.
struct SourceRgb {
    static constexpr bool kRowMajor = true;
    const uint8_t* rgb;
    const uint16_t* depth;
    unsigned W, H;
    int rotate180;
    __device__ __forceinline__ void pair(unsigned z, size_t)
    {
        rgb += (size_t)z * W * H * 3;
        depth += (size_t)z * W * H;
    }
    __device__ __forceinline__ float2 at(unsigned v, unsigned u) const
    {
        const size_t i = rotate180 ? (size_t)(H - 1 - v) * W + (W - 1 - u) : (size_t)v * W + u;
        return make_float2(gray_rgb(rgb[3 * i], rgb[3 * i + 1], rgb[3 * i + 2]), decode_depth_mm(depth[i]));
    }
};
struct SourcePlanes {   // column-major float planes of the pair's arena slice
    static constexpr bool kRowMajor = false;
    const float *col, *dep;
    unsigned W, H;
    __device__ __forceinline__ void pair(unsigned, size_t po)
    {
        col = pdflow::at(col, po);
        dep = pdflow::at(dep, po);
    }
    __device__ __forceinline__ float2 at(unsigned v, unsigned u) const
    {
        const size_t i = v + (size_t)u * H;
        return make_float2(col[i], dep[i]);
    }
};

// A frame's 32 x 32 tile through three pyramid levels in one pass: the source
// (levels + 0, W x H) is read once with a halo of 6 into shared memory, written
// as the first level where kWriteFirst, reduced to the tile's 16 x 16 of the
// second level with a halo of 2 (the halo pixels are the neighbours', computed
// again) and to its 8 x 8 of the third (count 2: stop at the second).  Bound by
// shared-memory reads and instruction issue of the 25 taps on a batch, by launch
// latency for one frame.  Against a launch a level, two pushes on a GB300: one 320x240
// frame 71 -> 34 us, one 640x480 89 -> 52, 64 716 -> 428.
constexpr int kPyrTile = 32, kPyrHalo = 6, kPyrSide = kPyrTile + 2 * kPyrHalo, kPyrMid = kPyrTile / 2 + 4;

// A tile's (intensity, depth) pixels, a column's even rows before its odd ones:
// the taps of consecutive pixels of the next level, two rows apart, are then
// consecutive in shared memory.
template <int kSide>
struct PyrTile {
    float2 px[kSide][kSide + 1];
    static __device__ __forceinline__ int slot(int row) { return (row & 1) * (kSide / 2) + (row >> 1); }
    __device__ __forceinline__ float2& operator()(int col, int row) { return px[col][slot(row)]; }
    // the tap k rows, l columns from (col, 2 half) of the next level's pixel
    __device__ __forceinline__ float2 tap(int col, int half, int k, int l) const
    {
        return px[col + l][(k & 1) * (kSide / 2) + half + (k >> 1)];
    }
};

template <class Source, bool kWriteFirst, unsigned kThreads>
__global__ void __launch_bounds__(kThreads) k_pyramid(Source src, PyrLevel l0, PyrLevel l1, PyrLevel l2, int count,
                                                        float fovh, size_t pstride, const unsigned* __restrict__ map)
{
    __shared__ PyrTile<kPyrSide> t0;
    __shared__ PyrTile<kPyrMid> t1;
    __shared__ float inv[3];   // the levels' focal factors (a tanf and a division each: once a tile)
    if (threadIdx.x < 3) inv[threadIdx.x] = inv_focal(fovh, src.W >> threadIdx.x);
    after_previous_kernel();   // the pass before writes this one's source
    allow_next_kernel();
    const size_t po = pair_off(map, pstride, blockIdx.z);
    src.pair(blockIdx.z, po);
    l1 = at(l1, po);
    const int W = (int)src.W, H = (int)src.H;
    const int U0 = (int)blockIdx.x * kPyrTile, V0 = (int)blockIdx.y * kPyrTile;
    // a warp a row (row-major sources) or a column of the tile and its halo (of
    // which two levels need 2 pixels)
    const int skip = count > 2 ? 0 : kPyrHalo - 2;
    for (int slow = skip + threadIdx.x / 32; slow < kPyrSide - skip; slow += kThreads / 32)
#pragma unroll
        for (int q = 0; q < 2; ++q) {
            const int fast = skip + q * 32 + (int)(threadIdx.x & 31);
            const int i = Source::kRowMajor ? fast : slow, j = Source::kRowMajor ? slow : fast;   // column, row
            const int u = U0 - kPyrHalo + i, v = V0 - kPyrHalo + j;
            if (fast < kPyrSide - skip && u >= 0 && u < W && v >= 0 && v < H) t0(i, j) = src.at((unsigned)v, (unsigned)u);
        }
    __syncthreads();
    if constexpr (kWriteFirst) {
        l0 = at(l0, po);
        for (int e = threadIdx.x; e < kPyrTile * kPyrTile; e += kThreads) {
            const int j = e % kPyrTile, i = e / kPyrTile, u = U0 + i, v = V0 + j;
            if (u < W && v < H)
                put_px(l0, H, W, v, u, t0(kPyrHalo + i, kPyrHalo + j), inv[0]);
        }
    }
    const int R1 = H / 2, C1 = W / 2, V1 = V0 / 2, U1 = U0 / 2;
    const int halo1 = count > 2 ? 2 : 0, side1 = kPyrTile / 2 + 2 * halo1;
    for (int e = threadIdx.x; e < side1 * side1; e += kThreads) {
        const int j = e % side1, i = e / side1, u = U1 - halo1 + i, v = V1 - halo1 + j;
        if (u < 0 || u >= C1 || v < 0 || v >= R1) continue;
        const int col = 2 * (i - halo1) + kPyrHalo, half = j - halo1 + kPyrHalo / 2;   // (2u, 2v) in t0
        const float2 x = down_px(v, u, R1, C1, [&](int k, int l) { return t0.tap(col, half, k, l); });
        if (i >= halo1 && i < halo1 + kPyrTile / 2 && j >= halo1 && j < halo1 + kPyrTile / 2)
            put_px(l1, R1, C1, v, u, x, inv[1]);
        if (count > 2) t1(i, j) = x;
    }
    if (count < 3) return;
    __syncthreads();
    l2 = at(l2, po);
    const int R2 = H / 4, C2 = W / 4;
    for (int e = threadIdx.x; e < kPyrTile / 4 * (kPyrTile / 4); e += kThreads) {
        const int j = e % (kPyrTile / 4), i = e / (kPyrTile / 4), u = U0 / 4 + i, v = V0 / 4 + j;
        if (u >= C2 || v >= R2) continue;
        put_px(l2, R2, C2, v, u,
               down_px(v, u, R2, C2, [&](int k, int l) { return t1.tap(2 * i + 2, j + 1, k, l); }), inv[2]);
    }
}

// A small result to pinned host memory in one launch, with the status word: bound
// by one trip over the chip-to-chip link, 16 bytes a thread (a 60x80 flow with the
// host's part 21 us, against 40 of four copies to pageable memory).
__global__ void k_flow_out(const float* __restrict__ dx, const float* __restrict__ dy, const float* __restrict__ dz,
                           size_t step, unsigned n4, const unsigned* status, float4* __restrict__ out,
                           unsigned* out_status)
{
    const unsigned i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i == 0 && blockIdx.y == 0 && blockIdx.z == 0) *out_status = *status;
    if (i >= n4) return;
    const float* src = blockIdx.y == 0 ? dx : blockIdx.y == 1 ? dy : dz;
    out[(size_t(blockIdx.y) * gridDim.z + blockIdx.z) * n4 + i] =
        reinterpret_cast<const float4*>(at(src, blockIdx.z * step))[i];
}

// ---------------------------------------------------------------------------
// Level set-up
// ---------------------------------------------------------------------------

// Connectivity weight (computeRij, pdflow_cudalib.cu:725-779) of the step from
// pixel i to i + d of back-projected coordinate x and depth z.
__device__ __forceinline__ float rij(const float* __restrict__ x, const float* __restrict__ z, unsigned i, unsigned d)
{
    return rfac(sub(x[i + d], x[i]), sub(z[i + d], z[i]));
}

// computeImGradients (pdflow_cudalib.cu:574-627) on the new frame, for every
// level of a solve in one launch: it needs the pyramid only, so it is off the
// path from one level's solution to the next level's iterations.  The new
// frame's weights (ri_2, rj_2) at the pixel, left of and above it are formed
// here instead of being stored and read back (16 VGA pairs: 0.088 ms for all
// six levels against 0.117 a launch a level, besides those planes' writes).
struct GradLevels {
    PyrLevel n[8];
    unsigned R[8], C[8], first_block[9];   // 256 pixels a block
    size_t aux[8];                         // the level's floats in the aux planes
    unsigned count;
};
__global__ void k_im_gradients(const __grid_constant__ GradLevels lv, LevelConsts L, size_t pstride,
                               const unsigned* __restrict__ map)
{
    allow_next_kernel();   // no wait before it: an ordinary launch, all before it has ended
    unsigned q = 0;
    while (q + 1 < lv.count && blockIdx.x >= lv.first_block[q + 1]) ++q;
    const size_t po = pair_off(map, pstride, blockIdx.y);
    const PyrLevel n = at(lv.n[q], po);
    L = at(L, po);
    const unsigned index = (blockIdx.x - lv.first_block[q]) * blockDim.x + threadIdx.x;
    const unsigned R = lv.R[q], C = lv.C[q];
    if (index >= R * C) return;
    const unsigned v = index % R, u = index / R;
    const size_t out = lv.aux[q] + index;
    const float* __restrict__ c = n.col;
    const float* __restrict__ d = n.dep;
    if (u == 0) {
        L.dcu_aux[out] = sub(c[index + R], c[index]);
        L.ddu_aux[out] = sub(d[index + R], d[index]);
    } else if (u == C - 1) {
        L.dcu_aux[out] = sub(c[index], c[index - R]);
        L.ddu_aux[out] = sub(d[index], d[index - R]);
    } else {
        const float r = rij(n.xx, d, index, R), rm = rij(n.xx, d, index - R, R);
        L.dcu_aux[out] = wgrad(r, rm, c[index + R], c[index], c[index - R]);
        L.ddu_aux[out] = (d[index] > 0.f) ? wgrad(r, rm, d[index + R], d[index], d[index - R]) : 0.f;
    }
    if (v == 0) {
        L.dcv_aux[out] = sub(c[index + 1], c[index]);
        L.ddv_aux[out] = sub(d[index + 1], d[index]);
    } else if (v == R - 1) {
        L.dcv_aux[out] = sub(c[index], c[index - 1]);
        L.ddv_aux[out] = sub(d[index], d[index - 1]);
    } else {
        const float r = rij(n.yy, d, index, 1), rm = rij(n.yy, d, index - 1, 1);
        L.dcv_aux[out] = wgrad(r, rm, c[index + 1], c[index], c[index - 1]);
        L.ddv_aux[out] = (d[index] > 0.f) ? wgrad(r, rm, d[index + 1], d[index], d[index - 1]) : 0.f;
    }
}

// performWarping (pdflow_cudalib.cu:629-652) at one pixel: both frames at (u +
// du, v + dv); aux: the level's offset in the gradient planes.
struct Warped {
    float dct, dcu, dcv, ddt, ddu, ddv;
};
__device__ __forceinline__ Warped warp_px(const PyrLevel& o, const PyrLevel& n, const LevelConsts& L, size_t aux,
                                          unsigned R, unsigned C, unsigned v, unsigned u, float du, float dv)
{
    const unsigned index = v + u * R;
    // the five plain interpolations at one position share their case analysis
    const Bilin b = bilin(R, C, add(float(u), du), add(float(v), dv));
    const float* const mats[5] = {n.col, L.dcu_aux + aux, L.dcv_aux + aux, L.ddu_aux + aux, L.ddv_aux + aux};
    float w5[5];
    bilin_blend_n<5>(mats, R, b, w5);
    const float wz = interp_depth_at(n.dep, R, b);
    return {sub(w5[0], o.col[index]), w5[1], w5[2], (wz > 0.f) ? sub(wz, o.dep[index]) : 0.f, w5[3], w5[4]};
}

// upsampleCopy + upsampleFilterPrevSolution (pdflow_cudalib.cu:460-569) of one
// coarse plane at a vertical pixel pair (rows 2a, 2a+1 of column u), as a
// gather over the coarse solution (the zero-inserted taps contribute exactly
// zero and are skipped): the even row's taps with a coarse sample are rows -2,
// 0, +2 and the odd row's -1, +1, and the column's parity fixes the columns
// (-2, 0, +2 or -1, +1), so both pixels read the same 3 x 3 (or 3 x 2) coarse
// neighbourhood and accumulate their taps in the reference's order (row, then
// column).  Bit r * 3 + e of `in`: the sample lies inside the level.
template <int kColTaps>
__device__ __forceinline__ float2 upsample_pair(const float* __restrict__ plane, const int (&at)[9], unsigned in,
                                                float scale)
{
    float c[3][kColTaps];
#pragma unroll
    for (int r = 0; r < 3; ++r)
#pragma unroll
        for (int e = 0; e < kColTaps; ++e) c[r][e] = (in >> (r * 3 + e)) & 1u ? mul(scale, plane[at[r * 3 + e]]) : 0.f;
    constexpr int l0 = kColTaps == 3 ? -2 : -1;
    float x0 = 0.f, x1 = 0.f;
#pragma unroll
    for (int r = 0; r < 3; ++r)   // even row: row taps -2, 0, +2 = coarse rows a-1, a, a+1
#pragma unroll
        for (int e = 0; e < kColTaps; ++e)
            if ((in >> (r * 3 + e)) & 1u) x0 = fm(mul(4.f, gmask(2 * r - 2, 2 * e + l0)), c[r][e], x0);
#pragma unroll
    for (int r = 1; r < 3; ++r)   // odd row: row taps -1, +1 = coarse rows a, a+1
#pragma unroll
        for (int e = 0; e < kColTaps; ++e)
            if ((in >> (r * 3 + e)) & 1u) x1 = fm(mul(4.f, gmask(2 * r - 3, 2 * e + l0)), c[r][e], x1);
    return make_float2(x0, x1);
}

// The mask's weight inside the image along one axis, in sixteenths: 16 less
// the taps of pixel x beyond [0, n).
__device__ __forceinline__ int mask_inside(int x, int n)
{
    return 16 - (x < 1 ? 5 : x < 2 ? 1 : 0) - (x > n - 2 ? 5 : x > n - 3 ? 1 : 0);
}

// A level's starting point: assignZeros / the upsampled solution
// (pdflow_cudalib.cu:439-569) and computeRij of the old frame (:725-779).  kPx
// pixels of a column per thread (2: rows 2a, 2a+1, stored as float2; 1: the
// coarsest level, whose rows are odd).
// start 0: zeros; 1: a predicted flow, duals from zero; 2: the coarse solution.
// Bound by instruction issue on a batch, by latency on one pair's small levels.
// One kernel with the warp below (the flow and weights in registers between
// them) needs 95 registers a thread and 0.57 ms for 16 pairs at 480x640 where
// the two take 0.33, and gains nothing on the small levels.
template <int kPx>
__global__ void __launch_bounds__(kBlock) k_level_start(LevelGeom g, int start, LevelSol cs, PyrLevel o,
                                                        LevelConsts L, State S, const float* seed)
{
    const size_t po = pair_off(g.map, g.pstride, blockIdx.y);
    cs = at(cs, po);
    o = at(o, po);
    L = at(L, po);
    S = at(S, po);
    const unsigned R = g.R, C = g.C, rows = R / kPx;
    const unsigned t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= rows * C) return;
    const unsigned a = t % rows, u = t / rows, v0 = kPx * a, index = v0 + u * R;
    // the old frame's weights need the pyramid only: formed while the kernel before ends
    float2 ri = make_float2(1.f, 1.f), rj = make_float2(1.f, 1.f);   // rfac(0, 0) at the far borders
    if (u != C - 1) {
        ri.x = rij(o.xx, o.dep, index, R);
        if (kPx == 2) ri.y = rij(o.xx, o.dep, index + 1, R);
    }
    if (v0 != R - 1) rj.x = rij(o.yy, o.dep, index, 1);
    if (kPx == 2 && v0 + 1 != R - 1) rj.y = rij(o.yy, o.dep, index + 1, 1);
    after_previous_kernel();
    allow_next_kernel();
    auto put = [&](float* plane, float2 x) {
        if constexpr (kPx == 2) *reinterpret_cast<float2*>(plane + index) = x;
        else plane[index] = x.x;
    };
    const float2 zero = make_float2(0.f, 0.f);
    float2 du = zero, dv = zero, dw = zero;
    float* const duals[7] = {S.pd, S.puu, S.puv, S.pvu, S.pvv, S.pwu, S.pwv};
    if (kPx == 2 && start == 2) {
        const int Rc = int(R / 2), Cc = int(C / 2), b = int(u >> 1), ca = int(a);
        const bool odd = u & 1u;
        int from[9];
        unsigned in = 0;
#pragma unroll
        for (int r = 0; r < 3; ++r)
#pragma unroll
            for (int e = 0; e < 3; ++e) {
                const int row = ca - 1 + r, col = odd ? b + e : b - 1 + e;
                from[r * 3 + e] = row + col * Rc;
                if (row >= 0 && row < Rc && col >= 0 && col < Cc) in |= 1u << (r * 3 + e);
            }
        // beyond the image's inner part the sum is divided by the mask's weight
        // inside the image, a multiple of 1/256 (elsewhere the factor is 1)
        const int wu = mask_inside(int(u), int(C));
        const float i0 = fdividef(1.f, float(mask_inside(int(v0), int(R)) * wu) / 256.f);
        const float i1 = fdividef(1.f, float(mask_inside(int(v0) + 1, int(R)) * wu) / 256.f);
        const bool inner = v0 > 1 && v0 + 1 < R - 2 && u > 1 && u < C - 2;
        auto up = [&](const float* plane, float scale) {
            float2 x = odd ? upsample_pair<2>(plane, from, in, scale) : upsample_pair<3>(plane, from, in, scale);
            if (!inner) x = make_float2(mul(x.x, i0), mul(x.y, i1));
            return x;
        };
        du = up(cs.du, 2.f);
        dv = up(cs.dv, 2.f);
        dw = up(cs.dw, 1.f);
        const float* const coarse[7] = {cs.pd, cs.puu, cs.puv, cs.pvu, cs.pvv, cs.pwu, cs.pwv};
#pragma unroll
        for (int q = 0; q < 7; ++q) put(duals[q], up(coarse[q], 1.f));
    } else {
        if (start == 1) {
            const float* sp = seed + (size_t)blockIdx.y * 3 * g.N + index;
            du = make_float2(sp[0], kPx == 2 ? sp[1] : 0.f);
            dv = make_float2(sp[g.N], kPx == 2 ? sp[g.N + 1] : 0.f);
            dw = make_float2(sp[2 * g.N], kPx == 2 ? sp[2 * g.N + 1] : 0.f);
        }
#pragma unroll
        for (int q = 0; q < 7; ++q) put(duals[q], zero);
    }
    put(L.du_prev, du);
    put(L.dv_prev, dv);
    put(S.du, zero);
    put(S.dv, zero);
    put(S.dua, zero);
    put(S.dva, zero);
    put(S.dw, dw);
    put(S.dwa, dw);
    put(L.ri, ri);
    put(L.rj, rj);
}

// performWarping (pdflow_cudalib.cu:629-652) + computeMu/computeStepSizes
// (:781-808), from the planes k_level_start wrote.  steps: which step-size
// planes to write (kStepsNone: only mu, the tile kernels recompute the step
// sizes from mu, ri, rj, ddu, ddv; there and beside the quad products the free
// spd plane holds powf(ddt, 2) for the level's median, so each pixel's square is
// taken once instead of once per neighbour).
__global__ void __launch_bounds__(kBlock) k_level_warp(LevelGeom g, PyrLevel o, PyrLevel n, LevelConsts L, Params p,
                                                       int steps, size_t aux)
{
    const size_t po = pair_off(g.map, g.pstride, blockIdx.y);
    o = at(o, po);
    n = at(n, po);
    L = at(L, po);
    const unsigned index = blockIdx.x * blockDim.x + threadIdx.x;
    if (index >= g.N) return;
    const unsigned R = g.R, C = g.C;
    const unsigned v = index % R, u = index / R;
    after_previous_kernel();
    allow_next_kernel();
    const Warped w = warp_px(o, n, L, aux, R, C, v, u, L.du_prev[index], L.dv_prev[index]);
    L.dct[index] = w.dct;
    L.dcu[index] = w.dcu;
    L.dcv[index] = w.dcv;
    L.ddt[index] = w.ddt;
    L.ddu[index] = w.ddu;
    L.ddv[index] = w.ddv;
    if (steps == kStepsNone || steps == kStepsQuads) L.spd[index] = powf(w.ddt, 2.f);   // the median's weight
    if (steps == kStepsNone) {
        L.mu[index] = data_weight(p.mu, w.ddu, w.ddv, w.ddt);
        return;
    }
    const float ri = L.ri[index], rj = L.rj[index];
    const float ri_m = (u > 0) ? L.ri[index - R] : 0.f;
    const float rj_m = (v > 0) ? L.rj[index - 1] : 0.f;
    const Steps s = mu_and_steps(p.mu, p.lambda_i, p.lambda_d, w.ddu, w.ddv, w.ddt, ri, rj, ri_m, rj_m, u > 0, v > 0);
    L.mu[index] = s.mu;
    if (steps == kStepsRaw || steps == kStepsAll) {
        L.spd[index] = s.spd;
        L.spuvx[index] = s.spuvx;
        L.spuvy[index] = s.spuvy;
        L.spwx[index] = s.spwx;
        L.spwy[index] = s.spwy;
        L.tu[index] = s.tu;
        L.tv[index] = s.tv;
        L.tw[index] = s.tw;
    }
    if (steps == kStepsQuads || steps == kStepsAll) {
        // the products the dual update forms (dual_update: mul(spd, mu), mul(spuvx, li), ...)
        L.qs[0][index] = mul(s.spd, s.mu);
        L.qs[1][index] = mul(s.spuvx, p.lambda_i);
        L.qs[2][index] = mul(s.spuvy, p.lambda_i);
        L.qs[3][index] = mul(s.spwx, p.lambda_d);
        L.qs[4][index] = mul(s.spwy, p.lambda_d);
        L.qs[5][index] = s.tu;
        L.qs[6][index] = s.tv;
        L.qs[7][index] = s.tw;
    }
}

// The new frame's weights as planes (the stage dump: the solve forms them
// where it needs them).
__global__ void k_rij2(LevelGeom g, PyrLevel n, LevelConsts L)
{
    const unsigned i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= g.N) return;
    const unsigned v = i % g.R, u = i / g.R;
    L.ri2[i] = u != g.C - 1 ? rij(n.xx, n.dep, i, g.R) : 1.f;
    L.rj2[i] = v != g.R - 1 ? rij(n.yy, n.dep, i, 1) : 1.f;
}

// ---------------------------------------------------------------------------
// Iteration kernels
// ---------------------------------------------------------------------------
__global__ void k_dual(LevelGeom g, LevelConsts L, State S, Params p)
{
    const size_t po = pair_off(g.map, g.pstride, blockIdx.y);
    L = at(L, po);
    S = at(S, po);
    const unsigned i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= g.N) return;
    const unsigned R = g.R, C = g.C;
    const unsigned v = i % R, u = i / R;
    const bool lu = (u == C - 1), lv = (v == R - 1);
    const unsigned iu = lu ? i : i + R, iv = lv ? i : i + 1;
    Duals d{S.pd[i], S.puu[i], S.puv[i], S.pvu[i], S.pvv[i], S.pwu[i], S.pwv[i]};
    dual_update(d, L.spd[i], L.spuvx[i], L.spuvy[i], L.spwx[i], L.spwy[i], L.mu[i], L.ddt[i], L.ddu[i], L.ddv[i],
                p.lambda_i, p.lambda_d, L.ri[i], L.rj[i], S.dua[i], S.dva[i], S.dwa[i], L.du_prev[i], L.dv_prev[i],
                S.dua[iu], S.dva[iu], S.dwa[iu], L.du_prev[iu], L.dv_prev[iu], S.dua[iv], S.dva[iv], S.dwa[iv],
                L.du_prev[iv], L.dv_prev[iv], lu, lv);
    S.pd[i] = d.pd;
    S.puu[i] = d.puu;
    S.puv[i] = d.puv;
    S.pvu[i] = d.pvu;
    S.pvv[i] = d.pvv;
    S.pwu[i] = d.pwu;
    S.pwv[i] = d.pwv;
}

__global__ void k_primal(LevelGeom g, LevelConsts L, State S, Params p, bool last, const float* depth_old)
{
    const size_t po = pair_off(g.map, g.pstride, blockIdx.y);
    L = at(L, po);
    S = at(S, po);
    depth_old = at(depth_old, po);
    const unsigned i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= g.N) return;
    const unsigned R = g.R, C = g.C;
    const unsigned v = i % R, u = i / R;
    const bool fu = (u == 0), lu = (u == C - 1), fv = (v == 0), lv = (v == R - 1);
    const unsigned im = fu ? i : i - R, jm = fv ? i : i - 1;
    const float ri = L.ri[i], rj = L.rj[i], ri_m = L.ri[im], rj_m = L.rj[jm];
    const float divu = divergence(ri, ri_m, rj, rj_m, S.puu[i], S.puu[im], S.puv[i], S.puv[jm], fu, lu, fv, lv);
    const float divv = divergence(ri, ri_m, rj, rj_m, S.pvu[i], S.pvu[im], S.pvv[i], S.pvv[jm], fu, lu, fv, lv);
    const float divw = divergence(ri, ri_m, rj, rj_m, S.pwu[i], S.pwu[im], S.pwv[i], S.pwv[jm], fu, lu, fv, lv);
    float du = S.du[i], dv = S.dv[i], dw = S.dw[i], dua, dva, dwa;
    primal_update(du, dv, dw, dua, dva, dwa, L.tu[i], L.tv[i], L.tw[i], L.mu[i], L.ddu[i], L.ddv[i], S.pd[i],
                  p.lambda_i, p.lambda_d, divu, divv, divw, L.dct[i], L.dcu[i], L.dcv[i]);
    if (last) {
        saturate(du, dv, dw, L.du_prev[i], L.dv_prev[i], depth_old[i]);
    } else {
        S.dua[i] = dua;
        S.dva[i] = dva;
        S.dwa[i] = dwa;
    }
    S.du[i] = du;
    S.dv[i] = dv;
    S.dw[i] = dw;
}

// saturateVariables alone, for a level scheduled with zero iterations.
__global__ void k_saturate(LevelGeom g, LevelConsts L, State S, const float* depth_old)
{
    const size_t po = pair_off(g.map, g.pstride, blockIdx.y);
    L = at(L, po);
    S = at(S, po);
    depth_old = at(depth_old, po);
    const unsigned i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= g.N) return;
    float du = S.du[i], dv = S.dv[i], dw = S.dw[i];
    saturate(du, dv, dw, L.du_prev[i], L.dv_prev[i], depth_old[i]);
    S.du[i] = du;
    S.dv[i] = dv;
    S.dw[i] = dw;
}

// ---------------------------------------------------------------------------
// filterSolution (pdflow_cudalib.cu:1040-1148) + computeMotionField (:1150-1167)
// ---------------------------------------------------------------------------
// Weighted median of up to 9 samples, register resident (the reference
// accumulates the weights in sorted order and walks to the first cumulative
// weight >= med, pdflow_cudalib.cu:1083-1132).
//
// Stable sort of up to 9 samples (the reference's bubbleSortDev,
// pdflow_cudalib.cu:1457-1473, swaps only on a strict '>', so equal values
// keep their input order) as an odd-even transposition network: 9 rounds of
// exchanges between neighbours (i, i+1), i of the round's parity, each on a
// strict '<'.  It sorts every 0/1 input and hence every input, and equal
// values never pass each other, so the order is the stable one.  Missing
// samples (n < 9) enter as (+inf, weight 0) after the present ones and stay
// there.  Then the cumulative weights are summed in sorted order, as the
// reference does, and the bracketing samples are interpolated; the result and
// the selected index are the reference's bit for bit.  Every index is a
// compile-time constant: nothing spills.
__device__ __forceinline__ float median9(const float (&f)[9], const float (&w)[9], unsigned present,
                                         float med_or_neg, float* total, int32_t* cont_out)
{
    // the samples in tap order, a missing one (bit clear in `present`) as +inf
    // of weight 0: the stable sort keeps the present samples in their order
    // and puts the missing ones after them, so its first n entries are those
    // of the reference's sort of the n present samples
    float sf[9], sw[9];
#pragma unroll
    for (int i = 0; i < 9; ++i) {
        const bool in = (present >> i) & 1u;
        sf[i] = in ? f[i] : INFINITY;
        sw[i] = in ? w[i] : 0.f;
    }
    // odd-even transposition sort: 9 rounds of adjacent exchanges on a strict
    // '<', so equal values never pass each other and the order is the stable
    // one of the reference's bubble sort, without carrying input indices
#pragma unroll
    for (int r = 0; r < 9; ++r)
#pragma unroll
        for (int a = r & 1; a + 1 < 9; a += 2) {
            const bool sw_ = sf[a + 1] < sf[a];
            const float tf = sf[a], tw = sw[a];
            sf[a] = sw_ ? sf[a + 1] : sf[a];
            sw[a] = sw_ ? sw[a + 1] : sw[a];
            sf[a + 1] = sw_ ? tf : sf[a + 1];
            sw[a + 1] = sw_ ? tw : sw[a + 1];
        }
    // cumulative weights; the missing samples (weight +0, sorted last) leave
    // the sum as it is (x + 0 == x for the non-negative sums), so cum[8] is
    // the reference's cum[n - 1]
    float cum[9];
    cum[0] = sw[0];
#pragma unroll
    for (int r = 1; r < 9; ++r) cum[r] = add(cum[r - 1], sw[r]);
    *total = cum[8];
    const float med = (med_or_neg < 0.f) ? mul(0.5f, cum[8]) : med_or_neg;
    // the reference counts the samples with med > cum (among the present
    // ones: a missing one's cum is the total, never below med) and
    // interpolates between that sample and the one before; cum does not
    // decrease, so the counted samples are a prefix and one pass finds both
    int cont = 0;
    float cr = 0.f, cl = 0.f, fr = 0.f, fl = 0.f;
#pragma unroll
    for (int r = 0; r < 8; ++r) {
        const bool t = med > cum[r];
        cont = t ? r + 1 : cont;
        cl = t ? cum[r] : cl;
        fl = t ? sf[r] : fl;
        cr = t ? cum[r + 1] : cr;
        fr = t ? sf[r + 1] : fr;
    }
    if (med > cum[8]) {   // past every sample: the reference finds no bracket
        cont = 9;
        cr = cl = fr = fl = 0.f;
    }
    *cont_out = cont;
    if (cont == 0) return sf[0];
    return median_lerp(cr, cl, med, fl, fr);
}

// The median's pixels in tiles of kMedRows x kMedCols (rows along
// threadIdx.x, so a warp's loads are one column's consecutive rows): the
// block first stages its tile and a one-pixel halo of the five planes the
// taps read, then every pixel takes its nine taps from shared memory at
// fixed offsets (outside the image the halo holds zeros; those taps are
// missing in `present` and never reach the median).
constexpr int kMedRows = 32, kMedCols = 8;
constexpr int kMedHR = kMedRows + 2, kMedHC = kMedCols + 2;

template <bool kDdtSq>   // L.spd holds powf(ddt, 2) (levels run as tiles)
__global__ void __launch_bounds__(kMedRows * kMedCols) k_median(LevelGeom g, bool finest, PyrLevel o, LevelConsts L,
                                                               State S, State Salt, LevelSol out, float* dx,
                                                               float* dy, float* dz, Params p, int32_t* sel)
{
    __shared__ float t_dep[kMedHC][kMedHR], t_sq[kMedHC][kMedHR], t_du[kMedHC][kMedHR], t_dv[kMedHC][kMedHR],
        t_dw[kMedHC][kMedHR];
    const size_t po = pair_off(g.map, g.pstride, blockIdx.z);
    const unsigned pf = pair_flags(g.map, blockIdx.z);
    finest = finest || (pf & kMapFinest);
    o = at(o, po);
    L = at(L, po);
    S = at((pf & kMapAlt) ? Salt : S, po);
    out = at(out, po);
    dx = at(dx, po);
    dy = at(dy, po);
    dz = at(dz, po);
    const int R = (int)g.R, C = (int)g.C;
    const int v0 = (int)blockIdx.x * kMedRows, u0 = (int)blockIdx.y * kMedCols;
    // the next level's start, as these CTAs end (no wait before it: this is an ordinary
    // launch, all before it has ended)
    allow_next_kernel();
    // the tile and its halo: rows v0-1 .. v0+kMedRows, columns u0-1 .. u0+kMedCols
    for (int e = threadIdx.y * kMedRows + threadIdx.x; e < kMedHR * kMedHC; e += kMedRows * kMedCols) {
        const int hr = e % kMedHR, hc = e / kMedHR, gv = v0 - 1 + hr, gu = u0 - 1 + hc;
        float z = 0.f, q = 0.f, a = 0.f, b = 0.f, c = 0.f;
        if (gv >= 0 && gv < R && gu >= 0 && gu < C) {
            const int j = gv + gu * R;
            z = o.dep[j];
            q = kDdtSq ? L.spd[j] : powf(L.ddt[j], 2.f);
            a = S.du[j];
            b = S.dv[j];
            c = S.dw[j];
        }
        t_dep[hc][hr] = z;
        t_sq[hc][hr] = q;
        t_du[hc][hr] = a;
        t_dv[hc][hr] = b;
        t_dw[hc][hr] = c;
    }
    __syncthreads();
    const int tv = (int)threadIdx.x, tu = (int)threadIdx.y;
    const int v = v0 + tv, u = u0 + tu;
    if (v >= R || u >= C) return;
    const unsigned index = (unsigned)(v + u * R);
    const float depth_old = t_dep[tu + 1][tv + 1];
    float ru, rv, rw;
    if (depth_old > 0.f) {
        // the nine taps in the reference's order (row offset, then column);
        // taps outside the image are marked missing (median9)
        unsigned present = 0x1ffu;
        if (v == 0) present &= ~0x007u;       // row offset -1: taps 0, 1, 2
        if (v == R - 1) present &= ~0x1c0u;   // row offset +1: taps 6, 7, 8
        if (u == 0) present &= ~0x049u;       // column offset -1: taps 0, 3, 6
        if (u == C - 1) present &= ~0x124u;   // column offset +1: taps 2, 5, 8
        float fu[9], fv[9], fw[9], wt[9];
#pragma unroll
        for (int k = -1; k < 2; k++)
#pragma unroll
            for (int l = -1; l < 2; l++) {
                const int q = 3 * (k + 1) + (l + 1);
                const int hc = tu + 1 + l, hr = tv + 1 + k;
                const float dz2 = (q == 4) ? pow2_diff_voted(depth_old, t_dep[hc][hr])   // the centre: z0 - z0
                                           : powf(sub(depth_old, t_dep[hc][hr]), 2.f);
                wt[q] = __frcp_rn(fm(10.f, t_sq[hc][hr], fm(5.f, dz2, 1.f)));
                fu[q] = t_du[hc][hr];
                fv[q] = t_dv[hc][hr];
                fw[q] = t_dw[hc][hr];
            }
        float tot;
        int32_t c0, c1, c2;
        ru = median9(fu, wt, present, -1.f, &tot, &c0);
        const float pres_med = mul(0.5f, tot);   // half of u's total, for all three (:1097)
        rv = median9(fv, wt, present, pres_med, &tot, &c1);
        rw = median9(fw, wt, present, pres_med, &tot, &c2);
        if (sel) { sel[index] = c0; sel[g.N + index] = c1; sel[2 * g.N + index] = c2; }
    } else {
        ru = t_du[tu + 1][tv + 1];
        rv = t_dv[tu + 1][tv + 1];
        rw = t_dw[tu + 1][tv + 1];
        if (sel) { sel[index] = -1; sel[g.N + index] = -1; sel[2 * g.N + index] = -1; }
    }
    out.du[index] = ru;
    out.dv[index] = rv;
    out.dw[index] = rw;
    // the duals go on to the next level (14 of the finest level's 27 planes of
    // traffic would be duals nobody reads; the stage form carries none)
    if (out.pd && !finest) {
        out.pd[index] = S.pd[index];
        out.puu[index] = S.puu[index];
        out.puv[index] = S.puv[index];
        out.pvu[index] = S.pvu[index];
        out.pvv[index] = S.pvv[index];
        out.pwu[index] = S.pwu[index];
        out.pwv[index] = S.pwv[index];
    }
    if (finest) {
        if (depth_old > 0) {
            // the finest level is cols wide (g.C == p.cols), also for a mixed batch's smaller pairs
            motion_field(depth_old, ru, rv, rw, o.xx[index], o.yy[index], inv_focal(p.fovh, g.C), dx[index],
                         dy[index], dz[index]);
        } else {
            dx[index] = 0.f;
            dy[index] = 0.f;
            dz[index] = 0.f;
        }
    }
}

// Per-level record of a solve (copyAllSolutions of the live application,
// called after every level: scene_flow_visualization.cpp:194-199).
__global__ void k_level_keep(LevelGeom g, LevelSol sol, PyrLevel o, Params p, float* __restrict__ keep,
                             size_t stride, size_t off)
{
    const unsigned y = blockIdx.y;
    const size_t po = pair_off(g.map, g.pstride, y);
    const unsigned slot = g.map ? (__ldg(g.map + y) & kMapSlotMask) : y;
    const unsigned i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= g.N) return;
    sol = at(sol, po);
    o = at(o, po);
    float* k = keep + (size_t)slot * stride + off;
    const float du = sol.du[i], dv = sol.dv[i], dw = sol.dw[i];
    k[i] = du;
    k[g.N + i] = dv;
    k[2 * g.N + i] = dw;
    const float z = o.dep[i];
    float dx = 0.f, dy = 0.f, dz = 0.f;
    if (z > 0.f) motion_field(z, du, dv, dw, o.xx[i], o.yy[i], inv_focal(p.fovh, p.cols), dx, dy, dz);
    k[3 * g.N + i] = dx;
    k[4 * g.N + i] = dy;
    k[5 * g.N + i] = dz;
}

// Frame t's pyramid becomes frame t-1's, for the mapped slots: the planes of all
// levels lie back to back (n float4, the padding between them included).
__global__ void k_pyr_copy(const float4* src, float4* dst, size_t n, size_t pstride, const unsigned* __restrict__ map)
{
    const size_t po = pair_off(map, pstride, blockIdx.y);
    src = at(src, po);
    dst = at(dst, po);
    for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x)
        dst[i] = src[i];
}

// Both frames at the solution's total image-plane flow, for the energy.
__global__ void k_energy_warp(LevelGeom g, LevelSol sol, PyrLevel o, PyrLevel n, LevelConsts L, Params p, size_t aux)
{
    const size_t po = pair_off(g.map, g.pstride, blockIdx.y);
    const unsigned i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= g.N) return;
    L = at(L, po);
    const Warped w = warp_px(at(o, po), at(n, po), L, aux, g.R, g.C, i % g.R, i / g.R, at(sol.du, po)[i],
                             at(sol.dv, po)[i]);
    L.dct[i] = w.dct;
    L.ddt[i] = w.ddt;
    L.mu[i] = data_weight(p.mu, w.ddu, w.ddv, w.ddt);
}

// 1024 accumulators per pair: accumulator t sums pixels t, t + 1024, ... in
// that order (32 one-warp CTAs per pair, so the FP64 work of one pair spreads
// over 32 SMs); k_energy_sum then adds the 1024 partial sums of a pair in a
// fixed tree, so the energy is deterministic and independent of the batch.
// With du = dv = 0 increments at the warp point the linearised data terms
// equal the warped residuals.
constexpr unsigned kEnergyAcc = 1024;

__global__ void __launch_bounds__(32) k_energy(LevelGeom g, LevelSol sol, LevelConsts L, Params p,
                                               double* __restrict__ part)
{
    const size_t po = pair_off(g.map, g.pstride, blockIdx.y);
    sol = at(sol, po);
    L = at(L, po);
    const unsigned R = g.R, C = g.C;
    const unsigned t = blockIdx.x * 32 + threadIdx.x;
    double acc = 0.0;
    for (unsigned i = t; i < g.N; i += kEnergyAcc) {
        const unsigned v = i % R, u = i / R;
        const float U = sol.du[i], V = sol.dv[i], W = sol.dw[i], ri = L.ri[i], rj = L.rj[i];
        const bool lu = u == C - 1, lv = v == R - 1;
        const float gu1 = lu ? 0.f : mul(ri, sub(sol.du[i + R], U)), gu2 = lv ? 0.f : mul(rj, sub(sol.du[i + 1], U));
        const float gv1 = lu ? 0.f : mul(ri, sub(sol.dv[i + R], V)), gv2 = lv ? 0.f : mul(rj, sub(sol.dv[i + 1], V));
        const float gw1 = lu ? 0.f : mul(ri, sub(sol.dw[i + R], W)), gw2 = lv ? 0.f : mul(rj, sub(sol.dw[i + 1], W));
        double e = fabs((double)L.dct[i]) + (double)L.mu[i] * fabs((double)L.ddt[i] - (double)W);
        e += (double)p.lambda_i * (hypot((double)gu1, (double)gu2) + hypot((double)gv1, (double)gv2));
        e += (double)p.lambda_d * hypot((double)gw1, (double)gw2);
        acc += e;
    }
    part[(size_t)blockIdx.y * kEnergyAcc + t] = acc;
}

__global__ void __launch_bounds__(kEnergyAcc) k_energy_sum(const double* __restrict__ part,
                                                           float* __restrict__ energies)
{
    __shared__ double red[kEnergyAcc];
    red[threadIdx.x] = part[(size_t)blockIdx.y * kEnergyAcc + threadIdx.x];
    __syncthreads();
    for (unsigned w = blockDim.x / 2; w > 0; w >>= 1) {
        if (threadIdx.x < w) red[threadIdx.x] += red[threadIdx.x + w];
        __syncthreads();
    }
    if (threadIdx.x == 0) energies[blockIdx.y] = (float)red[0];
}

}  // namespace

// ---------------------------------------------------------------------------
// Launchers
// ---------------------------------------------------------------------------
namespace {

// Up to this many pixels a pyramid is bound by latency: the first pass takes
// three levels (one launch less for 320x240 frames), 512 threads a tile.  Beyond,
// by instructions: two levels, so no second-level pixel is computed twice, and
// 256 threads, so that tiles overlap.  Two pushes on a GB300 (few / many form):
// one 320x240 frame 34 / 48 us, 8 52 / 64, 64 192 / 154; one 640x480 frame 52 / 61,
// two 66 / 66, four 82 / 75, 64 605 / 428.
constexpr size_t kPyrFewPixels = 2 * 640 * 480;

// One pass: count - 1 levels below `src` (and with kWriteFirst src's own planes).
template <bool kWriteFirst, class Source>
cudaError_t pyramid_pass(const Source& src, const PyrLevel* levels, unsigned count, bool few, float fovh,
                         unsigned pairs, size_t pstride, cudaStream_t st, const unsigned* map)
{
    const dim3 grid((src.W + kPyrTile - 1) / kPyrTile, (src.H + kPyrTile - 1) / kPyrTile, pairs);
    const PyrLevel &l1 = levels[1], &l2 = count > 2 ? levels[2] : levels[1];
    if (few)
        return launch_overlapped(k_pyramid<Source, kWriteFirst, 512>, grid, dim3(512), 0, st, src, levels[0], l1, l2,
                                 int(count), fovh, pstride, map);
    return launch_overlapped(k_pyramid<Source, kWriteFirst, 256>, grid, dim3(256), 0, st, src, levels[0], l1, l2,
                             int(count), fovh, pstride, map);
}

template <class Source>
cudaError_t pyramid(const Source& src, const PyrLevel* levels, unsigned count, float fovh, unsigned pairs,
                    size_t pstride, cudaStream_t st, const unsigned* map)
{
    if (count < 2) return cudaErrorInvalidValue;
    const bool few = size_t(src.W) * src.H * pairs <= kPyrFewPixels;
    const unsigned first = few ? std::min(count, 3u) : 2u;
    cudaError_t e = pyramid_pass<true>(src, levels, first, few, fovh, pairs, pstride, st, map);
    for (unsigned l = first - 1; l + 1 < count && e == cudaSuccess; l += 2) {   // levels l + 1, l + 2 from level l
        const SourcePlanes up{levels[l].col, levels[l].dep, src.W >> l, src.H >> l};
        e = pyramid_pass<false>(up, levels + l, std::min(count - l, 3u), few, fovh, pairs, pstride, st, map);
    }
    return e;
}

}  // namespace

cudaError_t launch_pyramid_u16(const uint8_t* img, const uint16_t* depth, unsigned W, unsigned H,
                               const PyrLevel* levels, unsigned count, float fovh, unsigned pairs, size_t pstride,
                               cudaStream_t st, const unsigned* map)
{
    return pyramid(SourceU16{img, depth, W, H}, levels, count, fovh, pairs, pstride, st, map);
}

cudaError_t launch_pyramid_rgb8_mm(const uint8_t* rgb, const uint16_t* depth, unsigned W, unsigned H,
                                   const PyrLevel* levels, unsigned count, float fovh, unsigned pairs, size_t pstride,
                                   cudaStream_t st, int rotate180)
{
    return pyramid(SourceRgb{rgb, depth, W, H, rotate180}, levels, count, fovh, pairs, pstride, st, nullptr);
}

cudaError_t launch_pyramid_planes(const float* I, const float* Z, unsigned W, unsigned H, const PyrLevel* levels,
                                  unsigned count, float fovh, unsigned pairs, size_t pstride, cudaStream_t st)
{
    return pyramid(SourcePlanes{I, Z, W, H}, levels, count, fovh, pairs, pstride, st, nullptr);
}

cudaError_t launch_pyr_copy(const PyrLevel* src, const PyrLevel* dst, unsigned levels, unsigned smallest, unsigned pairs,
                            size_t pstride, const unsigned* map, cudaStream_t st)
{
    const size_t n = (size_t(src[levels - 1].yy - src[0].col) + smallest + 3) / 4;   // whole float4 (planes are padded)
    const dim3 grid(unsigned(std::min<size_t>((n + kBlock - 1) / kBlock, 1024)), pairs);
    k_pyr_copy<<<grid, kBlock, 0, st>>>(reinterpret_cast<const float4*>(src[0].col), reinterpret_cast<float4*>(dst[0].col),
                                       n, pstride, map);
    return cudaGetLastError();
}

cudaError_t launch_flow_out(const float* dx, const float* dy, const float* dz, size_t step, unsigned n, size_t floats,
                            const unsigned* status, float* out, unsigned* out_status, cudaStream_t st)
{
    const unsigned n4 = unsigned(floats / 4);
    k_flow_out<<<dim3((n4 + kBlock - 1) / kBlock, 3, n), kBlock, 0, st>>>(
        dx, dy, dz, step, n4, status, reinterpret_cast<float4*>(out), out_status);
    return cudaGetLastError();
}

static dim3 level_grid(const LevelGeom& g) { return dim3(blocks_for(g.N), g.pairs); }

cudaError_t launch_im_gradients(const LevelGeom* levels, const PyrLevel* images, const size_t* aux, unsigned count,
                                LevelConsts L, cudaStream_t st)
{
    if (count == 0 || count > 8) return cudaErrorInvalidValue;
    GradLevels lv{};
    lv.count = count;
    for (unsigned q = 0; q < count; ++q) {
        lv.n[q] = images[q];
        lv.R[q] = levels[q].R;
        lv.C[q] = levels[q].C;
        lv.aux[q] = aux[q];
        lv.first_block[q + 1] = lv.first_block[q] + blocks_for(levels[q].N);
    }
    k_im_gradients<<<dim3(lv.first_block[count], levels[0].pairs), kBlock, 0, st>>>(lv, L, levels[0].pstride,
                                                                                  levels[0].map);
    return cudaGetLastError();
}

cudaError_t launch_level_setup(LevelGeom g, LevelStart start, LevelSol coarse, PyrLevel old_l, PyrLevel new_l,
                               LevelConsts L, State S, Params p, int steps, size_t aux, cudaStream_t st,
                               const float* seed)
{
    cudaError_t e;
    if (g.R % 2 == 0)
        e = launch_overlapped(k_level_start<2>, dim3(blocks_for(g.N / 2), g.pairs), dim3(kBlock), 0, st, g, int(start),
                              coarse, old_l, L, S, seed);
    else if (start == LevelStart::Coarse)
        return cudaErrorInvalidValue;   // a level above another has even rows
    else
        e = launch_overlapped(k_level_start<1>, level_grid(g), dim3(kBlock), 0, st, g, int(start), coarse, old_l, L, S,
                              seed);
    if (e != cudaSuccess) return e;
    return launch_overlapped(k_level_warp, level_grid(g), dim3(kBlock), 0, st, g, old_l, new_l, L, p, steps, aux);
}

cudaError_t launch_rij2(LevelGeom g, PyrLevel new_l, LevelConsts L, cudaStream_t st)
{
    k_rij2<<<level_grid(g), kBlock, 0, st>>>(g, new_l, L);
    return cudaGetLastError();
}

cudaError_t launch_dual(LevelGeom g, LevelConsts L, State S, Params p, cudaStream_t st)
{
    k_dual<<<level_grid(g), kBlock, 0, st>>>(g, L, S, p);
    return cudaGetLastError();
}

cudaError_t launch_primal(LevelGeom g, LevelConsts L, State S, Params p, bool last, const float* depth_old,
                          cudaStream_t st)
{
    k_primal<<<level_grid(g), kBlock, 0, st>>>(g, L, S, p, last, depth_old);
    return cudaGetLastError();
}

cudaError_t launch_saturate(LevelGeom g, LevelConsts L, State S, const float* depth_old, cudaStream_t st)
{
    k_saturate<<<level_grid(g), kBlock, 0, st>>>(g, L, S, depth_old);
    return cudaGetLastError();
}

cudaError_t launch_level_keep(LevelGeom g, LevelSol sol, PyrLevel old_l, Params p, float* keep, size_t stride,
                              size_t off, cudaStream_t st)
{
    k_level_keep<<<level_grid(g), kBlock, 0, st>>>(g, sol, old_l, p, keep, stride, off);
    return cudaGetLastError();
}

cudaError_t launch_median(LevelGeom g, bool finest, PyrLevel old_l, LevelConsts L, State S, LevelSol out, float* dx,
                          float* dy, float* dz, Params p, int32_t* sel, cudaStream_t st, const State* alt,
                          bool ddt_sq)
{
    const dim3 grid((g.R + kMedRows - 1) / kMedRows, (g.C + kMedCols - 1) / kMedCols, g.pairs);
    const dim3 block(kMedRows, kMedCols);
    // An ordinary launch: CTAs of it that start beside the last of the streamed
    // tiles' run with what L1 those leave, and so do the set-up kernels that follow
    // before the SM is next idle (a 64-pair VGA solve 31.28 ms, against 30.73; one
    // 320x240 pair 0.502, against 0.499).
    if (ddt_sq)
        k_median<true><<<grid, block, 0, st>>>(g, finest, old_l, L, S, alt ? *alt : S, out, dx, dy, dz, p, sel);
    else
        k_median<false><<<grid, block, 0, st>>>(g, finest, old_l, L, S, alt ? *alt : S, out, dx, dy, dz, p, sel);
    return cudaGetLastError();
}

cudaError_t launch_energy_warp(LevelGeom g, LevelSol sol, PyrLevel old_l, PyrLevel new_l, LevelConsts L, Params p,
                               size_t aux, cudaStream_t st)
{
    k_energy_warp<<<level_grid(g), kBlock, 0, st>>>(g, sol, old_l, new_l, L, p, aux);
    return cudaGetLastError();
}

cudaError_t launch_energy(LevelGeom g, LevelSol sol, LevelConsts L, Params p, float* energies, double* part,
                          cudaStream_t st)
{
    k_energy<<<dim3(kEnergyAcc / 32, g.pairs), 32, 0, st>>>(g, sol, L, p, part);
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return e;
    k_energy_sum<<<dim3(1, g.pairs), kEnergyAcc, 0, st>>>(part, energies);
    return cudaGetLastError();
}

}  // namespace pdflow
