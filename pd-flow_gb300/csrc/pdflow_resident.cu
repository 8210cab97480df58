// A small level's iterations in one launch, a thread-block cluster per pair
// ("resident tiles"): the deep-tile form (9) of levels that fit a cluster.
//
// Each CTA of a cluster keeps one tile (an interior plus a halo of 4) of the
// pair's level in registers for the whole level: the 13 state and 19 constant
// planes are read once, and every 4 iterations each CTA puts the ring of
// interior pixels that other tiles hold as halo into its shared memory, the
// cluster's barrier passes, and each CTA reloads its own halo from its
// neighbours' shared memory.  Per-pixel arithmetic is pdflow_region.cuh, so
// the bits are those of every other form.
//
// Bound: the iterations' dependent chain and two block barriers (5 or 12 warps
// an SM).  As deep streamed tiles these levels were a launch per 8 iterations,
// each loading 32 planes of 32 x 32 regions and storing 13: 1.6 us an iteration
// at 30x40 and 1.7 at 60x80 for one pair, here 0.65 and 0.99 (graph replay on a
// GB300).  Sixteen tiles of 8 x 12 (16 x 20 regions, 160 threads) take 30x40,
// fifteen of 24 x 16 (32 x 24 regions, 384 threads) 60x80, the smallest regions
// that cover them within a cluster.  A cooperative launch over all SMs with
// smaller tiles and counters in global memory for the exchange took 1.07 and
// 1.17 us an iteration and 22 us more per launch inside a graph.
#include <cuda_runtime.h>

#include "pdflow_iterate.cuh"
#include "pdflow_region.cuh"

namespace pdflow {

namespace {

using namespace region;

constexpr int kHalo = 4;              // iterations between two exchanges
constexpr unsigned kMostTiles = 16;   // CTAs of a cluster (more than 8 is opt-in)

struct ResidentArgs {
    LevelGeom g;
    const float* consts[19];   // in the order of PairConsts
    const float* src[13];      // in the order of PairState
    float* dst[13];
    const float* depth_old;
    float lambda_i, lambda_d;
    unsigned iters;
    const unsigned* pair_iters;   // iterations of each pair (null: iters)
    unsigned tiles_v, tiles;   // tiles per column of tiles, per pair (= the cluster's CTAs)
};

__device__ __forceinline__ void cluster_sync()
{
    __syncwarp();   // .aligned: the whole warp together
    asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
    asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
}

template <int kLanes, int kCols>
struct TileShape {
    static constexpr int kRows = 2 * kLanes, kPlane = kRows * kCols, kThreads = kLanes * kCols;
    static constexpr int kIntV = kRows - 2 * kHalo, kIntU = kCols - 2 * kHalo;
    static constexpr int kEdge = kIntV * kIntU / 2;   // float2 of a plane of the exchange buffer
    static_assert(kThreads % 32 == 0 && kIntV % 2 == 0, "whole warps, whole pairs");
    // exchange planes of the iteration, then two buffers of 13 interior planes
    static constexpr size_t kSmem = sizeof(float) * (6 * kPlane + 2 * 13 * 2 * kEdge);
};

template <int kLanes, int kCols>
__global__ void __launch_bounds__(kLanes* kCols) k_iterate_resident(const __grid_constant__ ResidentArgs a)
{
    using T = TileShape<kLanes, kCols>;
    extern __shared__ __align__(16) float sm[];
    float *X = sm, *Y = sm + 3 * T::kPlane;
    float2* edge = reinterpret_cast<float2*>(sm + 6 * T::kPlane);   // [buffer][plane][pair of the interior]
    const int t = threadIdx.x, c = t / kLanes, p = t % kLanes;
    const int me = c * T::kRows + 2 * p;
    const int right = (c + 1 < kCols ? c + 1 : c) * T::kRows + 2 * p;   // beyond the region: own storage
    const int left = (c > 0 ? c - 1 : c) * T::kRows + 2 * p;
    const unsigned y = blockIdx.x / a.tiles, tile = blockIdx.x - y * a.tiles;   // tile: the rank in the cluster
    const int R = (int)a.g.R, C = (int)a.g.C;
    const int tv = (int)(tile % a.tiles_v), tu = (int)(tile / a.tiles_v);
    const int iv0 = tv * T::kIntV, iu0 = tu * T::kIntU, iv1 = min(iv0 + T::kIntV, R), iu1 = min(iu0 + T::kIntU, C);
    const int v0 = max(iv0 - kHalo, 0) + 2 * p, u = max(iu0 - kHalo, 0) + c;
    const size_t po = pair_off(a.g.map, a.g.pstride, y), gi = (size_t)v0 + (size_t)u * (size_t)R;
    const bool live = u < C && v0 < R;            // rows are even: both pixels of the pair
    const bool inner = live && v0 >= iv0 && v0 < iv1 && u >= iu0 && u < iu1;
    // interior pixels some other tile holds as halo, and this tile's halo
    const bool ring = inner && ((tv > 0 && v0 < iv0 + kHalo) || (iv1 < R && v0 >= iv1 - kHalo) ||
                                (tu > 0 && u < iu0 + kHalo) || (iu1 < C && u >= iu1 - kHalo));
    const bool halo = live && !inner && v0 < iv1 + kHalo && u < iu1 + kHalo;
    // the pair's place in its owner's exchange planes, and (halo) the owner's
    const int ov = v0 / T::kIntV, ou = u / T::kIntU;
    const int slot = (u - ou * T::kIntU) * (T::kIntV / 2) + (v0 - ov * T::kIntV) / 2;
    uint32_t owner = smem_u32(edge);
    if (halo)
        asm("mapa.shared::cluster.u32 %0, %1, %2;"
            : "=r"(owner)
            : "r"(smem_u32(edge)), "r"((unsigned)ov + (unsigned)ou * a.tiles_v));

    const float2 zero = make_float2(0.f, 0.f);
    auto plane = [&](const float* q) {   // plain loads: the kernel before may write them while this one starts
        return live ? *reinterpret_cast<const float2*>(at(q, po) + gi) : zero;
    };
    const unsigned iters = a.pair_iters ? __ldg(a.pair_iters + y) : a.iters;   // the same for the whole cluster
    after_previous_kernel();
    allow_next_kernel();
    const PairConsts k{plane(a.consts[0]),  plane(a.consts[1]),  plane(a.consts[2]),  plane(a.consts[3]),
                       plane(a.consts[4]),  plane(a.consts[5]),  plane(a.consts[6]),  plane(a.consts[7]),
                       plane(a.consts[8]),  plane(a.consts[9]),  plane(a.consts[10]), plane(a.consts[11]),
                       plane(a.consts[12]), plane(a.consts[13]), plane(a.consts[14]), plane(a.consts[15]),
                       plane(a.consts[16]), plane(a.consts[17]), plane(a.consts[18])};
    PairState s{plane(a.src[0]), plane(a.src[1]), plane(a.src[2]),  plane(a.src[3]),  plane(a.src[4]),
                plane(a.src[5]), plane(a.src[6]), plane(a.src[7]),  plane(a.src[8]),  plane(a.src[9]),
                plane(a.src[10]), plane(a.src[11]), plane(a.src[12])};
    const PairDerived d(k);
    const PairPlace place{u == 0, u == C - 1, v0 == 0, v0 + 1 == R - 1};
    struct Hooks {
        const float* yl;
        __device__ __forceinline__ void sync() const { __syncthreads(); }
        __device__ __forceinline__ void carry(float2, float2, float2) const {}
        __device__ __forceinline__ const float* left(int q) const { return yl + q * T::kPlane; }
    };
    // Exchange x uses buffer x & 1: a CTA writes it again at exchange x + 2,
    // after the barrier of x + 1, which every CTA reaches after reading x.
    unsigned buffer = 0;
    for (unsigned done = 0;; buffer ^= 1u) {
        const unsigned kk = min(iters - done, (unsigned)kHalo);
        for (unsigned j = 0; j < kk; ++j)
            iterate_pair<true, kLanes, false>(s, k, d, X, Y, T::kPlane, me, right, place, a.lambda_i, a.lambda_d,
                                       Hooks{Y + left});
        done += kk;
        if (done >= iters) break;
        if (ring) {
            const float2 st[13] = {s.du, s.dv, s.dw, s.ua, s.va, s.wa, s.pd, s.puu, s.puv, s.pvu, s.pvv, s.pwu, s.pwv};
#pragma unroll
            for (int q = 0; q < 13; ++q) edge[(buffer * 13 + q) * T::kEdge + slot] = st[q];
        }
        cluster_sync();
        if (halo) {
            float2* to[13] = {&s.du, &s.dv, &s.dw, &s.ua, &s.va, &s.wa, &s.pd,
                              &s.puu, &s.puv, &s.pvu, &s.pvv, &s.pwu, &s.pwv};
#pragma unroll
            for (int q = 0; q < 13; ++q)
                asm volatile("ld.shared::cluster.v2.f32 {%0, %1}, [%2];"
                             : "=f"(to[q]->x), "=f"(to[q]->y)
                             : "r"(owner + 8u * ((buffer * 13 + q) * T::kEdge + slot))
                             : "memory");
        }
    }
    if (inner) {
        saturate_pair(s, k, __ldg(reinterpret_cast<const float2*>(at(a.depth_old, po) + gi)));
        const float2 st[13] = {s.du, s.dv, s.dw, s.ua, s.va, s.wa, s.pd, s.puu, s.puv, s.pvu, s.pvv, s.pwu, s.pwv};
#pragma unroll
        for (int q = 0; q < 13; ++q) *reinterpret_cast<float2*>(at(a.dst[q], po) + gi) = st[q];
    }
    cluster_sync();   // a neighbour may still be reading this CTA's shared memory
}

struct Shape {
    int rows, cols, threads;   // interior, threads
    size_t smem;
    const void* kernel;
};
template <int kLanes, int kCols>
Shape shape()
{
    using T = TileShape<kLanes, kCols>;
    return {T::kIntV, T::kIntU, T::kThreads, T::kSmem, (const void*)k_iterate_resident<kLanes, kCols>};
}
// The smallest region whose tiles fit a cluster.
const Shape kShapes[2] = {shape<8, 20>(), shape<16, 24>()};

unsigned shape_tiles(const Shape& s, const LevelGeom& g)
{
    return ((g.R + s.rows - 1) / s.rows) * ((g.C + s.cols - 1) / s.cols);
}

const Shape* shape_for(const LevelGeom& g)
{
    for (const Shape& s : kShapes)
        if (shape_tiles(s, g) <= kMostTiles) return &s;
    return nullptr;
}

}  // namespace

bool resident_eligible(const LevelGeom& g, const LevelConsts& L, const State& src, const State& dst, unsigned sms)
{
    const Shape* s = shape_for(g);
    // The small shape's CTAs share an SM; at 30x40 it wins at every batch measured
    // (per 85 iterations, against streamed tiles: 1 pair 0.063 / 0.140 ms, 24 pairs
    // 0.139 / 0.156, 128 pairs 0.520 / 0.625).  The large one's take an SM each: at
    // 60x80 it wins up to two rounds of CTAs (100 iterations: 1 pair 0.106 / 0.172,
    // 16 pairs 0.27 / 0.47 ms) and loses beyond (24 pairs 0.407 / 0.360).
    return s && (s == kShapes || shape_tiles(*s, g) * g.pairs <= 2 * sms) && stream_direct_eligible(g, L, src, dst);
}

cudaError_t prepare_resident()
{
    cudaError_t e = cudaSuccess;
    for (const Shape& s : kShapes) {
        if (e == cudaSuccess)
            e = cudaFuncSetAttribute(s.kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)s.smem);
        if (e == cudaSuccess) e = cudaFuncSetAttribute(s.kernel, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
    }
    return e;
}

cudaError_t launch_iterate_resident(LevelGeom g, LevelConsts L, State src, State dst, Params p,
                                    const float* depth_old, unsigned iters, cudaStream_t st,
                                    const unsigned* pair_iters)
{
    if (iters == 0 || reinterpret_cast<uintptr_t>(depth_old) % 8u != 0 || !shape_for(g) ||
        !stream_direct_eligible(g, L, src, dst))
        return cudaErrorInvalidValue;
    const Shape& s = *shape_for(g);
    ResidentArgs a{};
    a.g = g;
    const float* cg[19] = {L.ri, L.rj, L.dct, L.dcu, L.dcv, L.ddt, L.ddu, L.ddv, L.mu, L.du_prev, L.dv_prev,
                           L.qs[0], L.qs[1], L.qs[2], L.qs[3], L.qs[4], L.qs[5], L.qs[6], L.qs[7]};
    for (int q = 0; q < 19; ++q) a.consts[q] = cg[q];
    const float* sp[13] = {src.du, src.dv, src.dw, src.dua, src.dva, src.dwa, src.pd,
                           src.puu, src.puv, src.pvu, src.pvv, src.pwu, src.pwv};
    float* dp[13] = {dst.du, dst.dv, dst.dw, dst.dua, dst.dva, dst.dwa, dst.pd,
                     dst.puu, dst.puv, dst.pvu, dst.pvv, dst.pwu, dst.pwv};
    for (int q = 0; q < 13; ++q) {
        a.src[q] = sp[q];
        a.dst[q] = dp[q];
    }
    a.depth_old = depth_old;
    a.lambda_i = p.lambda_i;
    a.lambda_d = p.lambda_d;
    a.iters = iters;
    a.pair_iters = pair_iters;
    a.tiles_v = (g.R + s.rows - 1) / s.rows;
    a.tiles = shape_tiles(s, g);
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(a.tiles * g.pairs);
    cfg.blockDim = dim3(unsigned(s.threads));
    cfg.dynamicSmemBytes = s.smem;
    cfg.stream = st;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = a.tiles;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[1].val.programmaticStreamSerializationAllowed = 1;
    cfg.numAttrs = 2;
    void* args[] = {&a};
    return cudaLaunchKernelExC(&cfg, s.kernel, args);
}

}  // namespace pdflow
