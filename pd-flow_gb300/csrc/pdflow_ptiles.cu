// Persistent, register-resident tile iterations ("streamed tiles", iteration
// forms 8 and 9; the strips of form 10 below).
//
// One CTA per SM walks a list of tiles (every 24 x 24 interior of every pair
// of the launch, 4-pixel halo: 32 x 32 regions, as in pdflow_tiles2.cu).  A
// tile's 13 state planes and 19 level constants (11 set-up planes and the 8
// step products) live in registers while its kk <= 4 iterations run: each of
// the 512 threads owns a vertical pixel pair (rows 2p, 2p+1 of region column
// c) and computes it with packed FP32x2 instructions.  Meanwhile the TMA unit
// copies the next tile's 32 planes into a shared-memory staging buffer (two 4D
// tensor copies, one per run of planes the arena keeps back to back: the 13
// state planes and the 19 constants, pdflow_tmap.h; completing on an
// mbarrier), so the region loads run behind the arithmetic.
//
// Neighbours: the row below the pair (dual step) and above it (primal step)
// by warp shuffles inside the column's 16 lanes; the column to the right
// (dual) and to the left (primal) through six shared exchange planes, into
// which each thread publishes what its neighbours read (U = du_acc + du_prev,
// V = dv_acc + dv_prev, W = dw_acc; ri * the u-component of each TV dual).
// These are the same rounded expressions the reference evaluates
// (computeGradient, computeDivergence: pdflow_cudalib.cu:935-1013), so the
// results are bit-identical to every other iteration form.  Every pixel of
// the region is updated in every iteration; the stale ring at non-border
// region edges is never read by an exact pixel and only the interior is
// stored.  Needs rows % 4 == 0 (16-byte aligned tensor-copy rows); levels
// with an even row count otherwise (30x40, where form 8 was chosen: by default it
// runs resident, pdflow_resident.cu) run the tiles with each thread loading its
// pixel pair's 32 values directly (8-byte loads, no staging: such levels have
// about one region per CTA, nothing to stream).
//
// Strips (iteration form 10).  Of an iteration's column neighbours only the
// primal step's backward difference looks left (ri * the dual's u-component
// at column u - 1), and only the dual step's forward difference looks right.
// A CTA that walks a row of regions left to right can therefore hand the
// next region the left neighbour's exchange values of every iteration (a
// carry of 3 x 32 floats per iteration, in shared memory) instead of
// recomputing a left halo: after kk iterations columns [x, x + 32 - kk) of a
// region at column x are exact, 28 of 32 at kk = 4 instead of 24.  The
// units of work are whole strips (a pair's 24-row bands) and, for the last
// strips of the launch, column pieces of them, smaller towards the end (each
// starting with a region that recomputes a left halo of kk columns).  CTAs take units in order from
// a device counter as they finish the previous one: they walk vertically
// adjacent bands side by side (their row halos meet in L2 and their reads
// fill DRAM pages, as the tiles' do), and a CTA whose strips converge faster
// (the disc projection's work depends on the data) takes more of them; the
// pieces keep the last units short.  The last CTA to finish resets the
// counter for the next launch.
//
// Who does what.  Sixteen consumer warps hold the pixels; one lane of an
// extra warpgroup walks the regions, writes each one's descriptor and starts
// its copies as soon as the sixteen warps have read the staging planes (an
// mbarrier they arrive on), so the walk's index arithmetic, the unit counter's
// latency and the copies' issue are off the arithmetic's path, and a region
// has no block barrier but the iterations' two.  Bound: instruction issue and
// latency (16 warps an SM, the registers' limit; 51.3 % issue active, 6.63 warp
// instructions a pixel-iteration).  When
// thread 0 of the consumers did the walk behind a block barrier a region, 64
// VGA pairs took 35.74 ms and five 3.68 ms; with the producer 32.43 and 3.48.
//
// Launches of a level follow one another by programmatic dependent launch: a CTA
// starts as one of the launch before leaves its SM, prepares its barriers and its
// first region's descriptor, and waits for that launch's end before its first
// copy (one VGA pair, 25 launches of about 19 us at 480x640 and 22 of 7 at
// 240x320: 1237 -> 1191 us with its transfers), or, from a level's second launch
// on, before its first copy of state: the constants are final, so their 19 planes
// arrive while the launch before ends (one VGA solve 962 -> 928 us, one 320x240
// 500 -> 486, five VGA pairs 3007 -> 2932).
#include <cuda.h>

#include <algorithm>
#include <atomic>
#include <type_traits>

#include "pdflow_iterate.cuh"
#include "pdflow_math.cuh"
#include "pdflow_pack.cuh"
#include "pdflow_region.cuh"
#include "pdflow_tmap.h"

namespace pdflow {

namespace {

using namespace region;

constexpr int kSR = 32;                        // region rows and columns
// Interior and halo (= iterations per launch at most) are launch parameters:
// 24 + 2 x 4 (form 8) or 16 + 2 x 8 (form 9: twice the iterations per launch
// for levels whose launches are latency-bound, at four times the halo work).
constexpr int kSPlane = kSR * kSR;             // floats per shared plane
constexpr int kSThreads = kSR * kSR / 2;       // one thread per pixel pair (512)
constexpr int kSWarps = kSThreads / 32;
// The streamed launches add a producer warpgroup (setmaxnreg works on whole
// warpgroups; one lane of it does the work).  640 threads launch with 96
// registers each; the producer keeps 32 and the consumers take 112, which is
// exactly the launch's total (128 * 32 + 512 * 112 = 640 * 96).
constexpr int kSProducer = 128, kSLaunchRegs = 96, kSProducerRegs = 32, kSConsumerRegs = 112;
static_assert(kSProducer * kSProducerRegs + kSThreads * kSConsumerRegs == (kSProducer + kSThreads) * kSLaunchRegs,
              "the register split is the launch's total");

// staging planes (TMA destinations, in the arena's order): 13 state, 19
// constants; then the six exchange planes
enum { S_DU, S_DV, S_DW, S_UA, S_VA, S_WA, S_PD, S_PUU, S_PUV, S_PVU, S_PVV, S_PWU, S_PWV,
       K_RI, K_RJ, K_DCT, K_DCU, K_DCV, K_DDT, K_DDU, K_DDV, K_MU, K_DUP, K_DVP,
       K_S0, K_S1, K_S2, K_S3, K_S4, K_TU, K_TV, K_TW,
       N_STAGE,
       X_U = N_STAGE, X_V, X_W, Y_U, Y_V, Y_W, N_PLANES };

struct StreamArgs {
    LevelGeom g;
    const float* planes[32];   // direct loads: the 13 source state and 19 constant planes, in the staging order
    unsigned whole;            // strips: units 0 .. whole-1 are strips 0 .. whole-1
    unsigned tier_n[3], tier_p[3];   // strips: then tier i: tier_p[i] pieces of each of the next tier_n[i] strips
    unsigned* work;            // strips: [next unit - grid, CTAs finished], zero between launches
    float* dst[13];            // du dv dw du_acc dv_acc dw_acc pd puu puv pvu pvv pwu pwv (interior written)
    const float* depth_old;
    Params p;
    unsigned kk;
    bool last;
    bool follows;              // the kernel before in the stream is a launch of this level: the constants are final
    int tile, halo;            // interior rows and columns, halo width (tile + 2 halo = kSR)
    unsigned tiles_v;          // tiles per column of tiles
    unsigned tiles;            // tiles per pair
    unsigned total;            // tiles of the launch (tiles * pairs)
    unsigned* status;          // device word: kStreamTimeout when a bounded wait gives up
};

// 4D maps (rows, columns, planes, arena slots) of the 13 source state planes
// and of the 19 constant planes, box = one region of every plane of the group.
struct StreamMaps {
    CUtensorMap state, consts;
};

constexpr unsigned kStreamTimeout = 0x5354524Du;
constexpr uint32_t kStreamWaitLimit = 1u << 22;

// One region of a CTA's walk: its origin, the rows and columns it stores,
// and (strips) where the walk goes next.
struct Tile {
    unsigned y;                  // grid pair index
    int rv0, ru0, iv0, iv1, iu0, iu1;
    bool more;                   // a region to process
    bool carry_in, carry_out;    // strips: reads / writes the column carry
    unsigned k;                  // strips: the unit; tiles: the tile index
    int c1;                      // strips: the unit's end column
};

// What the consumer warps need of a region, as the producer writes it to
// shared memory (two 16-byte reads): its origin, the rows and columns to
// store (low and high halves of a word), the arena slot and flags.
struct Region {
    int rv0, ru0;
    unsigned iv, iu;
    unsigned slot, flags;
    unsigned pad[2];
};
constexpr unsigned kRegMore = 1u, kRegCarryIn = 2u, kRegCarryOut = 4u, kRegLast = 8u, kRegBorder = 16u,
                   kRegFinal = 32u;

__device__ __forceinline__ Region region_of(const StreamArgs& a, const Tile& t)
{
    Region r;
    const unsigned m = t.more && a.g.map ? __ldg(a.g.map + t.y) : t.y;
    const int R = (int)a.g.R, C = (int)a.g.C;
    r.rv0 = t.rv0;
    r.ru0 = t.ru0;
    r.iv = (unsigned)t.iv0 | (unsigned)t.iv1 << 16;
    r.iu = (unsigned)t.iu0 | (unsigned)t.iu1 << 16;
    r.slot = m & kMapSlotMask;
    r.flags = (t.more ? kRegMore : 0u) | (t.carry_in ? kRegCarryIn : 0u) | (t.carry_out ? kRegCarryOut : 0u) |
              (a.last || (a.g.map && (m & kMapLast)) ? kRegLast : 0u) |
              (t.ru0 > 0 && t.ru0 + kSR < C && t.rv0 > 0 && t.rv0 + kSR < R ? 0u : kRegBorder);
    r.pad[0] = r.pad[1] = 0u;
    return r;
}

// Tiles: the launch's tile n (regions of every pair, dealt round-robin).
__device__ __forceinline__ Tile tile_at(const StreamArgs& a, unsigned n)
{
    Tile t;
    t.more = n < a.total;
    t.k = n;
    t.c1 = 0;
    t.carry_in = t.carry_out = false;
    t.y = n / a.tiles;
    const unsigned x = n % a.tiles;
    const int R = (int)a.g.R, C = (int)a.g.C;
    const int tv = (int)(x % a.tiles_v), tu = (int)(x / a.tiles_v);
    t.iv0 = tv * a.tile;
    t.iu0 = tu * a.tile;
    t.iv1 = min(t.iv0 + a.tile, R);
    t.iu1 = min(t.iu0 + a.tile, C);
    t.rv0 = max(t.iv0 - a.halo, 0);
    t.ru0 = max(t.iu0 - a.halo, 0);
    return t;
}

// Strips: unit k, columns [c0, c1) of strip `strip` (strip s is row band
// s % tiles_v of pair s / tiles_v): a whole strip, or piece i of a strip of
// one of the tiers that follow (within a tier, pieces in order of i, then of
// the strip).
struct Segment {
    bool ok;
    unsigned strip;
    int c0, c1;
};
__device__ __forceinline__ Segment segment(const StreamArgs& a, unsigned k)
{
    const int C = (int)a.g.C;
    if (k < a.whole) return {true, k, 0, C};
    unsigned x = k - a.whole, base = a.whole;
#pragma unroll
    for (int i = 0; i < 3; ++i) {
        const unsigned n = a.tier_n[i], m = a.tier_p[i];
        if (x < n * m) {
            const int piece = (int)(x / n);
            return {true, base + x % n, C * piece / (int)m, C * (piece + 1) / (int)m};
        }
        x -= n * m;
        base += n;
    }
    return {false, 0, 0, 0};
}

// Strips: the first region of unit k.  It starts kk columns left of the
// unit's first (their values go stale from the left, one column per
// iteration) or at the image's first column.  Columns up to 32 - kk past the
// origin are exact (all of them when the region reaches the image's last
// column).
__device__ __forceinline__ Tile strip_at(const StreamArgs& a, unsigned k)
{
    Tile t;
    const Segment sg = segment(a, k);
    t.more = sg.ok;
    t.k = k;
    t.c1 = sg.c1;
    const int R = (int)a.g.R, C = (int)a.g.C, K = (int)a.kk;
    const int col = sg.c0;
    t.y = sg.strip / a.tiles_v;
    const int tv = (int)(sg.strip - t.y * a.tiles_v);
    t.iv0 = tv * a.tile;
    t.iv1 = min(t.iv0 + a.tile, R);
    t.rv0 = max(t.iv0 - a.halo, 0);
    t.ru0 = max(col - K, 0);
    const int exact = (t.ru0 + kSR >= C) ? C : t.ru0 + kSR - K;
    t.iu0 = col;
    t.iu1 = min(exact, sg.c1);
    t.carry_in = false;
    t.carry_out = t.iu1 == exact && t.iu1 < sg.c1;   // the next region continues the unit
    return t;
}

// Strips: the region after t within t's unit (t.iu1 < t.c1): the same rows,
// the columns from t's last exact one on, entered with the carry.
__device__ __forceinline__ Tile continue_unit(const StreamArgs& a, Tile t)
{
    const int C = (int)a.g.C, col = t.iu1;
    const int exact = (col + kSR >= C) ? C : col + kSR - (int)a.kk;
    t.ru0 = t.iu0 = col;
    t.iu1 = min(exact, t.c1);
    t.carry_in = true;
    t.carry_out = t.iu1 == exact && t.iu1 < t.c1;
    return t;
}

// The tensor copies of a region into the staging planes, completing on `bar`
// (every consumer warp has read staging).
__device__ __forceinline__ void expect_region(uint32_t bar)
{
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");   // earlier generic reads before async writes
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar),
                 "r"((uint32_t)N_STAGE * (uint32_t)kSPlane * 4u)
                 : "memory");
}
__device__ __forceinline__ void copy_group(const CUtensorMap& map, float* to, uint32_t bar, const Region& r)
{
    asm volatile(
        "cp.async.bulk.tensor.4d.shared::cluster.global.tile.mbarrier::complete_tx::bytes"
        " [%0], [%1, {%2, %3, %4, %5}], [%6];" ::"r"(smem_u32(to)),
        "l"(reinterpret_cast<uint64_t>(&map)), "r"(r.rv0), "r"(r.ru0), "r"(0), "r"((int)r.slot), "r"(bar)
        : "memory");
}
__device__ __forceinline__ void issue_region(const StreamMaps& tm, float* sm, uint32_t bar, const Region& r)
{
    expect_region(bar);
    copy_group(tm.state, sm + S_DU * kSPlane, bar, r);
    copy_group(tm.consts, sm + K_RI * kSPlane, bar, r);
}

// The producer lane: the CTA's walk (tiles blockIdx.x, + gridDim.x, ...; or,
// strips, unit blockIdx.x, then the units it takes from the counter).  Per
// region it waits until every consumer warp has read the staging planes of
// the one before, writes the region's descriptor and starts its copies.  The
// first region's are under way before the CTA's first barrier.  The walk ends
// with a region marked kRegFinal (tiles: the next index is known) or with a
// descriptor without kRegMore (strips: the next unit is taken only when the
// last region of the one before has been issued).
template <bool kStrips>
__device__ __forceinline__ Region walk_region(const StreamArgs& a, const Tile& t)
{
    Region r = region_of(a, t);
    if (!kStrips && t.k + gridDim.x >= a.total) r.flags |= kRegFinal;
    return r;
}
template <bool kStrips>
__device__ __forceinline__ void produce(const StreamArgs& a, const StreamMaps& tm, float* sm, Region* desc,
                                        uint32_t full, uint32_t empty, Tile t)
{
    for (uint32_t n = 1; t.more; ++n) {   // region 0 is on its way (or there is none)
        if constexpr (kStrips) {
            t = t.iu1 < t.c1 ? continue_unit(a, t) : strip_at(a, gridDim.x + atomicAdd(a.work, 1u));
        } else {
            t = tile_at(a, t.k + gridDim.x);
            if (!t.more) return;
        }
        const Region r = walk_region<kStrips>(a, t);
        if (!mbar_wait(empty, (n - 1u) & 1u, kStreamWaitLimit)) {
            atomicExch(a.status, kStreamTimeout);
            mbar_wait(full, (n - 1u) & 1u, kStreamWaitLimit);   // bounded: the copies still in flight
            return;
        }
        *desc = r;
        if (!t.more) {
            asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(full) : "memory");
            break;
        }
        issue_region(tm, sm, full, r);
    }
    // strips: the last CTA to finish (every CTA has taken its last unit)
    // clears the counter for the next launch
    if (kStrips && atomicAdd(a.work + 1, 1u) == gridDim.x - 1) {
        atomicExch(a.work, 0u);
        atomicExch(a.work + 1, 0u);
    }
}

// Barrier of the consumer warps (the producer warp takes no part).
__device__ __forceinline__ void consumer_sync()
{
    asm volatile("bar.sync 1, %0;" ::"n"(kSThreads) : "memory");
}

// carry (strips): [buffer][iteration][u, v, w][region row] of the column
// that the next region of the strip sees on its left
constexpr int kCarryFloats = 2 * 4 * 3 * kSR;

template <bool kStrips, bool kTma = true>
__global__ void __launch_bounds__(kTma ? kSThreads + kSProducer : kSThreads, 1)
    k_iterate_stream(StreamArgs a, const __grid_constant__ StreamMaps tm)
{
    static_assert(kTma || !kStrips, "the strips stream their regions");
    extern __shared__ __align__(128) float sm[];
    __shared__ __align__(8) unsigned long long full_mem, empty_mem;   // staging landed / staging read
    __shared__ __align__(16) Region desc;
    __shared__ unsigned failed;                    // a consumer's wait ran out
    const int t = threadIdx.x;
    const uint32_t full = smem_u32(&full_mem), empty = smem_u32(&empty_mem);
    if constexpr (kTma) {
        Tile first;
        if (t == kSThreads) {
            failed = 0u;
            asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(full));
            asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(empty), "n"(kSWarps));
            asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
            if constexpr (kStrips) first = strip_at(a, blockIdx.x);
            else first = tile_at(a, blockIdx.x);
            desc = walk_region<kStrips>(a, first);
            // the first region: its constants before the wait where they are final
            if (first.more) {
                expect_region(full);
                if (a.follows) copy_group(tm.consts, sm + K_RI * kSPlane, full, desc);
            }
            after_previous_kernel();
            if (first.more) {
                copy_group(tm.state, sm + S_DU * kSPlane, full, desc);
                if (!a.follows) copy_group(tm.consts, sm + K_RI * kSPlane, full, desc);
            } else {
                asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(full) : "memory");
            }
        }
        after_previous_kernel();
        __syncthreads();   // the mbarriers' initialisation before anyone waits on them
        if (t >= kSThreads) {
            asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(kSProducerRegs));
            if (t == kSThreads) allow_next_kernel();
            if (t == kSThreads) produce<kStrips>(a, tm, sm, &desc, full, empty, first);
            return;
        }
        asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(kSConsumerRegs));
    }
    const int c = t >> 4, p = t & 15;              // region column, pixel pair
    const int me = c * kSR + 2 * p;                 // the pair's offset in a shared plane
    const int right = (c + 1 < kSR ? c + 1 : c) * kSR + 2 * p;   // beyond the region: own storage
    const int left = (c > 0 ? c - 1 : c) * kSR + 2 * p;
    const int R = (int)a.g.R, C = (int)a.g.C;
    const float2 zero = make_float2(0.f, 0.f);
    float* carry = sm + N_PLANES * kSPlane;
    const int cc = kSR - 1 - (int)a.kk;              // strips: the column the next region needs
    for (unsigned n = 0;; ++n) {
        Region rg;
        if constexpr (kTma) {
            const bool ok = mbar_wait(full, n & 1u, kStreamWaitLimit);
            rg = desc;
            if (!ok) {   // go through this region's barriers without storing, then leave with the others
                rg.rv0 = rg.ru0 = 0;
                rg.iv = rg.iu = rg.slot = 0u;
                rg.flags = kRegMore;
                failed = 1u;
                atomicExch(a.status, kStreamTimeout);
            }
            if (!(rg.flags & kRegMore)) {
                // as many barriers as a region has, so that a warp whose wait
                // for this descriptor ran out does not wait for the others
                for (unsigned j = 0; j < 2 * a.kk; ++j) consumer_sync();
                break;
            }
        } else {
            rg = region_of(a, tile_at(a, blockIdx.x + n * gridDim.x));
            if (!(rg.flags & kRegMore)) break;
        }
        const size_t po = (size_t)rg.slot * a.g.pstride;
        const int u = rg.ru0 + c, v0 = rg.rv0 + 2 * p;
        const bool live = u < C && v0 < R;           // v0 < R implies v0 + 1 < R (R even)
        const PairPlace place{u == 0, u == C - 1, v0 == 0, v0 + 1 == R - 1};
        const bool last_launch = rg.flags & kRegLast;

        // the pair's value of plane k: from the staging copy, or loaded
        // directly (zero outside the image, as the tensor copy fills)
        auto ld2s = [&](int k) {
            if constexpr (kTma) return *reinterpret_cast<const float2*>(sm + k * kSPlane + me);
            return live ? __ldg(reinterpret_cast<const float2*>(at(a.planes[k], po) + v0 + (size_t)u * (size_t)R))
                        : zero;
        };
        PairState s{ld2s(S_DU), ld2s(S_DV), ld2s(S_DW), ld2s(S_UA), ld2s(S_VA), ld2s(S_WA), ld2s(S_PD),
                    ld2s(S_PUU), ld2s(S_PUV), ld2s(S_PVU), ld2s(S_PVV), ld2s(S_PWU), ld2s(S_PWV)};
        const PairConsts k{ld2s(K_RI), ld2s(K_RJ), ld2s(K_DCT), ld2s(K_DCU), ld2s(K_DCV), ld2s(K_DDT), ld2s(K_DDU),
                           ld2s(K_DDV), ld2s(K_MU), ld2s(K_DUP), ld2s(K_DVP), ld2s(K_S0), ld2s(K_S1), ld2s(K_S2),
                           ld2s(K_S3), ld2s(K_S4), ld2s(K_TU), ld2s(K_TV), ld2s(K_TW)};
        if constexpr (kTma) {   // this warp has read staging: the next region may land once all have
            __syncwarp();
            if ((t & 31) == 0) asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(empty) : "memory");
        }
        // the left neighbour's exchange values: the carry of the previous
        // region (strips, first column) or the exchange planes; j advances
        // the carry by one iteration
        const bool from_carry = kStrips && (rg.flags & kRegCarryIn) && c == 0;
        const float* yl = from_carry ? carry + ((n + 1) & 1) * (4 * 3 * kSR) + 2 * p : sm + Y_U * kSPlane + left;
        const int yl_k = from_carry ? kSR : kSPlane, yl_j = from_carry ? 3 * kSR : 0;
        float* yc = carry + (n & 1) * (4 * 3 * kSR) + 2 * p;
        const bool to_carry = kStrips && (rg.flags & kRegCarryOut) && c == cc;

        const PairDerived d(k);
        // the iterations, with the image-border cases (kBorder) or, for a region
        // that touches no image border, without them (the same expressions)
        struct Hooks {
            const float* yl;
            int yl_k;
            float* yc;
            bool to_carry;
            __device__ __forceinline__ void sync() const { consumer_sync(); }
            __device__ __forceinline__ void carry(float2 yu, float2 yv, float2 yw) const
            {
                if (to_carry) {
                    *reinterpret_cast<float2*>(yc) = yu;
                    *reinterpret_cast<float2*>(yc + kSR) = yv;
                    *reinterpret_cast<float2*>(yc + 2 * kSR) = yw;
                }
            }
            __device__ __forceinline__ const float* left(int c) const { return yl + c * yl_k; }
        };
        // saturated after the level's last iteration (strips: inside the loop, tiles:
        // after it; the strips' loop with it outside takes 64 VGA pairs from 32.1 to
        // 33.2 ms, the tiles' with it inside five from 3.44 to 3.46 ms)
        auto finish = [&]() {
            if (last_launch && live)
                saturate_pair(s, k, __ldg(reinterpret_cast<const float2*>(at(a.depth_old, po) + v0 +
                                                                          (size_t)u * (size_t)R)));
        };
        auto iterate = [&](auto border) {
            for (unsigned j = 0; j < a.kk; ++j) {
                iterate_pair<decltype(border)::value, kSR / 2, kStrips>(
                    s, k, d, sm + X_U * kSPlane, sm + Y_U * kSPlane, kSPlane, me, right, place, a.p.lambda_i,
                    a.p.lambda_d, Hooks{yl + (int)j * yl_j, yl_k, yc + (int)j * (3 * kSR), to_carry});
                if (kStrips && j + 1 == a.kk) finish();
            }
        };
        if (rg.flags & kRegBorder) iterate(std::true_type{});   // the same for the whole CTA
        else iterate(std::false_type{});
        const bool lost = kTma && *reinterpret_cast<volatile unsigned*>(&failed);   // set before this region's barriers
        if (lost) break;

        if (!kStrips) finish();
        // ---- the interior to the destination buffer ----
        if (live && v0 >= int(rg.iv & 0xffffu) && v0 < int(rg.iv >> 16) && u >= int(rg.iu & 0xffffu) &&
            u < int(rg.iu >> 16)) {
            const size_t gi = (size_t)v0 + (size_t)u * (size_t)R;
            const float2 st[13] = {s.du, s.dv, s.dw, s.ua, s.va, s.wa, s.pd, s.puu, s.puv, s.pvu, s.pvv, s.pwu, s.pwv};
#pragma unroll
            for (int q = 0; q < 13; ++q) *reinterpret_cast<float2*>(at(a.dst[q], po) + gi) = st[q];
        }
        if (!kStrips && (rg.flags & kRegFinal)) break;
        // the next region's first exchange stores (X planes, last read before
        // this region's last barrier) and its first Y and carry stores (after
        // its own first barrier) need no barrier here
    }
}

}  // namespace

size_t stream_smem_bytes() { return sizeof(float) * (N_PLANES * kSPlane + kCarryFloats); }

namespace {

// Regions of a unit's columns [c0, c1) (strip_at, continue_unit).
unsigned unit_regions(int c0, int c1, int C, int kk)
{
    unsigned n = 0;
    for (int col = c0; col < c1; ++n) {
        const int ru0 = n ? col : std::max(col - kk, 0);
        col = std::min(ru0 + kSR >= C ? C : ru0 + kSR - kk, c1);
    }
    return n;
}

// When the last CTA ends, in regions: CTAs take units in order as they finish.
// CTAs that end at the same time are one entry.  Regions take a little longer or
// shorter with the data, so a tenth of a last unit is added: short last units
// even that out.
class UnitQueue {
public:
    explicit UnitQueue(unsigned grid) { at_[0] = {0.f, grid}; }
    // n strips of m equal pieces each, piece by piece.
    void add(unsigned n, unsigned m, unsigned C, unsigned kk)
    {
        for (unsigned i = 0; i < m && n > 0; ++i)
            add(n, kUnitStart + float(unit_regions(int(C * i / m), int(C * (i + 1) / m), int(C), int(kk))));
    }
    float end() const { return at_[used_ - 1].time + 0.1f * last_; }

private:
    static constexpr float kUnitStart = 0.15f;   // what starting a unit costs beyond its regions
    static constexpr int kMost = 64;
    struct Group {
        float time;
        unsigned ctas;
    };
    Group at_[kMost];
    int used_ = 1;
    float last_ = 0.f;
    void add(unsigned n, float cost)
    {
        last_ = cost;
        while (n > 0) {
            const unsigned k = std::min(n, at_[0].ctas);
            const float time = at_[0].time + cost;
            n -= k;
            if ((at_[0].ctas -= k) == 0) {
                for (int i = 1; i < used_; ++i) at_[i - 1] = at_[i];
                --used_;
            }
            int i = 0;   // the first entry that ends no earlier
            while (i < used_ && at_[i].time < time - 1e-3f) ++i;
            if (i < used_ && at_[i].time < time + 1e-3f) {
                at_[i].ctas += k;
            } else if (used_ == kMost) {   // never seen: keep the bound, lose the detail
                at_[used_ - 1].ctas += k;
                at_[used_ - 1].time = std::max(at_[used_ - 1].time, time);
            } else {
                for (int q = used_; q > i; --q) at_[q] = at_[q - 1];
                at_[i] = {time, k};
                ++used_;
            }
        }
    }
};

float units_end(const StripUnits& u, unsigned C, unsigned kk, unsigned grid)
{
    UnitQueue q(grid);
    q.add(u.whole, 1, C, kk);
    for (int i = 0; i < 3; ++i) q.add(u.tier_n[i], u.tier_p[i], C, kk);
    return q.end();
}

StripUnits plan_units(unsigned strips_n, unsigned C, unsigned kk, unsigned grid)
{
    StripUnits su{};
    if (strips_n == 0 || C == 0 || kk == 0 || 2 * kk >= (unsigned)kSR || grid == 0) return su;
    const unsigned most = (C + (kSR - 2 * kk) - 1) / (kSR - 2 * kk);
    const unsigned regions = (C + (kSR - kk) - 1) / (kSR - kk);   // of a whole strip walked with the carry
    // many strips: whole ones, then the last grid / 8 in 2 pieces, in 4 and in 8
    unsigned left = strips_n;
    const unsigned tn[3] = {grid / 8, grid / 8, regions >= 16 ? grid / 4 : grid / 8}, tp[3] = {2, 4, 8};
    for (int i = 2; i >= 0; --i) {
        su.tier_n[i] = strips_n > grid ? std::min(tn[i], left) : 0u;
        su.tier_p[i] = std::min(tp[i], most);
        left -= su.tier_n[i];
    }
    if (strips_n <= grid) {
        su.tier_n[0] = strips_n;
        su.tier_p[0] = std::max(1u, std::min(grid / strips_n, most));
        left = 0;
    }
    su.whole = left;
    if (strips_n > 4 * grid) return su;
    // few strips a CTA: the first n in p1 pieces, the rest in p2 >= p1, of pieces
    // that waste few regions on restarts, if that ends clearly earlier (differences
    // below 4 % are within the model's error: 10 VGA pairs at 480x640, 32.9 against
    // 32.1 regions, took 3.55 against 3.61 ms)
    float best = units_end(su, C, kk, grid) * 0.96f;
    unsigned cuts[32], n_cuts = 0, fewest = ~0u, total[33];
    for (unsigned m = 1; m <= std::min(most, 32u); ++m) {
        total[m] = 0;
        for (unsigned i = 0; i < m; ++i)
            total[m] += unit_regions(int(C * i / m), int(C * (i + 1) / m), int(C), int(kk));
        fewest = std::min(fewest, total[m]);
    }
    for (unsigned m = 1; m <= std::min(most, 32u); ++m)
        if (total[m] * 8 <= fewest * 9) cuts[n_cuts++] = m;
    const unsigned step = std::max(1u, strips_n / 32);
    for (unsigned i = 0; i < n_cuts; ++i)
        for (unsigned j = i; j < n_cuts; ++j)
            for (unsigned n = i == j ? strips_n : step; n <= strips_n; n += step) {
                // no plan ends before its work spread evenly
                if (float(n * total[cuts[i]] + (strips_n - n) * total[cuts[j]]) >= best * float(grid)) continue;
                const StripUnits c{0, {n, strips_n - n, 0}, {cuts[i], cuts[j], 1}};
                const float end = units_end(c, C, kk, grid);
                if (end < best) {
                    best = end * 0.999f;
                    su = c;
                }
            }
    return su;
}

}  // namespace

static thread_local unsigned long long plans = 0;
unsigned long long strip_plans() { return plans; }

// Strip units.  Each piece of a strip recomputes a left halo, so many strips
// (over four a CTA) stay whole but for a short tail: on 64-pair VGA solves (1
// 280 strips of 23 regions at 480x640, 640 of 12 at 240x320) the last grid /
// 4, grid / 2 and grid strips in 8, 4 and 2 pieces took 38.06 ms, these tiers
// 37.3 ms.  With fewer the last round is nearly empty however the tail is cut
// (24 pairs at 240x320: 240 strips of 12 regions on 152 CTAs end after 24.3
// regions, the work is 18.9), so the cuts are chosen by when the queue ends:
// there 200 strips in 3 pieces and 40 in 4 end after 19.8 (85 iterations 2.76 ->
// 2.26 ms on a GB300; 13 pairs at 480x640 5.10 -> 4.56, 20 pairs 7.47 -> 6.78).
// The choice is a function of its arguments; the last 64 are kept (a search takes
// up to 0.5 ms of host time).
StripUnits strip_units(unsigned strips_n, unsigned C, unsigned kk, unsigned grid)
{
    struct Kept {
        unsigned key[4];
        StripUnits units;
    };
    thread_local Kept kept[64] = {};
    thread_local unsigned next = 0;
    const unsigned key[4] = {strips_n, C, kk, grid};
    for (const Kept& k : kept)
        if (std::equal(key, key + 4, k.key)) return k.units;
    ++plans;
    const StripUnits su = plan_units(strips_n, C, kk, grid);
    Kept& k = kept[next++ % 64u];
    std::copy(key, key + 4, k.key);
    k.units = su;
    return su;
}

float strips_end(const LevelGeom& g, unsigned ctas)
{
    constexpr unsigned kk = 4, rows = kSR - 2 * kk;
    const unsigned strips_n = g.pairs * ((g.R + rows - 1) / rows);
    return units_end(strip_units(strips_n, g.C, kk, ctas), g.C, kk, ctas);
}

// The direct loads and stores move a pixel pair as one float2: even rows and
// pair spacing, 8-byte aligned planes.
bool stream_direct_eligible(const LevelGeom& g, const LevelConsts& L, const State& src, const State& dst)
{
    if (g.R % 2 != 0 || g.slots == 0 || g.pstride % 2 != 0) return false;
    const float* cg[19] = {L.ri, L.rj, L.dct, L.dcu, L.dcv, L.ddt, L.ddu, L.ddv, L.mu, L.du_prev, L.dv_prev,
                           L.qs[0], L.qs[1], L.qs[2], L.qs[3], L.qs[4], L.qs[5], L.qs[6], L.qs[7]};
    const float* sd[26] = {src.du, src.dv, src.dw, src.dua, src.dva, src.dwa, src.pd, src.puu, src.puv,
                           src.pvu, src.pvv, src.pwu, src.pwv, dst.du, dst.dv, dst.dw, dst.dua, dst.dva,
                           dst.dwa, dst.pd, dst.puu, dst.puv, dst.pvu, dst.pvv, dst.pwu, dst.pwv};
    for (const float* q : cg)
        if (!q || reinterpret_cast<uintptr_t>(q) % 8u != 0) return false;
    for (const float* q : sd)
        if (!q || reinterpret_cast<uintptr_t>(q) % 8u != 0) return false;
    return true;
}

// Whether the kernels that stream their regions have the registers their split
// counts on (prepare_stream_tiles): with another count the consumers' setmaxnreg
// would wait for what the launch did not bring, so they do not run and levels take
// the tiles on direct loads.  The build refuses such a compiler's output.
static std::atomic<bool> streamed_copies{false};

static bool copies_eligible(const LevelGeom& g, const LevelConsts& L, const State& src, const State& dst)
{
    return streamed_copies && quads_eligible(g, L, src, dst);
}

bool stream_eligible(const LevelGeom& g, const LevelConsts& L, const State& src, const State& dst, int form)
{
    if (form == 7 ? quads_eligible(g, L, src, dst) : copies_eligible(g, L, src, dst)) return true;
    return (form == 8 || form == 9) && stream_direct_eligible(g, L, src, dst);
}

cudaError_t prepare_stream_tiles()
{
    cudaError_t e = cudaSuccess;
    for (const void* k : {(const void*)k_iterate_stream<false>, (const void*)k_iterate_stream<true>,
                          (const void*)k_iterate_stream<false, false>}) {
        if (e == cudaSuccess)
            e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)stream_smem_bytes());
        if (e == cudaSuccess) e = cudaFuncSetAttribute(k, cudaFuncAttributePreferredSharedMemoryCarveout, 100);
    }
    bool exact = e == cudaSuccess;
    for (const void* k : {(const void*)k_iterate_stream<false>, (const void*)k_iterate_stream<true>}) {
        cudaFuncAttributes fa{};
        if (e == cudaSuccess) e = cudaFuncGetAttributes(&fa, k);
        exact = exact && fa.numRegs == kSLaunchRegs;
    }
    if (e == cudaSuccess) streamed_copies = exact;
    return e;
}

cudaError_t launch_iterate_stream(LevelGeom g, LevelConsts L, State src, State dst, Params p, const float* depth_old,
                                  unsigned kk, bool last, cudaStream_t st, unsigned* status, unsigned ctas,
                                  StreamLayout layout, bool follows)
{
    // the region stays 32 x 32; rows of region origins stay multiples of 4
    // (16-byte tensor-copy coordinates): halo 4 (interior 24) or 8 (interior 16)
    const bool strips = layout == StreamLayout::Strips;
    const int kSH = layout == StreamLayout::Tiles16 ? 8 : 4, kST = kSR - 2 * kSH;
    // the tensor copies need the quad tiles' preconditions (16-byte aligned
    // planes at one spacing, rows % 4 == 0); the tiles also run on direct loads
    // where the rows are even
    const bool tma = copies_eligible(g, L, src, dst);
    if (kk == 0 || kk > (unsigned)kSH || !status || ctas == 0 || reinterpret_cast<uintptr_t>(depth_old) % 8u != 0 ||
        !(tma || (!strips && stream_direct_eligible(g, L, src, dst))))
        return cudaErrorInvalidValue;
    StreamArgs a;
    a.g = g;
    float* d13[13] = {dst.du, dst.dv, dst.dw, dst.dua, dst.dva, dst.dwa, dst.pd,
                      dst.puu, dst.puv, dst.pvu, dst.pvv, dst.pwu, dst.pwv};
    for (int k = 0; k < 13; ++k) a.dst[k] = d13[k];
    a.depth_old = depth_old;
    a.p = p;
    a.kk = kk;
    a.last = last;
    a.follows = follows;
    a.status = status;
    a.tile = kST;
    a.halo = kSH;
    a.tiles_v = (g.R + kST - 1) / kST;
    a.tiles = a.tiles_v * ((g.C + kST - 1) / kST);
    a.total = a.tiles * g.pairs;
    const unsigned grid = ctas < a.total ? ctas : a.total;
    const StripUnits su = strips ? strip_units(g.pairs * a.tiles_v, g.C, kk, grid) : StripUnits{};
    a.whole = su.whole;
    for (int i = 0; i < 3; ++i) {
        a.tier_n[i] = su.tier_n[i];
        a.tier_p[i] = su.tier_p[i];
    }
    a.work = status + 2;
    // the runs of planes (quads_eligible checked that each is equally spaced)
    const float* sg[13] = {src.du, src.dv, src.dw, src.dua, src.dva, src.dwa, src.pd,
                           src.puu, src.puv, src.pvu, src.pvv, src.pwu, src.pwv};
    const float* cg[19] = {L.ri, L.rj, L.dct, L.dcu, L.dcv, L.ddt, L.ddu, L.ddv, L.mu, L.du_prev, L.dv_prev,
                           L.qs[0], L.qs[1], L.qs[2], L.qs[3], L.qs[4], L.qs[5], L.qs[6], L.qs[7]};
    for (int k = 0; k < 13; ++k) a.planes[k] = sg[k];
    for (int k = 0; k < 19; ++k) a.planes[13 + k] = cg[k];
    StreamMaps maps{};
    if (!tma) {
        k_iterate_stream<false, false><<<grid, kSThreads, stream_smem_bytes(), st>>>(a, maps);
        return cudaGetLastError();
    }
    size_t ss = 0, cs = 0;
    if (!equally_spaced(sg, 13, &ss) || !equally_spaced(cg, 19, &cs) ||
        !encode_plane_group(&maps.state, sg[0], 13, ss, g.R, g.C, g.slots, g.pstride, kSR, kSR) ||
        !encode_plane_group(&maps.consts, cg[0], 19, cs, g.R, g.C, g.slots, g.pstride, kSR, kSR))
        return cudaErrorInvalidValue;
    return launch_overlapped(strips ? k_iterate_stream<true> : k_iterate_stream<false>, dim3(grid),
                             dim3(kSThreads + kSProducer), stream_smem_bytes(), st, a, maps);
}

}  // namespace pdflow
