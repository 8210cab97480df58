// One iteration of a 32-bit-float primal-dual pair of pixels held in registers,
// shared by the register-resident region kernels (pdflow_ptiles.cu,
// pdflow_resident.cu).
//
// A thread owns a vertical pixel pair (rows 2p, 2p + 1 of a region column);
// kLanes consecutive threads are one column of 2 kLanes rows.  Its state and
// the level's constants are in registers and it computes both pixels in packed
// FP32x2.  The row below the pair (dual step) and above it (primal step) come
// by warp shuffles inside the column's lanes; the column to the right (dual)
// and to the left (primal) through shared exchange planes, into which each
// thread publishes what its neighbours read (U = du_acc + du_prev, V = dv_acc
// + dv_prev, W = dw_acc; ri * the u-component of each TV dual).  These are the
// same rounded expressions the reference evaluates (computeGradient,
// computeDivergence: pdflow_cudalib.cu:935-1013).
#pragma once
#include <cuda_runtime.h>

#include "pdflow_math.cuh"
#include "pdflow_pack.cuh"

namespace pdflow {
namespace region {

using namespace pack;

__device__ __forceinline__ float clamp1(float pd) { return (fabsf(pd) > 1.f) ? ((pd > 1.f) ? 1.f : -1.f) : pd; }

// The three TV duals' projections onto the unit disc (updateDualVariables,
// pdflow_cudalib.cu:813-887) for both pixels of a pair, with disc_factor's
// expressions in packed FP32x2.  With kVote a warp whose 64 pixels have all three
// duals inside the disc (where the factors are 1 and the values stay) skips
// them: one vote for the three.  That pays where launches are many regions a CTA
// (the strips; GB300, against no vote: 64 VGA pairs 36.83 -> 36.62 ms, 16
// warm-started ones 8.94 -> 8.77; a vote a dual instead: 36.71, 8.87), and costs
// where a launch's time is its dependent chain (one VGA pair 1.020 -> 1.028 ms,
// five as tiles 3.71 -> 3.76).  A thread with a sum beyond disc_factor's range
// takes the scalar form.
struct Disc2 {
    float2 s;
    __device__ __forceinline__ Disc2(float2 a, float2 b)
    {
        const float2 hi = make_float2(max_nan(fabsf(a.x), fabsf(b.x)), max_nan(fabsf(a.y), fabsf(b.y)));
        const float2 lo = make_float2(fminf(fabsf(a.x), fabsf(b.x)), fminf(fabsf(a.y), fabsf(b.y)));
        s = fm2(hi, hi, mul2(lo, lo));
    }
    __device__ __forceinline__ float peak() const { return max_nan(s.x, s.y); }
    __device__ __forceinline__ void apply(float2& a, float2& b) const
    {
        const float2 f = make_float2(rsqrt_min1(s.x), rsqrt_min1(s.y));
        a = mul2(a, f);
        b = mul2(b, f);
    }
};
template <bool kVote>
__device__ __forceinline__ void project_duals(float2& puu, float2& puv, float2& pvu, float2& pvv, float2& pwu,
                                              float2& pwv)
{
    const Disc2 u(puu, puv), v(pvu, pvv), w(pwu, pwv);
    const float peak = max_nan(max_nan(u.peak(), v.peak()), w.peak());
    if (kVote && __all_sync(0xffffffffu, peak < 0.999f)) return;
    if (peak < kDiscLimit) {
        u.apply(puu, puv);
        v.apply(pvu, pvv);
        w.apply(pwu, pwv);
    } else {
        project_disc(puu.x, puv.x);
        project_disc(puu.y, puv.y);
        project_disc(pvu.x, pvv.x);
        project_disc(pvu.y, pvv.y);
        project_disc(pwu.x, pwv.x);
        project_disc(pwu.y, pwv.y);
    }
}

// L1 photometric shrinkage (pdflow_cudalib.cu:906-923) for both pixels of a
// pair: the step taken off du (dv) is the quotient a1 of / den inside the
// threshold and a1 with the sign of `of` outside it (du - (-a1) is du + a1),
// so one packed subtraction serves all three cases.  The quotients are
// div_rcp's in packed FP32x2, from na1 = -a1 and nrden = -RN(1 / den).
__device__ __forceinline__ float2 shrink_step2(float2 of, float2 den, float2 nrden, float2 na1, bool outx, bool outy)
{
    const float2 na = mul2(na1, of);
    const float2 q0 = mul2(na, nrden);
    const float2 q1 = fm2(fm2(q0, den, na), nrden, q0);
    const float2 q2 = fm2(fm2(q1, den, na), nrden, q1);
    return make_float2(outx ? signed_step(na1.x, of.x) : q2.x, outy ? signed_step(na1.y, of.y) : q2.y);
}
__device__ __forceinline__ void shrink_rcp2(float2& du, float2& dv, float2 of, float2 th, float2 den, float2 nrden,
                                            float2 na1, float2 nb1)
{
    const bool outx = fabsf(of.x) > th.x, outy = fabsf(of.y) > th.y;
    du = sub2(du, shrink_step2(of, den, nrden, na1, outx, outy));
    dv = sub2(dv, shrink_step2(of, den, nrden, nb1, outx, outy));
}

// The 13 state and 19 constant planes of a pair, in the arena's order.
struct PairState {
    float2 du, dv, dw, ua, va, wa, pd, puu, puv, pvu, pvv, pwu, pwv;
};
struct PairConsts {
    float2 ri, rj, dct, dcu, dcv, ddt, ddu, ddv, mu, dup, dvp, s0, s1, s2, s3, s4, tu, tv, tw;
};
// What a pair derives from its constants once.
struct PairDerived {
    float2 mudu, mudv, th, den, nrden, na1, nb1;   // the shrinkage's, pdflow_math.cuh
    bool rcp_ok;
    __device__ __forceinline__ explicit PairDerived(const PairConsts& k)
    {
        mudu = mul2(k.mu, k.ddu);
        mudv = mul2(k.mu, k.ddv);
        const float2 a1 = mul2(k.tu, k.dcu), b1 = mul2(k.tv, k.dcv);
        th = fm2(a1, k.dcu, mul2(b1, k.dcv));
        den = make_float2(add(th.x, 1e-10f), add(th.y, 1e-10f));
        nrden = make_float2(-__frcp_rn(den.x), -__frcp_rn(den.y));
        na1 = neg2(a1);
        nb1 = neg2(b1);
        rcp_ok = shrink_rcp_level_ok(a1.x, b1.x, th.x, den.x) && shrink_rcp_level_ok(a1.y, b1.y, th.y, den.y);
    }
};
// Where the pair lies in the image.
struct PairPlace {
    bool fu, lu, fv, lv;   // first / last column, first row (of the pair's .x), last row (of its .y)
};

// One iteration.  X: the three planes of the dual step's published values, me
// and right the pair's and its right neighbour's offsets in a plane (the own
// one beyond the region: read, then not needed); Y: the primal step's.  kBorder:
// the region touches the image border; kVote: project_duals'.  h.sync() is the barrier of the threads
// that exchange, h.carry(yu, yv, yw) sees the published primal-step values, and
// h.left(k) is where the left neighbour's value of component k is read.
template <bool kBorder, int kLanes, bool kVote, class Hooks>
__device__ __forceinline__ void iterate_pair(PairState& s, const PairConsts& k, const PairDerived& d, float* X,
                                             float* Y, int plane, int me, int right, const PairPlace& at, float li,
                                             float ld, Hooks h)
{
    const float2 li2 = make_float2(li, li), ld2 = make_float2(ld, ld), two = make_float2(2.f, 2.f);
    const float2 zero = make_float2(0.f, 0.f);
    // ---------------- dual step (computeGradient + updateDualVariables) ----------------
    {
        const float2 U = add2(s.ua, k.dup), V = add2(s.va, k.dvp);
        *reinterpret_cast<float2*>(X + me) = U;
        *reinterpret_cast<float2*>(X + plane + me) = V;
        *reinterpret_cast<float2*>(X + 2 * plane + me) = s.wa;
        const float Ub = __shfl_down_sync(0xffffffffu, U.x, 1, kLanes);   // the next pair's first row
        const float Vb = __shfl_down_sync(0xffffffffu, V.x, 1, kLanes);
        const float Wb = __shfl_down_sync(0xffffffffu, s.wa.x, 1, kLanes);
        h.sync();
        // borders by selects, not branches (the neighbour slot at the
        // region's right edge is the thread's own: read, then dropped)
        float2 gu1 = mul2(k.ri, sub2(*reinterpret_cast<const float2*>(X + right), U));
        float2 gv1 = mul2(k.ri, sub2(*reinterpret_cast<const float2*>(X + plane + right), V));
        float2 gw1 = mul2(k.ri, sub2(*reinterpret_cast<const float2*>(X + 2 * plane + right), s.wa));
        if (kBorder && at.lu) {
            gu1 = zero;
            gv1 = zero;
            gw1 = zero;
        }
        float2 gu2 = mul2(k.rj, sub2(make_float2(U.y, Ub), U));
        float2 gv2 = mul2(k.rj, sub2(make_float2(V.y, Vb), V));
        float2 gw2 = mul2(k.rj, sub2(make_float2(s.wa.y, Wb), s.wa));
        if (kBorder && at.lv) {
            gu2.y = 0.f;
            gv2.y = 0.f;
            gw2.y = 0.f;
        }
        const float2 data = fm2(k.ddv, s.va, fm2(k.ddu, s.ua, sub2(k.ddt, s.wa)));
        s.pd = fm2(k.s0, data, s.pd);
        s.puu = fm2(k.s1, gu1, s.puu);
        s.puv = fm2(k.s2, gu2, s.puv);
        s.pvu = fm2(k.s1, gv1, s.pvu);
        s.pvv = fm2(k.s2, gv2, s.pvv);
        s.pwu = fm2(k.s3, gw1, s.pwu);
        s.pwv = fm2(k.s4, gw2, s.pwv);
        s.pd.x = clamp1(s.pd.x);
        s.pd.y = clamp1(s.pd.y);
        project_duals<kVote>(s.puu, s.puv, s.pvu, s.pvv, s.pwu, s.pwv);
    }
    // ---------------- primal step (computeDivergence + updatePrimalVariables) ----------------
    {
        const float2 yu = mul2(k.ri, s.puu), yv = mul2(k.ri, s.pvu), yw = mul2(k.ri, s.pwu);
        *reinterpret_cast<float2*>(Y + me) = yu;
        *reinterpret_cast<float2*>(Y + plane + me) = yv;
        *reinterpret_cast<float2*>(Y + 2 * plane + me) = yw;
        h.carry(yu, yv, yw);
        const float2 zu = mul2(k.rj, s.puv), zv = mul2(k.rj, s.pvv), zw = mul2(k.rj, s.pwv);
        const float zua = __shfl_up_sync(0xffffffffu, zu.y, 1, kLanes);   // the previous pair's second row
        const float zva = __shfl_up_sync(0xffffffffu, zv.y, 1, kLanes);
        const float zwa = __shfl_up_sync(0xffffffffu, zw.y, 1, kLanes);
        h.sync();
        const float2 pu_[3] = {s.puu, s.pvu, s.pwu}, pv_[3] = {s.puv, s.pvv, s.pwv};
        const float2 zm_[3] = {make_float2(zua, zu.x), make_float2(zva, zv.x), make_float2(zwa, zw.x)};
        float2 div[3];
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            const float2 ym = neg2(*reinterpret_cast<const float2*>(h.left(c)));
            float2 g = fm2(k.ri, pu_[c], ym);
            // first / last / inner column
            if constexpr (kBorder) g = at.fu ? mul2(k.ri, pu_[c]) : (at.lu ? ym : g);
            float2 e = add2(g, fm2(k.rj, pv_[c], neg2(zm_[c])));
            if constexpr (kBorder) {
                if (at.fv) e.x = fm(k.rj.x, pv_[c].x, g.x);
                if (at.lv) e.y = fm(-k.rj.x, pv_[c].x, g.y);
            }
            div[c] = e;
        }
        const float2 du_old = s.du, dv_old = s.dv, dw_old = s.dw;
        s.du = fm2(neg2(k.tu), fm2(d.mudu, s.pd, neg2(mul2(li2, div[0]))), s.du);
        s.dv = fm2(neg2(k.tv), fm2(d.mudv, s.pd, neg2(mul2(li2, div[1]))), s.dv);
        {
            // per lane: see pdflow_pack.cuh on contraction of packed products
            const float2 tq = fm2(neg2(k.mu), s.pd, neg2(mul2(ld2, div[2])));
            s.dw.x = add(s.dw.x, mul(-k.tw.x, tq.x));
            s.dw.y = add(s.dw.y, mul(-k.tw.y, tq.y));
        }
        const float2 of = fm2(k.dcv, s.dv, fm2(k.dcu, s.du, k.dct));
        // quotients by the reciprocal when the whole warp is in its range
        if (__all_sync(0xffffffffu, d.rcp_ok && shrink_rcp_ok(of.x) && shrink_rcp_ok(of.y))) {
            shrink_rcp2(s.du, s.dv, of, d.th, d.den, d.nrden, d.na1, d.nb1);
        } else {
            shrink(s.du.x, s.dv.x, of.x, d.th.x, -d.na1.x, -d.nb1.x);
            shrink(s.du.y, s.dv.y, of.y, d.th.y, -d.na1.y, -d.nb1.y);
        }
        s.ua = fm2(two, s.du, neg2(du_old));
        s.va = fm2(two, s.dv, neg2(dv_old));
        s.wa = fm2(two, s.dw, neg2(dw_old));
    }
    // no barrier here: this iteration's exchange reads happen before the next
    // one's first barrier, and the next stores to the same planes after it
}

// saturateVariables (pdflow_cudalib.cu:1018-1038) after the level's last
// iteration; z = the old frame's depth at the pair.
__device__ __forceinline__ void saturate_pair(PairState& s, const PairConsts& k, float2 z)
{
    saturate(s.du.x, s.dv.x, s.dw.x, k.dup.x, k.dvp.x, z.x);
    saturate(s.du.y, s.dv.y, s.dw.y, k.dup.y, k.dvp.y, z.y);
}

}  // namespace region
}  // namespace pdflow
