// Gay-Berne family: gb_, gbr_, gbw_, gbc_, gbwc_ (fortran/force.f90:237-1030),
// FP32 per pair with (mu, nu) as parameters (the reference fixes (1,2) at :240).
//
// As in the reference, the shape (sig_x, sig_z) and energy (eps_x, eps_z)
// anisotropies are those of particle I. A per-particle prep pass hoists what
// depends on one particle only: the body z axis u (first column of the
// reference's U1 formula, :343-349), chi, chi' and 1/eps_z.
//
// The per-particle prep (gb_prep_one, step_epi.cuh) puts each particle's
// position and axis in one 32-byte record, so the range test reads them in
// one load.
//
// Near contact the envelope (r - sigma + 1)^-13 amplifies the rounding of the
// contact distance sigma = sig_x / sqrt(g) thirteenfold, and g = 1 - h cancels
// down to (1 - chi) / (1 + chi) for end-to-end pairs, so FP32 rounding of h
// reaches the 1e-5 force tolerance there. The range test therefore sorts the
// pairs it keeps into two classes: pairs within SG_GB_NEAR of contact are queued
// separately and evaluated with g, sigma and r - sigma in double-float
// arithmetic (from u and chi to 48 bits); the others in FP32.
// stats[3] (the fallbacks field of sg_ecp_stats) counts the precise class.
#include <algorithm>
#include <climits>
#include <cmath>

// The precise class: pairs with r below the approximate contact distance plus
// this margin (r - sigma + 1 < 1.02: overlapping pairs, where the envelope's
// amplification of the contact distance's rounding is largest).
#ifndef SG_GB_NEAR
#define SG_GB_NEAR 0.02f
#endif

#include "pair_common.cuh"
#include "dfloat.cuh"
#include "f32x2.cuh"
#include "step_epi.cuh"

namespace {

__global__ void k_gb_prep(int n, const float4* __restrict__ pos, const float4* __restrict__ quat,
                          const float4* __restrict__ shape, const float4* __restrict__ eshape, float muinv,
                          float4* prep) {
    int p = blockIdx.x * blockDim.x + threadIdx.x;
    if (p >= n) return;
    gb_prep_one(n, p, pos[p], quat[p], shape[p], eshape[p], muinv, prep);
}

// Shape term g = 1 - (chi/2) [sp^2 / (1 + chi uu) + sm^2 / (1 - chi uu)] / r^2
// (force.f90:266-306) in double-float, as
// 1 - (chi/2) [sp^2 (1 - chi uu) + sm^2 (1 + chi uu)] / [(1 - (chi uu)^2) r^2],
// from u and chi as hi + lo; rsq (r^2) is returned too.
SG_DEV dfl gb_shape_g_df(float3 r, float3 U1, float3 U1l, float3 U2, float3 U2l, dfl chi, dfl& rsq) {
    const dfl ru1 = df_dot3_lo(r, U1, U1l), ru2 = df_dot3_lo(r, U2, U2l), uu = df_dot3_dd(U1, U1l, U2, U2l);
    rsq = df_dot3(r, r);
    const dfl sp = df_add(ru1, ru2), sm = df_sub(ru1, ru2);
    const dfl cuu = df_mul(chi, uu);
    const dfl omc = df_sub(df_of(1.f), cuu), opc = df_add(df_of(1.f), cuu);
    const dfl num = df_add(df_mul(df_mul(sp, sp), omc), df_mul(df_mul(sm, sm), opc));
    const dfl den = df_mul(df_mul(opc, omc), rsq);
    const dfl h = df_div(df_mul_f(df_mul(chi, num), 0.5f), den);
    return df_sub(df_of(1.f), h);
}

// Shape (c = chi) or energy (c = chi') terms: a, b = (ru1 +- ru2) / (1 +- c uu)
// and g. inv_rsq = 1 / r^2: the divisions by r^2 of the reference become
// products. V: float, or two pairs in packed FP32 (f32x2.cuh).
template <class V>
struct GbTerms {
    V a, b, g;
};

template <class V>
SG_DEV GbTerms<V> gb_terms(V c, V ru1, V ru2, V uu, V inv_rsq) {
    auto rcp = [](float x) { return fast_rcp(x); };
    const V one = all_w<V>(1.f), sp = ru1 + ru2, sm = ru1 - ru2, cu = c * uu;
    GbTerms<V> t;
    t.a = sp * map_w(one + cu, rcp);
    t.b = sm * map_w(one - cu, rcp);
    t.g = fma_w(c * inv_rsq * all_w<V>(-0.5f), fma_w(sp, t.a, sm * t.b), one);
    return t;
}

template <class V>
struct GbPair {
    V x, y, z;             // r_ij
    V ux, uy, uz;          // axis of I
    V vx, vy, vz;          // axis of J
    V lprp, chi, xhi, inv_ez;
};

template <class V>
struct GbOut {
    V fx, fy, fz;          // force on I
    V tx, ty, tz;          // torque on I
    V sx, sy, sz;          // torque on J
    V pe, vir;
};

struct GbContact {         // the precise class: g, sigma and r - sigma from double-float arithmetic
    float g = 0.f, sigma = 0.f, rms = 0.f;
};

template <class V>
SG_DEV V dot_w(V ax, V ay, V az, V bx, V by, V bz) { return fma_w(az, bz, fma_w(ay, by, ax * bx)); }

SG_DEV bool in_zone(float x, float lo, float hi) { return x >= lo && x <= hi; }
SG_DEV mask2 in_zone(f2 x, f2 lo, f2 hi) { return not_above_w(lo, x) && not_above_w(x, hi); }

// Energy, force and torques of a Gay-Berne pair; returns whether it is in range.
// With dG/dr = P u1 + Q u2 + k r, dG/du1 = P r + q u2 and dG/du2 = Q r + q u1 for
// each of the two G (chi and chi', force.f90:266-306), everything the pair does
// is a combination of r, u1 and u2, whose scalar weights are summed first:
//   F = -(A r + B u1 + C u2), torques -u1 x (D u2 + B r) and -u2 x (D u1 + C r).
// r and sigma come from an approximate 1/sqrt and one Newton step whose last
// operation is a fused multiply-add of the exact product, so both are rounded
// once, as the square root and quotient they stand for; the other
// quotients are a 1-ulp reciprocal away (the force tolerance is 1e-5).
template <int KIND, bool PRECISE, class V>
SG_DEV typename MaskOf<V>::type gb_eval(const GbPair<V>& p, const GbContact& contact, float cutoff, float wf,
                                        float chirality, int mu, int nu, GbOut<V>& o) {
    constexpr bool kWeld = KIND == SG_GBW || KIND == SG_GBWC, kChiral = KIND == SG_GBC || KIND == SG_GBWC;
    constexpr bool kTaper = KIND != SG_GBR;
    auto k = [](float x) { return all_w<V>(x); };
    auto rcp = [](float x) { return fast_rcp(x); };
    auto rsqrt = [](float x) { return fast_rsqrt(x); };
    const V zero = k(0.f), one = k(1.f), half = k(0.5f);
    const V rsq = dot_w(p.x, p.y, p.z, p.x, p.y, p.z);
    const V ru1 = dot_w(p.x, p.y, p.z, p.ux, p.uy, p.uz), ru2 = dot_w(p.x, p.y, p.z, p.vx, p.vy, p.vz);
    const V uu = dot_w(p.ux, p.uy, p.uz, p.vx, p.vy, p.vz);
    const V inv_rsq = map_w(rsq, rcp);
    const V y0 = map_w(rsq, rsqrt), m0 = rsq * y0, hy = half * y0;
    const V rmag = fma_w(hy, fma_w(zero - m0, m0, rsq), m0);
    const V rinv = fma_w(hy, fma_w(zero - m0, y0, one), y0);
    const V cu = p.chi * uu;
    GbTerms<V> gc = gb_terms(p.chi, ru1, ru2, uu, inv_rsq);
    const GbTerms<V> gx = gb_terms(p.xhi, ru1, ru2, uu, inv_rsq);
    const V eps1 = map_w(fma_w(zero - cu, cu, one), [](float x) { return rsqrtf(x); });
    const V eps2 = gx.g * p.inv_ez;
    V sigma, rms;
    if constexpr (PRECISE) {
        gc.g = contact.g;
        sigma = contact.sigma;
        rms = contact.rms;
    } else {   // lprp / sqrt(g)
        const V s0 = map_w(gc.g, rsqrt), gs = gc.g * s0, er = fma_w(gc.g, s0, zero - gs);
        const V d = fma_w(zero - er, s0, fma_w(zero - gs, s0, one));   // 1 - g s0^2
        sigma = fma_w(p.lprp, s0, (p.lprp * s0) * (half * d));
        rms = rmag - sigma;
    }
    const V ginv = sigma * map_w(gc.g, rcp);
    const V reach = sigma + k(kWeld ? cutoff + wf - 1.f : cutoff - 1.f);
    const typename MaskOf<V>::type active = KIND == SG_GBR ? not_above_w(rms, zero) : less_w(rmag, reach);
    // 1 / (r - sigma + 1); correctly rounded in the precise class (sr^12
    // carries twelve times its error)
    auto contact_rcp = [](float x) { return PRECISE ? __frcp_rn(x) : fast_rcp(x); };
    const V sr = map_w(rms, [=](float x) {
        if (!kWeld) return contact_rcp(x + 1.f);
        return x < 0.f ? contact_rcp(x + 1.f) : x <= wf ? 1.f : contact_rcp(x + 1.f - wf);
    });
    const V sr2 = sr * sr, sr6 = sr2 * sr2 * sr2, sr12 = sr6 * sr6;
    V srx = fma_w(k(-2.f), sr6, sr12);
    if (KIND == SG_GBR) srx = srx + one;
    V srd = k(12.f) * (sr6 - sr12) * sr;
    // eps1^nu, eps2^(mu - 1) by products (mu, nu >= 1, warp-uniform)
    V e1n = eps1, e2p = one;
    for (int q = 1; q < nu; ++q) e1n = e1n * eps1;
    for (int q = 1; q < mu; ++q) e2p = e2p * eps2;
    const V e2m = e2p * eps2, ee = e1n * e2m;
    const V pe_fac = e1n * (k((float)mu) * e2p), e1_fac = e2m * (k((float)nu) * (e1n * eps1 * eps1));
    V pot = ee * srx;
    V lam = zero, del = zero;
    if (kChiral) {   // gbc_ / gbwc_ (force.f90:755-827)
        V cx, cd;
        if (KIND == SG_GBC) {
            cx = sr6 * sr;
            cd = k(-7.f) * sr6 * sr2;
        } else {
            cx = fma_w(k(-12.f / 7.f), sr6 * sr, sr12);
            cd = k(12.f) * (sr6 * sr2 - sr12 * sr);
        }
        const V wx = p.uy * p.vz - p.uz * p.vy, wy = p.uz * p.vx - p.ux * p.vz, wz = p.ux * p.vy - p.uy * p.vx;
        const V uur = dot_w(wx, wy, wz, p.x, p.y, p.z) * rinv;
        const V ch = k(chirality), chu = ch * uur * uu;
        pot = fma_w(ee * cx, chu, pot);
        srx = fma_w(cx, chu, srx);
        srd = fma_w(cd, chu, srd);
        del = ch * ee * cx * uur;
        lam = ch * ee * cx * uu * rinv;
    }
    const V Pc = zero - p.chi * inv_rsq * (gc.a + gc.b), Qc = zero - p.chi * inv_rsq * (gc.a - gc.b);
    const V Px = zero - p.xhi * inv_rsq * (gx.a + gx.b), Qx = zero - p.xhi * inv_rsq * (gx.a - gx.b);
    const V hr = half * rsq, ir2 = inv_rsq + inv_rsq;
    const V wr = ee * srd, wc = wr * half * ginv, wx = srx * pe_fac;
    V A = fma_w(wr, rinv, fma_w(wc, ir2 * (one - gc.g), wx * (ir2 * (one - gx.g))));
    const V B = fma_w(wc, Pc, wx * Px), C = fma_w(wc, Qc, wx * Qx);
    const V D = del + fma_w(srx * e1_fac, p.chi * p.chi * uu, hr * fma_w(wc, Pc * Qc, wx * (Px * Qx)));
    // u1 x u2, u1 x r, u2 x r
    auto cross = [](V a, V b, V c, V d) { return fma_w(a, d, all_w<V>(0.f) - b * c); };   // a d - b c
    const V ex = cross(p.uy, p.uz, p.vy, p.vz), ey = cross(p.uz, p.ux, p.vz, p.vx), ez = cross(p.ux, p.uy, p.vx, p.vy);
    const V ax = cross(p.uy, p.uz, p.y, p.z), ay = cross(p.uz, p.ux, p.z, p.x), az = cross(p.ux, p.uy, p.x, p.y);
    const V bx = cross(p.vy, p.vz, p.y, p.z), by = cross(p.vz, p.vx, p.z, p.x), bz = cross(p.vx, p.vy, p.x, p.y);
    if (kChiral) A = A - lam * rinv * (dot_w(ex, ey, ez, p.x, p.y, p.z) * rinv);
    o.fx = zero - fma_w(A, p.x, fma_w(B, p.ux, C * p.vx));
    o.fy = zero - fma_w(A, p.y, fma_w(B, p.uy, C * p.vy));
    o.fz = zero - fma_w(A, p.z, fma_w(B, p.uz, C * p.vz));
    o.tx = zero - fma_w(D, ex, B * ax);
    o.ty = zero - fma_w(D, ey, B * ay);
    o.tz = zero - fma_w(D, ez, B * az);
    o.sx = fma_w(D, ex, zero - C * bx);
    o.sy = fma_w(D, ey, zero - C * by);
    o.sz = fma_w(D, ez, zero - C * bz);
    if (kChiral) {   // what is perpendicular: lam u1 x u2 on F, and its torques
        o.fx = o.fx - lam * ex; o.fy = o.fy - lam * ey; o.fz = o.fz - lam * ez;
        o.tx = o.tx - lam * (ru1 * p.vx - uu * p.x);
        o.ty = o.ty - lam * (ru1 * p.vy - uu * p.y);
        o.tz = o.tz - lam * (ru1 * p.vz - uu * p.z);
        o.sx = o.sx - lam * (uu * p.x - ru2 * p.ux);
        o.sy = o.sy - lam * (uu * p.y - ru2 * p.uy);
        o.sz = o.sz - lam * (uu * p.z - ru2 * p.uz);
    }
    if (kTaper) {
        const V sw = k(0.9f) * reach;
        const typename MaskOf<V>::type on = in_zone(rmag, sw, reach);
        const V factor = map_w(reach - sw, rcp);
        const V xx = (rmag - sw) * factor, x2 = xx * xx, x3 = x2 * xx, x4 = x2 * x2, x5 = x3 * x2;
        const V taper = fma_w(k(-10.f), x3, fma_w(k(15.f), x4, fma_w(k(-6.f), x5, one)));
        const V slope = fma_w(k(-30.f), x2, fma_w(k(60.f), x3, k(-30.f) * x4));
        const V sub = select_w(on, slope * pot * factor, zero);   // taken from each component (reference quirk)
        const V sx = select_w(on, taper, one);
        o.fx = fma_w(sx, o.fx, zero - sub); o.fy = fma_w(sx, o.fy, zero - sub); o.fz = fma_w(sx, o.fz, zero - sub);
        o.tx = fma_w(sx, o.tx, zero - sub); o.ty = fma_w(sx, o.ty, zero - sub); o.tz = fma_w(sx, o.tz, zero - sub);
        o.sx = fma_w(sx, o.sx, zero - sub); o.sy = fma_w(sx, o.sy, zero - sub); o.sz = fma_w(sx, o.sz, zero - sub);
        pot = sx * pot;
    }
    o.pe = pot;
    o.vir = dot_w(p.x, p.y, p.z, o.fx, o.fy, o.fz);
    return active;
}

template <int KIND>
struct PotGB {
    static constexpr bool kTorque = true;
    static constexpr bool kStats = false;
    static constexpr bool kCountActive = true;
    static constexpr bool kWeld = (KIND == SG_GBW || KIND == SG_GBWC);
    static constexpr bool kFilterable = false;   // the filtered launch is k_pair_gb
    static constexpr int kMinBlocks = 1;
    const float4* __restrict__ prep;   // rec: 2 per particle
    const float4* __restrict__ aux;    // 1 per particle
    const float4* __restrict__ lo;     // 1 per particle: low parts of u and chi
    BoxF b;
    float cutoff, wf, chirality;
    int mu, nu;

    // A superset of eval's range test (r against the orientation-dependent
    // contact distance sigma of I's shape plus the cut-off), without its
    // correctly rounded square roots and division: approximate 1/sqrt for r
    // and sigma (a few ulp each), and a slack of 1e-5 (r + sigma), some 80
    // ulp of the larger, which also covers the rounding of sigma + shift. A
    // NaN anywhere keeps the pair: eval_r decides. r_ij is handed on to
    // eval_r. Returns 0 (out of range), 1 (in range) or 2 (in range and
    // within SG_GB_NEAR of the approximate contact distance: the precise class).
    SG_DEV int in_range_r(int i, int j, float3& r) const {
        float4 pi0, pi1, pj0, pj1;
        ld_f4x2(prep + 2 * i, pi0, pi1);
        ld_f4x2(prep + 2 * j, pj0, pj1);
        // (the precise class recomputes r_ij to ~1e-12: across the periodic
        // boundary this FP32 difference carries ulp(box)/2)
        r = pair_rij_of(make_float3(pi0.x, pi0.y, pi0.z), make_float3(pj0.x, pj0.y, pj0.z), i, b);
        const float rsq = r.x * r.x + r.y * r.y + r.z * r.z;
        const float3 U1 = make_float3(pi1.x, pi1.y, pi1.z), U2 = make_float3(pj1.x, pj1.y, pj1.z);
        const GbTerms<float> gc = gb_terms(pi1.w, dot3(r, U1), dot3(r, U2), dot3(U1, U2), fast_rcp(rsq));
        const float sigma = pi0.w * fast_rsqrt(gc.g);
        const float rmag = rsq * fast_rsqrt(rsq);
        if (0.99999f * rmag >= 1.00001f * sigma + reach_shift()) return 0;
        return rmag < sigma + SG_GB_NEAR ? 2 : 1;
    }
    SG_DEV float reach_shift() const {
        return (KIND == SG_GBR) ? 0.f : kWeld ? (cutoff + wf - 1.f) : (cutoff - 1.f);
    }

    // unfiltered launch: the range test's class picks the evaluation, as the
    // queues of the filtered launch do
    SG_DEV void eval(bool valid, int i, int j, int, PairOut& o, unsigned long long*) const {
        if (!valid) return;
        float3 r;
        if (in_range_r(i, j, r) == 2)
            eval_r<true>(valid, i, j, r, o);
        else
            eval_r<false>(valid, i, j, r, o);
    }

    template <bool PRECISE>
    SG_DEV void eval_r(bool valid, int i, int j, float3 r, PairOut& o) const {
        if (!valid) return;
        const float4* rec = prep;
        if (PRECISE) {
            // the minimum image to ~1e-12: across the periodic boundary the
            // FP32 difference carries ulp(box)/2, which the envelope amplifies
            const float4 a = rec[2 * i], c = rec[2 * j];
            r = pair_rij_of_precise(make_float3(a.x, a.y, a.z), make_float3(c.x, c.y, c.z), i, b);
        }
        const float4 pi1 = rec[2 * i + 1], pj1 = rec[2 * j + 1], ai = aux[i];
        GbPair<float> p;
        p.x = r.x; p.y = r.y; p.z = r.z;
        p.ux = pi1.x; p.uy = pi1.y; p.uz = pi1.z;
        p.vx = pj1.x; p.vy = pj1.y; p.vz = pj1.z;
        p.lprp = rec[2 * i].w;
        p.chi = pi1.w;
        p.xhi = ai.x;
        p.inv_ez = ai.y;
        GbContact c;
        if (PRECISE) {
            const float4 li = lo[i], lj = lo[j];
            dfl rsq_d;
            const dfl g = gb_shape_g_df(r, make_float3(p.ux, p.uy, p.uz), make_float3(li.x, li.y, li.z),
                                        make_float3(p.vx, p.vy, p.vz), make_float3(lj.x, lj.y, lj.z),
                                        dfl{p.chi, li.w}, rsq_d);
            const dfl sig_d = df_div(df_of(p.lprp), df_sqrt(g));
            const dfl d = df_sub(df_sqrt(rsq_d), sig_d);
            c.g = g.hi + g.lo;
            c.sigma = sig_d.hi + sig_d.lo;
            c.rms = d.hi + d.lo;
        }
        GbOut<float> w;
        const bool active = gb_eval<KIND, PRECISE>(p, c, cutoff, wf, chirality, mu, nu, w);
        if (!active) return;
        o.act = 1;
        o.pe = w.pe;
        o.vir = w.vir;
        o.f = make_float3(w.fx, w.fy, w.fz);
        o.ti = make_float3(w.tx, w.ty, w.tz);
        o.tj = make_float3(w.sx, w.sy, w.sz);
    }
};

// ------------------------------------------------------ half-list pairs ----
// The Gay-Berne kinds over the flat half list. The range test turns two thirds
// of a usual list away, so the pairs that pass it queue up per warp and are
// evaluated 64 at a time, two a lane in packed FP32 (f32x2.cuh), and the
// near-contact class 32 at a time in double-float (PotGB::eval_r<true>).
// A warp walks one contiguous span of the list, so its queue holds few rows:
// what a row's pairs add to particle I stays in the lanes and is reduced when
// the row ends; a batch of many short rows takes the segmented sums.
// What is left in the queues at the end is put together over the block's warps.
// Bound: the L1's wavefronts, three quarters of peak while it runs (a gather of
// 32 J records touches 32 lines, and so do the J particles' two additions), at
// 44 % issue with 16 warps an SM; 128 registers hold two pairs' evaluation (80
// spill: 112 us). Measured on the list of 32 768 particles (5.4 M listed, 36 % in
// range), whole kernel: one pair a lane, segmented sums and leftovers per warp
// 110 us; this 81. 200 000 particles 577 and 445, 4 999 28.2 and 22.4, 1 000
// 15.4 and 12.5; 512 replicas of the 1024-replica ensemble 1528 and 1027, 64 of
// 128 181 and 139, 8 of 16 38.5 and 27.5 (a block per replica with the records in
// shared memory took 1736, 1225 and 1041). J records one chunk ahead by cp.async
// cost twice the wavefronts (99 us), in registers more of those than it hid (103).
#define SG_GB_SLOTS 128   // ring of 64 to 127 waiting pairs: a chunk adds 64 at most
#define SG_GB_ROWS 6      // more rows than this in a batch: segmented sums
#define SG_GB_BLOCKS 2

struct GbQueue {   // one warp's waiting pairs of one class: r_ij
    int i[SG_GB_SLOTS], j[SG_GB_SLOTS];
    float x[SG_GB_SLOTS], y[SG_GB_SLOTS], z[SG_GB_SLOTS];
};
struct GbAxes {    // with the axis of J: six conflict-free wavefronts instead of another gather's 32
    float x[SG_GB_SLOTS], y[SG_GB_SLOTS], z[SG_GB_SLOTS];
};

template <int KIND, bool REPLICAS>
struct GbWarp {
    const PairLaunch& L;
    const PotGB<KIND>& pot;
    GbQueue* main;
    GbQueue* near;
    GbAxes* axes;   // of main
    float3 box, inv_box;                  // of replica box_r
    int box_r = -1;
    int lane;
    int nm = 0, hm = 0, nn = 0, hn = 0;   // waiting pairs and ring heads
    unsigned ranged = 0, precise = 0;
    F2Sum pe, vir;
    EnergySums es;                        // of the near-contact class
    int row = -1;                         // the row whose sums are held
    float3 f, t;

    SG_DEV GbWarp(const PairLaunch& l, const PotGB<KIND>& p, GbQueue* m, GbQueue* n, GbAxes* a)
        : L(l), pot(p), main(m), near(n), axes(a), lane(threadIdx.x & 31) {
        pe = vir = F2Sum{all_w<f2>(0.f), all_w<f2>(0.f)};
        f = t = make_float3(0.f, 0.f, 0.f);
        box = pot.b.box;
        inv_box = pot.b.periodic ? pot.b.inv_box : f;
    }

    SG_DEV void push(GbQueue* q, GbAxes* ax, int head, int& n, bool keep, int i, int j, float3 r, float3 u) {
        const unsigned m = __ballot_sync(0xffffffffu, keep);
        if (keep) {
            const int s = (head + n + __popc(m & ((1u << lane) - 1u))) & (SG_GB_SLOTS - 1);
            q->i[s] = i;
            q->j[s] = j;
            q->x[s] = r.x;
            q->y[s] = r.y;
            q->z[s] = r.z;
            if (ax) {
                ax->x[s] = u.x;
                ax->y[s] = u.y;
                ax->z[s] = u.z;
            }
        }
        n += __popc(m);
    }

    // Two listed pairs per lane: the superset range test of in_range_r, and
    // into the queues with what it keeps.
    SG_DEV void test(const PairChunk& c) {
        const int i0 = c.i0, j0 = c.j0, i1 = c.i1, j1 = c.j1;
        const bool v0 = lane < c.n, v1 = lane + 32 < c.n;
        float4 a0, a1, c0, c1, d0, d1, e0, e1;
        ld_f4x2(pot.prep + 2 * (size_t)j0, c0, c1);
        ld_f4x2(pot.prep + 2 * (size_t)j1, e0, e1);
        ld_f4x2(pot.prep + 2 * (size_t)i0, a0, a1);
        ld_f4x2(pot.prep + 2 * (size_t)i1, d0, d1);
        if (REPLICAS && c.r != box_r) {
            box_r = c.r;
            box = f3(pot.b.rbox[box_r]);
            inv_box = f3(pot.b.rinv[box_r]);
        }
        auto image = [](f2 d, float box, float inv_box) {   // see row_image
            const f2 big = all_w<f2>(12582912.f);
            const f2 n = fma_w(d, all_w<f2>(inv_box), big) - big;
            return fma_w(n, all_w<f2>(-box), d);
        };
        const f2 x = image(f2_of(a0.x - c0.x, d0.x - e0.x), box.x, inv_box.x);
        const f2 y = image(f2_of(a0.y - c0.y, d0.y - e0.y), box.y, inv_box.y);
        const f2 z = image(f2_of(a0.z - c0.z, d0.z - e0.z), box.z, inv_box.z);
        const f2 rsq = fma_w(z, z, fma_w(y, y, x * x));
        float3 r0, r1;
        f2_split(x, r0.x, r1.x);
        f2_split(y, r0.y, r1.y);
        f2_split(z, r0.z, r1.z);
        const float3 u0 = f3(a1), w0 = f3(c1), u1 = f3(d1), w1 = f3(e1);
        const GbTerms<f2> gc = gb_terms(f2_of(a1.w, d1.w), f2_of(dot3(r0, u0), dot3(r1, u1)),
                                        f2_of(dot3(r0, w0), dot3(r1, w1)), f2_of(dot3(u0, w0), dot3(u1, w1)),
                                        map_w(rsq, [](float v) { return fast_rcp(v); }));
        const f2 sigma = f2_of(a0.w, d0.w) * map_w(gc.g, [](float v) { return fast_rsqrt(v); });
        const f2 rmag = rsq * map_w(rsq, [](float v) { return fast_rsqrt(v); });
        float far0, far1, in0, in1, m0, m1, s0, s1;
        f2_split(rmag * all_w<f2>(0.99999f), far0, far1);
        f2_split(fma_w(sigma, all_w<f2>(1.00001f), all_w<f2>(pot.reach_shift())), in0, in1);
        f2_split(rmag, m0, m1);
        f2_split(sigma + all_w<f2>(SG_GB_NEAR), s0, s1);
        const bool k0 = v0 && !(far0 >= in0), k1 = v1 && !(far1 >= in1);   // a NaN keeps the pair
        const bool n0 = k0 && m0 < s0, n1 = k1 && m1 < s1;
        push(main, axes, hm, nm, k0 && !n0, i0, j0, r0, w0);
        push(main, axes, hm, nm, k1 && !n1, i1, j1, r1, w1);
        if (__any_sync(0xffffffffu, n0 || n1)) {
            const int before = nn;
            push(near, nullptr, hn, nn, n0, i0, j0, r0, w0);
            push(near, nullptr, hn, nn, n1, i1, j1, r1, w1);
            precise += nn - before;
        }
        __syncwarp();
    }

    SG_DEV void get(const GbQueue* q, int s, bool ok, int& i, int& j, float3& r) const {
        i = ok ? q->i[s] : -1;
        j = ok ? q->j[s] : 0;
        r = ok ? make_float3(q->x[s], q->y[s], q->z[s]) : make_float3(1.f, 0.f, 0.f);
    }

    SG_DEV float3 axis(const GbAxes* a, int s, bool ok) const {
        return ok ? make_float3(a->x[s], a->y[s], a->z[s]) : make_float3(1.f, 0.f, 0.f);
    }

    // The held row's sums to its particle: six values over 32 lanes by halving
    // (eight shuffles), which leaves one value in every lane.
    SG_DEV void end_row() {
        if (row < 0) return;
        const unsigned full = 0xffffffffu;
        const bool b4 = lane & 16, b3 = lane & 8, b2 = lane & 4;
        float v0 = b4 ? t.x : f.x, v1 = b4 ? t.y : f.y, v2 = b4 ? t.z : f.z;
        v0 += __shfl_xor_sync(full, b4 ? f.x : t.x, 16);
        v1 += __shfl_xor_sync(full, b4 ? f.y : t.y, 16);
        v2 += __shfl_xor_sync(full, b4 ? f.z : t.z, 16);
        float w0 = b3 ? v2 : v0, w1 = b3 ? 0.f : v1;
        w0 += __shfl_xor_sync(full, b3 ? v0 : v2, 8);
        w1 += __shfl_xor_sync(full, b3 ? v1 : 0.f, 8);
        float s = b2 ? w1 : w0;
        s += __shfl_xor_sync(full, b2 ? w0 : w1, 4);
        s += __shfl_xor_sync(full, s, 2);
        s += __shfl_xor_sync(full, s, 1);
        const int k = (b3 ? 2 : 0) + (b2 ? 1 : 0);   // component 0, 1, 2; 3: nothing
        if ((lane & 3) == 0 && k < 3) atomicAdd(reinterpret_cast<float*>((b4 ? L.torque : L.force) + row) + k, s);
        f = t = make_float3(0.f, 0.f, 0.f);
        row = -1;
    }

    // Two pairs per lane (slots lane and lane + 32 of a batch, in list order)
    SG_DEV void eval(int i0, int j0, float3 r0, float3 w0, int i1, int j1, float3 r1, float3 w1) {
        const unsigned full = 0xffffffffu;
        const bool ok0 = i0 >= 0, ok1 = i1 >= 0;
        const int k0 = max(i0, 0), k1 = max(i1, 0);
        GbPair<f2> p;
        {
            const float4 u0 = pot.prep[2 * (size_t)k0 + 1], u1 = pot.prep[2 * (size_t)k1 + 1];
            const float4 a0 = pot.aux[k0], a1 = pot.aux[k1];
            p.lprp = f2_of(pot.prep[2 * (size_t)k0].w, pot.prep[2 * (size_t)k1].w);
            p.x = f2_of(r0.x, r1.x); p.y = f2_of(r0.y, r1.y); p.z = f2_of(r0.z, r1.z);
            p.ux = f2_of(u0.x, u1.x); p.uy = f2_of(u0.y, u1.y); p.uz = f2_of(u0.z, u1.z);
            p.vx = f2_of(w0.x, w1.x); p.vy = f2_of(w0.y, w1.y); p.vz = f2_of(w0.z, w1.z);
            p.chi = f2_of(u0.w, u1.w);
            p.xhi = f2_of(a0.x, a1.x);
            p.inv_ez = f2_of(a0.y, a1.y);
        }
        GbOut<f2> o;
        const mask2 act = mask2{ok0, ok1} && gb_eval<KIND, false>(p, GbContact{}, pot.cutoff, pot.wf, pot.chirality,
                                                                  pot.mu, pot.nu, o);
        if (L.stats) ranged += __popc(__ballot_sync(full, act.lo)) + __popc(__ballot_sync(full, act.hi));
        {
            const f2 zero = all_w<f2>(0.f);
            pe.add(select_w(act, o.pe, zero));
            vir.add(select_w(act, o.vir, zero));
        }
        float3 f0, f1, t0, t1, s0, s1;
        f2_split(o.fx, f0.x, f1.x); f2_split(o.fy, f0.y, f1.y); f2_split(o.fz, f0.z, f1.z);
        f2_split(o.tx, t0.x, t1.x); f2_split(o.ty, t0.y, t1.y); f2_split(o.tz, t0.z, t1.z);
        f2_split(o.sx, s0.x, s1.x); f2_split(o.sy, s0.y, s1.y); f2_split(o.sz, s0.z, s1.z);
        if (act.lo) {
            atomic_add_f3(&L.force[j0], make_float3(-f0.x, -f0.y, -f0.z));
            atomic_add_f3(&L.torque[j0], s0);
        }
        if (act.hi) {
            atomic_add_f3(&L.force[j1], make_float3(-f1.x, -f1.y, -f1.z));
            atomic_add_f3(&L.torque[j1], s1);
        }
        // rows of the batch: the list goes by row, so their particles ascend
        const int up0 = __shfl_up_sync(full, i0, 1), up1 = __shfl_up_sync(full, i1, 1);
        const int rows = __popc(__ballot_sync(full, ok0 && (lane == 0 || i0 != up0))) +
                         __popc(__ballot_sync(full, ok1 && (lane == 0 || i1 != up1)));
        if (rows > SG_GB_ROWS) {
            end_row();
            if (!act.lo) f0 = t0 = make_float3(0.f, 0.f, 0.f);
            if (!act.hi) f1 = t1 = make_float3(0.f, 0.f, 0.f);
            segmented_scatter_i<true>(L, i0, f0, t0);
            segmented_scatter_i<true>(L, i1, f1, t1);
            return;
        }
        for (int at = -1;;) {
            const int a = ok0 && i0 > at ? i0 : INT_MAX, c = ok1 && i1 > at ? i1 : INT_MAX;
            at = __reduce_min_sync(full, min(a, c));
            if (at == INT_MAX) break;
            if (at != row) {
                end_row();
                row = at;
            }
            if (i0 == at && act.lo) {
                f.x += f0.x; f.y += f0.y; f.z += f0.z;
                t.x += t0.x; t.y += t0.y; t.z += t0.z;
            }
            if (i1 == at && act.hi) {
                f.x += f1.x; f.y += f1.y; f.z += f1.z;
                t.x += t1.x; t.y += t1.y; t.z += t1.z;
            }
        }
    }
    SG_DEV void drain_main() {
        int i0, j0, i1, j1;
        float3 r0, r1;
        const int s0 = (hm + lane) & (SG_GB_SLOTS - 1), s1 = (hm + 32 + lane) & (SG_GB_SLOTS - 1);
        get(main, s0, true, i0, j0, r0);
        get(main, s1, true, i1, j1, r1);
        const float3 w0 = axis(axes, s0, true), w1 = axis(axes, s1, true);
        hm = (hm + 64) & (SG_GB_SLOTS - 1);
        nm -= 64;
        __syncwarp();   // the slots are read before the next chunk writes them
        eval(i0, j0, r0, w0, i1, j1, r1, w1);
    }
    SG_DEV void eval_near(int i, int j, float3 r, bool ok) {
        PairOut o;
        o.f = o.ti = o.tj = make_float3(0.f, 0.f, 0.f);
        o.pe = o.vir = 0.f;
        o.act = 0;
        pot.template eval_r<true>(ok, ok ? i : 0, j, r, o);
        if (L.stats) ranged += __popc(__ballot_sync(0xffffffffu, o.act != 0));
        if (o.act) {
            atomic_add_f3(&L.force[j], make_float3(-o.f.x, -o.f.y, -o.f.z));
            atomic_add_f3(&L.torque[j], o.tj);
        }
        es.add(o.pe, o.vir);
        segmented_scatter_i<true>(L, ok ? i : -1, o.f, o.ti);
    }
    SG_DEV void drain_near() {
        int i, j;
        float3 r;
        get(near, (hn + lane) & (SG_GB_SLOTS - 1), true, i, j, r);
        hn = (hn + 32) & (SG_GB_SLOTS - 1);
        nn -= 32;
        __syncwarp();
        eval_near(i, j, r, true);
    }
};

template <int KIND, bool REPLICAS>
__global__ void __launch_bounds__(SG_PAIR_MAX_BLOCK, SG_GB_BLOCKS) k_pair_gb(PairLaunch L, PotGB<KIND> pot) {
    constexpr int W = SG_PAIR_MAX_BLOCK / 32;
    extern __shared__ float4 sg_gb_shared[];
    __shared__ int sh_left[2][W], sh_head[2][W];
    GbQueue* queues = reinterpret_cast<GbQueue*>(sg_gb_shared);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
    const int b0 = L.begin ? *L.begin : 0, np = *L.npairs;
    // equal spans of whole 64-pair chunks, the warps of a block side by side
    const int warps = gridDim.x * nw;
    const int span = (int)((((long long)np - b0 + warps - 1) / warps + 63) & ~63ll);
    GbAxes* axes = reinterpret_cast<GbAxes*>(queues + 2 * nw);
    GbWarp<KIND, REPLICAS> g(L, pot, queues + warp, queues + nw + warp, axes + warp);
    PairWalk w;
    const long long start = (long long)b0 + (long long)(blockIdx.x * nw + warp) * span;
    w.base = (int)min((long long)np, start);
    w.stop = (int)min((long long)np, start + span);
    w.r = 0;
    w.rend = np;
    w.shift = 0;
    if (REPLICAS && w.base < w.stop) {
        w.r = L.chunk_rep[w.base >> 5];
        w.enter(L);
    }
    unsigned listed = 0;
    PairChunk nxt;
    nxt.load(L, w, lane);
    while (nxt.n > 0) {
        const PairChunk c = nxt;
        if (REPLICAS) w.next(L);
        else w.base = w.end();
        nxt.load(L, w, lane);   // the next chunk's indices are in flight meanwhile
        listed += c.n;
        g.test(c);
        if (g.nm >= 64) g.drain_main();
        while (g.nn >= 32) g.drain_near();
    }
    // what is left, over the block
    if (lane == 0) {
        sh_left[0][warp] = g.nm;
        sh_left[1][warp] = g.nn;
        sh_head[0][warp] = g.hm;
        sh_head[1][warp] = g.hn;
    }
    __syncthreads();
    auto slot = [&](int q, int k, int& i, int& j, float3& r, float3& u) {   // k-th pair left of class q; i = -1 beyond
        int v = 0;
        while (v < nw && k >= sh_left[q][v]) k -= sh_left[q][v++];
        const bool ok = v < nw;
        const GbQueue* at = queues + q * nw + (ok ? v : 0);
        const int s = ok ? (sh_head[q][v] + k) & (SG_GB_SLOTS - 1) : 0;
        g.get(at, s, ok, i, j, r);
        u = q == 0 ? g.axis(axes + (ok ? v : 0), s, ok) : make_float3(0.f, 0.f, 0.f);
    };
    int left0 = 0, left1 = 0;
    for (int v = 0; v < nw; ++v) {
        left0 += sh_left[0][v];
        left1 += sh_left[1][v];
    }
    for (int k = 32 * (nw - 1 - warp); k < left1; k += 32 * nw) {   // the last warps first: the first take the others
        int i, j;
        float3 r, u;
        slot(1, k + lane, i, j, r, u);
        g.eval_near(i, j, r, i >= 0);
    }
    for (int k = 64 * warp; k < left0; k += 64 * nw) {
        int i0, j0, i1, j1;
        float3 r0, r1, u0, u1;
        slot(0, k + lane, i0, j0, r0, u0);
        slot(0, k + 32 + lane, i1, j1, r1, u1);
        g.eval(i0, j0, r0, u0, i1, j1, r1, u1);
    }
    g.end_row();
    // the pairs are done (see k_pair)
    pdl_trigger();
    if (L.stats && lane == 0) {
        if (listed) atomicAdd(&L.stats[0], (unsigned long long)listed);
        if (g.ranged) atomicAdd(&L.stats[1], (unsigned long long)g.ranged);
        if (g.precise) atomicAdd(&L.stats[3], (unsigned long long)g.precise);
    }
    float e[2], elo[2];
    auto total = [](const F2Sum& s, float x, float x_lo, float& hi, float& low) {
        const dfl d = s.total(), t = df_two_sum(d.hi, x);
        hi = t.hi;
        low = t.lo + d.lo + x_lo;
    };
    total(g.pe, g.es.pe, g.es.pe_lo, e[0], elo[0]);
    total(g.vir, g.es.vir, g.es.vir_lo, e[1], elo[1]);
    pair_sums_finish(e, elo, L.partials, L.done, L.acc, L.acc_total);
}

template <int KIND, bool REPLICAS>
int launch_gb_pairs(sg_ctx* ctx, const PotGB<KIND>& pot, int block) {
    if (!ctx->nl.initialized) return sg_fail(ctx, SG_ENOTREADY, "pair forces need sg_nlist_init first");
    if (int rc = sg_need_half_list(ctx, true)) return rc;
    PairLaunch L = make_pair_launch(ctx);
    const size_t smem = (sizeof(GbQueue) * 2 + sizeof(GbAxes)) * (size_t)(block / 32);
    const void* fn = (const void*)k_pair_gb<KIND, REPLICAS>;
    SG_CUDA(ctx, cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    int grid = sg_grid_for(ctx, fn, block, smem);
    const int64_t useful = (ctx->nl.pair_capacity + 2 * block - 1) / (2 * block);   // 64 pairs a warp
    grid = (int)std::max<int64_t>(1, std::min<int64_t>(grid, useful));
    if (int rc = sg_pair_slots(ctx, grid, &L.partials, &L.done)) return rc;
    k_pair_gb<KIND, REPLICAS><<<grid, block, smem, ctx->stream>>>(L, pot);
    SG_LAUNCH_CHECK(ctx, "k_pair_gb");
    return SG_OK;
}

template <int KIND>
int launch_gb(sg_ctx* ctx, const sg_pair_params* p, float4* prep, int mu, int nu) {
    PotGB<KIND> pot;
    pot.prep = prep;
    pot.aux = prep + 2 * (size_t)ctx->n;
    pot.lo = prep + 3 * (size_t)ctx->n;
    pot.b = make_boxf(ctx);
    pot.cutoff = (float)p->cutoff;
    pot.wf = (float)p->wf;
    pot.chirality = (float)p->chirality;
    pot.mu = mu;
    pot.nu = nu;
    const PairTune tune = sg_pair_tune_for(ctx, KIND, true);
    if (!tune.filter) return launch_pair(ctx, pot, KIND);
    return ctx->nrep ? launch_gb_pairs<KIND, true>(ctx, pot, tune.block)
                     : launch_gb_pairs<KIND, false>(ctx, pot, tune.block);
}

}  // namespace

int sg_launch_pair_gb(sg_ctx* ctx, const sg_pair_params* p) {
    int mu = p->mu, nu = p->nu;
    if (mu == 0 && nu == 0) { mu = 1; nu = 2; }
    if (mu < 1 || nu < 1 || mu > 8 || nu > 8) return sg_fail(ctx, SG_EINVAL, "GB exponents must be in 1..8");
    // prep buffer: reuse the ECP prep allocation (large enough: 4 float4 per particle)
    if (!ctx->ecp_prep) SG_CUDA(ctx, cudaMalloc(&ctx->ecp_prep, sizeof(float4) * SG_PREP_F4 * (size_t)ctx->n));
    if (ctx->step_prep_kind != SG_PREP_GB) {   // else written by the step's initial half step
        k_gb_prep<<<(ctx->n + 255) / 256, 256, 0, ctx->stream>>>(ctx->n, ctx->pos, ctx->quat, ctx->shape,
                                                                ctx->eshape, 1.f / (float)mu, ctx->ecp_prep);
        SG_LAUNCH_CHECK(ctx, "k_gb_prep");
    }
    switch (p->kind) {
        case SG_GB: return launch_gb<SG_GB>(ctx, p, ctx->ecp_prep, mu, nu);
        case SG_GBR: return launch_gb<SG_GBR>(ctx, p, ctx->ecp_prep, mu, nu);
        case SG_GBW: return launch_gb<SG_GBW>(ctx, p, ctx->ecp_prep, mu, nu);
        case SG_GBC: return launch_gb<SG_GBC>(ctx, p, ctx->ecp_prep, mu, nu);
        case SG_GBWC: return launch_gb<SG_GBWC>(ctx, p, ctx->ecp_prep, mu, nu);
        default: return sg_fail(ctx, SG_EINVAL, "unknown GB kind %d", p->kind);
    }
}
