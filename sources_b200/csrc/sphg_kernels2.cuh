// sphg_kernels2.cuh — the FP32 pair passes with two particles per lane pair
// (sphg_pairs2.cuh): the same terms as the one-particle passes of
// sphg_kernels.cuh, evaluated for both particles at once in packed FP32
// arithmetic.  What follows a particle's sums (EOS, plasticity, corrector) is
// shared with them.
#pragma once
#include "sphg_kernels.cuh"
#include "sphg_pairs2.cuh"

// Block size, resident blocks and staging space.  Bound: instruction issue, and
// the latency of each block's start (positions, cell bounds, bulk copies) and
// end (the corrector's state).  Measured at 912,016 particles (806,008 water,
// 106,008 soil), one kernel at a time, against the one-particle passes:
//   water_pass_a  124.0 -> 102.4 us   (12 or 14 blocks of 64 threads: 102, 99)
//   water_pass_b  169.4 -> 149.9 us   (8, 9, 10 blocks of 64: 158, 155, 154)
//   soil_pass      86.7 ->  62.6 us   (5, 6, 8 blocks of 64: 64, 63, 63)
//   step          421.3 -> 372.5 us
// and with the epilogue's loads before its stores, no predictor stored and the
// shorter cell list 85, 139, 57 and 312 us; with the checks of the sums (below)
// 86.5, 139.6, 57 and 314 (issue slots 58, 49 and 40 % used, 70, 98 and 177 warp
// instructions a particle);
// at 150k particles (Wendland, quadratic drag): 31.0 -> 27.1, 42.3 ->
// 41.9, 43.5 -> 36.0 us; soil only, 190k: 67.6 -> 53.8 us.  Neighbours come
// from shared memory: read through L1 (two particles and all candidates per
// lane) the passes took 112, 173 and 64 us.
#ifndef SPHG_TPB2
#define SPHG_TPB2 128
#endif
#ifndef SPHG_MINB_A2
#define SPHG_MINB_A2 6
#endif
#ifndef SPHG_MINB_B2
#define SPHG_MINB_B2 5
#endif
#ifndef SPHG_MINB_S2
#define SPHG_MINB_S2 4
#endif
// neighbours of one block of SPHG_TPB2 particles staged in shared memory
#ifndef SPHG_STAGE2
#define SPHG_STAGE2 576
#endif

// One value of both particles of the thread.
__device__ __forceinline__ float2 two(float a, float b) { return make_float2(a, b); }
__device__ __forceinline__ float2 neg2(float2 a) { return make_float2(-a.x, -a.y); }
__device__ __forceinline__ float2 zero2() { return make_float2(0.0f, 0.0f); }

// The two particles' own -v and rho.
struct Own2 {
    float2 nu, nv, rho;
    __device__ __forceinline__ Own2(const LanePair& p, const RecA<float>* rec) {
        const RecA<float> a = rec[p.k0], b = rec[p.k1];
        nu = two(-a.vx, -b.vx); nv = two(-a.vy, -b.vy); rho = two(a.rho, b.rho);
    }
};
// 1/rho, or 1 where rho is not positive (the sums are then not divided by it)
__device__ __forceinline__ float2 inv_rho(float2 rho) {
    return two(rho.x > 0.0f ? 1.0f / rho.x : 1.0f, rho.y > 0.0f ? 1.0f / rho.y : 1.0f);
}

// The pair factors of art_visc and av_vel from one reciprocal per pair.  d =
// v_b - v_a; mi = 2 m_b / (rho_a + rho_b); pi the viscous factor of grad W
// (approaching pairs only), mc = c_a + c_b.  ALONE: as the one-particle passes
// have it for any operand, with a reciprocal for each quotient (of an infinite
// density too) and no viscous factor where it is not called for.
template <bool ALONE>
__device__ __forceinline__ void visc_pair(const PairK& K, float2 rr, float2 dx, float2 dy, float2 du, float2 dv, float2 rho_a,
                                          float rho_b, float m_b, float2 mc, float2& mi, float2& pi) {
    // (kept above zero: a particle's own slot and coincident particles have r = 0, and etq may be 0)
    const float2 mr = add2(rho_a, splat2(rho_b)), de0 = add2(rr, splat2(K.h2e)), den = two(fmaxf(de0.x, 1e-30f), fmaxf(de0.y, 1e-30f));
    const float2 inv = rcp2(ALONE ? mr : mul2(mr, den));
    mi = mul2(splat2(m_b + m_b), inv);
    if (!ALONE) mi = mul2(mi, den);
    const float2 vr = fma2(du, dx, mul2(dv, dy));   // -(v_a - v_b) . (x_a - x_b)
    const float2 mu = mul2(mul2(splat2(K.nh), two(fmaxf(vr.x, 0.0f), fmaxf(vr.y, 0.0f))), ALONE ? rcp2(den) : mul2(inv, mr));
    pi = mul2(mul2(fma2(splat2(-K.beta), mu, mul2(splat2(K.alpha), mc)), mu), mi);
    if (ALONE) pi = sel2(vr.x > 0.0f, vr.y > 0.0f, pi);
}

// repulsive_force on the real particles of the pair from a virtual neighbour
__device__ __forceinline__ void wall_pair(const PairK& K, float2 rr, float2 dx, float2 dy, bool h0, bool h1, float2& ex,
                                          float2& ey) {
#pragma unroll
    for (int i = 0; i < 2; ++i) {
        const float r = sqrtf(i ? rr.y : rr.x);
        if ((i ? h1 : h0) && !(r > K.r0)) {
            const float f = K.dd * ((__powf(K.r0 / r, K.p1) - __powf(K.r0 / r, K.p2)) / (r * r));
            if (i) { ex.y += f * dx.y; ey.y += f * dy.y; }
            else { ex.x += f * dx.x; ey.x += f * dy.x; }
        }
    }
}

// Positions and records of a pass's neighbours, staged in shared memory when
// they fit (HASB: recB too): f(runs, xs, recA, recB, the two particles' own
// slots, the active halves) on each part of the pair's candidates.
template <bool HASB>
struct Staged2 {
    static constexpr int REC = HASB ? 64 : 32;
    static constexpr size_t BYTES = (size_t)SPHG_STAGE2 * REC;
};
extern __shared__ __align__(128) unsigned char stage_mem2[];

template <bool HASB, class F>
__device__ __forceinline__ void visit_pairs(const PhaseDev<float>& P, const GridGeom& g, const LanePair& p, int* timeout,
                                            F&& f) {
    __shared__ StageHdr H;
    double2* sxs = (double2*)stage_mem2;
    RecA<float>* sA = (RecA<float>*)(stage_mem2 + SPHG_STAGE2 * 16);
    RecB<float>* sB = (RecB<float>*)(stage_mem2 + SPHG_STAGE2 * 32);
    StageArrays<HASB ? 3 : 2> A;
    A.src[0] = P.xs; A.dst[0] = sxs; A.esize[0] = 16;
    A.src[1] = P.recA; A.dst[1] = sA; A.esize[1] = 16;
    if constexpr (HASB) { A.src[2] = P.recB; A.dst[2] = sB; A.esize[2] = 32; }
    PairRuns pr;
    pr.init(g, P.cell_start, p);
    const bool staged = stage_pairs<SPHG_TPB2>(H, A, g, P.cell_start, P.xs, P.n, SPHG_STAGE2, p, timeout);
    for (int i = 0, n = pr.parts(); i < n; ++i) {
        bool a0, a1;
        const Runs3 r = pr.part(g, P.cell_start, p, i, a0, a1);
        if (staged) {
            const int cy0 = p.lane ? p.oy : p.cy, cy1 = p.lane ? p.cy : p.oy;
            f(staged_runs3(H, r, pr.row(p, i)), (const double2*)sxs, (const RecA<float>*)sA, (const RecB<float>*)sB,
              staged_slot(H, p.k0, cy0), staged_slot(H, p.k1, cy1), a0, a1);
        } else {   // rare: the block's runs do not fit
            f(r, (const double2*)P.xs, (const RecA<float>*)P.recA, (const RecB<float>*)P.recB, p.k0, p.k1, a0, a1);
        }
    }
}

// ----------------------------------------------------------- water: pass A
// The two-phase sums of k_water_pass_a for both particles: ta = sum vol du gx
// and tb = sum vol dv gy (their combinations are the diagonal strain rates),
// tc the off-diagonal one, con, dl.
struct SumsA2 { float2 con, dl, ta, tb, tc; };
template <int SKF>
__device__ __forceinline__ void water_a_pair(const PairK& K, const Own2& o, SumsA2& s, const RecA<float>& rb, float2 dx, float2 dy,
                                             bool h0, bool h1) {
    float2 w, g;
    kernel_pair<SKF, true>(K, fma2(dx, dx, mul2(dy, dy)), h0, h1, w, g);
    const float2 vs = mul2(splat2(rb.vol), g);
    const float2 gx = mul2(vs, dx), gy = mul2(vs, dy);   // vol_b grad W
    s.dl = fma2(vs, add2(splat2(rb.rho), neg2(o.rho)), s.dl);
    // continuity and shear_strain_rate: v_b - v_a
    const float2 du = add2(splat2(rb.vx), o.nu), dv = add2(splat2(rb.vy), o.nv);
    const float2 xx = mul2(du, gx), yy = mul2(dv, gy);
    s.con = fma2(splat2(rb.rho), add2(xx, yy), s.con);
    s.ta = add2(s.ta, xx);
    s.tb = add2(s.tb, yy);
    s.tc = add2(s.tc, fma2(du, gy, mul2(dv, gx)));
}
template <int SKF>
__device__ __noinline__ SumsA2 water_a_alone(PhaseDev<float> P, GridGeom g, PairK K, LanePair p) {
    SumsA2 s{};
    const Own2 o(p, P.recA);
    visit_alone(g, P.cell_start, K.thr, P.xs, p, p.k,
                [&](int m, float2 dx, float2 dy, bool h0, bool h1) { water_a_pair<SKF>(K, o, s, P.recA[m], dx, dy, h0, h1); });
    return s;
}
template <int SKF>
__global__ void __launch_bounds__(SPHG_TPB2, SPHG_MINB_A2) k_water_pass_a2(PhaseDev<float> P, GridGeom g,
                                                                        const __grid_constant__ PairK K, SimConst c,
                                                                        DevCounters* cnt) {
    pdl_enter();
    const LanePair p(g, P.xs, P.n);
    const Own2 o(p, P.recA);
    SumsA2 s{};
    uint4 mask = make_uint4(0u, 0u, 0u, 0u);
    int hits0 = 0, hits1 = 0;
    visit_pairs<false>(P, g, p, &cnt->timeout, [&](const Runs3& r, const double2* xs, const RecA<float>* RA, const RecB<float>*,
                                                   int s0, int s1, bool a0, bool a1) {
        pair_scan<true>(r, p.lane, K.thr, xs, p.x0, p.x1, s0, s1, a0, a1, mask, hits0, hits1,
                        [&](int m, float2 dx, float2 dy, bool h0, bool h1) { water_a_pair<SKF>(K, o, s, RA[m], dx, dy, h0, h1); });
    });
    const int hits = p.mine(hits0, hits1);
    float con = p.mine(s.con), dl = p.mine(s.dl), ta = p.mine(s.ta), tb = p.mine(s.tb), tc = p.mine(s.tc);
    if (p.valid && !all_finite(con, dl, ta, tb, tc)) {
        const SumsA2 a = water_a_alone<SKF>(P, g, K, p);
        con = p.own(a.con); dl = p.own(a.dl); ta = p.own(a.ta); tb = p.own(a.tb); tc = p.own(a.tc);
    }
    if (p.v0) P.hmask[p.k] = mask;   // a lane without a particle of its own still has its half of the pair's candidates
    if (p.valid) {
        // delta_sph: 2 delta h c (rho_a - rho_b), c of the previous EOS call
        const float d = c.artificial_density ? -2.0f * K.ks * (float)(K.dh * P.c[P.perm[p.k]]) * dl : 0.0f;
        const float c23 = K.ks * (2.0f / 3.0f);
        water_a_finish<float, false>(P, c, p.k, -K.ks * con, d, c23 * (2.0f * ta - tb), K.ks * tc, c23 * (2.0f * tb - ta), 0.0f, hits);
    }
    count_stats_redux(cnt, 0, 0, hits, p.valid);
}

// ----------------------------------------------------------- water: pass B
// d1: pressure; e: viscous stress over rho_a, artificial viscosity, wall force; x: XSPH; c: the cross pairs
struct SumsB2 { float2 d1x, d1y, ex, ey, xx, xy, dvf, cdx, cdy, cdv, cv2; };
// visit(body): body(recA, recB, dx, dy, h0, h1) on every pair
template <int SKF, bool ALONE, class V>
__device__ __forceinline__ void water_b_pairs(const PhaseDev<float>& P, const PairK& K, const LanePair& p, const Own2& o, SumsB2& t,
                                              V&& visit) {
    const RecB<float> q0 = P.recB[p.k0], q1 = P.recB[p.k1];
    const float2 nphi = two(-q0.vof, -q1.vof), pa = two(q0.p, q1.p), ca = two(q0.c, q1.c), ira = inv_rho(o.rho);
    const float2 fxx = two(q0.vof * q0.sxx, q1.vof * q1.sxx), fxy = two(q0.vof * q0.sxy, q1.vof * q1.sxy),
                 fyy = two(q0.vof * q0.syy, q1.vof * q1.syy);
    const bool real0 = q0.itype > 0.0f, real1 = q1.itype > 0.0f;
    visit([&](const RecA<float>& rb, const RecB<float>& qb, float2 dx, float2 dy, bool h0, bool h1) {
        const float2 rr = fma2(dx, dx, mul2(dy, dy));
        float2 w, s, mi, pi;
        kernel_pair<SKF, false>(K, rr, h0, h1, w, s);
        const float2 gx = mul2(s, dx), gy = mul2(s, dy), vb = splat2(rb.vol);
        const float2 vp = mul2(vb, add2(pa, splat2(qb.p)));
        t.d1x = fma2(vp, gx, t.d1x);
        t.d1y = fma2(vp, gy, t.d1y);
        const float2 du = add2(splat2(rb.vx), o.nu), dv = add2(splat2(rb.vy), o.nv);   // v_b - v_a
        visc_pair<ALONE>(K, rr, dx, dy, du, dv, o.rho, rb.rho, rb.vol * rb.rho, add2(ca, splat2(qb.c)), mi, pi);
        const float2 xq = mul2(mi, w);
        t.xx = fma2(xq, du, t.xx);
        t.xy = fma2(xq, dv, t.xy);
        const float2 fb = splat2(qb.vof), vr = mul2(vb, ira);
        const float2 sxy = fma2(fb, splat2(qb.sxy), fxy);
        const float2 cx = fma2(vr, fma2(fb, splat2(qb.sxx), fxx), pi), cy = fma2(vr, fma2(fb, splat2(qb.syy), fyy), pi);
        const float2 cxy = mul2(vr, sxy);
        t.ex = fma2(cxy, gy, fma2(cx, gx, t.ex));
        t.ey = fma2(cxy, gx, fma2(cy, gy, t.ey));
        t.dvf = fma2(mul2(vb, add2(fb, nphi)), s, t.dvf);
        if (qb.itype < 0.0f) wall_pair(K, rr, dx, dy, h0 && real0, h1 && real1, t.ex, t.ey);
    });
}
// the water side of a cross pair (cross_water_sums); u = v_s - v_w
template <int SKF, bool FCH>
__device__ __forceinline__ void water_b_cross(const PhaseDev<float>& S, const PairK& K, const Own2& o, SumsB2& t, int m, float2 dx,
                                              float2 dy, bool h0, bool h1) {
    const RecA<float> rb = S.recA[m];
    const float phis = S.recB[m].vof;
    float2 w, s;
    kernel_pair<SKF, false>(K, fma2(dx, dx, mul2(dy, dy)), h0, h1, w, s);
    const float2 ux = add2(splat2(rb.vx), o.nu), uy = add2(splat2(rb.vy), o.nv);
    float2 q = mul2(splat2(rb.vol * phis), w);
    if constexpr (FCH) {
        const float2 u2 = fma2(ux, ux, mul2(uy, uy));
        q = mul2(q, fma2(splat2(K.kb), two(sqrtf(u2.x), sqrtf(u2.y)), splat2(1.0f)));
    }
    t.cdx = fma2(q, ux, t.cdx);
    t.cdy = fma2(q, uy, t.cdy);
    const float2 mb = splat2(rb.vol * rb.rho);
    t.cdv = fma2(mul2(mb, s), fma2(ux, dx, mul2(uy, dy)), t.cdv);
    t.cv2 = fma2(mb, w, t.cv2);
}
template <int SKF, bool FCH>
__device__ __noinline__ SumsB2 water_b_alone(PhaseDev<float> P, PhaseDev<float> S, GridGeom g, PairK K, LanePair p) {
    SumsB2 t{};
    const Own2 o(p, P.recA);
    water_b_pairs<SKF, true>(P, K, p, o, t, [&](auto&& body) {
        visit_alone(g, P.cell_start, K.thr, P.xs, p, p.k,
                    [&](int m, float2 dx, float2 dy, bool h0, bool h1) { body(P.recA[m], P.recB[m], dx, dy, h0, h1); });
    });
    visit_alone(g, S.cell_start, K.thr, S.xs, p, -1,
                [&](int m, float2 dx, float2 dy, bool h0, bool h1) { water_b_cross<SKF, FCH>(S, K, o, t, m, dx, dy, h0, h1); });
    return t;
}
template <int SKF, bool FCH>
__global__ void __launch_bounds__(SPHG_TPB2, SPHG_MINB_B2) k_water_pass_b2(PhaseDev<float> P, PhaseDev<float> S, GridGeom g,
                                                                        const __grid_constant__ PairK K, SimConst c, StepCtl u, DevCounters* cnt) {
    pdl_enter();
    const LanePair p(g, P.xs, P.n);
    const Own2 o(p, P.recA);
    SumsB2 t{};
    water_b_pairs<SKF, false>(P, K, p, o, t, [&](auto&& body) {
        const uint4 mask = p.v0 ? P.hmask[p.k] : make_uint4(0u, 0u, 0u, 0u);   // recorded by the step's first water pass
        visit_pairs<true>(P, g, p, &cnt->timeout, [&](const Runs3& r, const double2* xs, const RecA<float>* RA,
                                                           const RecB<float>* RB, int s0, int s1, bool a0, bool a1) {
            pair_replay(r, p.lane, K.thr, xs, p.x0, p.x1, s0, s1, a0, a1, mask,
                        [&](int m, float2 dx, float2 dy, bool h0, bool h1) { body(RA[m], RB[m], dx, dy, h0, h1); });
        });
    });
    int ch0 = 0, ch1 = 0;
    {
        PairRuns pr;
        pr.init(g, S.cell_start, p);
        for (int i = 0, n = pr.parts(); i < n; ++i) {
            bool a0, a1;
            const Runs3 r = pr.part(g, S.cell_start, p, i, a0, a1);
            uint4 unused;
            pair_scan<false>(r, p.lane, K.thr, S.xs, p.x0, p.x1, -1, -1, a0, a1, unused, ch0, ch1,
                             [&](int m, float2 dx, float2 dy, bool h0, bool h1) { water_b_cross<SKF, FCH>(S, K, o, t, m, dx, dy, h0, h1); });
        }
    }
    WaterB<float> w;
    auto sums = [&](const SumsB2& v, auto&& one) {
        w.mx = one(v.d1x); w.my = one(v.d1y);
        w.fx = K.ks * one(v.ex); w.fy = K.ks * one(v.ey);
        w.xsx = K.kw * one(v.xx); w.xsy = K.kw * one(v.xy);
        w.dvf = one(v.dvf);
        w.cdx = K.kw * one(v.cdx); w.cdy = K.kw * one(v.cdy); w.cdvof = K.ks * one(v.cdv); w.cv2 = K.kw * one(v.cv2);
    };
    sums(t, [&](float2 v) { return p.mine(v); });
    w.chits = p.mine(ch0, ch1);
    if (p.valid && !all_finite(w.mx, w.my, w.fx, w.fy, w.xsx, w.xsy, w.dvf, w.cdx, w.cdy, w.cdvof, w.cv2))
        sums(water_b_alone<SKF, FCH>(P, S, g, K, p), [&](float2 v) { return p.own(v); });
    if (p.valid) {
        const RecB<float> q = P.recB[p.k];
        w.mx *= -K.ks * q.vof; w.my *= -K.ks * q.vof;
        w.dvf = c.water_artificial_volume ? -2.0f * K.ks * (float)K.dh * q.c * w.dvf : 0.0f;
        water_b_finish<float, false>(P, g, c, u, cnt, p.k, p.lane ? o.rho.y : o.rho.x, q.vof, w);
    }
    count_stats_redux(cnt, 2, -1, w.chits, p.valid);
}

// ------------------------------------------------------------------ soil
// ta..td: sums of vol (du gx, dv gy, du gy, dv gx); m: pressure and stress over rho_a, artificial viscosity, wall force;
// x: XSPH; c: the cross pairs
struct SumsS2 { float2 con, dl, ta, tb, tc, td, mx, my, xx, xy, dpp, dsx, dsxy, dsy, cdx, cdy, cpx, cpy; };
template <int SKF, bool SINGLE, bool ALONE, class V>
__device__ __forceinline__ void soil_pairs(const PhaseDev<float>& P, const PairK& K, const LanePair& p, const Own2& o, SumsS2& t,
                                           V&& visit) {
    const RecB<float> q0 = P.recB[p.k0], q1 = P.recB[p.k1];
    const float2 npa = two(-q0.p, -q1.p), nsx = two(-q0.sxx, -q1.sxx), nsxy = two(-q0.sxy, -q1.sxy), nsy = two(-q0.syy, -q1.syy);
    const float2 nrho = neg2(o.rho), ira = inv_rho(o.rho);
    // minus the momentum factor of the particle's own stress: 1 (df, soil only) or vof / rho^2 (df3)
    const float2 nfa = SINGLE ? splat2(-1.0f) : two(-q0.vof / (o.rho.x * o.rho.x), -q1.vof / (o.rho.y * o.rho.y));
    const bool real0 = !SINGLE && q0.itype > 0.0f, real1 = !SINGLE && q1.itype > 0.0f;
    visit([&](const RecA<float>& rb, const RecB<float>& qb, float2 dx, float2 dy, bool h0, bool h1) {
        const float2 rr = fma2(dx, dx, mul2(dy, dy));
        float2 w, s, mi, pi;
        kernel_pair<SKF, SINGLE>(K, rr, h0, h1, w, s);
        const float2 gx = mul2(s, dx), gy = mul2(s, dy);
        const float2 du = add2(splat2(rb.vx), o.nu), dv = add2(splat2(rb.vy), o.nv);   // v_b - v_a
        const float2 vb = splat2(rb.vol), vu = mul2(vb, du), vv = mul2(vb, dv);
        const float mbs = rb.vol * rb.rho;
        const float2 xg = mul2(vu, gx), yg = mul2(vv, gy);
        t.con = fma2(splat2(rb.rho), add2(xg, yg), t.con);
        t.ta = add2(t.ta, xg);
        t.tb = add2(t.tb, yg);
        t.tc = fma2(vu, gy, t.tc);
        t.td = fma2(vv, gx, t.td);
        const float2 vs = mul2(vb, s);
        t.dl = fma2(vs, add2(splat2(rb.rho), nrho), t.dl);
        t.dpp = fma2(vs, add2(splat2(qb.p), npa), t.dpp);
        t.dsx = fma2(vs, add2(splat2(qb.sxx), nsx), t.dsx);
        t.dsxy = fma2(vs, add2(splat2(qb.sxy), nsxy), t.dsxy);
        t.dsy = fma2(vs, add2(splat2(qb.syy), nsy), t.dsy);
        visc_pair<ALONE>(K, rr, dx, dy, du, dv, o.rho, rb.rho, mbs, splat2(K.alpha_c), mi, pi);
        const float2 xq = mul2(mi, w);
        t.xx = fma2(xq, du, t.xx);
        t.xy = fma2(xq, dv, t.xy);
        // the pair stress f_a + f_b times the neighbour's volume (df) or mass (df3)
        const float fb = SINGLE ? 1.0f : qb.vof * rcp_approx(rb.rho * rb.rho);
        const float2 mw = SINGLE ? mul2(vb, ira) : splat2(mbs);
        const float pb = qb.p * fb;
        const float2 sxx = fma2(nfa, add2(nsx, neg2(npa)), splat2(fmaf(qb.sxx, fb, -pb)));
        const float2 syy = fma2(nfa, add2(nsy, neg2(npa)), splat2(fmaf(qb.syy, fb, -pb)));
        const float2 sxy = mul2(mw, fma2(nfa, nsxy, splat2(qb.sxy * fb)));
        const float2 cx = fma2(mw, sxx, pi), cy = fma2(mw, syy, pi);
        if constexpr (SINGLE) {   // the pair's two parts first, so that the sum itself is rounded once a pair
            t.mx = add2(fma2(sxy, gy, mul2(cx, gx)), t.mx);
            t.my = add2(fma2(sxy, gx, mul2(cy, gy)), t.my);
        } else {
            t.mx = fma2(sxy, gy, fma2(cx, gx, t.mx));
            t.my = fma2(sxy, gx, fma2(cy, gy, t.my));
        }
        if (!SINGLE && qb.itype < 0.0f) wall_pair(K, rr, dx, dy, h0 && real0, h1 && real1, t.mx, t.my);
    });
}
// the soil side of a cross pair (cross_soil_sums)
template <int SKF, bool FCH>
__device__ __forceinline__ void soil_cross(const PhaseDev<float>& W, const PairK& K, const Own2& o, SumsS2& t, int m, float2 dx,
                                           float2 dy, bool h0, bool h1) {
    const RecA<float> rb = W.recA[m];
    const RecB<float> qb = W.recB[m];
    float2 w, s;
    kernel_pair<SKF, false>(K, fma2(dx, dx, mul2(dy, dy)), h0, h1, w, s);
    float2 q = mul2(splat2(rb.vol * rb.rho * qb.vof), w);
    const float2 ux = add2(splat2(rb.vx), o.nu), uy = add2(splat2(rb.vy), o.nv);
    if constexpr (FCH) {
        const float2 u2 = fma2(ux, ux, mul2(uy, uy));
        q = mul2(q, fma2(splat2(K.kb), two(sqrtf(u2.x), sqrtf(u2.y)), splat2(1.0f)));
    }
    t.cdx = fma2(q, ux, t.cdx);
    t.cdy = fma2(q, uy, t.cdy);
    // the gradient with x_water - x_soil = -(x_a - x_b): the sign is applied to the sum
    const float2 mp = mul2(splat2(rb.vol * qb.p), s);
    t.cpx = fma2(mp, dx, t.cpx);
    t.cpy = fma2(mp, dy, t.cpy);
}
template <int SKF, bool SINGLE, bool FCH>
__device__ __noinline__ SumsS2 soil_alone(PhaseDev<float> P, PhaseDev<float> W, GridGeom g, PairK K, LanePair p) {
    SumsS2 t{};
    const Own2 o(p, P.recA);
    soil_pairs<SKF, SINGLE, true>(P, K, p, o, t, [&](auto&& body) {
        visit_alone(g, P.cell_start, K.thr, P.xs, p, p.k,
                    [&](int m, float2 dx, float2 dy, bool h0, bool h1) { body(P.recA[m], P.recB[m], dx, dy, h0, h1); });
    });
    if constexpr (!SINGLE)
        visit_alone(g, W.cell_start, K.thr, W.xs, p, -1,
                    [&](int m, float2 dx, float2 dy, bool h0, bool h1) { soil_cross<SKF, FCH>(W, K, o, t, m, dx, dy, h0, h1); });
    return t;
}
template <int SKF, bool SINGLE, bool FCH>
__global__ void __launch_bounds__(SPHG_TPB2, SPHG_MINB_S2) k_soil_pass2(PhaseDev<float> P, PhaseDev<float> W, GridGeom g,
                                                                     const __grid_constant__ PairK K, SimConst c, DevCounters* cnt, int slot,
                                                                     StepCtl u) {
    pdl_enter();
    const LanePair p(g, P.xs, P.n);
    const Own2 o(p, P.recA);
    SumsS2 t{};
    int hits0 = 0, hits1 = 0;
    soil_pairs<SKF, SINGLE, false>(P, K, p, o, t, [&](auto&& body) {
        visit_pairs<true>(P, g, p, &cnt->timeout, [&](const Runs3& r, const double2* xs, const RecA<float>* RA,
                                                              const RecB<float>* RB, int s0, int s1, bool a0, bool a1) {
            uint4 unused;
            pair_scan<false>(r, p.lane, K.thr, xs, p.x0, p.x1, s0, s1, a0, a1, unused, hits0, hits1,
                             [&](int m, float2 dx, float2 dy, bool h0, bool h1) {
                if (h0 || h1) body(RA[m], RB[m], dx, dy, h0, h1);
            });
        });
    });
    if constexpr (!SINGLE) {
        PairRuns pr;
        pr.init(g, W.cell_start, p);
        int ch0 = 0, ch1 = 0;
        for (int i = 0, n = pr.parts(); i < n; ++i) {
            bool a0, a1;
            const Runs3 r = pr.part(g, W.cell_start, p, i, a0, a1);
            uint4 unused;
            pair_scan<false>(r, p.lane, K.thr, W.xs, p.x0, p.x1, -1, -1, a0, a1, unused, ch0, ch1,
                             [&](int m, float2 dx, float2 dy, bool h0, bool h1) { soil_cross<SKF, FCH>(W, K, o, t, m, dx, dy, h0, h1); });
        }
    }
    const int hits = p.mine(hits0, hits1);
    const float c23 = K.ks * (2.0f / 3.0f), dh2 = -2.0f * K.ks * (float)K.dh;
    const float ps = c.soil_artificial_stress ? dh2 * (float)c.s_c : 0.0f;
    SoilSums<float> w;
    float con, dl;
    auto sums = [&](const SumsS2& v, auto&& one) {
        const float ta = one(v.ta), tb = one(v.tb), tc = one(v.tc), td = one(v.td);
        con = one(v.con); dl = one(v.dl);
        w.mx = w.my = SINGLE ? 0.0f : 0.0f * (p.lane ? o.rho.y : o.rho.x);   // df3's sums times rho over rho: NaN where rho is infinite
        w.fx = K.ks * one(v.mx); w.fy = K.ks * one(v.my);
        w.xsx = K.kw * one(v.xx); w.xsy = K.kw * one(v.xy);
        w.txx = c23 * (2.0f * ta - tb); w.txy = K.ks * (tc + td); w.tyy = c23 * (2.0f * tb - ta);
        w.vcc = K.ks * (ta + tb); w.wxy = 0.5f * K.ks * (tc - td);
        w.dp = ps * one(v.dpp); w.dsx = ps * one(v.dsx); w.dsxy = ps * one(v.dsxy); w.dsy = ps * one(v.dsy);
        w.cdx = w.cdy = w.cpx = w.cpy = 0.0f;
        if constexpr (!SINGLE) {
            w.cdx = K.kw * one(v.cdx); w.cdy = K.kw * one(v.cdy); w.cpx = -K.ks * one(v.cpx); w.cpy = -K.ks * one(v.cpy);
        }
    };
    sums(t, [&](float2 v) { return p.mine(v); });
    if (p.valid && !all_finite(con, dl, w.fx, w.fy, w.xsx, w.xsy, w.txx, w.txy, w.tyy, w.wxy, w.dp, w.dsx, w.dsxy, w.dsy, w.cdx,
                               w.cdy, w.cpx, w.cpy)) {
        sums(soil_alone<SKF, SINGLE, FCH>(P, W, g, K, p), [&](float2 v) { return p.own(v); });
        if (!c.soil_artificial_stress) w.dp = w.dsx = w.dsxy = w.dsy = 0.0f;   // not 0 times an infinite sum
    }
    w.hits = hits;
    int fail = 0, fail3 = 0;
    if (p.valid) {
        const RecB<float> q = P.recB[p.k];
        w.drho = -K.ks * con + (c.artificial_density ? dh2 * q.c * dl : 0.0f);   // delta_sph(rho) runs before pressure(): the old c
        soil_finish<float, SINGLE>(P, g, c, u, cnt, p.k, p.lane ? o.rho.y : o.rho.x, q.vof, w, fail, fail3);
    }
    count_stats_redux(cnt, slot, slot, hits, p.valid);
    if (c.plasticity == 3) count_fail(cnt, 2, fail);
    if (u.update && u.do_dp) count_fail(cnt, 3, fail3);
}
