// gsw_face.cuh -- the binary32 faces and update of the step kernels, without the IEEE
// division and square-root operators, and the column march that drives them.
//
// The step is bound by instruction issue (4096^2: 83 % of the issue slots, 16 % of the peak DRAM
// throughput). With the operators it takes 30.8 warp instructions per cell, of which their
// sequences, range tests and branches around their slow paths are a third; without them 24.5,
// and 17.5 in the fast arithmetic (20.3 before): 4096^2 step 0.538 -> 0.436 ms and 0.360 ->
// 0.310 ms, the compressed mesh (4096^2, 60 % active) 0.602 -> 0.449 ms and 0.399 -> 0.331 ms.
// Here the roots and quotients are the bare sequences:
//   * sqrt(x): y = rsqrt.approx(x), g = RN(x y), d = x - g g (one FMA, exact),
//     RN(g + d (y / 2)): Newton's correction with the exact residual (P. Markstein, "IA-64 and
//     Elementary Functions", 2000). Checked against the IEEE root for every binary32 x in
//     [2^-100, 2^100] (tests/test_face_gpu.py).
//   * a / b: y = RN(1/b) by one Newton step from rcp.approx (checked for every b in that
//     range and both signs), q = RN(a y), r = a - b q (exact), RN(q + r y). With y = RN(1/b)
//     the value rounded last differs from a / b by less than 3 * 2^-24 half-ulps, and a
//     quotient of two 24-bit significands closer than that to a rounding boundary satisfies
//     a 2^s - b M = c for an odd M and |c| <= 2; all such pairs (|c| <= 8) are enumerated by
//     the test and round correctly. Quotients by one divisor share y.
// The two hold while nothing underflows, so operands outside stated ranges (a non-finite
// value, a depth, bed or speed above 2^17, ...) raise a flag, and the row's face or update is
// evaluated again by the operators (srm_face, wetdry_friction): every value equals the IEEE
// operators' in either case. A nonzero momentum under 2^-100, which a long run holds in up to a
// cell in a hundred (friction and upwinding shrink it until it stays at a few binary32
// quanta), only has its own cell's velocities divided again.
//
// Two faces (or two rows) at a time in packed arithmetic (add/mul.rn.f32x2) was measured and
// is no faster: pairing the operands costs moves (21.0 and 22.4 instructions per cell, where
// the unpaired face took 25.1), and 100 to 128 registers leave half the resident warps
// (4096^2 step 0.472 and 0.459 ms, unpaired 0.453). ptxas also fuses a packed product into a packed sum, with
// --fmad=false too.
//
// In the fast arithmetic (GSW_FAST_ARITH) a root is x rsqrt.approx(x) and a quotient a rcp.approx(b),
// each within 2^-22 of the exact value; nothing is flagged, and divisors of 2^126 and more give 0
// and an infinite operand of a root NaN. The wave speed that sets dt is taken the same way. The
// depth error against binary64 after 16 steps on 3000x4096 is 8.2e-7 where sqrt.approx and
// div.full gave 8.1e-7.
#pragma once
#include "gsw_core.cuh"

namespace gsw {

__device__ __forceinline__ float rcp_approx(float x) {
    float y;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}
__device__ __forceinline__ float rsqrt_approx(float x) {
    float y;
    asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}

// Added to a root's argument: absorbed by any x >= 2^-100, and turns 0 into a finite rsqrt.
#define GSW_ROOT_TINY 0x1p-126f

// sqrt(x), correctly rounded for x = 0 or in [2^-100, 2^100]; for x below, a value under 2^-48.
__device__ __forceinline__ float sqrt_in(float x) {
    const float y = rsqrt_approx(x + GSW_ROOT_TINY);
    const float g = x * y;
#ifdef GSW_FAST_ARITH
    return g;
#else
    return fmaf(fmaf(-g, g, x), 0.5f * y, g);
#endif
}
// RN(1/b), and a / b by it.
__device__ __forceinline__ float rcp_in(float b) {
    const float y = rcp_approx(b);
#ifdef GSW_FAST_ARITH
    return y;
#else
    return fmaf(y, fmaf(-b, y, 1.0f), y);
#endif
}
__device__ __forceinline__ float div_in(float a, float b, float y) {
    const float q = a * y;
#ifdef GSW_FAST_ARITH
    return q;
#else
    return fmaf(fmaf(-b, q, a), y, q);
#endif
}

// The magnitude of x as an unsigned key in which 0 is the largest: one minimum over keys
// finds the smallest nonzero magnitude.
__device__ __forceinline__ uint32_t low_key(float x) { return 2u * __float_as_uint(x) - 1u; }
__device__ __forceinline__ uint32_t min3(uint32_t a, uint32_t b, uint32_t c) { return __vimin3_u32(a, b, c); }
#define GSW_KEY(e) (2u * ((uint32_t)(127 + (e)) << 23) - 1u)       // low_key(2^e)
// Depths, beds and speeds above this are left to the operators. With it as the limit M of a
// cell's |h| + |b| + |u| + |v|, a face's depths are at most 4 M, its wave speeds under 4 M (under 8 M
// from a velocity), the star speed's denominator under 2^6 M^2 = 2^40 and its numerator under
// 2^8 M^3 = 2^59, so that every quotient of a numerator above 2^-80 is a normal number and its
// residual exact. 2^17 leaves the usual no-data values (-9999, -32768, 99999) and elevations in
// feet or centimetres to these faces: at 2^14, terrain lifted by 20000 took 145 us per step where
// 86 is enough (1536x1500).
constexpr float kFaceMax = 0x1p17f;

// Whether gravity and the depth floor are in the ranges the bounds here use. Outside them the
// dense and flat steps take their operator kernels (1536x1500, g = 981: every row by the faces
// here and then again by the operators took 148 us where the operators alone take 100).
__host__ __device__ inline bool face_ranges(float g, float h_min) {
    return g >= 1.0f && g <= 128.0f && h_min >= 0x1p-24f && h_min <= 1.0f;
}
#ifdef GSW_FAST_ARITH
constexpr bool kFastArith = true;
#else
constexpr bool kFastArith = false;
#endif

// A cell as its faces need it: hgx, hgy are half_d times the central bed gradients.
struct FCell { float h, u, v, b, hgx, hgy; };

// RN(a / b) for any operands, through binary64: its quotient has more than twice binary32's
// digits, so rounding it once more gives the binary32 quotient, a subnormal one too. The slow
// paths are not inlined: their registers would count for the march, which calls them on few rows.
static __device__ __noinline__ float2 velocities_general(float hu, float hv, float h) {
    return make_float2((float)((double)hu / (double)h), (float)((double)hv / (double)h));
}

// Depth and velocities (make_prims). Returns whether the cell is outside the ranges of the
// faces.
__device__ __forceinline__ bool make_fcell(FCell& c, float h, float hu, float hv, float b, float h_min) {
    const bool wet = h > h_min;
    c.h = h; c.b = b;
    const float y = rcp_in(h);                          // not used where h is not above h_min
    c.u = wet ? div_in(hu, h, y) : 0.0f;
    c.v = wet ? div_in(hv, h, y) : 0.0f;
#ifdef GSW_FAST_ARITH
    return false;
#else
    const bool bad = !((fabsf(h) + fabsf(b)) + (fabsf(c.u) + fabsf(c.v)) <= kFaceMax);
    if (wet && (bad || min(low_key(hu), low_key(hv)) < GSW_KEY(-100))) {
        const float2 w = velocities_general(hu, hv, h);
        c.u = w.x; c.v = w.y;
    }
    return bad;
#endif
}

// A face's outputs as Face, already scaled by 1/d.
struct FFace { float Fh, Fn, Ft, srcL, srcR; };

// hinv: half of 1/d (a product by 1/2 is exact, so it may be folded into 1/d). g_recip: RN(1/g).
struct FacePhys { float inv_dx, inv_dy, hinv_dx, hinv_dy, half_dx, half_dy, g, g_recip, h_min; };

// The face between cells L and R along one axis (XAXIS: u normal), as srm_face and hllc in
// gsw_core.cuh. Returns whether a value left the range in which the roots and quotients are
// proven (the face is then invalid and srm_face has to evaluate it): a nonzero squared h_rt,
// face depth or numerator below 2^-80, a contact speed above 2^40, a star denominator below
// 2^-40.
// Differences in form, not in value:
//   * min(-a, -b) = -max(a, b); products by a power of two are exact and may be fused;
//   * two dry sides (SL = SR = 0) take the physical flux of L: the side choice and S are
//     forced instead of the speeds;
//   * the star flux is F + S (...) with S = min(SL, 0) on side L, max(SR, 0) on side R: S = 0
//     exactly where the physical flux is meant, and its denominator is then set to 1;
//   * a face whose two cells are below h_min gives zeros: its 1/d is set to zero. DRY_ZERO: also
//     where their beds are not finite, which only the sources show, and only in the fast
//     arithmetic (in the exact one such cells are flagged; 1.5 % of the fast step, which drops
//     these cells' momenta in any case, so only the fast residual has it).
template <bool XAXIS, bool DRY_ZERO>
__device__ __forceinline__ bool face_in(const FCell& L, const FCell& R, const FacePhys& p, FFace& F) {
    const float z = 0.0f;
    const float zL = L.b + (XAXIS ? L.hgx : L.hgy), zR = R.b - (XAXIS ? R.hgx : R.hgy);
    const float zf0 = L.b > R.b ? L.b : R.b;
    const float clip = zR - zL;
    const float dz = (R.b - L.b) - clip;
    const float eL = L.h + L.b, eR = R.h + R.b;
    const float de = eR - eL;
    const float hL = fmaxf(z, (eL + fmaxf(z, fminf(dz, de))) - zf0);
    const float hR = fmaxf(z, (eR + fmaxf(z, -fmaxf(dz, de))) - zf0);
    const float uL = XAXIS ? L.u : L.v, tL = XAXIS ? L.v : L.u, uR = XAXIS ? R.u : R.v, tR = XAXIS ? R.v : R.u;
    // bed sources
    const bool lowL = L.h < p.h_min, lowR = R.h < p.h_min;
    const float inv = lowL && lowR ? z : (XAXIS ? p.inv_dx : p.inv_dy);
    const float hg = 0.5f * p.g;
    {
        const float wL = zf0 - eL, wR = zf0 - eR;
        const float kL = fmaxf(z, fminf(lowR ? INFINITY : clip, wL));
        const float kR = fmaxf(z, fminf(lowL ? INFINITY : -clip, wR));
        F.srcL = ((hg * (hL + L.h)) * ((zf0 - kL) - L.b)) * inv;
        F.srcR = ((hg * (hR + R.h)) * ((zf0 - kR) - R.b)) * inv;
        if (DRY_ZERO) {
            F.srcL = lowL && lowR ? z : F.srcL;
            F.srcR = lowL && lowR ? z : F.srcR;
        }
    }
    // HLLC
    const float aL = sqrt_in(p.g * hL), aR = sqrt_in(p.g * hR);
    const float us = uL + uR;
    const float ust = fmaf(0.5f, us, aL) - aR;
    const float hrt = fmaf(0.5f, aL + aR, 0.25f * (uL - uR));
    const float m = fmaxf(hrt, z);
    const float m2 = m * m;
#ifdef GSW_FAST_ARITH
    const float ast = sqrt_in(p.g * (m2 * p.g_recip));
#else
    const float q0 = m2 * p.g_recip;
    const float ast = sqrt_in(p.g * fmaf(fmaf(-p.g, q0, m2), p.g_recip, q0));   // div_g
#endif
    const bool dryL = hL <= p.h_min, dryR = hR <= p.h_min, both = dryL && dryR;
    const float SL = dryL ? fmaf(-2.0f, aR, uR) : fminf(uL - aL, ust - ast);
    const float SR = dryR ? fmaf(2.0f, aL, uL) : fmaxf(uR + aR, ust + ast);
    const float cR = uR - SR, cL = uL - SL;
    const float den = hR * cR - hL * cL;
    const float num = (SL * hR) * cR - (SR * hL) * cL;
    const float SM = fabsf(den) > 1.0e-14f ? div_in(num, den, rcp_in(den)) : 0.5f * us;
    const bool side = both || SL >= z || SM >= z;                          // L
    const float hP = side ? hL : hR, uP = side ? uL : uR, tP = side ? tL : tR;
    const float S = both ? z : (side ? fminf(SL, z) : fmaxf(SR, z));
    const float D = S == z ? 1.0f : (S - SM) + 1.0e-30f;
    const float nS = S - uP;
    const float hu = hP * uP, ht = hP * tP;
    const float hK = hP * div_in(nS, D, rcp_in(D));
    F.Fh = (hu + S * (hK - hP)) * inv;
    F.Fn = ((hu * uP + (hg * hP) * hP) + S * (hK * SM - hu)) * inv;
    F.Ft = (hu * tP + S * (hK * tP - ht)) * inv;
#ifdef GSW_FAST_ARITH
    return false;
#else
    return !(fabsf(SM) <= 0x1p40f) || !(fabsf(D) >= 0x1p-40f) ||
           min3(min3(low_key(m2), low_key(hL), low_key(hR)), low_key(num), low_key(nS)) < GSW_KEY(-80);
#endif
}

// The same face by the operators (the slow rows).
template <bool XAXIS>
static __device__ __noinline__ void face_general(const FCell& L, const FCell& R, const FacePhys& p, FFace& F) {
    Cell<float> a, b;
    a.h = L.h; a.hu = 0.0f; a.hv = 0.0f; a.u = L.u; a.v = L.v; a.b = L.b; a.eta = L.h + L.b; a.gx = L.hgx; a.gy = L.hgy;
    b.h = R.h; b.hu = 0.0f; b.hv = 0.0f; b.u = R.u; b.v = R.v; b.b = R.b; b.eta = R.h + R.b; b.gx = R.hgx; b.gy = R.hgy;
    Face<float> f;
    srm_face<float, XAXIS>(a, b, 1.0f, XAXIS ? p.inv_dx : p.inv_dy, p.g, p.h_min, f, p.g_recip);
    F.Fh = f.Fh; F.Fn = f.Fn; F.Ft = f.Ft; F.srcL = f.srcL; F.srcR = f.srcR;
}

// bad: whether a cell of the face is outside the ranges (a y-face: the cell to the left is; the
// lane to the right holds the other).
template <bool XAXIS, bool DRY_ZERO>
__device__ __forceinline__ void face(const FCell& L, const FCell& R, const FacePhys& p, bool bad, FFace& F) {
    const bool out = face_in<XAXIS, DRY_ZERO>(L, R, p, F);
#ifndef GSW_FAST_ARITH
    bool slow = bad || out;
    if (__any_sync(0xffffffffu, slow)) {
        if (!XAXIS) slow = __shfl_down_sync(0xffffffffu, bad, 1) || slow;      // the cell to the right
        // a face of two cells below h_min is zero whatever their beds (no-data values among
        // them), so it does not send its warp to the operators
        if (__any_sync(0xffffffffu, slow && !(L.h < p.h_min && R.h < p.h_min))) {
            const FCell a = L, b = R;          // copies: the march's own stay in registers
            const FacePhys q = p;
            FFace G;
            face_general<XAXIS>(a, b, q, G);
            F = G;
        } else if (slow) {
            F.Fh = F.Fn = F.Ft = F.srcL = F.srcR = 0.0f;
        }
    }
#endif
}

// ----------------------------------------------------------------------------- update
struct FState { float h, hu, hv; uint32_t lam; };     // lam: the wave speed's bits

// The update by the operators.
template <bool FLAT, bool REFPOW>
static __device__ __noinline__ void update_general(FState& s, bool friction, float n, float dt, float g, float h_min,
                                                   float vcap, bool quadratic, bool keep_h, float h_cfl) {
    wetdry_friction<float>(s.h, s.hu, s.hv, friction, n, dt, g, h_min, vcap, quadratic, keep_h, REFPOW);
    s.lam = FLAT ? lam_flat_bits32(s.h, s.hu, s.hv, g, h_min, h_cfl) : lam_dense_bits32(s.h, s.hu, s.hv, g, h_cfl);
}

// wetdry_friction (quadratic friction, keep-h) and the wave speed of the new state in one:
// the reciprocal of the depth is shared by the friction's velocities and the wave speed's.
// FLAT: the flat loop's L2 speed of a cell that h_min_cfl does not floor (h_cfl is h_min there),
// else the dense loop's maximum norm.
// Returns whether a value is outside the proven ranges (s is then unchanged and
// update_general has to be used): non-finite or large values, a nonzero squared speed under
// 2^-100, a speed above vcap (its limiter divides again), a friction number above 2^100. A
// momentum under 2^-100 needs no test: its velocity is under 2^-76 whatever its last bits, and
// its square rounds to 0. Neither do the wave speed's own root and quotient: where one is not
// exact it is below 2^-48 and absorbed by sqrt(g h) >= 2^-12, or, in a dense cell between h_cfl
// and h_min, its momentum is 0 and g h at least 2^-90 by the host's test of h_cfl.
template <bool FLAT, bool REFPOW>
__device__ __forceinline__ bool update_in(FState& s, bool friction, float n, float dt, float g, float h_min, float vcap,
                                          float h_cfl) {
    const bool dry = s.h < h_min;
    float a = dry ? 0.0f : s.hu, b = dry ? 0.0f : s.hv;
    const float hs = dry ? h_min : s.h;
    const float y = rcp_in(hs);
    float u = div_in(a, hs, y), v = div_in(b, hs, y);
#ifndef GSW_FAST_ARITH
    bool bad = !(fabsf(s.h) + (fabsf(u) + fabsf(v)) <= kFaceMax);
#endif
    if (friction) {
        const float x = u * u + v * v;
        const float U = sqrt_in(x);
        const float h43 = REFPOW ? pow_m43_ref(hs) : pow_m43(hs);
#ifdef GSW_FAST_ARITH
        if (U > vcap) {
            const float c = gsqrt(gdiv(1.0f, (1.0e-10f + dt) * g * h43 * (U + 1.0e-30f)));
            if (c > n) n = c;
        }
#endif
        const float Cf = g * n * n * h43;
        const float X = fmaf(2.0f, 2.0f * dt * Cf * U, 1.0f);
        const float D = sqrt_in(X) + 1.0f;
        const float alpha = div_in(2.0f, D, rcp_in(D));
        a *= alpha; b *= alpha;
#ifndef GSW_FAST_ARITH
        bad = bad || U > vcap || !(X <= 0x1p100f) || low_key(x) < GSW_KEY(-100);
#endif
        if (FLAT) { u = div_in(a, hs, y); v = div_in(b, hs, y); }
    }
#ifndef GSW_FAST_ARITH
    if (bad) return true;
#endif
    s.hu = a; s.hv = b;
    if (dry) s.h = fmaxf(s.h, 0.0f);
    const float c = sqrt_in(g * s.h);
    const float w = FLAT ? sqrt_in(u * u + v * v) : div_in(fmaxf(fabsf(a), fabsf(b)), hs, y);
    s.lam = s.h < h_cfl ? 0u : __float_as_uint(w + c);
#ifdef GSW_FAST_ARITH   // a non-finite state has to show: fmaxf drops a NaN
    if (!(fabsf(s.h) + (fabsf(a) + fabsf(b)) <= 3.0e38f)) s.lam = 0x7f800000u;
#endif
    return false;
}

// ------------------------------------------------------------------------------ march
// n rows of one warp's 32 columns (lane = column; lanes 0 and 31 are halo columns), walked
// downwards with the x-face above the current row and the row itself in registers.
//   A: the rows' data. state(k, h, hu, hv), bed(k); bed_out(k): of lane 0 (31) the bed left
//      (right) of its own column.
//   U: what is done with a row. pre(k): loads issued before the faces; row(k, h, rh, rhu, rhv):
//      the row's old depth and residual. kDryZero: as face_in's DRY_ZERO.
// The march starts one row early, for the x-face above row 0 alone. Rows -2 .. n + 1 are read.
// `general` (warp-uniform): every row by the operators.
constexpr int kMarchUnroll = 1;
template <class A, class U>
__device__ __forceinline__ void march_rows(const A& acc, U& upd, int n, const FacePhys& ph, bool general) {
    const int lane = threadIdx.x;
    FCell cur, nx;
    float sh, shu, shv;
    acc.state(-1, sh, shu, shv);
    const float b0 = acc.bed(-2), b1 = acc.bed(-1);
    float bn = acc.bed(0), pb = acc.bed(1);
    bool bad_cur = make_fcell(cur, sh, shu, shv, b1, ph.h_min) || general;
    acc.state(0, sh, shu, shv);                // the next row's state, in flight during this row's faces
    cur.hgx = ph.half_dx * ((bn - b0) * ph.hinv_dx);
    cur.hgy = 0.0f;
    float wFh = 0.0f, wFn = 0.0f, wFt = 0.0f, wsR = 0.0f;
#pragma unroll kMarchUnroll
    for (int k = -1; k < n; ++k) {
        if (k >= 0) upd.pre(k);
        const bool bad_nx = make_fcell(nx, sh, shu, shv, bn, ph.h_min) || general;
        const float b2 = pb;
        if (k + 1 < n) {
            acc.state(k + 2, sh, shu, shv);
            pb = acc.bed(k + 3);
        }
        nx.hgx = ph.half_dx * ((b2 - cur.b) * ph.hinv_dx);
        {
            float bl = __shfl_up_sync(0xffffffffu, bn, 1), br = __shfl_down_sync(0xffffffffu, bn, 1);
            if (lane == 0 || lane == 31) {
                const float bo = acc.bed_out(k + 1);
                if (lane == 0) bl = bo; else br = bo;
            }
            nx.hgy = ph.half_dy * ((br - bl) * ph.hinv_dy);
        }
        float rh, rhu, rhv;
        // the residual, in the reference's order per component (E, W, N, S): the leading
        // 0 - E + W is formed as W - E (the same rounding; only a zero's sign can differ)
        // a row pair below h_min has no fluxes, whatever its beds
        if (__any_sync(0xffffffffu, !(cur.h < ph.h_min) || !(nx.h < ph.h_min))) {
            FFace E;
            face<true, U::kDryZero>(cur, nx, ph, bad_cur || bad_nx, E);
            rh = wFh - E.Fh;
            rhu = (wFn - (E.Fn + E.srcL)) + wsR;
            rhv = wFt - E.Ft;
            wFh = E.Fh; wFn = E.Fn; wFt = E.Ft; wsR = E.srcR;
            if (k >= 0) {
                FCell rn;
                rn.h = __shfl_down_sync(0xffffffffu, cur.h, 1);
                rn.u = __shfl_down_sync(0xffffffffu, cur.u, 1);
                rn.v = __shfl_down_sync(0xffffffffu, cur.v, 1);
                rn.b = __shfl_down_sync(0xffffffffu, cur.b, 1);
                rn.hgy = __shfl_down_sync(0xffffffffu, cur.hgy, 1);
                rn.hgx = rn.hgy;               // unused by a y-face
                FFace N;
                face<false, U::kDryZero>(cur, rn, ph, bad_cur, N);
                // the y-face left of the column comes from the lane to the left
                rh = (rh - N.Fh) + __shfl_up_sync(0xffffffffu, N.Fh, 1);
                rhu = (rhu - N.Ft) + __shfl_up_sync(0xffffffffu, N.Ft, 1);
                rhv = (((rhv - N.Fn) - N.srcL) + __shfl_up_sync(0xffffffffu, N.Fn, 1)) +
                      __shfl_up_sync(0xffffffffu, N.srcR, 1);
            }
        } else {                               // every cell of the two rows below h_min
            rh = wFh; rhu = wFn + wsR; rhv = wFt;
            wFh = wFn = wFt = wsR = 0.0f;
        }
        if (k >= 0) upd.row(k, cur.h, rh, rhu, rhv);
        cur = nx;
        bn = b2;
        bad_cur = bad_nx;
    }
}

}  // namespace gsw
