// gsw_flat_brick.cuh -- the per-brick march of the compressed mesh (shared by the flat
// solver's kernels and the ensemble's persistent step).
#pragma once
#include "gsw_common.cuh"
#include "gsw_face.cuh"

namespace gsw {

// Mesh arrays of one brick storage (a compressed mesh, or all members of an ensemble).
template <typename T>
struct FlatMesh {
    const T* q0; const T* q1; const T* q2;
    T* o0; T* o1; T* o2;
    const T* b;
    const uint8_t* flags;
    const uint8_t* ncls;
    T* max_h;
    const int32_t* bij; const int32_t* bnbr;
    int64_t nb; int bh;
};

// Physics of one solver (one ensemble member).
template <typename T>
struct FlatPhys {
    T inv_dx, inv_dy, half_dx, half_dy, g, h_min, h_min_cfl, vcap;
    int linf, quad, keep_h, rain_kind, ngh, nx, ny;
    const T* rain; const T* ntab;
    const int32_t* lookup;   // GSW_RAIN_LOOKUP: per-slot column of the rain row
    int ncol;
    T g_recip;               // RN(1/g) for the star depth's h / g, or 0 (gsw_core.cuh div_g)
    int ref_pow;             // 1: Manning's h^(-4/3) by powf (GSW_ARITH_EXACT), 0: by pow_m43 (read by
                             // the adjoint; the step kernels take it as their REFPOW parameter)
};

// Row segments per brick when the caller leaves the choice to the library: one warp
// per brick once the bricks fill the `warps` that can run at once twice over
// (throughput), else 2 or 4 warps per brick so that fewer bricks still keep enough
// warps busy and each warp's march is shorter (latency). A segment recomputes the
// x-face above its first row and reads two rows past each end.
__host__ __device__ __forceinline__ int auto_segments(int64_t bricks, int64_t warps, int bh) {
    int s = bricks >= 2 * warps ? 1 : (2 * bricks >= warps ? 2 : 4);
    while (s > 1 && bh % s != 0) s >>= 1;
    return s;
}

// For the flat kernels' argument struct
template <typename T>
struct FlatK {
    FlatMesh<T> m; FlatPhys<T> ph; const GswLoopState* st; unsigned long long* lam; int segs;
    int64_t b0, b1;    // bricks [b0, b1) are stepped
    bool general;      // binary32: outside the ranges of gsw_face.cuh
};

// Slot of brick-relative (row, lane). Lanes 0/31 of the rows above/below the brick are
// never used by an output cell; they read the zero brick.
struct BrickView {
    int64_t self, up, down, left, right, zero, BS;
    int bh;
    __device__ __forceinline__ int64_t slot(int r, int lane) const {
        if (r >= 0 && r < bh) {
            if (lane == 0) return left * BS + (int64_t)r * GSW_BRICK_PITCH + (GSW_BRICK_W - 1);
            if (lane == 31) return right * BS + (int64_t)r * GSW_BRICK_PITCH;
            return self * BS + (int64_t)r * GSW_BRICK_PITCH + (lane - 1);
        }
        if (lane == 0 || lane == 31) return zero * BS;
        if (r < 0) return up * BS + (int64_t)(bh + r) * GSW_BRICK_PITCH + (lane - 1);
        return down * BS + (int64_t)(r - bh) * GSW_BRICK_PITCH + (lane - 1);
    }
    // outer bed neighbour of the edge lanes, for the y-gradient
    __device__ __forceinline__ int64_t outer_b(int r, int lane) const {
        if (r < 0 || r >= bh) return zero * BS;
        if (lane == 0) return left * BS + (int64_t)r * GSW_BRICK_PITCH + (GSW_BRICK_W - 2);
        return right * BS + (int64_t)r * GSW_BRICK_PITCH + 1;
    }
};

template <typename T>
__device__ __forceinline__ T grad_y_flat(const FlatMesh<T>& m, const FlatPhys<T>& ph, const BrickView& v, T bc,
                                         int r, int lane) {
    T bl = __shfl_up_sync(0xffffffffu, bc, 1);
    T br = __shfl_down_sync(0xffffffffu, bc, 1);
    if (lane == 0)  bl = ld_state(m.b + v.outer_b(r, 0));
    if (lane == 31) br = ld_state(m.b + v.outer_b(r, 31));
    return (T)0.5 * (br - bl) * ph.inv_dy;
}

template <typename T>
__device__ __forceinline__ Cell<T> shfl_down_cell(const Cell<T>& c) {
    Cell<T> r;
    r.h = __shfl_down_sync(0xffffffffu, c.h, 1);
    r.u = __shfl_down_sync(0xffffffffu, c.u, 1);
    r.v = __shfl_down_sync(0xffffffffu, c.v, 1);
    r.eta = __shfl_down_sync(0xffffffffu, c.eta, 1);
    r.b = __shfl_down_sync(0xffffffffu, c.b, 1);
    r.gy = __shfl_down_sync(0xffffffffu, c.gy, 1);
    r.gx = r.gy; r.hu = r.h; r.hv = r.h;
    return r;
}

template <typename T>
__device__ __forceinline__ Face<T> shfl_up_face(const Face<T>& f) {
    Face<T> r;
    r.Fh = __shfl_up_sync(0xffffffffu, f.Fh, 1);
    r.Fn = __shfl_up_sync(0xffffffffu, f.Fn, 1);
    r.Ft = __shfl_up_sync(0xffffffffu, f.Ft, 1);
    r.srcR = __shfl_up_sync(0xffffffffu, f.srcR, 1);
    r.srcL = r.srcR;
    r.wet = true;   // unused: the residual adds a dry face's zeros
    return r;
}

__device__ __forceinline__ FacePhys face_phys(const FlatPhys<float>& ph) {
    return {ph.inv_dx, ph.inv_dy, 0.5f * ph.inv_dx, 0.5f * ph.inv_dy, ph.half_dx, ph.half_dy,
            ph.g, ph.g_recip != 0.0f ? ph.g_recip : rcp_in(ph.g), ph.h_min};
}

// Slots of one lane's rows of a brick, as BrickView::slot, by one base per row range. I: the
// slots' integer type, 32-bit where the mesh has fewer than 2^31 slots (a 64-bit base costs
// registers and address arithmetic on every access), else 64-bit.
template <typename I>
struct FlatRows {
    const FlatMesh<float>& m;
    I in, up, down, out;             // slots of row 0 continued from inside / above / below; lane 0/31: beyond
    I zero;
    int r0, bh;
    __device__ __forceinline__ I slot(int r) const {
        return (r < 0 ? up : (r >= bh ? down : in)) + (I)(r * GSW_BRICK_PITCH);
    }
    __device__ __forceinline__ void state(int k, float& h, float& hu, float& hv) const {
        const I s = slot(r0 + k);
        h = ld_state(m.q0 + s); hu = ld_state(m.q1 + s); hv = ld_state(m.q2 + s);
    }
    __device__ __forceinline__ float bed(int k) const { return ld_state(m.b + slot(r0 + k)); }
    __device__ __forceinline__ float bed_out(int k) const {
        const int r = r0 + k;
        return ld_state(m.b + (r < 0 || r >= bh ? zero : out + (I)(r * GSW_BRICK_PITCH)));
    }
};

template <typename I>
__device__ __forceinline__ FlatRows<I> flat_rows(const FlatMesh<float>& m, const BrickView& v, int r0, int lane) {
    const I BS = (I)(v.bh * GSW_BRICK_PITCH);
    FlatRows<I> a = {m, 0, 0, 0, 0, (I)v.zero * BS, r0, v.bh};
    const bool halo = lane == 0 || lane == 31;
    a.in = lane == 0 ? (I)v.left * BS + (GSW_BRICK_W - 1) : lane == 31 ? (I)v.right * BS : (I)v.self * BS + (lane - 1);
    a.up = (halo ? a.zero : (I)v.up * BS + (lane - 1)) + BS;         // halo lanes read the zero brick there
    a.down = (halo ? a.zero : (I)v.down * BS + (lane - 1)) - BS;
    a.out = lane == 0 ? (I)v.left * BS + (GSW_BRICK_W - 2) : (I)v.right * BS + 1;
    return a;
}

// One row's update (STEP) or its residual. REFPOW: Manning's h^(-4/3) by powf
// (GSW_ARITH_EXACT) instead of pow_m43. LEAN: the production configuration compiled in (rain
// none or uniform, quadratic friction, keep-h, the L2 wave-speed norm); the same bits as the
// general path.
template <typename I, bool STEP, bool REFPOW, bool LEAN>
struct FlatRow {
    static constexpr bool kDryZero = kFastArith && !STEP;
    const FlatMesh<float>& m;
    const FlatPhys<float>& ph;
    I base;                          // the lane's slot of row 0
    int bi, bj, r0, lane;
    float dt, rate;
    const float* frame;
    bool general;
    bool out_lane;
    uint32_t lam32 = 0u;             // the L2 norm's key
    unsigned long long lam64 = 0ull; // the general kernel's (either norm)
    uint8_t f = 0, cls = 0;
    float mh = 0.0f;
    __device__ __forceinline__ void pre(int k) {
        // the slot flag, class id and running maximum, loaded before the faces so that their
        // latency is hidden (the production kernel; the general one loads late)
        if (LEAN && STEP && out_lane) {
            const I o = base + (I)((r0 + k) * GSW_BRICK_PITCH);
            f = m.flags[o];
            if (m.ncls) cls = m.ncls[o];
            if (m.max_h != nullptr) mh = m.max_h[o];
        }
    }
    __device__ __forceinline__ void row(int k, float h, float rh, float rhu, float rhv) {
        if (!out_lane) return;
        const I o = base + (I)((r0 + k) * GSW_BRICK_PITCH);
        const uint8_t fl = (LEAN && STEP) ? f : m.flags[o];
        if (!(fl & GSW_SLOT_STORED)) return;
        const bool active = (fl & GSW_SLOT_ACTIVE) != 0;
        if (!STEP) {
            m.o0[o] = active ? rh : 0.0f; m.o1[o] = active ? rhu : 0.0f; m.o2[o] = active ? rhv : 0.0f;
            return;
        }
        FState s;
        s.h = h;
        s.hu = ld_state(m.q1 + o);                       // reloaded: not carried down the march
        s.hv = ld_state(m.q2 + o);
        if (active) {
            if (ph.rain_kind == GSW_RAIN_UNIFORM) rh = rh + rate;
            else if (!LEAN && ph.rain_kind == GSW_RAIN_GRIDDED) {
                const int i = bi * m.bh + r0 + k, j = bj * GSW_BRICK_W + (lane - 1);
                rh = rh + frame[(int64_t)(i - ph.ngh) * ph.ny + (j - ph.ngh)];
            } else if (!LEAN && ph.rain_kind == GSW_RAIN_LOOKUP) {
                rh = rh + frame[ph.lookup[o]];
            }
            s.h = h + dt * rh;
            s.hu = s.hu + dt * rhu;
            s.hv = s.hv + dt * rhv;
            const float n = m.ncls ? ph.ntab[LEAN ? cls : m.ncls[o]] : ph.ntab[0];
            // a wet cell whose wave speed divides by h_min_cfl instead of its depth
            bool slow = general || (!LEAN && (ph.quad == 0 || ph.keep_h == 0)) ||
                        (s.h < ph.h_min_cfl && !(s.h < ph.h_min));
            if (!slow) slow = update_in<true, REFPOW>(s, true, n, dt, ph.g, ph.h_min, ph.vcap, ph.h_min);
            if (slow) {
                FState g = s;                         // a copy: s itself stays in registers
                update_general<true, REFPOW>(g, true, n, dt, ph.g, ph.h_min, ph.vcap, LEAN || ph.quad != 0,
                                             LEAN || ph.keep_h != 0, ph.h_min_cfl);
                s = g;
            }
            if (LEAN || ph.linf == 0) {
                lam32 = max(lam32, s.lam);
            } else {
                const unsigned long long lb = lam_flat_bits(s.h, s.hu, s.hv, ph.g, ph.h_min, ph.h_min_cfl, true);
                lam64 = lb > lam64 ? lb : lam64;
            }
        }
        m.o0[o] = s.h; m.o1[o] = s.hu; m.o2[o] = s.hv;
        if (m.max_h != nullptr && s.h > (LEAN ? mh : m.max_h[o])) m.max_h[o] = s.h;
    }
};

// Rows [r0, r1) of one brick by the operators: binary64 (the adjoint's derivative checks), and
// binary32 outside the ranges of gsw_face.cuh. Template parameters and result as flat_brick's.
template <typename T, bool STEP, bool REFPOW, bool LEAN>
__device__ __forceinline__ unsigned long long flat_brick_operators(const FlatMesh<T>& m, const FlatPhys<T>& ph,
                                                                   const BrickView& v, int bi, int bj, int r0, int r1,
                                                                   T dt, T rate, const T* frame) {
    const int lane = threadIdx.x;
    const int64_t bidx = v.self;
    unsigned long long lam_local = 0ull;
    uint32_t lam32 = 0u;             // binary32: the L2 norm's key
    const int bh = m.bh;
    Cell<T> cur, nx;
    const T b_m2 = ld_state(m.b + v.slot(r0 - 2, lane));
    { const int64_t s = v.slot(r0 - 1, lane); cur.h = ld_state(m.q0 + s); cur.hu = ld_state(m.q1 + s); cur.hv = ld_state(m.q2 + s); cur.b = ld_state(m.b + s); }
    { const int64_t s = v.slot(r0, lane); nx.h = ld_state(m.q0 + s); nx.hu = ld_state(m.q1 + s); nx.hv = ld_state(m.q2 + s); nx.b = ld_state(m.b + s); }
    T b_next = ld_state(m.b + v.slot(r0 + 1, lane));
    // prefetch of the row after next (rows up to bh+1 exist: the brick below or the zero brick)
    int64_t sp = v.slot(r0 + 1, lane);
    T pf_h = ld_state(m.q0 + sp), pf_hu = ld_state(m.q1 + sp), pf_hv = ld_state(m.q2 + sp);
    T pf_b = ld_state(m.b + v.slot(r0 + 2, lane));
    make_prims(cur, ph.h_min);
    make_prims(nx, ph.h_min);
    cur.gx = (T)0.5 * (nx.b - b_m2) * ph.inv_dx;
    cur.gy = (T)0;
    nx.gx = (T)0.5 * (b_next - cur.b) * ph.inv_dx;
    nx.gy = grad_y_flat<T>(m, ph, v, nx.b, r0, lane);
    Face<T> Wf;
    srm_face<T, true>(cur, nx, ph.half_dx, ph.inv_dx, ph.g, ph.h_min, Wf, ph.g_recip);
    cur = nx;
    for (int r = r0; r < r1; ++r) {
        // loaded before the faces, as FlatRow::pre
        uint8_t f_r = 0, cls_r = 0;
        T mh_r = (T)0;
        if (LEAN && STEP && lane >= 1 && lane <= 30) {
            const int64_t o = bidx * v.BS + (int64_t)r * GSW_BRICK_PITCH + (lane - 1);
            f_r = m.flags[o];
            if (m.ncls) cls_r = m.ncls[o];
            if (m.max_h != nullptr) mh_r = m.max_h[o];
        }
        nx.h = pf_h; nx.hu = pf_hu; nx.hv = pf_hv;
        nx.b = b_next;
        const T b_p2 = pf_b;
        if (r + 1 < r1) {
            sp = v.slot(r + 2, lane);
            pf_h = ld_state(m.q0 + sp); pf_hu = ld_state(m.q1 + sp); pf_hv = ld_state(m.q2 + sp);
            pf_b = ld_state(m.b + v.slot(r + 3, lane));
        }
        make_prims(nx, ph.h_min);
        nx.gx = (T)0.5 * (b_p2 - cur.b) * ph.inv_dx;
        nx.gy = grad_y_flat<T>(m, ph, v, nx.b, r + 1, lane);
        Face<T> Ef;
        srm_face<T, true>(cur, nx, ph.half_dx, ph.inv_dx, ph.g, ph.h_min, Ef, ph.g_recip);
        // the residual in the reference's order (E, W, N, S per component; accumulate() in
        // gsw_core.cuh), the E and W parts before the y-face so that W is released early.
        // A dry face (skipped by the reference) holds +0 in every field, and adding or
        // subtracting +0 leaves these sums unchanged: they start at +0 and are never -0
        // (an IEEE sum or difference is -0 only from a -0 left operand; the fast
        // compilation's flush to zero can make one, whose sign may then differ), so no test of
        // the wet flag is needed.
        T rh = (T)0, rhu = (T)0, rhv = (T)0;
        rh = rh - Ef.Fh; rhu = rhu - Ef.Fn; rhv = rhv - Ef.Ft; rhu = rhu - Ef.srcL;
        rh = rh + Wf.Fh; rhu = rhu + Wf.Fn; rhv = rhv + Wf.Ft; rhu = rhu + Wf.srcR;
        Wf = Ef;
        const Cell<T> rn = shfl_down_cell<T>(cur);
        {
            Face<T> Nf;
            srm_face<T, false>(cur, rn, ph.half_dy, ph.inv_dy, ph.g, ph.h_min, Nf, ph.g_recip);
            const Face<T> Sf = shfl_up_face<T>(Nf);
            rh = rh - Nf.Fh; rhu = rhu - Nf.Ft; rhv = rhv - Nf.Fn; rhv = rhv - Nf.srcL;
            rh = rh + Sf.Fh; rhu = rhu + Sf.Ft; rhv = rhv + Sf.Fn; rhv = rhv + Sf.srcR;
        }
        if (lane >= 1 && lane <= 30) {
            const int64_t o = bidx * v.BS + (int64_t)r * GSW_BRICK_PITCH + (lane - 1);
            const uint8_t f = (LEAN && STEP) ? f_r : m.flags[o];
            if (f & GSW_SLOT_STORED) {
                const bool active = (f & GSW_SLOT_ACTIVE) != 0;
                if (!STEP) {
                    if (!active) { rh = (T)0; rhu = (T)0; rhv = (T)0; }
                    m.o0[o] = rh; m.o1[o] = rhu; m.o2[o] = rhv;
                } else if (!active) {
                    m.o0[o] = cur.h; m.o1[o] = ld_state(m.q1 + o); m.o2[o] = ld_state(m.q2 + o);
                    if (m.max_h != nullptr && cur.h > (LEAN ? mh_r : m.max_h[o])) m.max_h[o] = cur.h;
                } else {
                    T rr0 = rh;
                    if (ph.rain_kind == GSW_RAIN_UNIFORM) rr0 = rr0 + rate;
                    else if (!LEAN && ph.rain_kind == GSW_RAIN_GRIDDED) {
                        const int i = bi * bh + r, j = bj * GSW_BRICK_W + (lane - 1);
                        rr0 = rr0 + frame[(int64_t)(i - ph.ngh) * ph.ny + (j - ph.ngh)];
                    } else if (!LEAN && ph.rain_kind == GSW_RAIN_LOOKUP) {
                        rr0 = rr0 + frame[ph.lookup[o]];
                    }
                    T h = cur.h + dt * rr0;
                    T hu = ld_state(m.q1 + o) + dt * rhu;       // reloaded: not carried down the march
                    T hv = ld_state(m.q2 + o) + dt * rhv;
                    const T n = m.ncls ? ph.ntab[LEAN ? cls_r : m.ncls[o]] : ph.ntab[0];
                    wetdry_friction<T>(h, hu, hv, true, n, dt, ph.g, ph.h_min, ph.vcap,
                                       LEAN || ph.quad != 0, LEAN || ph.keep_h != 0, REFPOW);
                    m.o0[o] = h; m.o1[o] = hu; m.o2[o] = hv;
                    if (m.max_h != nullptr && h > (LEAN ? mh_r : m.max_h[o])) m.max_h[o] = h;
                    if (sizeof(T) == 4 && (LEAN || ph.linf == 0)) {
                        lam32 = max(lam32, lam_flat_bits32((float)h, (float)hu, (float)hv, (float)ph.g, (float)ph.h_min,
                                                           (float)ph.h_min_cfl));
                    } else {
                        const unsigned long long lb = lam_flat_bits(h, hu, hv, ph.g, ph.h_min, ph.h_min_cfl, ph.linf != 0);
                        lam_local = lb > lam_local ? lb : lam_local;
                    }
                }
            }
        }
        cur = nx;
        b_next = b_p2;
    }
    const unsigned long long l = lam_bits_of32(lam32);
    return l > lam_local ? l : lam_local;
}

// Rows [r0, r1) of one brick, walked by one warp. A segment reads rows r0-2 .. r1+1 through
// the brick view (the bricks above and below past the brick's edge) and recomputes the x-face
// above row r0 from the same inputs as the face below row r0-1, so splitting a brick's rows
// among warps changes no value. STEP: the fused step (returns this lane's wave speed bits);
// otherwise the residual. `frame` is the gridded rain frame, or null. I: as FlatRows. OPERATORS:
// every row by the operators; general (warp-uniform): the same where it is known on the device only
// (an ensemble's member), by the rows' fallback.
template <typename T, typename I, bool STEP, bool REFPOW, bool LEAN, bool OPERATORS>
__device__ __forceinline__ unsigned long long flat_brick(const FlatMesh<T>& m, const FlatPhys<T>& ph, int64_t bidx,
                                                         int r0, int r1, T dt, T rate, const T* frame,
                                                         bool general) {
    const int lane = threadIdx.x;
    BrickView v;
    v.BS = (int64_t)m.bh * GSW_BRICK_PITCH;
    v.bh = m.bh;
    v.self = bidx;
    v.up = m.bnbr[4 * bidx + 0]; v.down = m.bnbr[4 * bidx + 1];
    v.left = m.bnbr[4 * bidx + 2]; v.right = m.bnbr[4 * bidx + 3];
    v.zero = m.nb;
    const int bi = m.bij[2 * bidx], bj = m.bij[2 * bidx + 1];
    if constexpr (sizeof(T) == 4 && !OPERATORS) {
        const FlatRows<I> acc = flat_rows<I>(m, v, r0, lane);
        FlatRow<I, STEP, REFPOW, LEAN> upd = {m, ph, (I)(bidx * v.BS) + (lane - 1), bi, bj, r0, lane, dt, rate, frame, general,
                                           lane >= 1 && lane <= 30};
        march_rows(acc, upd, r1 - r0, face_phys(ph), general);
        const unsigned long long l = lam_bits_of32(upd.lam32);
        return LEAN || l > upd.lam64 ? l : upd.lam64;
    } else {
        return flat_brick_operators<T, STEP, REFPOW, LEAN>(m, ph, v, bi, bj, r0, r1, dt, rate, frame);
    }
}

}  // namespace gsw
