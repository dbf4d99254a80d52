// gsw_dense.cu -- dense-grid kernels of the GeoSWE step for sm_100a and their C ABI:
// the fused step and residual (the column march of gsw_dense_march.cuh), the standalone
// wave speed, the ghost fill, the stage boundary.
#include "gsw_dense_march.cuh"
#include "gsw_fast.h"

namespace gsw {

// Standalone wave speed of the current state over the interior (lammax_fp32_lean): a lane
// per column, four rows of loads in flight, no division of a cell index (8192^2: 0.43 ms with
// one, of a 0.12 ms copy's worth of bytes). A block's warps lie side by side over the columns, or,
// on a grid narrower than they are together, `1 << wshift` of them side by side and the others on
// the next rows (narrow grids left them idle: a step of 200000x12 728 us where 609 are enough).
template <typename T>
__global__ void __launch_bounds__(256) dense_lammax_kernel(DenseK<T> p, unsigned long long* out, int wshift) {
    chain_begin();
    const int nx = p.nxp - 2 * p.ngh, ny = p.nyp - 2 * p.ngh;
    unsigned long long lam = 0ull;
    const int iy = (int)(((blockIdx.x << wshift) + (threadIdx.y & ((1u << wshift) - 1u))) * 32 + threadIdx.x);
    const int rows = 8 >> wshift, step = (int)gridDim.y * rows;
    if (iy < ny) {
#pragma unroll 4
        for (int ix = blockIdx.y * rows + (threadIdx.y >> wshift); ix < nx; ix += step) {
            const int64_t o = (int64_t)(ix + p.ngh) * p.pitch + (iy + p.ngh);
            const T h = p.q0[o], hu = p.q1[o], hv = p.q2[o];
            const unsigned long long lb = lam_dense_bits(h, hu, hv, p.g, p.h_cfl);
            const bool skip = p.cfl_skip != nullptr && p.cfl_skip[(int64_t)ix * ny + iy] != 0;
            lam = !skip && lb > lam ? lb : lam;
        }
    }
    block_max_to(lam, out);
}

// Ghost fill (bc.py:50-172). apply_bc_2d fills the x faces over all columns, then the
// y faces over all rows, so a corner ends up as the y rule applied to the x-filled cell
// of its row. One launch computes every ghost directly from interior cells: x-ghost
// rows over interior columns, y-ghost columns over interior rows, and the corners by
// composing the two rules, which is what the two passes produce.
__device__ __forceinline__ int bc_src(int kind, int g, int n, int ngh) {
    // source index of ghost g along an axis of length n, for EXTRAPOLATE/WALL/PERIODIC
    if (g < ngh) {
        const int k = g;
        return kind == GSW_BC_WALL ? (2 * ngh - 1 - k) : kind == GSW_BC_PERIODIC ? (n - 2 * ngh + k) : ngh;
    }
    const int k = g - (n - ngh);
    return kind == GSW_BC_WALL ? (n - ngh - 1 - k) : kind == GSW_BC_PERIODIC ? (ngh + k) : (n - ngh - 1);
}

// blockIdx.y is the ghost row (over every column, corners included) or, from 2 ngh on, the ghost
// column (over the interior rows), so no thread divides a cell index: a step of a small grid
// waits for this kernel. Halos of more layers than a grid has rows of blocks take several each.
template <typename T>
__global__ void bc_fill_kernel(T* q0, T* q1, T* q2, int nxp, int nyp, int ngh, int64_t pitch,
                               int kxm, int kxp, int kym, int kyp, const GswLoopState* st) {
    chain_begin();
    if (st != nullptr && st->done) return;
    for (int64_t edge = blockIdx.y; edge < 4LL * ngh; edge += gridDim.y) {
        const bool rows = edge < 2LL * ngh;
        const int layer = (int)(rows ? edge : edge - 2LL * ngh);
        const bool low = layer < ngh;
        const int ghost = low ? layer : (rows ? nxp : nyp) - 2 * ngh + layer;
        const int lo = rows ? 0 : ngh, hi = rows ? nyp : nxp - ngh;
        for (int along = lo + blockIdx.x * blockDim.x + threadIdx.x; along < hi; along += gridDim.x * blockDim.x) {
            const int gi = rows ? ghost : along, gj = rows ? along : ghost;
            const int kx = !rows ? GSW_BC_NONE : low ? kxm : kxp;
            const bool corner = rows && (gj < ngh || gj >= nyp - ngh);
            const int ky = rows && !corner ? GSW_BC_NONE : gj < ngh ? kym : kyp;
            if (kx == GSW_BC_NONE && ky == GSW_BC_NONE) continue;
            // value of the x pass at (row gi, column cj)
            auto xval = [&](int cj, T& a, T& u, T& v) {
                if (kx == GSW_BC_FALL) { a = (T)0; u = (T)0; v = (T)0; return; }
                const int64_t o = (int64_t)(kx == GSW_BC_NONE ? gi : bc_src(kx, gi, nxp, ngh)) * pitch + cj;
                a = q0[o]; u = q1[o]; v = q2[o];
                if (kx == GSW_BC_WALL) u = -u;
            };
            T a, u, v;
            if (ky == GSW_BC_NONE) {                   // a ghost row, or a corner left to the x pass
                xval(gj, a, u, v);
            } else if (ky == GSW_BC_FALL) {
                a = (T)0; u = (T)0; v = (T)0;
            } else {
                xval(bc_src(ky, gj, nyp, ngh), a, u, v);
                if (ky == GSW_BC_WALL) v = -v;
            }
            const int64_t go = (int64_t)gi * pitch + gj;
            q0[go] = a; q1[go] = u; q2[go] = v;
        }
    }
}

// Stage boundary (forcing.py:315-377): eta(t_new) by clamped linear interpolation.
__device__ __forceinline__ double stage_eta(const double* ts, const double* ss, int n, double t) {
    if (t <= ts[0]) return ss[0];
    if (t >= ts[n - 1]) return ss[n - 1];
    int lo = 0, hi = n;                   // bisect_left
    while (lo < hi) { const int mid = (lo + hi) >> 1; if (ts[mid] < t) lo = mid + 1; else hi = mid; }
    const int i = lo;
    const double t0 = ts[i - 1], t1 = ts[i], s0 = ss[i - 1], s1 = ss[i];
    const double w = __ddiv_rn(__dsub_rn(t, t0), __dsub_rn(t1, t0));
    return __dadd_rn(s0, __dmul_rn(w, __dsub_rn(s1, s0)));
}

// With a wave-speed target, each cell's speed (at rest) is folded into it here.
template <typename T>
__global__ void stage_kernel(GswStageArgs a) {
    chain_begin();
    if (a.state->done) return;
    unsigned long long lam = 0ull;
    const double eta = stage_eta(a.time_s, a.stage_m, a.n_knots, a.state->t_new);
    T* q0 = (T*)a.q0; T* q1 = (T*)a.q1; T* q2 = (T*)a.q2;
    for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < a.n_cells; k += gridDim.x * blockDim.x) {
        T hn;
        if (a.bed_is_f32) {
            const float d = (float)eta - (float)a.bed64[k];
            hn = (T)(d > 0.0f ? d : 0.0f);
        } else {
            const double d = eta - a.bed64[k];
            hn = (T)(d > 0.0 ? d : 0.0);
        }
        const int64_t o = a.cell_off[k];
        q0[o] = hn; q1[o] = (T)0; q2[o] = (T)0;
        if (a.lam_target != nullptr && !(a.cfl_ghost != nullptr && a.cfl_ghost[k])) {
            const unsigned long long lb = lam_dense_bits(hn, (T)0, (T)0, (T)a.g, (T)a.h_cfl);
            lam = lb > lam ? lb : lam;
        }
    }
    if (a.lam_target != nullptr) block_max_to(lam, (unsigned long long*)a.lam_target);
}

// Fold the wave speed of listed cells into the loop's target (after all stage writes).
template <typename T>
__global__ void lam_cells_kernel(const T* q0, const T* q1, const T* q2, const int64_t* off, int n,
                                 const uint8_t* excl, T g, T h_cfl, unsigned long long* target,
                                 const GswLoopState* st) {
    chain_begin();
    if (st != nullptr && st->done) return;
    unsigned long long lam = 0ull;
    for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < n; k += gridDim.x * blockDim.x) {
        if (excl != nullptr && excl[k]) continue;
        const int64_t o = off[k];
        const unsigned long long lb = lam_dense_bits(q0[o], q1[o], q2[o], g, h_cfl);
        lam = lb > lam ? lb : lam;
    }
    block_max_to(lam, target);
}

}  // namespace gsw

using namespace gsw;

// Exact, portable or fast arithmetic; fast is binary32 only.
static int check_arith(const GswDenseArgs* a) {
    if (a->arith != GSW_ARITH_EXACT && a->arith != GSW_ARITH_FAST && a->arith != GSW_ARITH_PORTABLE)
        return set_error(GSW_ERR_INVALID, "dense: bad arith %d", a->arith);
    if (a->arith == GSW_ARITH_FAST && a->dtype != GSW_F32)
        return set_error(GSW_ERR_INVALID, "dense: fast arithmetic is binary32 only");
    return GSW_OK;
}

extern "C" int gsw_dense_step(const GswDenseArgs* a, void* stream) {
    GSW_CHECK_ABI(a);
    if (int rc = check_arith(a)) return rc;
    if (a->arith == GSW_ARITH_FAST) return gsw_fast_dense_launch(a, true, (cudaStream_t)stream);
    if (a->dtype == GSW_F32) return launch_march<float, true>(a, (cudaStream_t)stream);
    if (a->dtype == GSW_F64) return launch_march<double, true>(a, (cudaStream_t)stream);
    return set_error(GSW_ERR_INVALID, "dense step: bad dtype %d", a->dtype);
}

template <typename T>
static int launch_rhs(const GswDenseArgs* a, cudaStream_t s) {
    // cells outside the computed box (and ghost rows) read as 0
    const size_t rowb = (size_t)a->nyp * sizeof(T);
    for (void* o : {a->qn0, a->qn1, a->qn2}) {
        if (!o) return set_error(GSW_ERR_INVALID, "dense rhs: null output");
        if (cudaMemset2DAsync(o, (size_t)a->pitch * sizeof(T), 0, rowb, (size_t)a->nxp, s) != cudaSuccess)
            return set_error(GSW_ERR_CUDA, "dense rhs: cudaMemset2DAsync failed");
    }
    if (a->arith == GSW_ARITH_FAST) return gsw_fast_dense_launch(a, false, s);
    return launch_march<T, false>(a, s);
}

extern "C" int gsw_dense_rhs(const GswDenseArgs* a, void* stream) {
    GSW_CHECK_ABI(a);
    if (int rc = check_arith(a)) return rc;
    if (a->dtype == GSW_F32) return launch_rhs<float>(a, (cudaStream_t)stream);
    if (a->dtype == GSW_F64) return launch_rhs<double>(a, (cudaStream_t)stream);
    return set_error(GSW_ERR_INVALID, "dense rhs: bad dtype %d", a->dtype);
}

template <typename T>
static int launch_lammax(const GswDenseArgs* a, uint64_t* out, cudaStream_t s) {
    DenseK<T> k;
    int rc = fill_dense<T>(a, k, false);
    if (rc) return rc;
    if (!out) return set_error(GSW_ERR_INVALID, "lammax: null output");
    const int nx = k.nxp - 2 * k.ngh, ny = k.nyp - 2 * k.ngh;
    int wshift = 0;
    while (wshift < 3 && (32 << wshift) < ny) ++wshift;
    const int cols = 32 << wshift, rows = 8 >> wshift;
    const unsigned gx = (unsigned)((ny + cols - 1) / cols);
    const unsigned gy = (unsigned)std::min<int64_t>((nx + 4 * rows - 1) / (4 * rows), std::max<int64_t>(1, 8LL * sm_count() / gx));
    launch_chained(dense_lammax_kernel<T>, dim3(gx, std::min(gy, 65535u)), dim3(32, 8), s, k, (unsigned long long*)out, wshift);
    return check_launch("dense_lammax");
}

extern "C" int gsw_dense_lammax(const GswDenseArgs* a, uint64_t* lam_bits, void* stream) {
    GSW_CHECK_ABI(a);
    if (a->dtype == GSW_F32) return launch_lammax<float>(a, lam_bits, (cudaStream_t)stream);
    if (a->dtype == GSW_F64) return launch_lammax<double>(a, lam_bits, (cudaStream_t)stream);
    return set_error(GSW_ERR_INVALID, "lammax: bad dtype %d", a->dtype);
}

extern "C" int gsw_bc_fill(const GswBcArgs* a, void* stream) {
    GSW_CHECK_ABI(a);
    if (a->ngh < 1 || 2 * a->ngh >= a->nxp || 2 * a->ngh >= a->nyp || a->pitch < a->nyp)
        return set_error(GSW_ERR_INVALID, "bc: bad extents");
    for (int f = 0; f < 4; ++f)
        if (a->kinds[f] < 0 || a->kinds[f] > GSW_BC_NONE) return set_error(GSW_ERR_INVALID, "bc: bad kind %d", a->kinds[f]);
    const dim3 grid((unsigned)std::min((std::max(a->nxp, a->nyp) + 255) / 256, 64), (unsigned)std::min<int64_t>(4LL * a->ngh, 65535));
    cudaStream_t s = (cudaStream_t)stream;
    if (a->dtype == GSW_F32)
        launch_chained(bc_fill_kernel<float>, grid, dim3(256), s, (float*)a->q0, (float*)a->q1, (float*)a->q2, a->nxp, a->nyp,
                                                   a->ngh, a->pitch, a->kinds[0], a->kinds[1], a->kinds[2],
                                                   a->kinds[3], a->state);
    else if (a->dtype == GSW_F64)
        launch_chained(bc_fill_kernel<double>, grid, dim3(256), s, (double*)a->q0, (double*)a->q1, (double*)a->q2, a->nxp, a->nyp,
                                                    a->ngh, a->pitch, a->kinds[0], a->kinds[1], a->kinds[2],
                                                    a->kinds[3], a->state);
    else return set_error(GSW_ERR_INVALID, "bc: bad dtype");
    return check_launch("bc_fill");
}

extern "C" int gsw_stage_apply(const GswStageArgs* a, void* stream) {
    GSW_CHECK_ABI(a);
    if (a->n_cells <= 0) return GSW_OK;
    if (!a->cell_off || !a->bed64 || !a->time_s || !a->stage_m || a->n_knots < 1 || !a->state)
        return set_error(GSW_ERR_INVALID, "stage: null table or state");
    if (a->lam_target && !(a->h_cfl > 0.0))
        return set_error(GSW_ERR_INVALID, "stage: h_cfl (%g) must be > 0 (the wave speed's divisor floor)", a->h_cfl);
    cudaStream_t s = (cudaStream_t)stream;
    const int grid = std::min(sm_count() * 4, (a->n_cells + 255) / 256);
    if (a->dtype == GSW_F32) launch_chained(stage_kernel<float>, dim3(grid), dim3(256), s, *a);
    else if (a->dtype == GSW_F64) launch_chained(stage_kernel<double>, dim3(grid), dim3(256), s, *a);
    else return set_error(GSW_ERR_INVALID, "stage: bad dtype");
    return check_launch("stage");
}

extern "C" int gsw_lam_cells(const GswStageArgs* a, void* stream) {
    GSW_CHECK_ABI(a);
    if (a->n_cells <= 0) return GSW_OK;
    if (!a->cell_off || !a->lam_target) return set_error(GSW_ERR_INVALID, "lam_cells: null list or target");
    cudaStream_t s = (cudaStream_t)stream;
    const int grid = std::min(sm_count() * 4, (a->n_cells + 255) / 256);
    if (a->dtype == GSW_F32)
        launch_chained(lam_cells_kernel<float>, dim3(grid), dim3(256), s, (const float*)a->q0, (const float*)a->q1, (const float*)a->q2,
                                                     a->cell_off, a->n_cells, a->cfl_ghost, (float)a->g,
                                                     (float)a->h_cfl, (unsigned long long*)a->lam_target, a->state);
    else if (a->dtype == GSW_F64)
        launch_chained(lam_cells_kernel<double>, dim3(grid), dim3(256), s, (const double*)a->q0, (const double*)a->q1, (const double*)a->q2,
                                                      a->cell_off, a->n_cells, a->cfl_ghost, a->g, a->h_cfl,
                                                      (unsigned long long*)a->lam_target, a->state);
    else return set_error(GSW_ERR_INVALID, "lam_cells: bad dtype");
    return check_launch("lam_cells");
}
