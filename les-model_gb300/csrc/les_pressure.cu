// les_pressure.cu -- the pressure system of les-model src/pressure.cpp on the
// device: divergence RHS, b vector, stencil assembly, the 7-point SpMV, the
// Jacobi and Chebyshev preconditioners, PCG in FP64, the power iteration for
// lambda_max, the pressure boundary conditions and the stationary Jacobi
// solver.  (IC(0) and GS-SOR, which need wavefront ordering, are in
// les_wavefront.cu; the mixed-precision solve is in les_mixed.cu.)
//
// Compiled with -fmad=false: every elementwise expression keeps the
// reference's rounding.  Dot products and norms are deterministic two-stage
// reductions (block tree, then the last block sums the block partials in
// order), so they differ from the reference's sequential sum only by
// reassociation.
#include <cmath>
#include <random>
#include <utility>
#include <vector>

#include "les_internal.cuh"

using namespace les;

namespace les {
les_status ic_records64(les_ctx* c, const double* const* L);
les_status ic_apply_dev(les_ctx* c, const double* const* L, const double* r, double* z, int skip_done);
les_status wave_check(les_ctx* c);
les_status build_ic_dev(les_ctx* c);
les_status pcg_mixed(les_ctx* c, const les_pcg_opts* o, les_pcg_result* res);
bool pcg64_coop_used(const les_ctx* c, const les_pcg_opts* o, bool pow2);   // les_coop64.cu
les_status pcg64_coop(les_ctx* c, const les_pcg_opts* o, bool pow2, int keep_tol);
}

namespace {

__device__ __forceinline__ bool cell_coords(const Geo& g, int& i, int& j, int& k)
{
    k = blockIdx.x * TBK + threadIdx.x;
    j = blockIdx.y * TBJ + threadIdx.y;
    i = blockIdx.z;
    return k < g.nz && j < g.ny;
}

// fast_apply_laplacian body, src/pressure.cpp:721-744 (bounds tests kept so
// that the summation matches term for term).  POW2: every off-diagonal
// coefficient is a power of two (or its double, or zero), so its product is
// exact and one fused multiply-add rounds as the multiply and the add do.
template <bool POW2>
__device__ __forceinline__ double apply_row(const StencilView& A, const double* __restrict__ p,
                                            const Geo& g, int i, int j, int k, int id, double pc)
{
    Coef7 a = A.at(id);
    double val = a.c * pc;
    auto add = [&](double m, double x) { val = POW2 ? fma(m, x, val) : val + m * x; };
    if (i > 0) add(a.w, p[id - g.si]);
    if (i < g.nx - 1) add(a.e, p[id + g.si]);
    if (j > 0) add(a.s, p[id - g.sj]);
    if (j < g.ny - 1) add(a.n, p[id + g.sj]);
    if (k > 0) add(a.b, p[id - 1]);
    if (k < g.nz - 1) add(a.t, p[id + 1]);
    return val;
}

// How the rows of A are formed.  GB300 runs about two FP64 operations per SM
// and clock, so the FP64 kernels are bound by the number of operations of a
// row; each form gives the reference's roundings.
//   GENERAL  seven products and six sums (13), a matrix of the caller
//   POW2     one product and six fused multiply-adds (7), a device-built
//            matrix whose 1/h^2 are powers of two
//   SHARED   a device-built matrix of any spacing (8 to 10): the product
//            x1 * p of a cell is the same number for its two i-neighbours
//            (doubled exactly at a mirror, src/pressure.cpp:663-696), so it
//            is formed once per cell and handed on -- along i in registers as
//            the block marches, along j and k in shared memory; one product
//            serves all axes whose spacings are equal
// 256x128x128, general rows of one cell per thread -> POW2 / SHARED: SpMV
// 125 -> 58 / 91 us (with p.q 64 / 99); Chebyshev(4)-PCG iteration, with step 0
// and r.z in the kernels next to them, 735 -> 495 / 639 us (a matrix of the
// caller 735 -> 706).
enum RowForm { ROW_GENERAL = 0, ROW_POW2 = 1, ROW_SHARED = 2 };

struct RowTile {
    double v[2][2][TBJ + 2][TBK + 2];   // [plane parity][y, z products]
};

// multiplier 0, 1 or 2 of a base coefficient (its bit pattern: integer operations)
__device__ __forceinline__ double mult(unsigned pack, unsigned state)
{
    const unsigned m = (pack >> (2 * state)) & 3u;
    return __hiloint2double(m ? (int)(0x3fe00000u + (m << 20)) : 0, 0);
}

// Calls f(i, id, x_c, (A x)_c) for the cells of this thread's column on the
// planes [blockIdx.z * ci, + ci).  Every thread of the block must call it.
template <int FORM, class F>
__device__ __forceinline__ void march_rows(const StencilView& A, const double* __restrict__ x, const Geo& g, int ci,
                                           F f)
{
    const int k = blockIdx.x * TBK + threadIdx.x, j = blockIdx.y * TBJ + threadIdx.y;
    const int i0 = blockIdx.z * ci, i1 = min(g.nx, i0 + ci);
    const bool in = k < g.nz && j < g.ny;
    if (FORM != ROW_SHARED) {
        if (in)
            for (int i = i0; i < i1; ++i) {
                const int id = i * g.si + j * g.sj + k;
                const double xc = x[id];
                f(i, id, xc, apply_row<FORM == ROW_POW2>(A, x, g, i, j, k, id, xc));
            }
        return;
    }
    __shared__ RowTile tile;
    const StencilCoef& c = A.k;
    // (compared as bit patterns: a comparison of doubles takes the FP64 pipe)
    const bool same_y = __double_as_longlong(c.y1) == __double_as_longlong(c.x1);
    const bool same_z = __double_as_longlong(c.z1) == __double_as_longlong(c.y1);
    const int tj = threadIdx.y + 1, tk = threadIdx.x + 1;
    // The products around the tile: the row before it by warp 0, the row after it by
    // warp 1, the columns on either side by a half of warp 2 -- one FP64
    // instruction of a warp for up to 32 of them (by each row's own edge lanes:
    // two in every warp).
    const int j0 = blockIdx.y * TBJ, k0 = blockIdx.x * TBK;
    int hj = j, hk = k;
    bool halo = false;
    if (threadIdx.y == 0) {
        hj = j0 - 1;
        halo = hj >= 0 && k < g.nz;
    } else if (threadIdx.y == 1) {
        hj = j0 + TBJ;
        halo = hj < g.ny && k < g.nz;
    } else if (threadIdx.y == 2 && threadIdx.x < 2 * TBJ) {
        hj = j0 + (threadIdx.x & (TBJ - 1));
        hk = threadIdx.x < TBJ ? k0 - 1 : k0 + TBK;
        halo = hj < g.ny && hk >= 0 && hk < g.nz;
    }
    const bool halo_z = threadIdx.y == 2;
    const double halo_coef = halo_z ? c.z1 : c.y1;
    const int halo_off = hj * g.sj + hk, hr = hj - j0 + 1, hc = hk - k0 + 1;
    int id = i0 * g.si + j * g.sj + k;
    double xc = in ? x[id] : 0.0;
    double pw = in && i0 > 0 ? c.x1 * x[id - g.si] : 0.0, pc = c.x1 * xc;
    for (int i = i0; i < i1; ++i, id += g.si) {
        auto& ty = tile.v[i & 1][0];
        auto& tz = tile.v[i & 1][same_z ? 0 : 1];
        ty[tj][tk] = same_y ? pc : c.y1 * xc;
        if (!same_z) tz[tj][tk] = c.z1 * xc;
        if (halo) (halo_z ? tz : ty)[hr][hc] = halo_coef * x[i * g.si + halo_off];
        const double xe = in && i < g.nx - 1 ? x[id + g.si] : 0.0;
        const double pe = c.x1 * xe;
        __syncthreads();   // one barrier per plane: the planes alternate between two tiles
        if (in) {
            // code 0: an identity row, every multiplier 0 (and 0 times an infinity NaN)
            const unsigned code = A.code[id];
            const unsigned cd = code ? code - 1u : 3u, xs = cd % 5u, r = cd / 5u, ys = r & 3u, zs = r >> 2;
            const unsigned lo = code ? YL_PACK : 0u, hi = code ? YH_PACK : 0u;
            double val = (code ? c.c0 : 1.0) * xc;
            if (i > 0) val = fma(mult(XW_PACK, xs), pw, val);
            if (i < g.nx - 1) val = fma(mult(XE_PACK, xs), pe, val);
            if (j > 0) val = fma(mult(lo, ys), ty[tj - 1][tk], val);
            if (j < g.ny - 1) val = fma(mult(hi, ys), ty[tj + 1][tk], val);
            if (k > 0) val = fma(mult(lo, zs), tz[tj][tk - 1], val);
            if (k < g.nz - 1) val = fma(mult(hi, zs), tz[tj][tk + 1], val);
            f(i, id, xc, val);
        }
        xc = xe;
        pw = pc;
        pc = pe;
    }
}

// calculate_divergence (src/pressure.cpp:256-329) + build_b_vector
// (:566-599) in one pass, with ||b||^2 reduced on the side.
__global__ void k_div_b(Geo g, double scale, double idx, double idy, double idz, double idx1,
                        double idy1, double idz1, const double* __restrict__ un,
                        const double* __restrict__ vn, const double* __restrict__ wn,
                        const uint8_t* __restrict__ solid, double* __restrict__ rhs,
                        double* __restrict__ b, double* partials, unsigned* counter, SolverState* st,
                        double rel_tol, const double* dtp, double rho)
{
    __shared__ double sm[32];
    int i, j, k;
    double bb[1] = {0.0};
    if (dtp) scale = rho / *dtp;   // src/pressure.cpp:260, from the device dt
    if (cell_coords(g, i, j, k)) {
        const int id = i * g.si + j * g.sj + k;
        double r = 0.0;
        if (!(solid[id] || i == g.nx - 1)) {
            double du_dx, dv_dy, dw_dz;
            if (i == 0) du_dx = (un[id + g.si] - un[id]) * idx1;
            else du_dx = (un[id + g.si] - un[id - g.si]) * idx;
            if (j == 0) dv_dy = (vn[id + g.sj] - vn[id]) * idy1;
            else if (j == g.ny - 1) dv_dy = (vn[id] - vn[id - g.sj]) * idy1;
            else dv_dy = (vn[id + g.sj] - vn[id - g.sj]) * idy;
            if (k == 0) dw_dz = (wn[id + 1] - wn[id]) * idz1;
            else if (k == g.nz - 1) dw_dz = (wn[id] - wn[id - 1]) * idz1;
            else dw_dz = (wn[id + 1] - wn[id - 1]) * idz;
            r = scale * (du_dx + dv_dy + dw_dz);
            rhs[id] = r;
            double bv = -r;
            if (b) b[id] = bv;
            bb[0] = bv * bv;
        } else {
            rhs[id] = 0.0;
            if (b) b[id] = 0.0;
        }
    }
    if (!b) return;
    if (last_block_sum<1>(bb, partials, counter, sm)) {
        if (threadIdx.x == 0 && threadIdx.y == 0) {
            st->bnorm = sqrt(bb[0]);
            if (rel_tol > 0) st->tol = rel_tol * st->bnorm;
        }
    }
}

__global__ void k_build_b(Geo g, const double* __restrict__ rhs, const uint8_t* __restrict__ solid,
                          double* __restrict__ b)
{
    int i, j, k;
    if (!cell_coords(g, i, j, k)) return;
    const int id = i * g.si + j * g.sj + k;
    b[id] = (solid[id] || i == g.nx - 1) ? 0.0 : -rhs[id];
}

// build_stencil (src/pressure.cpp:608-699) as one code byte per cell.
__global__ void k_build_code(Geo g, const uint8_t* __restrict__ solid, uint8_t* __restrict__ code,
                             unsigned* any_solid)
{
    int i, j, k;
    if (!cell_coords(g, i, j, k)) return;
    const int id = i * g.si + j * g.sj + k;
    if (solid[id]) *any_solid = 1u;   // every writer stores the same value
    if (solid[id] || i == g.nx - 1) { code[id] = 0; return; }
    bool W = (i == 0) || solid[id - g.si];
    bool E1 = (i == g.nx - 2);
    bool E2 = !E1 && solid[id + g.si];
    unsigned xs;
    if (E1) xs = W ? 3u : 2u;
    else if (E2) xs = W ? 2u : 4u;
    else xs = W ? 1u : 0u;
    bool S = (j == 0) || solid[id - g.sj];
    bool N = (j == g.ny - 1) || solid[id + g.sj];
    unsigned ys = S ? (N ? 3u : 1u) : (N ? 2u : 0u);
    bool B = (k == 0) || solid[id - 1];
    bool T = (k == g.nz - 1) || solid[id + 1];
    unsigned zs = B ? (T ? 3u : 1u) : (T ? 2u : 0u);
    code[id] = (uint8_t)(1u + xs + 5u * (ys + 4u * zs));
}

__global__ void k_expand_stencil(Geo g, StencilView A, double* c, double* n, double* s, double* e,
                                 double* w, double* t, double* b)
{
    int i, j, k;
    if (!cell_coords(g, i, j, k)) return;
    const int id = i * g.si + j * g.sj + k;
    Coef7 a = A.at(id);
    c[id] = a.c; n[id] = a.n; s[id] = a.s; e[id] = a.e; w[id] = a.w; t[id] = a.t; b[id] = a.b;
}

// out = A in (+ optional dot in.out reduced into the state).
enum { DOT_NONE = 0, DOT_ALPHA = 1, DOT_SCAL0 = 2 };

template <int FORM, bool DOT>
__global__ void k_spmv(Geo g, StencilView A, int ci, const double* __restrict__ p, double* __restrict__ q,
                       double* partials, unsigned* counter, SolverState* st, int dot_mode)
{
    __shared__ double sm[32];
    if (dot_mode == DOT_ALPHA && st->done) return;
    double pq[1] = {0.0};
    march_rows<FORM>(A, p, g, ci, [&](int, int id, double pc, double val) {
        q[id] = val;
        if (DOT) pq[0] = fma(pc, val, pq[0]);
    });
    if (DOT && last_block_sum<1>(pq, partials, counter, sm)) {
        if (threadIdx.x == 0 && threadIdx.y == 0) {
            if (dot_mode == DOT_ALPHA) {
                st->pq = pq[0];
                st->alpha = st->rho / pq[0];   // src/pressure.cpp:378
            } else {
                st->scal[0] = pq[0];
            }
        }
    }
}

// r = b - q, ||r|| and the already-converged test of src/pressure.cpp:355-359.
__global__ void k_resid(Geo g, const double* __restrict__ b, const double* __restrict__ q,
                        double* __restrict__ r, double* partials, unsigned* counter, SolverState* st)
{
    __shared__ double sm[32];
    int i, j, k;
    double rr[1] = {0.0};
    if (cell_coords(g, i, j, k)) {
        const int id = i * g.si + j * g.sj + k;
        double v = b[id] - q[id];   // 1.0*b + (-1.0)*q
        r[id] = v;
        rr[0] = v * v;
    }
    if (last_block_sum<1>(rr, partials, counter, sm)) {
        if (threadIdx.x == 0 && threadIdx.y == 0) {
            double e = sqrt(rr[0]);
            st->rr = rr[0];
            st->err = e;
            st->k = 0;
            if (e < st->tol) { st->done = 1; st->iters = 0; st->status = LES_OK; }
            else if (!isfinite(e)) { st->done = 1; st->iters = st->max_iter; st->status = LES_NONFINITE; }
        }
    }
}

// x += alpha p; r -= alpha q; ||r||; convergence test; k += 1
// (src/pressure.cpp:381-392).  With the Jacobi preconditioner fused
// (z = r / A_c, :420-428) it also forms r.z and the next beta.
// z0 != nullptr: also the Chebyshev preconditioner's step 0, z0 = alpha0 r.
__global__ void k_update(Geo g, StencilView A, double* __restrict__ x, double* __restrict__ r,
                         const double* __restrict__ p, const double* __restrict__ q,
                         double* __restrict__ z, double* partials, unsigned* counter,
                         SolverState* st, int jacobi, DivBy by_c0, double alpha0, double* __restrict__ z0)
{
    __shared__ double sm[64];
    if (st->done) return;
    const double alpha = st->alpha;
    int i, j, k;
    double acc[2] = {0.0, 0.0};
    if (cell_coords(g, i, j, k))
        for (; i < g.nx; i += gridDim.z) {   // planes blockIdx.z, + gridDim.z, ...
            const int id = i * g.si + j * g.sj + k;
            x[id] += alpha * p[id];
            double rv = r[id] + (-alpha) * q[id];
            r[id] = rv;
            acc[0] = fma(rv, rv, acc[0]);
            if (jacobi) {
                const double zv = A.code ? (A.code[id] ? div_by(rv, by_c0) : rv) : rv / A.d[0][id];
                z[id] = zv;
                acc[1] = fma(rv, zv, acc[1]);
            }
            if (z0) z0[id] = fma(alpha0, rv, 0.0);
        }
    if (last_block_sum<2>(acc, partials, counter, sm)) {
        if (threadIdx.x == 0 && threadIdx.y == 0) {
            double e = sqrt(acc[0]);
            int kk = st->k + 1;
            st->k = kk;
            st->rr = acc[0];
            st->err = e;
            if (e < st->tol) { st->done = 1; st->iters = kk; st->status = LES_OK; }
            else if (!isfinite(e)) { st->done = 1; st->iters = st->max_iter; st->status = LES_NONFINITE; }
            else if (kk >= st->max_iter) { st->done = 1; st->iters = st->max_iter; st->status = LES_NOT_CONVERGED; }
            if (jacobi) {
                st->rz = acc[1];
                st->beta = acc[1] / st->rho;   // :399-402
                st->rho = acc[1];
            }
        }
    }
}

enum { RD_RHO = 0, RD_BETA = 1, RD_SCAL0 = 2, RD_NONE = 3 };

// What a kernel that ends with r.z does with the sum: RD_RHO sets rho (:369),
// RD_BETA forms beta = rz/rho and rho = rz (:399-408), RD_SCAL0 stores it.
__device__ __forceinline__ void dot_done(SolverState* st, int mode, double s)
{
    if (mode == RD_RHO) st->rho = s;
    else if (mode == RD_BETA) { st->rz = s; st->beta = s / st->rho; st->rho = s; }
    else st->scal[0] = s;
}

// dot(a, b) reduced into the state.  Bound by the FP64 pipe of the block sums, so
// its blocks are few and loop over planes (reduce_grid): 256x128x128, a block
// per plane and tile 87 us a call, capped 32.
__global__ void k_dot(Geo g, const double* __restrict__ a, const double* __restrict__ b,
                      double* partials, unsigned* counter, SolverState* st, int mode, int skip_done)
{
    __shared__ double sm[32];
    if (skip_done && st->done) return;
    int i, j, k;
    double s[1] = {0.0};
    if (cell_coords(g, i, j, k))
        for (; i < g.nx; i += gridDim.z) {   // planes blockIdx.z, + gridDim.z, ...
            const int id = i * g.si + j * g.sj + k;
            s[0] = fma(a[id], b[id], s[0]);
        }
    if (last_block_sum<1>(s, partials, counter, sm)) {
        if (threadIdx.x == 0 && threadIdx.y == 0) dot_done(st, mode, s[0]);
    }
}

// p = 1.0*z + beta*p (src/pressure.cpp:405).
// out = a*in1 + b*in2 (parallel_saxpy, src/pressure.cpp:995-1002; with
// a = 1, in1 = out it is parallel_axpy, :983-989).  out may alias either input.
__global__ void k_axpby(Geo g, double a, const double* in1, double b, const double* in2, double* out)
{
    int i, j, k;
    if (!cell_coords(g, i, j, k)) return;
    const int id = i * g.si + j * g.sj + k;
    out[id] = a * in1[id] + b * in2[id];
}

__global__ void k_pupdate(Geo g, const double* __restrict__ z, double* __restrict__ p, SolverState* st)
{
    if (st->done) return;
    const double beta = st->beta;
    int i, j, k;
    if (!cell_coords(g, i, j, k)) return;
    const int id = i * g.si + j * g.sj + k;
    p[id] = z[id] + beta * p[id];
}

__global__ void k_jacobi_pc(Geo g, StencilView A, const double* __restrict__ r, double* __restrict__ z,
                            SolverState* st, int skip_done, DivBy by_c0)
{
    if (skip_done && st->done) return;
    int i, j, k;
    if (!cell_coords(g, i, j, k)) return;
    const int id = i * g.si + j * g.sj + k;
    z[id] = A.code ? (A.code[id] ? div_by(r[id], by_c0) : r[id]) : r[id] / A.d[0][id];
}

// Chebyshev preconditioner, src/pressure.cpp:851-906.  Step 0:
// z = 0.0 + alpha0 * r (p_0 = res_0 = r is implicit).
__global__ void k_cheb0(Geo g, double alpha0, const double* __restrict__ r, double* __restrict__ z,
                        SolverState* st, int skip_done)
{
    if (skip_done && st->done) return;
    int i, j, k;
    if (!cell_coords(g, i, j, k)) return;
    const int id = i * g.si + j * g.sj + k;
    z[id] = fma(alpha0, r[id], 0.0);
}

// One inner step: res = r - A z; p = res + beta p; z' = z + alpha p.
// pin == nullptr means p_{k-1} = r (first step).  dot_mode != RD_NONE: also
// r.z' (the last step).
//
// Bound by the FP64 pipe: 7 to 10 operations for the row, 5 for the recurrence
// and one for r.z per cell (18 with every product rounded by itself; formed in
// every step, r.z cost 5 % of a Chebyshev(4)-PCG iteration).
template <int FORM, bool DOT>
__global__ void k_cheb_step(Geo g, StencilView A, int ci, double alpha, double beta,
                            const double* __restrict__ r, const double* __restrict__ zin,
                            const double* pin, double* pout, double* __restrict__ zout,
                            SolverState* st, int skip_done, double* partials, unsigned* counter, int dot_mode)
{
    __shared__ double sm[32];
    if (skip_done && st->done) return;
    double rz[1] = {0.0};
    march_rows<FORM>(A, zin, g, ci, [&](int, int id, double zc, double az) {
        const double rv = r[id];
        const double res = rv - az;
        const double pv = res + beta * (pin ? pin[id] : rv);
        if (pout) pout[id] = pv;
        const double zv = zc + alpha * pv;
        zout[id] = zv;
        if (DOT) rz[0] = fma(rv, zv, rz[0]);
    });
    if (DOT && last_block_sum<1>(rz, partials, counter, sm))
        if (threadIdx.x == 0 && threadIdx.y == 0) dot_done(st, dot_mode, rz[0]);
}

// apply_pressure_BCs, src/pressure.cpp:14-93, face part.  The ordered face
// loops leave every face cell equal to g(i, J(j), K(k)) where J, K clamp to
// [1, n-2] and g(i, j', k') = P(1, j', k') for i == 0, 0 for i == nx-1,
// P(i, j', k') otherwise (P: the values before the call).  `in` may equal
// `out` (faces read interior cells only).
// (One-dimensional blocks: GS-SOR ends here on grids of any number of planes.)
__global__ void k_pbc_faces(Geo g, const double* in, double* out)
{
    const int id = blockIdx.x * blockDim.x + threadIdx.x;
    if (id >= g.n) return;
    const int i = id / g.si, r = id - i * g.si, j = r / g.sj, k = r - j * g.sj;
    bool jk_in = j >= 1 && j <= g.ny - 2 && k >= 1 && k <= g.nz - 2;
    if (jk_in && i > 0 && i < g.nx - 1) return;
    if (i == g.nx - 1) { out[id] = 0.0; return; }
    int jj = j < 1 ? 1 : (j > g.ny - 2 ? g.ny - 2 : j);
    int kk = k < 1 ? 1 : (k > g.nz - 2 ? g.nz - 2 : k);
    int ii = i == 0 ? 1 : i;
    out[id] = in[ii * g.si + jj * g.sj + kk];
}

// Obstacle part (:73-92): first fluid neighbour in the order +i,-i,+j,-j,+k,-k.
__global__ void k_pbc_obstacle(Geo g, const int* __restrict__ list, int n, const uint8_t* __restrict__ solid,
                               double* __restrict__ p)
{
    int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= n) return;
    const int id = list[t];
    if (!solid[id + g.si]) p[id] = p[id + g.si];
    else if (!solid[id - g.si]) p[id] = p[id - g.si];
    else if (!solid[id + g.sj]) p[id] = p[id + g.sj];
    else if (!solid[id - g.sj]) p[id] = p[id - g.sj];
    else if (!solid[id + 1]) p[id] = p[id + 1];
    else if (!solid[id - 1]) p[id] = p[id - 1];
}

// Interior RHS of the stationary solvers, src/pressure.cpp:119-132 / :197-210.
__global__ void k_stat_rhs(Geo g, double coef, DivBy two_dx, DivBy two_dy, DivBy two_dz,
                           const double* __restrict__ u, const double* __restrict__ v,
                           const double* __restrict__ w, double* __restrict__ rhs)
{
    int i, j, k;
    if (!cell_coords(g, i, j, k)) return;
    const int id = i * g.si + j * g.sj + k;
    if (i < 1 || i > g.nx - 2 || j < 1 || j > g.ny - 2 || k < 1 || k > g.nz - 2) { rhs[id] = 0.0; return; }
    double div = div_by(u[id + g.si] - u[id - g.si], two_dx) + div_by(v[id + g.sj] - v[id - g.sj], two_dy) +
                 div_by(w[id + 1] - w[id - 1], two_dz);
    rhs[id] = coef * div;
}

// One Jacobi sweep, src/pressure.cpp:139-157, the faces of apply_pressure_BCs
// (:14-72: every face cell takes the new value of the interior cell it clamps
// to, the outlet 0, so that cell's thread stores it) and max|dp| (its bit
// pattern: the order of non-negative doubles is that of their patterns, and
// NaN is not selected).  The test of the sweep before, max|dp| < tol
// (:164-170), is made by every block here: three slots of maxdp rotate, one
// read, one formed, one cleared for the next sweep.
//
// Bound by the FP64 pipe: 10 operations per cell when the three 1/h^2 are the
// same power of two, 11 for three powers of two, 19 with divisions by a
// constant (45 with divisions as such).  Per sweep, 256x128x128: 550 -> 100 us
// (78 at the FP64 rate); 200x100x100, h = 1/100: 268 -> 116 us (75).
constexpr int JAC_PLANES = 4;   // planes per thread: one maximum for the block's four tiles
enum JacForm { JAC_DIV = 0, JAC_POW2 = 1, JAC_EQUAL = 2 };

template <int FORM>
__global__ void k_jacobi_sweep(Geo g, DivBy dx2, DivBy dy2, DivBy dz2, DivBy denom, const double* __restrict__ cur,
                               double* __restrict__ nxt, const double* __restrict__ rhs, unsigned long long* maxdp,
                               SolverState* st, int sweep, int cur_buf)
{
    __shared__ unsigned long long sm[TBJ];
    const bool first = blockIdx.x == 0 && blockIdx.y == 0 && blockIdx.z == 0 && threadIdx.x == 0 && threadIdx.y == 0;
    if (st->done) return;
    if (sweep > 0 && __longlong_as_double((long long)maxdp[(sweep + 2) % 3]) < st->tol) {
        if (first) {   // the sweep before met the tolerance
            st->iters = st->k = sweep;
            st->buf = cur_buf;
            st->status = LES_OK;
            st->done = 1;
        }
        return;
    }
    if (first) maxdp[(sweep + 1) % 3] = 0ull;
    const int k = blockIdx.x * TBK + threadIdx.x, j = blockIdx.y * TBJ + threadIdx.y;
    unsigned long long m = 0ull;
    if (j >= 1 && j <= g.ny - 2 && k >= 1 && k <= g.nz - 2) {
        const int i0 = max(1, (int)blockIdx.z * JAC_PLANES), i1 = min(g.nx - 1, ((int)blockIdx.z + 1) * JAC_PLANES);
        const bool edge = j == 1 || j == g.ny - 2 || k == 1 || k == g.nz - 2;
        int id = i0 * g.si + j * g.sj + k;
        double pw = i0 < i1 ? cur[id - g.si] : 0.0, pc = i0 < i1 ? cur[id] : 0.0;
        for (int i = i0; i < i1; ++i, id += g.si) {
            const double pe = cur[id + g.si];
            const double ew = pe + pw, ns = cur[id + g.sj] + cur[id - g.sj], tb = cur[id + 1] + cur[id - 1];
            double x;
            if (FORM == JAC_EQUAL) x = fma((ew + ns) + tb, dx2.y, -rhs[id]);
            else if (FORM == JAC_POW2) x = fma(tb, dz2.y, fma(ns, dy2.y, ew * dx2.y)) - rhs[id];
            else x = ((div_by(ew, dx2) + div_by(ns, dy2)) + div_by(tb, dz2)) - rhs[id];
            const double v = div_by(x, denom);
            nxt[id] = v;
            if (edge || i == 1 || i == g.nx - 2) {
                const int js[3] = {j, j == 1 ? 0 : -1, j == g.ny - 2 ? g.ny - 1 : -1};
                const int ks[3] = {k, k == 1 ? 0 : -1, k == g.nz - 2 ? g.nz - 1 : -1};
                for (int a = 0; a < 3; ++a)
                    for (int b = 0; b < 3; ++b) {
                        if (js[a] < 0 || ks[b] < 0) continue;
                        const int c = js[a] * g.sj + ks[b];
                        if (a || b) nxt[i * g.si + c] = v;
                        if (i == 1) nxt[c] = v;
                        if (i == g.nx - 2) nxt[(g.nx - 1) * g.si + c] = 0.0;
                    }
            }
            const unsigned long long r = (unsigned long long)__double_as_longlong(fabs(v - pc));
            if (r > m && r <= 0x7ff0000000000000ull) m = r;
            pw = pc;
            pc = pe;
        }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        const unsigned long long t = __shfl_xor_sync(0xffffffffu, m, o);
        m = t > m ? t : m;
    }
    if (threadIdx.x == 0) sm[threadIdx.y] = m;
    __syncthreads();
    if (threadIdx.x == 0 && threadIdx.y == 0) {
        for (int q = 1; q < TBJ; ++q) m = sm[q] > m ? sm[q] : m;
        if (m) atomicMax(maxdp + sweep % 3, m);
    }
}

// The test of the last sweep launched so far.
__global__ void k_jacobi_test(SolverState* st, const unsigned long long* maxdp, int sweeps, int buf)
{
    if (st->done) return;
    st->k = sweeps;
    st->buf = buf;
    if (__longlong_as_double((long long)maxdp[(sweeps + 2) % 3]) < st->tol) {
        st->iters = sweeps;
        st->status = LES_OK;
        st->done = 1;
    } else if (sweeps >= st->max_iter) {
        st->iters = sweeps;
        st->status = LES_NOT_CONVERGED;
        st->done = 1;
    }
}

__global__ void k_pbc_obstacle_guarded(Geo g, const int* __restrict__ list, int n,
                                       const uint8_t* __restrict__ solid, double* __restrict__ p,
                                       SolverState* st)
{
    if (st->done) return;
    int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= n) return;
    const int id = list[t];
    if (!solid[id + g.si]) p[id] = p[id + g.si];
    else if (!solid[id - g.si]) p[id] = p[id - g.si];
    else if (!solid[id + g.sj]) p[id] = p[id + g.sj];
    else if (!solid[id - g.sj]) p[id] = p[id - g.sj];
    else if (!solid[id + 1]) p[id] = p[id + 1];
    else if (!solid[id - 1]) p[id] = p[id - 1];
}

__global__ void k_scale_inv(Geo g, double* __restrict__ v, const double* __restrict__ w, SolverState* st)
{
    int i, j, k;
    if (!cell_coords(g, i, j, k)) return;
    const int id = i * g.si + j * g.sj + k;
    v[id] = w[id] / st->scal[1];
}

__global__ void k_norm_of(SolverState* st)
{
    st->scal[1] = sqrt(st->scal[0]);
}

__global__ void k_init_state(SolverState* st, double tol, int max_iter, int keep_tol)
{
    if (!keep_tol) st->tol = tol;
    st->max_iter = max_iter;
    st->k = 0;
    st->done = 0;
    st->iters = 0;
    st->status = LES_OK;
    st->buf = 0;
    st->err = 0.0;
}

}  // namespace

namespace les {

// Grid of the FP64 solver's reductions in its iterations: every (k, j) tile
// once and the i-planes shared out so that about eight blocks per SM run,
// each summing its planes before the grid sum -- one partial, fence and
// atomic per block instead of one per block and plane (16384 at
// 256x128x128).  The kernels loop over planes i = blockIdx.z + t gridDim.z,
// the row marches over chunks of consecutive planes.
static dim3 reduce_grid(const les_ctx* c)
{
    dim3 gr = cell_grid(c->g);
    const long long tiles = (long long)gr.x * gr.y;
    const long long z = (8LL * c->sms + tiles - 1) / tiles;
    gr.z = (unsigned)(z < 1 ? 1 : (z > c->g.nx ? c->g.nx : z));
    return gr;
}

// A row march's chunks: the reductions' split
struct MarchGrid {
    dim3 grid;
    int ci;
};

static MarchGrid march_grid(const les_ctx* c)
{
    MarchGrid m{reduce_grid(c), 0};
    m.ci = (c->g.nx + (int)m.grid.z - 1) / (int)m.grid.z;
    m.grid.z = (unsigned)((c->g.nx + m.ci - 1) / m.ci);
    return m;
}

static int row_form(const les_ctx* c)
{
    if (c->stencil_mode != 1) return ROW_GENERAL;
    auto pow2 = [](double v) { int e; return std::fabs(std::frexp(v, &e)) == 0.5; };
    return pow2(c->coef.x1) && pow2(c->coef.y1) && pow2(c->coef.z1) ? ROW_POW2 : ROW_SHARED;
}

// Rows without a sum behind them: where they share nothing along i a plane per
// block (general rows of 200x200x200, a Chebyshev(4) apply: 972 us; marched 1138)
static MarchGrid plain_grid(const les_ctx* c, int form)
{
    return form == ROW_GENERAL && c->g.nx <= 65535 ? MarchGrid{cell_grid(c->g), 1} : march_grid(c);
}

static void launch_spmv(les_ctx* c, int pid, const double* in, double* out, int dot_mode)
{
    const int f = row_form(c);
    const bool dot = dot_mode != DOT_NONE;
    const MarchGrid m = dot ? march_grid(c) : plain_grid(c, f);
    auto k = f == ROW_POW2 ? (dot ? k_spmv<ROW_POW2, true> : k_spmv<ROW_POW2, false>)
                           : (f == ROW_SHARED ? (dot ? k_spmv<ROW_SHARED, true> : k_spmv<ROW_SHARED, false>)
                                              : (dot ? k_spmv<ROW_GENERAL, true> : k_spmv<ROW_GENERAL, false>));
    if (pid >= 0) launch_p(c, pid, k, m.grid, cell_block(), c->g, stencil_view(c), m.ci, in, out, c->partials,
                           c->counters + 1, c->state, dot_mode);
    else launch(c, k, m.grid, cell_block(), c->g, stencil_view(c), m.ci, in, out, c->partials, c->counters + 1,
                c->state, dot_mode);
}

les_status spmv_dev(les_ctx* c, const double* in, double* out)
{
    if (!c->stencil_mode) return fail(c, LES_BAD_ARG, "no matrix: call les_build_stencil or les_set_stencil");
    launch_spmv(c, -1, in, out, DOT_NONE);
    return check_launch(c, "spmv");
}

les_status dot_dev(les_ctx* c, const double* a, const double* b, double* out_host)
{
    launch(c, k_dot, reduce_grid(c), cell_block(), c->g, a, b, c->partials, c->counters + 2, c->state, RD_SCAL0, 0);
    les_status st = check_launch(c, "dot");
    if (st) return st;
    st = read_state(c);
    if (st) return st;
    if (out_host) *out_host = c->h_state->scal[0];
    return LES_OK;
}

les_status div_b_dev(les_ctx* c, double dt, double rho, double rel_tol, const double* dtp)
{
    const les_mesh& m = c->mesh;
    launch(c, k_div_b, cell_grid(c->g), cell_block(),
        c->g, rho / dt, 1.0 / (2.0 * m.dx), 1.0 / (2.0 * m.dy), 1.0 / (2.0 * m.dz), 1.0 / m.dx,
        1.0 / m.dy, 1.0 / m.dz, c->slot[LES_U_NEW], c->slot[LES_V_NEW], c->slot[LES_W_NEW], c->mask,
        c->slot[LES_P_RHS], c->slot[LES_B], c->partials, c->counters + 3, c->state, rel_tol, dtp, rho);
    return check_launch(c, "divergence+b");
}

les_status pressure_bcs_dev(les_ctx* c, double* p)
{
    launch(c, k_pbc_faces, (c->g.n + 255) / 256, 256, c->g, p, p);
    if (c->n_solid)
        launch(c, k_pbc_obstacle, (c->n_solid + 255) / 256, 256, c->g, c->solid_list, c->n_solid,
                                                                          c->mask, p);
    return check_launch(c, "pressure bcs");
}

// the two buffers of a Chebyshev apply: step 0 lands so that the last step
// writes `z`
static double* cheb_z0(les_ctx* c, const les_pcg_opts* o, double* z) { return (o->degree - 1) % 2 == 0 ? z : c->w[6]; }

static double cheb_alpha0(const les_pcg_opts* o) { return 2.0 / ((o->lambda_max + o->lambda_min) / 2.0); }

// Preconditioner application r -> z for PCG; kernels are skipped once the
// state says done (skip_done).  dot_mode != RD_NONE: r.z too.  z0_done: the
// update kernel has written Chebyshev's step 0.
static les_status precond_dot(les_ctx* c, const les_pcg_opts* o, const double* r, double* z, int skip_done,
                              int dot_mode, bool z0_done)
{
    const Geo& g = c->g;
    StencilView A = stencil_view(c);
    les_status st = LES_OK;
    switch (o->precond) {
    case LES_PC_JACOBI:
        launch(c, k_jacobi_pc, cell_grid(g), cell_block(), g, A, r, z, c->state, skip_done, div_by_const(c->coef.c0));
        st = check_launch(c, "jacobi pc");
        break;
    case LES_PC_CHEBYSHEV: {
        if (o->degree < 1) return fail(c, LES_BAD_ARG, "Chebyshev degree must be >= 1");
        if ((st = ensure_work(c))) return st;
        const double d = (o->lambda_max + o->lambda_min) / 2.0;
        const double cc = (o->lambda_max - o->lambda_min) / 2.0;
        double alpha = cheb_alpha0(o);
        const int steps = o->degree - 1;
        double* zb[2] = {z, c->w[6]};
        int cur = (steps % 2 == 0) ? 0 : 1;
        if (!z0_done)
            launch(c, k_cheb0, cell_grid(g), cell_block(), g, alpha, r, zb[cur], c->state, skip_done);
        double* pbuf = c->w[7];
        const int f = row_form(c);
        const MarchGrid md = march_grid(c);
        const MarchGrid mc = plain_grid(c, f);
        auto kc = f == ROW_POW2 ? k_cheb_step<ROW_POW2, false>
                                : (f == ROW_SHARED ? k_cheb_step<ROW_SHARED, false> : k_cheb_step<ROW_GENERAL, false>);
        auto kd = f == ROW_POW2 ? k_cheb_step<ROW_POW2, true>
                                : (f == ROW_SHARED ? k_cheb_step<ROW_SHARED, true> : k_cheb_step<ROW_GENERAL, true>);
        for (int kq = 1; kq <= steps; ++kq) {
            double beta = (cc * alpha / 2.0) * (cc * alpha / 2.0);
            alpha = 1.0 / (d - beta);
            const bool last = kq == steps, dot = last && dot_mode != RD_NONE;
            const MarchGrid& m = dot ? md : mc;
            launch_p(c, PROF_CHEB64, dot ? kd : kc, m.grid, cell_block(), g, A, m.ci, alpha, beta, r,
                     (const double*)zb[cur], (const double*)(kq == 1 ? nullptr : pbuf), last ? nullptr : pbuf,
                     zb[cur ^ 1], c->state, skip_done, c->partials, c->counters + 2, dot_mode);
            cur ^= 1;
        }
        if (steps > 0) return check_launch(c, "chebyshev pc");   // the last step formed r.z
        st = check_launch(c, "chebyshev pc");
        break;
    }
    case LES_PC_IC:
    case LES_PC_IC_A:
        // with the records of ic_ready
        st = ic_apply_dev(c, (const double* const*)(o->precond == LES_PC_IC ? c->L : c->A), r, z, skip_done);
        break;
    default:
        return fail(c, LES_BAD_ARG, "unknown preconditioner");
    }
    if (!st && dot_mode != RD_NONE) {
        launch(c, k_dot, reduce_grid(c), cell_block(), g, r, (const double*)z, c->partials, c->counters + 2, c->state,
               dot_mode, skip_done);
        st = check_launch(c, "r.z");
    }
    return st;
}

// The IC-with-A mode needs A as arrays; expand the coded matrix on demand.
les_status ensure_stored_A(les_ctx* c)
{
    if (c->A_valid) return LES_OK;
    if (c->stencil_mode != 1) return fail(c, LES_BAD_ARG, "no matrix");
    const size_t nb = sizeof(double) * (size_t)c->g.n;
    for (int q = 0; q < 7; ++q)
        if (!c->A[q]) {
            les_status st = check_cuda(c, dev_malloc(c, &c->A[q], nb), "cudaMalloc(A)");
            if (st) return st;
        }
    launch(c, k_expand_stencil, cell_grid(c->g), cell_block(), 
        c->g, stencil_view(c), c->A[0], c->A[1], c->A[2], c->A[3], c->A[4], c->A[5], c->A[6]);
    // keep using the codes for the SpMV; the arrays are an exact copy
    c->A_valid = true;
    return check_launch(c, "expand stencil");
}

// Lays out the factor of an IC preconditioner for the applies that follow.
static les_status ic_ready(les_ctx* c, const les_pcg_opts* o)
{
    if (o->precond == LES_PC_IC) {
        if (!c->have_L) return fail(c, LES_BAD_ARG, "IC preconditioner needs les_build_ic or les_set_ic_factor");
        return ic_records64(c, (const double* const*)c->L);
    }
    if (o->precond == LES_PC_IC_A) {   // the factor arrays are A itself (src/pressure.cpp:363, :396)
        les_status st = ensure_stored_A(c);
        return st ? st : ic_records64(c, (const double* const*)c->A);
    }
    return LES_OK;
}

les_status precond_dev(les_ctx* c, const les_pcg_opts* o, const double* r, double* z, int skip_done)
{
    return precond_dot(c, o, r, z, skip_done, RD_NONE, false);
}

// PCG of src/pressure.cpp:342-414 in FP64 with the solution in P and the
// right-hand side in B.  The loop runs on the device; the host only polls
// the state between batches of iterations (kernels after convergence exit
// at once).
les_status pcg_fp64(les_ctx* c, const les_pcg_opts* o, les_pcg_result* res, int keep_tol)
{
    const Geo& g = c->g;
    les_status st = ensure_work(c);
    if (st) return st;
    if ((st = ic_ready(c, o))) return st;
    const bool pow2 = row_form(c) == ROW_POW2;
    if (pcg64_coop_used(c, o, pow2)) {
        if ((st = pcg64_coop(c, o, pow2, keep_tol))) return st;
        if ((st = wave_check(c))) return st;   // the exchanges' bounded waits
        if ((st = read_state(c))) return st;
        const SolverState& h = *c->h_state;
        if (res) {
            res->iters = h.iters;
            res->outer = 0;
            res->residual = h.err;
        }
        return (les_status)h.status;
    }
    StencilView A = stencil_view(c);
    double *x = c->slot[LES_P], *b = c->slot[LES_B];
    double *r = c->w[0], *z = c->w[1], *p = c->w[2], *q = c->w[3];
    const dim3 gr = cell_grid(g), bl = cell_block();
    launch(c, k_init_state, 1, 1, c->state, o->tol, o->max_iter, keep_tol);
    launch_spmv(c, -1, x, q, DOT_NONE);
    launch(c, k_resid, gr, bl, g, b, q, r, c->partials, c->counters + 4, c->state);
    st = precond_dot(c, o, r, p, 1, RD_RHO, false);
    if (st) return st;
    st = check_launch(c, "pcg init");
    if (st) return st;
    if (o->max_iter == 0) {
        // the reference's loop does not run; it returns max_iter (= 0)
        st = read_state(c);
        if (st) return st;
        if (res) { res->iters = 0; res->outer = 0; res->residual = c->h_state->err; }
        return c->h_state->done ? (les_status)c->h_state->status : LES_NOT_CONVERGED;
    }
    const bool jac = o->precond == LES_PC_JACOBI;
    const dim3 grr = reduce_grid(c);
    const bool cheb = o->precond == LES_PC_CHEBYSHEV;
    const double alpha0 = cheb ? cheb_alpha0(o) : 0.0;
    double* z0 = cheb ? cheb_z0(c, o, z) : nullptr;
    const DivBy by_c0 = div_by_const(c->coef.c0);
    int launched = 0, batch = 4;
    for (;;) {
        for (int it = 0; it < batch; ++it) {
            launch_spmv(c, PROF_SPMV64, p, q, DOT_ALPHA);
            launch_p(c, PROF_UPDATE64, k_update, grr, bl, g, A, x, r, (const double*)p, (const double*)q, z, c->partials,
                     c->counters + 5, c->state, jac ? 1 : 0, by_c0, alpha0, z0);
            if (!jac && (st = precond_dot(c, o, r, z, 1, RD_BETA, cheb))) return st;
            launch(c, k_pupdate, gr, bl, g, z, p, c->state);
        }
        launched += batch;
        st = check_launch(c, "pcg iteration");
        if (st) return st;
        st = read_state(c);
        if (st) return st;
        if (c->h_state->done || launched >= o->max_iter + 1) break;
        batch = batch < 32 ? batch * 2 : 32;
        if (launched + batch > o->max_iter + 1) batch = o->max_iter + 1 - launched;
        if (batch < 1) batch = 1;
    }
    if (o->precond == LES_PC_IC || o->precond == LES_PC_IC_A) {   // the wavefront's bounded waits
        st = wave_check(c);
        skew_trim(c);
        if (st) return st;
    }
    const SolverState& h = *c->h_state;
    if (res) {
        res->iters = h.iters;
        res->outer = 0;
        res->residual = h.err;
    }
    if (!h.done) return fail(c, LES_NOT_CONVERGED, "pcg: state not finalised");
    return (les_status)h.status;
}

les_status solve_jacobi_dev(les_ctx* c, double dt, double rho, int max_iter, double tol, int* sweeps)
{
    const Geo& g = c->g;
    les_status st = ensure_work(c);
    if (st) return st;
    const les_mesh& m = c->mesh;
    const dim3 gr = cell_grid(g), bl = cell_block();
    double* rhs = c->w[0];
    double* bufs[2] = {c->slot[LES_P], c->w[1]};
    const double dx2 = m.dx * m.dx, dy2 = m.dy * m.dy, dz2 = m.dz * m.dz;
    const double denom = 2 * (1.0 / dx2 + 1.0 / dy2 + 1.0 / dz2);
    launch(c, k_stat_rhs, gr, bl, g, rho / dt, div_by_const(2 * m.dx), div_by_const(2 * m.dy), div_by_const(2 * m.dz),
           (const double*)c->slot[LES_U], (const double*)c->slot[LES_V], (const double*)c->slot[LES_W], rhs);
    launch(c, k_init_state, 1, 1, c->state, tol, max_iter, 0);
    unsigned long long* const maxdp = reinterpret_cast<unsigned long long*>(c->partials);
    st = check_cuda(c, cudaMemsetAsync(maxdp, 0, 3 * sizeof *maxdp, c->stream), "memset");
    if (st) return st;
    // x / d for a power of two d is exactly x * (1 / d)
    auto pow2 = [](double v) { int e; return std::frexp(v, &e) == 0.5; };
    const bool p2 = pow2(dx2) && pow2(dy2) && pow2(dz2);
    auto sweep = !p2 ? k_jacobi_sweep<JAC_DIV>
                     : (dx2 == dy2 && dy2 == dz2 ? k_jacobi_sweep<JAC_EQUAL> : k_jacobi_sweep<JAC_POW2>);
    const dim3 gs(gr.x, gr.y, (g.nx + JAC_PLANES - 1) / JAC_PLANES);
    int launched = 0, batch = 16;
    int cur = 0;
    while (launched < max_iter) {
        for (int it = 0; it < batch && launched < max_iter; ++it, ++launched) {
            launch(c, sweep, gs, bl, g, div_by_const(dx2), div_by_const(dy2), div_by_const(dz2), div_by_const(denom),
                   (const double*)bufs[cur], bufs[cur ^ 1], (const double*)rhs, maxdp, c->state, launched, cur);
            cur ^= 1;
            if (c->n_solid)
                launch(c, k_pbc_obstacle_guarded, (c->n_solid + 255) / 256, 256, g, (const int*)c->solid_list,
                       c->n_solid, (const uint8_t*)c->mask, bufs[cur], c->state);
        }
        launch(c, k_jacobi_test, 1, 1, c->state, (const unsigned long long*)maxdp, launched, cur);
        st = check_launch(c, "jacobi sweeps");
        if (st) return st;
        st = read_state(c);
        if (st) return st;
        if (c->h_state->done) break;
        batch = 32;
    }
    if (max_iter <= 0) {
        if (sweeps) *sweeps = 0;
        return LES_OK;
    }
    // the converged field sits in bufs[state.buf]; mirror f.p.swap(p_new)
    if (c->h_state->buf == 1) std::swap(c->slot[LES_P], c->w[1]);
    if (sweeps) *sweeps = c->h_state->iters;
    return LES_OK;
}

}  // namespace les

extern "C" {

les_status les_divergence(les_ctx* c, double dt, double rho)
{
    if (!c) return LES_BAD_ARG;
    cudaSetDevice(c->device);
    const les_mesh& m = c->mesh;
    launch(c, k_div_b, cell_grid(c->g), cell_block(), 
        c->g, rho / dt, 1.0 / (2.0 * m.dx), 1.0 / (2.0 * m.dy), 1.0 / (2.0 * m.dz), 1.0 / m.dx,
        1.0 / m.dy, 1.0 / m.dz, c->slot[LES_U_NEW], c->slot[LES_V_NEW], c->slot[LES_W_NEW], c->mask,
        c->slot[LES_P_RHS], nullptr, c->partials, c->counters + 3, c->state, 0.0, nullptr, rho);
    return check_launch(c, "divergence");
}

les_status les_build_b(les_ctx* c)
{
    if (!c) return LES_BAD_ARG;
    cudaSetDevice(c->device);
    launch(c, k_build_b, cell_grid(c->g), cell_block(), c->g, c->slot[LES_P_RHS], c->mask,
                                                                c->slot[LES_B]);
    return check_launch(c, "build b");
}

les_status les_pressure_bcs(les_ctx* c)
{
    if (!c) return LES_BAD_ARG;
    cudaSetDevice(c->device);
    return pressure_bcs_dev(c, c->slot[LES_P]);
}

les_status les_build_stencil(les_ctx* c)
{
    if (!c) return LES_BAD_ARG;
    cudaSetDevice(c->device);
    if (!c->code) {
        les_status st = check_cuda(c, dev_malloc(c, &c->code, (size_t)c->g.n), "cudaMalloc(code)");
        if (st) return st;
    }
    const les_mesh& m = c->mesh;
    const double idx2 = 1.0 / (m.dx * m.dx), idy2 = 1.0 / (m.dy * m.dy), idz2 = 1.0 / (m.dz * m.dz);
    // src/pressure.cpp:613-623, and the doubled ghost coefficients of :663-696
    c->coef.c0 = (2.0 * idx2 + 2.0 * idy2 + 2.0 * idz2);
    c->coef.x1 = -idx2; c->coef.x2 = -idx2 + -idx2;
    c->coef.y1 = -idy2; c->coef.y2 = -idy2 + -idy2;
    c->coef.z1 = -idz2; c->coef.z2 = -idz2 + -idz2;
    unsigned* any_solid = c->counters + 30;
    les_status st = check_cuda(c, cudaMemsetAsync(any_solid, 0, sizeof(unsigned), c->stream), "memset");
    if (st) return st;
    launch(c, k_build_code, cell_grid(c->g), cell_block(), c->g, c->mask, c->code, any_solid);
    c->stencil_mode = 1;
    ++c->version;
    c->A_valid = false;   // a stale expansion of an older matrix must not be used
    if ((st = check_launch(c, "build stencil"))) return st;
    unsigned h = 1;
    st = check_cuda(c, cudaMemcpyAsync(&h, any_solid, sizeof(unsigned), cudaMemcpyDeviceToHost, c->stream), "copy");
    if (!st) st = check_cuda(c, cudaStreamSynchronize(c->stream), "build stencil");
    c->code_plain = st == LES_OK && h == 0u;
    return st;
}

les_status les_get_stencil(les_ctx* c, double* const* diag7)
{
    if (!c || !diag7) return LES_BAD_ARG;
    if (!c->stencil_mode) return fail(c, LES_BAD_ARG, "no matrix");
    cudaSetDevice(c->device);
    les_status st = ensure_work(c);
    if (st) return st;
    const size_t nb = sizeof(double) * (size_t)c->g.n;
    double* tmp[7];
    for (int q = 0; q < 7; ++q) {
        st = check_cuda(c, dev_malloc(c, &tmp[q], nb), "cudaMalloc(tmp)");
        if (st) return st;
    }
    launch(c, k_expand_stencil, cell_grid(c->g), cell_block(), c->g, stencil_view(c), tmp[0], tmp[1],
                                                                       tmp[2], tmp[3], tmp[4], tmp[5], tmp[6]);
    for (int q = 0; q < 7; ++q)
        if (diag7[q]) cudaMemcpyAsync(diag7[q], tmp[q], nb, cudaMemcpyDeviceToHost, c->stream);
    st = check_cuda(c, cudaStreamSynchronize(c->stream), "get stencil");
    for (int q = 0; q < 7; ++q) cudaFree(tmp[q]);
    return st;
}

les_status les_spmv(les_ctx* c, int in, int out)
{
    if (!c || in < 0 || in >= LES_NSLOTS || out < 0 || out >= LES_NSLOTS || in == out) return LES_BAD_ARG;
    cudaSetDevice(c->device);
    return spmv_dev(c, c->slot[in], c->slot[out]);
}

les_status les_dot(les_ctx* c, int a, int b, double* out)
{
    if (!c || a < 0 || a >= LES_NSLOTS || b < 0 || b >= LES_NSLOTS || !out) return LES_BAD_ARG;
    cudaSetDevice(c->device);
    return dot_dev(c, c->slot[a], c->slot[b], out);
}

les_status les_axpby(les_ctx* c, int out, double a, int in1, double b, int in2)
{
    if (!c || out < 0 || out >= LES_NSLOTS || in1 < 0 || in1 >= LES_NSLOTS || in2 < 0 || in2 >= LES_NSLOTS)
        return LES_BAD_ARG;
    cudaSetDevice(c->device);
    launch(c, k_axpby, cell_grid(c->g), cell_block(), c->g, a, (const double*)c->slot[in1], b,
           (const double*)c->slot[in2], c->slot[out]);
    return check_launch(c, "axpby");
}

les_status les_precond_apply(les_ctx* c, const les_pcg_opts* o, int in, int out)
{
    if (!c || !o || in < 0 || in >= LES_NSLOTS || out < 0 || out >= LES_NSLOTS || in == out) return LES_BAD_ARG;
    cudaSetDevice(c->device);
    if (!c->stencil_mode && o->precond != LES_PC_IC) return fail(c, LES_BAD_ARG, "no matrix");
    les_status st = ic_ready(c, o);
    if (!st) st = precond_dev(c, o, c->slot[in], c->slot[out], 0);
    if (o->precond == LES_PC_IC || o->precond == LES_PC_IC_A) {
        if (!st) st = wave_check(c);   // waits for the wavefront: LES_TIMEOUT if a bounded wait gave up
        skew_trim(c);
    }
    return st;
}

les_status les_pcg(les_ctx* c, const les_pcg_opts* o, les_pcg_result* res)
{
    if (!c || !o || o->max_iter < 0) return LES_BAD_ARG;
    if (!c->stencil_mode) return fail(c, LES_BAD_ARG, "no matrix: call les_build_stencil or les_set_stencil");
    cudaSetDevice(c->device);
    if (o->precision == LES_MIXED) return pcg_mixed(c, o, res);
    return pcg_fp64(c, o, res, 0);
}

les_status les_solve_jacobi(les_ctx* c, double dt, double rho, int max_iter, double tol, int* sweeps)
{
    if (!c || max_iter < 0) return LES_BAD_ARG;
    cudaSetDevice(c->device);
    return solve_jacobi_dev(c, dt, rho, max_iter, tol, sweeps);
}

les_status les_lambda_max(les_ctx* c, int n_iter, const double* v0, double* lambda)
{
    if (!c || !lambda || n_iter < 0) return LES_BAD_ARG;
    if (!c->stencil_mode) return fail(c, LES_BAD_ARG, "no matrix");
    cudaSetDevice(c->device);
    les_status st = ensure_work(c);
    if (st) return st;
    const Geo& g = c->g;
    std::vector<double> h;
    if (!v0) {
        // src/pressure.cpp:926-931 as drawn by one thread
        h.resize(g.n);
        std::mt19937 gen(1337);
        std::uniform_real_distribution<> dis(-1.0, 1.0);
        for (int i = 0; i < g.n; ++i) h[i] = dis(gen);
        v0 = h.data();
    }
    double *v = c->w[0], *w = c->w[1];
    st = check_cuda(c, cudaMemcpyAsync(v, v0, sizeof(double) * g.n, cudaMemcpyHostToDevice, c->stream), "upload v0");
    if (st) return st;
    const dim3 gr = cell_grid(g), bl = cell_block();
    double lam = 0.0;
    for (int it = 0; it < n_iter; ++it) {
        launch_spmv(c, -1, v, w, DOT_SCAL0);
        // lambda = v.w (spmv's fused dot is p.q = v.w)
        st = read_state(c);
        if (st) return st;
        lam = c->h_state->scal[0];
        launch(c, k_dot, reduce_grid(c), bl, g, w, w, c->partials, c->counters + 2, c->state, RD_SCAL0, 0);
        launch(c, k_norm_of, 1, 1, c->state);
        launch(c, k_scale_inv, gr, bl, g, v, w, c->state);   // v = w / ||w||
        st = check_launch(c, "lambda iteration");
        if (st) return st;
    }
    st = check_cuda(c, cudaStreamSynchronize(c->stream), "sync");
    if (st) return st;
    *lambda = lam;
    return LES_OK;
}

}  // extern "C"
