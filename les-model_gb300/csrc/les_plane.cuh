// les_plane.cuh -- device code of the plane marches: the FP32 inner PCG
// iteration of the mixed-precision solve (the two passes of les_col.cu) with
// a block, not a warp, as the unit that shares halos.
//
// A block owns a tile of the (j, k) plane and marches along i over a chunk of
// planes.  A thread holds four consecutive k cells (one 16-byte vector) of two
// neighbouring rows in registers for the planes a stencil needs.  The i
// neighbours of a cell are registers of its own thread, the k neighbours come
// from the adjacent lanes by shuffle, and the rows above and below a thread's
// two rows come from shared memory.  At march step I level L works on plane
// I-L, so the rows it needs from other threads belong to a plane that was
// finished in step I-1: each step publishes its rows in one of two buffers and
// reads the other, and one block barrier per step orders everything.
//
// Against the strips of les_col_march.cuh (a warp per strip, one cell per lane,
// 14 rows in registers for 8 owned ones) the tile is wider along k, so its
// k halo shrinks to nothing for rows of up to 128 cells, the j halo is shared
// by the block, loads and stores are 16 bytes wide, the arithmetic is packed
// (two cells per instruction) and 12 warps instead of 8 run on an SM.
// Microseconds per inner iteration, strips -> plane marches (GB300):
//   64x32x32 degree 4     22.6 -> 11.1     256x128x128 degree 4   46.4 -> 37.7
//   161x93x75 degree 5    36.5 -> 25.0     256x128x128 degree 7    138 -> 72
//   128x96x96 degree 4    28.3 -> 20.6     512x256x256 degree 4    335 -> 252
//   200x90x90 Jacobi      19.4 -> 15.4     384x200x257 degree 5    302 -> 220
// What bounds them: pass A at 512x256x256 the HBM rate (24 B per cell, 126 us:
// 6.4 TB/s, 0.95 of the measured copy).  Pass B the chain of a step (level,
// barrier and shared-memory latency) with three warps per scheduler: at
// 512x256x256 124 us for 16 B per cell, 0.65 of that rate.  Small grids the
// two grid sums of an iteration and the launches between them.
//
// Measured and dropped: operands staged through shared memory with cp.async
// three planes ahead (pass A of 512x256x256 126 -> 145 us, pass B 124 -> 146:
// the copies and reads take the shared-memory bandwidth that the published
// rows need); one step per loop pass with the rings moved (150 us); 512
// threads at 128 registers (282 us: 0.5 KB of spills).
//
// Layout.  The inner vectors' rows are padded to a multiple of four cells so
// that every row starts on a 16-byte boundary (plane_pitch); pads of r, z, p, q
// and e are kept at zero.
//
// The matrix is the position-dependent one of les_col.cu: mirrors at the inlet
// plane and at the j and k walls, no east coefficient on plane nx-2, identity
// rows on the outlet plane.  A tile that touches a wall takes the mirrored
// neighbour itself (west = east on plane 0, the row or cell inside for the row
// or cell outside), so tiles have halos only towards other tiles.
#pragma once
#include "les_col_march.cuh"

namespace les {

constexpr int PV = 4;   // cells per thread along k
constexpr int PR = 2;   // rows per thread

// Threads of a block: the largest whose registers hold the level rings of an
// unrolled march without a spill (three levels at 512 threads and 128
// registers spill 0.5 KB, and pass B of 512x256x256 takes 282 instead of
// 124 us; at 384 threads none).
__host__ __device__ constexpr int plane_threads_b(int S) { return S <= 2 ? 512 : (S == 3 ? 384 : 256); }
__host__ __device__ constexpr int plane_threads_a() { return 448; }

// A published vector's levels lie side by side, an odd number of 16-byte
// slots apart from the next vector's (no bank conflicts); a buffer has the
// largest block's size, so that levels and buffers are immediate offsets.
__host__ __device__ constexpr int plane_sp(int S) { return S | 1; }
__host__ __device__ constexpr int plane_pub(int threads, int levels) { return 2 * threads * PR * plane_sp(levels); }
constexpr size_t plane_smem(int threads, int levels) { return (size_t)16 * plane_pub(threads, levels); }

// ColCheb for the plane marches.  Level k is kept divided by s_k, the product
// of the levels' i weights, so that the i neighbours need no weight and the j
// and k weights (the ratios of the spacings) are the same for every level:
// fewer weights to hold in registers.  Each weight is stored twice, for the
// packed multiply-adds.
struct ChebPairs {
    float2 wy, wz;          // weights of the j and k neighbours
    float2 cc[6], ci[6];    // centre; on the outlet plane's identity rows
    float2 rr[6], gg[6];    // r' and z_{k-2} at the centre
    float2 zs;              // s_S: the last level's z
};

ChebPairs cheb_pairs(const ColCheb& c, int S);

struct PlaneArgsA {
    Geo g;            // strides of the padded layout
    PlaneMap m;
    Coef k;
    const float4 *z, *pold;
    float4 *pnew, *q, *e;
    SolverState *st, *outer;
    int pslot, total_cap;
    Defer df;
};

struct PlaneArgsB {
    Geo g;
    PlaneMap m;
    ChebPairs c3;
    float inv_c0;
    const float4 *r_in, *q;
    float4 *r_out, *z_out;
    SolverState *st, *outer;
    Defer df;
};

using KPA = void (*)(PlaneArgsA);
using KPB = void (*)(PlaneArgsB);
// form 0: rows of 32, 64 or 128 cells (whole rows per warp); 1: other
// multiples of four; 2: any length
KPB plane_pick_b_lo(int S, int form, bool first);   // S = 1..3
KPB plane_pick_b_hi(int S, int form, bool first);   // S = 4..6

}  // namespace les

namespace {

extern __shared__ float4 plane_sm[];

// Four cells as two pairs: the arithmetic is packed FP32 (two cells per
// instruction), the pairs those of a 16-byte load.
struct Vec {
    float2 lo, hi;
};

__device__ __forceinline__ Vec vec(const float4& a) { return Vec{make_float2(a.x, a.y), make_float2(a.z, a.w)}; }
__device__ __forceinline__ float4 f4(const Vec& a) { return make_float4(a.lo.x, a.lo.y, a.hi.x, a.hi.y); }
__device__ __forceinline__ Vec vzero() { return Vec{make_float2(0.f, 0.f), make_float2(0.f, 0.f)}; }
__device__ __forceinline__ float2 dup(float w) { return make_float2(w, w); }
__device__ __forceinline__ Vec vfma(float w, const Vec& a, const Vec& b)
{
    return Vec{__ffma2_rn(dup(w), a.lo, b.lo), __ffma2_rn(dup(w), a.hi, b.hi)};
}
__device__ __forceinline__ Vec vfma(float2 w, const Vec& a, const Vec& b)
{
    return Vec{__ffma2_rn(w, a.lo, b.lo), __ffma2_rn(w, a.hi, b.hi)};
}
__device__ __forceinline__ Vec vmul(float2 w, const Vec& a) { return Vec{__fmul2_rn(w, a.lo), __fmul2_rn(w, a.hi)}; }
__device__ __forceinline__ Vec vmul(float w, const Vec& a)
{
    return Vec{__fmul2_rn(dup(w), a.lo), __fmul2_rn(dup(w), a.hi)};
}
__device__ __forceinline__ Vec vadd(const Vec& a, const Vec& b) { return Vec{__fadd2_rn(a.lo, b.lo), __fadd2_rn(a.hi, b.hi)}; }
__device__ __forceinline__ float vdot(const Vec& a, const Vec& b)
{
    const float2 t = __ffma2_rn(a.hi, b.hi, __fmul2_rn(a.lo, b.lo));
    return t.x + t.y;
}

// vectors at 32-bit byte offsets from a uniform base
__device__ __forceinline__ Vec ldv(const float4* p, unsigned off)
{
    return vec(*reinterpret_cast<const float4*>(reinterpret_cast<const char*>(p) + off));
}
__device__ __forceinline__ void stv(float4* p, unsigned off, const Vec& v)
{
    *reinterpret_cast<float4*>(reinterpret_cast<char*>(p) + off) = f4(v);
}

// A thread's place in its block's tile.
struct TilePos {
    int i0, i1;          // owned planes
    unsigned off[PR];    // byte offset of each row's vector on plane 0
    int sm;              // index of row 0 in a published plane; row r at sm + r * lk
    int up, dn;          // published index of the row above row 0, below row 1
    int lane_l;          // vector of the row this thread holds
    int last;            // component that holds the row's last cell (-1: none of this vector)
    bool own[PR];        // rows owned by this thread (and its vector owned along k)
    bool left_wall;      // the vector starts at k = 0
    bool fix_l, fix_r;   // the k neighbour's lane is in another warp
    bool idle;           // no rows: takes part in barriers and shuffles only
};

template <int HALO>
__device__ __forceinline__ TilePos tile_pos(const Geo& g, const PlaneMap& m, int blk)
{
    TilePos t;
    const int kt = blk % m.nk, rest = blk / m.nk;
    const int jt = rest % m.nj, ch = rest / m.nj;
    t.i0 = ch * m.ci;
    t.i1 = min(g.nx, t.i0 + m.ci);
    const int tid = threadIdx.x;
    int gr = tid / m.lk;
    const int l = tid - gr * m.lk;
    t.idle = gr >= m.groups;
    gr = min(gr, m.groups - 1);
    const int H = m.groups * PR;
    const int jo0 = jt * m.tj, jo1 = min(g.ny, jo0 + m.tj), jt0 = max(0, jo0 - HALO);
    const int ko0 = kt * m.kw, ko1 = min(g.nz, ko0 + m.kw), kt0 = max(0, ko0 - ((HALO + 3) / 4) * 4);
    const int k = kt0 + PV * l;
    const bool kown = k >= ko0 && k < ko1;
    const int kc = min(k, g.sj - PV);   // vectors past the row read its last one (never used)
    const int r0 = gr * PR;
#pragma unroll
    for (int r = 0; r < PR; ++r) {
        const int j = jt0 + r0 + r;
        t.own[r] = !t.idle && kown && j >= jo0 && j < jo1;
        // the row past the wall mirrors
        t.off[r] = 4u * (unsigned)(max(j < g.ny ? j : 2 * (g.ny - 1) - j, 0) * g.sj + kc);
    }
    t.sm = r0 * m.lk + l;
    const int ja = jt0 + r0, jb = ja + PR - 1;
    const int tu = ja == 0 ? 1 : max(r0 - 1, 0);
    const int tb = r0 + PR - 1;
    const int td = jb == g.ny - 1 ? tb - 1 : (jb == g.ny ? max(tb - 3, 0) : min(tb + 1, H - 1));
    t.up = tu * m.lk + l;
    t.dn = td * m.lk + l;
    t.lane_l = l;
    t.last = (k <= g.nz - 1 && g.nz - 1 < k + PV) ? g.nz - 1 - k : -1;
    t.left_wall = k == 0;
    const int lane = tid & 31;
    t.fix_l = lane == 0 && l > 0;
    t.fix_r = lane == 31 && l < m.lk - 1;
    return t;
}

// Sums of the k neighbours of a vector's cells.  pub: the published place of
// this vector (for lanes whose neighbour is in another warp), SP the distance
// of its neighbours.
template <int FORM, int SP>
__device__ __forceinline__ Vec k_sum(const Vec& c, const TilePos& t, const float4* pub)
{
    float l = __shfl_up_sync(FULL, c.hi.y, 1), r = __shfl_down_sync(FULL, c.lo.x, 1);
    if (FORM != 0) {
        if (t.fix_l) l = pub[-SP].w;
        if (t.fix_r) r = pub[SP].x;
    }
    if (t.left_wall) l = c.lo.y;
    if (FORM == 2) {   // the neighbour past the row's last cell mirrors
        Vec s{make_float2(l + (t.last == 0 ? l : c.lo.y), c.lo.x + (t.last == 1 ? c.lo.x : c.hi.x)),
              make_float2(c.lo.y + (t.last == 2 ? c.lo.y : c.hi.y), c.hi.x + (t.last == 3 ? c.hi.x : r))};
        return s;
    }
    if (t.last == PV - 1) r = c.hi.x;
    return Vec{make_float2(l + c.lo.y, c.lo.x + c.hi.x), make_float2(c.lo.y + c.hi.y, c.hi.x + r)};
}

// cells past the end of the row (only with FORM 2) set to zero
template <int FORM>
__device__ __forceinline__ void zero_pads(Vec& v, const TilePos& t)
{
    if (FORM == 2 && t.last >= 0) {
        if (t.last < 1) v.lo.y = 0.f;
        if (t.last < 2) v.hi.x = 0.f;
        if (t.last < 3) v.hi.y = 0.f;
    }
}

// ---- the heads -------------------------------------------------------------------
// The deferred sums and decisions of head_a / head_b (les_col_march.cuh) for a
// few hundred partials at most, with nothing on the FP64 pipe where a
// dependent operation takes 64 cycles and more: the sums stay (hi, lo) pairs,
// quotients are formed from pairs on the FP32 pipe, and the root of ||r||^2 is
// taken once, at the end of a solve.  The partials and the state are read
// together.  64x32x32: 12.6 -> 11.5 us per iteration, 128x64x64:
// 16.4 -> 15.0, 256x128x128: 40.1 -> 38.7.

// num / den of pairs, rounded to FP32: both scaled by the power of two that
// brings d.hi to [1/4, 1/2) (a small one's reciprocal would be infinite), the
// quotient of the high parts by the reciprocal, and one correction by the
// remainder: within 2^-45 before the rounding, so that about one in 10^7 operands
// rounds differently from the pairs' FP64 quotient (a subnormal one may lose its
// last bits).  A quotient of the high parts that is zero or not finite stands as it
// is.  With a branch to FP64 for small operands instead an iteration at 128x64x64
// took 0.06 to 0.3 us longer.
__device__ __forceinline__ float df_quotient(const Acc& n, const Acc& d)
{
    const unsigned e = min((__float_as_uint(d.hi) >> 23) & 0xffu, 251u);
    const float s = __uint_as_float((252u - e) << 23);
    const float nh = __fmul_rn(n.hi, s), nl = __fmul_rn(n.lo, s), dh = __fmul_rn(d.hi, s), dl = __fmul_rn(d.lo, s);
    const float y = __frcp_rn(dh), q = __fmul_rn(nh, y);
    const float r = __fadd_rn(fmaf(-q, dh, nh), fmaf(-q, dl, nl));
    const bool plain = (__float_as_uint(q) << 1) - 1u < 0xfeffffffu;
    return plain ? fmaf(r, y, q) : q;
}

// Sums NV vectors of nb partials, the totals in thread 0.
template <int NV>
__device__ __forceinline__ void head_sum(const float2* __restrict__ part, int nb, Acc (&v)[NV], float2* sm)
{
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int nw = min((int)blockDim.x, (nb + 31) & ~31) >> 5;   // warps that hold partials
    if (warp < nw) {
        for (int b = threadIdx.x; b < nb; b += blockDim.x)
#pragma unroll
            for (int q = 0; q < NV; ++q) {
                const float2 t = __ldcg(part + q * nb + b);
                Acc x;
                x.hi = t.x;
                x.lo = t.y;
                v[q] = df_add(v[q], x);
            }
#pragma unroll
        for (int q = 0; q < NV; ++q)
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) {
                Acc t;
                t.hi = __shfl_down_sync(FULL, v[q].hi, o);
                t.lo = __shfl_down_sync(FULL, v[q].lo, o);
                v[q] = df_add(v[q], t);
            }
        if (lane == 0)
#pragma unroll
            for (int q = 0; q < NV; ++q) sm[q * 16 + warp] = make_float2(v[q].hi, v[q].lo);
    }
    __syncthreads();
    if (threadIdx.x == 0)
        for (int w = 1; w < nw; ++w)
#pragma unroll
            for (int q = 0; q < NV; ++q) {
                Acc x;
                x.hi = sm[q * 16 + w].x;
                x.lo = sm[q * 16 + w].y;
                v[q] = df_add(v[q], x);
            }
}

// The inner state's fields that the plane passes hand to each other in pairs
// lie in the double fields: rho, rho_next (bit patterns of float2).
__device__ __forceinline__ Acc get_pair(const double* f)
{
    const float2 t = __ldcg(reinterpret_cast<const float2*>(f));
    Acc a;
    a.hi = t.x;
    a.lo = t.y;
    return a;
}
__device__ __forceinline__ void put_pair(double* f, const Acc& a) { *reinterpret_cast<float2*>(f) = make_float2(a.hi, a.lo); }

// Pass A: pass B's sums ||r'||^2 and r'.z, the convergence test, beta.
template <bool FIRST>
__device__ __noinline__ HeadOut plane_head_a(const float2* __restrict__ pin, int nb_in, SolverState* st,
                                             SolverState* outer, int total_cap, int pslot, int blk)
{
    __shared__ float2 sm[32];
    __shared__ HeadOut so;
    Acc v[2], rho_old;
    double tol = 0.0;
    int done = 0, kk = 0, total = 0, max_iter = 0, frozen = 0;
    if (threadIdx.x == 0) {
        done = __ldcg(&st->done);
        if (!FIRST) {
            rho_old = get_pair(&st->rho);
            tol = __ldcg(&st->tol);
            kk = __ldcg(&st->k);   // committed by pass B
            total = __ldcg(&outer->iters);
            max_iter = __ldcg(&st->max_iter);
            frozen = __ldcg(&st->frozen);
        }
    }
    head_sum<2>(pin, nb_in, v, sm);
    if (threadIdx.x == 0) {
        const bool w0 = blk == 0;
        so.end = 1;
        if (!done) {
            int status = -1;
            so.coef = 0.f;
            if (!FIRST) {
                const double rr = (double)v[0].hi + (double)v[0].lo;
                if (rr < tol * tol) status = tol > 0.0 ? LES_OK : -1;
                else if (!(rr < 1.7976931348623157e308)) status = LES_NONFINITE;
                if (status < 0 && (kk >= max_iter || total >= total_cap)) status = LES_NOT_CONVERGED;
                if (frozen) status = -1;
                so.coef = frozen ? 0.f : df_quotient(v[1], rho_old);
            }
            if (w0) {
                if (status >= 0) {   // the solve ends at iteration kk: the final state
                    st->err = sqrt((double)v[0].hi + (double)v[0].lo);
                    st->status = status;
                    st->done = 1;
                } else {
                    put_pair(&st->rho_next, v[1]);
                    st->buf = pslot;   // buffer holding this iteration's p
                }
            }
            so.end = status >= 0;   // no work after the last iteration
        }
    }
    __syncthreads();
    return so;
}

// Pass B: pass A's sum p.q, alpha and the commit of the iteration.
__device__ __noinline__ HeadOut plane_head_b(const float2* __restrict__ pin, int nb_in, SolverState* st,
                                             SolverState* outer, int blk)
{
    __shared__ float2 sm[16];
    __shared__ HeadOut so;
    Acc v[1], rho;
    int done = 0, frozen = 0;
    if (threadIdx.x == 0) {
        done = __ldcg(&st->done);
        rho = get_pair(&st->rho_next);
        frozen = __ldcg(&st->frozen);
    }
    head_sum<1>(pin, nb_in, v, sm);
    if (threadIdx.x == 0) {
        so.end = done;
        so.coef = frozen ? 0.f : df_quotient(rho, v[0]);
        if (blk == 0 && !done) {
            st->alpha = (double)so.coef;
            put_pair(&st->rho, rho);
            st->k = st->k + 1;
            outer->iters = outer->iters + 1;
        }
    }
    __syncthreads();
    return so;
}

// ---- pass A -----------------------------------------------------------------
// p = z + beta p_old, e += alpha_prev p_old, q = A p, p.q (les_col.cu).
template <int TMAX, int FORM, bool FIRST>
__device__ __forceinline__ void plane_a(const PlaneArgsA& a, int blk, int nblk)
{
    __shared__ double sm[64];
    const Geo& g = a.g;
    const PlaneMap& m = a.m;
    const TilePos t = tile_pos<1>(g, m, blk);
    const unsigned si = 4u * (unsigned)g.si;
    const int is = t.i0 > 0 ? t.i0 - 1 : 0;
    // two planes ahead (one ahead in 512 threads: 20.8 us at 256x128x128, two in
    // 448: 19.7); planes past the outlet read the outlet plane (weight 0),
    // planes that are not owned some e (not used)
    Vec fz[2][PR], fp[2][PR], fe[2][PR];
    auto fetch = [&](int P, int s) {
        const unsigned at = (unsigned)min(P, g.nx - 1) * si;
#pragma unroll
        for (int r = 0; r < PR; ++r) {
            fz[s][r] = ldv(a.z, at + t.off[r]);
            if (!FIRST) {
                fp[s][r] = ldv(a.pold, at + t.off[r]);
                fe[s][r] = ldv(a.e, at + t.off[r]);
            }
        }
    };
    dep_wait();
    fetch(is, 0);   // on their way while the head sums
    fetch(is + 1, 1);
    const HeadOut h = plane_head_a<FIRST>(a.df.pin, a.df.nb_in, a.st, a.outer, a.total_cap, a.pslot, blk);
    if (h.end) return;
    const float beta = h.coef, aprev = FIRST ? 0.f : (float)a.st->alpha;
    Acc acc;
    // p of plane P in slot P - is modulo 4 (the steps are unrolled four times,
    // so slots, buffers and their addresses are known at compile time)
    Vec p[4][PR];
#pragma unroll
    for (int q = 0; q < 4; ++q) p[q][0] = p[q][1] = vzero();
    float4* const own = plane_sm + t.sm;
    const float4 *const up_at = plane_sm + t.up, *const dn_at = plane_sm + t.dn;
    const int lk = m.lk;
    for (int P0 = is; P0 <= t.i1; P0 += 4) {
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            const int P = P0 + u;
            if (P > t.i1) break;
            constexpr int BUF = TMAX * PR;
            const int put = (u & 1) * BUF, got = ((u & 1) ^ 1) * BUF;
            Vec(&vz)[PR] = fz[u & 1], (&vp)[PR] = fp[u & 1], (&ve)[PR] = fe[u & 1];
            Vec(&p0)[PR] = p[u], (&p1)[PR] = p[(u + 3) & 3], (&p2)[PR] = p[(u + 2) & 3];
            const unsigned at = (unsigned)P * si;
#pragma unroll
            for (int r = 0; r < PR; ++r) p0[r] = FIRST ? vz[r] : vfma(beta, vp[r], vz[r]);
            if (!t.idle) {
#pragma unroll
                for (int r = 0; r < PR; ++r) own[put + r * lk] = f4(p0[r]);
            }
            if (P >= t.i0 && P < t.i1) {
#pragma unroll
                for (int r = 0; r < PR; ++r)
                    if (t.own[r]) {
                        stv(a.pnew, at + t.off[r], p0[r]);
                        stv(a.e, at + t.off[r], FIRST ? vzero() : vfma(aprev, vp[r], ve[r]));
                    }
            }
            if (P + 1 < t.i1) fetch(P + 2, u & 1);
            const int C = P - 1;
            if (C >= t.i0) {
                const bool ident = C == g.nx - 1;
                const float cc = ident ? 1.f : a.k.c0, cy = ident ? 0.f : a.k.y1, cz = ident ? 0.f : a.k.z1;
                const float cw = ident || C == 0 ? 0.f : a.k.x1;
                const float ce = ident || C == g.nx - 2 ? 0.f : (C == 0 ? 2.f * a.k.x1 : a.k.x1);
                const Vec up = vec(up_at[got]), dn = vec(dn_at[got]);
                float s = 0.f;
#pragma unroll
                for (int r = 0; r < PR; ++r) {
                    const Vec js = vadd(r == 0 ? up : p1[0], r == 0 ? p1[1] : dn);
                    const Vec ks = k_sum<FORM, 1>(p1[r], t, own + got + r * lk);
                    Vec qv = vfma(cz, ks, vfma(cy, js, vfma(ce, p0[r], vfma(cw, p2[r], vmul(cc, p1[r])))));
                    zero_pads<FORM>(qv, t);
                    const float d = vdot(p1[r], qv);
                    if (t.own[r]) {
                        stv(a.q, at - si + t.off[r], qv);
                        s += d;
                    }
                }
                acc_add(acc, s);
            }
            __syncthreads();
        }
    }
    dep_signal();
    Acc v[1] = {acc};
    put_partials<1>(v, reinterpret_cast<float2*>(sm), a.df.pout, blk, nblk);
}

// ---- pass B -----------------------------------------------------------------
// The march of one block.  EDGE: the chunk reaches the inlet plane or the last
// two planes, whose level weights differ (plane-uniform selects); the other
// chunks take every weight as a constant.
template <int TMAX, int S, int FORM, bool FIRST, bool EDGE, class Fetch>
__device__ __forceinline__ void march_b(const PlaneArgsB& a, const TilePos& t, float alpha, int is, unsigned si,
                                        Vec (&vr)[PR], Vec (&vq)[PR], const Fetch& fetch, Acc& arr,
                                        Acc& arz)
{
    constexpr int NL = S > 1 ? S - 1 : 1;   // stored levels z_1 .. z_{S-1}
    // r' at planes I - d: level 1 reads three planes, level L >= 2 plane I - L
    constexpr int NP = S <= 3 ? 4 : S + 1;
    // Four steps per loop pass: buffers are known at compile time and the
    // rings are slots that rotate by renaming (r' of more than four planes
    // moves along rp).  Five and six levels would spill: one step per pass.
    constexpr int UN = S <= 4 ? 4 : 1;
    constexpr bool SLOT_R = S <= 3, SLOT_Z = UN == 4;
    constexpr int SP = plane_sp(S), BUF = TMAX * PR * SP;
    const int nx = a.g.nx, lk = a.m.lk, end = t.i1 + S;
    const ChebPairs& c3 = a.c3;
    Vec rp[NP][PR];
    Vec zr[NL][4][PR];       // z_L of step I: slot I - is modulo 4
#pragma unroll
    for (int r = 0; r < PR; ++r) {
#pragma unroll
        for (int d = 0; d < NP; ++d) rp[d][r] = vzero();
#pragma unroll
        for (int L = 0; L < NL; ++L) zr[L][0][r] = zr[L][1][r] = zr[L][2][r] = zr[L][3][r] = vzero();
    }
    // published planes: [parity][row, vector][r', z_1 .. z_{S-1}]
    float4* const own = plane_sm + t.sm * SP;
    const float4 *const up_at = plane_sm + t.up * SP, *const dn_at = plane_sm + t.dn * SP;
    const int row1 = lk * SP;
    for (int I0 = is; I0 < end; I0 += UN) {
#pragma unroll
        for (int u = 0; u < UN; ++u) {
            const int I = I0 + u;
            if (I >= end) break;
            const int par = UN == 4 ? u & 1 : (I - is) & 1;
            const int put = par * BUF, got = (par ^ 1) * BUF;
            const unsigned at = (unsigned)I * si;
            // plane I - d of r', z_L of d steps ago
            auto R = [&](int d) -> Vec(&)[PR] { return rp[SLOT_R ? (u + 8 - d) & 3 : d]; };
            auto Z = [&](int L, int d) -> Vec(&)[PR] { return zr[L - 1][SLOT_Z ? (u + 4 - d) & 3 : d]; };
            // ---- level 0 at plane I
            Vec(&r0)[PR] = R(0);
#pragma unroll
            for (int r = 0; r < PR; ++r) r0[r] = FIRST ? vr[r] : vfma(-alpha, vq[r], vr[r]);
            if (!t.idle) {
#pragma unroll
                for (int r = 0; r < PR; ++r) own[put + r * row1] = f4(r0[r]);
            }
            if (I >= t.i0 && I < t.i1) {
                float s = 0.f;
#pragma unroll
                for (int r = 0; r < PR; ++r) {
                    const float d = vdot(r0[r], r0[r]);
                    if (t.own[r]) {
                        stv(a.r_out, at + t.off[r], r0[r]);
                        s += d;
                    }
                }
                acc_add(arr, s);
            }
            if (I + 1 < end) fetch(I + 1);
            // ---- Chebyshev levels 1..S at planes I-1 .. I-S
#pragma unroll
            for (int LV = 1; LV <= S; ++LV) {
                const int Pk = I - LV;
                const bool ident = EDGE && Pk == nx - 1;   // identity rows
                const float2 none = make_float2(0.f, 0.f), one2 = make_float2(1.f, 1.f);
                // the inlet plane's west neighbour is its east one; the plane
                // before the outlet has no east coefficient
                const float2 wc = ident ? c3.ci[LV - 1] : c3.cc[LV - 1];
                const float2 ww = EDGE && (ident || Pk == 0) ? none : one2;
                const float2 we = EDGE && (ident || Pk == nx - 2) ? none : (EDGE && Pk == 0 ? make_float2(2.f, 2.f) : one2);
                const float2 wy = ident ? none : c3.wy, wz = ident ? none : c3.wz;
                const Vec up = vec(up_at[got + LV - 1]), dn = vec(dn_at[got + LV - 1]);
                // level 1: the stencil of z_0 = a0 r' (a0 is in the weights)
                constexpr int one = 1;
                const Vec(&zc)[PR] = LV == 1 ? R(1) : Z(LV < 2 ? one : LV - 1, 1);
                const Vec(&zw)[PR] = LV == 1 ? R(2) : Z(LV < 2 ? one : LV - 1, 2);
                const Vec(&ze)[PR] = LV == 1 ? R(0) : Z(LV < 2 ? one : LV - 1, 0);
                Vec zk[PR];
#pragma unroll
                for (int r = 0; r < PR; ++r) {
                    const Vec js = vadd(r == 0 ? up : zc[0], r == 0 ? zc[1] : dn);
                    const Vec ks = k_sum<FORM, SP>(zc[r], t, own + got + r * row1 + LV - 1);
                    Vec v = EDGE ? vfma(we, ze[r], vmul(ww, zw[r])) : vadd(ze[r], zw[r]);
                    v = vfma(wz, ks, vfma(wy, js, vfma(wc, zc[r], v)));
                    if (LV >= 2) v = vfma(c3.rr[LV - 1], R(LV)[r], v);
                    if (LV >= 3) v = vfma(c3.gg[LV - 1], Z(LV < 3 ? one : LV - 2, 2)[r], v);
                    zk[r] = v;
                }
                if (LV < S) {
#pragma unroll
                    for (int r = 0; r < PR; ++r) {
                        Z(LV < S ? LV : one, 0)[r] = zk[r];
                        if (!t.idle) own[put + r * row1 + LV] = f4(zk[r]);
                    }
                }
                if (LV == S && Pk >= t.i0 && Pk < t.i1) {
                    float s = 0.f;
#pragma unroll
                    for (int r = 0; r < PR; ++r) {
                        zk[r] = vmul(c3.zs, zk[r]);
                        zero_pads<FORM>(zk[r], t);
                        const float d = vdot(R(S)[r], zk[r]);
                        if (t.own[r]) {
                            stv(a.z_out, at - S * si + t.off[r], zk[r]);
                            s += d;
                        }
                    }
                    acc_add(arz, s);
                }
            }
#pragma unroll
            for (int r = 0; r < PR; ++r) {
                if (!SLOT_R) {
#pragma unroll
                    for (int d = NP - 1; d >= 1; --d) rp[d][r] = rp[d - 1][r];
                }
                if (!SLOT_Z) {
#pragma unroll
                    for (int L = 0; L < S - 1; ++L) {
                        zr[L][2][r] = zr[L][1][r];
                        zr[L][1][r] = zr[L][0][r];
                    }
                }
            }
            __syncthreads();
        }
    }
}

// r' = r - alpha q, ||r'||^2, z = Chebyshev(r') in S levels (ChebPairs), r'.z.
template <int TMAX, int S, int FORM, bool FIRST>
__device__ __forceinline__ void plane_b(const PlaneArgsB& a, int blk, int nblk)
{
    __shared__ double sm[64];
    const Geo& g = a.g;
    const PlaneMap& m = a.m;
    const TilePos t = tile_pos<S>(g, m, blk);
    const unsigned si = 4u * (unsigned)g.si;
    const int is = max(0, t.i0 - S);
    Vec vr[PR], vq[PR];
    auto fetch = [&](int P) {   // planes past the outlet read the outlet plane (weight 0)
        const unsigned at = (unsigned)min(P, g.nx - 1) * si;
#pragma unroll
        for (int r = 0; r < PR; ++r) {
            vr[r] = ldv(a.r_in, at + t.off[r]);
            if (!FIRST) vq[r] = ldv(a.q, at + t.off[r]);
        }
    };
    dep_wait();
    fetch(is);   // on its way while the head sums
    float alpha = 0.f;
    if (!FIRST) {   // pass A's sum, alpha and the commit of the iteration
        const HeadOut h = plane_head_b(a.df.pin, a.df.nb_in, a.st, a.outer, blk);
        if (h.end) return;
        alpha = h.coef;
    } else if (a.st->done) {
        return;
    }
    Acc arr, arz;
    {   // the first step reads the other buffer: finite values that reach no owned cell
        constexpr int BUF = TMAX * PR * plane_sp(S);
        const int n = m.groups * PR * m.lk * plane_sp(S);
        for (int q = threadIdx.x; q < n; q += blockDim.x) plane_sm[BUF + q] = make_float4(0.f, 0.f, 0.f, 0.f);
        __syncthreads();
    }
    if (is == 0 || t.i1 + S > g.nx - 2)
        march_b<TMAX, S, FORM, FIRST, true>(a, t, alpha, is, si, vr, vq, fetch, arr, arz);
    else
        march_b<TMAX, S, FORM, FIRST, false>(a, t, alpha, is, si, vr, vq, fetch, arr, arz);
    dep_signal();
    Acc v[2] = {arr, arz};
    put_partials<2>(v, reinterpret_cast<float2*>(sm), a.df.pout, blk, nblk);
}

// Jacobi: r' = r - alpha q, z = r' / A_c; no stencil, so no tile: the vectors
// of all planes, a grid-strided loop.
template <bool FIRST>
__device__ __forceinline__ void plane_b0(const PlaneArgsB& a, int blk, int nblk)
{
    __shared__ double sm[64];
    const Geo& g = a.g;
    dep_wait();
    float alpha = 0.f;
    if (!FIRST) {
        const HeadOut h = plane_head_b(a.df.pin, a.df.nb_in, a.st, a.outer, blk);
        if (h.end) return;
        alpha = h.coef;
    } else if (a.st->done) {
        return;
    }
    const int n = g.nx * (g.si / PV), ident = (g.nx - 1) * (g.si / PV);   // identity rows from there
    Acc arr, arz;
    for (int id = blk * blockDim.x + threadIdx.x; id < n; id += nblk * blockDim.x) {
        const Vec r = vec(a.r_in[id]);
        const float d = id >= ident ? 1.f : a.inv_c0;
        const Vec rv = FIRST ? r : vfma(-alpha, vec(a.q[id]), r), zv = vmul(d, rv);
        a.r_out[id] = f4(rv);
        a.z_out[id] = f4(zv);
        acc_add(arr, vdot(rv, rv));
        acc_add(arz, vdot(rv, zv));
    }
    dep_signal();
    Acc v[2] = {arr, arz};
    put_partials<2>(v, reinterpret_cast<float2*>(sm), a.df.pout, blk, nblk);
}

template <int FORM, bool FIRST>
__global__ void __launch_bounds__(plane_threads_a(), 1) k_plane_a(const __grid_constant__ PlaneArgsA a)
{
    plane_a<plane_threads_a(), FORM, FIRST>(a, blockIdx.x, gridDim.x);
}

template <int S, int FORM, bool FIRST>
__global__ void __launch_bounds__(plane_threads_b(S), 1) k_plane_b(const __grid_constant__ PlaneArgsB a)
{
    plane_b<plane_threads_b(S), S, FORM, FIRST>(a, blockIdx.x, gridDim.x);
}

template <int S>
KPB plane_pick_b_s(int form, bool first)
{
    switch (form) {
    case 0: return first ? k_plane_b<S, 0, true> : k_plane_b<S, 0, false>;
    case 1: return first ? k_plane_b<S, 1, true> : k_plane_b<S, 1, false>;
    default: return first ? k_plane_b<S, 2, true> : k_plane_b<S, 2, false>;
    }
}

}  // namespace
