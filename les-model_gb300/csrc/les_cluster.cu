// les_cluster.cu -- the FP32 inner solve of a small grid (the iteration of
// les_col.cu) in one launch of one thread-block cluster.
//
// On a small grid the two passes of an iteration are a few microseconds of
// launches, grid sums and march latency around very little work.  Here the
// whole solve stays in the shared memory of the 16 blocks of one cluster, each
// with a range of planes and one plane of every vector beyond either end;
// blocks exchange end planes and partial sums by stores to each other's shared
// memory, and the cluster's hardware barrier orders an iteration in 1 + S
// steps (S Chebyshev levels):
//     beta, p = z + beta p, e += alpha_prev p_old, q = A p, p.q      barrier
//     alpha, r' = r - alpha q, levels 1 .. S of z = M^-1 r', a barrier each;
//     the last with ||r'||^2 and r'.z
// p and r' of the planes beyond the ends are updated by both blocks (from the
// exchanged z and q).  Every cell's arithmetic is that of the plane marches
// (les_plane.cuh); the sums differ by reassociation.
//
// Microseconds per inner iteration, plane marches -> cluster (GB300, degree 4):
//     16x32x32 10.0 -> 3.8    64x32x32 10.3 -> 5.3
//     48x48x32 10.6 -> 6.4    60x40x40 12.1 -> 8.7
// (Jacobi at 64x32x32 7.4 -> 3.4, degree 7 16.8 -> 8.3).
// What bounds it: a barrier with the stores before it takes 0.35 us (the
// smallest grids: 0.4 us per level); at 64x32x32 a level takes 0.85 us, half of
// it shared-memory reads of the neighbours' cells.
#include "les_plane.cuh"

#include <algorithm>

namespace les {

struct ClusterArgs {
    int nx, ny, nz;
    int pv, ncol;       // vectors per row, per plane
    int vmax;           // most planes of a block
    int groups, per;    // thread groups that share a block's planes, planes of each
    Coef k;
    ChebPairs c3;
    float inv_c0;
    const float4* r;
    float4 *p, *e;
    SolverState *st, *outer;
    int total_cap;
};

}  // namespace les

namespace {

constexpr int NB = 16;              // blocks of the cluster (more than 8 is opt-in)
constexpr int CL_THREADS = 640;     // most threads of a block
constexpr int CL_WARPS = CL_THREADS / 32;
constexpr size_t CL_SMEM = 225 * 1024;

__device__ __forceinline__ unsigned smem_addr(const void* p) { return (unsigned)__cvta_generic_to_shared(p); }
// the same place in block `rank` of the cluster
__device__ __forceinline__ unsigned peer_addr(unsigned a, int rank)
{
    unsigned r;
    asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(rank));
    return r;
}
__device__ __forceinline__ void peer_store(unsigned a, const float4& v)
{
    asm volatile("st.shared::cluster.v4.f32 [%0], {%1, %2, %3, %4};" ::"r"(a), "f"(v.x), "f"(v.y), "f"(v.z), "f"(v.w)
                 : "memory");
}
// orders all shared-memory stores of the cluster before all loads after it
__device__ __forceinline__ void cluster_barrier()
{
    __syncwarp();
    asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
    asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
}

// a + b of pairs, not renormalised: the high part is ready after one addition
// and the rounding errors gather in the low part (a tree of a few levels)
__device__ __forceinline__ Acc pair_add(const Acc& a, const Acc& b)
{
    const float s = __fadd_rn(a.hi, b.hi), bp = __fsub_rn(s, a.hi);
    const float err = __fadd_rn(__fsub_rn(a.hi, __fsub_rn(s, bp)), __fsub_rn(b.hi, bp));
    return Acc{s, __fadd_rn(__fadd_rn(a.lo, b.lo), err)};
}
// the sum of the pairs of N neighbouring lanes, in each of them
template <int N>
__device__ __forceinline__ void lane_sum(Acc& v)
{
#pragma unroll
    for (int o = N / 2; o > 0; o >>= 1) {
        Acc t;
        t.hi = __shfl_xor_sync(FULL, v.hi, o);
        t.lo = __shfl_xor_sync(FULL, v.lo, o);
        v = pair_add(v, t);
    }
}

// PER > 0: a thread's PER planes of every vector also stay in registers, and
// shared memory is read for other threads' cells only; 0: any number of planes,
// all in shared memory.
template <int S, int PER>
struct ClusterSolve {
    static constexpr int N = PER > 0 ? PER : 1;
    const ClusterArgs& a;
    float4 *R, *P, *Q, *Z[2], *E;
    float4 *part[2], *warp_part;   // blocks' sums: p.q; ||r'||^2 and r'.z; this block's warps' sums
    int rank, g0, np;          // this block's first plane and number of planes
    int np_lo;                 // planes of the block before
    int nw;
    int i0, i1;                // this thread's planes (relative to g0)
    int col, up, dn;           // its column of vectors, the rows above and below
    bool halo_lo, halo_hi;     // it also updates p and r' of the planes beyond the ends
    TilePos t;
    Acc s0, s1;
    Vec rr[N], pp[N], qq[N], ee[N], zz[2][N];

    __device__ ClusterSolve(const ClusterArgs& args, float4* sm) : a(args)
    {
        const int plane = (a.vmax + 2) * a.ncol;
        R = sm;
        P = R + plane;
        Q = P + plane;
        Z[0] = Q + plane;
        Z[1] = Z[0] + plane;
        E = Z[1] + plane;
        part[0] = E + a.vmax * a.ncol;
        part[1] = part[0] + NB;
        warp_part = part[1] + NB;
        rank = blockIdx.x;
        g0 = first(rank);
        np = first(rank + 1) - g0;
        np_lo = rank ? g0 - first(rank - 1) : 0;
        nw = blockDim.x >> 5;
        const int seg = threadIdx.x / a.ncol;
        const bool idle = seg >= a.groups;
        col = idle ? 0 : threadIdx.x - seg * a.ncol;
        const int j = col / a.pv, l = col - j * a.pv, k = PV * l, lane = threadIdx.x & 31;
        i0 = idle ? 0 : min(np, seg * a.per);
        i1 = idle ? 0 : min(np, i0 + a.per);
        halo_lo = !idle && seg == 0;
        halo_hi = !idle && seg == a.groups - 1;
        up = (j == 0 ? 1 : j - 1) * a.pv + l;
        dn = (j == a.ny - 1 ? a.ny - 2 : j + 1) * a.pv + l;
        t.left_wall = k == 0;
        t.last = (k <= a.nz - 1 && a.nz - 1 < k + PV) ? a.nz - 1 - k : -1;
        t.fix_l = !idle && lane == 0 && l > 0;
        t.fix_r = !idle && lane == 31 && l < a.pv - 1;
    }
    __device__ int first(int b) const { return a.nx * b / NB; }

    // vector of plane i (-1 and np: beyond the ends) of this thread's column
    __device__ float4* at(float4* v, int i) const { return v + (i + 1) * a.ncol + col; }

    __device__ int count() const { return PER > 0 ? PER : a.per; }
    // plane i0 + n of one of this thread's vectors
    __device__ Vec get(const Vec (&own)[N], float4* v, int n) const { return PER > 0 ? own[n] : vec(*at(v, min(i0 + n, np - 1))); }
    __device__ void put(Vec (&own)[N], float4* v, int n, const Vec& x) const
    {
        if (PER > 0) own[n] = x;
        if (i0 + n < i1) *at(v, i0 + n) = f4(x);
    }

    // stores a vector of plane i here, and in the neighbour whose end it is
    __device__ void publish(float4* v, int i, const Vec& x) const
    {
        float4* const own = at(v, i);
        *own = f4(x);
        if (i == 0 && rank > 0) peer_store(peer_addr(smem_addr(v + (np_lo + 1) * a.ncol + col), rank - 1), f4(x));
        if (i == np - 1 && rank < NB - 1) peer_store(peer_addr(smem_addr(v + col), rank + 1), f4(x));
    }

    // This block's sums to every block: a few remote stores (sixteen from each
    // warp crowd the network between the blocks: 7.65 -> 6.50 us per iteration
    // at 64x32x32)
    __device__ void put_sums(int which)
    {
        const int lane = threadIdx.x & 31;
        lane_sum<32>(s0);
        if (which == 1) lane_sum<32>(s1);
        if (lane == 0) warp_part[threadIdx.x >> 5] = make_float4(s0.hi, s0.lo, s1.hi, s1.lo);
        __syncthreads();
        if (threadIdx.x < 32) {
            const float4 x = lane < nw ? warp_part[lane] : make_float4(0.f, 0.f, 0.f, 0.f);
            s0 = Acc{x.x, x.y};
            s1 = Acc{x.z, x.w};
            lane_sum<PER == 2 ? 16 : 32>(s0);   // PER = 2: at most 16 warps
            if (which == 1) lane_sum<PER == 2 ? 16 : 32>(s1);
            if (lane < NB) peer_store(peer_addr(smem_addr(part[which] + rank), lane), make_float4(s0.hi, s0.lo, s1.hi, s1.lo));
        }
    }
    // the totals, in the same order in every warp
    __device__ void get_sums(int which)
    {
        const float4 x = part[which][threadIdx.x & (NB - 1)];
        s0 = Acc{x.x, x.y};
        s1 = Acc{x.z, x.w};
        lane_sum<NB>(s0);
        if (which == 1) lane_sum<NB>(s1);
    }

    // Calls f(n, mine, i, west, centre, east, js, ks) for this thread's planes of
    // the stencil of v; every thread of the block makes as many calls (shuffles),
    // those past its planes on some plane of the block.
    template <class F>
    __device__ void stencil(const Vec (&own)[N], float4* v, F f)
    {
        Vec w = vec(*at(v, i0 - 1)), c = PER > 0 ? own[0] : vec(*at(v, min(i0, np)));
#pragma unroll(PER > 0 ? PER : 1)
        for (int n = 0; n < count(); ++n) {
            const int i = min(i0 + n, np - 1);
            Vec e;
            if (PER > 0 && n + 1 < PER && i0 + n + 1 < i1) e = own[n + 1 < N ? n + 1 : 0];
            else e = vec(*at(v, i + 1));
            float4* const row = v + (i + 1) * a.ncol;
            const Vec js = vadd(vec(row[up]), vec(row[dn]));
            const Vec ks = k_sum<2, 1>(c, t, row + col);
            f(n, i0 + n < i1, i, w, c, e, js, ks);
            w = c;
            c = e;
        }
    }

    // z = M^-1 r' and r'.z; barriers after the levels 1 .. S-1
    template <bool EDGE>
    __device__ void levels()
    {
#pragma unroll
        for (int LV = 1; LV <= S; ++LV) {
            float4 *const src = LV == 1 ? R : Z[(LV - 1) & 1], *const dst = Z[LV & 1];
            const ChebPairs& c3 = a.c3;
            stencil(LV == 1 ? rr : zz[(LV - 1) & 1], src,
                    [&](int n, bool mine, int i, const Vec& w, const Vec& c, const Vec& e, const Vec& js, const Vec& ks) {
                const int g = g0 + i;
                const bool ident = EDGE && g == a.nx - 1;
                const float2 none = make_float2(0.f, 0.f), one = make_float2(1.f, 1.f);
                const float2 wc = ident ? c3.ci[LV - 1] : c3.cc[LV - 1];
                const float2 ww = EDGE && (ident || g == 0) ? none : one;
                const float2 we = EDGE && (ident || g == a.nx - 2) ? none : (EDGE && g == 0 ? make_float2(2.f, 2.f) : one);
                const float2 wy = ident ? none : c3.wy, wz = ident ? none : c3.wz;
                Vec v = EDGE ? vfma(we, e, vmul(ww, w)) : vadd(e, w);
                v = vfma(wz, ks, vfma(wy, js, vfma(wc, c, v)));
                const Vec rc = LV == 1 ? c : get(rr, R, n);
                if (LV >= 2) v = vfma(c3.rr[LV - 1], rc, v);
                if (LV >= 3) v = vfma(c3.gg[LV - 1], get(zz[LV & 1], dst, n), v);   // z_{LV-2} is replaced
                if (LV == S) {
                    v = vmul(c3.zs, v);
                    zero_pads<2>(v, t);
                }
                if (PER > 0) zz[LV & 1][n] = v;
                if (mine) {
                    publish(dst, i, v);
                    if (LV == S) acc_add(s1, vdot(rc, v));
                }
            });
            if (LV < S) cluster_barrier();
        }
    }

    // r' = r - alpha q with ||r'||^2 (Jacobi: and z, r'.z), then the levels
    template <bool EDGE>
    __device__ void residual_and_z(float alpha)
    {
        s0 = s1 = Acc{};
        auto diag = [&](int i) { return g0 + i == a.nx - 1 ? 1.f : a.inv_c0; };
#pragma unroll(PER > 0 ? PER : 1)
        for (int n = 0; n < count(); ++n) {
            const Vec rv = vfma(-alpha, get(qq, Q, n), get(rr, R, n));
            put(rr, R, n, rv);
            const Vec zv = vmul(diag(i0 + n), rv);
            if (S == 0) put(zz[0], Z[0], n, zv);
            if (i0 + n < i1) {
                acc_add(s0, vdot(rv, rv));
                if (S == 0) acc_add(s1, vdot(rv, zv));
            }
        }
        auto beyond = [&](int i) {
            const Vec rv = vfma(-alpha, vec(*at(Q, i)), vec(*at(R, i)));
            *at(R, i) = f4(rv);
            if (S == 0) *at(Z[0], i) = f4(vmul(diag(i), rv));
        };
        if (halo_lo) beyond(-1);
        if (halo_hi) beyond(np);
        if (S > 0) {
            __syncthreads();
            levels<EDGE>();
        }
        put_sums(1);
        cluster_barrier();
        get_sums(1);
    }

    template <bool EDGE>
    __device__ void run()
    {
        float4* const z = Z[S & 1];
        const double tol = a.st->tol;
        const int max_iter = a.st->max_iter, total0 = a.outer->iters;
        // r with the planes beyond the ends; everything else zero
        const int plane = (a.vmax + 2) * a.ncol;
        for (int q = threadIdx.x; q < plane * 4 + a.vmax * a.ncol; q += blockDim.x) P[q] = make_float4(0.f, 0.f, 0.f, 0.f);
        for (int q = threadIdx.x; q < plane; q += blockDim.x) {
            const int g = g0 - 1 + q / a.ncol;
            R[q] = g >= 0 && g < a.nx && g <= g0 + np ? a.r[(size_t)g * a.ncol + q % a.ncol] : make_float4(0.f, 0.f, 0.f, 0.f);
        }
#pragma unroll
        for (int n = 0; n < N; ++n) {
            pp[n] = qq[n] = ee[n] = zz[0][n] = zz[1][n] = vzero();
            rr[n] = vzero();
        }
        cluster_barrier();   // every block has started, and its vectors are set
        if (PER > 0)
#pragma unroll
            for (int n = 0; n < N; ++n)
                if (i0 + n < i1) rr[n] = vec(*at(R, i0 + n));
        residual_and_z<EDGE>(0.f);
        float alpha = 0.f;
        Acc rho;
        int k = 0, status = -1;
        double rr = 0.0;
        const float tol2 = (float)(1.0001 * tol * tol);
        for (;;) {
            // s0, s1: ||r'||^2, r'.z
            // the test on pairs' high parts while it is clear, else in FP64 (a
            // few FP64 operations in every warp: 6.50 -> 5.88 us at 64x32x32)
            if (k > 0) {
                if (!(s0.hi > tol2 && s0.hi < 3e38f)) {
                    rr = (double)s0.hi + (double)s0.lo;
                    if (rr < tol * tol) status = tol > 0.0 ? LES_OK : -1;
                    else if (!(rr < 1.7976931348623157e308)) status = LES_NONFINITE;
                }
                if (status < 0 && (k >= max_iter || total0 + k >= a.total_cap)) status = LES_NOT_CONVERGED;
                if (status >= 0) break;
            }
            const float beta = k ? df_quotient(s1, rho) : 0.f;
            rho = s1;
#pragma unroll(PER > 0 ? PER : 1)
            for (int n = 0; n < count(); ++n) {
                const Vec old = get(pp, P, n);
                put(pp, P, n, vfma(beta, old, get(zz[S & 1], z, n)));
                if (PER > 0) {
                    ee[n] = vfma(alpha, old, ee[n]);
                } else if (i0 + n < i1) {
                    float4* const e = E + (i0 + n) * a.ncol + col;
                    *e = f4(vfma(alpha, old, vec(*e)));
                }
            }
            if (halo_lo) *at(P, -1) = f4(vfma(beta, vec(*at(P, -1)), vec(*at(z, -1))));
            if (halo_hi) *at(P, np) = f4(vfma(beta, vec(*at(P, np)), vec(*at(z, np))));
            __syncthreads();
            s0 = s1 = Acc{};
            stencil(pp, P, [&](int n, bool mine, int i, const Vec& w, const Vec& c, const Vec& e, const Vec& js, const Vec& ks) {
                const int g = g0 + i;
                const bool ident = EDGE && g == a.nx - 1;
                const float cc = ident ? 1.f : a.k.c0, cy = ident ? 0.f : a.k.y1, cz = ident ? 0.f : a.k.z1;
                const float cw = EDGE && (ident || g == 0) ? 0.f : a.k.x1;
                const float ce = EDGE && (ident || g == a.nx - 2) ? 0.f : (EDGE && g == 0 ? 2.f * a.k.x1 : a.k.x1);
                Vec q = vfma(cz, ks, vfma(cy, js, vfma(ce, e, vfma(cw, w, vmul(cc, c)))));
                zero_pads<2>(q, t);
                if (PER > 0) qq[n] = q;
                if (mine) {
                    publish(Q, i, q);
                    acc_add(s0, vdot(c, q));
                }
            });
            put_sums(0);
            cluster_barrier();
            get_sums(0);
            alpha = df_quotient(rho, s0);
            ++k;
            residual_and_z<EDGE>(alpha);
        }
#pragma unroll(PER > 0 ? PER : 1)
        for (int n = 0; n < count(); ++n)
            if (i0 + n < i1) {
                const size_t id = (size_t)(g0 + i0 + n) * a.ncol + col;
                a.p[id] = f4(get(pp, P, n));
                a.e[id] = PER > 0 ? f4(ee[n]) : E[(i0 + n) * a.ncol + col];
            }
        if (rank == 0 && threadIdx.x == 0) {
            a.st->err = sqrt((double)s0.hi + (double)s0.lo);
            a.st->alpha = (double)alpha;
            a.st->k = k;
            a.st->buf = 0;
            a.st->status = status;
            a.st->done = 1;
            a.outer->iters = total0 + k;
        }
    }
};

// Threads of a block: those that leave a thread the registers of its planes.
constexpr int cl_threads(int per) { return per == 2 ? 512 : CL_THREADS; }

template <int S, int PER>
__global__ void __launch_bounds__(cl_threads(PER), 1) k_cluster_solve(const __grid_constant__ ClusterArgs a)
{
    if (a.st->done) return;   // in every block: this kernel sets it after its last barrier
    ClusterSolve<S, PER> c(a, plane_sm);
    // the inlet plane and the last two have weights of their own
    if (c.g0 == 0 || c.g0 + c.np >= a.nx - 1) c.template run<true>();
    else c.template run<false>();
}

using KCL = void (*)(ClusterArgs);

template <int PER>
KCL pick(int S)
{
    switch (S) {
    case 0: return k_cluster_solve<0, PER>;
    case 1: return k_cluster_solve<1, PER>;
    case 2: return k_cluster_solve<2, PER>;
    case 3: return k_cluster_solve<3, PER>;
    case 4: return k_cluster_solve<4, PER>;
    case 5: return k_cluster_solve<5, PER>;
    default: return k_cluster_solve<6, PER>;
    }
}

// How a block's planes are split: as few planes per thread as its threads
// allow, in registers up to two (degree 4 at 64x32x32 5.88 -> 5.29 us per
// iteration, 32x32x32 4.98 -> 4.55; four planes in the registers of 384
// threads lose: 48x48x32 6.16 -> 6.47).
struct Split {
    KCL k;
    int groups, per;
};

Split split_of(int vmax, int ncol, int S)
{
    auto with = [&](int threads) {
        const int groups = std::max(1, std::min(vmax, threads / ncol)), per = (vmax + groups - 1) / groups;
        return Split{nullptr, (vmax + per - 1) / per, per};
    };
    auto fits = [&](const Split& s, int per) { return s.per <= per && s.groups * ncol <= cl_threads(per); };
    Split s = with(cl_threads(1));
    if (fits(s, 1)) { s.k = pick<1>(S); return s; }
    s = with(cl_threads(2));
    if (fits(s, 2)) { s.k = pick<2>(S); return s; }
    s = with(CL_THREADS);
    s.k = pick<0>(S);
    return s;
}

size_t cluster_bytes(int vmax, int ncol)
{
    return sizeof(float4) * ((size_t)(6 * vmax + 10) * ncol + 2 * NB + CL_WARPS);
}

cudaLaunchConfig_t config(int threads, size_t smem, cudaStream_t s, cudaLaunchAttribute* at)
{
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = NB;
    cfg.blockDim = threads;
    cfg.dynamicSmemBytes = smem;
    cfg.stream = s;
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = NB;
    at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    return cfg;
}

}  // namespace

namespace les {

// The cluster serves the solves of the plane marches whose vectors fit its
// shared memory (up to about 100 000 cells) and whose planes fit a block's
// threads.  Not while kernels are timed one by one.
bool cluster_used(les_ctx* c, const les_pcg_opts* o, int S)
{
    const Geo& g = c->g;
    const int ncol = g.ny * (plane_pitch(g.nz) / PV), vmax = (g.nx + NB - 1) / NB;
    if (!plane_used(c, o) || c->prof_on) return false;
    if (g.nx < NB || ncol > CL_THREADS || cluster_bytes(vmax, ncol) > CL_SMEM) return false;
    const Split sp = split_of(vmax, ncol, S);
    const void* fn = (const void*)sp.k;
    cudaLaunchAttribute at[1];
    cudaLaunchConfig_t cfg = config((sp.groups * ncol + 31) / 32 * 32, cluster_bytes(vmax, ncol), c->stream, at);
    int n = 0;
    const bool ok = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)CL_SMEM) == cudaSuccess &&
                    cudaFuncSetAttribute(fn, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) == cudaSuccess &&
                    cudaOccupancyMaxActiveClusters(&n, fn, &cfg) == cudaSuccess && n > 0;
    if (!ok) cudaGetLastError();
    return ok;
}

les_status cluster_solve(les_ctx* c, const ColPlan& P)
{
    const Geo& g = c->g;
    ClusterArgs a{g.nx, g.ny, g.nz, plane_pitch(g.nz) / PV, g.ny * (plane_pitch(g.nz) / PV), (g.nx + NB - 1) / NB};
    const Split sp = split_of(a.vmax, a.ncol, P.S);
    a.groups = sp.groups;
    a.per = sp.per;
    a.k = Coef{P.A.k.c0, P.A.k.x1, P.A.k.y1, P.A.k.z1};
    a.c3 = cheb_pairs(P.c3, P.S);
    a.inv_c0 = P.inv_c0;
    a.r = reinterpret_cast<const float4*>(c->f[0]);
    a.p = reinterpret_cast<float4*>(c->f[2]);
    a.e = reinterpret_cast<float4*>(c->f[5]);
    a.st = P.in;
    a.outer = P.out;
    a.total_cap = P.cap;
    cudaLaunchAttribute at[1];
    const cudaLaunchConfig_t cfg =
        config((a.groups * a.ncol + 31) / 32 * 32, cluster_bytes(a.vmax, a.ncol), c->stream, at);
    les_status st = check_cuda(c, cudaLaunchKernelEx(&cfg, sp.k, a), "cluster solve");
    ++c->launches;
    return st;
}

}  // namespace les
