// les_coop64.cu -- the FP64 PCG (src/pressure.cpp:342-414 and :762-835) of a
// small or medium grid in one cooperative launch.
//
// Launch by launch an iteration is three (Jacobi) to six (Chebyshev, degree 4)
// kernels of a few microseconds of work each, with a reduction tail, a launch
// gap and the host's own launch rate between them: 26 us per Jacobi iteration
// at 64x32x32, most of it waiting (the FP64 pipe needs 3).  Here the blocks stay resident, each with
// its own range of cells, and meet in an exchange where the iteration needs
// one: the two inner products, and wherever neighbours' values of a new vector
// are read.  The operations and their order are those of the kernels in
// les_pressure.cu; the sums differ by reassociation.  What is left at 64x32x32,
// 13 us: three exchanges of about 2.5 us (arrival, one poll, the partial sums),
// block sums and divisions on a pipe where a dependent operation takes 64
// cycles and more.  Compiled with -fmad=false.
#include "les_internal.cuh"

using namespace les;

namespace {

constexpr int MAX_STEPS = 31;  // Chebyshev steps after step 0

// The exchange of the blocks: an arrival counter that one thread of each block
// polls, and the blocks' partial sums, [parity][value][block].  Two parities
// suffice: a block stores to exchange e + 2 only after every block has arrived
// at e + 1, after reading e.  (Slots that carry a number beside the value, all
// polled by every block, save a round trip but crowd the few cache lines: 3 us
// until a block saw even its own.)
struct Meet {
    double* part;
    unsigned* count;
    int* err;
    unsigned arrive;   // 1; 0: this block never arrives (LES_OPT_TEST_STALL)
    unsigned nb, number;
};

// Sum over the block in thread 0: through shared memory to four warps (one
// per sub-partition), two or four values a lane, then a shuffle tree each: a
// warp's FP64 instruction holds its sub-partition's unit for about 64 cycles.
template <int NV, int CT>
__device__ __forceinline__ void block_total(double (&v)[NV], double (*sm)[CT])
{
    __shared__ double part[NV][4];
#pragma unroll
    for (int q = 0; q < NV; ++q) sm[q][threadIdx.x] = v[q];
    __syncthreads();
    if (threadIdx.x < 128) {
#pragma unroll
        for (int q = 0; q < NV; ++q) {
            v[q] = sm[q][threadIdx.x] + sm[q][threadIdx.x + 128];
            if (CT == 512) v[q] += sm[q][threadIdx.x + 256] + sm[q][threadIdx.x + 384];
        }
        warp_sum<NV>(v);
        if ((threadIdx.x & 31) == 0)
#pragma unroll
            for (int q = 0; q < NV; ++q) part[q][threadIdx.x >> 5] = v[q];
    }
    __syncthreads();
    if (threadIdx.x == 0)
#pragma unroll
        for (int q = 0; q < NV; ++q) v[q] = (part[q][0] + part[q][1]) + (part[q][2] + part[q][3]);
}

// Scalars that one thread forms for its block (a division in each of 16 warps
// would hold the FP64 pipe for over a microsecond)
struct Scalars {
    double a;
    int end;   // 0: go on, 1: the solve is done, 2: a wait gave up
};

// Sums v over all blocks in the same order and calls decide(totals, &out) in
// thread 0; out.end in every thread.  The blocks' stores before the exchange
// are visible to (L2) loads after it.  SUM = false: only that.  A wait that
// gives up (about 2 s) ends the solve in every block.
template <int NV, bool SUM = true, int CT, class F>
__device__ __forceinline__ int meet(Meet& m, double (&v)[NV], double (*sm)[CT], Scalars& out, F decide)
{
    if (SUM) block_total<NV, CT>(v, sm);   // a block barrier after the caller's stores
    else __syncthreads();
    const unsigned e = ++m.number;
    double* const s = m.part + (size_t)(e & 1u) * 2u * m.nb;
    int ok = 1;
    if (threadIdx.x == 0) {
        if (SUM)
#pragma unroll
            for (int q = 0; q < NV; ++q) __stcg(s + q * m.nb + blockIdx.x, v[q]);
        __threadfence();   // the block's stores before the arrival
        atomicAdd(m.count, m.arrive);
        const unsigned target = e * m.nb;
        unsigned spins = 0;
        unsigned long long t0 = 0;
        for (;;) {
            unsigned c;
            asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(c) : "l"(m.count) : "memory");
            if ((int)(c - target) >= 0) break;
            if ((++spins & 255u) == 0u) {   // bounded: about 2 s, or another block gave up
                const unsigned long long t = globaltimer_ns();
                if (t0 == 0) t0 = t;
                if (*(volatile int*)m.err || t - t0 > 2000000000ull) {
                    atomicExch(m.err, 1);
                    ok = 0;
                    break;
                }
            }
        }
    }
    ok = __syncthreads_and(ok);
    if (SUM) {
#pragma unroll
        for (int q = 0; q < NV; ++q) v[q] = threadIdx.x < m.nb ? __ldcg(s + q * m.nb + threadIdx.x) : 0.0;
        block_total<NV, CT>(v, sm);
    }
    if (threadIdx.x == 0) {
        out.end = ok ? 0 : 2;
        if (ok) decide(v, out);
    }
    __syncthreads();
    return out.end;
}

// A row of A through L2 (other blocks' values of this launch).  ld(id) loads a
// neighbour.  PLAIN: a device-built matrix without solid cells, where a neighbour
// outside the grid always has the multiplier 0, so its load is clamped instead of
// tested.  (A fluid cell between a wall and a solid cell has the multiplier 1 for
// the neighbour in the wall, src/pressure.cpp:663-696; the row leaves that
// neighbour out, :721-744.  With the tests, and the cell's place for them, an
// iteration at 128x64x64 takes 32.1 us instead of 30.3, Chebyshev degree 4 89.0
// instead of 85.4.)
template <bool PLAIN, bool POW2, class Load>
__device__ __forceinline__ double row(const StencilView& A, const Geo& g, int id, double c, Load ld)
{
    const Coef7 a = PLAIN ? decode(A.code[id], A.k) : A.at(id);
    double v = a.c * c;
    auto add = [&](double m, double x) { v = POW2 ? fma(m, x, v) : v + m * x; };
    if (PLAIN) {
        const int n = g.n - 1;
        add(a.w, ld(max(id - g.si, 0)));
        add(a.e, ld(min(id + g.si, n)));
        add(a.s, ld(max(id - g.sj, 0)));
        add(a.n, ld(min(id + g.sj, n)));
        add(a.b, ld(max(id - 1, 0)));
        add(a.t, ld(min(id + 1, n)));
        return v;
    }
    const int i = id / g.si, r = id - i * g.si, j = r / g.sj, k = r - j * g.sj;
    if (i > 0) add(a.w, ld(id - g.si));
    if (i < g.nx - 1) add(a.e, ld(id + g.si));
    if (j > 0) add(a.s, ld(id - g.sj));
    if (j < g.ny - 1) add(a.n, ld(id + g.sj));
    if (k > 0) add(a.b, ld(id - 1));
    if (k < g.nz - 1) add(a.t, ld(id + 1));
    return v;
}

struct Args {
    Geo g;
    StencilView A;
    double *x, *r, *p, *q, *z, *z2, *pc;   // pc: Chebyshev's own direction
    const double* b;
    SolverState* st;
    double* part;
    unsigned* count;
    int* err;
    int stall;
    double tol;
    int keep_tol, max_iter, degree;        // degree 0: Jacobi
    double alpha0, alpha[MAX_STEPS], beta[MAX_STEPS];   // Chebyshev's coefficients, :878-899
    DivBy by_c0;
};

template <int CT, bool PLAIN, bool POW2>
__global__ void __launch_bounds__(CT, 1) k_pcg64(const __grid_constant__ Args a)
{
    __shared__ double sm[2][CT];
    __shared__ Scalars sc;
    const Geo& g = a.g;
    Meet m{a.part, a.count, a.err, a.stall && blockIdx.x == 0 ? 0u : 1u, gridDim.x, 0};
    const int per = (g.n + (int)gridDim.x - 1) / (int)gridDim.x;
    const int c0 = (int)blockIdx.x * per + (int)threadIdx.x, c1 = min(g.n, ((int)blockIdx.x + 1) * per);
    const double tol = a.keep_tol ? a.st->tol : a.tol;
    const double far = tol * tol * (1.0 + 1e-12);   // sqrt(rr) > tol above it
    const int steps = a.degree - 1;
    double rho = 0.0;   // in thread 0
    auto each = [&](auto f) {
        for (int c = c0; c < c1; c += CT) f(c);
    };
    // ||r||^2 after k iterations: the test of src/pressure.cpp:355-359 and :386-392
    auto test = [&](int k, double rr, Scalars& o) {
        // far above the tolerance the root is not needed
        if (rr > far && rr < 1.7976931348623157e308 && k < a.max_iter) return;
        const double err = sqrt(rr);
        int status = -1, iters = k;
        if (err < tol) status = LES_OK;
        else if (!isfinite(err)) { status = LES_NONFINITE; iters = a.max_iter; }
        else if (k >= a.max_iter) { status = LES_NOT_CONVERGED; iters = a.max_iter; }
        if (status < 0) return;
        o.end = 1;
        if (blockIdx.x) return;
        a.st->tol = tol;
        a.st->max_iter = a.max_iter;
        a.st->k = k;
        a.st->iters = iters;
        a.st->status = status;
        a.st->err = err;
        a.st->rr = rr;
        a.st->buf = 0;
        a.st->done = 1;
    };
    // M^-1 r of the pointwise preconditioners (Jacobi, src/pressure.cpp:420-428;
    // Chebyshev's step 0), formed where r is
    auto point = [&](int c, double rv) {
        const double zv = a.degree == 0 ? (PLAIN || a.A.code ? (a.A.code[c] ? div_by(rv, a.by_c0) : rv) : rv / a.A.d[0][c])
                                        : fma(a.alpha0, rv, 0.0);
        if (steps <= 0) a.z[c] = zv;
        return zv;
    };
    // beta = rz / rho and rho = rz (:399-408); first: rho = rz
    auto set_beta = [&](double rz, bool first, Scalars& o) {
        o.a = first ? 0.0 : rz / rho;
        rho = rz;
    };
    // Chebyshev's steps 1.. (:888-905); the last exchange forms beta
    const double* zbuf = a.z;
    auto chebyshev = [&](bool first) {
        double alpha = a.alpha0;
        double *zi = a.z, *zo = a.z2;
        for (int q = 1; q <= steps; ++q) {
            const double beta = a.beta[q - 1];
            alpha = a.alpha[q - 1];
            double rz[1] = {0.0};
            each([&](int c) {
                const double rv = a.r[c];
                const double zc = q == 1 ? fma(a.alpha0, rv, 0.0) : zi[c];
                const double az = q == 1 ? row<PLAIN, POW2>(a.A, g, c, zc, [&](int id) { return fma(a.alpha0, __ldcg(a.r + id), 0.0); })
                                         : row<PLAIN, POW2>(a.A, g, c, zc, [&](int id) { return __ldcg(zi + id); });
                const double res = rv - az;
                const double pv = res + beta * (q == 1 ? rv : a.pc[c]);
                if (q < steps) a.pc[c] = pv;
                const double zv = zc + alpha * pv;
                zo[c] = zv;
                if (q == steps) rz[0] = fma(rv, zv, rz[0]);
            });
            double* const t = zi;
            zi = zo;
            zo = t;
            const int end = q < steps ? meet<1, false>(m, rz, sm, sc, [](double (&)[1], Scalars&) {})
                                      : meet<1>(m, rz, sm, sc,
                                                [&](double (&s)[1], Scalars& o) { set_beta(s[0], first, o); });
            if (end) return end;
        }
        zbuf = zi;
        return 0;
    };
    // r = b - A x, ||r||, z, rho, p = z
    double s2[2] = {0.0, 0.0}, s1[1] = {0.0};
    each([&](int c) {
        const double v = a.b[c] - row<PLAIN, POW2>(a.A, g, c, a.x[c], [&](int id) { return a.x[id]; });
        a.r[c] = v;
        s2[0] = fma(v, v, s2[0]);
        s2[1] = fma(v, point(c, v), s2[1]);
    });
    if (meet<2>(m, s2, sm, sc, [&](double (&s)[2], Scalars& o) {
            test(0, s[0], o);
            set_beta(s[1], true, o);
        }))
        return;
    if (steps > 0 && chebyshev(true)) return;
    each([&](int c) { a.p[c] = zbuf[c]; });
    for (int k = 1;; ++k) {
        if (meet<1, false>(m, s1, sm, sc, [](double (&)[1], Scalars&) {})) return;   // p is in place
        s1[0] = 0.0;
        each([&](int c) {
            const double pv = a.p[c];
            const double v = row<PLAIN, POW2>(a.A, g, c, pv, [&](int id) { return __ldcg(a.p + id); });
            a.q[c] = v;
            s1[0] = fma(pv, v, s1[0]);
        });
        if (meet<1>(m, s1, sm, sc, [&](double (&s)[1], Scalars& o) { o.a = rho / s[0]; })) return;   // :378
        const double alpha = sc.a;
        s2[0] = s2[1] = 0.0;
        each([&](int c) {
            a.x[c] += alpha * a.p[c];
            const double v = a.r[c] + (-alpha) * a.q[c];
            a.r[c] = v;
            s2[0] = fma(v, v, s2[0]);
            s2[1] = fma(v, point(c, v), s2[1]);
        });
        if (meet<2>(m, s2, sm, sc, [&](double (&s)[2], Scalars& o) {
                test(k, s[0], o);
                if (steps <= 0) set_beta(s[1], false, o);
            }))
            return;
        if (steps > 0 && chebyshev(false)) return;
        const double beta = sc.a;
        each([&](int c) { a.p[c] = zbuf[c] + beta * a.p[c]; });
    }
}

template <int CT>
const void* pick(bool plain, bool pow2)
{
    if (plain) return pow2 ? (const void*)k_pcg64<CT, true, true> : (const void*)k_pcg64<CT, true, false>;
    return pow2 ? (const void*)k_pcg64<CT, false, true> : (const void*)k_pcg64<CT, false, false>;
}

}  // namespace

namespace les {

// Cells up to which the cooperative form is taken.  Microseconds per iteration,
// launch by launch and cooperative (GB300), of Jacobi / Chebyshev degree 4:
//   64x32x32     26.5 / 13.2     48 / 28      90x90x90    70.3 / 48.2    164 / 149
//   80x80x80     60.3 / 37.4    133 / 111     100x100x100 93.3 / 62.2    228 / 196
//   128x128x64   71.0 / 51.4    157 / 153     degree 7 243 / 244
// (h = 0.01 but for the first and the last).  It was also ahead at 160x128x100,
// the largest timed (132 / 90, 330 / 284; h = 0.01 155 / 116, 420 / 387); the line
// stays at the size up to which every degree was.
// A spacing that is no power of two has rows of thirteen operations here and of
// eight to ten in the launched kernels, which come out ahead from degree 3 where
// their tiles of 8 x 32 cells fill the plane: 128x128x64, h = 0.01, degree 3 155 /
// 161, degree 7 303 / 336; 128x80x64 degree 3 117 / 106, degree 7 219 / 219.
constexpr long long COOP_CELLS = 1 << 20, COOP_CELLS_WHOLE = 5 << 17;

bool pcg64_coop_used(const les_ctx* c, const les_pcg_opts* o, bool pow2)
{
    const bool cheb = o->precond == LES_PC_CHEBYSHEV;
    if (!(o->precond == LES_PC_JACOBI || (cheb && o->degree >= 1 && o->degree <= MAX_STEPS + 1))) return false;
    const bool whole = c->stencil_mode == 1 && !pow2 && cheb && o->degree > 2 && c->g.ny % TBJ == 0 && c->g.nz % TBK == 0;
    return o->max_iter > 0 && !c->prof_on && c->g.n <= (whole ? COOP_CELLS_WHOLE : COOP_CELLS);
}

// The whole solve in one launch; the state is read back (and a wait that gave
// up reported) by the caller.
les_status pcg64_coop(les_ctx* c, const les_pcg_opts* o, bool pow2, int keep_tol)
{
    Args a{};
    a.g = c->g;
    a.A = stencil_view(c);
    a.x = c->slot[LES_P];
    a.b = c->slot[LES_B];
    a.r = c->w[0];
    a.z = c->w[1];
    a.p = c->w[2];
    a.q = c->w[3];
    a.z2 = c->w[6];
    a.pc = c->w[7];
    a.st = c->state;
    a.err = (int*)(c->gsync + 2);
    a.stall = c->test_stall;
    a.tol = o->tol;
    a.keep_tol = keep_tol;
    a.max_iter = o->max_iter;
    a.degree = o->precond == LES_PC_JACOBI ? 0 : o->degree;
    if (a.degree) {
        const double d = (o->lambda_max + o->lambda_min) / 2.0, cc = (o->lambda_max - o->lambda_min) / 2.0;
        double alpha = a.alpha0 = 2.0 / d;
        for (int q = 0; q < a.degree - 1; ++q) {
            a.beta[q] = (cc * alpha / 2.0) * (cc * alpha / 2.0);
            a.alpha[q] = alpha = 1.0 / (d - a.beta[q]);
        }
    }
    a.by_c0 = div_by_const(c->coef.c0);
    const bool plain = c->stencil_mode == 1 && c->code_plain;
    // fewer threads make the block sums cheaper, more hide the loads of more
    // cells; one block per SM at most, no more than give every fourth thread a cell
    const int threads = c->g.n <= 512 * c->sms ? 256 : 512;
    const void* fn = threads == 256 ? pick<256>(plain, pow2) : pick<512>(plain, pow2);
    int grid = (c->g.n + threads / 4 - 1) / (threads / 4);
    grid = grid < 1 ? 1 : (grid > c->sms ? c->sms : grid);
    if (grid > threads || (size_t)grid * 4 > c->partials_len) return fail(c, LES_BAD_ARG, "internal: exchange too small");
    a.part = c->partials;
    a.count = c->gsync;
    les_status st = check_cuda(c, cudaMemsetAsync(c->gsync, 0, sizeof(unsigned) * 2, c->stream), "reset exchange");
    if (st) return st;
    void* args[] = {&a};
    st = check_cuda(c, cudaLaunchCooperativeKernel(fn, dim3(grid), dim3(threads), args, 0, c->stream), "cooperative solve");
    ++c->launches;
    return st;
}

}  // namespace les
