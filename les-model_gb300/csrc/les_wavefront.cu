// les_wavefront.cu -- the three lexicographically ordered loops of les-model
// src/pressure.cpp on the device: the IC(0) factorisation (:495-556), the
// IC forward/backward substitution (:442-482) and the GS-SOR sweep
// (:212-246).
//
// Each cell of these loops depends only on its (i-1), (j-1), (k-1)
// neighbours (the backward solve: on i+1, j+1, k+1), so any order that
// computes a cell after those neighbours performs exactly the same
// floating-point operations on exactly the same operand values as the serial
// lexicographic loop: the results are bit-identical to the reference.
//
// The substitution and the SOR sweep run as a pipelined wavefront with no
// grid barrier inside a sweep.  The (j, k) plane is cut into tiles of TJ rows
// by 32 columns; a block of TJ warps owns a tile and marches along i, warp w
// on the tile's row w and lane l on column l, working at block step tau on
// plane tau - l - w (lanes and warps skewed by one plane each).  So the k-1
// neighbour of a cell is the previous lane's result of the step before (a
// warp shuffle), the j-1 neighbour the previous warp's result of the step
// before (shared memory, one block barrier per step), and the i-1 neighbour
// the thread's own result of the step before.  The rows of a tile run on the
// SM's four sub-partitions at once: a single warp would push all of them
// through one sub-partition's FP64 unit.  Only a tile's first row and first
// lane need other tiles' values: the tile below in j and the tile before in
// k publish their progress (steps completed, one counter per tile, release
// store after a fence) every WB steps, and a block waits (acquire load,
// bounded by %globaltimer) for the progress its next WB steps need, then
// reads those neighbours through L2.  The backward solve mirrors every
// direction.  Tiles are handed out to the resident blocks in an order in
// which each tile's producers come first, so the waits always end.
// The IC factorisation (set-up, once) keeps the simpler form: hyperplanes
// i+j+k = s in order, one grid barrier between them.  Every wait is bounded
// (about 2 s); a wait that gives up sets an error flag, every warp leaves,
// and the host reports LES_TIMEOUT.  Compiled with -fmad=false.
#include <cmath>

#include "les_internal.cuh"

using namespace les;

namespace les {
les_status pressure_bcs_dev(les_ctx* c, double* p);
}

namespace {

struct Plane {
    int nx, ny, nz, si, sj;
};

__device__ __forceinline__ int gtid() { return blockIdx.x * blockDim.x + threadIdx.x; }
__device__ __forceinline__ int gthreads() { return gridDim.x * blockDim.x; }

// IC(0) factorisation, src/pressure.cpp:506-555, hyperplane by hyperplane.
// L arrays must be zero on entry (fresh matrix semantics).
__global__ void k_ic_build(Plane P, StencilView A, double* Lc, double* Lw, double* Ls, double* Lb,
                           GridSync gs)
{
    const double small_val = 1e-30;
    const int smax = P.nx + P.ny + P.nz - 3;
    const int njk = P.ny * P.nz;
    for (int s = 0; s <= smax; ++s) {
        for (int t = gtid(); t < njk; t += gthreads()) {
            int j = t / P.nz, k = t - j * P.nz;
            int i = s - j - k;
            if (i < 0 || i >= P.nx) continue;
            int id = i * P.si + j * P.sj + k;
            Coef7 a = A.at(id);
            double sum_sq = 0.0;
            if (i > 0) {
                double lc = __ldcg(Lc + id - P.si);
                if (fabs(lc) > small_val) { double l = a.w / lc; Lw[id] = l; sum_sq += l * l; }
            }
            if (j > 0) {
                double lc = __ldcg(Lc + id - P.sj);
                if (fabs(lc) > small_val) { double l = a.s / lc; Ls[id] = l; sum_sq += l * l; }
            }
            if (k > 0) {
                double lc = __ldcg(Lc + id - 1);
                if (fabs(lc) > small_val) { double l = a.b / lc; Lb[id] = l; sum_sq += l * l; }
            }
            double diag = a.c - sum_sq;
            Lc[id] = (diag <= small_val) ? 1.0 : sqrt(diag);
        }
        if (!grid_barrier(gs)) return;
    }
}

// ---- pipelined wavefront -----------------------------------------------------
#ifndef LES_WAVE_WB
#define LES_WAVE_WB 4
#endif
#ifndef LES_WAVE_TJ
#define LES_WAVE_TJ 4
#endif
#ifndef LES_WAVE_WD
#define LES_WAVE_WD 8
#endif
constexpr int WB = LES_WAVE_WB;        // steps between progress publications
constexpr int WAVE_TJ = LES_WAVE_TJ;   // rows per tile = warps per block (one per SM sub-partition)
constexpr int WT = 32 * WAVE_TJ;

struct Wave {
    int nx, ny, nz, si, sj;    // the swept box (interior for GS-SOR) and the strides
    int off;                   // index of the box's first cell
    int wj, wk, ntiles;        // tiles along j and k
    int steps;                 // marching steps of a tile: planes + 31 lane skews + TJ-1 row skews
    int* prog;                 // progress counter per tile
    int* err;                  // set by a wait that gives up
    int stall;                 // tile that withholds its progress (LES_OPT_TEST_STALL), or -1
};

__device__ __forceinline__ int ld_acquire(const int* p)
{
    int v;
    asm volatile("ld.acquire.gpu.global.s32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
}

__device__ __forceinline__ void st_release(int* p, int v)
{
    asm volatile("st.release.gpu.global.s32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}

// Waits until *p has reached target (wrap-safe); false once the wait gave up
// (~2 s) or another block raised the error flag.  seen: the last value read.
__device__ bool wait_progress(const int* p, int target, int* err, int& seen)
{
    if ((seen = ld_acquire(p)) - target >= 0) return true;
    const unsigned long long t0 = globaltimer_ns();
    unsigned spins = 0;
    for (;;) {
        if ((seen = ld_acquire(p)) - target >= 0) return true;
        if (*(volatile int*)err) return false;
        if ((++spins & 63u) == 0u && globaltimer_ns() - t0 > 2000000000ull) {
            atomicExch(err, 1);
            return false;
        }
        __nanosleep(32);
    }
}

// One counter that a lane of warp 0 watches for its block: before the steps
// up to tend, *p must have reached base + min(tend + ahead, steps).  A value
// seen earlier that already covers the target saves the read.
struct Watch {
    const int* p;   // nullptr: nothing to wait for
    int base, ahead, seen;
};

// Waits for every lane's counter (all lanes at once: a read costs an L2 round
// trip); false in every thread when a wait gave up.
__device__ __forceinline__ bool wait_steps(const Wave& W, Watch& w, int tend, int* flag)
{
    if (threadIdx.x < 32) {
        bool ok = true;
        if (w.p && tend + w.ahead > 0) {
            const int target = w.base + min(tend + w.ahead, W.steps);
            if (w.seen - target < 0) ok = wait_progress(w.p, target, W.err, w.seen);
        }
        ok = __all_sync(0xffffffffu, ok);
        if (threadIdx.x == 0) *flag = ok;
    }
    __syncthreads();
    return *flag != 0;
}

// Publishes `value` as the tile's progress; after a block barrier that follows
// every thread's stores (the release covers what the barrier ordered).
__device__ __forceinline__ void publish(int* p, int value)
{
    if (threadIdx.x == 0) st_release(p, value);
}

// Tile t's producers: DIR > 0 the tiles below in j (t-1) and before in k
// (t-wj); DIR < 0 the tiles above (t+1) and after (t+wj).
struct TileDeps {
    int dj, dk;
};

template <int DIR>
__device__ __forceinline__ TileDeps tile_deps(const Wave& W, int J, int K, int t)
{
    TileDeps d;
    if (DIR > 0) {
        d.dj = J > 0 ? t - 1 : -1;
        d.dk = K > 0 ? t - W.wj : -1;
    } else {
        d.dj = J < W.wj - 1 ? t + 1 : -1;
        d.dk = K < W.wk - 1 ? t + W.wj : -1;
    }
    return d;
}

// The producers' counters, lanes 0 and 1.  A tile's row next to this one is its
// row TJ-1 (skewed TJ-1 steps behind its row 0), so the j-producer must be
// TJ-1 steps ahead; the k-producer's far lane reaches a plane 31 steps after
// its near lane.
__device__ __forceinline__ Watch watch_producers(const int* prog, const TileDeps& d, int base)
{
    Watch w{nullptr, base, 0, base - (1 << 20)};
    if (threadIdx.x == 0 && d.dj >= 0) { w.p = prog + d.dj; w.ahead = WAVE_TJ - 1; }
    if (threadIdx.x == 1 && d.dk >= 0) { w.p = prog + d.dk; w.ahead = 31; }
    return w;
}

// ---- operand staging: every step's read-only (or not yet written) operands
// are copied into shared memory WD steps ahead with cp.async, so a step
// never waits on a global load; only the cross-tile neighbours (after the
// batch's wait) are read directly.
constexpr int WD = LES_WAVE_WD;   // steps staged ahead (a power of two)

template <int BYTES>
__device__ __forceinline__ void cp_async(void* smem, const void* gmem)
{
    const unsigned s = (unsigned)__cvta_generic_to_shared(smem);
    asm volatile("cp.async.ca.shared.global [%0], [%1], %2;" ::"r"(s), "l"(gmem), "n"(BYTES) : "memory");
}
__device__ __forceinline__ void cp_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }

// A tile: rows jb.. of TJ rows (the last tile in j may have fewer) by the 32
// columns K*32..; warp w works on the tile's row w (in the sweep's order) and
// lane l on column K*32 + l.  At block step tau, warp w lane l works on plane
// tau - skew(l) - w (forward planes ascend, backward descend; skew(l) is l
// forward, 31-l backward), so:
//   the i-neighbour is the thread's own result of the step before,
//   the k-neighbour the previous lane's result of the step before (shuffle),
//   the j-neighbour the previous warp's result of the step before, handed
//   over in shared memory (double-buffered by step parity, one block barrier
//   per step); row 0 takes it from the tile before in j.
template <typename T>
struct IcStage {
    T v[WD][5][WAVE_TJ][32];   // rhs (forward r, backward the cell's forward result), Lw, Ls, Lb, Lc
    T xs[2][WAVE_TJ][32];      // each row's result of the last two steps
    int flag;
};

// IC(0) substitution of one tile, src/pressure.cpp:442-482.  DIR > 0: the
// forward solve L y = r (z = y); DIR < 0: the backward solve L^T z = y.
template <typename T, int DIR>
__device__ bool ic_tile(const Wave& W, int t, int base, const T* __restrict__ Lc, const T* __restrict__ Lw,
                        const T* __restrict__ Ls, const T* __restrict__ Lb, const T* __restrict__ r, T* z,
                        IcStage<T>& sg)
{
    constexpr unsigned FULL = 0xffffffffu;
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const int J = t % W.wj, K = t / W.wj;
    const int jb = J * WAVE_TJ, rows = min(WAVE_TJ, W.ny - jb);
    const int k = K * 32 + lane;
    const bool kin = k < W.nz;
    const int kc = min(k, W.nz - 1);                          // every address stays inside the grid
    const int sk = DIR > 0 ? lane : 31 - lane;
    const TileDeps d = tile_deps<DIR>(W, J, K, t);
    const bool wact = w < rows;                               // this warp's row exists
    // this warp's grid row (rows past the grid repeat the last one; dropped)
    const int jr = DIR > 0 ? jb + min(w, rows - 1) : jb + rows - 1 - min(w, rows - 1);
    const int rb = W.off + jr * W.sj + kc;
    const bool jin = DIR > 0 ? jr > 0 : jr < W.ny - 1;        // the row has its j-neighbour
    const bool kbn = DIR > 0 ? k > 0 : k < W.nz - 1;
    // row 0's neighbour row in the tile before, the near lane's neighbour column
    const int jn = DIR > 0 ? max(jb - 1, 0) : min(jb + rows, W.ny - 1);
    const int kn = DIR > 0 ? max(K * 32 - 1, 0) : min(K * 32 + 32, W.nz - 1);
    const int near = DIR > 0 ? 0 : 31;
    auto plane = [&](int tau, int skew) { return DIR > 0 ? tau - skew - w : W.nx - 1 - (tau - skew - w); };
    auto clampi = [&](int i) { return min(max(i, 0), W.nx - 1); };
    // the operands of step tau into slot tau % WD (one commit group per step);
    // the factors of a missing neighbour are read from the cell and not used
    auto stage = [&](int tau) {
        const int i = clampi(plane(tau, sk));
        const int sl = tau & (WD - 1);
        const int id = rb + i * W.si;
        const int ie = DIR > 0 ? 0 : (i < W.nx - 1 ? W.si : 0);
        const int je = DIR > 0 ? 0 : (jin ? W.sj : 0);
        const int ke = DIR > 0 ? 0 : (kbn ? 1 : 0);
        cp_async<sizeof(T)>(&sg.v[sl][0][w][lane], (DIR > 0 ? r : z) + id);
        cp_async<sizeof(T)>(&sg.v[sl][1][w][lane], Lw + id + ie);
        cp_async<sizeof(T)>(&sg.v[sl][2][w][lane], Ls + id + je);
        cp_async<sizeof(T)>(&sg.v[sl][3][w][lane], Lb + id + ke);
        cp_async<sizeof(T)>(&sg.v[sl][4][w][lane], Lc + id);
        cp_commit();
    };
    Watch watch = watch_producers(W.prog, d, base);
    T prev = T(0), outp = T(0);
    sg.xs[0][w][lane] = sg.xs[1][w][lane] = T(0);
#pragma unroll
    for (int q = 0; q < WD - 1; ++q) stage(q);
    for (int tau0 = 0; tau0 < W.steps; tau0 += WB) {
        const int tend = min(tau0 + WB, W.steps);
        if (!wait_steps(W, watch, tend, &sg.flag)) {
            cp_wait<0>();
            return false;
        }
        // the batch's cross-tile neighbours through L2 (clamped loads,
        // selected): row 0's j-neighbour for every step (own column), and the
        // k-neighbours of this warp's near lane (lane q holds step tau0 + q's)
        T zj[WB];
#pragma unroll
        for (int q = 0; q < WB; ++q) {
            const T v = __ldcg(z + W.off + clampi(plane(tau0 + q, sk)) * W.si + jn * W.sj + kc);
            zj[q] = d.dj >= 0 ? v : T(0);
        }
        T zk0;
        {
            const T v = __ldcg(z + W.off + clampi(plane(tau0 + (lane & (WB - 1)), 0)) * W.si + jr * W.sj + kn);
            zk0 = d.dk >= 0 ? v : T(0);
        }
#pragma unroll
        for (int q = 0; q < WB; ++q) {
            const int tau = tau0 + q;
            if (tau >= tend) break;   // block-uniform
            stage(tau + WD - 1);      // past the last step: clamped copies, never used
            cp_wait<WD - 1>();        // step tau's operands are in
            const int i = plane(tau, sk);
            const bool act = wact && kin && i >= 0 && i < W.nx;
            const int sl = tau & (WD - 1);
            const bool ib = DIR > 0 ? i > 0 : i < W.nx - 1;
            T zk = DIR > 0 ? __shfl_up_sync(FULL, outp, 1) : __shfl_down_sync(FULL, outp, 1);
            const T v0 = __shfl_sync(FULL, zk0, q);
            zk = lane == near ? v0 : zk;
            const T zjv = w == 0 ? zj[q] : sg.xs[(tau - 1) & 1][w - 1][lane];
            // :451-463 / :469-481, the terms in the reference's order
            T sum = sg.v[sl][0][w][lane];
            T a = sum - sg.v[sl][1][w][lane] * prev;
            sum = ib ? a : sum;
            a = sum - sg.v[sl][2][w][lane] * zjv;
            sum = jin ? a : sum;
            a = sum - sg.v[sl][3][w][lane] * zk;
            sum = kbn ? a : sum;
            const T out = sum / sg.v[sl][4][w][lane];
            if (act) z[rb + i * W.si] = out;
            prev = outp = out;
            sg.xs[tau & 1][w][lane] = out;
            __syncthreads();          // the next step reads this step's rows
        }
        if (t != W.stall) publish(W.prog + t, base + tend);   // block-uniform
    }
    cp_wait<0>();
    return true;
}

// apply_ic_preconditioner, src/pressure.cpp:442-482: the forward solve over
// all tiles, one grid barrier, the backward solve.  T = double is the
// reference's arithmetic; T = float serves the FP32 inner solve of the
// mixed-precision path (st == nullptr: never skipped).
template <typename T>
__global__ void __launch_bounds__(WT) k_ic_wave(Wave W, int base, const T* __restrict__ Lc, const T* __restrict__ Lw,
                                                const T* __restrict__ Ls, const T* __restrict__ Lb,
                                                const T* __restrict__ r, T* z, GridSync gs, const SolverState* st,
                                                int skip_done)
{
    if (skip_done && st && st->done) return;   // uniform across blocks: no barrier is entered
    __shared__ IcStage<T> sg;
    const int b = blockIdx.x, nb = gridDim.x;  // one tile per block at a time
    bool ok = true;
    for (int t = b; t < W.ntiles && ok; t += nb) ok = ic_tile<T, 1>(W, t, base, Lc, Lw, Ls, Lb, r, z, sg);
    if (!grid_barrier(gs) || !ok) return;
    for (int t = b; t < W.ntiles && ok; t += nb)
        ok = ic_tile<T, -1>(W, W.ntiles - 1 - t, base + W.steps + 1, Lc, Lw, Ls, Lb, r, z, sg);
}

// ---- GS-SOR, src/pressure.cpp:212-246 -------------------------------------------
// p = (1-omega) p + omega coef ((p_e + p_w)/dx2 + (p_n + p_s)/dy2 + (p_t + p_b)/dz2 - rhs)
// with the west, south and bottom neighbours already updated in this sweep
// and the east, north and top ones not yet; after each sweep
// apply_pressure_BCs and the test max|dp| < tol.
//
// Sweeps in flight.  A cell of sweep s needs, besides the new values of its
// west, south and bottom neighbours, only values of sweep s-1 one hyperplane
// ahead, so sweep s can follow sweep s-1 through the grid.  A block runs every
// Q-th sweep of its tile and Q blocks share a tile, each waiting for the
// progress of the one before on its own tile and on the tiles above, after
// and diagonal to it (watch_old), in addition to the producers of its own
// sweep.  One sweep at a time spends 700 of its 1000 steps filling and
// draining the wavefront with one warp per SM sub-partition (256x128x128: 1.18
// ms per sweep, FP64 pipe idle); in flight the sweeps keep several blocks on
// every SM busy.  256x128x128: 1180 -> 195 us per sweep (the FP64 pipe alone
// needs about 95); h = 1/161, 191x161x115: 2070 -> 370 us; 67x46x53: 570 -> 80.
//
// Boundary conditions inside a run of sweeps.  Faces: the value that
// apply_pressure_BCs leaves on the face next to an interior cell is that
// cell's own new value (0 at the outlet), so the cell's thread stores it.
// Obstacle: a solid cell with a fluid neighbour takes that neighbour's value
// after the sweep.  p keeps what the sweep computed (the sweep's own later
// cells read that), and the value the next sweep must see as the cell's old
// one goes to rep[sweep & 1], stored by the thread that computes the source
// cell; two buffers, because a source west, south or below of its cell is
// computed before the cell's old value is read.  A source's next-but-one value
// cannot overtake a reader: source and cell are neighbours, so the source's
// sweep s+2 waits for the cell's sweep s+1.  Which cells read rep (bit `planes`
// words `rd`) or store to it (`wr`, with directions in `fl`) is found once per
// solve (k_gs_flags).
//
// The test.  Sweeps run in batches of 1, 2, 4, ... 32; a batch records every
// sweep's max|dp|.  If one before the batch's last was below tol, the field is
// restored to the batch's start and exactly that many sweeps are run: the
// result is that of testing after every sweep.
//
// Layout.  The lanes of a warp work on 32 different planes at a time, so in the
// field's own layout every lane's 8 bytes lie in another sector (424 us per
// sweep at 256x128x128, bound by those accesses).  The solve therefore runs on
// skewed copies of p's interior and of the right-hand side: element (tile,
// step, warp, lane) holds the cell that this thread works on at that step.
// Every access of a step is then contiguous, and the old values of the east,
// north and top neighbours are the next step's own elements of the same
// thread, the next warp and the next lane: a step copies one new value per
// cell instead of four.  Faces stay in p.
struct Skew {
    int wj, steps;
    __device__ __forceinline__ size_t at(int i, int j, int k) const   // interior coordinates
    {
        const int l = k & 31, w = j % WAVE_TJ, t = (k >> 5) * wj + j / WAVE_TJ;
        return ((size_t)t * steps + (i + l + w)) * WT + w * 32 + l;
    }
};

struct GsArgs {
    Wave W;
    int Q, nb;                  // sweeps in flight, blocks per sweep
    DivBy dx, dy, dz;           // dx2, dy2, dz2
    double omega, coef, tol;
    int max_iter;
    double* p;                  // the field: its faces during the sweeps
    const double* rhs;          // skewed, like the next ones
    double* ps;                 // p's interior
    double* rep[2];
    size_t len;                 // elements of a skewed array
    double *ps_back, *face_back, *rep_back;
    const unsigned *rd, *wr;    // per column (j, k) of the grid and 32 planes: cells that read / store rep
    const uint8_t* fl;          // per cell: bits 0..5 directions to store to, bit 7 the cell's own old value is 0
    const int* solid_list;
    int n_solid;
    unsigned long long* gmax;   // max|dp| of each sweep of a batch (bit pattern)
    SolverState* st;
    GridSync gs;
    int nx, ny, nz;
};
constexpr int GS_BATCH = 32;    // most sweeps in a batch
constexpr int GS_MAX_FLIGHT = 8;
// FP64 operations of a cell: divisions by any d (19), products by powers of
// two joined to the sums (11), equal powers of two applied once (10) -- the
// same roundings.
enum GsForm { GS_DIV = 0, GS_POW2 = 1, GS_EQUAL = 2 };

// Copied WD steps ahead: the cells' old values and rhs, the row above the
// tile's last row and the column after its last lane.
struct GsStage {
    double own[WD][WAVE_TJ][32], rhs[WD][WAVE_TJ][32];
    double north[WD][32], top[WD][WAVE_TJ];
    double inlet[WAVE_TJ][32];      // the inlet face next to each column's first cell
    double xs[2][WAVE_TJ][32];      // each row's result of the last two steps
    int flag, flag0;
};

// The counters of sweep s-1, lanes 2 to 5: on this tile and the ones above,
// after and diagonal to it.  The copies of a step read old values of its own
// hyperplane and the next one, and the sources of solid cells there one more,
// so this tile's sweep s-1 must be two steps past the last copied one; the
// tile above reaches the same hyperplane TJ-1 of its own steps earlier (its
// first row), the tile after 31 (its first lane).
__device__ __forceinline__ void watch_old(Watch& w, const Wave& W, const int* prog, int J, int K, int t, int base)
{
    const bool n = J < W.wj - 1, top = K < W.wk - 1;
    const int q = threadIdx.x;
    if (q < 2 || q > 5) return;
    if ((q == 3 && !n) || (q == 4 && !top) || (q == 5 && !(n && top))) return;
    w.p = prog + t + (q == 3 || q == 5 ? 1 : 0) + (q == 4 || q == 5 ? W.wj : 0);
    w.base = base;
    w.ahead = WD - 1 + 3 - (q == 3 || q == 5 ? WAVE_TJ - 1 : 0) - (q == 4 || q == 5 ? 31 : 0);
    w.seen = base - (1 << 20);
}

// Sweep `s` of a batch over tile t, the solve's sweep number `num`.  base:
// progress value of this sweep's start (the one before: base - steps - 1).
template <int FORM>
__device__ bool gs_tile(const GsArgs& A, int t, int s, int num, int base, double one_m_omega, double omega_coef,
                        unsigned long long& maxr, GsStage& sg)
{
    constexpr unsigned FULL = 0xffffffffu;
    const Wave& W = A.W;
    int* const prog = W.prog + (s % A.Q) * W.ntiles;
    const int* const prog_old = W.prog + ((s + A.Q - 1) % A.Q) * W.ntiles;
    double* const p = A.p;
    const Skew sk{W.wj, W.steps};
    double* const rep_new = A.rep[num & 1];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const int J = t % W.wj, K = t / W.wj;
    const int jb = J * WAVE_TJ, rows = min(WAVE_TJ, W.ny - jb), kb = K * 32, cols = min(32, W.nz - kb);
    const TileDeps d = tile_deps<1>(W, J, K, t);
    const bool cell = w < rows && lane < cols;    // this thread has a column
    const int jr = jb + min(w, rows - 1), k = kb + min(lane, cols - 1);
    const int ssi = W.si, ssj = W.sj;
    const int rb = W.off + jr * ssj + k;          // (i = 0) in the field
    const bool last_row = w == rows - 1, last_col = lane == cols - 1;
    const bool wall_n = jr == W.ny - 1, wall_t = k == W.nz - 1;
    const size_t tile = (size_t)W.steps * WT;     // elements of a tile
    const size_t tb = t * tile + threadIdx.x;
    const size_t nb = (t + 1) * tile + lane, ob = (t + W.wj) * tile + w * 32;   // the tiles above and after
    // which old values lie in rep: bits of 32 planes of this column, the one
    // above and the one after
    const bool use_rep = num > 0 && A.n_solid > 0;
    const int col = (jr + 1) * A.nz + k + 1, ncol = A.ny * A.nz;
    const double* const rep_old = A.rep[(num & 1) ^ 1];
    unsigned ro = 0, rn = 0, rt = 0, wo = 0;
    int word = -1, wword = -1;
    auto stage = [&](int tau) {
        const int i = tau - lane - w, sl = tau & (WD - 1);
        if (i >= 0 && i < W.nx && cell) {
            const double *po = A.ps, *pn = A.ps, *pt = A.ps;
            if (use_rep) {
                const int gi = i + 1;   // grid plane
                if ((gi >> 5) != word) {
                    word = gi >> 5;
                    const unsigned* const c = A.rd + (size_t)word * ncol + col;
                    ro = __ldg(c);
                    rn = __ldg(c + A.nz);
                    rt = __ldg(c + 1);
                }
                if ((ro >> (gi & 31)) & 1u) po = rep_old;
                if ((rn >> (gi & 31)) & 1u) pn = rep_old;
                if ((rt >> (gi & 31)) & 1u) pt = rep_old;
            }
            const size_t at = tb + (size_t)tau * WT;
            cp_async<8>(&sg.own[sl][w][lane], po + at);
            cp_async<8>(&sg.rhs[sl][w][lane], A.rhs + at);
            if (last_row) cp_async<8>(&sg.north[sl][lane], wall_n ? p + rb + i * ssi + ssj : pn + nb + (size_t)(tau - w) * WT);
            if (last_col) cp_async<8>(&sg.top[sl][w], wall_t ? p + rb + i * ssi + 1 : pt + ob + (size_t)(tau - lane) * WT);
            if (i == 0) cp_async<8>(&sg.inlet[w][lane], p + rb - ssi);
        }
        cp_commit();
    };
    // the outlet face is 0 after every sweep
    const double outlet = num == 0 ? __ldcg(p + rb + W.nx * ssi) : 0.0;
    double prev = 0.0, outp = 0.0;
    sg.xs[0][w][lane] = sg.xs[1][w][lane] = 0.0;
    Watch watch = watch_producers(prog, d, base);
    if (s > 0) {
        watch_old(watch, W, prog_old, J, K, t, base - W.steps - 1);
        if (!wait_steps(W, watch, 0, &sg.flag0)) return false;
    }
#pragma unroll
    for (int q = 0; q < WD - 1; ++q) stage(q);
    cp_wait<WD - 3>();   // steps 0 and 1; the barrier of the first wait makes them visible
    for (int tau0 = 0; tau0 < W.steps; tau0 += WB) {
        const int tend = min(tau0 + WB, W.steps);
        if (!wait_steps(W, watch, tend, &sg.flag)) {
            cp_wait<0>();
            return false;
        }
        // new values of other tiles, through L2: the last row of the tile below
        // (or the wall's face) for every step of warp 0, and the last lane of
        // the tile before (lane q holds step tau0 + q's)
        double ps0[WB], pb0 = 0.0;
#pragma unroll
        for (int q = 0; q < WB; ++q) {
            const int i = tau0 + q - lane;
            ps0[q] = 0.0;
            if (w == 0 && cell && i >= 0 && i < W.nx)
                ps0[q] = __ldcg(d.dj >= 0 ? A.ps + (t - 1) * tile + (size_t)(tau0 + q + WAVE_TJ - 1) * WT + 32 * (WAVE_TJ - 1) + lane
                                          : p + rb + i * ssi - ssj);
        }
        {
            const int q = lane & (WB - 1), i = tau0 + q - w;
            if (w < rows && i >= 0 && i < W.nx)
                pb0 = __ldcg(d.dk >= 0 ? A.ps + (t - W.wj) * tile + (size_t)(tau0 + q + 31) * WT + w * 32 + 31
                                       : p + W.off + jr * ssj + i * ssi - 1);
        }
#pragma unroll
        for (int q = 0; q < WB; ++q) {
            const int tau = tau0 + q;
            if (tau >= tend) break;   // block-uniform
            stage(tau + WD - 1);
            const int i = tau - lane - w;
            const bool act = cell && i >= 0 && i < W.nx;
            const int sl = tau & (WD - 1), sn = (tau + 1) & (WD - 1);
            const double po = sg.own[sl][w][lane], rh = sg.rhs[sl][w][lane];
            const double pe = i == W.nx - 1 ? outlet : sg.own[sn][w][lane];
            const double pn = last_row ? sg.north[sl][lane] : sg.own[sn][min(w + 1, WAVE_TJ - 1)][lane];
            const double pt = last_col ? sg.top[sl][w] : sg.own[sn][w][min(lane + 1, 31)];
            const double pw = i == 0 ? sg.inlet[w][lane] : prev;
            double pb = __shfl_up_sync(FULL, outp, 1);
            const double v0 = __shfl_sync(FULL, pb0, q);
            pb = lane == 0 ? v0 : pb;
            const double ps = w == 0 ? ps0[q] : sg.xs[(tau - 1) & 1][w - 1][lane];
            const double ew = pe + pw, ns = pn + ps, tb2 = pt + pb;
            double x;
            if (FORM == GS_EQUAL) x = fma((ew + ns) + tb2, A.dx.y, -rh);
            else if (FORM == GS_POW2) x = fma(tb2, A.dz.y, fma(ns, A.dy.y, ew * A.dx.y)) - rh;
            else x = ((div_by(ew, A.dx) + div_by(ns, A.dy)) + div_by(tb2, A.dz)) - rh;
            const double v = one_m_omega * po + omega_coef * x;
            if (act) {
                A.ps[tb + (size_t)tau * WT] = v;
                // the faces next to this cell, src/pressure.cpp:14-72
                const int id = rb + i * ssi;
                if (i == 0) p[id - ssi] = v;
                if (i == W.nx - 1) p[id + ssi] = 0.0;
                if (jr == 0) p[id - ssj] = v;
                if (wall_n) p[id + ssj] = v;
                if (k == 0) p[id - 1] = v;
                if (wall_t) p[id + 1] = v;
                if (A.n_solid > 0) {
                    const int gi = i + 1;
                    if ((gi >> 5) != wword) {
                        wword = gi >> 5;
                        wo = __ldg(A.wr + (size_t)wword * ncol + col);
                    }
                    if ((wo >> (gi & 31)) & 1u) {   // the source of solid cells, or solid next to the outlet
                        const unsigned f = A.fl[id];
                        if (f & 1u) rep_new[sk.at(i + 1, jr, k)] = v;
                        if (f & 2u) rep_new[sk.at(i - 1, jr, k)] = v;
                        if (f & 4u) rep_new[sk.at(i, jr + 1, k)] = v;
                        if (f & 8u) rep_new[sk.at(i, jr - 1, k)] = v;
                        if (f & 16u) rep_new[sk.at(i, jr, k + 1)] = v;
                        if (f & 32u) rep_new[sk.at(i, jr, k - 1)] = v;
                        if (f & 128u) rep_new[sk.at(i, jr, k)] = 0.0;
                    }
                }
                // max over non-negative doubles by their bit patterns; NaN is not selected
                const unsigned long long r = (unsigned long long)__double_as_longlong(fabs(v - po));
                if (r > maxr && r <= 0x7ff0000000000000ull) maxr = r;
            }
            prev = outp = v;
            sg.xs[tau & 1][w][lane] = v;
            cp_wait<WD - 3>();        // steps tau + 1 and tau + 2 of this thread are in
            __syncthreads();          // the next step reads this step's rows and others' copies
        }
        if (t != W.stall) publish(prog + t, base + tend);   // block-uniform
    }
    cp_wait<0>();
    return true;
}

// Flags of the obstacle copy, src/pressure.cpp:73-92: a solid interior cell
// takes its first fluid neighbour's value, in the order +i, -i, +j, -j, +k, -k.
// If that neighbour is a face, the face next to the cell holds the cell's own
// value (nothing to do) or, at the outlet, 0.
__device__ __forceinline__ int first_fluid(const uint8_t* solid, int id, int si, int sj)
{
    if (!solid[id + si]) return 0;
    if (!solid[id - si]) return 1;
    if (!solid[id + sj]) return 2;
    if (!solid[id - sj]) return 3;
    if (!solid[id + 1]) return 4;
    if (!solid[id - 1]) return 5;
    return 6;
}

// One thread per column and word of 32 planes.
__global__ void k_gs_flags(int nx, int ny, int nz, const uint8_t* __restrict__ solid, unsigned* __restrict__ rd,
                           unsigned* __restrict__ wr, uint8_t* __restrict__ fl)
{
    const int si = ny * nz, sj = nz;
    const int col = blockIdx.x * blockDim.x + threadIdx.x, wi = blockIdx.y;
    if (col >= si) return;
    const int j = col / nz, k = col - j * nz;
    unsigned r = 0u, w = 0u;
    auto interior = [&](int i, int jj, int kk) {
        return i >= 1 && i <= nx - 2 && jj >= 1 && jj <= ny - 2 && kk >= 1 && kk <= nz - 2;
    };
    for (int b = 0; b < 32; ++b) {
        const int i = wi * 32 + b;
        if (i >= nx) break;
        const int id = i * si + col;
        unsigned f = 0u;
        if (interior(i, j, k)) {
            if (solid[id]) {
                const int q = first_fluid(solid, id, si, sj);
                const int di[7] = {1, -1, 0, 0, 0, 0, 0}, dj[7] = {0, 0, 1, -1, 0, 0, 0}, dk[7] = {0, 0, 0, 0, 1, -1, 0};
                if (q < 6) {
                    if (interior(i + di[q], j + dj[q], k + dk[q])) r |= 1u << b;
                    else if (q == 0) { r |= 1u << b; f = 128u; }   // the outlet face
                }
            } else {   // the solid neighbours this cell is the first fluid neighbour of
                if (interior(i + 1, j, k) && solid[id + si] && first_fluid(solid, id + si, si, sj) == 1) f |= 1u;
                if (interior(i - 1, j, k) && solid[id - si] && first_fluid(solid, id - si, si, sj) == 0) f |= 2u;
                if (interior(i, j + 1, k) && solid[id + sj] && first_fluid(solid, id + sj, si, sj) == 3) f |= 4u;
                if (interior(i, j - 1, k) && solid[id - sj] && first_fluid(solid, id - sj, si, sj) == 2) f |= 8u;
                if (interior(i, j, k + 1) && solid[id + 1] && first_fluid(solid, id + 1, si, sj) == 5) f |= 16u;
                if (interior(i, j, k - 1) && solid[id - 1] && first_fluid(solid, id - 1, si, sj) == 4) f |= 32u;
            }
        }
        if (f) w |= 1u << b;
        fl[id] = (uint8_t)f;
    }
    rd[(size_t)wi * si + col] = r;
    wr[(size_t)wi * si + col] = w;
}

// Skewed copies: p's interior and the right-hand side, src/pressure.cpp:197-210.
__global__ void k_gs_skew(Geo g, Skew sk, double coef, DivBy two_dx, DivBy two_dy, DivBy two_dz,
                          const double* __restrict__ u, const double* __restrict__ v, const double* __restrict__ w,
                          const double* __restrict__ p, double* __restrict__ ps, double* __restrict__ rhs)
{
    const int k = blockIdx.x * TBK + threadIdx.x, j = blockIdx.y * TBJ + threadIdx.y, i = blockIdx.z;
    if (i < 1 || i > g.nx - 2 || j < 1 || j > g.ny - 2 || k < 1 || k > g.nz - 2) return;
    const int id = i * g.si + j * g.sj + k;
    const size_t at = sk.at(i - 1, j - 1, k - 1);
    const double div = div_by(u[id + g.si] - u[id - g.si], two_dx) + div_by(v[id + g.sj] - v[id - g.sj], two_dy) +
                       div_by(w[id + 1] - w[id - 1], two_dz);
    ps[at] = p[id];
    rhs[at] = coef * div;
}

__global__ void k_gs_unskew(Geo g, Skew sk, const double* __restrict__ ps, double* __restrict__ p)
{
    const int k = blockIdx.x * TBK + threadIdx.x, j = blockIdx.y * TBJ + threadIdx.y, i = blockIdx.z;
    if (i < 1 || i > g.nx - 2 || j < 1 || j > g.ny - 2 || k < 1 || k > g.nz - 2) return;
    p[i * g.si + j * g.sj + k] = ps[sk.at(i - 1, j - 1, k - 1)];
}

// What a batch may have to go back to: p's interior and faces, and the old
// values of solid cells (rep of the sweep before the batch); to: into the
// backup, else from it.
__device__ void gs_backup(const GsArgs& A, int num, bool to, int gt, int gn)
{
    auto move = [&](double* x, double* b) {
        if (to) *b = __ldcg(x);
        else *x = *b;
    };
    for (size_t c = gt; c < A.len; c += gn) move(A.ps + c, A.ps_back + c);
    // the faces that sweeps read: next to the interior
    const int mi = A.nx - 2, mj = A.ny - 2, mk = A.nz - 2, si = A.ny * A.nz, sj = A.nz;
    const int fi = mj * mk, fj = mi * mk, fk = mi * mj;
    for (int q = gt; q < 2 * (fi + fj + fk); q += gn) {
        int e = q, id;
        if (e < 2 * fi) {
            const int h = e >= fi;
            e -= h * fi;
            id = (h ? A.nx - 1 : 0) * si + (1 + e / mk) * sj + 1 + e % mk;
        } else if ((e -= 2 * fi) < 2 * fj) {
            const int h = e >= fj;
            e -= h * fj;
            id = (1 + e / mk) * si + (h ? A.ny - 1 : 0) * sj + 1 + e % mk;
        } else {
            e -= 2 * fj;
            const int h = e >= fk;
            e -= h * fk;
            id = (1 + e / mj) * si + (1 + e % mj) * sj + (h ? A.nz - 1 : 0);
        }
        move(A.p + id, A.face_back + q);
    }
    if (num > 0) {
        const Skew sk{A.W.wj, A.W.steps};
        for (int q = gt; q < A.n_solid; q += gn) {
            const int id = A.solid_list[q], i = id / si, r = id - i * si, j = r / sj, k = r - j * sj;
            move(A.rep[(num & 1) ^ 1] + sk.at(i - 1, j - 1, k - 1), A.rep_back + q);
        }
    }
}

template <int FORM>
__global__ void __launch_bounds__(WT, FORM == GS_DIV ? 5 : 6) k_gs_wave(const __grid_constant__ GsArgs A, int base)
{
    __shared__ GsStage sg;
    __shared__ unsigned long long wmax[WAVE_TJ];
    const Wave& W = A.W;
    const int blk = blockIdx.x % A.nb, q0 = blockIdx.x / A.nb;   // this block's tiles and sweeps
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const int gt = blockIdx.x * WT + threadIdx.x, gn = gridDim.x * WT;
    const double one_m_omega = 1 - A.omega, omega_coef = A.omega * A.coef;
    int done = 0, run = 1, epoch = base;   // sweeps finished, sweeps of this batch, its first progress value
    bool converged = false, redo = false;
    while (done < A.max_iter && !converged) {
        if (!redo) {
            run = min(run, A.max_iter - done);
            if (run > 1) gs_backup(A, done, true, gt, gn);
        }
        if (gt < GS_BATCH) A.gmax[gt] = 0ull;
        if (!grid_barrier(A.gs)) return;
        bool ok = true;
        for (int s = q0; s < run && ok; s += A.Q) {
            unsigned long long maxr = 0ull;
            for (int t = blk; t < W.ntiles && ok; t += A.nb)
                ok = gs_tile<FORM>(A, t, s, done + s, epoch + s * (W.steps + 1), one_m_omega, omega_coef, maxr, sg);
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) {
                const unsigned long long x = __shfl_xor_sync(0xffffffffu, maxr, o);
                maxr = x > maxr ? x : maxr;
            }
            if (lane == 0) wmax[w] = maxr;
            __syncthreads();
            if (threadIdx.x == 0) {
                for (int q = 1; q < WAVE_TJ; ++q) maxr = wmax[q] > maxr ? wmax[q] : maxr;
                atomicMax(A.gmax + s, maxr);
            }
            __syncthreads();
        }
        if (!grid_barrier(A.gs) || !ok) return;
        epoch += GS_BATCH * (W.steps + 1);
        // the first sweep whose max|dp| is below tol (the same in every thread)
        int hit = run;
        for (int s = 0; s < run && hit == run; ++s)
            if (__longlong_as_double((long long)__ldcg(A.gmax + s)) < A.tol) hit = s;
        if (hit < run - 1) {   // before the batch's last: run that many again from its start
            run = hit + 1;
            redo = true;
            gs_backup(A, done, false, gt, gn);
        } else {
            done += run;
            converged = hit < run;
            redo = false;
            run = min(2 * run, GS_BATCH);
        }
        if (!grid_barrier(A.gs)) return;   // every thread has read gmax; restored values are in place
    }
    if (gt == 0) {
        A.st->iters = done;
        A.st->k = done;
        A.st->done = 1;
        A.st->status = converged ? LES_OK : LES_NOT_CONVERGED;
    }
}

Plane plane_of(const Geo& g) { return Plane{g.nx, g.ny, g.nz, g.si, g.sj}; }

les_status coop_launch(les_ctx* c, const void* fn, void** args, int* grid_out, int pid = -1)
{
    int per_sm = 0;
    les_status st = check_cuda(c, cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, fn, 256, 0), "occupancy");
    if (st) return st;
    if (per_sm < 1) return fail(c, LES_CUDA_ERROR, "wavefront kernel cannot be resident");
    int grid = c->sms;   // one block per SM: enough threads for the widest hyperplane
    if (grid_out) *grid_out = grid;
    // count and generation only: the error word stays set until the host reads it
    st = check_cuda(c, cudaMemsetAsync(c->gsync, 0, sizeof(unsigned) * 2, c->stream), "reset barrier");
    if (st) return st;
    cudaEvent_t e1 = nullptr;
    if (pid >= 0 && c->prof_on) prof_begin(c, pid, &e1);
    st = check_cuda(c, cudaLaunchCooperativeKernel(fn, dim3(grid), dim3(256), args, 0, c->stream),
                    "cooperative launch");
    ++c->launches;
    if (e1) cudaEventRecord(e1, c->stream);
    return st;
}

GridSync grid_sync(les_ctx* c, int grid)
{
    GridSync gs;
    gs.count = c->gsync + 0;
    gs.gen = c->gsync + 1;
    gs.error = (int*)(c->gsync + 2);
    gs.nblocks = (unsigned)grid;
    return gs;
}

les_status check_barrier(les_ctx* c)
{
    unsigned h[4];
    les_status st = check_cuda(c, cudaMemcpyAsync(h, c->gsync, sizeof(h), cudaMemcpyDeviceToHost, c->stream),
                               "read barrier");
    if (st) return st;
    st = check_cuda(c, cudaStreamSynchronize(c->stream), "sync");
    if (st) return st;
    if (h[2]) {
        st = check_cuda(c, cudaMemsetAsync(c->gsync + 2, 0, sizeof(unsigned), c->stream), "clear error");
        if (st) return st;
        return fail(c, LES_TIMEOUT, "a bounded wavefront wait timed out");
    }
    return LES_OK;
}

// The warp tiles of a pipelined sweep over the box [0,nx)x[0,ny)x[0,nz)
// starting at grid cell `off`, and the progress base of this launch: the
// launch uses progress values in (base, base + span]; the counters are only
// compared against later bases, so they need no reset between launches.
// sets: progress counters per tile (GS-SOR: one set per sweep in flight).
les_status wave_setup(les_ctx* c, int nx, int ny, int nz, int off, long long span, int sets, Wave& W, int& base)
{
    W.nx = nx;
    W.ny = ny;
    W.nz = nz;
    W.si = c->g.si;
    W.sj = c->g.sj;
    W.off = off;
    W.wj = (ny + WAVE_TJ - 1) / WAVE_TJ;
    W.wk = (nz + 31) / 32;
    W.ntiles = W.wj * W.wk;
    W.steps = nx + 31 + WAVE_TJ - 1;
    const int len = W.ntiles * sets;
    if (c->wave_prog_len < len) {
        cudaFree(c->wave_prog);
        c->wave_prog = nullptr;
        c->wave_prog_len = 0;
        les_status st = check_cuda(c, cudaMalloc(&c->wave_prog, sizeof(int) * (size_t)len), "cudaMalloc(wave)");
        if (st) return st;
        c->wave_prog_len = len;
        c->wave_epoch = 0;
        st = check_cuda(c, cudaMemsetAsync(c->wave_prog, 0, sizeof(int) * (size_t)len, c->stream), "memset");
        if (st) return st;
    }
    if (span < 0 || span > (1 << 29)) return fail(c, LES_BAD_ARG, "wavefront: too many sweeps in one launch");
    if (c->wave_epoch > (1 << 30) - (int)span) {   // restart the counters well before the int range ends
        les_status st = check_cuda(c, cudaMemsetAsync(c->wave_prog, 0, sizeof(int) * (size_t)c->wave_prog_len,
                                                      c->stream), "memset");
        if (st) return st;
        c->wave_epoch = 0;
    }
    base = c->wave_epoch;
    c->wave_epoch += (int)span + 1;
    W.prog = c->wave_prog;
    W.err = (int*)(c->gsync + 2);
    W.stall = c->test_stall ? 0 : -1;
    return LES_OK;
}

// Cooperative launch of a pipelined sweep: one tile per block at a time, as many blocks
// as tiles but no more than can be resident at once (the tiles are handed out
// in producer-first order, so any resident count finishes).
// grid: blocks, no more than wave_resident.
les_status wave_resident(les_ctx* c, const void* fn, int* blocks)
{
    int per_sm = 0;
    les_status st = check_cuda(c, cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, fn, WT, 0), "occupancy");
    if (st) return st;
    if (per_sm < 1) return fail(c, LES_CUDA_ERROR, "wavefront kernel cannot be resident");
    *blocks = per_sm * c->sms;
    return LES_OK;
}

les_status wave_launch(les_ctx* c, const void* fn, void** args, int grid, int pid)
{
    // count and generation only: the error word stays set until the host reads it
    les_status st = check_cuda(c, cudaMemsetAsync(c->gsync, 0, sizeof(unsigned) * 2, c->stream), "reset barrier");
    if (st) return st;
    cudaEvent_t e1 = nullptr;
    if (pid >= 0 && c->prof_on) prof_begin(c, pid, &e1);
    st = check_cuda(c, cudaLaunchCooperativeKernel(fn, dim3(grid), dim3(WT), args, 0, c->stream),
                    "cooperative launch");
    ++c->launches;
    if (e1) cudaEventRecord(e1, c->stream);
    return st;
}

}  // namespace

namespace les {

// LES_TIMEOUT (and the flag cleared) if a wavefront wait gave up since the last check.
les_status wave_check(les_ctx* c) { return check_barrier(c); }

les_status ic_apply_dev(les_ctx* c, const double* r, double* z, const double* const* Lsrc, int skip_done)
{
    const double* const* L = Lsrc ? Lsrc : (const double* const*)c->L;
    Wave W;
    int base = 0;
    les_status st = wave_setup(c, c->g.nx, c->g.ny, c->g.nz, 0, 2 * (c->g.nx + 32 + WAVE_TJ), 1, W, base);
    if (st) return st;
    const double *Lc = L[0], *Lw = L[4], *Ls = L[2], *Lb = L[6];
    const void* fn = (const void*)k_ic_wave<double>;
    int resident = 0;
    st = wave_resident(c, fn, &resident);
    if (st) return st;
    const int grid = W.ntiles < resident ? W.ntiles : resident;
    GridSync gs = grid_sync(c, grid);
    const SolverState* stp = c->state;
    int skip = skip_done;
    void* args[] = {&W, &base, (void*)&Lc, (void*)&Lw, (void*)&Ls, (void*)&Lb, (void*)&r, (void*)&z, &gs,
                    (void*)&stp, &skip};
    return wave_launch(c, fn, args, grid, PROF_IC);
}

les_status ic_apply_dev32(les_ctx* c, const float* r, float* z, const float* const* L, SolverState* st)
{
    Wave W;
    int base = 0;
    les_status s2 = wave_setup(c, c->g.nx, c->g.ny, c->g.nz, 0, 2 * (c->g.nx + 32 + WAVE_TJ), 1, W, base);
    if (s2) return s2;
    const float *Lc = L[0], *Lw = L[4], *Ls = L[2], *Lb = L[6];
    const void* fn = (const void*)k_ic_wave<float>;
    int resident = 0;
    s2 = wave_resident(c, fn, &resident);
    if (s2) return s2;
    const int grid = W.ntiles < resident ? W.ntiles : resident;
    GridSync gs = grid_sync(c, grid);
    const SolverState* stp = st;
    int skip = st ? 1 : 0;
    void* args[] = {&W, &base, (void*)&Lc, (void*)&Lw, (void*)&Ls, (void*)&Lb, (void*)&r, (void*)&z, &gs,
                    (void*)&stp, &skip};
    return wave_launch(c, fn, args, grid, PROF_IC);
}

les_status build_ic_dev(les_ctx* c)
{
    const size_t nb = sizeof(double) * (size_t)c->g.n;
    for (int q = 0; q < 7; ++q) {
        if (!c->L[q]) {
            les_status st = check_cuda(c, cudaMalloc(&c->L[q], nb), "cudaMalloc(L)");
            if (st) return st;
        }
        cudaMemsetAsync(c->L[q], 0, nb, c->stream);
    }
    Plane P = plane_of(c->g);
    StencilView A = stencil_view(c);
    GridSync gs = grid_sync(c, c->sms);
    double *Lc = c->L[0], *Lw = c->L[4], *Ls = c->L[2], *Lb = c->L[6];
    void* args[] = {&P, &A, &Lc, &Lw, &Ls, &Lb, &gs};
    les_status st = coop_launch(c, (const void*)k_ic_build, args, nullptr);
    if (st) return st;
    st = check_barrier(c);
    if (st) return st;
    c->have_L = true;
    return LES_OK;
}

les_status solve_gs_dev(les_ctx* c, double dt, double rho, int max_iter, double omega, double tol, int* sweeps)
{
    les_status st = ensure_work(c);
    if (st) return st;
    const les_mesh& m = c->mesh;
    const double dx2 = m.dx * m.dx, dy2 = m.dy * m.dy, dz2 = m.dz * m.dz;
    const double coef = 1.0 / (2.0 * (1.0 / dx2 + 1.0 / dy2 + 1.0 / dz2));
    const Geo& g = c->g;
    if (g.nx < 3 || g.ny < 3 || g.nz < 3) return fail(c, LES_BAD_ARG, "GS-SOR needs an interior");
    // x / d2 for a power of two d2 is exactly x * (1 / d2)
    auto pow2 = [](double v) { int e; return std::frexp(v, &e) == 0.5; };
    const bool p2 = pow2(dx2) && pow2(dy2) && pow2(dz2);
    const void* fn = !p2 ? (const void*)k_gs_wave<GS_DIV>
                         : (dx2 == dy2 && dy2 == dz2 ? (const void*)k_gs_wave<GS_EQUAL> : (const void*)k_gs_wave<GS_POW2>);
    int resident = 0;
    st = wave_resident(c, fn, &resident);
    if (st) return st;
    // Sweeps in flight: as many as there are resident blocks for, up to what a
    // sweep's length has room for (a sweep starts about 20 steps behind the
    // one before: the staging depth, the waits' granularity).
    const int ntiles = ((g.ny - 2 + WAVE_TJ - 1) / WAVE_TJ) * ((g.nz - 2 + 31) / 32);
    const int room = (g.nx - 2 + 31 + WAVE_TJ - 1) / 20 + 1;
    int Q = resident / ntiles;
    Q = Q < 1 ? 1 : (Q > room ? room : Q);
    if (Q > GS_MAX_FLIGHT) Q = GS_MAX_FLIGHT;
    if (Q > max_iter && max_iter > 0) Q = max_iter;
    GsArgs a{};
    int base = 0;
    // progress values: every batch (about max_iter / GS_BATCH and the doubling
    // ones before, one run again) takes GS_BATCH sweeps' worth
    const long long batches = max_iter / GS_BATCH + 8;
    st = wave_setup(c, g.nx - 2, g.ny - 2, g.nz - 2, g.si + g.sj + 1,
                    batches * GS_BATCH * (long long)(g.nx - 2 + 32 + WAVE_TJ), Q, a.W, base);
    if (st) return st;
    a.len = (size_t)a.W.ntiles * a.W.steps * WT;
    if (c->gs_len < 5 * a.len) {   // the skewed arrays, kept for the next solve
        cudaFree(c->gs_buf);
        c->gs_buf = nullptr;
        c->gs_len = 0;
        st = check_cuda(c, cudaMalloc(&c->gs_buf, sizeof(double) * 5 * a.len), "cudaMalloc(skewed sweeps)");
        if (st) return st;
        c->gs_len = 5 * a.len;
    }
    const int words = (g.nx + 31) / 32;
    a.Q = Q;
    a.nb = ntiles < resident ? ntiles : resident;
    a.dx = div_by_const(dx2);
    a.dy = div_by_const(dy2);
    a.dz = div_by_const(dz2);
    a.omega = omega;
    a.coef = coef;
    a.tol = tol;
    a.max_iter = max_iter;
    a.p = c->slot[LES_P];
    a.ps = c->gs_buf;
    double* const rhs = c->gs_buf + a.len;
    a.rhs = rhs;
    a.ps_back = c->gs_buf + 2 * a.len;
    a.rep[0] = c->gs_buf + 3 * a.len;
    a.rep[1] = c->gs_buf + 4 * a.len;
    a.face_back = c->w[0];
    a.rep_back = c->w[1];
    unsigned* const rd = reinterpret_cast<unsigned*>(c->w[2]);   // two words per column and 32 planes: n doubles hold them
    uint8_t* const fl = reinterpret_cast<uint8_t*>(c->w[3]);
    a.rd = rd;
    a.wr = rd + (size_t)words * g.si;
    a.fl = fl;
    a.solid_list = c->solid_list;
    a.n_solid = c->n_solid;
    a.gmax = reinterpret_cast<unsigned long long*>(c->partials);
    a.st = c->state;
    a.nx = g.nx;
    a.ny = g.ny;
    a.nz = g.nz;
    const int grid = a.nb * Q;
    a.gs = grid_sync(c, grid);
    const Skew sk{a.W.wj, a.W.steps};
    launch(c, k_gs_skew, cell_grid(g), cell_block(), g, sk, rho / dt, div_by_const(2 * m.dx), div_by_const(2 * m.dy),
           div_by_const(2 * m.dz), (const double*)c->slot[LES_U], (const double*)c->slot[LES_V],
           (const double*)c->slot[LES_W], (const double*)a.p, a.ps, rhs);
    if (c->n_solid)
        launch(c, k_gs_flags, dim3((g.si + 255) / 256, words), 256, g.nx, g.ny, g.nz, (const uint8_t*)c->mask, rd,
               rd + (size_t)words * g.si, fl);
    if ((st = check_launch(c, "gs set-up"))) return st;
    void* args[] = {&a, &base};
    if (max_iter > 0) {
        st = wave_launch(c, fn, args, grid, -1);
        if (st) return st;
        launch(c, k_gs_unskew, cell_grid(g), cell_block(), g, sk, (const double*)a.ps, a.p);
        if ((st = pressure_bcs_dev(c, a.p))) return st;   // of the last sweep
    }
    st = check_barrier(c);
    if (st) return st;
    st = read_state(c);
    if (st) return st;
    if (sweeps) *sweeps = max_iter > 0 ? c->h_state->iters : 0;
    return LES_OK;
}

}  // namespace les

extern "C" {

les_status les_build_ic(les_ctx* c)
{
    if (!c) return LES_BAD_ARG;
    if (!c->stencil_mode) return fail(c, LES_BAD_ARG, "no matrix: call les_build_stencil or les_set_stencil");
    cudaSetDevice(c->device);
    return build_ic_dev(c);
}

les_status les_solve_gs(les_ctx* c, double dt, double rho, int max_iter, double omega, double tol, int* sweeps)
{
    if (!c || max_iter < 0) return LES_BAD_ARG;
    cudaSetDevice(c->device);
    return solve_gs_dev(c, dt, rho, max_iter, omega, tol, sweeps);
}

}  // extern "C"
