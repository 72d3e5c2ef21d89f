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
// by 32 columns; TJ warps of a block own a tile and march along i, warp w on
// the tile's row w and lane l on column l, working at block step tau on plane
// tau - l - w (lanes and warps skewed by one plane each).  So the k-1
// neighbour of a cell is the previous lane's result of the step before (a
// warp shuffle), the j-1 neighbour the previous warp's result of the step
// before (shared memory, one barrier per step), and the i-1 neighbour the
// thread's own result of the step before.  The rows of a tile run on the
// SM's four sub-partitions at once: a single warp would push all of them
// through one sub-partition's FP64 unit.  Only a tile's first row and first
// lane need other tiles' values: the tile below in j and the tile before in
// k publish their progress (steps completed, one counter per tile, a release
// store) every few steps, and a block waits (acquire load, bounded by
// %globaltimer) for the progress its next steps need, then reads those
// neighbours through L2.  The backward solve mirrors every direction.  Tiles
// are handed out to the resident blocks in an order in which each tile's
// producers come first, so the waits always end.
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
constexpr int WB = LES_WAVE_WB;        // GS-SOR: steps between progress publications
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
__device__ __forceinline__ void cp_async16(void* smem, const void* gmem)
{
    const unsigned s = (unsigned)__cvta_generic_to_shared(smem);
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(s), "l"(gmem) : "memory");
}
__device__ __forceinline__ void cp_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }

// Skewed arrays.  The lanes of a warp work on 32 different planes at a time, so
// in the fields' own layout every lane's value lies in another sector.  A solve
// therefore runs on copies in the order of the work: element (tile, step, warp,
// lane) is the cell that this thread works on at that step.
struct Skew {
    int wj, steps;
    __device__ __forceinline__ size_t at(int i, int j, int k) const   // interior coordinates
    {
        const int l = k & 31, w = j % WAVE_TJ, t = (k >> 5) * wj + j / WAVE_TJ;
        return ((size_t)t * steps + (i + l + w)) * WT + w * 32 + l;
    }
};

// IC(0) substitution, src/pressure.cpp:442-482.
//
// Work: a tile has TJ rows (the last in j may have fewer) by 32 columns.  In
// the forward solve warp w works on row w and lane l on column l, at step tau
// on plane tau - l - w.  The backward solve is its mirror image: warp w on row
// TJ-1-w, lanes from the last column, at step tau on the cell of forward step
// steps-1-tau.  So in both
//   the i-neighbour is the thread's own result of the step before,
//   the k-neighbour the adjacent lane's result of the step before (shuffle),
//   the j-neighbour the previous warp's result of the step before, handed
//   over in shared memory (double-buffered by step parity, one block barrier
//   per step); warp 0 takes it from the next tile in j.
//
// Data: per tile and step one record of eight values for each of the 128 cells
//   Lw Ls Lb | Lc 1/Lc | Lw(i+1) Ls(j+1) Lb(k+1)
// of which the forward solve reads the first five and the backward solve the
// last five, and the right-hand side, overwritten by the result: 6 KB per step
// (FP64), contiguous, copied eight steps ahead in 16-byte pieces.  The records
// are laid out once per solve (ic_records).  COPY = false: no records; the
// operands are read from the factor's and the vectors' own arrays, cell by cell
// (a context without the memory for the copies): 96x64x64 694 us an apply,
// 256x128x128 2015.
//
// Roles: four warps compute; a fifth waits for the producers and brings their
// values into shared memory, up to RING batches ahead, and a sixth publishes
// the tile's progress.  So a polled round trip, a load through L2 and a fence
// (about a microsecond each) lengthen the distance between tiles, not each
// batch of steps.
//
// Bound by the chain of a step: nine FP64 operations that hold a sub-partition's
// unit about 64 cycles each (three for the division with the reciprocal at
// hand, see div_by, instead of ten or more), the shuffle and the barrier.
// Apply, 96x64x64: 960 -> 464 us; 256x128x128: 2930 -> 1616 us.
constexpr int REC = 8;    // values of a record
constexpr int IWB = 4;    // steps of a batch (1: 498, 2: 477, 4: 464 us for 96x64x64)
constexpr int RING = 8;   // batches of neighbours' values in flight
constexpr int IC_THREADS = WT + 64;
template <typename T>
struct IcStage {
    T v[WD][6][WT];                // five factors and the right-hand side
    T xs[2][WAVE_TJ][32];          // each row's result of the last two steps
    T zj[RING][IWB][32];            // the row next to warp 0's
    T zk[RING][IWB][WAVE_TJ];       // the column next to the near lane's
    volatile int ready, done, fail;   // batches brought in, computed; a wait gave up
    int go;
};

// The computing warps' barrier.
__device__ __forceinline__ void compute_barrier() { asm volatile("bar.sync 1, %0;" ::"n"(WT) : "memory"); }

// One lane waits until *p has reached n; false once `fail` is set (the waits
// on other blocks are the bounded ones) or after about 4 s.
__device__ __forceinline__ bool wait_shared(const volatile int* p, int n, const volatile int* fail)
{
    unsigned spins = 0;
    unsigned long long t0 = 0;
    while (*p < n) {
        if (*fail) return false;
        if ((++spins & 1023u) == 0u) {
            const unsigned long long t = globaltimer_ns();
            if (t0 == 0) t0 = t;
            if (t - t0 > 4000000000ull) return false;
        }
    }
    __threadfence_block();
    return true;
}

// sum / Lc with y = RN(1/Lc); y = 0 marks an Lc outside the range (see div_by)
__device__ __forceinline__ double ic_divide(double sum, double lc, double y)
{
    const int hi = __double2hiint(sum), e = (hi >> 20) & 0x7ff;
    const double q = sum * y;
    if (y != 0.0) {
        if (e > 1023 - 500 && e < 1023 + 500) return fma(fma(-q, lc, sum), y, q);
        if (((hi << 1) | __double2loint(sum)) == 0) return q;   // 0 with its sign
    }
    return div_slow(sum, lc);
}
__device__ __forceinline__ float ic_divide(float sum, float lc, float) { return sum / lc; }

// A factor's own arrays (COPY = false)
struct IcFactor {
    const double *Lc, *Lw, *Ls, *Lb;
};
__device__ __forceinline__ void copy_in(double* smem, const double* gmem) { cp_async<8>(smem, gmem); }
__device__ __forceinline__ void copy_in(float* smem, const float* gmem) { cp_async<4>(smem, gmem); }
__device__ __forceinline__ void copy_in(float* smem, const double* gmem) { *smem = (float)__ldg(gmem); }

// zs: the right-hand side, overwritten by the result, in the records' order;
// COPY = false: the result z, and r the right-hand side of the forward solve.
template <typename T, int DIR, bool COPY>
__device__ bool ic_tile(const Wave& W, int t, int base, const T* __restrict__ rec, const IcFactor& L,
                        const T* __restrict__ r_in, T* zs, IcStage<T>& sg)
{
    constexpr unsigned FULL = 0xffffffffu;
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const int J = t % W.wj, K = t / W.wj;
    const int rows = min(WAVE_TJ, W.ny - J * WAVE_TJ);
    const TileDeps d = tile_deps<DIR>(W, J, K, t);
    const int near = DIR > 0 ? 0 : 31;
    const size_t tile = (size_t)W.steps * WT, tb = (size_t)t * tile;
    const int batches = (W.steps + IWB - 1) / IWB;
    auto fstep = [&](int tau) { return DIR > 0 ? tau : W.steps - 1 - tau; };   // the forward step of the same cells
    if (threadIdx.x == 0) sg.ready = sg.done = sg.fail = 0;
    __syncthreads();

    if (w == WAVE_TJ) {   // the neighbours' values
        Watch watch{nullptr, base, 0, base - (1 << 20)};
        if (lane == 0 && d.dj >= 0) { watch.p = W.prog + d.dj; watch.ahead = WAVE_TJ - 1; }
        if (lane == 1 && d.dk >= 0) { watch.p = W.prog + d.dk; watch.ahead = 31; }
        // row 0 or TJ-1 of the tile next in j; column 0 or 31 of the tile next in k
        const T* const zj_at = zs + (size_t)(DIR > 0 ? t - 1 : t + 1) * tile + (DIR > 0 ? 32 * (WAVE_TJ - 1) : 0) + lane;
        const int q0 = lane & (IWB - 1), row0 = (lane / IWB) & (WAVE_TJ - 1);
        const T* const zk_at = zs + (size_t)(DIR > 0 ? t - W.wj : t + W.wj) * tile + row0 * 32 + (DIR > 0 ? 31 : 0);
        const int rj = DIR > 0 ? 0 : WAVE_TJ - 1;   // the row that needs the j-neighbour
        // the same row and column of the grid
        const int jn = J * WAVE_TJ + (DIR > 0 ? -1 : WAVE_TJ), kj = K * 32 + lane, kn = K * 32 + (DIR > 0 ? -1 : 32);
        for (int n = 0; n < batches; ++n) {
            const int tau0 = n * IWB, tend = min(tau0 + IWB, W.steps);
            bool ok = true;
            if (watch.p) {
                const int target = base + min(tend + watch.ahead, W.steps);
                if (watch.seen - target < 0) ok = wait_progress(watch.p, target, W.err, watch.seen);
            }
            if (lane == 2) ok = wait_shared(&sg.done, n - RING + 1, &sg.fail);   // the ring's place is free
            if (!__all_sync(FULL, ok)) {
                sg.fail = 1;
                break;
            }
            __syncwarp();   // the lanes that waited order the others' loads and stores (a vote orders nothing)
            const int sl = n & (RING - 1);
            T zj[IWB], zk = T(0);
#pragma unroll
            for (int q = 0; q < IWB; ++q) {
                const int f = fstep(tau0 + q), i = f - lane - rj;
                zj[q] = T(0);
                if (d.dj >= 0 && i >= 0 && i < W.nx && (COPY || kj < W.nz))
                    zj[q] = __ldcg(COPY ? zj_at + (size_t)(f + (DIR > 0 ? WAVE_TJ - 1 : 1 - WAVE_TJ)) * WT
                                        : zs + i * W.si + jn * W.sj + kj);
            }
            {
                const int f = fstep(tau0 + q0), i = f - near - row0;
                if (d.dk >= 0 && lane < IWB * WAVE_TJ && i >= 0 && i < W.nx && (COPY || row0 < rows))
                    zk = __ldcg(COPY ? zk_at + (size_t)(f + (DIR > 0 ? 31 : -31)) * WT
                                     : zs + i * W.si + (J * WAVE_TJ + row0) * W.sj + kn);
            }
#pragma unroll
            for (int q = 0; q < IWB; ++q) sg.zj[sl][q][lane] = zj[q];
            if (lane < IWB * WAVE_TJ) sg.zk[sl][q0][row0] = zk;
            __threadfence_block();
            __syncwarp();
            if (lane == 0) sg.ready = n + 1;
        }
    } else if (w == WAVE_TJ + 1) {   // the tile's progress
        if (lane == 0 && t != W.stall)
            for (int n = 0; n < batches;) {
                if (!wait_shared(&sg.done, n + 1, &sg.fail)) break;
                n = sg.done;   // a release takes longer than a batch: the latest
                __threadfence_block();
                st_release(W.prog + t, base + min(n * IWB, W.steps));
            }
    } else {
        const int row = DIR > 0 ? w : WAVE_TJ - 1 - w;
        const int j = J * WAVE_TJ + row, k = K * 32 + lane, el = row * 32 + lane;
        const bool cell = row < rows && k < W.nz;
        const bool jin = DIR > 0 ? j > 0 : j < W.ny - 1, kin = DIR > 0 ? k > 0 : k < W.nz - 1;
        constexpr int PER = 16 / sizeof(T), NREC = 5 * WT / PER, NALL = 6 * WT / PER;   // 16-byte pieces
        auto stage = [&](int tau) {
            if (!COPY) {
                const int i = fstep(tau) - lane - row;
                if (tau < W.steps && cell && i >= 0 && i < W.nx) {
                    const int id = i * W.si + j * W.sj + k;
                    T* const to = &sg.v[tau & (WD - 1)][0][el];
                    constexpr int F = DIR > 0 ? 0 : 2, C = DIR > 0 ? 3 : 0;
                    // (factors of a missing neighbour are not used)
                    copy_in(to + F * WT, L.Lw + id + (DIR > 0 || i == W.nx - 1 ? 0 : W.si));
                    copy_in(to + (F + 1) * WT, L.Ls + id + (DIR > 0 || !jin ? 0 : W.sj));
                    copy_in(to + (F + 2) * WT, L.Lb + id + (DIR > 0 || !kin ? 0 : 1));
                    copy_in(to + C * WT, L.Lc + id);
                    to[(C + 1) * WT] = T(0);   // no reciprocal: a division
                    copy_in(to + 5 * WT, (DIR > 0 ? r_in : zs) + id);
                }
            } else if (tau < W.steps) {
                const int f = fstep(tau), sl = tau & (WD - 1);
                const T* const r = rec + ((size_t)t * W.steps + f) * (REC * WT) + (DIR > 0 ? 0 : 3 * WT);
                const T* const z = zs + tb + (size_t)f * WT;
                T* const to = &sg.v[sl][0][0];
#pragma unroll
                for (int c = threadIdx.x; c < NALL; c += WT)
                    cp_async16(to + c * PER, c < NREC ? r + c * PER : z + (c - NREC) * PER);
            }
            cp_commit();
        };
        T prev = T(0);
        sg.xs[0][w][lane] = sg.xs[1][w][lane] = T(0);
#pragma unroll
        for (int q = 0; q < WD - 1; ++q) stage(q);
        cp_wait<WD - 2>();   // step 0
        compute_barrier();
        for (int n = 0; n < batches; ++n) {
            const int tau0 = n * IWB, tend = min(tau0 + IWB, W.steps), nr = n & (RING - 1);
            if (threadIdx.x == 0) {   // one thread decides, so that the warps leave together
                sg.go = wait_shared(&sg.ready, n + 1, &sg.fail);
                if (!sg.go) sg.fail = 1;
            }
            compute_barrier();
            if (!sg.go) break;
#pragma unroll
            for (int q = 0; q < IWB; ++q) {
                const int tau = tau0 + q;
                if (tau >= tend) break;   // block-uniform
                stage(tau + WD - 1);
                const int i = fstep(tau) - lane - row, sl = tau & (WD - 1);
                const bool act = cell && i >= 0 && i < W.nx;
                const bool ib = DIR > 0 ? i > 0 : i < W.nx - 1;
                T zk = DIR > 0 ? __shfl_up_sync(FULL, prev, 1) : __shfl_down_sync(FULL, prev, 1);
                if (lane == near) zk = sg.zk[nr][q][row];
                const T zj = w == 0 ? sg.zj[nr][q][lane] : sg.xs[(tau - 1) & 1][w - 1][lane];
                // :451-463 / :469-481, the terms in the reference's order
                constexpr int F = DIR > 0 ? 0 : 2, C = DIR > 0 ? 3 : 0;   // the factors', the diagonal's place
                T sum = sg.v[sl][5][el];
                T a = sum - sg.v[sl][F][el] * prev;
                sum = ib ? a : sum;
                a = sum - sg.v[sl][F + 1][el] * zj;
                sum = jin ? a : sum;
                a = sum - sg.v[sl][F + 2][el] * zk;
                sum = kin ? a : sum;
                // (the lanes outside the grid hold anything: not through the slow path)
                T out = T(0);
                if (act) {
                    out = ic_divide(sum, sg.v[sl][C][el], sg.v[sl][C + 1][el]);
                    zs[COPY ? tb + (size_t)fstep(tau) * WT + el : (size_t)(i * W.si + j * W.sj + k)] = out;
                }
                prev = out;
                sg.xs[tau & 1][w][lane] = out;
                cp_wait<WD - 2>();        // this thread's pieces of the next step are in
                compute_barrier();        // the next step reads this step's rows and others' pieces
            }
            if (threadIdx.x == 0) {
                __threadfence_block();
                sg.done = n + 1;
            }
        }
        cp_wait<0>();
    }
    __syncthreads();
    const bool good = sg.fail == 0;
    __syncthreads();   // the next tile clears it
    return good;
}

// apply_ic_preconditioner, src/pressure.cpp:442-482: the forward solve over
// all tiles, one grid barrier, the backward solve.  T = double is the
// reference's arithmetic; T = float serves the FP32 inner solve of the
// mixed-precision path (st == nullptr: never skipped).
template <typename T, bool COPY>
__global__ void __launch_bounds__(IC_THREADS) k_ic_wave(Wave W, int base, const T* __restrict__ rec, IcFactor L,
                                                        const T* __restrict__ r, T* zs, GridSync gs,
                                                        const SolverState* st, int skip_done)
{
    if (skip_done && st && st->done) return;   // uniform across blocks: no barrier is entered
    extern __shared__ char ic_sm[];
    IcStage<T>& sg = *reinterpret_cast<IcStage<T>*>(ic_sm);
    const int b = blockIdx.x, nb = gridDim.x;  // one tile per block at a time
    bool ok = true;
    for (int t = b; t < W.ntiles && ok; t += nb) ok = ic_tile<T, 1, COPY>(W, t, base, rec, L, r, zs, sg);
    if (!grid_barrier(gs) || !ok) return;
    for (int t = b; t < W.ntiles && ok; t += nb)
        ok = ic_tile<T, -1, COPY>(W, W.ntiles - 1 - t, base + W.steps + 1, rec, L, r, zs, sg);
}

// One thread per cell of the grid, in a one-dimensional grid of blocks (the
// other dimensions end at 65535 blocks, a wavefront's planes need not).
constexpr int FLAT = 256;
inline unsigned flat_grid(const Geo& g) { return (unsigned)((g.n + FLAT - 1) / FLAT); }
struct CellAt {
    int id, i, j, k;
};
__device__ __forceinline__ bool flat_cell(const Geo& g, CellAt& c)
{
    c.id = blockIdx.x * FLAT + threadIdx.x;
    if (c.id >= g.n) return false;
    c.i = c.id / g.si;
    const int r = c.id - c.i * g.si;
    c.j = r / g.sj;
    c.k = r - c.j * g.sj;
    return true;
}

// The records of a factor (its FP64 diagonals).
template <typename T>
__global__ void k_ic_records(Geo g, Skew sk, const double* __restrict__ Lc, const double* __restrict__ Lw,
                             const double* __restrict__ Ls, const double* __restrict__ Lb, T* __restrict__ rec)
{
    CellAt q;
    if (!flat_cell(g, q)) return;
    const int id = q.id, i = q.i, j = q.j, k = q.k;
    const size_t at = sk.at(i, j, k);
    T* const r = rec + at / WT * (REC * WT) + at % WT;
    const T c = (T)Lc[id];
    r[0] = (T)Lw[id];
    r[WT] = (T)Ls[id];
    r[2 * WT] = (T)Lb[id];
    r[3 * WT] = c;
    const int e = (__double2hiint((double)c) >> 20) & 0x7ff;
    r[4 * WT] = e > 1023 - 400 && e < 1023 + 400 ? T(1) / c : T(0);
    r[5 * WT] = i < g.nx - 1 ? (T)Lw[id + g.si] : T(0);
    r[6 * WT] = j < g.ny - 1 ? (T)Ls[id + g.sj] : T(0);
    r[7 * WT] = k < g.nz - 1 ? (T)Lb[id + 1] : T(0);
}

template <typename T, bool IN>
__global__ void k_ic_skew(Geo g, Skew sk, const T* __restrict__ from, T* __restrict__ to, const SolverState* st,
                          int skip_done)
{
    if (skip_done && st && st->done) return;
    CellAt q;
    if (!flat_cell(g, q)) return;
    const int id = q.id, i = q.i, j = q.j, k = q.k;
    if (IN) to[sk.at(i, j, k)] = from[id];
    else to[id] = from[sk.at(i, j, k)];
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
// every SM busy.  256x128x128: 1180 -> 190 us per sweep (the FP64 pipe alone
// needs about 95); h = 1/161, 191x161x115: 2070 -> 318 us; 67x46x53: 570 -> 80.
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
// Layout.  The solve runs on skewed copies of p's interior and of the
// right-hand side: every access of a step is then contiguous (in the field's
// own layout: 424 us per sweep at 256x128x128, bound by those accesses), and
// the old values of the east, north and top neighbours are the next step's own
// elements of the same thread, the next warp and the next lane: a step copies
// one new value per cell instead of four.  Faces stay in p.
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
//
// COPY = false: no copies (a context without the memory for them): ps is the
// field itself and rhs, rep lie in the fields' layout; one sweep at a time, with
// the divisions that serve any spacing.  256x128x128: 954 us per sweep.
template <int FORM, bool COPY>
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
            const int id = rb + i * ssi;
            const size_t at = COPY ? tb + (size_t)tau * WT : (size_t)id;
            cp_async<8>(&sg.own[sl][w][lane], po + at);
            cp_async<8>(&sg.rhs[sl][w][lane], A.rhs + at);
            if (last_row)
                cp_async<8>(&sg.north[sl][lane], wall_n ? p + id + ssj : pn + (COPY ? nb + (size_t)(tau - w) * WT : id + ssj));
            if (last_col)
                cp_async<8>(&sg.top[sl][w], wall_t ? p + id + 1 : pt + (COPY ? ob + (size_t)(tau - lane) * WT : id + 1));
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
                ps0[q] = __ldcg(COPY && d.dj >= 0 ? A.ps + (t - 1) * tile + (size_t)(tau0 + q + WAVE_TJ - 1) * WT + 32 * (WAVE_TJ - 1) + lane
                                          : p + rb + i * ssi - ssj);
        }
        {
            const int q = lane & (WB - 1), i = tau0 + q - w;
            if (w < rows && i >= 0 && i < W.nx)
                pb0 = __ldcg(COPY && d.dk >= 0 ? A.ps + (t - W.wj) * tile + (size_t)(tau0 + q + 31) * WT + w * 32 + 31
                                       : p + W.off + jr * ssj + i * ssi + kb - 1);
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
            double x = 0.0;   // (the lanes outside the grid hold anything: not through the slow path)
            if (!act) {
            } else if (FORM == GS_EQUAL) x = fma((ew + ns) + tb2, A.dx.y, -rh);
            else if (FORM == GS_POW2) x = fma(tb2, A.dz.y, fma(ns, A.dy.y, ew * A.dx.y)) - rh;
            else x = ((div_by(ew, A.dx) + div_by(ns, A.dy)) + div_by(tb2, A.dz)) - rh;
            const double v = one_m_omega * po + omega_coef * x;
            if (act) {
                const int id = rb + i * ssi;
                A.ps[COPY ? tb + (size_t)tau * WT : (size_t)id] = v;
                // the faces next to this cell, src/pressure.cpp:14-72
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
                        auto rep = [&](int di, int dj, int dk) -> double& {
                            return rep_new[COPY ? sk.at(i + di, jr + dj, k + dk) : (size_t)(id + di * ssi + dj * ssj + dk)];
                        };
                        if (f & 1u) rep(1, 0, 0) = v;
                        if (f & 2u) rep(-1, 0, 0) = v;
                        if (f & 4u) rep(0, 1, 0) = v;
                        if (f & 8u) rep(0, -1, 0) = v;
                        if (f & 16u) rep(0, 0, 1) = v;
                        if (f & 32u) rep(0, 0, -1) = v;
                        if (f & 128u) rep(0, 0, 0) = 0.0;
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

// One thread per column, its words of 32 planes shared out along y.
__global__ void k_gs_flags(int nx, int ny, int nz, const uint8_t* __restrict__ solid, unsigned* __restrict__ rd,
                           unsigned* __restrict__ wr, uint8_t* __restrict__ fl)
{
    const int si = ny * nz, sj = nz;
    const int col = blockIdx.x * blockDim.x + threadIdx.x;
    if (col >= si) return;
    const int j = col / nz, k = col - j * nz;
    auto interior = [&](int i, int jj, int kk) {
        return i >= 1 && i <= nx - 2 && jj >= 1 && jj <= ny - 2 && kk >= 1 && kk <= nz - 2;
    };
    for (int wi = blockIdx.y; wi * 32 < nx; wi += gridDim.y) {
        unsigned r = 0u, w = 0u;
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
}

// p's interior (COPY) and the right-hand side, src/pressure.cpp:197-210.
template <bool COPY>
__global__ void k_gs_skew(Geo g, Skew sk, double coef, DivBy two_dx, DivBy two_dy, DivBy two_dz,
                          const double* __restrict__ u, const double* __restrict__ v, const double* __restrict__ w,
                          const double* __restrict__ p, double* __restrict__ ps, double* __restrict__ rhs)
{
    CellAt q;
    if (!flat_cell(g, q)) return;
    const int id = q.id, i = q.i, j = q.j, k = q.k;
    if (i < 1 || i > g.nx - 2 || j < 1 || j > g.ny - 2 || k < 1 || k > g.nz - 2) return;
    const size_t at = COPY ? sk.at(i - 1, j - 1, k - 1) : (size_t)id;
    const double div = div_by(u[id + g.si] - u[id - g.si], two_dx) + div_by(v[id + g.sj] - v[id - g.sj], two_dy) +
                       div_by(w[id + 1] - w[id - 1], two_dz);
    if (COPY) ps[at] = p[id];
    rhs[at] = coef * div;
}

__global__ void k_gs_unskew(Geo g, Skew sk, const double* __restrict__ ps, double* __restrict__ p)
{
    CellAt q;
    if (!flat_cell(g, q)) return;
    const int i = q.i, j = q.j, k = q.k;
    if (i < 1 || i > g.nx - 2 || j < 1 || j > g.ny - 2 || k < 1 || k > g.nz - 2) return;
    p[q.id] = ps[sk.at(i - 1, j - 1, k - 1)];
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

template <int FORM, bool COPY>
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
            if (COPY && run > 1) gs_backup(A, done, true, gt, gn);
        }
        if (gt < GS_BATCH) A.gmax[gt] = 0ull;
        if (!grid_barrier(A.gs)) return;
        bool ok = true;
        for (int s = q0; s < run && ok; s += A.Q) {
            unsigned long long maxr = 0ull;
            for (int t = blk; t < W.ntiles && ok; t += A.nb)
                ok = gs_tile<FORM, COPY>(A, t, s, done + s, epoch + s * (W.steps + 1), one_m_omega, omega_coef, maxr, sg);
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
        epoch += (COPY ? GS_BATCH : 1) * (W.steps + 1);
        // the first sweep whose max|dp| is below tol (the same in every thread)
        int hit = run;
        for (int s = 0; s < run && hit == run; ++s)
            if (__longlong_as_double((long long)__ldcg(A.gmax + s)) < A.tol) hit = s;
        if (COPY && hit < run - 1) {   // before the batch's last: run that many again from its start
            run = hit + 1;
            redo = true;
            gs_backup(A, done, false, gt, gn);
        } else {
            done += run;
            converged = hit < run;
            redo = false;
            if (COPY) run = min(2 * run, GS_BATCH);
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
    if (span < 0 || span > (1 << 30)) return fail(c, LES_BAD_ARG, "wavefront: too many sweeps in one launch");
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
les_status wave_resident(les_ctx* c, const void* fn, int threads, size_t smem, int* blocks)
{
    int per_sm = 0;
    les_status st = check_cuda(c, cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, fn, threads, smem), "occupancy");
    if (st) return st;
    if (per_sm < 1) return fail(c, LES_CUDA_ERROR, "wavefront kernel cannot be resident");
    *blocks = per_sm * c->sms;
    return LES_OK;
}

les_status wave_launch(les_ctx* c, const void* fn, void** args, int grid, int threads, size_t smem, int pid)
{
    // count and generation only: the error word stays set until the host reads it
    les_status st = check_cuda(c, cudaMemsetAsync(c->gsync, 0, sizeof(unsigned) * 2, c->stream), "reset barrier");
    if (st) return st;
    cudaEvent_t e1 = nullptr;
    if (pid >= 0 && c->prof_on) prof_begin(c, pid, &e1);
    st = check_cuda(c, cudaLaunchCooperativeKernel(fn, dim3(grid), dim3(threads), args, smem, c->stream),
                    "cooperative launch");
    ++c->launches;
    if (e1) cudaEventRecord(e1, c->stream);
    return st;
}

}  // namespace

namespace les {

// LES_TIMEOUT (and the flag cleared) if a wavefront wait gave up since the last check.
les_status wave_check(les_ctx* c) { return check_barrier(c); }

// The skewed arrays.  false: the context works without them (LES_OPT_WAVE_COPIES)
// or the memory cannot be had; the solve then runs on the fields' own layout.
// Arrays of up to SKEW_KEEP are kept from solve to solve, larger ones given back
// at its end: cudaMalloc and cudaFree of 0.34 GB take 0.25 ms, of 1.3 GB 1.0 ms.
constexpr size_t SKEW_KEEP = size_t(1) << 30;

static bool skew_buffer(les_ctx* c, size_t doubles)
{
    if (!c->wave_copies) return false;
    if (c->skew_len >= doubles) return true;
    skew_free(c);
    if (cudaMalloc(&c->skew_buf, sizeof(double) * doubles) != cudaSuccess) {
        cudaGetLastError();
        c->skew_buf = nullptr;
        return false;
    }
    c->skew_len = doubles;
    return true;
}

void skew_free(les_ctx* c)
{
    cudaFree(c->skew_buf);
    c->skew_buf = nullptr;
    c->skew_len = 0;
}

void skew_trim(les_ctx* c)
{
    if (sizeof(double) * c->skew_len > SKEW_KEEP) skew_free(c);
}

static Skew ic_skew(const les_ctx* c, size_t* len)
{
    const Geo& g = c->g;
    const Skew sk{(g.ny + WAVE_TJ - 1) / WAVE_TJ, g.nx + 31 + WAVE_TJ - 1};
    *len = (size_t)sk.wj * ((g.nz + 31) / 32) * sk.steps * WT;
    return sk;
}

// doubles that hold the records and the vector
template <typename T>
static size_t ic_doubles(size_t len)
{
    return ((REC + 1) * len * sizeof(T) + sizeof(double) - 1) / sizeof(double);
}

// Lays out the records of the factor L (c, n, s, e, w, t, b) for the applies
// that follow.
template <typename T>
static les_status ic_records(les_ctx* c, const double* const* L)
{
    size_t len;
    const Skew sk = ic_skew(c, &len);
    if (!skew_buffer(c, ic_doubles<T>(len))) return LES_OK;
    launch(c, k_ic_records<T>, flat_grid(c->g), FLAT, c->g, sk, L[0], L[4], L[2], L[6],
           reinterpret_cast<T*>(c->skew_buf));
    return check_launch(c, "ic records");
}

les_status ic_records64(les_ctx* c, const double* const* L) { return ic_records<double>(c, L); }
les_status ic_records32(les_ctx* c, const double* const* L) { return ic_records<float>(c, L); }

// z = M^-1 r with the factor L whose records were laid out last.
template <typename T>
static les_status ic_apply(les_ctx* c, const double* const* L, const T* r, T* z, const SolverState* state, int skip_done)
{
    size_t len;
    const Skew sk = ic_skew(c, &len);
    const bool copy = c->wave_copies && c->skew_len >= ic_doubles<T>(len);
    const T* rec = reinterpret_cast<const T*>(c->skew_buf);
    T* zs = copy ? reinterpret_cast<T*>(c->skew_buf) + REC * len : z;
    IcFactor F{L[0], L[4], L[2], L[6]};
    Wave W;
    int base = 0;
    les_status st = wave_setup(c, c->g.nx, c->g.ny, c->g.nz, 0, 2 * (c->g.nx + 32 + WAVE_TJ), 1, W, base);
    if (st) return st;
    const void* fn = copy ? (const void*)k_ic_wave<T, true> : (const void*)k_ic_wave<T, false>;
    const size_t smem = sizeof(IcStage<T>);
    st = check_cuda(c, cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem), "smem attribute");
    if (st) return st;
    int resident = 0;
    if ((st = wave_resident(c, fn, IC_THREADS, smem, &resident))) return st;
    const int grid = W.ntiles < resident ? W.ntiles : resident;
    GridSync gs = grid_sync(c, grid);
    if (copy) launch(c, k_ic_skew<T, true>, flat_grid(c->g), FLAT, c->g, sk, r, zs, state, skip_done);
    void* args[] = {&W, &base, (void*)&rec, &F, (void*)&r, (void*)&zs, &gs, (void*)&state, &skip_done};
    if ((st = wave_launch(c, fn, args, grid, IC_THREADS, smem, PROF_IC))) return st;
    if (copy) launch(c, k_ic_skew<T, false>, flat_grid(c->g), FLAT, c->g, sk, (const T*)zs, z, state, skip_done);
    return check_launch(c, "ic apply");
}

les_status ic_apply_dev(les_ctx* c, const double* const* L, const double* r, double* z, int skip_done)
{
    return ic_apply<double>(c, L, r, z, c->state, skip_done);
}

les_status ic_apply_dev32(les_ctx* c, const double* const* L, const float* r, float* z, SolverState* st)
{
    return ic_apply<float>(c, L, r, z, st, st ? 1 : 0);
}

les_status build_ic_dev(les_ctx* c)
{
    const size_t nb = sizeof(double) * (size_t)c->g.n;
    for (int q = 0; q < 7; ++q) {
        if (!c->L[q]) {
            les_status st = check_cuda(c, dev_malloc(c, &c->L[q], nb), "cudaMalloc(L)");
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
    // progress values of a sweep, and the most sweeps of a solve
    const long long per = g.nx - 2 + 32 + WAVE_TJ;
    if (max_iter * per > (1 << 29)) return fail(c, LES_BAD_ARG, "wavefront: too many sweeps in one launch");
    // the skewed arrays first: the work is split for the form that runs
    const Skew sk{(g.ny - 2 + WAVE_TJ - 1) / WAVE_TJ, g.nx - 2 + 31 + WAVE_TJ - 1};
    const int ntiles = sk.wj * ((g.nz - 2 + 31) / 32);
    const size_t len = (size_t)ntiles * sk.steps * WT;
    const bool copy = 8 * GS_BATCH * per <= (1 << 29) && skew_buffer(c, 5 * len);   // (room for the batches below)
    const void* fn = !copy ? (const void*)k_gs_wave<GS_DIV, false>
                   : !p2   ? (const void*)k_gs_wave<GS_DIV, true>
                   : (dx2 == dy2 && dy2 == dz2 ? (const void*)k_gs_wave<GS_EQUAL, true> : (const void*)k_gs_wave<GS_POW2, true>);
    int resident = 0;
    st = wave_resident(c, fn, WT, 0, &resident);
    if (st) return st;
    // Sweeps in flight: as many as there are resident blocks for, up to what a
    // sweep's length has room for (a sweep starts about 20 steps behind the
    // one before: the staging depth, the waits' granularity).
    const int room = sk.steps / 20 + 1;
    int Q = copy ? resident / ntiles : 1;
    Q = Q < 1 ? 1 : (Q > room ? room : Q);
    if (Q > GS_MAX_FLIGHT) Q = GS_MAX_FLIGHT;
    if (Q > max_iter && max_iter > 0) Q = max_iter;
    GsArgs a{};
    int base = 0;
    // progress values: every batch (about max_iter / GS_BATCH and the doubling
    // ones before, one run again) takes GS_BATCH sweeps' worth; without the
    // copies a sweep takes its own
    const long long sweeps_worth = copy ? (long long)(max_iter / GS_BATCH + 8) * GS_BATCH : max_iter;
    st = wave_setup(c, g.nx - 2, g.ny - 2, g.nz - 2, g.si + g.sj + 1, sweeps_worth * per, Q, a.W, base);
    if (st) return st;
    a.len = len;
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
    a.ps = copy ? c->skew_buf : a.p;
    double* const rhs = copy ? c->skew_buf + len : c->w[4];
    a.rhs = rhs;
    a.ps_back = copy ? c->skew_buf + 2 * len : nullptr;
    a.rep[0] = copy ? c->skew_buf + 3 * len : c->w[5];
    a.rep[1] = copy ? c->skew_buf + 4 * len : c->w[6];
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
    launch(c, copy ? k_gs_skew<true> : k_gs_skew<false>, flat_grid(g), FLAT, g, sk, rho / dt, div_by_const(2 * m.dx), div_by_const(2 * m.dy),
           div_by_const(2 * m.dz), (const double*)c->slot[LES_U], (const double*)c->slot[LES_V],
           (const double*)c->slot[LES_W], (const double*)a.p, a.ps, rhs);
    if (c->n_solid)
        launch(c, k_gs_flags, dim3((g.si + 255) / 256, words < 65535 ? words : 65535), 256, g.nx, g.ny, g.nz, (const uint8_t*)c->mask, rd,
               rd + (size_t)words * g.si, fl);
    if ((st = check_launch(c, "gs set-up"))) return st;
    void* args[] = {&a, &base};
    if (max_iter > 0) {
        st = wave_launch(c, fn, args, grid, WT, 0, -1);
        if (st) return st;
        if (copy) launch(c, k_gs_unskew, flat_grid(g), FLAT, g, sk, (const double*)a.ps, a.p);
        if ((st = pressure_bcs_dev(c, a.p))) return st;   // of the last sweep
    }
    st = check_barrier(c);
    if (st) return st;
    st = read_state(c);
    if (st) return st;
    skew_trim(c);
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
