// les_plane.cu -- plane-march passes (les_plane.cuh): pass A, Jacobi's pass B,
// the choice of tiles and the launches.
#include "les_plane.cuh"

#include <algorithm>
#include <cmath>

namespace {

template <bool FIRST>
__global__ void __launch_bounds__(512, 2) k_plane_b0(const __grid_constant__ PlaneArgsB a)
{
    plane_b0<FIRST>(a, blockIdx.x, gridDim.x);
}

template <int FORM>
KPA pick_a_f(bool first)
{
    return first ? k_plane_a<FORM, true> : k_plane_a<FORM, false>;
}

KPA pick_a(int form, bool first)
{
    return form == 0 ? pick_a_f<0>(first) : (form == 1 ? pick_a_f<1>(first) : pick_a_f<2>(first));
}

KPB pick_b(int S, int form, bool first)
{
    if (S == 0) return first ? k_plane_b0<true> : k_plane_b0<false>;
    return S <= 3 ? plane_pick_b_lo(S, form, first) : plane_pick_b_hi(S, form, first);
}

constexpr size_t SMEM_MAX = 225 * 1024;   // of the SM's 227 KB, less the kernels' static arrays

int form_of(const Geo& g, const PlaneMap& m) { return g.nz % PV ? 2 : (32 % m.lk ? 1 : 0); }

// A tile of nk x nj for halo h in at most `threads` threads; false if it does
// not fit.
bool tile_fit(const Geo& g, int nk, int nj, int h, int threads, PlaneMap& m)
{
    const int pj = plane_pitch(g.nz), hk = (h + 3) / 4 * 4;
    m = PlaneMap{};
    m.kw = ((g.nz + nk - 1) / nk + PV - 1) / PV * PV;
    m.nk = (g.nz + m.kw - 1) / m.kw;
    m.lk = std::min(pj, m.kw + (m.nk == 1 ? 0 : (m.nk == 2 ? hk : 2 * hk))) / PV;
    m.tj = (g.ny + nj - 1) / nj;
    m.nj = (g.ny + m.tj - 1) / m.tj;
    const int rows = std::min(g.ny, m.tj + (m.nj == 1 ? 0 : (m.nj == 2 ? h : 2 * h)));
    m.groups = (rows + PR - 1) / PR;
    m.threads = (m.lk * m.groups + 31) / 32 * 32;
    return m.threads <= threads;
}

// Tiles and chunks of one pass on one grid: of the tiles that fit a block, and
// of the chunk counts that fill one to four waves of resident blocks, the one
// with the fewest marched steps (a chunk's halo planes and a pass's head
// included).  A step takes about as long with 4 warps on an SM as with 16 --
// its chain of level, barrier and load latency -- so a larger tile beats a
// longer chunk: 256x128x128, pass B in 11-warp tiles of 20 steps 23.6 us, in
// 9-warp tiles of 24 steps 27.3 us; hence a step counts the same up to 20
// warps.  Among equals the one with the fewest warps on an SM, which spreads the
// work over more of them: 96x64x64, pass B in 144 blocks instead of 96, an
// iteration 13.5 -> 12.7 us.
// best == nullptr: only whether there is a tile that fits.
bool plane_tiles(const Geo& g, int h, int levels, int threads, int sms, PlaneMap* best)
{
    double best_t = 1e30;
    int best_w = 0;
    for (int nk = 1; nk <= 16; ++nk) {
        int tried = 0;
        PlaneMap m;
        tile_fit(g, nk, 1, h, threads, m);   // (for lk)
        const int most = PR * (threads / m.lk);   // rows that fit, the fewest row tiles:
        for (int nj = most ? (g.ny + most - 1) / most : g.ny + 1; nj <= g.ny && tried < 8; ++nj) {
            if (!tile_fit(g, nk, nj, h, threads, m)) continue;
            if (m.nk != nk || m.nj != nj) continue;   // the same tiles as a smaller count's
            if (!best) return true;
            ++tried;
            int res = threads / m.threads;
            const size_t by_smem = SMEM_MAX / plane_smem(threads, levels);
            if ((size_t)res > by_smem) res = (int)by_smem;
            if (res < 1) res = 1;
            const int tiles = m.nk * m.nj;
            for (int w = 1; w <= 4; ++w) {
                int nch = (int)((long long)res * sms * w / tiles);
                nch = std::max(1, std::min(nch, (g.nx + 1) / 2));
                m.ci = (g.nx + nch - 1) / nch;
                nch = (g.nx + m.ci - 1) / m.ci;
                m.items = tiles * nch;
                const int per_sm = std::min(res, (m.items + sms - 1) / sms);
                const int waves = (m.items + per_sm * sms - 1) / (per_sm * sms);
                const int steps = m.ci + (nch == 1 ? h : 2 * h);
                const int warps = per_sm * (m.threads / 32);   // on an SM
                const double t = waves * (steps + 4.0) * std::max(20, warps);
                if (t < best_t || (t == best_t && warps < best_w)) {
                    best_t = t;
                    best_w = warps;
                    *best = m;
                }
            }
        }
        if (plane_pitch(g.nz) / nk <= 32) break;   // narrower tiles only add halo
    }
    return best_t < 1e30;
}

Geo padded(const Geo& g)
{
    Geo p = g;
    p.sj = plane_pitch(g.nz);
    p.si = g.ny * p.sj;
    return p;
}

}  // namespace

namespace les {

ChebPairs cheb_pairs(const ColCheb& c, int S)
{
    ChebPairs p{};
    auto two = [](double v) { return make_float2((float)v, (float)v); };
    if (S < 1) return p;
    p.wy = two((double)c.cy[0] / c.cx[0]);
    p.wz = two((double)c.cz[0] / c.cx[0]);
    double s[7] = {1.0};   // level 0 is r' itself (a0 is in level 1's weights)
    for (int k = 1; k <= S; ++k) {
        s[k] = s[k - 1] * c.cx[k - 1];
        p.cc[k - 1] = two((double)c.cc[k - 1] / c.cx[k - 1]);
        p.ci[k - 1] = two((double)c.ci[k - 1] / c.cx[k - 1]);
        p.rr[k - 1] = two(c.rr[k - 1] / s[k]);
        p.gg[k - 1] = two(k >= 3 ? c.gg[k - 1] * s[k - 2] / s[k] : 0.0);
    }
    p.zs = two(s[S]);
    return p;
}

// The scaled levels are larger than r': a bound of their growth, from the sums
// of the weights' magnitudes.
static double level_growth(const ChebPairs& p, int S)
{
    double before = 0.0, g = 1.0, most = 1.0;   // levels k-2, k-1
    for (int k = 0; k < S; ++k) {
        const double cc = std::max(std::fabs(p.cc[k].x), std::fabs(p.ci[k].x));
        const double v = (cc + 2.0 + 2.0 * std::fabs(p.wy.x) + 2.0 * std::fabs(p.wz.x)) * g + std::fabs(p.rr[k].x) +
                         std::fabs(p.gg[k].x) * before;
        before = g;
        g = v;
        if (!(g <= most)) most = g;
    }
    return most;
}

// Growth 2^60 at most: the square of r' is an FP32 number, so |r'| < 2^64 and the
// levels stay below 2^124; and with the last weight normal nothing is lost at the
// lower end.  Cubes have 2^24 at degree 7 and 2^12 at degree 4; the line lies at
// about dx / dy = 10 for degree 7, 300 for degree 4.  (The strips do not scale
// their levels.)
static bool levels_fit(const les_ctx* c, const les_pcg_opts* o, int S)
{
    if (S < 1) return true;
    const ChebPairs p = cheb_pairs(col_cheb(o, (float)c->coef.c0, (float)c->coef.x1, (float)c->coef.y1, (float)c->coef.z1), S);
    return level_growth(p, S) <= 0x1p60 && std::fabs(p.zs.x) >= 0x1p-126f;
}

// a, b: nullptr to ask only whether there are plans
static bool plane_plan(const les_ctx* c, int S, PlaneMap* a, PlaneMap* b)
{
    const Geo& g = c->g;
    const double share = c->share > 0 && c->share <= 1 ? c->share : 1.0;
    const int sms = std::max(1, (int)(c->sms * share));
    if (!plane_tiles(g, 1, 1, plane_threads_a(), sms, a)) return false;
    if (S > 0) return plane_tiles(g, S, S, plane_threads_b(S), sms, b);
    if (b) {
        *b = PlaneMap{};
        b->threads = 512;
        b->items = std::max(1, std::min(2 * sms, (g.nx * (padded(g).si / PV) + 511) / 512));
    }
    return true;
}

// The plane marches serve the solves of the register-column passes: they were
// faster on every grid measured, 24x16x16 to 512x256x256, rows of 16 to 512
// cells, Jacobi and degrees 3 to 7 (1.10 to 2.07 times, les_plane.cuh).  The
// strips run where a caller asked for a strip shape or the autotuner found
// one faster, in batched ensembles, for vectors of 4 GB and more (32-bit byte
// offsets) and for spacings whose scaled levels would leave FP32 (levels_fit).
bool plane_used(const les_ctx* c, const les_pcg_opts* o)
{
    if (!col_supported(c, o)) return false;
    if ((unsigned long long)c->g.nx * c->g.ny * plane_pitch(c->g.nz) >= (1ull << 30)) return false;
    if ((c->tune_tja || c->tune_tjb || c->tune_cia || c->tune_cib) && !c->tune_plane) return false;
    const int S = o->precond == LES_PC_JACOBI ? 0 : o->degree - 1;
    return levels_fit(c, o, S) && plane_plan(c, S, nullptr, nullptr);
}

les_status plane_maps(les_ctx* c, const les_pcg_opts* o, ColPlan& P)
{
    if (!plane_plan(c, P.S, &P.pa, &P.pb)) return fail(c, LES_BAD_ARG, "plane march: no tile fits");
    P.blocks_a = P.pa.items;
    P.blocks_b = P.pb.items;
    return LES_OK;
}

// a kernel's dynamic shared memory limit, raised before its first launch or capture
static les_status smem_limit(les_ctx* c, const void* fn)
{
    return check_cuda(c, cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)SMEM_MAX),
                      "shared memory limit");
}

les_status plane_pass_a(les_ctx* c, const ColPlan& P, bool first, int pc)
{
    float2* const part = reinterpret_cast<float2*>(c->partials);   // pass B's pairs, then pass A's
    PlaneArgsA a{padded(c->g), P.pa, Coef{P.A.k.c0, P.A.k.x1, P.A.k.y1, P.A.k.z1}};
    float* pb[2] = {c->f[2], c->f[3]};
    a.z = reinterpret_cast<const float4*>(c->f[1]);
    a.pold = reinterpret_cast<const float4*>(pb[pc]);
    a.pnew = reinterpret_cast<float4*>(pb[pc ^ 1]);
    a.q = reinterpret_cast<float4*>(c->f[4]);
    a.e = reinterpret_cast<float4*>(c->f[5]);
    a.st = P.in;
    a.outer = P.out;
    a.pslot = pc ^ 1;
    a.total_cap = P.cap;
    a.df = Defer{part, P.blocks_b, part + 2 * (size_t)P.blocks_b};
    const KPA k = pick_a(form_of(c->g, P.pa), first);
    les_status st = smem_limit(c, (const void*)k);
    if (st) return st;
    launch_pdl(c, PROF_IN_SPMV, plane_smem(plane_threads_a(), 1), k, P.blocks_a, P.pa.threads, a);
    return check_launch(c, "plane pass A");
}

les_status plane_pass_b(les_ctx* c, const ColPlan& P, bool first, int rin)
{
    float2* const part = reinterpret_cast<float2*>(c->partials);
    float* r[2] = {c->f[0], c->f[6]};
    PlaneArgsB a{padded(c->g), P.pb, cheb_pairs(P.c3, P.S), P.inv_c0};
    a.r_in = reinterpret_cast<const float4*>(r[rin]);
    a.q = reinterpret_cast<const float4*>(c->f[4]);
    a.r_out = reinterpret_cast<float4*>(r[rin ^ 1]);
    a.z_out = reinterpret_cast<float4*>(c->f[1]);
    a.st = P.in;
    a.outer = P.out;
    a.df = Defer{part + 2 * (size_t)P.blocks_b, P.blocks_a, part};
    const KPB k = pick_b(P.S, P.S ? form_of(c->g, P.pb) : 0, first);
    les_status st = P.S ? smem_limit(c, (const void*)k) : LES_OK;
    if (st) return st;
    launch_pdl(c, PROF_IN_CHEB, P.S ? plane_smem(plane_threads_b(P.S), P.S) : 0, k, P.blocks_b, P.pb.threads, a);
    return check_launch(c, "plane pass B");
}

}  // namespace les
