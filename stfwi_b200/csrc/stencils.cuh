// Stencil kernels of the forward and adjoint steps (sm_100a).
//
// Four kernels per time step pair: fwd_vel (U, V), fwd_str (the stresses,
// receivers, history), adj_a (P, Q) and adj_b (the strain adjoints and the
// gradient sums), each over every tile of every shot of the launch, with the
// tiling and the stencil pieces of stencil_parts.cuh.
#pragma once
#include <type_traits>

#include "stencil_parts.cuh"

namespace stfwi {

__device__ __forceinline__ float f2c(const float2 &v, int c) { return c == 0 ? v.x : v.y; }

// arithmetic on the two columns of a thread
__device__ __forceinline__ float2 dup2(float s) { return make_float2(s, s); }
__device__ __forceinline__ float2 add2(float2 a, float2 b) { return make_float2(a.x + b.x, a.y + b.y); }
__device__ __forceinline__ float2 sub2(float2 a, float2 b) { return make_float2(a.x - b.x, a.y - b.y); }
__device__ __forceinline__ float2 mul2(float2 a, float2 b) { return make_float2(a.x * b.x, a.y * b.y); }
__device__ __forceinline__ float2 fma2(float2 a, float2 b, float2 c)
{
    return make_float2(fmaf(a.x, b.x, c.x), fmaf(a.y, b.y, c.y));
}

// Coefficients of the masked stencils.  A term is dropped only within 2K cells
// of an edge, so a table holds one entry for each of the first and the last
// eight positions and one for all between; a block builds it in shared memory
// while its first boxes are on their way.  A dropped term is a zero
// coefficient: fma(0, f, d) = d exactly.
constexpr int TAB = 17;
__device__ __forceinline__ int tab_at(int t, int n) { return n <= TAB ? min(t, TAB - 1) : t < 8 ? t : min(max(t - n + TAB, 8), TAB - 1); }
__device__ __forceinline__ int tab_pos(int e, int n) { return n <= TAB || e <= 8 ? e : n - TAB + e; }

__device__ __forceinline__ float v4k(const float4 &v, int k) { return k == 1 ? v.x : k == 2 ? v.y : k == 3 ? v.z : v.w; }
template <int FD, class Pred> __device__ __forceinline__ float4 cvec(Pred p)
{
    auto c = [&](int k) { return k <= FD / 2 && p(k) ? cf<FD>(k) : 0.f; };
    return make_float4(c(1), c(2), c(3), c(4));
}
// sets: D+ and D-; A and B of the transposed D+ and of the transposed D- (of positions below lim)
template <int FD> __device__ __forceinline__ float4 cv_P(int t, int n)
{
    return cvec<FD>([&](int k) { return mP(t, k, n); });
}
template <int FD> __device__ __forceinline__ float4 cv_M(int t, int n)
{
    return cvec<FD>([&](int k) { return mM(t, k, n); });
}
template <int FD> __device__ __forceinline__ float4 cv_tPA(int t, int n)
{
    return cvec<FD>([&](int k) { return mP(t - k, k, n); });
}
template <int FD> __device__ __forceinline__ float4 cv_tPB(int t, int n)
{
    return cvec<FD>([&](int k) { return mP(t + k - 1, k, n); });
}
template <int FD> __device__ __forceinline__ float4 cv_tMA(int t, int n, int lim)
{
    return cvec<FD>([&](int k) { return mM(t - k + 1, k, n) && t - k + 1 < lim; });
}
template <int FD> __device__ __forceinline__ float4 cv_tMB(int t, int n, int lim)
{
    return cvec<FD>([&](int k) { return mM(t + k, k, n) && t + k < lim; });
}
// forward kernels: x sets (P, M), z sets (P, M)
struct FwdTab { float4 x[2][TAB], z[2][TAB]; };
// adjoint kernels: x and z sets (tPA, tPB, tMA, tMB); the strain update
// transposes D- as formed below the last column and row
struct AdjTab { float4 x[4][TAB], z[4][TAB]; };

template <int FD> __device__ __forceinline__ void fill(FwdTab *tb, const Geo &g, int tid)
{
    if (tid >= 4 * TAB) return;
    const int set = tid / TAB, e = tid % TAB, n = set < 2 ? g.nx : g.nz, t = tab_pos(e, n);
    float4 *o = set < 2 ? &tb->x[set][e] : &tb->z[set - 2][e];
    *o = (set & 1) == 0 ? cv_P<FD>(t, n) : cv_M<FD>(t, n);
}
template <int FD> __device__ __forceinline__ void fill(AdjTab *tb, const Geo &g, int tid, int below)
{
    if (tid >= 8 * TAB) return;
    const int set = tid / TAB, e = tid % TAB, n = set < 4 ? g.nx : g.nz, t = tab_pos(e, n), lim = n - below;
    float4 *o = set < 4 ? &tb->x[set][e] : &tb->z[set - 4][e];
    const int k = set & 3;
    *o = k == 0 ? cv_tPA<FD>(t, n) : k == 1 ? cv_tPB<FD>(t, n) : k == 2 ? cv_tMA<FD>(t, n, lim) : cv_tMB<FD>(t, n, lim);
}

// a table entry, loaded where it is used: the entries of a thread's columns
// are the same for all its rows, and kept in registers they would spill
__device__ __forceinline__ float4 entry(const float4 *p)
{
    float4 v;
    asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(smem_u32(p)));
    return v;
}

// x stencils of a thread's two columns from their neighbourhood a: with the
// plain coefficients, or (XB) with those of the table rows A (and B) at e0, e1
template <int FD, bool XB> __device__ __forceinline__ float2 x_dp(const float (&a)[10], const float4 *A, int e0, int e1)
{
    if (!XB) {
        auto c = [](int k) { return cf<FD>(k); };
        return make_float2(a_dp<FD>(a, 0, c), a_dp<FD>(a, 1, c));
    }
    const float4 v0 = entry(A + e0), v1 = entry(A + e1);
    return make_float2(a_dp<FD>(a, 0, [&](int k) { return v4k(v0, k); }), a_dp<FD>(a, 1, [&](int k) { return v4k(v1, k); }));
}
template <int FD, bool XB> __device__ __forceinline__ float2 x_dm(const float (&a)[10], const float4 *A, int e0, int e1)
{
    if (!XB) {
        auto c = [](int k) { return cf<FD>(k); };
        return make_float2(a_dm<FD>(a, 0, c), a_dm<FD>(a, 1, c));
    }
    const float4 v0 = entry(A + e0), v1 = entry(A + e1);
    return make_float2(a_dm<FD>(a, 0, [&](int k) { return v4k(v0, k); }), a_dm<FD>(a, 1, [&](int k) { return v4k(v1, k); }));
}
template <int FD, bool XB>
__device__ __forceinline__ float2 x_tdp(const float (&a)[10], const float4 *A, const float4 *B, int e0, int e1)
{
    if (!XB) {
        auto c = [](int k) { return cf<FD>(k); };
        return make_float2(a_tdp<FD>(a, 0, c, c), a_tdp<FD>(a, 1, c, c));
    }
    const float4 u0 = entry(A + e0), v0 = entry(B + e0), u1 = entry(A + e1), v1 = entry(B + e1);
    return make_float2(a_tdp<FD>(a, 0, [&](int k) { return v4k(u0, k); }, [&](int k) { return v4k(v0, k); }),
                       a_tdp<FD>(a, 1, [&](int k) { return v4k(u1, k); }, [&](int k) { return v4k(v1, k); }));
}
template <int FD, bool XB>
__device__ __forceinline__ float2 x_tdm(const float (&a)[10], const float4 *A, const float4 *B, int e0, int e1)
{
    if (!XB) {
        auto c = [](int k) { return cf<FD>(k); };
        return make_float2(a_tdm<FD>(a, 0, c, c), a_tdm<FD>(a, 1, c, c));
    }
    const float4 u0 = entry(A + e0), v0 = entry(B + e0), u1 = entry(A + e1), v1 = entry(B + e1);
    return make_float2(a_tdm<FD>(a, 0, [&](int k) { return v4k(u0, k); }, [&](int k) { return v4k(v0, k); }),
                       a_tdm<FD>(a, 1, [&](int k) { return v4k(u1, k); }, [&](int k) { return v4k(v1, k); }));
}
// z stencils of the pair at row r of the thread from its window w (row r at
// w[r + K]): plain coefficients, or (GUARD) those of the table entry at A (and B)
template <int FD, bool GUARD, int W>
__device__ __forceinline__ float2 z_dp(const float2 (&w)[W], int r, const float4 *A)
{
    constexpr int K = FD / 2;
    float4 v;
    if (GUARD) v = entry(A);
    float2 d = make_float2(0.f, 0.f);
#pragma unroll
    for (int k = 1; k <= K; ++k) d = fma2(dup2(GUARD ? v4k(v, k) : cf<FD>(k)), sub2(w[r + K + k], w[r + K - k + 1]), d);
    return d;
}
template <int FD, bool GUARD, int W>
__device__ __forceinline__ float2 z_dm(const float2 (&w)[W], int r, const float4 *A)
{
    constexpr int K = FD / 2;
    float4 v;
    if (GUARD) v = entry(A);
    float2 d = make_float2(0.f, 0.f);
#pragma unroll
    for (int k = 1; k <= K; ++k) d = fma2(dup2(GUARD ? v4k(v, k) : cf<FD>(k)), sub2(w[r + K + k - 1], w[r + K - k]), d);
    return d;
}
template <int FD, bool GUARD, int W>
__device__ __forceinline__ float2 z_tdp(const float2 (&w)[W], int r, const float4 *A, const float4 *B)
{
    constexpr int K = FD / 2;
    float4 u, v;
    if (GUARD) { u = entry(A); v = entry(B); }
    float2 d = make_float2(0.f, 0.f);
#pragma unroll
    for (int k = 1; k <= K; ++k) {
        d = fma2(dup2(GUARD ? v4k(u, k) : cf<FD>(k)), w[r + K - k], d);
        d = fma2(dup2(GUARD ? -v4k(v, k) : -cf<FD>(k)), w[r + K + k - 1], d);
    }
    return d;
}
template <int FD, bool GUARD, int W>
__device__ __forceinline__ float2 z_tdm(const float2 (&w)[W], int r, const float4 *A, const float4 *B)
{
    constexpr int K = FD / 2;
    float4 u, v;
    if (GUARD) { u = entry(A); v = entry(B); }
    float2 d = make_float2(0.f, 0.f);
#pragma unroll
    for (int k = 1; k <= K; ++k) {
        d = fma2(dup2(GUARD ? v4k(u, k) : cf<FD>(k)), w[r + K - k + 1], d);
        d = fma2(dup2(GUARD ? -v4k(v, k) : -cf<FD>(k)), w[r + K + k], d);
    }
    return d;
}

// z window of the pair
template <int W, int RPT>
__device__ __forceinline__ void zwin(float2 (&w)[W], const float *s, int ty, int tx)
{
#pragma unroll
    for (int m = 0; m < W; ++m) w[m] = *reinterpret_cast<const float2 *>(s + (ty * RPT + m) * SW4 + XO4 + 2 * tx);
}
__device__ __forceinline__ float2 pair_at(const float *p) { return *reinterpret_cast<const float2 *>(p); }

// ------------------------------------------------------------- work and pipeline
//
// A block takes a run of shots of one tile (an item is one of them), and
// loads the tile's constants once.
//
// The items' boxes arrive by TMA in a ring of NST stages.  Every warp waits
// for a stage by itself and arrives at the stage's second barrier once it has
// read it; the last warp to arrive refills the stage with the item NST further
// on.  No barrier joins the warps of a block.

struct Run {
    uint32_t tile;      // row << 16 | column
    int q, shot, n;     // number of the run, its first shot, its shots
    __device__ __forceinline__ int j0() const { return (tile & 0xffffu) * TX4; }
    __device__ __forceinline__ int i0(int tzh) const { return (tile >> 16) * tzh; }
    __device__ __forceinline__ int number(const Work &w) const { return (tile >> 16) * w.ntx + (tile & 0xffffu); }
};

// ring state in shared memory
template <int NST> struct Ring {
    uint64_t full[NST];     // a stage's copies have landed
    uint64_t empty[NST];    // every warp has read the stage
    uint32_t issued;        // items issued by this block
};

// a wait ran out at the block's item `it`: record it and wait (bounded) for
// every copy issued that this warp has not seen land.  A warp sees land or
// waits here for all that it issued itself, so the block never exits under a
// copy in flight; and as this warp leaves no stage from `it` on, the others
// issue at most one round more.
template <int NST> __device__ __forceinline__ void ring_abort(Ring<NST> *r, int it, int *status)
{
    if (threadIdx.x == 0) {
        atomicOr(status, ST_TIMEOUT3);
        const int n = (int)*(volatile uint32_t *)&r->issued;
        for (int k = it; k < n; ++k) mbar_wait_bounded(r->full + k % NST, (k / NST) & 1, WAIT3);
    }
    __syncwarp();
}

// this warp has read its item from stage st (round parity ph): true in lane 0
// of the last warp out, which then issues the item NST further on.  The
// arrivals release the warps' reads and the wait, which finds the phase
// complete, acquires them, so the copy comes after all of them.
template <int NST> __device__ __forceinline__ bool ring_leave(Ring<NST> *r, int st, int ph, bool more)
{
    __syncwarp();
    if (threadIdx.x != 0 || !more) return false;
    if (mbar_arrive_pending(r->empty + st) != 1 || !mbar_try_wait(r->empty + st, ph)) return false;
    asm volatile("red.relaxed.cta.shared::cta.add.u32 [%0], 1;" ::"r"(smem_u32(&r->issued)) : "memory");
    return true;
}

// stage sizes (floats) and ring depths: as many stages as two blocks an SM
// have room for
template <int FD, int R, int NW> struct Stage {
    using T = G4<FD, R, NW>;
    static constexpr int OWN2 = al32_3(2 * T::TZH * TX4), OWN3 = al32_3(3 * T::TZH * TX4);
    static constexpr int VEL = T::S3 + OWN2, STR = T::S2 + OWN3;
    // adjoint stages: four planes, each a copy of its own that starts on 128
    // bytes, then the own boxes; at FD 2 a plane's rows do not end on 128 bytes
    static constexpr int SNA = al32_3(T::SN), SOWN = 4 * SNA;
    static constexpr int ADA = SOWN + OWN2, ADB = SOWN + 2 * OWN3;
    static_assert(SNA % 32 == 0 && SOWN >= 3 * SNA + T::SN && ADA >= SOWN + 2 * T::TZH * TX4 &&
                      ADB >= SOWN + OWN3 + 3 * T::TZH * TX4,
                  "a stage holds all that its copies write");
    static constexpr int fit(int floats) { return imin(4, (113 * 1024 - 256 - (int)sizeof(AdjTab)) / (floats * 4)); }
    static constexpr int imin(int a, int b) { return a < b ? a : b; }
    static constexpr int NVEL = fit(VEL), NSTR = fit(STR), NADA = fit(ADA), NADB = fit(ADB);
    // stages, coefficient table, ring
    static constexpr size_t bytes(int floats, int nst) { return (size_t)floats * nst * 4 + sizeof(AdjTab) + 16 * nst + 16; }
};

// ------------------------------------------------------------- guarded paths
//
// Which work a cell needs is decided per tile for the columns and per warp
// (RPT rows) for the rows: a warp takes the unguarded path when neither a
// slice mask nor a C-PML strip applies to its cells.  GUARD rows test the
// masks of their row, uniform over the warp, XB tiles (the first and last of
// a tile row) also those of their columns.

// columns [j0, j0 + TX4) clear of the `lo` first and `hi` last columns
__device__ __forceinline__ bool cols_plain(const Geo &g, int j0, int lo, int hi)
{
    return j0 >= lo && j0 + TX4 <= g.nx - hi;
}
// rows [a, b] clear of the `lo` first and `hi` last rows
__device__ __forceinline__ bool rows_plain(const Geo &g, int a, int b, int lo, int hi)
{
    return a >= lo && b < g.nz - hi;
}

// x-strip indices of columns jb, jb + 1; outside the strips and the grid the
// index of the row's last memory, which stays zero
__device__ __forceinline__ int2 xstrip_pair(const Geo &g, int jb)
{
    const int a = jb < g.nx ? xstrip_index(g, jb) : -1, b = jb + 1 < g.nx ? xstrip_index(g, jb + 1) : -1;
    return make_int2(a < 0 ? g.xs_n - 1 : a, b < 0 ? g.xs_n - 1 : b);
}

// a 16-byte C-PML entry (constant during a launch)
__device__ __forceinline__ float4 ldt(const float4 *p) { return __ldg(p); }

// The C-PML memories of a warp's rows (two arrays a, b) and coefficients, on
// their way into L1 before the warp waits for its stage: loaded into registers
// there they would be live across the stencils, loaded row by row from L2 each
// row would wait for its own.
__device__ __forceinline__ void prefetch_l1(const void *p) { asm volatile("prefetch.global.L1 [%0];" ::"l"(p)); }
template <int RPT>
__device__ __forceinline__ void prefetch_x(const Geo &g, int iw, int2 xs, const float *a, const float *b)
{
    const int x = min(xs.x, xs.y);
    if (x == g.xs_n - 1) return;
#pragma unroll
    for (int r = 0; r < RPT; ++r) {
        const int o = min(iw + r, g.nz - 1) * g.xs_n + x;
        prefetch_l1(a + o);
        prefetch_l1(b + o);
    }
}
template <int RPT>
__device__ __forceinline__ void prefetch_z(const Geo &g, int iw, int jb, const float *a, const float *b)
{
#pragma unroll
    for (int r = 0; r < RPT; ++r) {
        const int zs = zstrip_index(g, min(iw + r, g.nz - 1));
        if (zs < 0 || jb >= g.nx) continue;
        prefetch_l1(a + zs * g.P + jb);
        prefetch_l1(b + zs * g.P + jb);
    }
}
// a row's memories of the columns jb, jb + 1 in an x strip.  Outside the strips
// the coefficients are (0, 0, 1) and the memory 0, not some other column's: that
// could be infinite, and 0 times it is no zero.
__device__ __forceinline__ float2 mem_x(const float *row, int2 xs) { return make_float2(row[xs.x], row[xs.y]); }

// C-PML (fwi/forward.py:107-112: psi' = b psi + a D, D' = D/k + psi') of a pair
// of x-derivatives on one row (c0, c1: the columns' (b, a, 1/k),
// old: their memories, p: the memory's row) / of z-derivatives (p: the pair's memory)
__device__ __forceinline__ void pml_x2(const Geo &g, float2 &d, const float4 &c0, const float4 &c1, int2 xs, float2 old, float *p)
{
    const float p0 = c0.x * old.x + c0.y * d.x, p1 = c1.x * old.y + c1.y * d.y;
    if (xs.x < g.xs_n - 1) p[xs.x] = p0;
    if (xs.y < g.xs_n - 1) p[xs.y] = p1;
    d = make_float2(d.x * c0.z + p0, d.y * c1.z + p1);
}
__device__ __forceinline__ void pml_z2(float2 &d, const float4 &zc, float2 old, float *p)
{
    const float2 pn = fma2(dup2(zc.x), old, mul2(dup2(zc.y), d));
    *reinterpret_cast<float2 *>(p) = pn;
    d = fma2(d, dup2(zc.z), pn);
}
// transposed C-PML of a pair (the memory kept as phi = psi / (dt / d)): x' = (1/k + a) x + a phi, phi' = b (x + phi)
__device__ __forceinline__ void adj_x2(const Geo &g, float2 &v, const float4 &c0, const float4 &c1, int2 xs, float2 phi, float *p)
{
    if (xs.x < g.xs_n - 1) p[xs.x] = c0.x * (v.x + phi.x);
    if (xs.y < g.xs_n - 1) p[xs.y] = c1.x * (v.y + phi.y);
    v = make_float2((c0.z + c0.y) * v.x + c0.y * phi.x, (c1.z + c1.y) * v.y + c1.y * phi.y);
}
__device__ __forceinline__ void adj_z2(float2 &v, const float4 &zc, float2 phi, float *p)
{
    *reinterpret_cast<float2 *>(p) = mul2(dup2(zc.x), add2(v, phi));
    v = fma2(dup2(zc.z + zc.y), v, mul2(dup2(zc.y), phi));
}
// the same at one cell (receiver injection): a value s added before the transform
__device__ __forceinline__ float adj_inject(float s, const float4 &c, bool strip, float *p)
{
    if (strip) atomicAdd(p, c.x * s);
    return strip ? (c.z + c.y) * s : s;
}

// add v to component k (0 or 1) of a pair, nothing for any other k
__device__ __forceinline__ void add_at(float2 &p, int k, float v)
{
    if (k == 0) p.x = p.x + v;
    if (k == 1) p.y = p.y + v;
}
// store a pair (XB: only its first column where it is the row's last)
template <bool XB> __device__ __forceinline__ void store_pair(float *p, float2 v, int left)
{
    if (!XB || left >= 2) *reinterpret_cast<float2 *>(p) = v;
    else if (left == 1) *p = v.x;
}


// a material of columns jb, jb + 1 of row i (its rows start on 128 bytes, jb
// is even).  Off the grid it is some other cell's: nothing computed there is
// kept, and a select on the loaded value would wait for it.
__device__ __forceinline__ float2 mat_pair(const Geo &g, const float *a, int i, int jb)
{
    return *reinterpret_cast<const float2 *>(a + (long long)min(i, g.nz - 1) * g.P + (jb < g.nx ? jb : 0));
}

// start of a launch: the block's run, the ring's barriers, the first NST items
// on their way (by the first warp's first lane), and meanwhile, by the other
// warps, the coefficient tables.  All that reads what the launch before wrote
// comes after the dependency wait: where a launch may start before its
// predecessor ends, only the part before the wait overlaps.
template <int NST, class Issue, class Fill>
__device__ __forceinline__ void ring_start(Ring<NST> *ring, const Work &w, Run &c, Issue issue, Fill fill_tab)
{
    if (w.single) {
        // one item a block, the grid being (tile columns, tile rows, shots):
        // nothing to look up before the first copy can start
        c.tile = blockIdx.y << 16 | blockIdx.x;
        c.q = w.run0 + blockIdx.z;
        c.shot = w.s0 + c.q;
        c.n = 1;
    } else {
        const unsigned pos = blockIdx.x / (unsigned)w.runs;
        c.tile = __ldg(w.order + pos);
        c.q = w.run0 + (int)(blockIdx.x - pos * w.runs);
        c.shot = w.first(c.q);
        c.n = w.base + (c.q < w.longer ? 1 : 0);
    }
    const bool lead = threadIdx.x == 0 && threadIdx.y == 0;
    if (lead) {
        for (int b = 0; b < NST; ++b) {
            mbar_init(ring->full + b, 1);
            mbar_init(ring->empty + b, blockDim.y);
        }
        ring->issued = min(NST, c.n);
        fence_async_shared();
    }
    if (threadIdx.y > 0) fill_tab((threadIdx.y - 1) * TX + threadIdx.x);
    grid_dependency_start();
    grid_dependency_wait();
    if (lead) {
#pragma unroll 1
        for (int b = 0; b < NST && b < c.n; ++b) issue(c.shot + b, b);
    }
    __syncthreads();
}

// ------------------------------------------------------------- forward: velocities

template <int FD, int RPT, int NW>
__global__ void __launch_bounds__(TX *NW, NW == 8 ? 2 : 1)
    st_fwd_vel(const __grid_constant__ Geo g, const __grid_constant__ Mat m, const __grid_constant__ Shots sh, float *F,
               float *PX, float *PZ, int n, const __grid_constant__ Work w, int *status,
               const __grid_constant__ CUtensorMap tmS, const __grid_constant__ CUtensorMap tmUo)
{
    using T = G4<FD, RPT, NW>;
    using Sg = Stage<FD, RPT, NW>;
    constexpr int K = T::K, SN = T::SN, STG = Sg::VEL, NST = Sg::NVEL, PL = T::TZH * TX4;
    extern __shared__ __align__(128) float sm[];
    FwdTab *tab = reinterpret_cast<FwdTab *>(sm + STG * NST);
    Ring<NST> *ring = reinterpret_cast<Ring<NST> *>(tab + 1);
    const int tx = threadIdx.x, ty = threadIdx.y;
    Run c;
    auto issue = [&](int s, int st) {
        mbar_arrive_expect_tx(ring->full + st, (3 * SN + 2 * PL) * 4);
        tma_load_4d(sm + st * STG, &tmS, ring->full + st, c.j0() - XO4, c.i0(T::TZH) - K, F_EX, s);
        tma_load_4d(sm + st * STG + T::S3, &tmUo, ring->full + st, c.j0(), c.i0(T::TZH), F_U, s);
    };
    ring_start(ring, w, c, issue, [&](int i) { fill<FD>(tab, g, i); });
    // columns (of the tile) and rows (of this warp) where no slice mask and no
    // C-PML strip applies; the strips are at least K wide, so they hold the
    // masked columns and rows except those below a free surface
    const int jb = c.j0() + 2 * tx, iw = c.i0(T::TZH) + ty * RPT;
    const bool xin = cols_plain(g, c.j0(), g.pad, g.pad);
    const bool zin = rows_plain(g, iw, iw + RPT - 1, g.fs ? K : g.pad, g.pad);
    float2 B[RPT];
#pragma unroll
    for (int r = 0; r < RPT; ++r) B[r] = mat_pair(g, m.B, iw + r, jb);
    for (int it = 0; it < c.n; ++it) {
        const int st = it % NST, ph = it / NST & 1;   // stage, parity of its round
        const int s = c.shot + it;
        const int4 src = __ldg(sh.pos + s);
        const float *S = sm + st * STG, *own = S + T::S3;   // own: [U, V][TZH][TX4] of the tile's own cells
        float *U = F + ((long long)s * F_N + F_U) * g.fstride;
        float *V = F + ((long long)s * F_N + F_V) * g.fstride;
        float *pSXX = px_ptr(g, PX, s, PX_SXX), *pSXZx = px_ptr(g, PX, s, PX_SXZ);
        float *pSXZz = pz_ptr(g, PZ, s, PZ_SXZ), *pSZZ = pz_ptr(g, PZ, s, PZ_SZZ);
        auto rows = [&](auto gd, auto xb) -> bool {
            constexpr bool GUARD = decltype(gd)::value, XB = decltype(xb)::value;
            int2 xs = make_int2(g.xs_n - 1, g.xs_n - 1);
            const int e0 = XB ? tab_at(jb, g.nx) : 0, e1 = XB ? tab_at(jb + 1, g.nx) : 0;   // the columns' table entries
            if (XB) {
                xs = xstrip_pair(g, jb);
                prefetch_x<RPT>(g, iw, xs, pSXX, pSXZx);
                prefetch_l1(g.pmx + jb);
            }
            if (GUARD) {
                prefetch_z<RPT>(g, iw, jb, pSXZz, pSZZ);
                prefetch_l1(g.pmz + iw);
            }
            if (!mbar_wait_bounded(ring->full + st, ph, g.wait_polls)) return false;
            float2 dzxz[RPT], dzz[RPT];
            {
                float2 wn[T::W];
                zwin<T::W, RPT>(wn, S + 2 * SN, ty, tx);
#pragma unroll
                for (int r = 0; r < RPT; ++r) {
                    dzxz[r] = z_dm<FD, GUARD>(wn, r, &tab->z[1][tab_at(iw + r, g.nz)]);
                    if (GUARD && g.fs && iw + r == 0) dzxz[r] = mul2(dup2(2.f * cf<FD>(1)), wn[r + K]);
                }
                zwin<T::W, RPT>(wn, S + SN, ty, tx);
#pragma unroll
                for (int r = 0; r < RPT; ++r) dzz[r] = z_dp<FD, GUARD>(wn, r, &tab->z[0][tab_at(iw + r, g.nz)]);
            }
#pragma unroll
            for (int r = 0; r < RPT; ++r) {
                const int i = iw + r, zr = ty * RPT + r, q = (zr + K) * SW4 + XO4 + 2 * tx;
                if (GUARD && i >= g.nz - 1) continue;   // row nz - 1 keeps its value
                float a[10];
                xrow(a, S, q);
                float2 dxx = x_dp<FD, XB>(a, tab->x[0], e0, e1);
                xrow(a, S + 2 * SN, q);
                float2 dxxz = x_dm<FD, XB>(a, tab->x[1], e0, e1);
                const float2 u2 = pair_at(own + zr * TX4 + 2 * tx), v2 = pair_at(own + PL + zr * TX4 + 2 * tx);
                if (XB) {
                    const float4 c0 = ldt(g.pmx + jb), c1 = ldt(g.pmx + jb + 1);
                    const float2 m0 = mem_x(pSXX + i * g.xs_n, xs), m1 = mem_x(pSXZx + i * g.xs_n, xs);
                    pml_x2(g, dxx, c0, c1, xs, m0, pSXX + i * g.xs_n);
                    pml_x2(g, dxxz, c0, c1, xs, m1, pSXZx + i * g.xs_n);
                }
                if (GUARD) {
                    const float4 zc = ldt(g.pmz + i);
                    const int zs = __float_as_int(zc.w);
                    if (zs >= 0 && (!XB || jb < g.nx)) {
                        const float2 m0 = pair_at(pSXZz + zs * g.P + jb), m1 = pair_at(pSZZ + zs * g.P + jb);
                        pml_z2(dzxz[r], zc, m0, pSXZz + zs * g.P + jb);
                        pml_z2(dzz[r], zc, m1, pSZZ + zs * g.P + jb);
                    }
                }
                const float2 bx = mul2(dup2(g.dtdx), B[r]), bz = mul2(dup2(g.dtdz), B[r]);
                float2 un = fma2(bz, dzxz[r], fma2(bx, dxx, u2));
                float2 vn = fma2(bz, dzz[r], fma2(bx, dxxz, v2));
                const long long o = (long long)i * g.P + jb;
                if (XB) {
                    // columns 0 and nx - 1 keep their value
                    if (jb < 1 || jb >= g.nx - 1) { un.x = u2.x; vn.x = v2.x; }
                    if (jb + 1 >= g.nx - 1) { un.y = u2.y; vn.y = v2.y; }
                }
                if (src.x == i && src.z == 0 && (!XB || (src.y >= 1 && src.y < g.nx - 1)))   // force source
                    add_at(vn, src.y - jb, sh.fcoef[s] * sh.wav[(long long)s * g.nt + n]);
                store_pair<XB>(U + o, un, g.nx - jb);
                store_pair<XB>(V + o, vn, g.nx - jb);
            }
            return true;
        };
        if (!(!xin ? rows(std::true_type{}, std::true_type{})
                   : !zin ? rows(std::true_type{}, std::false_type{}) : rows(std::false_type{}, std::false_type{}))) {
            ring_abort(ring, it, status);
            return;
        }
        if (ring_leave(ring, st, ph, it + NST < c.n)) issue(s + NST, st);
    }
}

// ------------------------------------------------------------- forward: stresses

template <int FD, int RPT, int NW, bool ENERGY>
__global__ void __launch_bounds__(TX *NW, NW == 8 ? 2 : 1)
    st_fwd_str(const __grid_constant__ Geo g, const __grid_constant__ Mat m, const __grid_constant__ Shots sh,
               const __grid_constant__ Recv rv, float *F, float *PX, float *PZ, int n, const __grid_constant__ Work w,
               const __grid_constant__ FwdOut out, const __grid_constant__ CUtensorMap tmV,
               const __grid_constant__ CUtensorMap tmSo)
{
    using T = G4<FD, RPT, NW>;
    using Sg = Stage<FD, RPT, NW>;
    constexpr int K = T::K, SN = T::SN, STG = Sg::STR, NST = Sg::NSTR, PL = T::TZH * TX4;
    extern __shared__ __align__(128) float sm[];
    FwdTab *tab = reinterpret_cast<FwdTab *>(sm + STG * NST);
    Ring<NST> *ring = reinterpret_cast<Ring<NST> *>(tab + 1);
    const int tx = threadIdx.x, ty = threadIdx.y;
    Run c;
    auto issue = [&](int s, int st) {
        mbar_arrive_expect_tx(ring->full + st, (2 * SN + 3 * PL) * 4);
        tma_load_4d(sm + st * STG, &tmV, ring->full + st, c.j0() - XO4, c.i0(T::TZH) - K, F_U, s);
        tma_load_4d(sm + st * STG + T::S2, &tmSo, ring->full + st, c.j0(), c.i0(T::TZH), F_EX, s);
    };
    ring_start(ring, w, c, issue, [&](int i) { fill<FD>(tab, g, i); });
    const int jb = c.j0() + 2 * tx, iw = c.i0(T::TZH) + ty * RPT;
    const bool xin = cols_plain(g, c.j0(), g.pad, g.pad);   // as in st_fwd_vel
    const bool zin = rows_plain(g, iw, iw + RPT - 1, g.fs ? K : g.pad, g.pad);
    const int r0 = rv.tile_start[c.number(w)], r1 = rv.tile_start[c.number(w) + 1];
    float2 ml2m[RPT], ml[RPT], mm[RPT];
    constexpr int RG = ENERGY ? RPT : 1;
    double eacc[RG][2];
#pragma unroll
    for (int r = 0; r < RPT; ++r) {
        ml2m[r] = mat_pair(g, m.L2M, iw + r, jb);
        ml[r] = mat_pair(g, m.L, iw + r, jb);
        mm[r] = mat_pair(g, m.M, iw + r, jb);
    }
#pragma unroll
    for (int r = 0; r < RG; ++r) eacc[r][0] = eacc[r][1] = 0.0;
    // energy sums of the run's shots
    auto leave = [&]() {
        if constexpr (ENERGY) {
#pragma unroll
            for (int r = 0; r < RG; ++r)
#pragma unroll
                for (int cc = 0; cc < 2; ++cc)
                    if (iw + r < g.nz && jb + cc < g.nx)
                        atomicAdd(out.energy + (long long)(iw + r) * g.nx + jb + cc, eacc[r][cc]);
        }
    };
    const float2 dtdx2 = dup2(g.dtdx), dtdz2 = dup2(g.dtdz);
    // history rows as float pairs when every pair starts on 8 bytes
    const bool hist2 = ((g.pad | g.nx_dom) & 1) == 0;
    for (int it = 0; it < c.n; ++it) {
        const int st = it % NST, ph = it / NST & 1;   // stage, parity of its round
        const int s = c.shot + it;
        const int4 src = __ldg(sh.pos + s);
        const float *S = sm + st * STG, *own = S + T::S2;   // own: [sxx, szz, sxz][TZH][TX4] of the tile's own cells
        float *sxx = F + ((long long)s * F_N + F_EX) * g.fstride;
        float *szz = F + ((long long)s * F_N + F_EZ) * g.fstride;
        float *sxz = F + ((long long)s * F_N + F_ES) * g.fstride;
        float *pDXU = px_ptr(g, PX, s, PX_DXU), *pDXV = px_ptr(g, PX, s, PX_DXV);
        float *pDZV = pz_ptr(g, PZ, s, PZ_DZV), *pDZU = pz_ptr(g, PZ, s, PZ_DZU);
        float *snap_s = out.snap ? out.snap + ((long long)s * out.slots + out.slot) * g.snf * g.nd : nullptr;
        auto rows = [&](auto gd, auto xb) -> bool {
            constexpr bool GUARD = decltype(gd)::value, XB = decltype(xb)::value;
            int2 xs = make_int2(g.xs_n - 1, g.xs_n - 1);
            const int e0 = XB ? tab_at(jb, g.nx) : 0, e1 = XB ? tab_at(jb + 1, g.nx) : 0;   // the columns' table entries
            if (XB) {
                xs = xstrip_pair(g, jb);
                prefetch_x<RPT>(g, iw, xs, pDXU, pDXV);
                prefetch_l1(g.pmx + jb);
            }
            if (GUARD) {
                prefetch_z<RPT>(g, iw, jb, pDZV, pDZU);
                prefetch_l1(g.pmz + iw);
            }
            if (!mbar_wait_bounded(ring->full + st, ph, g.wait_polls)) return false;
            float2 dzv_[RPT], dzu_[RPT];
            {
                float2 wn[T::W];
                zwin<T::W, RPT>(wn, S + SN, ty, tx);
#pragma unroll
                for (int r = 0; r < RPT; ++r) dzv_[r] = z_dm<FD, GUARD>(wn, r, &tab->z[1][tab_at(iw + r, g.nz)]);
                zwin<T::W, RPT>(wn, S, ty, tx);
#pragma unroll
                for (int r = 0; r < RPT; ++r) dzu_[r] = z_dp<FD, GUARD>(wn, r, &tab->z[0][tab_at(iw + r, g.nz)]);
            }
#pragma unroll
            for (int r = 0; r < RPT; ++r) {
                const int i = iw + r, zr = ty * RPT + r, q = (zr + K) * SW4 + XO4 + 2 * tx, qo = zr * TX4 + 2 * tx;
                if (GUARD && i >= g.nz) continue;
                const bool last = GUARD && i >= g.nz - 1;
                float a[10];
                // column 0 has no D- term, column nx - 1 no D+ term: their
                // derivatives and memories stay zero
                xrow(a, S, q);
                float2 dxu = x_dm<FD, XB>(a, tab->x[1], e0, e1);
                const float2 uu = make_float2(a[4], a[5]);
                xrow(a, S + SN, q);
                float2 dxv = x_dp<FD, XB>(a, tab->x[0], e0, e1);
                const float2 vv = make_float2(a[4], a[5]);
                float2 dzv = dzv_[r], dzu = dzu_[r];
                const float2 e1 = pair_at(own + qo), e2 = pair_at(own + PL + qo), e3 = pair_at(own + 2 * PL + qo);
                if (last) dxv = make_float2(0.f, 0.f);
                if (XB) {
                    const float4 c0 = ldt(g.pmx + jb), c1 = ldt(g.pmx + jb + 1);
                    const float2 m0 = mem_x(pDXU + i * g.xs_n, xs), m1 = mem_x(pDXV + i * g.xs_n, xs);
                    pml_x2(g, dxu, c0, c1, xs, m0, pDXU + i * g.xs_n);
                    if (!last) pml_x2(g, dxv, c0, c1, xs, m1, pDXV + i * g.xs_n);
                }
                if (GUARD) {
                    if (g.fs && i == 0) {
                        // the free surface fixes d(vz)/dz
                        dzv.x = ((!XB || jb < g.nx) ? m.Lr[jb] : 0.f) * dxu.x * g.dzdx;
                        dzv.y = ((!XB || jb + 1 < g.nx) ? m.Lr[jb + 1] : 0.f) * dxu.y * g.dzdx;
                    }
                    if (XB) {
                        if (jb >= g.nx - 1) dzv.x = 0.f;
                        if (jb + 1 >= g.nx - 1) dzv.y = 0.f;
                        if (jb < 1) dzu.x = 0.f;
                    }
                    const float4 zc = ldt(g.pmz + i);
                    const int zs = __float_as_int(zc.w);
                    if (zs >= 0 && (!XB || jb < g.nx)) {
                        const float2 m0 = pair_at(pDZV + zs * g.P + jb), m1 = pair_at(pDZU + zs * g.P + jb);
                        pml_z2(dzv, zc, m0, pDZV + zs * g.P + jb);
                        pml_z2(dzu, zc, m1, pDZU + zs * g.P + jb);
                    }
                }
                const float2 dex = mul2(dtdx2, dxu), dez = mul2(dtdz2, dzv);
                float2 des = mul2(dup2(0.5f), fma2(dtdx2, dxv, mul2(dtdz2, dzu)));
                if (last) des = make_float2(0.f, 0.f);
                if (XB) {
                    if (jb >= g.nx - 1) des.x = 0.f;
                    if (jb + 1 >= g.nx - 1) des.y = 0.f;
                }
                float2 axx = fma2(ml[r], dez, fma2(ml2m[r], dex, e1));
                float2 azz = fma2(ml2m[r], dez, fma2(ml[r], dex, e2));
                const float2 axz = fma2(mul2(dup2(2.f), mm[r]), des, e3);
                if (src.x == i && src.z == 1) {   // moment source
                    const int sj = src.y - jb;
                    const float stm = sh.wav[(long long)s * g.nt + n] * g.dt / sh.mcoef[s];
                    const float f = sj == 0 ? ml2m[r].x + ml[r].x : ml2m[r].y + ml[r].y;
                    add_at(axx, sj, f * stm);
                    add_at(azz, sj, f * stm);
                }
                const int pi = i - g.z0, pj = jb - g.pad;
                if (snap_s && (!GUARD || (pi >= 0 && pi < g.nz_dom))) {
                    float *sp = snap_s + (long long)pi * g.nx_dom + pj;
                    const bool px0 = !XB || (pj >= 0 && pj < g.nx_dom), px1 = !XB || (pj + 1 >= 0 && pj + 1 < g.nx_dom);
                    if (hist2) {
                        if (px0) {   // an even pair is inside or outside as a whole
                            __stcs(reinterpret_cast<float2 *>(sp), axx);
                            __stcs(reinterpret_cast<float2 *>(sp + g.nd), azz);
                            __stcs(reinterpret_cast<float2 *>(sp + 2 * g.nd), axz);
                            if (g.snf == 5) {   // velocities of this step (density gradient)
                                __stcs(reinterpret_cast<float2 *>(sp + 3 * g.nd), uu);
                                __stcs(reinterpret_cast<float2 *>(sp + 4 * g.nd), vv);
                            }
                        }
                    } else {
                        if (px0) {
                            __stcs(sp, axx.x); __stcs(sp + g.nd, azz.x); __stcs(sp + 2 * g.nd, axz.x);
                            if (g.snf == 5) { __stcs(sp + 3 * g.nd, uu.x); __stcs(sp + 4 * g.nd, vv.x); }
                        }
                        if (px1) {
                            __stcs(sp + 1, axx.y); __stcs(sp + g.nd + 1, azz.y); __stcs(sp + 2 * g.nd + 1, axz.y);
                            if (g.snf == 5) { __stcs(sp + 3 * g.nd + 1, uu.y); __stcs(sp + 4 * g.nd + 1, vv.y); }
                        }
                    }
                }
                if (GUARD && out.row0 && g.fs && i == 0) {
                    float *rp = out.row0 + ((long long)s * out.slots + out.slot_row0) * g.nx_dom + pj;
                    if (!XB || (pj >= 0 && pj < g.nx_dom)) rp[0] = dxu.x;
                    if (!XB || (pj + 1 >= 0 && pj + 1 < g.nx_dom)) rp[1] = dxu.y;
                }
                if (ENERGY) {
#pragma unroll
                    for (int cc = 0; cc < 2; ++cc) {
                        if (XB && jb + cc >= g.nx) continue;
                        float f;
                        if (out.energy_comp < 2) {
                            f = out.energy_comp == 0 ? f2c(uu, cc) : f2c(vv, cc);
                        } else {
                            float ex, ez, es;
                            strains_of(f2c(axx, cc), f2c(azz, cc), f2c(axz, cc), f2c(ml2m[r], cc), f2c(ml[r], cc),
                                       f2c(mm[r], cc), ex, ez, es);
                            f = out.energy_comp == 2 ? ex : ez;
                        }
                        eacc[r % RG][cc] += (double)f * (double)f;
                    }
                }
                const long long o = (long long)i * g.P + jb;
                store_pair<XB>(sxx + o, axx, g.nx - jb);
                store_pair<XB>(szz + o, azz, g.nx - jb);
                store_pair<XB>(sxz + o, axz, g.nx - jb);
            }
            return true;
        };
        if (!(!xin ? rows(std::true_type{}, std::true_type{})
                   : !zin ? rows(std::true_type{}, std::false_type{}) : rows(std::false_type{}, std::false_type{}))) {
            ring_abort(ring, it, out.status);
            return;
        }
        if (ring_leave(ring, st, ph, it + NST < c.n)) issue(s + NST, st);
        if (r1 > r0) {
            // receivers on this warp's rows, which its own lanes have just written
            __syncwarp();
            const float *U = F + ((long long)s * F_N + F_U) * g.fstride;
            const float *V = F + ((long long)s * F_N + F_V) * g.fstride;
            for (int qq = r0 + tx; qq < r1; qq += TX) {
                const int rid = rv.tile_rec[qq], ri = rv.rz[rid];
                if (ri < iw || ri >= iw + RPT) continue;
                const long long o = (long long)ri * g.P + rv.rx[rid];
                float ex, ez, es;
                strains_of(sxx[o], szz[o], sxz[o], m.L2M[o], m.L[o], m.M[o], ex, ez, es);
                const float v0 = U[o], v1 = V[o];
                float *dst = out.rec + (long long)s * 4 * g.nt * g.nrec + (long long)n * g.nrec + rid;
                dst[0] = v0;
                dst[(long long)g.nt * g.nrec] = v1;
                dst[2LL * g.nt * g.nrec] = ex;
                dst[3LL * g.nt * g.nrec] = ez;
                if (!(isfinite(v0) && isfinite(v1) && isfinite(ex) && isfinite(ez))) atomicOr(out.status, 1);
            }
        }
    }
    leave();
}

// ------------------------------------------------------------- adjoint
//
// The transposed C-PML acts on the values that a transposed stencil then
// gathers, so a reader next to a strip needs the image of its neighbours'
// cells.  The writer makes it: each strain (velocity) update, holding the new
// value and the memory of its own cells in registers, also stores the images
// that the next velocity (strain) update will differentiate, in arrays that
// cover only the cells some strip-touching box reads ([jl, jr) x [it, ib) is
// left out): x images in bands of columns, z images in bands of rows.  The
// memories are then private to a cell's owner, one copy each.

// does the staged box of a tile touch an x strip / a z strip
__device__ __forceinline__ bool box_x(const Geo &g, int j0)
{
    return j0 - XO4 < g.pad || j0 + TX4 + XO4 > g.nx - g.pad;
}
__device__ __forceinline__ bool box_z(const Geo &g, int i0, int tzh, int K)
{
    return i0 + tzh + K > g.nz - g.pad || (!g.fs && i0 - K < g.pad);
}
// place of column j / row i in the image bands
__device__ __forceinline__ int band_x(const Geo &g, int j) { return j < g.jl ? j : j - g.jr + g.jl; }
__device__ __forceinline__ int band(int i, int lo, int hi) { return i < lo ? i : i - hi + lo; }

// ------------------------------------------------------------- adjoint: P = B U_a, Q = B V_a

template <int FD, int RPT, int NW>
__global__ void __launch_bounds__(TX *NW, NW == 8 ? 2 : 1)
    st_adj_a(const __grid_constant__ Geo g, const __grid_constant__ Mat m, const __grid_constant__ Recv rv, float *A,
             float *PX, float *PZ, const __grid_constant__ Images im, int n, const __grid_constant__ Work w,
             const __grid_constant__ AdjIn in, int *status,
             const __grid_constant__ CUtensorMap tmE, const __grid_constant__ CUtensorMap tmPQo,
             const __grid_constant__ CUtensorMap tmX, const __grid_constant__ CUtensorMap tmZ)
{
    using T = G4<FD, RPT, NW>;
    using Sg = Stage<FD, RPT, NW>;
    constexpr int SNA = Sg::SNA, SOWN = Sg::SOWN;
    constexpr int K = T::K, SN = T::SN, STG = Sg::ADA, NST = Sg::NADA, PL = T::TZH * TX4;
    extern __shared__ __align__(128) float sm[];
    AdjTab *tab = reinterpret_cast<AdjTab *>(sm + STG * NST);
    Ring<NST> *ring = reinterpret_cast<Ring<NST> *>(tab + 1);
    const int tx = threadIdx.x, ty = threadIdx.y;
    // planes of the staged box: what the step differentiates.  Away from the
    // C-PML strips these are the strain adjoints themselves; where the box
    // touches a strip, their transposed-C-PML images (adj_b writes them), x
    // and z images separately, and the exz image for x is a plane of its own.
    Run c;
    auto issue = [&](int s, int st) {
        const bool bx = box_x(g, c.j0()), bz = box_z(g, c.i0(T::TZH), T::TZH, K);
        constexpr int PB = SN * 4, OB = 2 * T::TZH * TX4 * 4;
        uint64_t *bar = ring->full + st;
        float *d = sm + st * STG;
        const int x = c.j0() - XO4, y = c.i0(T::TZH) - K;
        const int xi = x >= g.jr ? x - g.jr + g.jl : x, yi = y >= g.iba ? y - g.iba + g.ita : y;
        mbar_arrive_expect_tx(bar, (bx || bz ? 4 : 3) * PB + OB);
        if (bx) tma_load_4d(d, &tmX, bar, xi, y, 0, s);
        else tma_load_4d(d, &tmE, bar, x, y, F_EX, s);
        if (bz) {
            tma_load_4d(d + SNA, &tmZ, bar, x, yi, 0, s);
            tma_load_4d(d + 2 * SNA, &tmZ, bar, x, yi, 1, s);
        } else {
            tma_load_4d(d + SNA, &tmE, bar, x, y, F_EZ, s);
            tma_load_4d(d + 2 * SNA, &tmE, bar, x, y, F_ES, s);
        }
        if (bx) tma_load_4d(d + 3 * SNA, &tmX, bar, xi, y, 1, s);
        else if (bz) tma_load_4d(d + 3 * SNA, &tmE, bar, x, y, F_ES, s);
        tma_load_4d(d + SOWN, &tmPQo, bar, c.j0(), c.i0(T::TZH), F_U, s);
    };
    ring_start(ring, w, c, issue, [&](int i) { fill<FD>(tab, g, i, 0); });
    // transposed masks reach 2K - 1 (low edge) and 2K (high edge) cells inwards
    const int mlo = max(g.pad, 2 * K - 1), mhi = max(g.pad, 2 * K);
    const float hdtdz = 0.5f * g.dtdz, hdtdx = 0.5f * g.dtdx;
    const int jb = c.j0() + 2 * tx, iw = c.i0(T::TZH) + ty * RPT;
    const bool xin = cols_plain(g, c.j0(), mlo, mhi);
    const bool zin = rows_plain(g, iw, iw + RPT - 1, g.fs ? 2 * K - 1 : mlo, mhi);
    const bool bx = box_x(g, c.j0()), bz = box_z(g, c.i0(T::TZH), T::TZH, K);
    const bool xband = jb < g.nx && (jb < g.jl || jb >= g.jr), zband = iw < g.itb || iw + RPT > g.ibb;
    const int r0 = rv.tile_start[c.number(w)], r1 = rv.tile_start[c.number(w) + 1];
    float2 Bc[RPT];
#pragma unroll
    for (int r = 0; r < RPT; ++r) Bc[r] = mat_pair(g, m.B, iw + r, jb);
    for (int it = 0; it < c.n; ++it) {
        const int st = it % NST, ph = it / NST & 1;   // stage, parity of its round
        const int s = c.shot + it;
        const float *S = sm + st * STG;
        const float *own = S + SOWN;   // [P, Q][TZH][TX4] of the tile's own cells
        float *Pp = A + ((long long)s * F_N + F_U) * g.fstride;
        float *Qp = A + ((long long)s * F_N + F_V) * g.fstride;
        float *iXX = im.xb + (long long)s * 2 * g.txs, *iXXZ = iXX + g.txs;
        float *iZXZ = im.zb + (long long)s * 2 * g.tzs, *iZZ = iZXZ + g.tzs;
        const float *aDxU = S, *aDzV = S + SNA, *aDzU = S + 2 * SNA, *aDxV = (bx || bz) ? S + 3 * SNA : aDzU;
        float *fXX = px_ptr(g, PX, s, PX_NFWD + PXA_XX), *fXXZ = px_ptr(g, PX, s, PX_NFWD + PXA_XXZ);
        float *fZXZ = pz_ptr(g, PZ, s, PZ_NFWD + PZA_ZXZ), *fZZ = pz_ptr(g, PZ, s, PZ_NFWD + PZA_ZZ);
        auto rows = [&](auto gd, auto xb) -> bool {
            constexpr bool GUARD = decltype(gd)::value, XB = decltype(xb)::value;
            int2 xs = make_int2(g.xs_n - 1, g.xs_n - 1);
            const int e0 = XB ? tab_at(jb, g.nx) : 0, e1 = XB ? tab_at(jb + 1, g.nx) : 0;   // the columns' table entries
            if (XB) {
                xs = xstrip_pair(g, jb);
                prefetch_x<RPT>(g, iw, xs, fXX, fXXZ);
                prefetch_l1(g.pmx + jb);
            }
            if (GUARD) {
                prefetch_z<RPT>(g, iw, jb, fZXZ, fZZ);
                prefetch_l1(g.pmz + iw);
            }
            if (!mbar_wait_bounded(ring->full + st, ph, g.wait_polls)) return false;
            float2 zu_[RPT], zv_[RPT];
            {
                float2 wn[T::W];
                zwin<T::W, RPT>(wn, aDzU, ty, tx);
#pragma unroll
                for (int r = 0; r < RPT; ++r) zu_[r] = z_tdp<FD, GUARD>(wn, r, &tab->z[0][tab_at(iw + r, g.nz)], &tab->z[1][tab_at(iw + r, g.nz)]);
                zwin<T::W, RPT>(wn, aDzV, ty, tx);
#pragma unroll
                for (int r = 0; r < RPT; ++r) zv_[r] = z_tdm<FD, GUARD>(wn, r, &tab->z[2][tab_at(iw + r, g.nz)], &tab->z[3][tab_at(iw + r, g.nz)]);
            }
#pragma unroll
            for (int r = 0; r < RPT; ++r) {
                const int i = iw + r, zr = ty * RPT + r, q = (zr + K) * SW4 + XO4 + 2 * tx;
                if (GUARD && i >= g.nz) continue;
                const bool last = GUARD && i >= g.nz - 1;
                float a[10];
                xrow(a, aDxU, q);
                if (GUARD && g.fs && i == 0 && !bx) {
                    // free surface: d(vz)/dz is d(vx)/dx times Lr there, so
                    // exx_a receives Lr ezz_a (the x images already hold it)
                    float az[10];
                    xrow(az, aDzV, q);
#pragma unroll
                    for (int k = 0; k < 10; ++k) a[k] = m.Lr[jb - 4 + k] * az[k] + a[k];
                }
                const float2 tdm = x_tdm<FD, XB>(a, tab->x[2], tab->x[3], e0, e1);
                xrow(a, aDxV, q);
                float2 tdp = x_tdp<FD, XB>(a, tab->x[0], tab->x[1], e0, e1), zu = zu_[r], zv = zv_[r];
                const float2 p2 = pair_at(own + zr * TX4 + 2 * tx), q2 = pair_at(own + PL + zr * TX4 + 2 * tx);
                if (last) tdp = make_float2(0.f, 0.f);
                if (XB) {
                    if (jb < 1 || jb >= g.nx - 1) zu.x = 0.f;
                    if (jb + 1 >= g.nx - 1) zu.y = 0.f;
                    if (jb >= g.nx - 1) zv.x = 0.f;
                    if (jb + 1 >= g.nx - 1) zv.y = 0.f;
                }
                const float2 gu = fma2(dup2(g.dtdx), tdm, mul2(dup2(hdtdz), zu));
                const float2 gv = fma2(dup2(g.dtdz), zv, mul2(dup2(hdtdx), tdp));
                const float2 np = fma2(Bc[r], gu, p2), nq = fma2(Bc[r], gv, q2);
                if (GUARD && in.want_exact && g.fs && i == 0) {
                    // dJ/dLr on the free-surface row
#pragma unroll
                    for (int cc = 0; cc < 2; ++cc) {
                        const int j = jb + cc, pj = j - g.pad;
                        if (pj >= 0 && pj < g.nx_dom && j < g.nx - 1) {
                            const float du = in.row0[((long long)s * in.slots + in.slot) * g.nx_dom + pj];
                            in.accLr[(long long)s * g.nx_dom + pj] += (double)(g.dtdz * aDzV[q + cc]) * (double)du * (double)g.dzdx;
                        }
                    }
                }
                const long long o = (long long)i * g.P + jb;
                store_pair<XB>(Pp + o, np, g.nx - jb);
                store_pair<XB>(Qp + o, nq, g.nx - jb);
                if (xband || zband) {
                    // images for the strain update, which reads P and Q on [0, nz - 1) x [1, nx - 1) only
                    float2 pv = np, qv = nq;
                    if (last) pv = qv = make_float2(0.f, 0.f);
                    if (XB) {
                        if (jb < 1 || jb >= g.nx - 1) pv.x = qv.x = 0.f;
                        if (jb + 1 >= g.nx - 1) pv.y = qv.y = 0.f;
                    }
                    if (xband) {
                        float2 vXX = pv, vXXZ = qv;
                        if (XB) {
                            const float4 c0 = ldt(g.pmx + jb), c1 = ldt(g.pmx + jb + 1);
                            const float2 m0 = mem_x(fXX + i * g.xs_n, xs), m1 = mem_x(fXXZ + i * g.xs_n, xs);
                            adj_x2(g, vXX, c0, c1, xs, m0, fXX + i * g.xs_n);
                            adj_x2(g, vXXZ, c0, c1, xs, m1, fXXZ + i * g.xs_n);
                        }
                        const long long b = (long long)i * g.wxp + band_x(g, jb);
                        *reinterpret_cast<float2 *>(iXX + b) = vXX;
                        *reinterpret_cast<float2 *>(iXXZ + b) = vXXZ;
                    }
                    if ((i < g.itb || i >= g.ibb) && (!XB || jb < g.nx)) {
                        float2 vZXZ = pv, vZZ = qv;
                        if (GUARD) {
                            const float4 zc = ldt(g.pmz + i);
                            const int zs = __float_as_int(zc.w);
                            if (zs >= 0) {
                                const float2 m0 = pair_at(fZXZ + zs * g.P + jb), m1 = pair_at(fZZ + zs * g.P + jb);
                                adj_z2(vZXZ, zc, m0, fZXZ + zs * g.P + jb);
                                adj_z2(vZZ, zc, m1, fZZ + zs * g.P + jb);
                            }
                        }
                        const long long b = (long long)band(i, g.itb, g.ibb) * g.P + jb;
                        *reinterpret_cast<float2 *>(iZXZ + b) = vZXZ;
                        *reinterpret_cast<float2 *>(iZZ + b) = vZZ;
                    }
                }
            }
            return true;
        };
        if (!(!xin ? rows(std::true_type{}, std::true_type{})
                   : !zin ? rows(std::true_type{}, std::false_type{}) : rows(std::false_type{}, std::false_type{}))) {
            ring_abort(ring, it, status);
            return;
        }
        if (ring_leave(ring, st, ph, it + NST < c.n)) issue(s + NST, st);
        if (r1 > r0) {
            // receivers on this warp's rows, whose cells its own lanes have just written
            __syncwarp();
            for (int qq = r0 + tx; qq < r1; qq += TX) {
                const int rid = rv.tile_rec[qq], i = rv.rz[rid], j = rv.rx[rid];
                if (i < iw || i >= iw + RPT) continue;
                const long long o = (long long)i * g.P + j;
                const float *src = in.rec_adj + (long long)s * 4 * g.nt * g.nrec + (long long)n * g.nrec + rid;
                const float b = m.B[o], dp = b * src[0], dq = b * src[(long long)g.nt * g.nrec];
                atomicAdd(Pp + o, dp);
                atomicAdd(Qp + o, dq);
                if (i >= g.nz - 1 || j < 1 || j >= g.nx - 1) continue;
                if (j < g.jl || j >= g.jr) {
                    const int xs = xstrip_index(g, j);
                    const float4 xc = ldt(g.pmx + j);
                    const long long t = (long long)i * g.wxp + band_x(g, j);
                    atomicAdd(iXX + t, adj_inject(dp, xc, xs >= 0, fXX + i * g.xs_n + xs));
                    atomicAdd(iXXZ + t, adj_inject(dq, xc, xs >= 0, fXXZ + i * g.xs_n + xs));
                }
                if (i < g.itb || i >= g.ibb) {
                    const float4 zc = ldt(g.pmz + i);
                    const int zs = __float_as_int(zc.w);
                    const long long t = (long long)band(i, g.itb, g.ibb) * g.P + j, pz = (long long)zs * g.P + j;
                    atomicAdd(iZXZ + t, adj_inject(dp, zc, zs >= 0, fZXZ + pz));
                    atomicAdd(iZZ + t, adj_inject(dq, zc, zs >= 0, fZZ + pz));
                }
            }
        }
    }
}

// ------------------------------------------------------------- adjoint: strains + gradient

// receiver adjoints e1 (exx) and e3 (ezz) at cell (i, j) of shot s, after the
// cell's own update: into the strain adjoints and into the images st_adj_a
// differentiates
__device__ __forceinline__ void inject_strain(const Geo &g, const Mat &m, const Images &im, float *A, float *PX,
                                              float *PZ, int s, int i, int j, float e1, float e3)
{
    const long long o = (long long)i * g.P + j;
    atomicAdd(A + ((long long)s * F_N + F_EX) * g.fstride + o, e1);
    atomicAdd(A + ((long long)s * F_N + F_EZ) * g.fstride + o, e3);
    const float4 zc = ldt(g.pmz + i);
    const int zs = __float_as_int(zc.w);
    float d3 = e3;
    if (zs >= 0) d3 = adj_inject(e3, zc, true, pz_ptr(g, PZ, s, PZ_NFWD + PZA_DZV) + (long long)zs * g.P + j);
    if (i < g.ita || i >= g.iba)
        atomicAdd(im.za + (long long)s * 2 * g.tzs + (long long)band(i, g.ita, g.iba) * g.P + j, d3);
    if (j < g.jl || j >= g.jr) {
        float d1 = j >= 1 ? e1 : 0.f;
        if (g.fs && i == 0 && j < g.nx - 1) d1 = m.Lr[j] * d3 + d1;
        const int xs = xstrip_index(g, j);
        if (xs >= 0)
            d1 = adj_inject(d1, ldt(g.pmx + j), true, px_ptr(g, PX, s, PX_NFWD + PXA_DXU) + (long long)i * g.xs_n + xs);
        atomicAdd(im.xa + (long long)s * 2 * g.txs + (long long)i * g.wxp + band_x(g, j), d1);
    }
}

template <int FD, int RPT, int NW, bool EXACT, bool IMG, bool RHO>
__global__ void __launch_bounds__(TX *NW, NW == 8 ? 2 : 1)
    st_adj_b(const __grid_constant__ Geo g, const __grid_constant__ Mat m, const __grid_constant__ Shots sh,
             const __grid_constant__ Recv rv, float *A, float *PX, float *PZ, const __grid_constant__ Images im, int n,
             const __grid_constant__ Work w, const __grid_constant__ AdjOut o, int *status, const __grid_constant__ CUtensorMap tmP, const __grid_constant__ CUtensorMap tmEo,
             const __grid_constant__ CUtensorMap tmH, const __grid_constant__ CUtensorMap tmX,
             const __grid_constant__ CUtensorMap tmZ)
{
    // one history box per item from [shot][slot * snf + field][nz_dom][nx_dom]
    // at the tile's physical coordinates (cells outside arrive as 0): the
    // carry-in stresses of the exact gradient, or the carry-out ones of the
    // imaging condition
    const int hslot = EXACT ? o.slot_in : o.slot_img;
    const bool htma = (EXACT || IMG) && o.hist_tma && hslot >= 0;
    using T = G4<FD, RPT, NW>;
    using Sg = Stage<FD, RPT, NW>;
    constexpr int SNA = Sg::SNA, SOWN = Sg::SOWN;
    constexpr int K = T::K, SN = T::SN, STG = Sg::ADB, NST = Sg::NADB, PL = T::TZH * TX4;
    extern __shared__ __align__(128) float sm[];
    AdjTab *tab = reinterpret_cast<AdjTab *>(sm + STG * NST);
    Ring<NST> *ring = reinterpret_cast<Ring<NST> *>(tab + 1);
    const int tx = threadIdx.x, ty = threadIdx.y;
    // planes as in st_adj_a: P and Q, or their images where the box touches a
    // strip; the z image of P and the x image of Q are planes of their own
    Run c;
    auto issue = [&](int s, int st) {
        const bool bx = box_x(g, c.j0()), bz = box_z(g, c.i0(T::TZH), T::TZH, K);
        constexpr int PB = SN * 4, OB = 3 * T::TZH * TX4 * 4;
        uint64_t *bar = ring->full + st;
        float *d = sm + st * STG;
        const int x = c.j0() - XO4, y = c.i0(T::TZH) - K;
        const int xi = x >= g.jr ? x - g.jr + g.jl : x, yi = y >= g.ibb ? y - g.ibb + g.itb : y;
        mbar_arrive_expect_tx(bar, (bx || bz ? 4 : 2) * PB + OB + (htma ? OB : 0));
        if (bx) tma_load_4d(d, &tmX, bar, xi, y, 0, s);
        else tma_load_4d(d, &tmP, bar, x, y, F_U, s);
        if (bz) tma_load_4d(d + SNA, &tmZ, bar, x, yi, 1, s);
        else tma_load_4d(d + SNA, &tmP, bar, x, y, F_V, s);
        if (bx || bz) {
            if (bz) tma_load_4d(d + 2 * SNA, &tmZ, bar, x, yi, 0, s);
            else tma_load_4d(d + 2 * SNA, &tmP, bar, x, y, F_U, s);
            if (bx) tma_load_4d(d + 3 * SNA, &tmX, bar, xi, y, 1, s);
            else tma_load_4d(d + 3 * SNA, &tmP, bar, x, y, F_V, s);
        }
        tma_load_4d(d + SOWN, &tmEo, bar, c.j0(), c.i0(T::TZH), F_EX, s);
        if (htma)
            tma_load_4d_hint(d + SOWN + Sg::OWN3, &tmH, bar, c.j0() - g.pad, c.i0(T::TZH) - g.z0, hslot * g.snf, s, l2_evict_first());
    };
    ring_start(ring, w, c, issue, [&](int i) { fill<FD>(tab, g, i, 1); });
    const int mlo = max(g.pad, 2 * K - 1), mhi = max(g.pad, 2 * K);
    const float2 dtdx2 = dup2(g.dtdx), dtdz2 = dup2(g.dtdz);
    const bool hist2 = ((g.pad | g.nx_dom) & 1) == 0;   // history pairs start on 8 bytes
    constexpr int RE = EXACT ? RPT : 1, RI = IMG ? RPT : 1;
    const int jb = c.j0() + 2 * tx, iw = c.i0(T::TZH) + ty * RPT;
    const bool xin = cols_plain(g, c.j0(), mlo, mhi);
    const bool zin = rows_plain(g, iw, iw + RPT - 1, g.fs ? 2 * K - 1 : mlo, mhi);
    const bool bx = box_x(g, c.j0()), bz = box_z(g, c.i0(T::TZH), T::TZH, K);
    const bool xband = jb < g.nx && (jb < g.jl || jb >= g.jr), zband = iw < g.ita || iw + RPT > g.iba;
    const int r0 = n > 0 ? rv.tile_start[c.number(w)] : 0, r1 = n > 0 ? rv.tile_start[c.number(w) + 1] : 0;
    float2 ml2m[RPT], ml[RPT], mm[RPT];
#pragma unroll
    for (int r = 0; r < RPT; ++r) {
        ml2m[r] = mat_pair(g, m.L2M, iw + r, jb);
        ml[r] = mat_pair(g, m.L, iw + r, jb);
        mm[r] = mat_pair(g, m.M, iw + r, jb);
    }
    // sums over the run's shots, in FP32; over steps and runs in FP64 (the
    // reductions of leave() and k_finalize).  The exact gradient sums the
    // carry-in stresses s against the stress adjoints, sA = sum(s1 sxx_a + s2
    // szz_a), sB = sum(s2 sxx_a + s1 szz_a), sC = sum(s3 sxz_a); k_finalize
    // applies the strain-recovery factors.
    float2 sA[RE], sB[RE], sC[RE], glam[RI], gmu[RI];
    // density terms (history with velocities): dJ/dB of the exact gradient
    // and the rho term of the imaging formula
    constexpr int RB = (EXACT && RHO) ? RPT : 1, RR = (IMG && RHO) ? RPT : 1;
    float2 gB[RB], grl[RR];
    const float2 zero = make_float2(0.f, 0.f);
#pragma unroll
    for (int r = 0; r < RE; ++r) sA[r] = sB[r] = sC[r] = zero;
#pragma unroll
    for (int r = 0; r < RI; ++r) glam[r] = gmu[r] = zero;
#pragma unroll
    for (int r = 0; r < RB; ++r) gB[r] = zero;
#pragma unroll
    for (int r = 0; r < RR; ++r) grl[r] = zero;
    // the run's sums into its group's FP64 planes, to which no other block
    // adds at these cells: the order of the additions is that of the steps
    auto leave = [&]() {
        if (!EXACT && !IMG) return;
        double *base = o.acc + (long long)c.q * o.accp * g.nd;
#pragma unroll
        for (int r = 0; r < RPT; ++r)
#pragma unroll
            for (int cc = 0; cc < 2; ++cc) {
                const int pi = iw + r - g.z0, pj = jb + cc - g.pad;
                if (pi < 0 || pi >= g.nz_dom || pj < 0 || pj >= g.nx_dom) continue;
                double *acc = base + (long long)pi * g.nx_dom + pj;
                if (EXACT) {
                    atomicAdd(acc, (double)f2c(sC[r % RE], cc));
                    atomicAdd(acc + g.nd, (double)f2c(sB[r % RE], cc));
                    atomicAdd(acc + 2 * g.nd, (double)f2c(sA[r % RE], cc));
                }
                if (IMG) {
                    atomicAdd(acc + 3 * g.nd, (double)f2c(glam[r % RI], cc));
                    atomicAdd(acc + 4 * g.nd, (double)f2c(gmu[r % RI], cc));
                }
                if (EXACT && RHO) atomicAdd(acc + 5 * g.nd, (double)f2c(gB[r % RB], cc));
                if (IMG && RHO) atomicAdd(acc + 6 * g.nd, (double)f2c(grl[r % RR], cc));
            }
    };
    for (int it = 0; it < c.n; ++it) {
        const int st = it % NST, ph = it / NST & 1;   // stage, parity of its round
        const int s = c.shot + it;
        const float *S = sm + st * STG;
        const float *own = S + SOWN;             // [ex_a, ez_a, es_a][TZH][TX4] of the tile's own cells
        const float *hown = own + Sg::OWN3;      // [sxx, szz, sxz][TZH][TX4] of the history slot (htma)
        float *E = A + ((long long)s * F_N + F_EX) * g.fstride;   // exx_a, ezz_a, exz_a follow one another
        const float *Pp = A + ((long long)s * F_N + F_U) * g.fstride, *Qp = Pp + g.fstride;
        // history slots of the shot: carry-in, carry-out, and the next step's carry-out (none below 0)
        auto slot = [&](int k) { return o.snap + ((long long)s * o.slots + k) * g.snf * g.nd; };
        const int4 src = __ldg(sh.pos + s);
        const float *aXX = S, *aZZ = S + SNA;
        const float *aZXZ = (bx || bz) ? S + 2 * SNA : aXX, *aXXZ = (bx || bz) ? S + 3 * SNA : aZZ;
        auto rows = [&](auto gd, auto xb) -> bool {
            constexpr bool GUARD = decltype(gd)::value, XB = decltype(xb)::value;
            int2 xs = make_int2(g.xs_n - 1, g.xs_n - 1);
            const int e0 = XB ? tab_at(jb, g.nx) : 0, e1 = XB ? tab_at(jb + 1, g.nx) : 0;   // the columns' table entries
            if (XB) {
                xs = xstrip_pair(g, jb);
                prefetch_x<RPT>(g, iw, xs, px_ptr(g, PX, s, PX_NFWD + PXA_DXU), px_ptr(g, PX, s, PX_NFWD + PXA_DXV));
                prefetch_l1(g.pmx + jb);
            }
            if (GUARD) {
                prefetch_z<RPT>(g, iw, jb, pz_ptr(g, PZ, s, PZ_NFWD + PZA_DZV), pz_ptr(g, PZ, s, PZ_NFWD + PZA_DZU));
                prefetch_l1(g.pmz + iw);
            }
            if (!mbar_wait_bounded(ring->full + st, ph, g.wait_polls)) return false;
            // centred differences of P and Q for the imaging condition come
            // from the staged boxes where these hold P and Q themselves
            const bool boxed = IMG && !GUARD && !bx && !bz;
            float2 zp_[RPT], zm_[RPT], dzP[RI], dzQ[RI];
            {
                float2 wn[T::W];
                zwin<T::W, RPT>(wn, aZZ, ty, tx);
#pragma unroll
                for (int r = 0; r < RPT; ++r) {
                    zp_[r] = z_tdp<FD, GUARD>(wn, r, &tab->z[0][tab_at(iw + r, g.nz)], &tab->z[1][tab_at(iw + r, g.nz)]);
                    if (IMG) dzQ[r % RI] = sub2(wn[r + K + 1], wn[r + K - 1]);
                }
                zwin<T::W, RPT>(wn, aZXZ, ty, tx);
#pragma unroll
                for (int r = 0; r < RPT; ++r) {
                    zm_[r] = z_tdm<FD, GUARD>(wn, r, &tab->z[2][tab_at(iw + r, g.nz)], &tab->z[3][tab_at(iw + r, g.nz)]);
                    if (GUARD && g.fs && iw + r == 0) zm_[r] = fma2(dup2(2.f * cf<FD>(1)), wn[r + K], zm_[r]);
                    if (IMG) dzP[r % RI] = sub2(wn[r + K + 1], wn[r + K - 1]);
                }
            }
#pragma unroll
            for (int r = 0; r < RPT; ++r) {
                const int i = iw + r, zr = ty * RPT + r, q = (zr + K) * SW4 + XO4 + 2 * tx, qo = zr * TX4 + 2 * tx;
                if (GUARD && i >= g.nz) continue;
                const bool last = GUARD && i >= g.nz - 1;
                float a[10];
                xrow(a, aXX, q);
                float2 tdp = x_tdp<FD, XB>(a, tab->x[0], tab->x[1], e0, e1);
                const float2 dxP = make_float2(a[5] - a[3], a[6] - a[4]);
                xrow(a, aXXZ, q);
                float2 tdm = x_tdm<FD, XB>(a, tab->x[2], tab->x[3], e0, e1);
                const float2 dxQ = make_float2(a[5] - a[3], a[6] - a[4]);
                float2 zp = zp_[r], zm = zm_[r];
                const float2 ea = pair_at(own + qo), za = pair_at(own + PL + qo), sa = pair_at(own + 2 * PL + qo);
                if (last) tdp = tdm = make_float2(0.f, 0.f);
                if (XB) {
                    if (jb < 1 || jb >= g.nx - 1) zp.x = zm.x = 0.f;
                    if (jb + 1 >= g.nx - 1) zp.y = zm.y = 0.f;
                }
                const float2 sxx = mul2(dtdx2, tdp), szz = mul2(dtdz2, zp);
                const float2 sxz = fma2(dtdx2, tdm, mul2(dtdz2, zm));
                const float2 nex = fma2(ml[r], szz, fma2(ml2m[r], sxx, ea));
                const float2 nez = fma2(ml2m[r], szz, fma2(ml[r], sxx, za));
                const float2 nes = fma2(mul2(dup2(2.f), mm[r]), sxz, sa);
                if (src.x == i && (jb == src.y || jb + 1 == src.y)) {
                    // the source's cell
                    const int cc = src.y - jb;
                    const float e = f2c(ea, cc) + f2c(za, cc);
                    if (src.z == 0) {
                        if (o.src_a) o.src_a[(long long)s * g.nt + n] = g.dtdxdz * Qp[(long long)i * g.P + jb + cc];
                    } else {
                        if (o.src_a) o.src_a[(long long)s * g.nt + n] = (g.dt / sh.mcoef[s]) * e;
                        if (EXACT) {
                            // the moment factor's (L + M) term, one FP64 sum per shot
                            const double lm = sh.lm[s], wv = sh.wav[(long long)s * g.nt + n];
                            o.mterm[s] += -(wv * g.dt / ((double)sh.mcoef[s] / lm)) / (lm * lm) * (double)e;
                        }
                    }
                }
                const long long off = (long long)i * g.P + jb;
                store_pair<XB>(E + off, nex, g.nx - jb);
                store_pair<XB>(E + g.fstride + off, nez, g.nx - jb);
                store_pair<XB>(E + 2 * g.fstride + off, nes, g.nx - jb);
                if (xband || zband) {
                    // images for the velocity update
                    float2 vzv = nez, h = nes;
                    if (last) h = make_float2(0.f, 0.f);
                    if (XB) {
                        if (jb >= g.nx - 1) h.x = 0.f;
                        if (jb + 1 >= g.nx - 1) h.y = 0.f;
                    }
                    if (!XB || jb < g.nx) {
                        float2 vzu = h;
                        if (GUARD) {
                            const float4 zc = ldt(g.pmz + i);
                            const int zs = __float_as_int(zc.w);
                            if (zs >= 0) {
                                float *fDZV = pz_ptr(g, PZ, s, PZ_NFWD + PZA_DZV), *fDZU = pz_ptr(g, PZ, s, PZ_NFWD + PZA_DZU);
                                const float2 m0 = pair_at(fDZV + zs * g.P + jb), m1 = pair_at(fDZU + zs * g.P + jb);
                                adj_z2(vzv, zc, m0, fDZV + zs * g.P + jb);
                                adj_z2(vzu, zc, m1, fDZU + zs * g.P + jb);
                            }
                        }
                        if (i < g.ita || i >= g.iba) {
                            const long long b = (long long)band(i, g.ita, g.iba) * g.P + jb;
                            float *iz = im.za + (long long)s * 2 * g.tzs + b;
                            *reinterpret_cast<float2 *>(iz) = vzv;
                            *reinterpret_cast<float2 *>(iz + g.tzs) = vzu;
                        }
                    }
                    if (xband) {
                        float2 d = nex, v = h;
                        if (XB && jb < 1) d.x = 0.f;
                        if (GUARD && g.fs && i == 0) {
                            // the free surface's d(vz)/dz term (columns below nx - 1)
                            if (!XB || jb < g.nx - 1) d.x = m.Lr[jb] * vzv.x + d.x;
                            if (!XB || jb + 1 < g.nx - 1) d.y = m.Lr[jb + 1] * vzv.y + d.y;
                        }
                        if (XB) {
                            float *fDXU = px_ptr(g, PX, s, PX_NFWD + PXA_DXU), *fDXV = px_ptr(g, PX, s, PX_NFWD + PXA_DXV);
                            const float4 c0 = ldt(g.pmx + jb), c1 = ldt(g.pmx + jb + 1);
                            const float2 m0 = mem_x(fDXU + i * g.xs_n, xs), m1 = mem_x(fDXV + i * g.xs_n, xs);
                            adj_x2(g, d, c0, c1, xs, m0, fDXU + i * g.xs_n);
                            adj_x2(g, v, c0, c1, xs, m1, fDXV + i * g.xs_n);
                        }
                        const long long b = (long long)i * g.wxp + band_x(g, jb);
                        float *ix = im.xa + (long long)s * 2 * g.txs + b;
                        *reinterpret_cast<float2 *>(ix) = d;
                        *reinterpret_cast<float2 *>(ix + g.txs) = v;
                    }
                }
                const int pi = i - g.z0, pj0 = jb - g.pad;
                const bool prow = !GUARD || (pi >= 0 && pi < g.nz_dom);
                const bool p0 = prow && (!XB || (pj0 >= 0 && pj0 < g.nx_dom));
                const bool p1 = prow && (!XB || (pj0 + 1 >= 0 && pj0 + 1 < g.nx_dom));
                // a history plane's pair at this cell (outside the physical grid: 0)
                auto hist = [&](const float *pl) {
                    const float *a = pl + (long long)pi * g.nx_dom + pj0;
                    float2 v = make_float2(0.f, 0.f);
                    if (hist2) {
                        if (p0) v = __ldcs(reinterpret_cast<const float2 *>(a));
                    } else {
                        if (p0) v.x = __ldcs(a);
                        if (p1) v.y = __ldcs(a + 1);
                    }
                    return v;
                };
                float2 h1, h2, h3;
                if (htma) {
                    h1 = pair_at(hown + qo);
                    h2 = pair_at(hown + PL + qo);
                    h3 = pair_at(hown + 2 * PL + qo);
                }
                if (EXACT && o.slot_in >= 0) {
                    if (!htma) {
                        const float *in = slot(o.slot_in);
                        h1 = hist(in); h2 = hist(in + g.nd); h3 = hist(in + 2 * g.nd);
                    }
                    sA[r % RE] = add2(sA[r % RE], fma2(h1, sxx, mul2(h2, szz)));
                    sB[r % RE] = add2(sB[r % RE], fma2(h2, sxx, mul2(h1, szz)));
                    sC[r % RE] = fma2(h3, sxz, sC[r % RE]);
                }
                if (RHO && (p0 || p1)) {
                    const long long off = (long long)i * g.P + jb;
                    const float2 pc = *reinterpret_cast<const float2 *>(Pp + off), qc = *reinterpret_cast<const float2 *>(Qp + off);
                    const float2 bb = mat_pair(g, m.B, i, jb);
                    const float *in = slot(o.slot_in), *img = slot(o.slot_img), *nxt = slot(o.slot_next);
                    if (EXACT && o.slot_in >= 0 && o.slot_img >= 0) {
                        // dJ/dB: U_a dU/B + V_a dV/B with U_a = P/B and the
                        // step's velocity increments from the history
                        const float2 du = sub2(hist(img + 3 * g.nd), hist(in + 3 * g.nd));
                        const float2 dv = sub2(hist(img + 4 * g.nd), hist(in + 4 * g.nd));
                        if (p0) gB[r % RB].x += (pc.x * du.x + qc.x * dv.x) / (bb.x * bb.x);
                        if (p1) gB[r % RB].y += (pc.y * du.y + qc.y * dv.y) / (bb.y * bb.y);
                    }
                    if (IMG) {
                        // -1/2 U_a(n) (vx(n-1) - vx(n+1)), the rho term of the
                        // imaging formula regrouped by adjoint step
                        float2 t = make_float2(0.f, 0.f);
                        const float2 ua = make_float2(p0 ? pc.x / bb.x : 0.f, p1 ? pc.y / bb.y : 0.f);
                        const float2 va = make_float2(p0 ? qc.x / bb.x : 0.f, p1 ? qc.y / bb.y : 0.f);
                        if (n >= 2 && o.slot_in >= 0)
                            t = add2(t, fma2(ua, hist(in + 3 * g.nd), mul2(va, hist(in + 4 * g.nd))));
                        if (n <= g.nt - 3 && o.slot_next >= 0)
                            t = sub2(t, fma2(ua, hist(nxt + 3 * g.nd), mul2(va, hist(nxt + 4 * g.nd))));
                        grl[r % RR] = fma2(dup2(-0.5f), t, grl[r % RR]);
                    }
                }
                if (IMG && o.slot_img >= 0 && (p0 || p1)) {
                    if (EXACT || !htma) {
                        const float *img = slot(o.slot_img);
                        h1 = hist(img); h2 = hist(img + g.nd); h3 = hist(img + 2 * g.nd);
                    }
#pragma unroll
                    for (int cc = 0; cc < 2; ++cc) {
                        if (!(cc ? p1 : p0)) continue;
                        float dxBU, dzBU, dxBV, dzBV;
                        if (boxed) {
                            dxBU = f2c(dxP, cc) * g.inv2dx;
                            dxBV = f2c(dxQ, cc) * g.inv2dx;
                            dzBU = f2c(dzP[r % RI], cc) * g.inv2dz;
                            dzBV = f2c(dzQ[r % RI], cc) * g.inv2dz;
                        } else {
                            // periodic at the edges of the padded grid, as jnp.roll
                            const int j = jb + cc, ip = (i + 1) % g.nz, im1 = (i - 1 + g.nz) % g.nz;
                            const int jp = (j + 1) % g.nx, jm = (j - 1 + g.nx) % g.nx;
                            const long long oxp = (long long)i * g.P + jp, oxm = (long long)i * g.P + jm;
                            const long long ozp = (long long)ip * g.P + j, ozm = (long long)im1 * g.P + j;
                            dxBU = (Pp[oxp] - Pp[oxm]) * g.inv2dx;
                            dzBV = (Qp[ozp] - Qp[ozm]) * g.inv2dz;
                            dzBU = (Pp[ozp] - Pp[ozm]) * g.inv2dz;
                            dxBV = (Qp[oxp] - Qp[oxm]) * g.inv2dx;
                        }
                        const float l2m = f2c(ml2m[r], cc), l = f2c(ml[r], cc);
                        const float t1 = f2c(h1, cc), t2 = f2c(h2, cc), id = 1.0f / ((l2m - l) * (l2m + l));
                        const float e1 = (l2m * t1 - l * t2) * id, e2 = (l2m * t2 - l * t1) * id;
                        const float e3 = f2c(h3, cc) * (1.0f / (2.f * f2c(mm[r], cc)));
                        const float gl = -g.dt * ((e1 + e2) * (dxBU + dzBV));
                        const float gm = -g.dt * (2.f * e1 * dxBU + 2.f * e2 * dzBV + e3 * (dzBU + dxBV));
                        if (cc) { glam[r % RI].y += gl; gmu[r % RI].y += gm; }
                        else { glam[r % RI].x += gl; gmu[r % RI].x += gm; }
                    }
                }
            }
            return true;
        };
        if (!(!xin ? rows(std::true_type{}, std::true_type{})
                   : !zin ? rows(std::true_type{}, std::false_type{}) : rows(std::false_type{}, std::false_type{}))) {
            ring_abort(ring, it, status);
            return;
        }
        if (ring_leave(ring, st, ph, it + NST < c.n)) issue(s + NST, st);
        if (r1 > r0) {
            // receivers of step n - 1 on this warp's rows, whose cells its own lanes have just written
            __syncwarp();
            for (int qq = r0 + tx; qq < r1; qq += TX) {
                const int rid = rv.tile_rec[qq], i = rv.rz[rid];
                if (i < iw || i >= iw + RPT) continue;
                const float *src = o.rec_adj + (long long)s * 4 * g.nt * g.nrec + (long long)(n - 1) * g.nrec + rid;
                inject_strain(g, m, im, A, PX, PZ, s, i, rv.rx[rid], src[2LL * g.nt * g.nrec], src[3LL * g.nt * g.nrec]);
            }
        }
    }
    leave();
}

}  // namespace stfwi
