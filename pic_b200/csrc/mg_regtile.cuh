// Register tiles of the multigrid's graph- and host-loop V-cycle (included by
// multigrid.cu): the down and up phases of one level, and of two levels in one
// launch, for up to kRtMaxSweeps red-black sweeps.
//
// A block of 8, 12 or 16 warps works a region of a level held in registers, 64
// columns by 4 rows per warp: warp w has rows 4w .. 4w+3, lane l the columns 2l
// and 2l+1 of each.  Region origins are even in both directions, so a node's
// colour follows from its row and column index at compile time, every lane
// updates one node per row in every half-sweep, and a half-sweep costs one warp
// shuffle (the neighbour in the next lane) and about eight arithmetic
// instructions per update.  Rows on either side of a warp's four travel through
// shared memory, two values per lane and one barrier per half-sweep.  The
// Dirichlet mask comes as bit columns (LevelDev::fb), two words per lane and
// column.
//
// What bounds these phases is instruction issue at large grids and the chain
// load - sweeps - store at small ones; shared-memory tiles of 32 x 32 (down_tile,
// up_tile) spend about 370 instructions per node, most of them on addresses,
// index bounds and mask bytes, with half their threads idle in a half-sweep.
#pragma once

namespace pic {

constexpr int kRtRows = 4;       // rows per warp
constexpr int kRtMaxWarps = 16;
constexpr int kRtMaxThreads = 32 * kRtMaxWarps;
constexpr int kRtCols = 64;      // region columns, = 2 * 32
constexpr unsigned kRtRowMask = (1u << kRtRows) - 1u;

// How far a phase of S sweeps reaches into the region, from its border (depth
// 0).  A half-sweep is right one node deeper than what it reads; the first
// half-sweep of a down phase starts from zero and reads no neighbour.
//   down   e at depth 2S - 1, the residual at 2S, its restriction at 2S + 1
//   up     e at depth 2S; with the FP64 residual, e one node around the core
// Core and left halo are even (two levels: multiples of four), so that every
// origin keeps its parity.  core(n): the core of n region rows or columns.
template <int S>
struct RtDown {
    static constexpr int HL = 2 * S + 2;
    static constexpr __host__ __device__ int core(int n) { return n - HL - 2 * S; }
};
template <int S, bool RES>
struct RtUp {
    static constexpr int HL = RES ? 2 * S + 2 : 2 * S;
    static constexpr __host__ __device__ int core(int n) { return n - 2 * HL; }
};
// Two levels, F (the region) and C (half as many columns and rows, one node
// per lane and row).
//   down2  C's right-hand side is right on C nodes [ceil((2S+1)/2),
//          floor((n-2-2S)/2)], its restriction 2S + 1 nodes inside that
//   up2    C is right on [2S, n/2 - 2 - 2S] (the last lane's prolongation is
//          not formed), F's prolongation on [4S, n - 4 - 4S], F on
//          [6S, n - 4 - 6S]
template <int S>
struct RtDown2 {
    static constexpr int C0 = (S + 1 + 2 * S + 1 + 1) / 2 * 2, HL = 2 * C0;  // C0: the first C2 centre
    static constexpr __host__ __device__ int core(int n) {
        const int c1 = ((n - 2 - 2 * S) / 2 - 2 * S - 1) / 2 * 2;  // the last one
        return 2 * (c1 + 2 - C0);
    }
};
template <int S>
struct RtUp2 {
    static constexpr int HL = (6 * S + 3) / 4 * 4;
    static constexpr __host__ __device__ int core(int n) { return (n - 4 - 6 * S - HL + 1) / 4 * 4; }
};

__device__ __forceinline__ int rt_warps() { return int(blockDim.x) >> 5; }
__device__ __forceinline__ int rt_side() { return kRtRows * rt_warps(); }  // region rows

// Column bits of up to 32 rows from row j of column i: bit r is 1 when node
// (i, j + r) is free.
__device__ __forceinline__ unsigned rt_free_bits(const uint32_t* __restrict__ fb, int nx, int nwords, int i, int j,
                                                 unsigned mask) {
    const int w = j >> 5;  // floor, j may be negative
    const bool ci = i >= 0 && i < nx;
    const unsigned lo = (ci && w >= 0 && w < nwords) ? __ldg(fb + long(w) * nx + i) : 0u;
    const unsigned hi = (ci && w + 1 >= 0 && w + 1 < nwords) ? __ldg(fb + long(w + 1) * nx + i) : 0u;
    return __funnelshift_r(lo, hi, unsigned(j & 31)) & mask;
}

// The coefficients of an update; r-z rows keep {wN, wS, 1/diag, D} in registers.
template <class T, int ROWS, bool CYL>
struct RtCoef {
    T cx, cy, inv_diag, omega;
    T rz[CYL ? ROWS : 1][4];
    __device__ __forceinline__ void load(const LevelDev<T>& L, T om, int j0) {
        cx = L.cx;
        cy = L.cy;
        inv_diag = L.inv_diag;
        omega = om;
        if constexpr (CYL) {
#pragma unroll
            for (int r = 0; r < ROWS; ++r) {
                const int j = j0 + r;
                const bool in = j >= 0 && j < L.ny;
#pragma unroll
                for (int q = 0; q < 4; ++q) rz[r][q] = in ? __ldg(L.rz + 4 * j + q) : T(0);
            }
        }
    }
    // The over-relaxed value of a node of row r (relaxed, relaxed_rz).
    __device__ __forceinline__ T update(int r, T old, T ew, T s, T n, T g) const {
        if constexpr (CYL) return relaxed_rz(old, ew, s, n, g, cx, rz[r][0], rz[r][1], rz[r][2], omega);
        else return relaxed(old, ew, s, n, g, cx, cy, inv_diag, omega);
    }
};

// One region of F: 4 rows x 2 columns per lane, and the rows on either side.
template <class T>
struct RtTile {
    T e[kRtRows][2], g[kRtRows][2];
    T up[2], dn[2];  // row -1 (the warp above) and row 4, per column
    unsigned fr[2];  // free bits of the rows, per column
};

// Shared exchange rows, two buffers used in turn: a buffer is written again
// only after the barrier between its readers and the next-but-one exchange.
template <class T>
struct RtShared {
    T x[2][kRtMaxWarps][2][32];
};

// Publishes, of the nodes of one colour, row 0 (its column COLOR & 1) and the
// last row (its other column), and reads the neighbouring warps' into up and dn.
template <class T, int COLOR>
__device__ __forceinline__ void rt_exchange(RtTile<T>& t, RtShared<T>& s, int& buf) {
    const int w = threadIdx.x >> 5, l = threadIdx.x & 31;
    constexpr int c0 = COLOR & 1, c1 = (kRtRows - 1 + COLOR) & 1;
    s.x[buf][w][0][l] = t.e[0][c0];
    s.x[buf][w][1][l] = t.e[kRtRows - 1][c1];
    __syncthreads();
    if (w > 0) t.up[c1] = s.x[buf][w - 1][1][l];
    if (w < rt_warps() - 1) t.dn[c0] = s.x[buf][w + 1][0][l];
    buf ^= 1;
}

// One half-sweep (COLOR 0: red, (i + j) even).
template <class T, int COLOR, bool CYL>
__device__ __forceinline__ void rt_half_sweep(RtTile<T>& t, const RtCoef<T, kRtRows, CYL>& cf) {
#pragma unroll
    for (int r = 0; r < kRtRows; ++r) {
        const int c = (r + COLOR) & 1;
        const T side = c ? __shfl_down_sync(0xffffffffu, t.e[r][0], 1) : __shfl_up_sync(0xffffffffu, t.e[r][1], 1);
        const T s = r > 0 ? t.e[r - 1][c] : t.up[c];
        const T n = r < kRtRows - 1 ? t.e[r + 1][c] : t.dn[c];
        const T v = cf.update(r, t.e[r][c], side + t.e[r][1 - c], s, n, t.g[r][c]);
        if ((t.fr[c] >> r) & 1u) t.e[r][c] = v;
    }
}

// S sweeps.  FROM_ZERO: e = 0 everywhere before the first half-sweep, which
// reads no neighbour; else the initial rows are exchanged first.  LAST: the
// black rows after the last half-sweep are exchanged too (for a residual).
template <class T, int S, bool CYL, bool FROM_ZERO, bool LAST>
__device__ __forceinline__ void rt_sweeps(RtTile<T>& t, const RtCoef<T, kRtRows, CYL>& cf, RtShared<T>& sh, int& buf) {
    t.up[0] = t.up[1] = t.dn[0] = t.dn[1] = T(0);
    if constexpr (!FROM_ZERO) {
        rt_exchange<T, 1>(t, sh, buf);
    }
#pragma unroll
    for (int s = 0; s < S; ++s) {
        if (FROM_ZERO && s == 0) {
#pragma unroll
            for (int r = 0; r < kRtRows; ++r) {
                const int c = r & 1;
                t.e[r][c] = ((t.fr[c] >> r) & 1u) ? cf.update(r, T(0), T(0), T(0), T(0), t.g[r][c]) : T(0);
                t.e[r][1 - c] = T(0);
            }
        } else {
            rt_half_sweep<T, 0, CYL>(t, cf);
        }
        rt_exchange<T, 0>(t, sh, buf);
        rt_half_sweep<T, 1, CYL>(t, cf);
        if (LAST || s < S - 1) rt_exchange<T, 1>(t, sh, buf);
    }
}

// The residual g - A e of the region, 0 on Dirichlet nodes (r-z: weighted by
// the row's volume).
template <class T, bool CYL>
__device__ __forceinline__ void rt_residual(const RtTile<T>& t, const RtCoef<T, kRtRows, CYL>& cf,
                                            T (&res)[kRtRows][2]) {
#pragma unroll
    for (int r = 0; r < kRtRows; ++r) {
        const T w = __shfl_up_sync(0xffffffffu, t.e[r][1], 1), ea = __shfl_down_sync(0xffffffffu, t.e[r][0], 1);
#pragma unroll
        for (int c = 0; c < 2; ++c) {
            const T e = t.e[r][c];
            const T wv = c ? t.e[r][0] : w, ev = c ? ea : t.e[r][1];
            const T s = r > 0 ? t.e[r - 1][c] : t.up[c];
            const T n = r < kRtRows - 1 ? t.e[r + 1][c] : t.dn[c];
            T v;
            if constexpr (CYL) {
                const T lap = cf.cx * (wv + ev - T(2) * e) + cf.rz[r][0] * (n - e) + cf.rz[r][1] * (s - e);
                v = cf.rz[r][3] * (t.g[r][c] - lap);
            } else {
                v = t.g[r][c] - weighted(cf.cx, wv + ev - T(2) * e, cf.cy, s + n - T(2) * e);
            }
            res[r][c] = ((t.fr[c] >> r) & 1u) ? v : T(0);
        }
    }
}

// The full weighting of a coarse node from its fine row {west, centre, east}
// and the rows below and above, in restrict_fw's order.
template <class T>
struct RtRow3 {
    T w, c, e;
};
template <class T>
__device__ __forceinline__ T rt_weight(const RtRow3<T>& s, const RtRow3<T>& m, const RtRow3<T>& n) {
    T v = T(0.25) * m.c;
    v += T(0.125) * (m.w + m.e + s.c + n.c);
    v += T(0.0625) * (s.w + s.e + n.w + n.e);
    return v;
}

// Full weighting of the coarse rows of this warp (the fine rows 0 and 2) at
// the even columns; J0: the coarse row of fine row 0.
template <class T, bool CYL>
__device__ __forceinline__ void rt_restrict(const T (&res)[kRtRows][2], RtShared<T>& sh, int& buf, int J0,
                                            T (&out)[kRtRows / 2]) {
    const int w = threadIdx.x >> 5, l = threadIdx.x & 31;
    sh.x[buf][w][0][l] = res[kRtRows - 1][0];
    sh.x[buf][w][1][l] = res[kRtRows - 1][1];
    __syncthreads();
    RtRow3<T> below{T(0), T(0), T(0)};
    if (w > 0) {
        below.c = sh.x[buf][w - 1][0][l];
        below.e = sh.x[buf][w - 1][1][l];
        below.w = sh.x[buf][w - 1][1][max(l - 1, 0)];
    }
    buf ^= 1;
#pragma unroll
    for (int q = 0; q < kRtRows / 2; ++q) {
        auto row = [&](int r) {
            return RtRow3<T>{__shfl_up_sync(0xffffffffu, res[r][1], 1), res[r][0], res[r][1]};
        };
        const RtRow3<T> above = row(2 * q + 1);
        T v = rt_weight(below, row(2 * q), above);
        // r-z: divided by the stencil's weighted volume (2J; 5/16 on the axis)
        if constexpr (CYL) v *= J0 + q == 0 ? T(3.2) : T(0.5) / T(J0 + q);
        out[q] = v;
        below = above;
    }
}

// Loads the free bits of a lane's rows, per column.
template <class T>
__device__ __forceinline__ void rt_load_bits(const LevelDev<T>& L, int i0, int j0, RtTile<T>& t) {
    const int nw = (L.ny + 31) >> 5;
    t.fr[0] = rt_free_bits(L.fb, L.nx, nw, i0, j0, kRtRowMask);
    t.fr[1] = rt_free_bits(L.fb, L.nx, nw, i0 + 1, j0, kRtRowMask);
}

// The region's nodes of a field; nodes outside the grid take the value of the
// nearest one inside (they are never free, and what a Dirichlet node holds is
// not used), so that no load carries a bound test.
template <class T, class G>
__device__ __forceinline__ void rt_load_rows(const G* src, int nx, int ny, int i0, int j0, T (&v)[kRtRows][2]) {
    const int c0 = min(max(i0, 0), nx - 1), c1 = min(max(i0 + 1, 0), nx - 1);
#pragma unroll
    for (int r = 0; r < kRtRows; ++r) {
        const G* p = src + long(min(max(j0 + r, 0), ny - 1)) * nx;
        v[r][0] = T(p[c0]);
        v[r][1] = T(p[c1]);
    }
}

// Stores the core's nodes of a field of the region.
// (cx, cy: the core's columns and rows; HL: its left halo)
template <class T, int HL>
__device__ __forceinline__ void rt_store_core(T* dst, const T (&v)[kRtRows][2], int nx, int ny, int i0, int j0, int cx,
                                              int cy) {
    const int w = threadIdx.x >> 5, l = threadIdx.x & 31;
    if (2 * l < HL || 2 * l >= HL + cx) return;
    T* p = dst + long(j0) * nx + i0;
#pragma unroll
    for (int r = 0; r < kRtRows; ++r) {
        const int lr = w * kRtRows + r;
        if (lr < HL || lr >= HL + cy || j0 + r >= ny) continue;
        if (i0 < nx) p[long(r) * nx] = v[r][0];
        if (i0 + 1 < nx) p[long(r) * nx + 1] = v[r][1];
    }
}

// ---- one level -----------------------------------------------------------------------

// The first residual of a solve, formed by the first cycle's down phase.
struct RtInit {
    const double *phi, *f, *rz0;
    double* r64;
    double cx, cy;
};

// Rows -1 and 4 of a warp's FP64 potential, both columns.
struct RtShared64 {
    double x[kRtMaxWarps][2][2][32];
};

// r = f - A phi on the region's free nodes (right from depth 1 on), 0
// elsewhere, in the association of k_mg_r0; the core's r goes to r64 and its
// squares, and those of f, to r2 and f2.
template <class T, int HL, bool CYL>
__device__ __forceinline__ void rt_first_residual(const RtInit& I, const LevelDev<T>& F, int i0, int j0, int cx,
                                                  int cy, RtTile<T>& t, RtShared64& sh, double& r2, double& f2) {
    const int w = threadIdx.x >> 5, l = threadIdx.x & 31;
    double p[kRtRows][2], fv[kRtRows][2], up[2] = {0.0, 0.0}, dn[2] = {0.0, 0.0};
    rt_load_rows<double, double>(I.phi, F.nx, F.ny, i0, j0, p);
    rt_load_rows<double, double>(I.f, F.nx, F.ny, i0, j0, fv);
#pragma unroll
    for (int c = 0; c < 2; ++c) {
        sh.x[w][0][c][l] = p[0][c];
        sh.x[w][1][c][l] = p[kRtRows - 1][c];
    }
    __syncthreads();
#pragma unroll
    for (int c = 0; c < 2; ++c) {
        if (w > 0) up[c] = sh.x[w - 1][1][c][l];
        if (w < rt_warps() - 1) dn[c] = sh.x[w + 1][0][c][l];
    }
    const bool core_col = 2 * l >= HL && 2 * l < HL + cx;
#pragma unroll
    for (int r = 0; r < kRtRows; ++r) {
        const int lr = w * kRtRows + r, j = j0 + r;
        const double ww = __shfl_up_sync(0xffffffffu, p[r][1], 1), ee = __shfl_down_sync(0xffffffffu, p[r][0], 1);
        const bool in = core_col && lr >= HL && lr < HL + cy && j < F.ny;
#pragma unroll
        for (int c = 0; c < 2; ++c) {
            const double e = p[r][c];
            const double wv = c ? p[r][0] : ww, ev = c ? ee : p[r][1];
            const double s = r > 0 ? p[r - 1][c] : up[c], n = r < kRtRows - 1 ? p[r + 1][c] : dn[c];
            const bool fr = (t.fr[c] >> r) & 1u;
            double lap;
            if constexpr (CYL) {
                const bool jin = j >= 0 && j < F.ny;
                const double wn = jin ? __ldg(I.rz0 + 4 * j) : 0.0, ws = jin ? __ldg(I.rz0 + 4 * j + 1) : 0.0;
                lap = I.cx * ((wv - e) + (ev - e)) + wn * (n - e) + ws * (s - e);
            } else {
                lap = I.cx * ((wv - e) + (ev - e)) + I.cy * ((s - e) + (n - e));
            }
            const double res = fr ? fv[r][c] - lap : 0.0;
            t.g[r][c] = T(res);
            if (in && i0 + c < F.nx) {
                I.r64[long(j) * F.nx + i0 + c] = res;
                r2 += res * res;
                if (fr) f2 += fv[r][c] * fv[r][c];
            }
        }
    }
}

// The decision, the same in every warp; `writer` (one thread of the grid) records
// it.  True: the solve has stopped, now or before.  ref: ||f||^2.
__device__ __forceinline__ bool rt_pending_stop(const RtPending& P, bool writer, double& ref) {
    // a flag that this grid's writer has set already is this decision
    if (!P.fblocks && stopped(P.N.stop)) return true;
    const int l = threadIdx.x & 31;
    double r2 = 0.0, f2 = 0.0;
#pragma unroll
    for (int u = 0; u < kRtPendingMax / 32; ++u) {
        const int q = l + 32 * u;
        if (q < P.nb) r2 += P.N.partial[q];
        if (q < P.fblocks) f2 += P.N.fpart[q];
    }
    ref = P.fblocks ? 0.0 : P.N.norms[0];
    r2 = warp_sum(r2);
    if (P.fblocks) ref = warp_sum(f2);
    const bool conv = r2 < P.tol2 * (ref > 0.0 ? ref : 1.0);
    const bool stop = conv || P.done >= P.max_cycles;
    if (writer) {
        if (P.fblocks) P.N.norms[0] = ref;
        P.N.norms[1] = r2;
        *P.N.cycles = P.done;
        *P.N.total += P.inc;
        *P.N.converged = conv ? 1 : 0;
        *P.N.stop = stop ? 1 : 0;
    }
    return stop;
}

// How a tile's phase follows the one before it.  RtLaunched: a launch of its own
// in the chain, which waits for its predecessor and does nothing once the solve
// has stopped.  RtInLoop: a phase of k_rt_rest, after a grid barrier.  Loads of
// what the phase before did not write come ahead of wait().
struct RtLaunched {
    const int* stop;
    __device__ __forceinline__ void wait() const {
        pdl_wait();
        pdl_trigger();
    }
    __device__ __forceinline__ bool done() const { return stopped(stop); }
};
struct RtPendingLaunched {
    const int* stop;
    const RtPending& P;
    __device__ __forceinline__ void wait() const {
        pdl_wait();
        pdl_trigger();
    }
    __device__ __forceinline__ bool done() const {
        double ref;
        return P.nb ? rt_pending_stop(P, threadIdx.x == 0 && blockIdx.x + blockIdx.y == 0, ref) : stopped(stop);
    }
};
struct RtInLoop {
    __device__ __forceinline__ void wait() const {}
    __device__ __forceinline__ bool done() const { return false; }
};

// What follows a down phase's right-hand side (in t.g): smooth from zero, store
// the core's correction (and, on level 0, its right-hand side in the V-cycle's
// precision), restrict the residual.  (cx, cy: the core's columns and rows.)
template <class T, int S, bool CYL>
__device__ __forceinline__ void rt_down_rest(const LevelDev<T>& F, const LevelDev<T>& C, RtTile<T>& t,
                                             const RtCoef<T, kRtRows, CYL>& cf, RtShared<T>& sh, int i0, int j0, int cx,
                                             int cy, bool store_g, unsigned cfr) {
    constexpr int HL = RtDown<S>::HL;
    const int w = threadIdx.x >> 5, l = threadIdx.x & 31;
    // the coarse column and rows this lane restricts to (i0, j0 are even)
    const int I = i0 >> 1, J0 = j0 >> 1;
    int buf = 0;
    rt_sweeps<T, S, CYL, true, true>(t, cf, sh, buf);
    rt_store_core<T, HL>(F.e, t.e, F.nx, F.ny, i0, j0, cx, cy);
    if (store_g) rt_store_core<T, HL>(F.g, t.g, F.nx, F.ny, i0, j0, cx, cy);
    T res[kRtRows][2], out[kRtRows / 2];
    rt_residual<T, CYL>(t, cf, res);
    rt_restrict<T, CYL>(res, sh, buf, J0, out);
    if (2 * l < HL || 2 * l >= HL + cx || I >= C.nx) return;
#pragma unroll
    for (int q = 0; q < kRtRows / 2; ++q) {
        const int lr = w * kRtRows + 2 * q;
        if (lr < HL || lr >= HL + cy || J0 + q >= C.ny) continue;
        C.g[long(J0 + q) * C.nx + I] = ((cfr >> q) & 1u) ? out[q] : T(0);
    }
}

// The down phase (see k_mg_down) of the tile (bx, by): smooth from zero,
// restrict the residual.
template <class T, int S, bool CYL, class Sync>
__device__ __forceinline__ void rt_down_tile(const LevelDev<T>& F, const LevelDev<T>& C, T omega, const double* g64,
                                             int bx, int by, RtShared<T>& sh, const Sync& sync) {
    constexpr int HL = RtDown<S>::HL;
    const int w = threadIdx.x >> 5, l = threadIdx.x & 31;
    const int cx = RtDown<S>::core(kRtCols), cy = RtDown<S>::core(rt_side());
    const int i0 = bx * cx - HL + 2 * l, j0 = by * cy - HL + kRtRows * w;
    RtTile<T> t;
    RtCoef<T, kRtRows, CYL> cf;
    rt_load_bits(F, i0, j0, t);
    const unsigned cfr = rt_free_bits(C.fb, C.nx, (C.ny + 31) >> 5, i0 >> 1, j0 >> 1, (1u << (kRtRows / 2)) - 1u);
    cf.load(F, omega, j0);
    sync.wait();
    if (g64) rt_load_rows<T, double>(g64, F.nx, F.ny, i0, j0, t.g);
    else rt_load_rows<T, T>(F.g, F.nx, F.ny, i0, j0, t.g);
    if (sync.done()) return;
    rt_down_rest<T, S, CYL>(F, C, t, cf, sh, i0, j0, cx, cy, g64 != nullptr, cfr);
}

template <class T, int S, bool CYL>
__global__ void __launch_bounds__(kRtMaxThreads) k_rt_down(LevelDev<T> F, LevelDev<T> C, T omega,
                                                           const double* __restrict__ g64, const int* stop,
                                                           const __grid_constant__ RtPending P) {
    __shared__ RtShared<T> sh;
    rt_down_tile<T, S, CYL>(F, C, omega, g64, blockIdx.x, blockIdx.y, sh, RtPendingLaunched{stop, P});
}

// The finest down phase of a solve's first cycle: the right-hand side is the
// first residual, formed here.  Its region is right from depth 1 on, so the
// core is the residual up phase's.  decide: also the norms of the residual and
// of f and the first loop decision; else the blocks' shares of ||f||^2, for the
// decision after the first cycles (NormState::fpart).
// Two blocks to an SM where 64 registers hold it (2049^2 69 us with one block,
// 49 with two; r-z would spill: 129 x 97 step 1.7 us slower).
template <class T, int S, bool CYL>
__global__ void __launch_bounds__(kRtMaxThreads, sizeof(T) == 4 && !CYL ? 2 : 1)
    k_rt_init(LevelDev<T> F, LevelDev<T> C, T omega, RtInit I, NormState N, double tol2, int max_cycles, int decide) {
    constexpr int HL = RtDown<S>::HL;
    static_assert(HL == RtUp<S, true>::HL, "the first residual's tiles are the residual up phase's");
    __shared__ RtShared<T> sh;
    __shared__ RtShared64 sh64;
    const int w = threadIdx.x >> 5, l = threadIdx.x & 31;
    const int cx = RtUp<S, true>::core(kRtCols), cy = RtUp<S, true>::core(rt_side());
    const int i0 = int(blockIdx.x) * cx - HL + 2 * l, j0 = int(blockIdx.y) * cy - HL + kRtRows * w;
    RtTile<T> t;
    RtCoef<T, kRtRows, CYL> cf;
    rt_load_bits(F, i0, j0, t);
    const unsigned cfr = rt_free_bits(C.fb, C.nx, (C.ny + 31) >> 5, i0 >> 1, j0 >> 1, (1u << (kRtRows / 2)) - 1u);
    cf.load(F, omega, j0);
    pdl_wait();
    pdl_trigger();
    double r2 = 0.0, f2 = 0.0;
    rt_first_residual<T, HL, CYL>(I, F, i0, j0, cx, cy, t, sh64, r2, f2);
    rt_down_rest<T, S, CYL>(F, C, t, cf, sh, i0, j0, cx, cy, true, cfr);
    if (decide) {
        norm_reduce_decide(r2, f2, N, tol2, max_cycles, 1, cudaGraphConditionalHandle{}, 0);
        return;
    }
    __shared__ double ws[kRtMaxWarps];
    f2 = warp_sum(f2);
    if (l == 0) ws[w] = f2;
    __syncthreads();
    if (threadIdx.x == 0) {
        double s = 0.0;
        for (int q = 0; q < rt_warps(); ++q) s += ws[q];
        N.fpart[blockIdx.y * gridDim.x + blockIdx.x] = s;
    }
}

// Adds the bilinear prolongation of the coarse rows cv (of the fine rows 0, 2
// and 4) and their east neighbours ce on the free nodes; e is 0 elsewhere.
template <class T>
__device__ __forceinline__ void rt_prolong(RtTile<T>& t, const T (&cv)[kRtRows / 2 + 1], const T (&ce)[kRtRows / 2 + 1]) {
#pragma unroll
    for (int r = 0; r < kRtRows; ++r) {
        const int q = r >> 1;
        T a = cv[q], b = T(0.5) * (cv[q] + ce[q]);
        if (r & 1) {
            a = T(0.5) * (cv[q] + cv[q + 1]);
            b = T(0.25) * (cv[q] + ce[q] + cv[q + 1] + ce[q + 1]);
        }
        t.e[r][0] = ((t.fr[0] >> r) & 1u) ? t.e[r][0] + a : T(0);
        t.e[r][1] = ((t.fr[1] >> r) & 1u) ? t.e[r][1] + b : T(0);
    }
}

// An 8-byte copy from global to shared memory that the thread goes on past
// (rows of an odd number of nodes allow no wider ones), and the wait for all of
// this thread's.
__device__ __forceinline__ void rt_copy8(double* dst, const double* src) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(unsigned(__cvta_generic_to_shared(dst))), "l"(src)
                 : "memory");
}
__device__ __forceinline__ void rt_copy_wait() { asm volatile("cp.async.wait_all;" ::: "memory"); }
constexpr int kRtUp = 0, kRtRes = 1, kRtResStaged = 2;  // the up phase's modes
constexpr int kRtStage = 4 * kRtRows;  // staged doubles per thread of the residual up phase

// The up phase (see k_mg_up, k_mg_up_res) of the tile (bx, by): add the
// prolonged coarse correction and smooth; kRtRes (level 0): phi += e and the
// FP64 residual r -= A e on the core, its squares in r2.  phi and r are loaded
// before the wait, into registers (kRtRes) or shared memory (kRtResStaged, 128
// bytes per thread and 64 registers): see rt_staged.  A 2049^2 grid's phase
// moves 172 MB, 26 us at the copy rate, in 72 us from registers (one block of
// 512 threads to an SM: load, sweeps and store follow each other) and in 50
// staged (two).
template <class T, int S, bool CYL, int MODE, class Sync>
__device__ __forceinline__ bool rt_up_tile(const LevelDev<T>& F, const LevelDev<T>& C, T omega, double* phi,
                                           const ResArgs& R, int bx, int by, RtShared<T>& sh, double* stage,
                                           double& r2, const Sync& sync) {
    constexpr bool RES = MODE != kRtUp;
    using G = RtUp<S, RES>;
    const int w = threadIdx.x >> 5, l = threadIdx.x & 31;
    const int cx = G::core(kRtCols), cy = G::core(rt_side());
    const int i0 = bx * cx - G::HL + 2 * l, j0 = by * cy - G::HL + kRtRows * w;
    RtTile<T> t;
    RtCoef<T, kRtRows, CYL> cf;
    rt_load_bits(F, i0, j0, t);
    cf.load(F, omega, j0);
    // everything but the coarse correction was written two or more launches back
    rt_load_rows<T, T>(F.e, F.nx, F.ny, i0, j0, t.e);
    rt_load_rows<T, T>(F.g, F.nx, F.ny, i0, j0, t.g);
    const bool core_col = 2 * l >= G::HL && 2 * l < G::HL + cx;
    constexpr bool STAGED = MODE == kRtResStaged;
    double pv[RES && !STAGED ? kRtRows : 1][2], rv[RES && !STAGED ? kRtRows : 1][2];
    double* st = STAGED ? stage + threadIdx.x : nullptr;
    if constexpr (RES) {
#pragma unroll
        for (int r = 0; r < kRtRows; ++r) {
            const int lr = w * kRtRows + r;
            const bool in = core_col && lr >= G::HL && lr < G::HL + cy && j0 + r < F.ny;
            const long k = long(j0 + r) * F.nx + i0;
#pragma unroll
            for (int c = 0; c < 2; ++c) {
                const bool ic = in && i0 + c < F.nx;
                if constexpr (STAGED) {
                    if (!ic) continue;
                    rt_copy8(st + (4 * r + c) * blockDim.x, phi + k + c);
                    rt_copy8(st + (4 * r + 2 + c) * blockDim.x, R.r64 + k + c);
                } else {
                    pv[r][c] = ic ? phi[k + c] : 0.0;
                    rv[r][c] = ic ? R.r64[k + c] : 0.0;
                }
            }
        }
    }
    sync.wait();
    {
        const int I = i0 >> 1, J0 = j0 >> 1;
        T cv[kRtRows / 2 + 1], ce[kRtRows / 2 + 1];
#pragma unroll
        for (int q = 0; q < kRtRows / 2 + 1; ++q) {
            const int J = J0 + q;
            const bool in = J >= 0 && J < C.ny;
            const T* p = C.ec + long(J) * C.nx + I;
            cv[q] = (in && I >= 0 && I < C.nx) ? p[0] : T(0);
            // the last lane's east neighbour is not in the warp
            const T x = (l == 31 && in && I + 1 >= 0 && I + 1 < C.nx) ? p[1] : T(0);
            const T y = __shfl_down_sync(0xffffffffu, cv[q], 1);
            ce[q] = l == 31 ? x : y;
        }
        if (sync.done()) {
            if constexpr (STAGED) rt_copy_wait();  // no block ends with copies into it under way
            return false;
        }
        rt_prolong(t, cv, ce);
    }
    int buf = 0;
    // the red rows' neighbours are black: they are exchanged before the first half-sweep
    rt_sweeps<T, S, CYL, false, RES>(t, cf, sh, buf);
    if constexpr (!RES) {
        rt_store_core<T, G::HL>(F.ec, t.e, F.nx, F.ny, i0, j0, cx, cy);
    } else {
        r2 = 0.0;
        if constexpr (STAGED) rt_copy_wait();
#pragma unroll
        for (int r = 0; r < kRtRows; ++r) {
            const int lr = w * kRtRows + r, j = j0 + r;
            const T ww = __shfl_up_sync(0xffffffffu, t.e[r][1], 1), ee = __shfl_down_sync(0xffffffffu, t.e[r][0], 1);
            const bool in = core_col && lr >= G::HL && lr < G::HL + cy && j < F.ny;
            const long k = long(j) * F.nx + i0;
#pragma unroll
            for (int c = 0; c < 2; ++c) {
                if (!in || i0 + c >= F.nx) continue;
                phi[k + c] = (STAGED ? st[(4 * r + c) * blockDim.x] : pv[STAGED ? 0 : r][c]) + double(t.e[r][c]);
                if (!((t.fr[c] >> r) & 1u)) continue;
                // f - A(phi + e) = r - A e, in the association of k_mg_r0's Laplacian
                const double e = double(t.e[r][c]);
                const double wv = double(c ? t.e[r][0] : ww), ev = double(c ? ee : t.e[r][1]);
                const double s = double(r > 0 ? t.e[r - 1][c] : t.up[c]);
                const double n = double(r < kRtRows - 1 ? t.e[r + 1][c] : t.dn[c]);
                double lap;
                if constexpr (CYL)
                    lap = R.cx * ((wv - e) + (ev - e)) + R.rz0[4 * j] * (n - e) + R.rz0[4 * j + 1] * (s - e);
                else
                    lap = R.cx * ((wv - e) + (ev - e)) + R.cy * ((s - e) + (n - e));
                const double rr = (STAGED ? st[(4 * r + 2 + c) * blockDim.x] : rv[STAGED ? 0 : r][c]) - lap;
                R.r64[k + c] = rr;
                r2 += rr * rr;
            }
        }
    }
    return true;
}

// The sum over the block's warps, in thread 0.
__device__ __forceinline__ double rt_block_sum(double v) {
    __shared__ double ws[kRtMaxWarps];
    v = warp_sum(v);
    if ((threadIdx.x & 31) == 0) ws[threadIdx.x >> 5] = v;
    __syncthreads();
    double s = 0.0;
    if (threadIdx.x == 0)
        for (int q = 0; q < rt_warps(); ++q) s += ws[q];
    return s;
}

// The phase as a launch; RES: its norm and the loop decision too.
template <class T, int S, bool CYL, int MODE>
__global__ void __launch_bounds__(kRtMaxThreads, MODE == kRtResStaged ? 2 : 1)
    k_rt_up(LevelDev<T> F, LevelDev<T> C, T omega, double* __restrict__ phi, ResArgs R, const int* stop) {
    __shared__ RtShared<T> sh;
    extern __shared__ double rt_stage[];
    double r2 = 0.0;
    if (!rt_up_tile<T, S, CYL, MODE>(F, C, omega, phi, R, blockIdx.x, blockIdx.y, sh, rt_stage, r2, RtLaunched{stop}))
        return;
    if constexpr (MODE != kRtUp) {
        if (R.decide == 2) {
            // the block's sum for rt_pending_stop
            const double s = rt_block_sum(r2);
            if (threadIdx.x == 0) R.N.partial[blockIdx.y * gridDim.x + blockIdx.x] = s;
        } else if (R.decide)
            norm_reduce_decide(r2, 0.0, R.N, R.tol2, R.max_cycles, 0, R.cond, R.use_cond, R.inc, R.fblocks);
    }
}

// ---- two levels in one launch ---------------------------------------------------------
//
// C's region: lane l has column C-origin + l, warp w the rows 2w and 2w+1.  The
// origin is even, so a node's colour is (l + row) & 1: in a half-sweep a lane
// updates one of its two rows, the odd or the even one by its parity.

constexpr int kRtCRows = kRtRows / 2;
static_assert(kRtCRows == 2, "one pair of coarse rows per warp");

template <class T>
struct RtCTile {
    T e[2], g[2];
    T up, dn;  // rows -1 and 2
    unsigned fr;
};

template <class T>
__device__ __forceinline__ void rt_c_exchange(RtCTile<T>& t, RtShared<T>& s, int& buf) {
    const int w = threadIdx.x >> 5, l = threadIdx.x & 31;
    s.x[buf][w][0][l] = t.e[0];
    s.x[buf][w][1][l] = t.e[1];
    __syncthreads();
    if (w > 0) t.up = s.x[buf][w - 1][1][l];
    if (w < rt_warps() - 1) t.dn = s.x[buf][w + 1][0][l];
    buf ^= 1;
}

template <class T, bool CYL>
__device__ __forceinline__ void rt_c_half_sweep(RtCTile<T>& t, const RtCoef<T, kRtCRows, CYL>& cf, int color) {
    const bool odd = ((threadIdx.x + color) & 1) != 0;  // which of its rows this lane updates
    // the neighbouring lanes update the other row: they send this lane's
    const T send = odd ? t.e[0] : t.e[1];
    const T wv = __shfl_up_sync(0xffffffffu, send, 1), ev = __shfl_down_sync(0xffffffffu, send, 1);
    const T s = odd ? t.e[0] : t.up, n = odd ? t.dn : t.e[1];
    const T old = odd ? t.e[1] : t.e[0], g = odd ? t.g[1] : t.g[0];
    T v;
    if constexpr (CYL)
        v = relaxed_rz(old, wv + ev, s, n, g, cf.cx, odd ? cf.rz[1][0] : cf.rz[0][0], odd ? cf.rz[1][1] : cf.rz[0][1],
                       odd ? cf.rz[1][2] : cf.rz[0][2], cf.omega);
    else v = cf.update(0, old, wv + ev, s, n, g);
    if (!odd && (t.fr & 1u)) t.e[0] = v;
    if (odd && (t.fr & 2u)) t.e[1] = v;
}

// S sweeps of C; every exchange carries both colours' boundary rows.
template <class T, int S, bool CYL, bool FROM_ZERO>
__device__ __forceinline__ void rt_c_sweeps(RtCTile<T>& t, const RtCoef<T, kRtCRows, CYL>& cf, RtShared<T>& sh, int& buf) {
    t.up = t.dn = T(0);
    if (!FROM_ZERO) rt_c_exchange(t, sh, buf);
#pragma unroll
    for (int s = 0; s < S; ++s) {
        rt_c_half_sweep<T, CYL>(t, cf, 0);
        rt_c_exchange(t, sh, buf);
        rt_c_half_sweep<T, CYL>(t, cf, 1);
        rt_c_exchange(t, sh, buf);
    }
}

template <class T, int S, bool CYL, class Sync>
__device__ __forceinline__ void rt_down2_tile(const LevelDev<T>& F, const LevelDev<T>& C, const LevelDev<T>& C2, T omega,
                                             int bx, int by, RtShared<T>& sh, const Sync& sync) {
    using G = RtDown2<S>;
    const int w = threadIdx.x >> 5, l = threadIdx.x & 31;
    const int cx = G::core(kRtCols), cy = G::core(rt_side());
    const int i0 = bx * cx - G::HL + 2 * l, j0 = by * cy - G::HL + kRtRows * w;
    const int I = i0 >> 1, J0 = j0 >> 1;
    RtTile<T> t;
    RtCTile<T> ct;
    RtCoef<T, kRtRows, CYL> cf;
    RtCoef<T, kRtCRows, CYL> cc;
    rt_load_bits(F, i0, j0, t);
    ct.fr = rt_free_bits(C.fb, C.nx, (C.ny + 31) >> 5, I, J0, (1u << (kRtRows / 2)) - 1u);
    const unsigned c2fr = rt_free_bits(C2.fb, C2.nx, (C2.ny + 31) >> 5, I >> 1, J0 >> 1, 1u);
    cf.load(F, omega, j0);
    cc.load(C, omega, J0);
    sync.wait();
    rt_load_rows<T, T>(F.g, F.nx, F.ny, i0, j0, t.g);
    if (sync.done()) return;
    int buf = 0;
    rt_sweeps<T, S, CYL, true, true>(t, cf, sh, buf);
    rt_store_core<T, G::HL>(F.e, t.e, F.nx, F.ny, i0, j0, cx, cy);
    T res[kRtRows][2], out[kRtCRows];
    rt_residual<T, CYL>(t, cf, res);
    rt_restrict<T, CYL>(res, sh, buf, J0, out);
#pragma unroll
    for (int q = 0; q < kRtCRows; ++q) {
        ct.g[q] = ((ct.fr >> q) & 1u) ? out[q] : T(0);
        ct.e[q] = T(0);
    }
    rt_c_sweeps<T, S, CYL, true>(ct, cc, sh, buf);
    // C's core: its e and g for the up phase
    const bool ccol = 2 * l >= G::HL && 2 * l < G::HL + cx && I < C.nx;
#pragma unroll
    for (int q = 0; q < kRtCRows; ++q) {
        const int lr = w * kRtRows + 2 * q;
        if (!ccol || lr < G::HL || lr >= G::HL + cy || J0 + q >= C.ny) continue;
        const long K = long(J0 + q) * C.nx + I;
        C.e[K] = ct.e[q];
        C.g[K] = ct.g[q];
    }
    // C's residual
    RtRow3<T> rc[kRtCRows];
#pragma unroll
    for (int q = 0; q < kRtCRows; ++q) {
        const T e = ct.e[q];
        const T wv = __shfl_up_sync(0xffffffffu, e, 1), ev = __shfl_down_sync(0xffffffffu, e, 1);
        const T s = q > 0 ? ct.e[q - 1] : ct.up, n = q < kRtCRows - 1 ? ct.e[q + 1] : ct.dn;
        T v;
        if constexpr (CYL) {
            const T lap = cc.cx * (wv + ev - T(2) * e) + cc.rz[q][0] * (n - e) + cc.rz[q][1] * (s - e);
            v = cc.rz[q][3] * (ct.g[q] - lap);
        } else {
            v = ct.g[q] - weighted(cc.cx, wv + ev - T(2) * e, cc.cy, s + n - T(2) * e);
        }
        const T r = ((ct.fr >> q) & 1u) ? v : T(0);
        rc[q] = RtRow3<T>{__shfl_up_sync(0xffffffffu, r, 1), r, __shfl_down_sync(0xffffffffu, r, 1)};
    }
    sh.x[buf][w][1][l] = rc[1].c;
    __syncthreads();
    RtRow3<T> below{T(0), T(0), T(0)};
    if (w > 0) {
        const T* x = sh.x[buf][w - 1][1];
        below = RtRow3<T>{x[max(l - 1, 0)], x[l], x[min(l + 1, 31)]};
    }
    buf ^= 1;
    // one C2 row per warp, on the even lanes
    const int I2 = I >> 1, J2 = J0 >> 1, lr = w * kRtRows;
    if ((l & 1) || !ccol || I2 >= C2.nx || lr < G::HL || lr >= G::HL + cy || J2 >= C2.ny) return;
    T v = rt_weight(below, rc[0], rc[1]);
    if constexpr (CYL) v *= J2 == 0 ? T(3.2) : T(0.5) / T(J2);
    C2.g[long(J2) * C2.nx + I2] = (c2fr & 1u) ? v : T(0);
}

template <class T, int S, bool CYL>
__global__ void __launch_bounds__(kRtMaxThreads) k_rt_down2(LevelDev<T> F, LevelDev<T> C, LevelDev<T> C2, T omega,
                                                           const int* stop) {
    __shared__ RtShared<T> sh;
    rt_down2_tile<T, S, CYL>(F, C, C2, omega, blockIdx.x, blockIdx.y, sh, RtLaunched{stop});
}

template <class T, int S, bool CYL, class Sync>
__device__ __forceinline__ void rt_up2_tile(const LevelDev<T>& F, const LevelDev<T>& C, const LevelDev<T>& C2, T omega,
                                             int bx, int by, RtShared<T>& sh, const Sync& sync) {
    using G = RtUp2<S>;
    const int w = threadIdx.x >> 5, l = threadIdx.x & 31;
    const int cx = G::core(kRtCols), cy = G::core(rt_side());
    const int i0 = bx * cx - G::HL + 2 * l, j0 = by * cy - G::HL + kRtRows * w;
    const int I = i0 >> 1, J0 = j0 >> 1;
    RtTile<T> t;
    RtCTile<T> ct;
    RtCoef<T, kRtRows, CYL> cf;
    RtCoef<T, kRtCRows, CYL> cc;
    rt_load_bits(F, i0, j0, t);
    ct.fr = rt_free_bits(C.fb, C.nx, (C.ny + 31) >> 5, I, J0, (1u << (kRtRows / 2)) - 1u);
    cf.load(F, omega, j0);
    cc.load(C, omega, J0);
    rt_load_rows<T, T>(F.e, F.nx, F.ny, i0, j0, t.e);
    rt_load_rows<T, T>(F.g, F.nx, F.ny, i0, j0, t.g);
#pragma unroll
    for (int q = 0; q < kRtCRows; ++q) {
        const long K = long(min(max(J0 + q, 0), C.ny - 1)) * C.nx + min(max(I, 0), C.nx - 1);
        ct.e[q] = C.e[K];
        ct.g[q] = C.g[K];
    }
    sync.wait();
    {
        // C2's correction prolonged onto C: an odd column takes the mean of
        // its own C2 column and the next lane's
        const int I2 = I >> 1, J2 = J0 >> 1;
        T v2[2], e2[2];
#pragma unroll
        for (int q = 0; q < 2; ++q) {
            const int J = J2 + q;
            const bool in = J >= 0 && J < C2.ny && I2 >= 0 && I2 < C2.nx;
            v2[q] = in ? C2.ec[long(J) * C2.nx + I2] : T(0);
            e2[q] = __shfl_down_sync(0xffffffffu, v2[q], 1);
        }
        const bool odd = (l & 1) != 0;
        const T v[kRtCRows] = {odd ? T(0.5) * (v2[0] + e2[0]) : v2[0],
                               odd ? T(0.25) * (v2[0] + e2[0] + v2[1] + e2[1]) : T(0.5) * (v2[0] + v2[1])};
#pragma unroll
        for (int q = 0; q < kRtCRows; ++q) ct.e[q] = ((ct.fr >> q) & 1u) ? ct.e[q] + v[q] : T(0);
    }
    if (sync.done()) return;
    int buf = 0;
    rt_c_sweeps<T, S, CYL, false>(ct, cc, sh, buf);
    {
        T cv[kRtCRows + 1] = {ct.e[0], ct.e[1], ct.dn}, ce[kRtCRows + 1];
#pragma unroll
        for (int q = 0; q < kRtCRows + 1; ++q) ce[q] = __shfl_down_sync(0xffffffffu, cv[q], 1);
        rt_prolong(t, cv, ce);
    }
    rt_sweeps<T, S, CYL, false, false>(t, cf, sh, buf);
    rt_store_core<T, G::HL>(F.ec, t.e, F.nx, F.ny, i0, j0, cx, cy);
}

template <class T, int S, bool CYL>
__global__ void __launch_bounds__(kRtMaxThreads) k_rt_up2(LevelDev<T> F, LevelDev<T> C, LevelDev<T> C2, T omega,
                                                           const int* stop) {
    __shared__ RtShared<T> sh;
    rt_up2_tile<T, S, CYL>(F, C, C2, omega, blockIdx.x, blockIdx.y, sh, RtLaunched{stop});
}

// ---- the cycles after the launched ones, in one cooperative launch ----------------------

// The cycles a solve still needs after those launched in line, on grids whose
// every phase is one wave of tiles: nothing when the solve has stopped (the
// usual case), else V-cycles with a grid barrier between phases until it
// converges or reaches max_cycles.  A conditional node costs a solve 6.6 us on
// the device also when its condition is false, and the graph that holds one
// more time to launch; this launch costs 2 us (a simulation's step to 1e-8 with
// the node and with this launch: 129 x 97 68.5 and 57.2 us, 513 x 513 104.9 and
// 89.4).  A cycle in here takes about 10 us more than one of the node's (129 x
// 129 27 us against 17.5): a barrier costs 1 to 2 us where a launch in line
// costs 1, and the phases' code leaves the instruction cache.
template <class T>
struct RtRest {
    int lc;     // levels above the direct solve: [0, lc)
    int fuse2;  // levels lc - 2 and lc - 1 in one phase each way
    LevelDev<T> lv[kMgMaxLevels];
    DirectDesc<T> direct;
    int direct64;  // its inverse is FP64
    ResArgs res;
    RtPending pending;
    double* phi;
    T omega;
    GridBar* bar;
    int* error;
    unsigned long long polls;
};

template <class T, class MT>
__device__ __forceinline__ void rt_direct(const DirectDesc<T>& D, MT* gs) {
    const int w = threadIdx.x >> 5, l = threadIdx.x & 31;
    const MT* __restrict__ ainv = static_cast<const MT*>(D.ainv);
    for (int k = threadIdx.x; k < D.n; k += blockDim.x) gs[k] = MT(D.g[__ldg(D.idx + k)]);
    if (blockIdx.x == 0)
        for (int k = threadIdx.x; k < D.nz; k += blockDim.x) D.e[D.zidx[k]] = T(0);
    __syncthreads();
    for (int row = int(blockIdx.x) * rt_warps() + w; row < D.n; row += int(gridDim.x) * rt_warps()) {
        MT s = MT(0);
#pragma unroll 5
        for (int u = 0; u < kDirectCols; ++u) {
            const int c = l + 32 * u;
            if (c < D.n) s += __ldg(ainv + long(row) * D.n + c) * gs[c];
        }
        const double t = warp_sum(double(s));
        if (l == 0) D.e[__ldg(D.idx + row)] = T(t);
    }
}

template <class T, int S, bool CYL>
__global__ void __launch_bounds__(kRtMaxThreads, 1) k_rt_rest(const __grid_constant__ RtRest<T> D) {
    double f2;
    if (rt_pending_stop(D.pending, threadIdx.x == 0 && blockIdx.x == 0, f2)) return;
    // after a barrier that gave up its counter is not in order: nothing runs in
    // here, and solves end unconverged, until the host has read the error
    if (*reinterpret_cast<const volatile int*>(D.error)) return;
    __shared__ RtShared<T> sh;
    __shared__ double gs[kDirectMaxFree];
    const int bid = int(blockIdx.x), nb = int(gridDim.x), l = threadIdx.x & 31;
    const NormState& N = D.res.N;
    const int before = D.pending.done;
    const double lim = D.res.tol2 * (f2 > 0.0 ? f2 : 1.0);
    const int lsingle = D.fuse2 ? D.lc - 2 : D.lc;
    const RtInLoop go{};
    int seq = 0, n = 0;
    double r2 = 0.0;
    bool conv = false;
    auto barrier = [&]() { return grid_barrier(D.bar, D.error, seq++, D.polls); };
    // this block's tile of a phase on level L (every phase has at most nb tiles)
    auto tile = [&](const LevelDev<T>& L, int cx, int cy, int& bx, int& by) {
        const int tx = (L.nx + cx - 1) / cx;
        bx = bid % tx;
        by = bid / tx;
        return by * cy < L.ny;
    };
    do {
        int bx, by;
        for (int k = 0; k < lsingle; ++k) {
            if (tile(D.lv[k], RtDown<S>::core(kRtCols), RtDown<S>::core(rt_side()), bx, by))
                rt_down_tile<T, S, CYL>(D.lv[k], D.lv[k + 1], D.omega, k == 0 ? D.res.r64 : nullptr, bx, by, sh, go);
            if (!barrier()) return;
        }
        if (D.fuse2) {
            if (tile(D.lv[lsingle], RtDown2<S>::core(kRtCols), RtDown2<S>::core(rt_side()), bx, by))
                rt_down2_tile<T, S, CYL>(D.lv[lsingle], D.lv[lsingle + 1], D.lv[lsingle + 2], D.omega, bx, by, sh, go);
            if (!barrier()) return;
        }
        if (D.direct64) rt_direct<T, double>(D.direct, gs);
        else rt_direct<T, T>(D.direct, reinterpret_cast<T*>(gs));
        if (!barrier()) return;
        if (D.fuse2) {
            if (tile(D.lv[lsingle], RtUp2<S>::core(kRtCols), RtUp2<S>::core(rt_side()), bx, by))
                rt_up2_tile<T, S, CYL>(D.lv[lsingle], D.lv[lsingle + 1], D.lv[lsingle + 2], D.omega, bx, by, sh, go);
            if (!barrier()) return;
        }
        for (int k = lsingle - 1; k >= 1; --k) {
            double u;
            if (tile(D.lv[k], RtUp<S, false>::core(kRtCols), RtUp<S, false>::core(rt_side()), bx, by))
                rt_up_tile<T, S, CYL, kRtUp>(D.lv[k], D.lv[k + 1], D.omega, nullptr, D.res, bx, by, sh, nullptr, u, go);
            if (!barrier()) return;
        }
        r2 = 0.0;
        if (tile(D.lv[0], RtUp<S, true>::core(kRtCols), RtUp<S, true>::core(rt_side()), bx, by))
            rt_up_tile<T, S, CYL, kRtRes>(D.lv[0], D.lv[1], D.omega, D.phi, D.res, bx, by, sh, nullptr, r2, go);
        // the norm: the blocks' sums, added by every block in the same order
        r2 = rt_block_sum(r2);
        if (threadIdx.x == 0) N.partial[bid] = r2;
        if (!barrier()) return;
        r2 = 0.0;
        for (int q = l; q < nb; q += 32) r2 += reinterpret_cast<const volatile double*>(N.partial)[q];
        r2 = warp_sum(r2);
        ++n;
        conv = r2 < lim;
    } while (!conv && before + n < D.res.max_cycles);
    if (bid == 0 && threadIdx.x == 0) {
        N.norms[1] = r2;
        *N.cycles = before + n;
        *N.total += n;
        *N.converged = conv ? 1 : 0;
        *N.stop = 1;
    }
}

// ---- launch tables ----------------------------------------------------------------------

template <class T>
using RtUpKernel = void (*)(LevelDev<T>, LevelDev<T>, T, double*, ResArgs, const int*);
template <class T>
using RtInitKernel = void (*)(LevelDev<T>, LevelDev<T>, T, RtInit, NormState, double, int, int);

template <class T, bool CYL>
static RtDownKernel<T> rt_down_kernel(int s) {
    static const RtDownKernel<T> k[kRtMaxSweeps + 1] = {nullptr, k_rt_down<T, 1, CYL>, k_rt_down<T, 2, CYL>,
                                                      k_rt_down<T, 3, CYL>};
    return k[s];
}

template <class T, bool CYL>
static RtInitKernel<T> rt_init_kernel(int s) {
    static const RtInitKernel<T> k[kRtMaxSweeps + 1] = {nullptr, k_rt_init<T, 1, CYL>, k_rt_init<T, 2, CYL>,
                                                        k_rt_init<T, 3, CYL>};
    return k[s];
}

template <class T, bool CYL, int MODE>
static RtUpKernel<T> rt_up_kernel(int s) {
    static const RtUpKernel<T> k[kRtMaxSweeps + 1] = {nullptr, k_rt_up<T, 1, CYL, MODE>, k_rt_up<T, 2, CYL, MODE>,
                                                      k_rt_up<T, 3, CYL, MODE>};
    return k[s];
}

template <class T, bool CYL>
static RtFused2Kernel<T> rt_down2_kernel(int s) {
    static const RtFused2Kernel<T> k[kRtMaxSweeps + 1] = {nullptr, k_rt_down2<T, 1, CYL>, k_rt_down2<T, 2, CYL>,
                                                        k_rt_down2<T, 3, CYL>};
    return k[s];
}

template <class T, bool CYL>
static RtFused2Kernel<T> rt_up2_kernel(int s) {
    static const RtFused2Kernel<T> k[kRtMaxSweeps + 1] = {nullptr, k_rt_up2<T, 1, CYL>, k_rt_up2<T, 2, CYL>,
                                                        k_rt_up2<T, 3, CYL>};
    return k[s];
}

static size_t rt_stage_bytes(int threads) { return sizeof(double) * kRtStage * threads; }

template <class T>
using RtRestKernel = void (*)(const RtRest<T>);
template <class T, bool CYL>
static RtRestKernel<T> rt_rest_kernel(int s) {
    static const RtRestKernel<T> k[kRtMaxSweeps + 1] = {nullptr, k_rt_rest<T, 1, CYL>, k_rt_rest<T, 2, CYL>,
                                                        k_rt_rest<T, 3, CYL>};
    return k[s];
}

// The launch shape of a phase on an nx x ny level: of 8, 12 and 16 warps per
// block, the one that gives the busiest SM the fewest warps (a region row costs
// the same in every shape, but the halo is shared by more rows in the taller
// ones: small levels spread over more SMs, large ones take 16).
struct RtShape {
    dim3 grid;
    int threads;
};
template <class Core>
static RtShape rt_shape(int nx, int ny, Core core) {
    RtShape best{};
    long cost = 0;
    for (int w : {16, 12, 8}) {
        const int cy = core(kRtRows * w);
        if (cy < 4) continue;
        const dim3 g(div_up(nx, core(kRtCols)), div_up(ny, cy));
        const long c = long(div_up(long(g.x) * g.y, num_sms())) * w;
        if (!best.threads || c < cost) {
            best = RtShape{g, 32 * w};
            cost = c;
        }
    }
    return best;
}
static RtShape rt_down_shape(int s, int nx, int ny) {
    return rt_shape(nx, ny, [=](int n) {
        return s == 1 ? RtDown<1>::core(n) : s == 2 ? RtDown<2>::core(n) : RtDown<3>::core(n);
    });
}
static RtShape rt_up_shape(int s, int nx, int ny, bool res) {
    return rt_shape(nx, ny, [=](int n) {
        if (res) return s == 1 ? RtUp<1, true>::core(n) : s == 2 ? RtUp<2, true>::core(n) : RtUp<3, true>::core(n);
        return s == 1 ? RtUp<1, false>::core(n) : s == 2 ? RtUp<2, false>::core(n) : RtUp<3, false>::core(n);
    });
}
static RtShape rt_down2_shape(int s, int nx, int ny) {
    return rt_shape(nx, ny, [=](int n) {
        return s == 1 ? RtDown2<1>::core(n) : s == 2 ? RtDown2<2>::core(n) : RtDown2<3>::core(n);
    });
}
static RtShape rt_up2_shape(int s, int nx, int ny) {
    return rt_shape(nx, ny, [=](int n) {
        return s == 1 ? RtUp2<1>::core(n) : s == 2 ? RtUp2<2>::core(n) : RtUp2<3>::core(n);
    });
}

}  // namespace pic
