// Multigrid levels as two launches each: one for the way down (one smoothing
// step from a zero iterate, residual, restriction) and one for the way up
// (prolongation, correction, one smoothing step). The per-phase kernels of
// mg.cu make 9 launches (2 colours) or 15 (4 colours) of the same work, each
// a pass over the level in memory.
//
// A block owns a core of cx x cy columns and works on it plus a halo in
// shared memory; every phase recomputes the halo columns that the following
// phases of the core need, so no phase waits for another block. With nc
// colours the halo is
//   uniform levels  down 3: colour 0 at distance <= 3 of the core, colour 1 at
//                   <= 2, residual at <= 1; up 2.
//   cross levels    down nc + 3: bottom rows at <= nc + 3, colour c at
//                   <= nc + 2 - c, bottom rows again at <= 2, residual at <= 1;
//                   up nc + 2. (FP32: one more on the way down.)
// The arithmetic per row is the colour pass's (mg_device.cuh) up to the order
// of the sums, on FP32 cross levels in the same order.
//
// What bounds them: the latency of the phases, not bytes. On a B200, per level
// and V-cycle: 1025x257x17 FP64 flat 125 us (55 down, 70 up) against about 300
// of the per-phase kernels, FP32 83 us; a 97x49x9 level 14 us; sloping 257x33x9
// FP64 50 us, FP32 56 us. All levels of a V-cycle below 160000 points: 41 us
// (97x49x9), 125 us (257x33x9) against 180 and 345 us in the cooperative kernel.
//
// On uniform levels one thread solves one column bottom to top: the sums over
// neighbour columns do not depend on the row below, only
// x_k = q_k - g_k x_{k-1} is a chain. On cross levels, whose rows cost an
// order more, the lanes of a segment share a column. Columns lie in shared
// memory with an odd pitch and the columns of one parity of i side by side, so that the threads
// of a warp, which take every other column, meet no bank conflict.
#include "mg_tile.cuh"
#include "mg_device.cuh"

#include <algorithm>

namespace ow3d {

namespace {
using namespace mgdev;

constexpr int kCrossThreads = 512, kUniThreads = 320, kOrderedThreads = 512;
constexpr size_t kTileSmemMax = 220 * 1024, kTileSmemTwo = 112 * 1024;
constexpr int kTileMaxRows = 65535;   // blocks of a grid in y: longer basins take the per-phase kernels

// Core and staged region of a block, 1-based columns; on a periodic level i
// runs past the ends and is taken cyclically (gcol).
struct Reg {
    int ia, ib, ra, rb, W;   // core and region in x
    int ja, jb, sa, sb, H;   // in y
};

// Core t of columns 1..n (the first `rem` cores hold q + 1 columns, the others
// q). A core holds three columns or more, so a wall's ghost column always lies
// in a core with the two interior columns that determine it.
__host__ __device__ inline void span(int n, int t, int q, int rem, int halo, int& a, int& b, int& ra, int& rb) {
    a = 1 + t * q + (t < rem ? t : rem);
    b = a + q - 1 + (t < rem ? 1 : 0);
    ra = a - halo > 1 ? a - halo : 1;
    if (ra <= 3) ra = 1;                 // a region that holds column 2 or 3 holds the ghost column too
    rb = b + halo < n ? b + halo : n;
    if (rb >= n - 2) rb = n;
}
__host__ __device__ inline Reg region(int Nxg, int Nyg, int per, const TileGeo& g, int bx, int by, bool three) {
    Reg r;
    if (per) {
        span(Nxg, bx, g.qx, g.remx, 0, r.ia, r.ib, r.ra, r.rb);
        r.ia += 1; r.ib += 1;            // the distinct columns 2..Nxg-2
        r.ra = r.ia - g.halo;
        r.rb = r.ib + g.halo;
    } else {
        span(Nxg, bx, g.qx, g.remx, g.halo, r.ia, r.ib, r.ra, r.rb);
    }
    if (three) span(Nyg, by, g.qy, g.remy, g.halo, r.ja, r.jb, r.sa, r.sb);
    else r.ja = r.jb = r.sa = r.sb = 1;
    r.W = r.rb - r.ra + 1;
    r.H = r.sb - r.sa + 1;
    return r;
}
// Whether the region touches a wall (and so holds ghost columns).
__device__ __forceinline__ bool at_wall(int Nxg, int Nyg, int per, const Reg& r, bool three) {
    return (!per && (r.ra == 1 || r.rb == Nxg)) || (three && (r.sa == 1 || r.sb == Nyg));
}
// Periodic x: the distinct column that stands at i.
__device__ __forceinline__ int gcol(int i, int Nxg, int per) {
    if (!per) return i;
    const int M = Nxg - 3;
    int t = (i - 2) % M;
    if (t < 0) t += M;
    return 2 + t;
}

// a / b for 0 <= a < 2^20, 1 <= b, rb = recip(b): exact (the quotient of
// a + 1/2 is at least 1 / (2 b) away from an integer, the error of the product
// below that), a few instructions where an integer division is some twenty-five.
__device__ __forceinline__ int quot(int a, float rb) { return (int)(((float)a + 0.5f) * rb); }
__device__ __forceinline__ float recip(int b) { return __fdividef(1.0f, (float)b); }

template <typename T> struct Pair;
template <> struct Pair<double> { using type = double2; };
template <> struct Pair<float> { using type = float2; };
template <typename T>
__device__ __forceinline__ typename Pair<T>::type pair_at(const T* p) {
    return *reinterpret_cast<const typename Pair<T>::type*>(p);
}

// Visit H rows of W columns of Nzg values each: a thread keeps one place k in
// the column (N rows: 2 where Nzg is even -- a pair then lies on its own
// alignment -- else 1) and steps through the columns, U visits in flight, so
// that an access costs a few additions of index arithmetic. acc.ld(v, c, q)
// only loads what column c of row q needs (no branch, no arithmetic on the
// values: either would hold up the loads of the visits after it), acc.st(c, q,
// v) does the rest; acc is made for the thread's k.
template <int N, int U, typename MAKE>
__device__ __forceinline__ void sweep_n(int W, int H, int Nzg, MAKE make) {
    const int nu = Nzg / N;
    const float rnu = recip(nu), rw = recip(W);
    const int cg = quot(threadIdx.x, rnu), step = quot(blockDim.x, rnu);
    if (cg >= step) return;
    const auto acc = make(N * (threadIdx.x - cg * nu));
    int q = quot(cg, rw), c = cg - q * W;
    const int dq = quot(step, rw), dc = step - dq * W;
    while (q < H) {
        typename decltype(make(0))::template Val<N> v[U];
        int cc[U], qq[U];
#pragma unroll
        for (int m = 0; m < U; ++m) {
            cc[m] = c;
            qq[m] = q;
            if (q < H) acc.ld(v[m], c, q);
            c += dc;
            q += dq;
            if (c >= W) { c -= W; ++q; }
        }
#pragma unroll
        for (int m = 0; m < U; ++m)
            if (qq[m] < H) acc.st(cc[m], qq[m], v[m]);
    }
}
template <int U, typename MAKE>
__device__ __forceinline__ void sweep(int W, int H, int Nzg, MAKE make) {
    if ((Nzg & 1) == 0) sweep_n<2, U>(W, H, Nzg, make);
    else sweep_n<1, U>(W, H, Nzg, make);
}
template <typename T>
__device__ __forceinline__ void put_pair(T* p, T a, T b) {
    typename Pair<T>::type q;
    q.x = a; q.y = b;
    *reinterpret_cast<typename Pair<T>::type*>(p) = q;
}
// N values to a staged array; VEC: its columns have an even pitch (uniform
// levels), so that pairs go in one access.
template <int N, bool VEC, typename T>
__device__ __forceinline__ void put(T* p, const T* v) {
    if constexpr (N == 2 && VEC) put_pair(p, v[0], v[1]);
    else if constexpr (N == 2) { p[0] = v[0]; p[1] = v[1]; }
    else p[0] = v[0];
}
template <int N, typename T>
__device__ __forceinline__ void get(T* v, const T* p) {
    if constexpr (N == 2) { const auto q = pair_at(p); v[0] = q.x; v[1] = q.y; }
    else v[0] = p[0];
}

// Offset of column (li, lj) of the region (0-based) in a staged array.
__device__ __forceinline__ int slot(const TileGeo& g, int li, int lj) {
    return ((lj * 2 + (li & 1)) * g.HW + (li >> 1)) * g.NZP;
}
// The same within a row (add row_slot of its row).
__device__ __forceinline__ int col_slot(const TileGeo& g, int li) { return ((li & 1) * g.HW + (li >> 1)) * g.NZP; }
__device__ __forceinline__ int row_slot(const TileGeo& g, int lj) { return 2 * lj * g.HW * g.NZP; }
// Offsets to the left and right neighbour columns of a column of parity li & 1.
__device__ __forceinline__ int near_l(const TileGeo& g, int li) { return li & 1 ? -g.HW * g.NZP : (g.HW - 1) * g.NZP; }
__device__ __forceinline__ int near_r(const TileGeo& g, int li) { return li & 1 ? (1 - g.HW) * g.NZP : g.HW * g.NZP; }

// The interior columns of `colour` at distance <= d of the core, one per
// thread in turn: f(i, j).
template <bool THREE, typename F>
__device__ __forceinline__ void colour_columns(int Nxg, int Nyg, int per, const Reg& r, int ncolor, int colour, int d,
                                               F f) {
    int ilo = r.ia - d, ihi = r.ib + d, jlo = 1, jhi = 1;
    if (!per) { ilo = max(ilo, 2); ihi = min(ihi, Nxg - 1); }
    if (THREE) { jlo = max(r.ja - d, 2); jhi = min(r.jb + d, Nyg - 1); }
    const bool four = ncolor == 4;
    int js = 1;
    if (THREE && four) {
        jlo += (jlo ^ (colour >> 1)) & 1;
        js = 2;
    }
    const int ni = (ihi - ilo + 2) >> 1, nj = jhi >= jlo ? (jhi - jlo) / js + 1 : 0;
    const float rni = recip(ni);
    for (int t = threadIdx.x; t < ni * nj; t += blockDim.x) {
        const int tj = quot(t, rni), j = jlo + tj * js;
        const int par = four ? colour & 1 : (colour + j) & 1;
        const int i = ilo + ((ilo ^ par) & 1) + 2 * (t - tj * ni);
        if (i <= ihi) f(i, j);
    }
}

// All interior columns at distance <= d of the core.
template <bool THREE, typename F>
__device__ __forceinline__ void all_columns(int Nxg, int Nyg, int per, const Reg& r, int d, F f) {
    int ilo = r.ia - d, ihi = r.ib + d, jlo = 1, jhi = 1;
    if (!per) { ilo = max(ilo, 2); ihi = min(ihi, Nxg - 1); }
    if (THREE) { jlo = max(r.ja - d, 2); jhi = min(r.jb + d, Nyg - 1); }
    // in a row first every other column, then the rest: a warp's columns lie
    // side by side in shared memory
    const int ni = max(ihi - ilo + 1, 0), nj = max(jhi - jlo + 1, 0), first = (ni + 1) >> 1;
    const float rni = recip(ni);
    for (int t = threadIdx.x; t < ni * nj; t += blockDim.x) {
        const int tj = quot(t, rni), q = t - tj * ni;
        f(ilo + (q < first ? 2 * q : 2 * (q - first) + 1), jlo + tj);
    }
}

// The ghost columns of the region (corners excluded): f(place of row k in the
// ghost column, in its nearest and in its second interior column, i and j of
// the nearest, whether the wall is an x wall, 0 or 1 for the low or high one)
// for the 0-based rows k = 1..Nzg-1. All walls in one loop.
template <bool THREE, typename F>
__device__ __forceinline__ void ghost_rows(int Nxg, int Nyg, int per, int Nzg, const Reg& r, const TileGeo& g, F f) {
    const int jlo = THREE ? max(r.sa, 2) : 1, jhi = THREE ? min(r.sb, Nyg - 1) : 1;
    const int ilo = per ? r.ra : max(r.ra, 2), ihi = per ? r.rb : min(r.rb, Nxg - 1);
    const int nx = jhi - jlo + 1, ny = ihi - ilo + 1;
    const int n0 = !per && r.ra == 1 ? nx : 0, n1 = n0 + (!per && r.rb == Nxg ? nx : 0);
    const int n2 = n1 + (THREE && r.sa == 1 ? ny : 0), n3 = n2 + (THREE && r.sb == Nyg ? ny : 0);
    const int row = 2 * g.HW * g.NZP, nk = Nzg - 1;
    const float rnk = recip(nk);
    for (int t = threadIdx.x; t < n3 * nk; t += blockDim.x) {
        const int q = quot(t, rnk), k = 1 + t - q * nk;
        const bool xw = q < n1;
        const int side = xw ? (q >= n0) : (q >= n2);
        const int p = q - (xw ? (side ? n0 : 0) : (side ? n2 : n1));
        if (xw) {
            const int gi = side ? Nxg : 1, d = side ? -1 : 1, j = jlo + p, li = gi - r.ra, lj = j - r.sa;
            f(slot(g, li, lj) + k, slot(g, li + d, lj) + k, slot(g, li + 2 * d, lj) + k, gi + d, j, true, side);
        } else {
            const int gj = side ? Nyg : 1, d = side ? -1 : 1, i = ilo + p, s = slot(g, i - r.ra, gj - r.sa) + k;
            f(s, s + d * row, s + 2 * d * row, i, gj + d, false, side);
        }
    }
}

// The same two rows at a time (arrays of even pitch): f(place of the pair in
// the ghost column, the nearest, the second; i + j of the nearest; x wall;
// side; first row).
template <bool THREE, typename F>
__device__ __forceinline__ void ghost_pairs(int Nxg, int Nyg, int per, const Reg& r, const TileGeo& g, F f) {
    const int jlo = THREE ? max(r.sa, 2) : 1, jhi = THREE ? min(r.sb, Nyg - 1) : 1;
    const int ilo = per ? r.ra : max(r.ra, 2), ihi = per ? r.rb : min(r.rb, Nxg - 1);
    const int nx = jhi - jlo + 1, ny = ihi - ilo + 1;
    const int n0 = !per && r.ra == 1 ? nx : 0, n1 = n0 + (!per && r.rb == Nxg ? nx : 0);
    const int n2 = n1 + (THREE && r.sa == 1 ? ny : 0), n3 = n2 + (THREE && r.sb == Nyg ? ny : 0);
    const int row = row_slot(g, 1);
    const float rnp = recip(g.np);
    for (int t = threadIdx.x; t < n3 * g.np; t += blockDim.x) {
        const int q = quot(t, rnp), k = 2 * (t - q * g.np);
        const bool xw = q < n1;
        const int side = xw ? (q >= n0) : (q >= n2);
        const int p = q - (xw ? (side ? n0 : 0) : (side ? n2 : n1));
        if (xw) {
            const int d = side ? -1 : 1, li = (side ? Nxg : 1) - r.ra, o = row_slot(g, jlo + p - r.sa) + k;
            f(o + col_slot(g, li), o + col_slot(g, li + d), o + col_slot(g, li + 2 * d), li + d + r.ra + jlo + p, true, side, k);
        } else {
            const int d = side ? -row : row, s = slot(g, ilo + p - r.ra, (side ? Nyg : 1) - r.sa) + k;
            f(s, s + d, s + 2 * d, ilo + p + (side ? Nyg - 1 : 2), false, side, k);
        }
    }
}

// Owned coarse columns of a core span [a, b] of an axis of nf fine and nc
// coarse columns, coarsened (F = 2) or not (F = 1).
__device__ __forceinline__ void owned(int a, int b, int nf, int nc, int F, int per, int& lo, int& hi) {
    const int s = F - 1;
    if (per) { lo = 2 + ((a - 2 + s) >> s); hi = 2 + ((b - 2) >> s); return; }
    lo = a == 1 ? 1 : (a == nf ? nc : 2 + ((a - 2 + s) >> s));
    hi = b == nf ? nc : (b == 1 ? 1 : 2 + ((b - 2) >> s));
}

// Restrict the residual staged in rs to the owned coarse columns
// (MGRestriction3DExplicit.f90:19-128; on a uniform grid the weights in x and
// y are 1/4, 1/2, 1/4). The residual is zero on the ghost columns, in the
// bottom rows and in the free-surface row: a smoothing step ends with these
// rows relaxed last. Four lanes share a coarse column.
template <bool THREE, bool VEC, typename T>
__device__ __forceinline__ void restrict_tile(const LevelDev<T>& F, const LevelDev<T>& Cc, const TileGeo& g,
                                              const Reg& r, int bx, const T* rs, T* __restrict__ rc,
                                              T* __restrict__ zero) {
    const int per = F.per, Ncz = Cc.Nzg, xc = Cc.xc, yc = THREE ? Cc.yc : 0;
    int clo, chi, dlo = 1, dhi = 1;
    owned(r.ia, r.ib, F.Nxg, Cc.Nxg, 1 + xc, per, clo, chi);
    if (THREE) owned(r.ja, r.jb, F.Nyg, Cc.Nyg, 1 + yc, 0, dlo, dhi);
    const int nx = chi - clo + 1, ny = dhi - dlo + 1;
    constexpr int P = 4;
    const int part = threadIdx.x % P;
    const float rnx = recip(nx);
    for (int cq = threadIdx.x / P; cq < nx * ny; cq += blockDim.x / P) {
        const int cj = quot(cq, rnx), ic = clo + cq - cj * nx, jc = dlo + cj;
        T* const ro = rc + (int64_t)Ncz * ((ic - 1) + Cc.Nxg * (jc - 1));
        T* const zo = zero ? zero + (ro - rc) : nullptr;
        const bool ghost = (!per && (ic == 1 || ic == Cc.Nxg)) || (THREE && (jc == 1 || jc == Cc.Nyg));
        const int i = 2 + (ic - 2) * (1 + xc), j = THREE ? 2 + (jc - 2) * (1 + yc) : 1;
        const int li = ghost ? 0 : i - r.ra, lj = ghost ? 0 : j - r.sa;
        const T* const p = rs + slot(g, li, lj);
        const int nl = near_l(g, li), nr = near_r(g, li), row = row_slot(g, 1);
        // zero weight for ghost neighbours
        const T wl = !per && i == 2 ? T(0) : T(0.25), wr = !per && i == F.Nxg - 1 ? T(0) : T(0.25);
        const T wd = j == 2 ? T(0) : T(0.25), wu = j == F.Nyg - 1 ? T(0) : T(0.25);
        auto xsum = [&](const T* q) -> T { return xc ? T(0.5) * q[0] + (wl * q[nl] + wr * q[nr]) : q[0]; };
        auto plane = [&](int k) -> T {
            const T* const q = p + k;
            return yc ? T(0.5) * xsum(q) + (wd * xsum(q - row) + wu * xsum(q + row)) : xsum(q);
        };
        if (VEC && !Cc.zc && (Ncz & 1) == 0) {   // two rows at a time
            for (int kc = 2 * part; kc < Ncz; kc += 2 * P) {
                T v0 = 0, v1 = 0;
                if (!ghost) {
                    auto xsum2 = [&](const T* q, T& a, T& b) {
                        const auto m = pair_at(q);
                        if (!xc) { a = m.x; b = m.y; return; }
                        const auto l = pair_at(q + nl), h = pair_at(q + nr);
                        a = T(0.5) * m.x + (wl * l.x + wr * h.x);
                        b = T(0.5) * m.y + (wl * l.y + wr * h.y);
                    };
                    xsum2(p + kc, v0, v1);
                    if (yc) {
                        T d0, d1, u0, u1;
                        xsum2(p + kc - row, d0, d1);
                        xsum2(p + kc + row, u0, u1);
                        v0 = T(0.5) * v0 + (wd * d0 + wu * u0);
                        v1 = T(0.5) * v1 + (wd * d1 + wu * u1);
                    }
                    if (kc == 0) v0 = 0;
                    if (kc + 2 == Ncz) v1 = 0;
                }
                put_pair(ro + kc, v0, v1);
                if (zo) put_pair(zo + kc, T(0), T(0));
            }
            continue;
        }
        for (int kc = part; kc < Ncz; kc += P) {
            T v = 0;
            if (!ghost && kc >= 1 && kc <= Ncz - 2) {
                if (!Cc.zc) {
                    v = plane(kc);
                } else {
                    const int k = 1 + (kc - 1) * 2;   // 0-based fine row
                    const double dU = F.z[k + 1] - F.z[k], dD = F.z[k] - F.z[k - 1];
                    const T h = T(0.5) * T(F.iz[k]);
                    v = T(0.5) * plane(k);
                    if (k > 1) v += h * T(dD) * plane(k - 1);
                    if (k + 1 <= F.Nzg - 2) v += h * T(dU) * plane(k + 1);
                }
            }
            ro[kc] = v;
            if (zo) zo[kc] = T(0);
        }
    }
    if (per && bx == 0) {   // the coarse image columns
        for (int t = threadIdx.x; t < 3 * ny * Ncz; t += blockDim.x) {
            const int cq = t / Ncz, k = t - cq * Ncz, jc = dlo + cq / 3, w = cq % 3;
            const int col = w == 0 ? 1 : (w == 1 ? Cc.Nxg - 1 : Cc.Nxg);
            const int o = k + Ncz * ((col - 1) + Cc.Nxg * (jc - 1));
            rc[o] = T(0);
            if (zero) zero[o] = T(0);
        }
    }
}

// A level's right-hand side as the kernels read it: of the level's own type, or
// for the finest level the solver's FP64 vector times *scale (null: 1), which
// saves a pass that scales and converts it.
template <typename TB>
struct Rhs {
    const TB* p;
    const double* scale;
};
// Sums and products kept apart (the ordered form's transfers).
__device__ __forceinline__ float mul_rn(float a, float b) { return __fmul_rn(a, b); }
__device__ __forceinline__ float add_rn(float a, float b) { return __fadd_rn(a, b); }
__device__ __forceinline__ double mul_rn(double a, double b) { return a * b; }
__device__ __forceinline__ double add_rn(double a, double b) { return a + b; }

// Place of column (c, q) of the region: by column parity (slot), or FLAT: row
// by row, as the ordered cross form keeps it.
template <bool FLAT>
__device__ __forceinline__ int tile_slot(const TileGeo& g, int c, int q) {
    return FLAT ? (2 * g.HW * q + c) * g.NZP : slot(g, c, q);
}

template <typename T, typename TB>
__device__ __forceinline__ T rhs_value(TB v, double s) {
    if constexpr (sizeof(TB) == 8) return T(s * v);
    else return v;
}

// Accessor of stage_up (sweep_n).
template <typename T, typename TB, bool THREE, bool VEC, bool FLAT>
struct UpAcc {
    const TB* b;                // at column 1 of the region's first row and the thread's k
    double scale;
    const T *x, *xc;            // likewise; the coarse field at the thread's k
    T *xs, *bs;
    const LevelDev<T>& F;
    const LevelDev<T>& Cc;
    const TileGeo& g;
    int ra, sa, k;
    bool first, last;           // this k is the bottom row / ends in the free-surface row
    template <int N>
    struct Val { T x[N]; TB b[N]; T c[THREE ? 4 : 2][N]; };
    // the coarse columns around fine column i (0-based, in values), row j's two
    __device__ __forceinline__ void coarse_cols(int i, int& i0, int& i1) const {
        i0 = Cc.xc ? 1 + ((i - 2) >> 1) : i - 1;
        i1 = Cc.xc ? i0 + (i & 1) : i0;
        if (F.per && i1 == Cc.Nxg - 2) i1 = 1;
        i0 *= Cc.Nzg;
        i1 *= Cc.Nzg;
    }
    __device__ __forceinline__ void coarse_rows(int j, const T*& c0, const T*& c1) const {
        const int nrow = Cc.Nzg * Cc.Nxg, j0 = !THREE ? 0 : (Cc.yc ? 1 + ((j - 2) >> 1) : j - 1);
        c0 = xc + nrow * j0;
        c1 = c0 + (THREE && Cc.yc && (j & 1) ? nrow : 0);
    }
    template <int N>
    __device__ __forceinline__ void ld(Val<N>& v, int c, int q) const {
        const int i = gcol(ra + c, F.Nxg, F.per);
        const int e = F.Nzg * (i - 1 + F.Nxg * q);
        get<N>(v.x, x + e);
        get<N>(v.b, b + e);
        if (Cc.zc) return;      // (uniform) the sigma form loads in st
        int i0, i1;             // in range on ghost columns too
        coarse_cols(i, i0, i1);
        const T *c0, *c1;
        coarse_rows(sa + q, c0, c1);
        get<N>(v.c[0], c0 + i0);
        get<N>(v.c[1], c0 + i1);
        if constexpr (THREE) {
            get<N>(v.c[2], c1 + i0);
            get<N>(v.c[3], c1 + i1);
        }
    }
    template <int N>
    __device__ __forceinline__ void st(int c, int q, const Val<N>& v) const {
        const int i = gcol(ra + c, F.Nxg, F.per), j = sa + q;
        const bool ghost = (!F.per && (i == 1 || i == F.Nxg)) || (THREE && (j == 1 || j == F.Nyg));
        T xv[N], bv[N];
#pragma unroll
        for (int n = 0; n < N; ++n) {
            xv[n] = v.x[n];
            bv[n] = rhs_value<T>(v.b[n], scale);
            if (!Cc.zc) {
                T d = v.c[0][n] + v.c[1][n];
                if constexpr (THREE) d = T(0.25) * (d + (v.c[2][n] + v.c[3][n]));
                else d = T(0.5) * d;
                if (!ghost && !(first && n == 0) && !(last && n == N - 1)) xv[n] += d;
            } else if (!ghost && k + n >= 1 && k + n <= F.Nzg - 2) {
                int i0, i1;
                coarse_cols(i, i0, i1);
                const T *c0, *c1;
                coarse_rows(j, c0, c1);
                auto avg = [&](int z) -> T {
                    const T d = c0[i0 + z] + c0[i1 + z];
                    return THREE ? T(0.25) * (d + (c1[i0 + z] + c1[i1 + z])) : T(0.5) * d;
                };
                const int kk = k + n;
                const T w1 = __ldg(F.pwz + 2 * kk + 1);
                T d = mul_rn(__ldg(F.pwz + 2 * kk), avg(__ldg(F.piz + 2 * kk) - 1));
                if (w1 != T(0)) d += w1 * avg(__ldg(F.piz + 2 * kk + 1) - 1);
                xv[n] = add_rn(xv[n], d);
            }
        }
        const int s = tile_slot<FLAT>(g, c, q);
        put<N, VEC>(xs + s, xv);
        put<N, VEC>(bs + s, bv);
    }
};

// Stage the corrected iterate xin + P xc (MGProlongation3DExplicit.f90:19-110;
// in x and y the average of the one, two or four coarse columns around a
// point, in sigma by the level's table where the coarse grid is coarsened
// there too; ghost columns, bottom and free-surface rows take no correction)
// in xs and the right-hand side in bs.
template <bool THREE, bool VEC, bool FLAT, typename T, typename TB>
__device__ __forceinline__ void stage_up(const LevelDev<T>& F, const LevelDev<T>& Cc, const TileGeo& g, const Reg& r,
                                         const TB* __restrict__ b, const double* __restrict__ bscale,
                                         const T* __restrict__ xin, const T* __restrict__ xc, T* xs, T* bs) {
    const int64_t o = (int64_t)F.Nzg * F.Nxg * (r.sa - 1);
    const double scale = bscale ? *bscale : 1.0;
    sweep<2>(r.W, r.H, F.Nzg, [&](int k) {
        const int end = k + ((F.Nzg & 1) == 0 ? 1 : 0);
        return UpAcc<T, TB, THREE, VEC, FLAT>{b + o + k, scale, xin + o + k, xc + (Cc.zc ? 0 : k), xs + k, bs + k, F, Cc, g,
                                        r.ra, r.sa, k, k == 0, end == F.Nzg - 1};
    });
}

// Accessor of stage_down (sweep_n); INPLACE: the right-hand side goes where the
// iterate will be.
template <typename T, typename TB, bool THREE, bool VEC, bool INPLACE, bool FLAT>
struct DownAcc {
    const TB* b;                // at column 1 of the region's first row and the thread's k
    double scale;
    T *xs, *bs;
    const TileGeo& g;
    const T (*gx)[3], (*gy)[3];
    int ra, sa, Nxg, Nyg, per, nz;
    bool first;                 // this k is the bottom row
    bool wall;                  // the region touches a wall
    template <int N>
    struct Val { TB b[N]; };
    template <int N>
    __device__ __forceinline__ void ld(Val<N>& v, int c, int q) const {
        get<N>(v.b, b + nz * (gcol(ra + c, Nxg, per) - 1 + Nxg * q));
    }
    template <int N>
    __device__ __forceinline__ void st(int c, int q, const Val<N>& v) const {
        const int s = tile_slot<FLAT>(g, c, q), i = ra + c, j = sa + q;
        T bv[N], x[N];
#pragma unroll
        for (int n = 0; n < N; ++n) { bv[n] = rhs_value<T>(v.b[n], scale); x[n] = INPLACE ? bv[n] : T(0); }
        if (!INPLACE) put<N, VEC>(bs + s, bv);
        const bool x0 = !per && i == 1, x1 = !per && i == Nxg, y0 = THREE && j == 1, y1 = THREE && j == Nyg;
        if (wall && (x0 || x1 || y0 || y1)) {
            const T w = (x0 || x1) && (y0 || y1) ? T(1) : (gx ? (x0 || x1 ? gx[x1][2] : gy[y1][2]) : T(0));
#pragma unroll
            for (int n = 0; n < N; ++n) x[n] = first && n == 0 ? bv[n] : w * bv[n];
        }
        put<N, VEC>(xs + s, x);
    }
};

// Stage the right-hand side in bs and in xs the zero iterate (INPLACE: in xs
// the right-hand side) with the identity rows (corner columns, level 1 of the
// ghost columns: b) and, gx[w][2] and gy[w][2] being one over the ghost weight
// of wall w, the ghost rows relaxed (null: left at zero).
template <bool THREE, bool VEC, bool INPLACE, bool FLAT, typename T, typename TB>
__device__ __forceinline__ void stage_down(const LevelDev<T>& F, const TileGeo& g, const Reg& r,
                                           const TB* __restrict__ b, const double* __restrict__ bscale, T* xs, T* bs,
                                           const T (*gx)[3], const T (*gy)[3]) {
    const int64_t o = (int64_t)F.Nzg * F.Nxg * (r.sa - 1);
    const double scale = bscale ? *bscale : 1.0;
    sweep<4>(r.W, r.H, F.Nzg, [&](int k) {
        return DownAcc<T, TB, THREE, VEC, INPLACE, FLAT>{b + o + k, scale, xs + k, bs + k, g, gx, gy, r.ra, r.sa, F.Nxg, F.Nyg, F.per,
                                          F.Nzg, k == 0, at_wall(F.Nxg, F.Nyg, F.per, r, THREE)};
    });
}

// Accessor of write_core (sweep_n).
template <typename T, bool VEC>
struct CoreAcc {
    const T* xs;                // at the thread's k
    T* out;                     // at the core's first column and the thread's k
    const TileGeo& g;
    int c0, q0, nz, Nxg;
    template <int N>
    struct Val { T x[N]; };
    template <int N>
    __device__ __forceinline__ void ld(Val<N>& v, int c, int q) const {
        const T* const p = xs + slot(g, c + c0, q + q0);
        if constexpr (N == 2 && VEC) {
            get<2>(v.x, p);
        } else {
#pragma unroll
            for (int n = 0; n < N; ++n) v.x[n] = p[n];
        }
    }
    template <int N>
    __device__ __forceinline__ void st(int c, int q, const Val<N>& v) const {
        put<N, true>(out + nz * (c + Nxg * q), v.x);
    }
};

// Write the core columns of the staged array (periodic x: and zeros in the
// image columns).
template <bool THREE, bool VEC, typename T>
__device__ __forceinline__ void write_core(const LevelDev<T>& F, const Reg& r, const TileGeo& g, int bx, const T* xs,
                                           T* __restrict__ out) {
    const int Nzg = F.Nzg, Nxg = F.Nxg, H = r.jb - r.ja + 1;
    T* const o = out + (int64_t)Nzg * ((r.ia - 1) + (int64_t)Nxg * (r.ja - 1));
    sweep<4>(r.ib - r.ia + 1, H, Nzg, [&](int k) {
        return CoreAcc<T, VEC>{xs + k, o + k, g, r.ia - r.ra, r.ja - r.sa, Nzg, Nxg};
    });
    if (F.per && bx == 0)
        for (int t = threadIdx.x; t < 3 * H * Nzg; t += blockDim.x) {
            const int cq = t / Nzg, k = t - cq * Nzg, w = cq % 3;
            const int col = w == 0 ? 1 : (w == 1 ? Nxg - 1 : Nxg);
            out[k + Nzg * ((col - 1) + Nxg * (r.ja + cq / 3 - 1))] = T(0);
        }
}

// ----------------------------------------------------------- uniform levels

// A uniform column's rows lie in pairs (even pitch): every access of the
// column code below moves two rows, half the shared-memory instructions.
// Pitch / 2 is odd, so that the pairs of neighbouring columns, which the
// threads of a warp take together, fall on different banks.

// Neighbour columns' part of rows k and k + 1.
template <bool THREE, typename T>
__device__ __forceinline__ void uni_off(const UniTab<T>& u, const T* xp, int l, int r, int row, int k, T* o) {
    const auto a = pair_at(xp + l + k), b = pair_at(xp + r + k);
    o[0] = u.wxl * a.x + u.wxr * b.x;
    o[1] = u.wxl * a.y + u.wxr * b.y;
    if (THREE) {
        const auto d = pair_at(xp - row + k), e = pair_at(xp + row + k);
        o[0] += u.wyd * d.x + u.wyu * e.x;
        o[1] += u.wyd * d.y + u.wyu * e.y;
    }
}

// Rows of a column whose sums are formed together: enough loads in flight,
// few enough for the registers of two blocks per SM (18 rows at once spill).
__host__ __device__ constexpr int uni_chunk(int nzg) { return nzg == 0 ? 8 : (nzg <= 10 ? (nzg + 1) / 2 * 2 : 6); }

// Rows 2..Nzg-1 of the column at xp bottom to top, then its bottom row and
// its free-surface row: x_k = (b_k - off_k - up_k x_{k+1}) id_k - g_k x_{k-1}.
// A chunk's sums are formed before its first new value is stored, so their
// loads are in flight together and only the chain's one multiply-add per row
// is serial. off(k, o): the neighbour columns' part of rows k, k + 1; ZERO: the
// column's own old iterate is zero.
template <int NZG, bool ZERO, typename T, typename OFF>
__device__ __forceinline__ void uni_column(const UniTab<T>& u, int nzg, T* xp, const T* bp, OFF off) {
    const int Nzg = NZG > 0 ? NZG : nzg;
    constexpr int CH = uni_chunk(NZG);
    const T b1 = bp[0];
    T xprev = ZERO ? b1 * u.t6 : (b1 - u.t0 * xp[1] - u.t1 * xp[2]) * u.t6;
    T x2 = 0, x3 = 0;
#pragma unroll
    for (int k0 = 0; k0 < Nzg; k0 += CH) {
        T q[CH], xo[CH + 1];
        if (!ZERO) {
#pragma unroll
            for (int m = 0; m < CH; m += 2)
                if (k0 + m < Nzg) { const auto v = pair_at(xp + k0 + m); xo[m] = v.x; xo[m + 1] = v.y; }
            xo[CH] = k0 + CH < Nzg ? xp[k0 + CH] : T(0);
        }
#pragma unroll
        for (int m = 0; m < CH; m += 2) {
            if (k0 + m >= Nzg) continue;
            const auto v = pair_at(bp + k0 + m);
            T o[2];
            off(k0 + m, o);
            q[m] = v.x; q[m + 1] = v.y;
#pragma unroll
            for (int n = 0; n < 2; ++n) {
                const int k = k0 + m + n;
                if (k >= 1 && k < Nzg - 1)
                    q[m + n] = ((ZERO ? q[m + n] : q[m + n] - u.up[k] * xo[m + n + 1]) - o[n]) * u.id[k];
            }
        }
#pragma unroll
        for (int m = 0; m < CH; ++m) {
            const int k = k0 + m;
            if (k >= 1 && k < Nzg - 1) {
                xprev = q[m] - u.g[k] * xprev;
                q[m] = xprev;
                if (k == 1) x2 = xprev;
                if (k == 2) x3 = xprev;
            }
        }
#pragma unroll
        for (int m = 0; m < CH; m += 2)
            if (k0 + m < Nzg) put_pair(xp + k0 + m, q[m], q[m + 1]);   // the free-surface row: b
    }
    xp[0] = (b1 - u.t0 * x2 - u.t1 * x3) * u.t6;
}

// Down, in place: xs holds b and is overwritten by the iterate column by
// column -- from x = 0 a colour-0 column reads no column but ghosts, a colour-1
// column only colour-0 and ghost columns -- and then by the residual, which
// follows from what changed after a row was solved, so b is not needed again:
//   colour 1: -up x_{k+1};  colour 0: that and -w x of its colour-1
//   neighbours; next to a wall, the change of the ghost value; in row 2 the
//   second update of the bottom row.
// Colour 0's residual first (it reads colour 1's iterate), then colour 1's
// (its own column only).

// Colour 0 (FIRST) or 1 of the smoothing step, at distance <= 3 or 2.
template <bool THREE, int NZG, bool FIRST, typename T>
__device__ __forceinline__ void uni_first(const LevelDev<T>& F, const UniTab<T>& u, const TileGeo& g, const Reg& r, T* xs) {
    const int Nxg = F.Nxg, Nyg = F.Nyg, per = F.per, row = row_slot(g, 1);
    colour_columns<THREE>(Nxg, Nyg, per, r, 2, FIRST ? 0 : 1, FIRST ? 3 : 2, [&](int i, int j) {
        const int li = i - r.ra, l = near_l(g, li), h = near_r(g, li);
        T* const xp = xs + slot(g, li, j - r.sa);
        if (!FIRST) {
            uni_column<NZG, true>(u, F.Nzg, xp, xp, [&](int k, T* o) { uni_off<THREE>(u, xp, l, h, row, k, o); });
            return;
        }
        const bool el = !per && i == 2, er = !per && i == Nxg - 1, ed = THREE && j == 2, eu = THREE && j == Nyg - 1;
        if (el || er || ed || eu) {
            uni_column<NZG, true>(u, F.Nzg, xp, xp, [&](int k, T* o) {
                o[0] = o[1] = T(0);
                auto add = [&](bool on, T w, int at) {
                    if (!on) return;
                    const auto v = pair_at(xp + at + k);
                    o[0] += w * v.x;
                    o[1] += w * v.y;
                };
                add(el, u.wxl, l);
                add(er, u.wxr, h);
                add(ed, u.wyd, -row);
                add(eu, u.wyu, row);
            });
        } else {
            uni_column<NZG, true>(u, F.Nzg, xp, xp, [&](int, T* o) { o[0] = o[1] = T(0); });
        }
    });
}

// The columns of one colour at distance <= 1: residual in place.
template <bool THREE, int NZG, bool FIRST, typename T>
__device__ __forceinline__ void uni_residual(const LevelDev<T>& F, const UniTab<T>& u, const TileGeo& g, const Reg& r,
                                             T* xs) {
    const int Nxg = F.Nxg, Nyg = F.Nyg, per = F.per, row = row_slot(g, 1), Nzg = NZG > 0 ? NZG : F.Nzg;
    constexpr int CH = uni_chunk(NZG);
    // add(k, q): the side terms of rows k, k + 1
    auto column = [&](T* xp, auto add) {
        const T c2 = u.lo[1] * u.t6 * (u.t0 * xp[1] + u.t1 * xp[2]);   // the bottom row's second update
#pragma unroll
        for (int k0 = 0; k0 < Nzg; k0 += CH) {
            T x[CH + 1], q[CH];
#pragma unroll
            for (int m = 0; m < CH; m += 2)
                if (k0 + m < Nzg) { const auto v = pair_at(xp + k0 + m); x[m] = v.x; x[m + 1] = v.y; }
            x[CH] = k0 + CH < Nzg ? xp[k0 + CH] : T(0);
#pragma unroll
            for (int m = 0; m < CH; m += 2) {
                if (k0 + m >= Nzg) continue;
                T o[2] = {T(0), T(0)};
                add(k0 + m, o);
#pragma unroll
                for (int n = 0; n < 2; ++n) {
                    const int k = k0 + m + n;
                    q[m + n] = x[m + n];
                    if (k >= 1 && k < Nzg - 1) q[m + n] = o[n] - u.up[k] * x[m + n + 1] + (k == 1 ? c2 : T(0));
                }
            }
#pragma unroll
            for (int m = 0; m < CH; m += 2)
                if (k0 + m < Nzg) put_pair(xp + k0 + m, q[m], q[m + 1]);
        }
    };
    colour_columns<THREE>(Nxg, Nyg, per, r, 2, FIRST ? 0 : 1, 1, [&](int i, int j) {
        const int li = i - r.ra, l = near_l(g, li), h = near_r(g, li);
        T* const xp = xs + slot(g, li, j - r.sa);
        const bool el = !per && i == 2, er = !per && i == Nxg - 1, ed = THREE && j == 2, eu = THREE && j == Nyg - 1;
        if (el || er || ed || eu) {
            column(xp, [&](int k, T* o) {
                // a ghost neighbour moved by -(wa x_near + wb x_second) / wg since the row was solved
                auto side = [&](bool wall, T w, const T* gw, int at, int opposite) {
                    if (wall) {
                        const auto v = pair_at(xp + k);
                        const T c = w * gw[2];
                        T d0 = gw[0] * v.x, d1 = gw[0] * v.y;
                        if (FIRST) { const auto z = pair_at(xp + opposite + k); d0 += gw[1] * z.x; d1 += gw[1] * z.y; }
                        o[0] += c * d0;
                        o[1] += c * d1;
                    } else if (FIRST) {
                        const auto z = pair_at(xp + at + k);
                        o[0] -= w * z.x;
                        o[1] -= w * z.y;
                    }
                };
                side(el, u.wxl, u.gx[0], l, h);
                side(er, u.wxr, u.gx[1], h, l);
                if (THREE) {
                    side(ed, u.wyd, u.gy[0], -row, row);
                    side(eu, u.wyu, u.gy[1], row, -row);
                }
            });
        } else if (FIRST) {
            column(xp, [&](int k, T* o) {
                uni_off<THREE>(u, xp, l, h, row, k, o);
                o[0] = -o[0];
                o[1] = -o[1];
            });
        } else {
            column(xp, [&](int, T*) {});
        }
    });
}

template <typename T, typename TB, bool THREE, int NZG>
__global__ void __launch_bounds__(kUniThreads, sizeof(T) == 8 ? 2 : 3)
    k_mg_down_uni(LevelDev<T> F, LevelDev<T> Cc, const TB* __restrict__ b, const double* __restrict__ scale,
                  T* __restrict__ xout, T* __restrict__ rc, T* __restrict__ zero, const __grid_constant__ UniTab<T> u,
                  TileGeo g) {
    pdl_entry();
    extern __shared__ __align__(16) unsigned char tile_smem[];
    T* const xs = reinterpret_cast<T*>(tile_smem);
    const int bx = blockIdx.x, by = blockIdx.y;
    const Reg r = region(F.Nxg, F.Nyg, F.per, g, bx, by, THREE);
    const bool wall = at_wall(F.Nxg, F.Nyg, F.per, r, THREE);
    stage_down<THREE, true, true, false>(F, g, r, b, scale, xs, xs, u.gx, u.gy);
    __syncthreads();
    // ghost rows: the contribution of the colour just solved
    auto ghosts = [&](int colour) {
        if (!wall) return;
        ghost_pairs<THREE>(F.Nxg, F.Nyg, F.per, r, g, [&](int s, int sa, int sb, int ij, bool xw, int side, int k) {
            const T* const w = xw ? u.gx[side] : u.gy[side];
            const bool near = (ij & 1) == colour;
            const auto v = pair_at(xs + s), a = pair_at(xs + (near ? sa : sb));
            const T c = (near ? w[0] : w[1]) * w[2];
            put_pair(xs + s, k == 0 ? v.x : v.x - c * a.x, v.y - c * a.y);   // level 1: an identity row
        });
        __syncthreads();
    };
    uni_first<THREE, NZG, true>(F, u, g, r, xs);
    __syncthreads();
    ghosts(0);
    uni_first<THREE, NZG, false>(F, u, g, r, xs);
    __syncthreads();
    ghosts(1);
    write_core<THREE, true>(F, r, g, bx, xs, xout);
    __syncthreads();
    uni_residual<THREE, NZG, true>(F, u, g, r, xs);
    __syncthreads();
    uni_residual<THREE, NZG, false>(F, u, g, r, xs);
    __syncthreads();
    restrict_tile<THREE, true>(F, Cc, g, r, bx, xs, rc, zero);
}

// One smoothing step on the staged iterate: colour c at distance <= 1 - c, the
// ghost rows relaxed before, between and after.
template <bool THREE, int NZG, typename T>
__device__ __forceinline__ void uni_smooth(const LevelDev<T>& F, const UniTab<T>& u, const TileGeo& g, const Reg& r,
                                           T* xs, const T* bs) {
    const bool wall = at_wall(F.Nxg, F.Nyg, F.per, r, THREE);
    auto ghosts = [&]() {
        if (!wall) return;
        ghost_pairs<THREE>(F.Nxg, F.Nyg, F.per, r, g, [&](int s, int sa, int sb, int, bool xw, int side, int k) {
            const T* const w = xw ? u.gx[side] : u.gy[side];
            const auto b = pair_at(bs + s), a = pair_at(xs + sa), c = pair_at(xs + sb);
            const T v0 = (b.x - w[0] * a.x - w[1] * c.x) * w[2], v1 = (b.y - w[0] * a.y - w[1] * c.y) * w[2];
            put_pair(xs + s, k == 0 ? b.x : v0, v1);   // level 1: an identity row
        });
        __syncthreads();
    };
    ghosts();
    const int row = row_slot(g, 1);
    for (int colour = 0; colour < 2; ++colour) {
        colour_columns<THREE>(F.Nxg, F.Nyg, F.per, r, 2, colour, 1 - colour, [&](int i, int j) {
            const int li = i - r.ra, s = slot(g, li, j - r.sa), l = near_l(g, li), h = near_r(g, li);
            T* const xp = xs + s;
            uni_column<NZG, false>(u, F.Nzg, xp, bs + s, [&](int k, T* o) { uni_off<THREE>(u, xp, l, h, row, k, o); });
        });
        __syncthreads();
        ghosts();
    }
}

template <typename T, typename TB, bool THREE, int NZG>
__global__ void __launch_bounds__(256, sizeof(T) == 8 ? 2 : 3) k_mg_up_uni(LevelDev<T> F, LevelDev<T> Cc, const TB* __restrict__ b,
                                                   const double* __restrict__ scale,
                                                   const T* __restrict__ xin, const T* __restrict__ xc,
                                                   T* __restrict__ out, const __grid_constant__ UniTab<T> u, TileGeo g) {
    pdl_entry();
    extern __shared__ __align__(16) unsigned char tile_smem[];
    T* const xs = reinterpret_cast<T*>(tile_smem);
    T* const bs = xs + 2 * g.HW * g.PH * g.NZP;
    const int bx = blockIdx.x, by = blockIdx.y;
    const Reg r = region(F.Nxg, F.Nyg, F.per, g, bx, by, THREE);
    stage_up<THREE, true, false>(F, Cc, g, r, b, scale, xin, xc, xs, bs);
    __syncthreads();
    uni_smooth<THREE, NZG>(F, u, g, r, xs, bs);
    write_core<THREE, true>(F, r, g, bx, xs, out);
}

// ------------------------------------------------------------- cross levels

// The mixed derivatives d2/dxds (replicated over three y planes) and d2/dyds
// (over three x planes) of row k are om_k sum_m z_m D(k-1+m) with one
// horizontal 9-point sum per level
//   D(k) = sum_ab 2 (ca sx_a + cb sy_b) x(i-1+a, j-1+b, k),
// the factors ca = h_x/h, cb = h_y/h taken out of the sums (54 products per
// row as the two sums are written, 9 this way).
template <typename T, bool THREE>
struct CrossCol {
    T ih, ca, cb, c3;           // 1/h, h_x/h, h_y/h and the sigma-3 factor
    T W[THREE ? 9 : 3];
    __device__ __forceinline__ CrossCol(const T* cf, const RowTab<T>& t) : ih(cf[0]), ca(cf[1]), cb(cf[2]), c3(cf[3]) {
#pragma unroll
        for (int b = 0; b < (THREE ? 3 : 1); ++b)
#pragma unroll
            for (int a = 0; a < 3; ++a) {
                W[3 * b + a] = T(2) * ca * t.sx1[a];
                if (THREE) W[3 * b + a] += T(2) * cb * t.sy1[b];
            }
    }
    __device__ __forceinline__ T centre() const { return W[THREE ? 4 : 1]; }
    // row coefficients below, on and above the diagonal without the mixed terms
    __device__ __forceinline__ void row(const RowTab<T>& t, int k, T& lo, T& dg, T& up) const {
        const T om = t.om[k], s3 = om * c3, cz = om * om * (ca * ca + cb * cb) + ih * ih;
        lo = s3 * t.z0[k] + cz * t.y0[k];
        dg = s3 * t.z1[k] + cz * t.y1[k] + t.sx2[1] + (THREE ? t.sy2[1] : T(0));
        up = s3 * t.z2[k] + cz * t.y2[k];
    }
};

// Staged arrays of a cross tile: the columns' coefficients ([slot][4]), the
// iterate, and the right-hand side (replaced by the residual on the way down).
template <typename T>
struct CrossTile {
    T *cf, *xs, *bs;
};

// D(k) without the own column at p = the column's row k; off: the axis
// neighbours' part of the row (d2/dx2, d2/dy2).
template <typename T, bool THREE>
__device__ __forceinline__ T cross_sum(const CrossCol<T, THREE>& c, const RowTab<T>& t, const T* p, int nl, int nr,
                                       int nrow, T& off) {
    const T xl = p[nl], xr = p[nr];
    off = t.sx2[0] * xl + t.sx2[2] * xr;
    if (!THREE) return c.W[0] * xl + c.W[2] * xr;
    const T xd = p[-nrow], xu = p[nrow];
    off += t.sy2[0] * xd + t.sy2[2] * xu;
    return (c.W[0] * p[nl - nrow] + c.W[1] * xd + c.W[2] * p[nr - nrow]) + (c.W[3] * xl + c.W[5] * xr) +
           (c.W[6] * p[nl + nrow] + c.W[7] * xu + c.W[8] * p[nr + nrow]);
}

// D(1), the level below the bottom, the own column included, next to a wall:
// its stencils are shifted off the ghost corner columns.
template <typename T, bool THREE>
__device__ T cross_level1(const CrossCol<T, THREE>& c, const RowTab<T>& t, const TileGeo& g, const T* xs, int Nxg,
                          int Nyg, int i, int j, int li, int lj) {
    const int sh = i == 2 ? 1 : (i == Nxg - 1 ? -1 : 0);
    const int shy = !THREE ? 0 : (j == 2 ? 1 : (j == Nyg - 1 ? -1 : 0));
    const T* const wx = sh == 0 ? t.sx1 : t.ex[sh > 0 ? 0 : 1];
    T vx = 0, vy = 0;
    for (int b = (THREE ? -1 : 0); b <= (THREE ? 1 : 0); ++b)
        for (int a = 0; a < 3; ++a) vx += wx[a] * xs[slot(g, li - 1 + sh + a, lj + b)];
    if (THREE) {
        const T* const wy = shy == 0 ? t.sy1 : t.ey[shy > 0 ? 0 : 1];
        for (int a = -1; a <= 1; ++a)
            for (int b = 0; b < 3; ++b) vy += wy[b] * xs[slot(g, li + a, lj - 1 + shy + b)];
    }
    return T(2) * c.ca * vx + T(2) * c.cb * vy;
}

// Columns of `colour` at distance <= d of the core, one per segment of S
// lanes, lane r holding rows 1+2r and 2+2r (0-based): the sums of a column's
// rows are formed by its lanes together, and the chain over the rows is a
// shuffle scan of the lanes' composed maps x -> a x + b. (One thread per
// column instead: 31-33 us per launch at any level size, the latency of 8
// rows one after another per colour.) RES: replace the right-hand side by the
// residual instead of solving.
template <typename T, bool THREE, int S, bool RES>
__device__ __forceinline__ void cross_pass(const LevelDev<T>& F, const RowTab<T>& t, const TileGeo& g, const Reg& r,
                                           const CrossTile<T>& w, int ncolor, int colour, int d) {
    const int Nxg = F.Nxg, Nyg = F.Nyg, Nzg = F.Nzg;
    const int ilo = max(r.ia - d, 2), ihi = min(r.ib + d, Nxg - 1);
    int jlo = 1, jhi = 1, js = 1;
    if (THREE) { jlo = max(r.ja - d, 2); jhi = min(r.jb + d, Nyg - 1); }
    const bool four = ncolor == 4;
    if (!RES && THREE && four) { jlo += (jlo ^ (colour >> 1)) & 1; js = 2; }
    const int ni = RES ? max(ihi - ilo + 1, 0) : (ihi - ilo + 2) >> 1, nj = jhi >= jlo ? (jhi - jlo) / js + 1 : 0;
    const int total = ni * nj, lane = threadIdx.x & 31, rr = lane & (S - 1);
    const int per_warp = 32 / S, step = (blockDim.x >> 5) * per_warp;
    const int ka = 1 + 2 * rr, kb = ka + 1;
    const int kac = min(ka, Nzg - 1), kbc = min(kb, Nzg - 1);
    const int nrow = row_slot(g, 1);
    const float rni = recip(ni);
    for (int base = (threadIdx.x >> 5) * per_warp; base < total; base += step) {
        const int q = base + lane / S;
        const int tq = min(q, total - 1), tj = quot(tq, rni), j = jlo + tj * js;
        const int par = four ? colour & 1 : (colour + j) & 1;
        int i = RES ? ilo + tq - tj * ni : ilo + ((ilo ^ par) & 1) + 2 * (tq - tj * ni);
        const bool act = q < total && i <= ihi;
        if (i > ihi) i = ihi;                       // an idle segment reads a column in range
        const int li = i - r.ra, lj = j - r.sa;
        const int cs = (lj * 2 + (li & 1)) * g.HW + (li >> 1), s = cs * g.NZP;
        const int nl = near_l(g, li), nr = near_r(g, li);
        const CrossCol<T, THREE> c(w.cf + 4 * cs, t);
        T* const p = w.xs + s;
        T* const bp = w.bs + s;
        const T wc = c.centre();
        T offa, offb, offx;
        T Da = cross_sum<T, THREE>(c, t, p + kac, nl, nr, nrow, offa);
        T Db = cross_sum<T, THREE>(c, t, p + kbc, nl, nr, nrow, offb);
        // lane 0: the level below the bottom; the last row's lane: the free surface
        const int kx = rr == 0 ? 0 : Nzg - 1;
        T Dx = cross_sum<T, THREE>(c, t, p + kx, nl, nr, nrow, offx);
        if (rr == 0) {
            if (i == 2 || i == Nxg - 1 || (THREE && (j == 2 || j == Nyg - 1)))
                Dx = cross_level1<T, THREE>(c, t, g, w.xs, Nxg, Nyg, i, j, li, lj);
            else
                Dx += wc * p[0];
        }
        if (RES) {
            Da += wc * p[kac];
            Db += wc * p[kbc];
            if (rr != 0) Dx += wc * p[kx];
        }
        T Dm = __shfl_up_sync(0xffffffffu, Db, 1, S), Dn = __shfl_down_sync(0xffffffffu, Da, 1, S);
        if (rr == 0) Dm = Dx;
        if (kb == Nzg - 2) Dn = Dx;
        const T xka = p[kac], xkb = p[kbc], xkn = p[min(kb + 1, Nzg - 1)];
        const int ra = min(ka, Nzg - 2), rb = min(kb, Nzg - 2);   // row constants
        T loa, dga, upa, lob, dgb, upb;
        c.row(t, ra, loa, dga, upa);
        c.row(t, rb, lob, dgb, upb);
        const T oma = t.om[ra], omb = t.om[rb];
        T fa = bp[kac] - offa - oma * (t.z0[ra] * Dm + t.z1[ra] * Da + t.z2[ra] * Db);
        T fb = bp[kbc] - offb - omb * (t.z0[rb] * Da + t.z1[rb] * Db + t.z2[rb] * Dn);
        if (RES) {
            if (act) {
                if (ka <= Nzg - 2) bp[ka] = fa - loa * p[kac - 1] - dga * xka - upa * xkb;
                if (kb <= Nzg - 2) bp[kb] = fb - lob * xka - dgb * xkb - upb * xkn;
            }
        } else {
            // the own column's mixed terms join the chain (row 2's lower one is in D(1))
            const T wa = oma * wc, wb = omb * wc;
            if (rr != 0) loa += wa * t.z0[ra];
            dga += wa * t.z1[ra]; upa += wa * t.z2[ra];
            lob += wb * t.z0[rb]; dgb += wb * t.z1[rb]; upb += wb * t.z2[rb];
            const T ida = T(1) / dga, idb = T(1) / dgb;
            const T qa = (fa - upa * xkb) * ida, ga = loa * ida;
            const T qb = (fb - upb * xkn) * idb, gb = lob * idb;
            const bool va = ka <= Nzg - 2, vb = kb <= Nzg - 2;
            T a = 1, bb = 0;
            if (va) { bb = qa; a = -ga; }
            if (vb) { bb = qb - gb * bb; a = -gb * a; }
#pragma unroll
            for (int dd = 1; dd < S; dd <<= 1) {
                const T ap = __shfl_up_sync(0xffffffffu, a, dd, S);
                const T bq = __shfl_up_sync(0xffffffffu, bb, dd, S);
                if (rr >= dd) { bb = a * bq + bb; a = a * ap; }
            }
            const T ae = __shfl_up_sync(0xffffffffu, a, 1, S), be = __shfl_up_sync(0xffffffffu, bb, 1, S);
            const T x1 = p[0];                       // the bottom row is fixed during the pass
            const T xin = rr == 0 ? x1 : ae * x1 + be;
            const T xa = qa - ga * xin, xb = qb - gb * xa;
            const T xf = bp[Nzg - 1];
            __syncwarp();
            if (act) {
                if (va) p[ka] = xa;
                if (vb) p[kb] = xb;
                if (rr == 0) p[Nzg - 1] = xf;
            }
        }
    }
}

// Bottom row (k = 1) of every interior column at distance <= d, from its rows
// 2, 3 and the neighbours' row 2 (BuildLinearSystemMatrix.f90:50-70, the row
// times 1/h). FIRST: the iterate is zero.
template <typename T, bool THREE, bool FIRST>
__device__ __forceinline__ void cross_bottoms(const LevelDev<T>& F, const RowTab<T>& t, const TileGeo& g, const Reg& r,
                                              const CrossTile<T>& w, int d) {
    const int Nxg = F.Nxg, Nyg = F.Nyg, nrow = row_slot(g, 1);
    all_columns<THREE>(Nxg, Nyg, 0, r, d, [&](int i, int j) {
        const int li = i - r.ra, lj = j - r.sa;
        const int cs = (lj * 2 + (li & 1)) * g.HW + (li >> 1), s = cs * g.NZP;
        const T ih = w.cf[4 * cs], ca = w.cf[4 * cs + 1], cb = w.cf[4 * cs + 2];
        const T f = ih * ih + t.om[1] * (ca * ca + cb * cb);
        T* const p = w.xs + s;
        T v = w.bs[s] * ih;
        if (!FIRST) {
            const T* const p2 = p + 1;
            v -= f * (t.z1[1] * p[1] + t.z2[1] * p[2]) +
                 ca * (t.sx1[0] * p2[near_l(g, li)] + t.sx1[1] * p[1] + t.sx1[2] * p2[near_r(g, li)]);
            if (THREE) v -= cb * (t.sy1[0] * p2[-nrow] + t.sy1[1] * p[1] + t.sy1[2] * p2[nrow]);
        }
        p[0] = v / (f * t.z0[1]);
    });
    __syncthreads();
}

// Relax ghost rows from the current values: those whose stencil holds a
// column of colour `post` (just solved) and those next to a column of colour
// `pre` (to be solved, which reads them).
template <typename T, bool THREE>
__device__ __forceinline__ void cross_ghosts(const LevelDev<T>& F, const RowTab<T>& t, const Reg& r, const TileGeo& g,
                                             const CrossTile<T>& w, int ncolor, int post, int pre) {
    ghost_rows<THREE>(F.Nxg, F.Nyg, 0, F.Nzg, r, g, [&](int s, int sa, int sb, int ni, int nj, bool xw,
                                                                        int side) {
        auto has = [&](int i, int j, int colour) {
            return ncolor == 4 ? ((i & 1) == (colour & 1) && (j & 1) == (colour >> 1)) : ((i + j) & 1) == colour;
        };
        const int di = xw ? (side ? -1 : 1) : 0, dj = xw ? 0 : (side ? -1 : 1);
        const bool a = post >= 0 && (has(ni, nj, post) || has(ni + di, nj + dj, post));
        if (!a && !(pre < ncolor && has(ni, nj, pre))) return;
        const T* const gw = xw ? t.gx[side] : t.gy[side];
        w.xs[s] = (w.bs[s] - gw[0] * w.xs[sa] - gw[1] * w.xs[sb]) * gw[2];
    });
    __syncthreads();
}

// The colours of one smoothing step on the staged iterate (colour c at
// distance <= d1 - c), then the bottom rows at <= d2.
template <typename T, bool THREE, int S>
__device__ __forceinline__ void cross_smooth(const LevelDev<T>& F, const RowTab<T>& t, const TileGeo& g, const Reg& r,
                                             const CrossTile<T>& w, int d1, int d2) {
    const int nc = F.ncolor;
    const bool wall = at_wall(F.Nxg, F.Nyg, 0, r, THREE);
    if (wall) cross_ghosts<T, THREE>(F, t, r, g, w, nc, -1, 0);
    for (int c = 0; c < nc; ++c) {
        cross_pass<T, THREE, S, false>(F, t, g, r, w, nc, c, d1 - c);
        __syncthreads();
        if (wall) cross_ghosts<T, THREE>(F, t, r, g, w, nc, c, c + 1);
    }
    cross_bottoms<T, THREE, false>(F, t, g, r, w, d2);
}

template <typename T>
__device__ __forceinline__ CrossTile<T> cross_arrays(const TileGeo& g, T* sm) {
    const int cols = 2 * g.HW * g.PH;
    return CrossTile<T>{sm, sm + 4 * cols, sm + (4 + g.NZP) * cols};
}
template <bool THREE, typename T>
__device__ __forceinline__ void stage_cf(const LevelDev<T>& F, const TileGeo& g, const Reg& r, T* cf) {
    const float rw = recip(r.W);
    for (int q = threadIdx.x; q < r.W * r.H; q += blockDim.x) {
        const int lj = quot(q, rw), li = q - lj * r.W;
        T a, b, c, d;
        load_cf(F.cf, (int64_t)(r.ra + li - 1) + (int64_t)F.Nxg * (r.sa + lj - 1), a, b, c, d);
        T* const o = cf + 4 * ((lj * 2 + (li & 1)) * g.HW + (li >> 1));
        o[0] = a; o[1] = b; o[2] = THREE ? c : T(0); o[3] = d;
    }
}

template <typename T, bool THREE, int S>
__global__ void __launch_bounds__(kCrossThreads) k_mg_down_cross(LevelDev<T> F, LevelDev<T> Cc, const T* __restrict__ b,
                                                       const double* __restrict__ scale,
                                                                 T* __restrict__ xout, T* __restrict__ rc,
                                                                 T* __restrict__ zero,
                                                                 const __grid_constant__ RowTab<T> t, TileGeo g) {
    pdl_entry();
    extern __shared__ __align__(16) unsigned char tile_smem[];
    const CrossTile<T> w = cross_arrays(g, reinterpret_cast<T*>(tile_smem));
    const int nc = F.ncolor, bx = blockIdx.x, by = blockIdx.y;
    const Reg r = region(F.Nxg, F.Nyg, 0, g, bx, by, THREE);
    stage_cf<THREE>(F, g, r, w.cf);
    stage_down<THREE, false, false, false>(F, g, r, b, scale, w.xs, w.bs, (const T(*)[3])nullptr, (const T(*)[3])nullptr);
    __syncthreads();
    cross_bottoms<T, THREE, true>(F, t, g, r, w, g.halo);
    cross_smooth<T, THREE, S>(F, t, g, r, w, nc + 2, 2);
    write_core<THREE, false>(F, r, g, bx, w.xs, xout);
    cross_pass<T, THREE, S, true>(F, t, g, r, w, nc, 0, 1);
    __syncthreads();
    restrict_tile<THREE, false>(F, Cc, g, r, bx, w.bs, rc, zero);
}

template <typename T, bool THREE, int S>
__global__ void __launch_bounds__(kCrossThreads) k_mg_up_cross(LevelDev<T> F, LevelDev<T> Cc, const T* __restrict__ b,
                                                       const double* __restrict__ scale,
                                                               const T* __restrict__ xin, const T* __restrict__ xc,
                                                               T* __restrict__ out,
                                                               const __grid_constant__ RowTab<T> t, TileGeo g) {
    pdl_entry();
    extern __shared__ __align__(16) unsigned char tile_smem[];
    const CrossTile<T> w = cross_arrays(g, reinterpret_cast<T*>(tile_smem));
    const int nc = F.ncolor, bx = blockIdx.x, by = blockIdx.y;
    const Reg r = region(F.Nxg, F.Nyg, 0, g, bx, by, THREE);
    stage_cf<THREE>(F, g, r, w.cf);
    stage_up<THREE, false, false>(F, Cc, g, r, b, scale, xin, xc, w.xs, w.bs);
    __syncthreads();
    cross_bottoms<T, THREE, false>(F, t, g, r, w, nc + 1);
    cross_smooth<T, THREE, S>(F, t, g, r, w, nc, 0);
    write_core<THREE, false>(F, r, g, bx, w.xs, out);
}

// ------------------------------------------- cross levels in FP32 (ordered)
//
// In FP32 another order of the sums moves the steep basins' results by up to
// 1e-8 (see tile_level in ow3d.cu), so these levels keep every sum of the
// per-phase kernels (mg_device.cuh) in its order: the bottom rows, residual and
// restriction are the same functions on the staged tile (the level's
// description with its vectors' base and pitch replaced by the tile's), the
// colour tasks the same operations with the difference's weights at hand. The
// results are the per-phase kernels' bit for bit. TWO: the form of
// the column task that levels above the fused coarse kernel's size take there
// (two rows per lane), else one row per lane.
using LevelF = LevelDev<float>;

// The tile's level: F with vectors xs and bs of the region.
__device__ __forceinline__ void tile_view(LevelF& L, const LevelF& F, const TileGeo& g, const Reg& r, float* xs,
                                          float* bs) {
    if (threadIdx.x == 0) {
        L = F;
        L.pitch = 2 * g.HW;
        const int64_t o = (int64_t)F.Nzg * ((r.ra - 1) + (int64_t)L.pitch * (r.sa - 1));
        L.xv = xs - o;
        L.bv = bs - o;
        L.rv = bs - o;
    }
}

// Every point of the columns ilo..ihi x jlo..jhi of the region: f(place in the
// staged vectors, place in the level's vectors, k, i, j), all 1-based.
template <typename F_>
__device__ __forceinline__ void box_points(const LevelF& F, const TileGeo& g, const Reg& r, int ilo, int ihi, int jlo,
                                           int jhi, F_ f) {
    const int Nzg = F.Nzg, len = (ihi - ilo + 1) * Nzg;
    for (int j = jlo + threadIdx.x / 32; j <= jhi; j += blockDim.x / 32) {
        const int s0 = (2 * g.HW * (j - r.sa) + ilo - r.ra) * Nzg, p0 = Nzg * ((ilo - 1) + F.Nxg * (j - 1));
#pragma unroll 2
        for (int e = threadIdx.x % 32; e < len; e += 32) {
            const int c = (int)div32((uint32_t)e, F.mz32, F.sz32);
            f(s0 + e, p0 + e, e - c * Nzg + 1, ilo + c, j);
        }
    }
}

// The mixed-derivative sums of a row, in the per-phase kernels' order: over
// three planes (x: y planes, y: x planes) and three levels the three columns of
// the centred difference (w; its centre weight is zero up to rounding, and
// where it is exactly zero, cw false, its terms change nothing and are left
// out). p: the row in the column's staged values; oa, ob: offsets along the
// difference and across the planes. sh: in row 2 next to a wall, the shift of
// the level below the bottom's stencil off the ghost column (weights e). JOIN:
// the own column's terms go to lo, dg, up, times f = 2 s2 or 2 s4 (top: row
// Nzg-1, whose upper one does not), else into the sum like the others.
template <bool PLANES, bool JOIN>
__device__ __forceinline__ float mixed_sum(const float* w, const float* e, int sh, bool cw, bool top, const float* p,
                                           float z0, float z1, float z2, int oa, int ob, float f, float& lo, float& dg,
                                           float& up) {
    float xz = 0;
#pragma unroll
    for (int b = PLANES ? -1 : 0; b <= (PLANES ? 1 : 0); ++b)
#pragma unroll
        for (int kk = 0; kk < 3; ++kk) {
            const float* const q = p + b * ob + kk - 1;
            const float z = kk == 0 ? z0 : (kk == 1 ? z1 : z2);
            float dx;
            if (kk == 0 && sh != 0) {
                dx = 0;
#pragma unroll
                for (int m = 0; m < 3; ++m) {
                    const int a = sh - 1 + m;
                    if (JOIN && a == 0 && b == 0) lo = __fmaf_rn(__fmul_rn(f, z), e[m], lo);
                    else dx = __fmaf_rn(e[m], q[a * oa], dx);
                }
            } else {
                dx = __fmul_rn(w[0], q[-oa]);
                if (cw) {
                    if (JOIN && b == 0 && !(kk == 2 && top)) {
                        float& c = kk == 0 ? lo : (kk == 1 ? dg : up);
                        c = __fmaf_rn(__fmul_rn(f, z), w[1], c);
                    } else {
                        dx = __fmaf_rn(w[1], q[0], dx);
                    }
                }
                dx = __fmaf_rn(w[2], q[oa], dx);
            }
            xz = __fmaf_rn(z, dx, xz);
        }
    return xz;
}

// Row k of a column as the map x_k = q - g x_{k-1} (colour_col1 /
// colour_col2): x0, xp the old values of rows k, k + 1; shx, shy as above.
template <bool THREE>
__device__ __forceinline__ void ordered_row(const RowTab<float>& t, const RowConst<float>& rk, const float* p, float bk,
                                            float x0, float xp, float ih, float ca, float cb, float c3, int ox, int oy,
                                            int shx, int shy, bool top, float& qo, float& go) {
    const float xl = p[-ox], xr = p[ox];
    const float xd = THREE ? p[-oy] : 0.0f, xu = THREE ? p[oy] : 0.0f;
    const float om = rk.om;
    const float s2 = om * ca, s4 = THREE ? om * cb : 0.0f;
    const float s3 = om * c3;
    const float cz = s2 * s2 + s4 * s4 + ih * ih;
    float off = t.sx2[0] * xl + t.sx2[2] * xr;
    float diag = t.sx2[1] + s3 * rk.z1 + cz * rk.zz1;
    if (THREE) { off += t.sy2[0] * xd + t.sy2[2] * xu; diag += t.sy2[1]; }
    float lo = s3 * rk.z0 + cz * rk.zz0;
    float up = s3 * rk.z2 + cz * rk.zz2;
    if (s2 != 0.0f) {
        const float f = 2.0f * s2;
        off = __fmaf_rn(f, mixed_sum<THREE, true>(t.sx1, t.ex[shx < 0], shx, t.sx1[1] != 0.0f, top, p, rk.z0, rk.z1,
                                                  rk.z2, ox, oy, f, lo, diag, up), off);
    }
    if (THREE && s4 != 0.0f) {
        const float f = 2.0f * s4;
        off = __fmaf_rn(f, mixed_sum<true, true>(t.sy1, t.ey[shy < 0], shy, t.sy1[1] != 0.0f, top, p, rk.z0, rk.z1, rk.z2,
                                                 oy, ox, f, lo, diag, up), off);
    }
    const float id = 1.0f / diag;
    qo = x0 + (bk - diag * x0 - up * xp - off) * id;
    go = lo * id;
}

// A x at row k (2..Nzg-1) of an interior column (lo_interior).
template <bool THREE>
__device__ __forceinline__ float ordered_interior(const LevelF& L, const RowTab<float>& t, const float* p, int k, int i,
                                                  int j, int ox, int oy) {
    float ih, ca, cb, c3;
    load_cf(L.cf, (int64_t)(i - 1) + (int64_t)L.Nxg * (j - 1), ih, ca, cb, c3);
    const float om = 1.0f - __ldg(L.zs + k - 1);
    const float s2 = om * ca, s4 = THREE ? om * cb : 0.0f;
    const float s3 = om * c3;
    const float cz = s2 * s2 + s4 * s4 + ih * ih;
    float acc = 0;
#pragma unroll
    for (int m = 0; m < 3; ++m) acc = __fmaf_rn(t.sx2[m], p[(m - 1) * ox], acc);
    if (THREE) {
#pragma unroll
        for (int m = 0; m < 3; ++m) acc = __fmaf_rn(t.sy2[m], p[(m - 1) * oy], acc);
    }
    const float z[3] = {t.z0[k - 1], t.z1[k - 1], t.z2[k - 1]}, y[3] = {t.y0[k - 1], t.y1[k - 1], t.y2[k - 1]};
    float dz = 0, dzz = 0;
#pragma unroll
    for (int m = 0; m < 3; ++m) {
        const float v = p[m - 1];
        dz = __fmaf_rn(z[m], v, dz);
        dzz = __fmaf_rn(y[m], v, dzz);
    }
    acc += s3 * dz + cz * dzz;
    const int shx = k != 2 ? 0 : (i == 2 ? 1 : (i == L.Nxg - 1 ? -1 : 0));
    const int shy = !THREE || k != 2 ? 0 : (j == 2 ? 1 : (j == L.Nyg - 1 ? -1 : 0));
    float none;
    if (s2 != 0.0f)
        acc = __fmaf_rn(2.0f * s2, mixed_sum<THREE, false>(t.sx1, t.ex[shx < 0], shx, t.sx1[1] != 0.0f, false, p, z[0],
                                                           z[1], z[2], ox, oy, 0.0f, none, none, none), acc);
    if (THREE && s4 != 0.0f)
        acc = __fmaf_rn(2.0f * s4, mixed_sum<true, false>(t.sy1, t.ey[shy < 0], shy, t.sy1[1] != 0.0f, false, p, z[0],
                                                          z[1], z[2], oy, ox, 0.0f, none, none, none), acc);
    return acc;
}

// The colour task of column (i, j) (act), S lanes each: colour_col2 (TWO) or
// colour_col1 on the staged tile.
template <bool THREE, int S, bool TWO>
__device__ __forceinline__ void ordered_task(const LevelF& L, const RowTab<float>& t, int i, int j, bool act,
                                             const RowConst<float>& ra, const RowConst<float>& rb) {
    const int Nxg = L.Nxg, Nyg = L.Nyg, Nzg = L.Nzg, R = Nzg - 2, lane = threadIdx.x & 31, r = lane & (S - 1);
    const int ox = Nzg, oy = Nzg * L.pitch;
    float* const X = L.xv;
    const float* const B = L.bv;
    float* const xc = X + IC(L, i, j) * Nzg;
    const float* const bc = B + IC(L, i, j) * Nzg;
    const int ka = TWO ? 2 + 2 * r : min(r + 2, Nzg - 1), kb = ka + 1;
    const bool va = act && (TWO ? ka <= Nzg - 1 : r < R), vb = TWO && act && kb <= Nzg - 1;
    const int last = TWO ? (R - 1) / 2 : R - 1;
    const bool edge = act && (i <= 3 || i >= Nxg - 2 || (THREE && (j <= 3 || j >= Nyg - 2)));
    // ghost column at offset og from the column, the two columns of its stencil
    // at oa (weight wa) and ob (wb); own: which of them is this column (its new
    // values are xna, xnb, xfs once post is set)
    auto relax = [&](int og, int oa, float wa, int ob, float wb, float wg, int own, bool post, float xna, float xnb,
                     float xfsn) {
        auto row = [&](int kk, float xo) {
            const float v1 = (post && own == 1) ? xo : xc[oa + kk - 1];
            const float v2 = (post && own == 2) ? xo : xc[ob + kk - 1];
            xc[og + kk - 1] = (bc[og + kk - 1] - (wa * v1 + wb * v2)) / wg;
        };
        if (TWO) {
            if (ka <= Nzg - 1) row(ka, xna);
            if (kb <= Nzg - 1) row(kb, xnb);
        } else if (r < R) {
            row(r + 2, xna);
        }
        if (r == last) row(Nzg, xfsn);
    };
    auto ghosts = [&](bool post, float xna, float xnb, float xfsn) {
        // low walls: stencil of position 2, columns 1 (ghost), 2, 3; high walls
        // of position n - 1, columns n - 2, n - 1, n (ghost)
        if (i == 2 || (post && i == 3))
            relax((1 - i) * ox, (2 - i) * ox, t.sx1[1], (3 - i) * ox, t.sx1[2], t.sx1[0], i == 2 ? 1 : 2, post, xna, xnb,
                  xfsn);
        if (i == Nxg - 1 || (post && i == Nxg - 2))
            relax((Nxg - i) * ox, (Nxg - 2 - i) * ox, t.sx1[0], (Nxg - 1 - i) * ox, t.sx1[1], t.sx1[2],
                  i == Nxg - 1 ? 2 : 1, post, xna, xnb, xfsn);
        if (THREE) {
            if (j == 2 || (post && j == 3))
                relax((1 - j) * oy, (2 - j) * oy, t.sy1[1], (3 - j) * oy, t.sy1[2], t.sy1[0], j == 2 ? 1 : 2, post, xna,
                      xnb, xfsn);
            if (j == Nyg - 1 || (post && j == Nyg - 2))
                relax((Nyg - j) * oy, (Nyg - 2 - j) * oy, t.sy1[0], (Nyg - 1 - j) * oy, t.sy1[1], t.sy1[2],
                      j == Nyg - 1 ? 2 : 1, post, xna, xnb, xfsn);
        }
    };
    if (edge) {
        // (corner columns hold b from the staging)
        ghosts(false, 0.0f, 0.0f, 0.0f);
    }
    __syncwarp();
    float qa = 0, ga = 0, qb = 0, gb = 0, x1 = 0;
    if (act) {
        float ih, ca, cb, c3;
        load_cf(L.cf, (int64_t)(i - 1) + (int64_t)Nxg * (j - 1), ih, ca, cb, c3);
        const int kra = min(ka, Nzg - 1), krb = min(kb, Nzg - 1);
        const int shx = kra != 2 ? 0 : (i == 2 ? 1 : (i == Nxg - 1 ? -1 : 0));
        const int shy = !THREE || kra != 2 ? 0 : (j == 2 ? 1 : (j == Nyg - 1 ? -1 : 0));
        const float x0a = xc[kra - 1], xpa = xc[kra], xpb = xc[krb];
        ordered_row<THREE>(t, ra, xc + kra - 1, bc[kra - 1], x0a, xpa, ih, ca, cb, c3, ox, oy, shx, shy,
                           kra == Nzg - 1, qa, ga);
        if (TWO)
            ordered_row<THREE>(t, rb, xc + krb - 1, bc[krb - 1], xpa, xpb, ih, ca, cb, c3, ox, oy, 0, 0, krb == Nzg - 1,
                               qb, gb);
        if (!va) { qa = 0; ga = 0; }
        if (!vb) { qb = 0; gb = 0; }
        x1 = xc[0];
    }
    float xna, xnb = 0;
    if constexpr (TWO) {
        float a = 1, bb = 0;
        if (va) { bb = qa; a = -ga; }
        if (vb) { bb = qb - gb * bb; a = -gb * a; }
#pragma unroll
        for (int d = 1; d < S; d <<= 1) {
            const float ap = __shfl_up_sync(0xffffffffu, a, d, S);
            const float bp = __shfl_up_sync(0xffffffffu, bb, d, S);
            if (r >= d) { bb = a * bp + bb; a = a * ap; }
        }
        const float ae = __shfl_up_sync(0xffffffffu, a, 1, S), be = __shfl_up_sync(0xffffffffu, bb, 1, S);
        const float xin = (r == 0) ? x1 : ae * x1 + be;
        xna = qa - ga * xin;
        xnb = qb - gb * xna;
    } else {
        float a = -ga, bb = qa;
#pragma unroll
        for (int d = 1; d < S; d <<= 1) {
            const float ap = __shfl_up_sync(0xffffffffu, a, d, S);
            const float bp = __shfl_up_sync(0xffffffffu, bb, d, S);
            if (r >= d) { bb = a * bp + bb; a = a * ap; }
        }
        xna = a * x1 + bb;
    }
    const float xfs = act ? bc[Nzg - 1] : 0.0f;
    __syncwarp();
    if (va) xc[ka - 1] = xna;
    if (vb) xc[kb - 1] = xnb;
    if (act && r == last) xc[Nzg - 1] = xfs;
    if (edge) ghosts(true, xna, xnb, xfs);
}

template <bool THREE>
__device__ __forceinline__ void ordered_bottoms(const LevelF& L, const Reg& r, int d) {
    all_columns<THREE>(L.Nxg, L.Nyg, 0, r, d, [&](int i, int j) { bottom_column<float, THREE>(L, i, j); });
    __syncthreads();
}

// The colour tasks at distance <= d, one column per segment of S lanes.
template <bool THREE, int S, bool TWO>
__device__ __forceinline__ void ordered_colour(const LevelF& L, const RowTab<float>& t, const Reg& r, int colour, int d) {
    const int Nxg = L.Nxg, Nyg = L.Nyg, Nzg = L.Nzg;
    const int ilo = max(r.ia - d, 2), ihi = min(r.ib + d, Nxg - 1);
    int jlo = 1, jhi = 1, js = 1;
    if (THREE) { jlo = max(r.ja - d, 2); jhi = min(r.jb + d, Nyg - 1); }
    const bool four = L.ncolor == 4;
    if (THREE && four) { jlo += (jlo ^ (colour >> 1)) & 1; js = 2; }
    const int ni = max((ihi - ilo + 2) >> 1, 0), nj = jhi >= jlo ? (jhi - jlo) / js + 1 : 0, total = ni * nj;
    const int lane = threadIdx.x & 31, rr = lane & (S - 1);
    const int per_warp = 32 / S, step = (blockDim.x >> 5) * per_warp;
    const RowConst<float> ra = TWO ? row_const_k<float>(L, 2 + 2 * rr) : row_const<float, S>(L);
    const RowConst<float> rb = TWO ? row_const_k<float>(L, 3 + 2 * rr) : ra;
    const float rni = recip(ni);
    for (int base = (threadIdx.x >> 5) * per_warp; base < total; base += step) {
        const int q = base + lane / S;
        int i = 2, j = THREE ? 2 : 1;
        bool act = q < total;
        if (act) {
            const int tj = quot(q, rni);
            j = jlo + tj * js;
            const int par = four ? colour & 1 : (colour + j) & 1;
            i = ilo + ((ilo ^ par) & 1) + 2 * (q - tj * ni);
            act = i <= ihi;
        }
        ordered_task<THREE, S, TWO>(L, t, i, j, act, ra, rb);
    }
    __syncthreads();
}

template <bool THREE, int S, bool TWO>
__global__ void __launch_bounds__(kOrderedThreads) k_mg_down_ordered(LevelF F, LevelF Cc, const float* __restrict__ b,
                                                                     float* __restrict__ xout, float* __restrict__ rc,
                                                                     const __grid_constant__ RowTab<float> t,
                                                                     TileGeo g) {
    pdl_entry();
    extern __shared__ __align__(16) unsigned char tile_smem[];
    __shared__ LevelF L;
    float* const xs = reinterpret_cast<float*>(tile_smem);
    float* const bs = xs + 2 * g.HW * g.PH * F.Nzg;
    const int Nxg = F.Nxg, Nyg = F.Nyg, nc = F.ncolor;
    const Reg r = region(Nxg, Nyg, 0, g, blockIdx.x, blockIdx.y, THREE);
    tile_view(L, F, g, r, xs, bs);
    // x = 0; the bottom pass over it sets the ghost columns' level 1 (the
    // corner columns, which only the column diagonal to them reads, after it
    // has set them, may hold b already)
    stage_down<THREE, true, false, true>(F, g, r, b, (const double*)nullptr, xs, bs, (const float(*)[3])nullptr,
                                         (const float(*)[3])nullptr);
    __syncthreads();
    ordered_bottoms<THREE>(L, r, nc + 3);
    for (int c = 0; c < nc; ++c) ordered_colour<THREE, S, TWO>(L, t, r, c, nc + 2 - c);
    ordered_bottoms<THREE>(L, r, 2);
    // the iterate of the core, and at distance <= 1 the residual where the
    // right-hand side was
    box_points(F, g, r, max(r.ia - 1, 1), min(r.ib + 1, Nxg), THREE ? max(r.ja - 1, 1) : 1,
               THREE ? min(r.jb + 1, Nyg) : 1, [&](int s, int p, int k, int i, int j) {
        if (i >= r.ia && i <= r.ib && j >= r.ja && j <= r.jb) xout[p] = xs[s];
        float v, dg;
        if (i == 1 || i == Nxg || (THREE && (j == 1 || j == Nyg))) v = lo_ghost<float, THREE>(L, L.xv, k, i, j, dg);
        else if (k == F.Nzg) v = xs[s];
        else if (k == 1) v = lo_bottom<float, THREE>(L, L.xv, i, j, dg);
        else v = ordered_interior<THREE>(F, t, xs + s, k, i, j, F.Nzg, F.Nzg * 2 * g.HW);
        bs[s] = bs[s] - v;
    });
    __syncthreads();
    int clo, chi, dlo = 1, dhi = 1;
    owned(r.ia, r.ib, Nxg, Cc.Nxg, 1 + Cc.xc, 0, clo, chi);
    if (THREE) owned(r.ja, r.jb, Nyg, Cc.Nyg, 1 + Cc.yc, 0, dlo, dhi);
    const int Ncz = Cc.Nzg, len = (chi - clo + 1) * Ncz;
    const float rlen = recip(len);
    for (int e = threadIdx.x; e < len * (dhi - dlo + 1); e += blockDim.x) {
        const int q = quot(e, rlen);
        restrict_item<float>(L, Cc, L.rv, rc, Cc.xv,
                              (e - q * len) + Ncz * ((clo - 1) + (int64_t)Cc.Nxg * (dlo + q - 1)));
    }
}

template <bool THREE, int S, bool TWO>
__global__ void __launch_bounds__(kOrderedThreads) k_mg_up_ordered(LevelF F, LevelF Cc, const float* __restrict__ b,
                                                                   const float* __restrict__ xin,
                                                                   const float* __restrict__ xc,
                                                                   float* __restrict__ out,
                                                                   const __grid_constant__ RowTab<float> t, TileGeo g) {
    pdl_entry();
    extern __shared__ __align__(16) unsigned char tile_smem[];
    __shared__ LevelF L;
    float* const xs = reinterpret_cast<float*>(tile_smem);
    float* const bs = xs + 2 * g.HW * g.PH * F.Nzg;
    const int nc = F.ncolor;
    const Reg r = region(F.Nxg, F.Nyg, 0, g, blockIdx.x, blockIdx.y, THREE);
    tile_view(L, F, g, r, xs, bs);
    stage_up<THREE, true, true>(F, Cc, g, r, b, (const double*)nullptr, xin, xc, xs, bs);
    __syncthreads();
    ordered_bottoms<THREE>(L, r, nc + 1);
    for (int c = 0; c < nc; ++c) ordered_colour<THREE, S, TWO>(L, t, r, c, nc - c);
    ordered_bottoms<THREE>(L, r, 0);
    box_points(F, g, r, r.ia, r.ib, r.ja, r.jb, [&](int s, int p, int, int, int) { out[p] = xs[s]; });
}

// ------------------------------------------------------------ host side

// Column pitch in shared memory. Cross levels, whose lanes take rows of a
// column one by one: odd. Uniform levels, two rows at a time: twice an odd
// number.
inline int tile_pitch(int nzg, bool cross) { return cross ? nzg | 1 : ((nzg + 1) / 2 | 1) * 2; }

// Whether the per-phase kernels take the level's columns with two rows per lane
// (the levels above the fused coarse kernel's size).
template <typename T>
bool two_rows(const LevelDev<T>& L) { return L.N > g_coop_max_points.load(std::memory_order_relaxed); }

// Cores, slots and shared memory of a launch over all its tiles.
template <typename T>
void size_geo(const LevelDev<T>& L, TileGeo& g, int cx, int cy, bool cross, bool down) {
    const bool three = L.Nyg > 1;
    auto cores = [](int n, int c, int& nt, int& q, int& rem, int& most) {
        nt = (n + c - 1) / c;
        if (n / nt < 3) nt = n / 3;      // n >= 4: of a periodic level the distinct columns (tile_level)
        q = n / nt;
        rem = n - q * nt;
        most = q + (rem > 0 ? 1 : 0);
    };
    cores(L.per ? L.Nxg - 3 : L.Nxg, cx, g.ntx, g.qx, g.remx, g.cx);
    if (three) cores(L.Nyg, cy, g.nty, g.qy, g.remy, g.cy);
    else { g.nty = 1; g.qy = 1; g.remy = 0; g.cy = 1; }
    const bool ordered = cross && sizeof(T) == 4;
    g.NZP = ordered ? L.Nzg : tile_pitch(L.Nzg, cross);
    g.np = (L.Nzg + 1) / 2;
    int W = 0, H = 0;
    for (int bx = 0; bx < g.ntx; ++bx) W = std::max(W, region(L.Nxg, L.Nyg, L.per, g, bx, 0, three).W);
    for (int by = 0; by < g.nty; ++by) H = std::max(H, region(L.Nxg, L.Nyg, L.per, g, 0, by, three).H);
    g.HW = (W + 1) / 2;
    g.PH = H;
    const size_t cols = (size_t)2 * g.HW * g.PH;
    // iterate, right-hand side (uniform levels on the way down: in one place), coefficients
    g.smem = (cols * g.NZP * (cross || !down ? 2 : 1) + (cross && !ordered ? 4 * cols : 0)) * sizeof(T);
}

}  // namespace

template <typename T>
void tile_geometry(const LevelDev<T>& L, TileLevel<T>& t) {
    const bool three = L.Nyg > 1, cross = t.mode == kTileCross;
    // Of the cores that leave shared memory for two blocks per SM (the smallest
    // core: for one), the one of least waves x (columns of a tile with its halo
    // + 200): a tile's time is its columns' share of the staging and the phases
    // plus the phases' latency, worth some 200 columns. Levels of few tiles so
    // take smaller cores, and large ones the largest that fits (way up at
    // 1025x257x17 FP64: 16x8 80 us, 24x8 70 us; one level below, 561 tiles of
    // 16x8 21 us, 374 of 24x8 23 us). Uniform levels run two blocks per SM, as
    // the waves are counted (FP64 96 to 128 registers at 256 or 320 threads).
    // The 3-D sloping forms do not: at 98 to 128 registers a block of 384
    // threads or more is alone on its SM, so 165 tiles (257x33x9 FP64, finest
    // level) are a second wave of 17 tiles, 27 and 23 us a launch against 17
    // and 15 us for the 51 tiles of the level below. In FP64 the smallest core,
    // 8x8 with its halo of 7, fits up to 22 sigma levels on a wide level;
    // taller ones take the per-phase kernels.
    static const int uni3[][2] = {{32, 8}, {24, 8}, {16, 8}, {8, 4}}, cross3[][2] = {{16, 16}, {16, 8}, {8, 8}};
    static const int line[][2] = {{64, 1}, {32, 1}, {16, 1}};
    const int (*cand)[2] = three ? (cross ? cross3 : uni3) : line;
    const int ncand = three && !cross ? 4 : 3;
    auto pick = [&](TileGeo& g, int halo, bool down) {
        g.halo = halo;
        bool found = false;
        int64_t least = 0;
        TileGeo best{};
        for (int q = 0; q < ncand; ++q) {
            size_geo(L, g, cand[q][0], cand[q][1], cross, down);
            if (g.nty > kTileMaxRows) continue;
            if (g.smem > kTileSmemMax || (g.smem > kTileSmemTwo && (found || q + 1 < ncand))) continue;
            int lanes = cross ? (L.Nzg <= 10 ? 4 : (L.Nzg <= 18 ? 8 : 16)) : 1;
            if (cross && sizeof(T) == 4 && !two_rows(L)) lanes *= 2;
            const int cols = (g.cx + 2 * halo) * (three ? g.cy + 2 * halo : 1) / L.ncolor * lanes;
            const int most = cross ? kCrossThreads : (down ? kUniThreads : 256);
            g.threads = std::min(most, std::max(256, (cols + 31) / 32 * 32));
            const int64_t waves = (g.ntx * g.nty + 2 * 148 - 1) / (2 * 148), cost = waves * (2 * g.HW * g.PH + 200);
            if (found && cost >= least) continue;
            found = true;
            least = cost;
            best = g;
        }
        g = best;
        return found;
    };
    if (t.mode == kTileNone) return;
    // (the ordered form's first bottom pass reads one column further)
    const int nc = L.ncolor, extra = sizeof(T) == 4 ? 1 : 0;
    if (!pick(t.down, cross ? nc + 3 + extra : 3, true) || !pick(t.up, cross ? nc + 2 : 2, false)) t.mode = kTileNone;
}

namespace {
template <typename K>
void allow_smem(K kernel, std::atomic<unsigned long long>& set) {
    int dev = 0;
    cudaGetDevice(&dev);
    const unsigned long long bit = 1ull << (dev & 63);
    if (!(set.load(std::memory_order_relaxed) & bit)) {
        cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kTileSmemMax);
        set.fetch_or(bit, std::memory_order_relaxed);
    }
}

template <typename T, typename TB, bool THREE, int NZG>
void down_uni(const LevelDev<T>& F, const LevelDev<T>& Cc, const TileLevel<T>& t, Rhs<TB> b, T* xs, T* rc, T* zero,
              cudaStream_t st) {
    static std::atomic<unsigned long long> set{0ull};
    const TileGeo& g = t.down;
    allow_smem(k_mg_down_uni<T, TB, THREE, NZG>, set);
    launch_k(k_mg_down_uni<T, TB, THREE, NZG>, dim3((unsigned)g.ntx, (unsigned)g.nty), dim3((unsigned)g.threads), g.smem,
             st, F, Cc, b.p, b.scale, xs, rc, zero, t.u, g);
}
template <typename T, typename TB, bool THREE, int NZG>
void up_uni(const LevelDev<T>& F, const LevelDev<T>& Cc, const TileLevel<T>& t, Rhs<TB> b, const T* xs, const T* xc,
            T* out, cudaStream_t st) {
    static std::atomic<unsigned long long> set{0ull};
    const TileGeo& g = t.up;
    allow_smem(k_mg_up_uni<T, TB, THREE, NZG>, set);
    launch_k(k_mg_up_uni<T, TB, THREE, NZG>, dim3((unsigned)g.ntx, (unsigned)g.nty), dim3((unsigned)g.threads), g.smem,
             st, F, Cc, b.p, b.scale, xs, xc, out, t.u, g);
}
template <typename T, typename TB, bool THREE, int S>
void down_cross(const LevelDev<T>& F, const LevelDev<T>& Cc, const TileLevel<T>& t, Rhs<TB> b, T* xs, T* rc, T* zero,
                cudaStream_t st) {
    static std::atomic<unsigned long long> set{0ull};
    const TileGeo& g = t.down;
    allow_smem(k_mg_down_cross<T, THREE, S>, set);
    launch_k(k_mg_down_cross<T, THREE, S>, dim3((unsigned)g.ntx, (unsigned)g.nty), dim3((unsigned)g.threads), g.smem, st,
             F, Cc, b.p, b.scale, xs, rc, zero, t.r, g);
}
template <typename T, typename TB, bool THREE, int S>
void up_cross(const LevelDev<T>& F, const LevelDev<T>& Cc, const TileLevel<T>& t, Rhs<TB> b, const T* xs, const T* xc,
              T* out, cudaStream_t st) {
    static std::atomic<unsigned long long> set{0ull};
    const TileGeo& g = t.up;
    allow_smem(k_mg_up_cross<T, THREE, S>, set);
    launch_k(k_mg_up_cross<T, THREE, S>, dim3((unsigned)g.ntx, (unsigned)g.nty), dim3((unsigned)g.threads), g.smem, st, F,
             Cc, b.p, b.scale, xs, xc, out, t.r, g);
}

template <bool THREE, int S, bool TWO>
void down_ordered(const LevelF& F, const LevelF& Cc, const TileLevel<float>& t, Rhs<float> b, float* xs, float* rc, float*,
                  cudaStream_t st) {
    static std::atomic<unsigned long long> set{0ull};
    const TileGeo& g = t.down;
    allow_smem(k_mg_down_ordered<THREE, S, TWO>, set);
    launch_k(k_mg_down_ordered<THREE, S, TWO>, dim3((unsigned)g.ntx, (unsigned)g.nty), dim3((unsigned)g.threads), g.smem,
             st, F, Cc, b.p, xs, rc, t.r, g);
}
template <bool THREE, int S, bool TWO>
void up_ordered(const LevelF& F, const LevelF& Cc, const TileLevel<float>& t, Rhs<float> b, const float* xs,
                const float* xc, float* out, cudaStream_t st) {
    static std::atomic<unsigned long long> set{0ull};
    const TileGeo& g = t.up;
    allow_smem(k_mg_up_ordered<THREE, S, TWO>, set);
    launch_k(k_mg_up_ordered<THREE, S, TWO>, dim3((unsigned)g.ntx, (unsigned)g.nty), dim3((unsigned)g.threads), g.smem, st,
             F, Cc, b.p, xs, xc, out, t.r, g);
}

// Uniform levels: the columns of 9 and, in 3-D, 17 sigma levels, the usual
// counts, unrolled, any other by the general form, which takes those two as
// well but slower: a V cycle at 1025x257x17 258 us unrolled against 347 (FP32
// 209, 294), at 1025x257x9 162 against 220, of a 513x9 flume 24 against 35; at
// 1025x257x13, by the general form, 280. (The unrolled FP64 way up of 17 levels
// spills 76 bytes a thread at the 128 registers of two blocks per SM.) Cross
// levels: the lanes per column (FP64, and FP32 with two rows per lane: two
// rows each; else one).
#define OW3D_TILE(way, ...)                                                     \
    do {                                                                        \
        if (t.mode == kTileUniform) {                                           \
            if (F.Nyg > 1) {                                                    \
                if (F.Nzg == 18) way##_uni<T, TB, true, 18>(__VA_ARGS__);       \
                else if (F.Nzg == 10) way##_uni<T, TB, true, 10>(__VA_ARGS__);  \
                else way##_uni<T, TB, true, 0>(__VA_ARGS__);                    \
            } else {                                                            \
                if (F.Nzg == 10) way##_uni<T, TB, false, 10>(__VA_ARGS__);      \
                else way##_uni<T, TB, false, 0>(__VA_ARGS__);                   \
            }                                                                   \
        } else if constexpr (sizeof(T) == 8) {                                  \
            if (F.Nyg > 1) {                                                    \
                if (F.Nzg <= 10) way##_cross<T, TB, true, 4>(__VA_ARGS__);      \
                else if (F.Nzg <= 18) way##_cross<T, TB, true, 8>(__VA_ARGS__); \
                else way##_cross<T, TB, true, 16>(__VA_ARGS__);                 \
            } else {                                                            \
                if (F.Nzg <= 10) way##_cross<T, TB, false, 4>(__VA_ARGS__);     \
                else if (F.Nzg <= 18) way##_cross<T, TB, false, 8>(__VA_ARGS__); \
                else way##_cross<T, TB, false, 16>(__VA_ARGS__);                \
            }                                                                   \
        } else if constexpr (sizeof(TB) == 4) {                                 \
            if (F.Nyg > 1 && two_rows(F)) {                                     \
                if (F.Nzg <= 10) way##_ordered<true, 4, true>(__VA_ARGS__);     \
                else if (F.Nzg <= 18) way##_ordered<true, 8, true>(__VA_ARGS__); \
                else way##_ordered<true, 16, true>(__VA_ARGS__);                \
            } else if (F.Nyg > 1) {                                             \
                if (F.Nzg <= 10) way##_ordered<true, 8, false>(__VA_ARGS__);    \
                else if (F.Nzg <= 18) way##_ordered<true, 16, false>(__VA_ARGS__); \
                else way##_ordered<true, 32, false>(__VA_ARGS__);               \
            } else if (two_rows(F)) {                                           \
                if (F.Nzg <= 10) way##_ordered<false, 4, true>(__VA_ARGS__);    \
                else if (F.Nzg <= 18) way##_ordered<false, 8, true>(__VA_ARGS__); \
                else way##_ordered<false, 16, true>(__VA_ARGS__);               \
            } else {                                                            \
                if (F.Nzg <= 10) way##_ordered<false, 8, false>(__VA_ARGS__);   \
                else if (F.Nzg <= 18) way##_ordered<false, 16, false>(__VA_ARGS__); \
                else way##_ordered<false, 32, false>(__VA_ARGS__);              \
            }                                                                   \
        }                                                                       \
    } while (0)

template <typename T, typename TB>
void down(const LevelDev<T>& F, const LevelDev<T>& Cc, const TileLevel<T>& t, Rhs<TB> b, T* xs, T* rc, T* zero,
          cudaStream_t st) {
    OW3D_TILE(down, F, Cc, t, b, xs, rc, zero, st);
}
template <typename T, typename TB>
void up(const LevelDev<T>& F, const LevelDev<T>& Cc, const TileLevel<T>& t, Rhs<TB> b, const T* xs, const T* xc, T* out,
        cudaStream_t st) {
    OW3D_TILE(up, F, Cc, t, b, xs, xc, out, st);
}
}  // namespace

template <typename T>
void launch_tile_down(const LevelDev<T>& F, const LevelDev<T>& Cc, const TileLevel<T>& t, const double* src,
                      const double* scale, T* xs, T* rc, T* zero, cudaStream_t st) {
    if (src) down<T, double>(F, Cc, t, Rhs<double>{src, scale}, xs, rc, zero, st);
    else down<T, T>(F, Cc, t, Rhs<T>{F.bv, nullptr}, xs, rc, zero, st);
}
template <typename T>
void launch_tile_up(const LevelDev<T>& F, const LevelDev<T>& Cc, const TileLevel<T>& t, const double* src,
                    const double* scale, const T* xs, const T* xc, T* out, cudaStream_t st) {
    if (src) up<T, double>(F, Cc, t, Rhs<double>{src, scale}, xs, xc, out, st);
    else up<T, T>(F, Cc, t, Rhs<T>{F.bv, nullptr}, xs, xc, out, st);
}

#define OW3D_INST(T)                                                                                              \
    template void tile_geometry<T>(const LevelDev<T>&, TileLevel<T>&);                                            \
    template void launch_tile_down<T>(const LevelDev<T>&, const LevelDev<T>&, const TileLevel<T>&, const double*, \
                                      const double*, T*, T*, T*, cudaStream_t);                                   \
    template void launch_tile_up<T>(const LevelDev<T>&, const LevelDev<T>&, const TileLevel<T>&, const double*,   \
                                    const double*, const T*, const T*, T*, cudaStream_t);
OW3D_INST(double)
OW3D_INST(float)
#undef OW3D_INST

}  // namespace ow3d
