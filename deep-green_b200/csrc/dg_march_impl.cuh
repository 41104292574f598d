// dg_march_impl.cuh -- the one-cell-per-lane step kernel: compute_step
// (deep-green src/rs/src/physics.rs:595-681) with the reference's rounding in
// FP64 and FP32 (RefArith; built with --fmad=false), and with fused
// arithmetic in FP64 (FusedArith).  The FP32 production step is the packed
// kernel of dg_sweep_impl.cuh.
//
// Decomposition.  A block owns TY rows (y) x 32 columns (z) and marches along
// x through a chunk of planes, one warp per row and one cell per lane, so
// that a 64-bit value takes the registers an FP32 pair takes in the packed
// kernel: 16 warps of 128 registers per SM instead of 6 of 255.  Each plane
// arrives by one 4-D TMA copy (36 columns x (TY + 4) rows x 5 fields) in a
// ring of R slots and is converted to primitives once, into a buffer of two
// planes; its conserved totals are read again from L2 when its cells are
// updated, which keeps the ring short enough for the tile.
//   * Owned warps (TY): row y0 + r, lane l the cell z0 + l.
//   * Halo warp A: the row below the tile, the halo columns left (lanes 0-15)
//     and right (lanes 16-31) of it, and the TMA copies.
//   * Halo warp B: the row above, the columns outside those (conversion
//     only), the face above the tile's top row and the faces on its right
//     edge.
// All warps run one loop body (run_warp).  One barrier per plane.  Iteration
// j, before it: convert plane j + 1; slopes and prediction of plane j; the x
// face between planes j - 1 and j; publish face states.  After it: update
// plane j - 1, whose six fluxes are now known, in the reference's summation
// order; the y and z faces of plane j.
//
// What bounds it: the FP64 pipe (2 warp instructions per clock and SM) and,
// in FP32 with the reference's rounding, issue; the divisions cost most.  The
// reference divides about 70 times per cell, by few divisors: ds or 2 ds
// (slopes), the cell volume, gamma - 1, and per face the star density five
// times.  Quotients with a shared divisor take one correctly rounded
// reciprocal and three operations each (div_shared), bit for bit the IEEE
// quotient.
//
// Ghost-layer rules of the derived arrays: as listed in dg_sweep_impl.cuh.
#pragma once
#include "dg_common.cuh"
#include "dg_host.h"
#include "dg_sweep_impl.cuh"

namespace dg {
namespace march {

constexpr int kTileZ = 32;            // tile columns: one cell per lane
constexpr int kBoxZ = kTileZ + 4;     // staged columns

// ---------------------------------------------------------------------------
// Correctly rounded quotients with a shared divisor.  y = RN(1/b);
// q0 = RN(a y), the residual b q0 - a is exact in one fused multiply-add, and
// RN(q0 - residual y) is RN(a/b) as long as nothing over- or underflows
// (Markstein 1990; Brisebarre, Muller & Raina, IEEE Trans. Computers 53(8),
// 2004, for a divisor known in advance).  The residual's sign is chosen so
// that a signed zero keeps its sign for b > 0.  Operands outside the ranges
// below (zero numerators are inside) take the plain division instead.
// ---------------------------------------------------------------------------
template <class T> __device__ __forceinline__ T div_shared(T a, T b, T y) {
    const T q0 = a * y;
    const T nr = fma(b, q0, -a);
    return fma(-nr, y, q0);
}

// Exponent-ordered magnitude of a numerator: an unsigned key that compares
// like |a| and is zero only for a zero.
__device__ __forceinline__ unsigned mag_key(float a) { return __float_as_uint(a) & 0x7fffffffu; }
__device__ __forceinline__ unsigned mag_key(double a) {
    const unsigned hi = (unsigned)__double2hiint(a) & 0x7fffffffu;
    return hi | (__double2loint(a) != 0 ? 1u : 0u);
}
// Bounds of the safe ranges.  FP32: numerators 0 or 2^-75 .. 2^60, divisors
// 2^-40 .. 2^20: quotients stay within 2^-95 .. 2^100 and residuals are
// multiples of 2^-122.  FP64: numerators 0 or 2^-400 .. 2^400, divisors
// 2^-300 .. 2^300.
template <class T> struct SafeRange;
template <> struct SafeRange<float> {
    static constexpr unsigned nlo = (127u - 75u) << 23, nhi = (127u + 60u) << 23;
    static constexpr unsigned dlo = (127u - 40u) << 23, dhi = (127u + 20u) << 23;
};
template <> struct SafeRange<double> {
    static constexpr unsigned nlo = (1023u - 400u) << 20, nhi = (1023u + 400u) << 20;
    static constexpr unsigned dlo = (1023u - 300u) << 20, dhi = (1023u + 300u) << 20;
};
template <class T> __device__ __forceinline__ bool safe_divisor(T b) {
    const unsigned h = mag_key(b);
    return b > T(0) && h >= SafeRange<T>::dlo && h <= SafeRange<T>::dhi;
}
// Running bounds over the numerators of one group: zeros wrap to the top of
// `lo`'s order and are ignored by it.
struct KeyBounds {
    unsigned lo = 0xffffffffu, hi = 0;
    template <class T> __device__ __forceinline__ void add(T a) {
        const unsigned h = mag_key(a);
        lo = min(lo, h - 1u);
        hi = max(hi, h);
    }
    template <class T> __device__ __forceinline__ bool safe() const {
        return lo >= SafeRange<T>::nlo - 1u && hi <= SafeRange<T>::nhi;
    }
};

// The plain division of the rare paths, out of line: inlined, the dozens of
// IEEE divisions behind the range tests made the march's code several times
// larger than what runs, and its instruction fetches the leading stall.
__device__ __noinline__ float plain_div(float a, float b) { return a / b; }
__device__ __noinline__ double plain_div(double a, double b) { return a / b; }

__device__ __forceinline__ float rcp_rn(float x) { return __frcp_rn(x); }
__device__ __forceinline__ double rcp_rn(double x) { return __drcp_rn(x); }

// ---------------------------------------------------------------------------
// Reference rounding: the reference's expressions (physics.rs; each function
// cites the lines it follows), operation for operation.  Face states are
// xt + hs / xt - hs with hs = slope * ds / 2.
// ---------------------------------------------------------------------------
template <class T> struct RefArith {
    using Ph = Phys<T, true>;
    struct K {
        T dt, dtds;
        bool safe;   // ds, 2 ds, the volume and gamma - 1 are safe divisors
    };
    static __device__ __forceinline__ K make(const GridArgs<T> &a, T dt) {
        K k;
        k.dt = dt;
        k.dtds = dt * a.k.ds;
        k.safe = safe_divisor(a.k.ds) && safe_divisor(a.k.two_ds) && safe_divisor(a.k.vol) && safe_divisor(a.k.gm1);
        return k;
    }
    // calc_primitives, physics.rs:112-140
    static __device__ __forceinline__ void prim(const T u[5], T w[5], const GridArgs<T> &a, const K &k) {
        const Consts<T> &c = a.k;
        KeyBounds kb;
#pragma unroll
        for (int f = 0; f < 5; ++f) kb.add(u[f]);
        const T r = div_shared(u[0], c.vol, c.inv_vol);
        const T rv = r * c.vol;
        if (k.safe && kb.safe<T>() && safe_divisor(rv)) {
            const T y = rcp_rn(rv);
            const T vx = div_shared(u[1], rv, y), vy = div_shared(u[2], rv, y), vz = div_shared(u[3], rv, y);
            w[0] = r;
            w[1] = vx;
            w[2] = vy;
            w[3] = vz;
            w[4] = (div_shared(u[4], c.vol, c.inv_vol) - T(0.5) * r * (vx * vx + vy * vy + vz * vz)) * c.gm1;
        } else {
            const T r1 = plain_div(u[0], c.vol), rv1 = r1 * c.vol;
            const T vx = plain_div(u[1], rv1), vy = plain_div(u[2], rv1), vz = plain_div(u[3], rv1);
            w[0] = r1;
            w[1] = vx;
            w[2] = vy;
            w[3] = vz;
            w[4] = (plain_div(u[4], c.vol) - T(0.5) * r1 * (vx * vx + vy * vy + vz * vz)) * c.gm1;
        }
    }
    // slopes of the five fields from the lower, own and upper value:
    // calc_gradients, physics.rs:206-208 (LIM 0); minmod of the one-sided
    // differences (LIM 1)
    template <int LIM>
    static __device__ __forceinline__ void slopes(const T qm[5], const T q[5], const T qp[5], T g[5],
                                                  const GridArgs<T> &a, const K &k) {
        const Consts<T> &c = a.k;
        KeyBounds kb;
        bool slow = !k.safe;
        if constexpr (LIM == 0) {
#pragma unroll
            for (int f = 0; f < 5; ++f) {
                const T d = qp[f] - qm[f];
                kb.add(d);
                g[f] = div_shared(d, c.two_ds, c.inv_2ds);
            }
        } else {
            // minmod(dm / ds, dp / ds): division by ds > 0 keeps signs and
            // order, so the difference of smaller magnitude is divided.  The
            // limiter's test is the sign of the quotients' product; the
            // differences' product p decides it unless p is so small that
            // either product may underflow
            // (the quotients' is at least p 2^-40 or p 2^-600 for a safe ds).
            constexpr T tiny = sizeof(T) == 4 ? T(0x1p-105) : T(0x1p-470);
#pragma unroll
            for (int f = 0; f < 5; ++f) {
                const T dm = q[f] - qm[f], dp = qp[f] - q[f];
                const T p = dm * dp;
                const T d = fabs(dm) < fabs(dp) ? dm : dp;
                const bool pos = p > tiny;
                slow |= !pos && !(p < T(0)) && d != T(0);
                const T dd = pos ? d : T(0);
                kb.add(dd);
                g[f] = div_shared(dd, c.ds, c.inv_ds);
            }
        }
        if (slow || !kb.safe<T>()) {
#pragma unroll
            for (int f = 0; f < 5; ++f)
                g[f] = LIM == 0 ? plain_div(qp[f] - qm[f], c.two_ds)
                                : minmod(plain_div(q[f] - qm[f], c.ds), plain_div(qp[f] - q[f], c.ds));
        }
    }
    static __device__ __forceinline__ void predict(const T q[5], const T gx[5], const T gy[5], const T gz[5],
                                                   const GridArgs<T> &a, const K &k, T out[5]) {
        Ph::predict(q, gx, gy, gz, k.dt, a.k, out);
    }
    static __device__ __forceinline__ T hs(T g, const GridArgs<T> &a) { return g * a.k.half_ds; }
    // gravity height of a z face (physics.rs:366-372)
    static __device__ __forceinline__ T grav(const GridArgs<T> &a, int klow) {
        return (T(a.nz) - T(2.0) * T(2)) * a.k.ds - (T(klow) - T(2.0)) * a.k.ds;
    }
    // calc_flux_reconstruction, physics.rs:313-405 (the final *ds included),
    // from the two face states: lo = the lower cell's (reference "r"), up =
    // the upper cell's ("l"), N = 1, 2, 3: index of the normal velocity.  heat:
    // the first face of a lower conducting wall, whose energy flux takes Q / V
    // after the advective part (kernels.h:561-575); xt is the lower cell's
    // predicted state up to its mirrored velocity.
    template <int N, bool GRAV>
    static __device__ __forceinline__ void face(const T lo[5], const T up[5], T h, bool heat, const T xt[5],
                                                const GridArgs<T> &a, const K &k, T F[5]) {
        constexpr int T1 = N == 1 ? 2 : 1, T2 = N == 3 ? 2 : 3;
        const Consts<T> &c = a.k;
        const T rl = up[0], vxl = up[N], vyl = up[T1], vzl = up[T2], pl = up[4];
        const T rr = lo[0], vxr = lo[N], vyr = lo[T1], vzr = lo[T2], pr = lo[4];
        const T mxl = rl * vxl, mxr = rr * vxr, myl = rl * vyl, myr = rr * vyr, mzl = rl * vzl, mzr = rr * vzr;
        const T rho_star = (rl + rr) / T(2.0);
        const T mx = (mxl + mxr) / T(2.0);
        const T my = (myl + myr) / T(2.0);
        const T mz = (mzl + mzr) / T(2.0);
        T el = div_shared(pl, c.gm1, c.inv_gm1), er = div_shared(pr, c.gm1, c.inv_gm1);
        KeyBounds kb;
        kb.add(pl);
        kb.add(pr);
        const T y = rcp_rn(rho_star);
        const T xx = mx * mx, xy = mx * my, xz = mx * mz;
        const T kin = T(0.5) * (mx * mx + my * my + mz * mz);
        kb.add(kin);
        kb.add(xx);
        kb.add(xy);
        kb.add(xz);
        kb.add(mx);
        T qk = div_shared(kin, rho_star, y), qxx = div_shared(xx, rho_star, y), qxy = div_shared(xy, rho_star, y),
          qxz = div_shared(xz, rho_star, y), qx = div_shared(mx, rho_star, y);
        if (!(k.safe && safe_divisor(rho_star) && kb.safe<T>())) {
            el = plain_div(pl, c.gm1);
            er = plain_div(pr, c.gm1);
            qk = plain_div(kin, rho_star);
            qxx = plain_div(xx, rho_star);
            qxy = plain_div(xy, rho_star);
            qxz = plain_div(xz, rho_star);
            qx = plain_div(mx, rho_star);
        }
        const T en_left = T(0.5) * (rl * (vxl * vxl + vyl * vyl + vzl * vzl)) + el;
        const T en_right = T(0.5) * (rr * (vxr * vxr + vyr * vyr + vzr * vzr)) + er;
        const T en_star = T(0.5) * (en_left + en_right);
        const T p_star = c.gm1 * (en_star - qk);
        T f1 = qxx + p_star;
        T f2 = qxy;
        T f3 = qxz;
        T f4 = (en_star + p_star) * qx;
        if (heat) f4 += wall_heat(xt[0], xt[4], c.ds);
        if constexpr (GRAV) {
            f1 += T(1.0) * rho_star * c.g * h;
            f4 += T(0.5) * rho_star * (vxl + vxr) * c.g * h;
        }
        const T c_l = sqrt(c.gamma * pl / rl) + fabs(vxl);
        const T c_r = sqrt(c.gamma * pr / rr) + fabs(vxr);
        const T c_star = fmax(c_l, c_r);
        const T f0 = mx - T(0.5) * c_star * (rl - rr);
        f1 -= c_star * (mxl - mxr) / T(2.0);
        f2 -= c_star * (myl - myr) / T(2.0);
        f3 -= c_star * (mzl - mzr) / T(2.0);
        f4 -= c_star * (en_left - en_right) / T(2.0);
        F[0] = f0 * c.ds;
        F[N] = f1 * c.ds;
        F[T1] = f2 * c.ds;
        F[T2] = f3 * c.ds;
        F[4] = f4 * c.ds;
    }
    // add_fluxes, physics.rs:548-554 (the caller sums in the same order)
    static __device__ __forceinline__ T update(T u, T sum, int, const K &k) { return u - k.dtds * sum; }
    // c_s + |v| of an updated cell (calc_timestep, physics.rs:187-189): ds
    // over its maximum is the minimum of the reference's ds / (c_s + |v|),
    // division being monotone
    static __device__ __forceinline__ T speed(const T u[5], const GridArgs<T> &a, const K &k) {
        T w[5];
        prim(u, w, a, k);
        return sqrt(a.k.gamma * w[4] / w[0]) + sqrt(w[1] * w[1] + w[2] * w[2] + w[3] * w[3]);
    }
};

// ---------------------------------------------------------------------------
// Fused arithmetic in FP64: the packed kernel's formulas on scalars (half
// primitives, half slopes, fluxes 2F and 4F).
// ---------------------------------------------------------------------------
struct FusedArith {
    using T = double;
    struct K {
        sweep::K<double> s;
        RefArith<double>::K r;
    };
    static __device__ __forceinline__ K make(const GridArgs<T> &a, T dt) {
        return K{sweep::make_k(a, dt), RefArith<double>::make(a, dt)};
    }
    static __device__ __forceinline__ void prim(const T u[5], T w[5], const GridArgs<T> &, const K &k) {
        sweep::prim_half(u, w, k.s);
    }
    template <int LIM>
    static __device__ __forceinline__ void slopes(const T qm[5], const T q[5], const T qp[5], T g[5],
                                                  const GridArgs<T> &, const K &) {
#pragma unroll
        for (int f = 0; f < 5; ++f) g[f] = sweep::slope1<LIM>(q[f] - qm[f], qp[f] - q[f]);
    }
    static __device__ __forceinline__ void predict(const T q[5], const T gx[5], const T gy[5], const T gz[5],
                                                   const GridArgs<T> &, const K &k, T out[5]) {
        sweep::predict(q, gx, gy, gz, k.s, out);
    }
    static __device__ __forceinline__ T hs(T g, const GridArgs<T> &) { return g; }
    static __device__ __forceinline__ T grav(const GridArgs<T> &a, int klow) { return sweep::grav_h(a, klow); }
    template <int N, bool GRAV>
    static __device__ __forceinline__ void face(const T lo[5], const T up[5], T gh, bool heat, const T xt[5],
                                                const GridArgs<T> &, const K &k, T F[5]) {
        sweep::face<N, GRAV>(lo, up, gh, k.s, F);
        if (heat) F[4] += sweep::heat4(xt[0], xt[4], k.s);
    }
    static __device__ __forceinline__ T update(T u, T sum, int f, const K &k) { return fma(k.s.sc[f], sum, u); }
    // the state reduction's own expression (reference rounding), so that the
    // fused dt equals the reduction's bit for bit
    static __device__ __forceinline__ T speed(const T u[5], const GridArgs<T> &a, const K &k) {
        return RefArith<double>::speed(u, a, k.r);
    }
};

template <class T, int TY, int R> struct Smem {
    static constexpr int kRows = TY + 4;                  // staged rows y0-2 .. y0+TY+1
    static constexpr int kFieldElems = kRows * kBoxZ;
    static constexpr int kBoxBytes = 5 * kFieldElems * (int)sizeof(T);
    static constexpr int kSlotElems = ((kBoxBytes + 127) / 128) * 128 / (int)sizeof(T);
    T ring[R * kSlotElems];                               // conserved totals as staged
    T pb[2][5][kRows][kBoxZ];                             // primitives of the staged cells, by plane parity
    T colq[2][5][32];                                     // the halo columns' cells, by lane of warp A
    T ypl[2][TY + 1][5][kTileZ];                          // upper y state, rows y0-1 .. y0+TY-1
    T fy[2][TY + 1][5][kTileZ];                           // flux of the lower y face, rows y0 .. y0+TY
    T fz[TY][5][kTileZ + 2];                              // flux of the lower z face (own warp's rows only)
    T fxl[TY][5][kTileZ];                                 // the lanes' flux of the x face behind
    T ytop[2][5][kTileZ];                                 // top row's xt (wall) or lower state (outflow)
    T zl[2][TY][5];                                       // left halo column: upper z state (wall: +hs)
    T zr[2][TY][5];                                       // right halo column: lower z state (wall: hs)
    T zeu[2][TY][5];                                      // last column's upper z state
    T zex[2][TY][5];                                      // last column's xt (wall) or lower state (outflow)
    T fzr[2][TY][5];                                      // flux of the right edge face
    uint64_t bar[R];
    unsigned long long wmax;                              // finish_speed
    int abort_flag[2];                                    // by plane parity
    int skip;
};

template <class T, class P, int TY, int R, int LIM, bool GRAV> struct March {
    using Sm = Smem<T, TY, R>;
    using K = typename P::K;
    using Mode = sweep::Mode;
    static_assert(TY <= 14, "halo warps hold two columns of TY rows and four of TY + 2");
    static constexpr int W = TY + 2;      // warps: TY owned rows, A, B
    static constexpr int NT = 32 * W;
    static constexpr int WA = TY, WB = TY + 1;

    static __device__ __forceinline__ T *slot(Sm &s, int l) { return s.ring + (l % R) * Sm::kSlotElems; }
    static __device__ __forceinline__ T mirror(T v, bool on) { return on ? -v : v; }
    static __device__ __forceinline__ float smax_of(float m, float v) { return max_nan(m, v); }
    static __device__ __forceinline__ double smax_of(double m, double v) {
        return (m != m || v != v) ? (m + v) : fmax(m, v);
    }
    static __device__ __forceinline__ void barrier() { asm volatile("bar.sync 0;" ::: "memory"); }

    struct Tile {
        long long budget;
        int y0, z0, xs, xe, np, vy, vz;
        int ylo, yhi, zlo, zhi;
        K k;
        T gh, ghe;   // gravity terms: the lane's lower z face, the right edge face
    };

    static __device__ __forceinline__ bool wait_plane(Sm &s, int l, long long budget) {
        return mbar_wait(&s.bar[l % R], (l / R) & 1, budget);
    }
    // Plane nx-3 with a non-periodic upper x face: the ghost rule's operands
    // wait one plane in the y-state slot of parity (nx-2) & 1, which the row
    // above reads until the end of plane nx-4; every role takes one more
    // barrier first.
    static __device__ __forceinline__ bool upper_stash(const GridArgs<T> &a, int j) {
        return j == a.nx - 3 && a.bc[1] != kPeriodic;
    }
    // staged cell (row ry, column cz of the box) of plane l as primitives
    static __device__ __forceinline__ void load_prim(Sm &s, int l, int ry, int cz, const GridArgs<T> &a, const K &k,
                                                     T q[5]) {
        const T *sl = slot(s, l);
        T u[5];
#pragma unroll
        for (int f = 0; f < 5; ++f) u[f] = sl[(f * Sm::kRows + ry) * kBoxZ + cz];
        P::prim(u, q, a, k);
    }
    static __device__ __forceinline__ void load_pb(Sm &s, int par, int row, int col, T q[5]) {
#pragma unroll
        for (int f = 0; f < 5; ++f) q[f] = s.pb[par][f][row][col];
    }
    // Slopes of the cell at (row, col) of plane parity par: x from qm, qn; y
    // and z from the cells around it.
    static __device__ __forceinline__ void slopes_at(Sm &s, int par, int row, int col, const T qm[5], const T q[5],
                                                     const T qn[5], const GridArgs<T> &a, const K &k, T gx[5], T gy[5],
                                                     T gz[5]) {
        P::template slopes<LIM>(qm, q, qn, gx, a, k);
        T m[5], p[5];
        load_pb(s, par, row - 1, col, m);
        load_pb(s, par, row + 1, col, p);
        P::template slopes<LIM>(m, q, p, gy, a, k);
        load_pb(s, par, row, col - 1, m);
        load_pb(s, par, row, col + 1, p);
        P::template slopes<LIM>(m, q, p, gz, a, k);
    }

    // ---------------------------------------------------------------------
    // The march of one warp.  All warps run the same code on cells of their
    // own: warp r < TY the cells of row y0 + r, warp A those of the row below
    // the tile and then those of the halo columns (lane l < 16: left of row l,
    // else right of row l - 16), warp B those of the row above.  A and B also
    // convert the staged cells nobody owns.  A loop per role made the kernels
    // 145 (FP32) to 190 KB of code, and waiting for instructions their leading
    // stall: 128^3 FP64 472 -> 374 us per step with this one, FP32 292 -> 247
    // (reference rounding); fused FP64, 93 KB, lost some (251 -> 279 at
    // 150x97x131).  What a lane carries from plane to plane beyond lox stays in
    // shared memory for the registers' sake.  Returns the number of planes
    // warp A requested.
    // ---------------------------------------------------------------------
    static __device__ int run_warp(Sm &s, const GridArgs<T> &a, const CUtensorMap *tmap, const Tile &t, int w, int lane,
                                   T &smax) {
        const unsigned full = 0xffffffffu;
        const K &k = t.k;
        const bool isa = w == WA, isb = w == WB, own = w < TY, active = own && w < t.vy;
        const int r = w;
        // staged row of the warp's cells; the staged columns each lane converts
        // and computes on: lanes past the tile's last column work on its halo
        // columns again, so that no lane computes on cells outside the grid
        const int prow = isa ? 1 : (isb ? t.vy + 2 : r + 2);
        const int ccol = 2 + min(lane, t.vz + 1), col = 2 + min(lane, t.vz);
        const int crow = min(lane & 15, t.vy - 1), cz = lane < 16 ? 1 : t.vz + 2;   // warp A's halo column cell
        const int y = t.y0 + r, z = t.z0 + min(lane, t.vz - 1), edge = t.vz - 1;
        const bool valid = lane < t.vz;
        const bool yout = own && r == 0 && t.ylo == sweep::kOut, ywall = own && r == 0 && t.ylo == sweep::kWallM;
        const bool ytop = active && r == t.vy - 1 && t.yhi != sweep::kNormal;
        const bool zheat = lane == 0 && t.zlo == sweep::kWallM && (a.heat & 4);
        const unsigned ybits = active ? image_bits(y, a.ny, a.bc[2], a.bc[3]) : 0;
        const unsigned zbits = active && valid ? image_bits(z, a.nz, a.bc[4], a.bc[5]) : 0;
        const long long cell0 = (long long)y * a.pitch + z;
        const long long plane = (long long)a.ny * a.pitch;
        const int fidx = isb ? t.vy : r;   // the y face this warp computes
        int issued = t.np < R ? t.np : R;
        // carried along the march: lox, the lower state of the x face ahead
        // (and s.fxl, the flux of the x face behind)
        T lox[5];
#pragma unroll
        for (int f = 0; f < 5; ++f) lox[f] = T(0);

        // iterations xs-3 and xs-2 only convert planes xs-2 and xs-1
        for (int j = t.xs - 3; j <= t.xe; ++j) {
            const int l = j - t.xs + 3, pj = j & 1;
            const bool pub = j >= t.xs && j < t.xe;   // plane j's y and z faces belong to this chunk
            T xt[5], hsx[5], hsy[5], hsz[5], d[5];
            if (upper_stash(a, j)) barrier();
            if (!wait_plane(s, l, t.budget)) s.abort_flag[pj] = 1;
            if (active || !own) {
                // The cell at planes j and j-1, read before the conversion of
                // plane j+1 takes plane j-1's place.  Slopes and prediction
                // always, so that they interleave with the conversion: before
                // plane xs-1, and for a ghost row of outflow, nothing uses them.
                T q[5], qm[5], qn[5], gx[5], gy[5], gz[5];
                load_pb(s, pj, prow, col, q);
                load_pb(s, pj ^ 1, prow, col, qm);
                load_prim(s, l, prow, ccol, a, k, qn);
#pragma unroll
                for (int f = 0; f < 5; ++f) s.pb[pj ^ 1][f][prow][ccol] = qn[f];
                slopes_at(s, pj, prow, col, qm, q, qn, a, k, gx, gy, gz);
                P::predict(q, gx, gy, gz, a, k, xt);
#pragma unroll
                for (int f = 0; f < 5; ++f) {
                    hsx[f] = P::hs(gx[f], a);
                    hsy[f] = P::hs(gy[f], a);
                    hsz[f] = P::hs(gz[f], a);
                }
                if (!isb && pub) {
                    const bool wall = isa && t.ylo == sweep::kWallM;   // a ghost row's own half slope
#pragma unroll
                    for (int f = 0; f < 5; ++f) s.ypl[pj][prow - 1][f][lane] = wall ? hsy[f] : xt[f] + hsy[f];
                }
            }
            if (!own) {
                // the staged cells nobody owns: the outermost row (A, B) and the
                // columns outside the lanes' (B); A's halo column cells last
#pragma unroll 1
                for (int task = 1; task < (isa ? 3 : 4); ++task) {
                    const bool cols = isa && task == 2;
                    const int row = task == 1 ? (isa ? 0 : t.vy + 3) : (isa ? crow + 2 : 1 + min(lane >> 1, t.vy + 1));
                    const int cc = task == 1 ? ccol : (isa ? cz : ((lane & 1) ? t.vz + 2 : 0) + task - 2);
                    T cq[5], cm[5], cn[5];
#pragma unroll
                    for (int f = 0; f < 5; ++f) {
                        cq[f] = s.colq[pj][f][lane];
                        cm[f] = s.colq[pj ^ 1][f][lane];
                    }
                    load_prim(s, l, row, cc, a, k, cn);
#pragma unroll
                    for (int f = 0; f < 5; ++f) s.pb[pj ^ 1][f][row][cc] = cn[f];
                    if (!cols) continue;
#pragma unroll
                    for (int f = 0; f < 5; ++f) s.colq[pj ^ 1][f][lane] = cn[f];
                    if (!pub || (t.zlo == sweep::kOut && t.zhi == sweep::kOut)) continue;
                    T gx[5], gy[5], gz[5], ct[5];
                    slopes_at(s, pj, row, cc, cm, cq, cn, a, k, gx, gy, gz);
                    P::predict(cq, gx, gy, gz, a, k, ct);
                    if ((lane & 15) < t.vy) {
#pragma unroll
                        for (int f = 0; f < 5; ++f) {
                            const T h = P::hs(gz[f], a);
                            if (lane < 16) s.zl[pj][crow][f] = t.zlo == sweep::kWallM ? h : ct[f] + h;
                            else s.zr[pj][crow][f] = t.zhi == sweep::kWallM ? h : ct[f] - h;
                        }
                    }
                }
            }
            if (active && j >= t.xs - 1) {
                // a wall's ghost plane 1 keeps its own half slope for the
                // face ahead; an upper ghost plane takes the last plane's
                // operands, stashed one plane earlier
                const bool wall_lo = a.bc[0] == kWall, hi_rule = a.bc[1] != kPeriodic;
                T *stash = &s.ypl[(a.nx - 2) & 1][r + 1][0][lane];
                if (j == a.nx - 3 && hi_rule) {
#pragma unroll
                    for (int f = 0; f < 5; ++f)
                        stash[f * kTileZ] = a.bc[1] == kOutflow ? xt[f] - hsx[f] : mirror(xt[f], f == 1);
                }
                if (j >= t.xs) {
                    T lo[5], up[5], fx[5];
#pragma unroll
                    for (int f = 0; f < 5; ++f) {
                        lo[f] = lox[f];
                        up[f] = xt[f] - hsx[f];
                    }
                    if (j == 2 && wall_lo) {
#pragma unroll
                        for (int f = 0; f < 5; ++f) lo[f] = mirror(xt[f], f == 1) + lo[f];
                    }
                    if (j == a.nx - 2 && hi_rule) {
#pragma unroll
                        for (int f = 0; f < 5; ++f) {
                            const T v = stash[f * kTileZ];
                            up[f] = a.bc[1] == kOutflow ? v : v - hsx[f];
                        }
                    }
                    P::template face<1, false>(lo, up, T(0), j == 2 && (a.heat & 1), xt, a, k, fx);
                    // on a lower outflow x face plane 2 sees no x divergence
                    const bool xo = j - 1 == 2 && a.bc[0] == kOutflow;
#pragma unroll
                    for (int f = 0; f < 5; ++f) {
                        d[f] = fx[f] - (xo ? fx[f] : s.fxl[r][f][lane]);
                        s.fxl[r][f][lane] = fx[f];
                    }
                }
#pragma unroll
                for (int f = 0; f < 5; ++f) lox[f] = j == 1 && wall_lo ? hsx[f] : xt[f] + hsx[f];
                if (pub) {
                    if (ytop) {
#pragma unroll
                        for (int f = 0; f < 5; ++f) s.ytop[pj][f][lane] = t.yhi == sweep::kOut ? xt[f] - hsy[f] : xt[f];
                    }
                    if (lane == edge) {
#pragma unroll
                        for (int f = 0; f < 5; ++f) {
                            s.zeu[pj][r][f] = xt[f] + hsz[f];
                            s.zex[pj][r][f] = t.zhi == sweep::kOut ? xt[f] - hsz[f] : xt[f];
                        }
                    }
                }
            }
            fence_proxy_async();
            barrier();
            if (s.abort_flag[pj]) break;
            if (isa) {
                // the barrier freed the slot converted before it
                const int nl = l + R;
                if (nl < t.np) {
                    if (lane == 0) {
                        mbar_expect_tx(&s.bar[nl % R], Sm::kBoxBytes);
                        tma_load_4d(slot(s, nl), tmap, t.z0 - 2, t.y0 - 2, t.xs - 2 + nl, 0, &s.bar[nl % R]);
                    }
                    issued = nl + 1;
                }
                continue;
            }
            if (active && j > t.xs) {
                // ---- update of plane j-1 (its totals loaded here: earlier, they
                // cost registers that spilled, 400 against 374 us)
                const int pp = pj ^ 1;
                T u[5], u0[5];
                const T *src = a.src + (long long)(j - 1) * plane + cell0;
#pragma unroll
                for (int f = 0; f < 5; ++f) u0[f] = src[f * a.fstride];
#pragma unroll
                for (int f = 0; f < 5; ++f) {
                    const T fyh = s.fy[pp][r + 1][f][lane];
                    const T fyl = yout ? fyh : s.fy[pp][r][f][lane];
                    const T fzh = lane >= edge ? s.fzr[pp][r][f] : s.fz[r][f][lane + 1];
                    const T fzl = lane == 0 && t.zlo == sweep::kOut ? fzh : s.fz[r][f][lane];
                    u[f] = P::update(u0[f], d[f] + fyh - fyl + fzh - fzl, f, k);
                }
                __syncwarp();
                if (valid) {
                    T *dst = a.dst + (long long)(j - 1) * plane + cell0;
#pragma unroll
                    for (int f = 0; f < 5; ++f) dst[f * a.fstride] = u[f];
                    smax = smax_of(smax, P::speed(u, a, k));
                    const int xu = j - 1;
                    const unsigned xbits = xu <= 3 || xu >= a.nx - 4 ? image_bits(xu, a.nx, a.bc[0], a.bc[1]) : 0;
                    if (xbits | ybits | zbits) {
                        // ghost images: every combination of the cell and its
                        // images along the axes, but the cell itself (bit 0:
                        // the cell's own index, bit 1 + g: ghost index g)
                        for (unsigned bx = (xbits & 15u) << 1 | 1u; bx; bx &= bx - 1) {
                            const int gx = __ffs(bx) - 2;
                            for (unsigned by = (ybits & 15u) << 1 | 1u; by; by &= by - 1) {
                                const int gy = __ffs(by) - 2;
                                for (unsigned bz = (zbits & 15u) << 1 | (gx >= 0 || gy >= 0); bz; bz &= bz - 1) {
                                    const int gz = __ffs(bz) - 2;
                                    T *g = a.dst + ((long long)(gx < 0 ? xu : ghost_at(gx, a.nx)) * a.ny +
                                                    (gy < 0 ? y : ghost_at(gy, a.ny))) * a.pitch +
                                           (gz < 0 ? z : ghost_at(gz, a.nz));
                                    g[0] = u[0];
                                    g[a.fstride] = gx >= 0 && ((xbits >> (4 + gx)) & 1) ? -u[1] : u[1];
                                    g[2 * a.fstride] = gy >= 0 && ((ybits >> (4 + gy)) & 1) ? -u[2] : u[2];
                                    g[3 * a.fstride] = gz >= 0 && ((zbits >> (4 + gz)) & 1) ? -u[3] : u[3];
                                    g[4 * a.fstride] = u[4];
                                }
                            }
                        }
                    }
                }
                __syncwarp();
            }
            if (!pub || !(active || isb)) continue;
            // ---- y and z faces of plane j: an owned row's lower y face and its
            // cells' lower z faces; warp B the face above the top row and the
            // right edge faces (one row per lane)
            T lo[5], up[5], F[5];
            if (!yout) {
#pragma unroll
                for (int f = 0; f < 5; ++f) {
                    lo[f] = s.ypl[pj][fidx][f][lane];
                    // wall ghost row: mirrored prediction of this row + its own half slope
                    if (ywall) lo[f] = mirror(xt[f], f == 2) + lo[f];
                    up[f] = xt[f] - hsy[f];
                }
                if (isb && t.yhi != sweep::kNormal) {
#pragma unroll
                    for (int f = 0; f < 5; ++f) {
                        const T x = s.ytop[pj][f][lane];
                        up[f] = t.yhi == sweep::kOut ? x : mirror(x, f == 2) - hsy[f];
                    }
                }
                P::template face<2, false>(lo, up, T(0), ywall && (a.heat & 2), xt, a, k, F);
#pragma unroll
                for (int f = 0; f < 5; ++f) s.fy[pj][fidx][f][lane] = F[f];
            }
            if (isb) {
                const int er = min(lane, t.vy - 1);
#pragma unroll
                for (int f = 0; f < 5; ++f) {
                    lo[f] = s.zeu[pj][er][f];
                    const T zr = s.zr[pj][er][f], zx = s.zex[pj][er][f];
                    up[f] = t.zhi == sweep::kNormal ? zr : (t.zhi == sweep::kOut ? zx : mirror(zx, f == 3) - zr);
                }
            } else {
#pragma unroll
                for (int f = 0; f < 5; ++f) {
                    const T left = __shfl_up_sync(full, xt[f] + hsz[f], 1);
                    lo[f] = lane == 0 ? s.zl[pj][r][f] : left;
                    up[f] = xt[f] - hsz[f];
                }
                if (t.zlo == sweep::kWallM) {
                    if (lane == 0) {
#pragma unroll
                        for (int f = 0; f < 5; ++f) lo[f] = mirror(xt[f], f == 3) + lo[f];
                    }
                }
            }
            P::template face<3, GRAV>(lo, up, isb ? t.ghe : t.gh, own && zheat, xt, a, k, F);
            if (!isb) {
#pragma unroll
                for (int f = 0; f < 5; ++f) s.fz[r][f][lane] = F[f];
            } else if (lane < t.vy) {
#pragma unroll
                for (int f = 0; f < 5; ++f) s.fzr[pj][lane][f] = F[f];
            }
            __syncwarp();
        }
        return issued;
    }

    static __device__ void run(const GridArgs<T> &a, const CUtensorMap *tmap, int chunk, unsigned char *raw) {
        Sm &s = *reinterpret_cast<Sm *>(raw);
        const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
        const int tiles_z = (a.nz - 4 + kTileZ - 1) / kTileZ, tiles_y = (a.ny - 4 + TY - 1) / TY;
        int b = blockIdx.x;
        const int tz = b % tiles_z; b /= tiles_z;
        const int ty = b % tiles_y; b /= tiles_y;
        Tile t;
        t.budget = wait_budget_of(a);
        t.y0 = 2 + ty * TY;
        t.z0 = 2 + tz * kTileZ;
        t.xs = 2 + b * chunk;
        t.xe = min(t.xs + chunk, a.nx - 2);
        t.np = t.xe - t.xs + 4;
        t.vy = min(TY, a.ny - 2 - t.y0);
        t.vz = min(kTileZ, a.nz - 2 - t.z0);
        t.ylo = sweep::side_mode(t.y0 == 2, a.bc[2]);
        t.yhi = sweep::side_mode(t.y0 + t.vy == a.ny - 2, a.bc[3]);
        t.zlo = sweep::side_mode(t.z0 == 2, a.bc[4]);
        t.zhi = sweep::side_mode(t.z0 + t.vz == a.nz - 2, a.bc[5]);
        const unsigned step = (unsigned)a.ctl->step;
        t.k = P::make(a, (T)a.ctl->dt[step & 1]);
        t.gh = t.ghe = T(0);
        if constexpr (GRAV) {
            t.gh = P::grav(a, grav_klow(t.z0 + lane - 1, a.nz, a.bc[4]));
            t.ghe = P::grav(a, t.z0 + t.vz - 1);
        }
        // an earlier step's wait gave up: leave the state alone (read once,
        // so every thread of the block takes the same branch)
        if (tid == 0) {
            s.skip = (*(volatile unsigned *)&a.ctl->flags & kStatusTimeout) != 0;
            s.abort_flag[0] = s.abort_flag[1] = 0;
            s.wmax = 0;
            if (!s.skip) {
                for (int i = 0; i < R; ++i) mbar_init(&s.bar[i], 1);
                fence_mbar_init();
            }
        }
        __syncthreads();
        if (s.skip) return;
        if (warp == WA && lane == 0) {
            for (int l = 0; l < R && l < t.np; ++l) {
                mbar_expect_tx(&s.bar[l], Sm::kBoxBytes);
                tma_load_4d(slot(s, l), tmap, t.z0 - 2, t.y0 - 2, t.xs - 2 + l, 0, &s.bar[l]);
            }
        }
        T smax = T(0);
        const int issued = run_warp(s, a, tmap, t, warp, lane, smax);
        __syncthreads();
        if (s.abort_flag[0] | s.abort_flag[1]) {
            if (warp == WA && lane == 0) {
                // let the copies in flight land before the block exits
                for (int l2 = issued > R ? issued - R : 0; l2 < issued; ++l2)
                    mbar_wait(&s.bar[l2 % R], (l2 / R) & 1, kWaitBudget);
                atomicOr(&a.ctl->flags, kStatusTimeout);
            }
            return;
        }
        if (a.chain & kChainLet) asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
        finish_speed<true>(a, smax, &s.wmax, gridDim.x);
    }
};

template <class T, int TY, int R> constexpr int smem_bytes() {
    static_assert(sizeof(Smem<T, TY, R>) + 1024 <= 232448, "tile exceeds the 227 KB of shared memory per block");
    return (int)sizeof(Smem<T, TY, R>) + 1024;
}

template <class T, class P, int TY, int R, int LIM, bool GRAV>
__global__ void __launch_bounds__(32 * (TY + 2), 1)
    march_step_kernel(const GridArgs<T> a, const __grid_constant__ CUtensorMap tmap, int chunk) {
    extern __shared__ __align__(1024) unsigned char smem_raw[];
    if (a.chain & kChainWait) asm volatile("griddepcontrol.wait;" ::: "memory");
    March<T, P, TY, R, LIM, GRAV>::run(a, &tmap, chunk, smem_raw);
}

template <class T, class P, int TY, int R, int LIM, bool GRAV>
cudaError_t launch_one(const GridArgs<T> &a, const CUtensorMap *tmap, int blocks, int chunk, cudaStream_t st) {
    auto kern = march_step_kernel<T, P, TY, R, LIM, GRAV>;
    constexpr int smem = smem_bytes<T, TY, R>();
    static std::atomic<unsigned long long> attr_set{0};
    const cudaError_t e = ensure_dynamic_smem(kern, smem, attr_set);
    if (e != cudaSuccess) return e;
    return launch_after(kern, blocks, 32 * (TY + 2), smem, st, (a.chain & kChainWait) != 0, a, *tmap, chunk);
}

template <class T, class P, int TY, int R>
cudaError_t launch(const GridArgs<T> &a, const CUtensorMap *tmap, int blocks, int chunk, cudaStream_t st) {
    if (a.gravity)
        return a.limiter == 0 ? launch_one<T, P, TY, R, 0, true>(a, tmap, blocks, chunk, st)
                              : launch_one<T, P, TY, R, 1, true>(a, tmap, blocks, chunk, st);
    return a.limiter == 0 ? launch_one<T, P, TY, R, 0, false>(a, tmap, blocks, chunk, st)
                          : launch_one<T, P, TY, R, 1, false>(a, tmap, blocks, chunk, st);
}

}  // namespace march
}  // namespace dg
