// wave.cu -- wave action balance of one step (wavestep, Wavestep.cu:755-1167;
// arithmetic of the reference's CPU judge, wave_CPU.cpp).
//
// Kernels (launch order):
//   k_disp       dispersion (wave_CPU.cpp:154-205) per cell -> k, c, cg and
//                propagtheta's sigma / sinh(2 kh)
//   k_wave_tma   rows 1..ny-2 with TMA plane tiles (the default; see there)
//   k_wave_fast  rows 1..ny-2, one thread per cell, bins streamed in order:
//                offshore boundary + sanity + action, x/y/theta second-order
//                upwind advection of ee and rr with the Euler step (in energy
//                units), then energint, roelvink|baldock, dissipation,
//                meandir, radstress.  Each bin's ee/rr plane tile (32 x 8
//                cells + 2-cell halo) streams into shared memory by cp.async
//                three bins ahead (five buffers, one barrier per bin), and
//                the cell's own bins for the theta fluxes come from the
//                resident tiles; ctheta
//                (propagtheta) is evaluated on the fly from per-cell slopes;
//                the theta-face flux is computed once and carried to the
//                next bin.  The threads of rows 1 and ny-2 then also
//                finish rows 0 and ny-1, whose ee/rr are copies of theirs
//                (rollerlatbnd, wave_CPU.cpp:830-870) around the
//                dissipation.  Emits the per-block WAVEDT minimum.
//   k_wave_force wavforce + twodimbnd(noix) + breakerdelay + twodimbnd(ust).
#include <type_traits>

#include "xbg_common.cuh"
#include "../../include/xbg.h"

namespace xbg {

// dispersion relation, wave_CPU.cpp:154-205 (golden-ratio relaxation)
template <class R>
__device__ void disp_cell(const Konst<R>& K, R sg, R h, R& k_, R& c_, R& cg_, R& sig_) {
    R g = K.g;
    R L0 = K.twopi * g / (sg * sg);
    R L1 = L0, L2, errdisp;
    // FP32: the relaxation in float (the reference promotes tanh's argument to
    // double through its pi; the stopping rule |L2 - L1| <= 1e-4 m bounds the
    // difference).  FP64: as written.
    const R kh0 = (R)(2 * XBG_PI) * h;
    for (int n = 1; n < 200; n++) {
        if constexpr (sizeof(R) == 4) L2 = L0 * tanhf(kh0 / L1);
        else L2 = (R)((double)L0 * ::tanh(2 * XBG_PI * (double)h / (double)L1));
        errdisp = DM<R>::fabs(L2 - L1);
        L1 = (L1 * K.aphi + L2 * K.bphi);
        if (errdisp <= 0.0001f) break;
        if (n == 199) {
            L1 = L0 * DM<R>::pow(DM<R>::tanh(DM<R>::pow(sg * sg * h / g, (R)(3.0f / 4.0f))), (R)(2.0f / 3.0f));
            break;
        }
    }
    R kk = (R)(2 * XBG_PI / (double)L1);
    k_ = kk;
    R cc = sg / kk;
    c_ = cc;
    R kkhh = cmin(kk * h, (R)10.0f);
    R s2kh = DM<R>::sinh((R)2.0f * kkhh);
    cg_ = cc * ((R)0.5f + kkhh / s2kh);
    sig_ = sg / s2kh;   // propagtheta's sigma / sinh(2 kh)
}

template <class R>
__device__ __forceinline__ void b_disp(const Dev<R>& S, const Konst<R>& K, const int bix, const int biy) {
    const bool off = wave_off(S.clk);   // tested once the cell's loads are issued (see halted())
    int i = bix * blockDim.x + threadIdx.x;
    if (i >= S.C) return;
    const R sg = (R)S.clk->sigm, h = ld(S.f[HH] + i);
    loads_before_here();
    if (off) return;
    R k_, c_, cg_, sig_;
    disp_cell(K, sg, h, k_, c_, cg_, sig_);
    S.f[WK][i] = k_;
    S.f[CC_][i] = c_;
    S.f[CG][i] = cg_;
    S.tmp[T_SIG][i] = sig_;
}
XBG_KERNELS(disp)

// Per-cell slope terms of propagtheta (wave_CPU.cpp:226-306).
template <class R>
struct CthCoef { R s, dhdx, dhdy, dudx, dudy, dvdx, dvdy, wci, sg; };

template <class R>
__device__ __forceinline__ CthCoef<R> cth_coef(const Dev<R>& S, const Konst<R>& K, int ix, int iy, R sg) {
    const int nx = K.nx, ny = K.ny;
    const R* hh = S.f[HH]; const R* uu = S.f[UU]; const R* vv = S.f[VV];
    int xm = mm(ix), xp = pp(ix, nx), ym = mm(iy), yp = pp(iy, ny);
    R dxf = K.dx;
    R sx = (R)(xp - xm) * dxf, sy = (R)(yp - ym) * dxf;
    CthCoef<R> c;
    c.dhdx = (ld(hh + xp + iy * nx) - ld(hh + xm + iy * nx)) / sx;
    c.dudx = (ld(uu + xp + iy * nx) - ld(uu + xm + iy * nx)) / sx;
    c.dvdx = (ld(vv + xp + iy * nx) - ld(vv + xm + iy * nx)) / sx;
    c.dhdy = (ld(hh + ix + yp * nx) - ld(hh + ix + ym * nx)) / sy;
    c.dudy = (ld(uu + ix + yp * nx) - ld(uu + ix + ym * nx)) / sy;
    c.dvdy = (ld(vv + ix + yp * nx) - ld(vv + ix + ym * nx)) / sy;
    int i = ix + iy * nx;
    R h = ld(hh + i);
    c.s = ld(S.tmp[T_SIG] + i);   // sigma / sinh(2 kh), from the dispersion pass
    c.wci = K.wci * cmin(h / K.hwci, (R)1.0f);
    c.sg = sg;
    return c;
}
template <class R>
__device__ __forceinline__ R cth_eval(const CthCoef<R>& c, R cx, R sx) {
    R ctht = (c.s) * (c.dhdx * sx - c.dhdy * cx) +
             c.wci * (cx * (sx * c.dudx - cx * c.dudy) + sx * (sx * c.dvdx - cx * c.dvdy));
    return cmin(cmax(ctht, (R)(-0.25f * c.sg)), (R)(0.25f * c.sg));
}

template <class R>
__device__ __forceinline__ void block_min_store(R v, R* dst) {
    // warp shuffle, then one value per warp through shared memory
    for (int o = 16; o > 0; o >>= 1) v = DM<R>::fmin(v, __shfl_xor_sync(0xffffffffu, v, o));
    __shared__ R wmin[32];
    int tid = threadIdx.x + threadIdx.y * blockDim.x;
    int nw = (blockDim.x * blockDim.y + 31) / 32;
    if ((tid & 31) == 0) wmin[tid >> 5] = v;
    __syncthreads();
    if (tid < 32) {
        R m = tid < nw ? wmin[tid] : (R)3.0e38f;
        for (int o = 16; o > 0; o >>= 1) m = DM<R>::fmin(m, __shfl_xor_sync(0xffffffffu, m, o));
        if (tid == 0) *dst = m;
    }
}

#define WT_X 32
#define WT_Y 8
#define WT_TX (WT_X + 4)
#define WT_TY (WT_Y + 4)
#define WT_N (WT_TX * WT_TY)
// ------------------------------------------------------------------------
// Fast rows pass.  Same algorithm as k_wave_tile, arranged for instruction
// throughput (the pass is issue-bound, not HBM-bound):
//  - ee is advected in energy units: action (ee/sigm), the Euler step and
//    energy (*sigm) of the reference cancel for the uniform sigm, and the
//    upwind selection is scale invariant, so A*sigm = ee - dt*(fluxes of ee);
//  - upwind choices are selects instead of branches (no divergence);
//  - reciprocals of the uniform divisors (dtheta, idiv, D/E) multiply;
//  - WAVEDT's min over bins of a/|ctheta| is a/max|ctheta| (one division);
//  - the theta tables live in shared memory, plane pointers advance by C.
// Results agree with the reference arithmetic to a few ulps per operation.
template <class R>
__device__ __forceinline__ R upw(R a, R b) {   // 1.5a - 0.5b, first-order fallback
    R v = DM<R>::fma((R)1.5, a, (R)-0.5 * b);
    return v < (R)0 ? a : v;
}
// The upwind side is chosen first and one extrapolation evaluated (the same
// value as evaluating both sides and selecting).
template <class R>
__device__ __forceinline__ R flux2(R qm2, R qm, R qi, R qp, R qp2, R cf, R cfmin) {
    const bool pin = cf > (R)0, pmin = cfmin > (R)0;
    const R arrin = upw(pin ? qi : qp, pin ? qm : qp2) * cf;
    const R arrmin = upw(pmin ? qm : qi, pmin ? qm2 : qp) * cfmin;
    return arrin - arrmin;
}
// Without wave-current interaction every face speed of a bin is a cell
// constant times cos(theta) (x) or sin(theta) (y).  The cell constants carry
// dt / dx (kin, kmin: the face speeds 0.5 (cg_i + cg_j) dt / dx), so a bin's
// x or y flux difference is cos (sin) times fk(), and its Euler update
// A = e - (cos fk_x + sin fk_y + dt / dtheta (theta-face difference)).  The
// upwind side is the one of cos (sin): pos.  The box-fed rows pass evaluates the
// same expressions on pairs of cells (xy_flux; bit-identical results).
template <class R>
__device__ __forceinline__ R flux2kv(R qm2, R qm, R qi, R qp, R qp2, bool pos, R kin, R kmin) {
    const R ain = upw(pos ? qi : qp, pos ? qm : qp2);
    const R amin = upw(pos ? qm : qi, pos ? qm2 : qp);
    return DM<R>::fma(ain, kin, -(amin * kmin));
}
template <class R>
__device__ __forceinline__ R euler_k(R e, R ct, R st, R fkx, R fky, R ft, R kth) {
    return e - DM<R>::fma(ct, fkx, DM<R>::fma(st, fky, ft * kth));
}

// theta-face flux between bins t and t+1 (the arrint of bin t, which is the
// arrmint of bin t+1): e(t-1), e(t), e(t+1), e(t+2), ctheta(t), ctheta(t+1)
template <class R>
__device__ __forceinline__ R theta_face(R em, R e0, R ep, R ep2, R c0, R cp) {
    const R cb = (R)0.5f * (c0 + cp);
    const bool p = cb > (R)0;
    const R a = p ? e0 : ep, b = p ? em : ep2;
    R u = DM<R>::fma((R)1.5f, a, DM<R>::mul((R)-0.5f, b));
    u = u < (R)0 ? a : u;
    return cb * u;
}

// Direction tables of the bins in shared memory: (cos, sin) and
// (cos^2, sin^2, sin cos, theta), one vector load each.
template <class R> struct alignas(2 * sizeof(R)) Dir2 { R c, s; };
template <class R> struct alignas(4 * sizeof(R)) Dir4 { R c2, s2, cs, th; };

// energint + roelvink|baldock (wave_CPU.cpp:873-1028) of one cell from the sum
// over bins of its sanitised advected ee: 1/idiv, Dv and Dv / max(Eint, 1e-7).
template <class R>
__device__ __forceinline__ void wave_breaking(const Konst<R>& K, R esum, R hh, R k, R fw, R Trep, R& ridiv, R& Dv,
                                              R& Dq) {
    const R rho = K.rho, g = K.g;
    const R Etmp = esum * K.dtheta;
    R Htmp = DM<R>::sqrt(Etmp / (rho * g / (R)8.0f));
    const R hr = Htmp / (K.gammax * hh);
    const R idiv = DM<R>::fmax((R)1.0f, hr * hr);
    ridiv = (R)1 / idiv;
    Htmp = DM<R>::fmin(Htmp, K.gammax * hh);
    const R Eint = (rho * g * Htmp * Htmp) / (R)8.0f;
    if (K.breakmodel == 1) {   // roelvinkCPU
        R Ht = DM<R>::sqrt(Eint * (R)(8.0 / (double)rho / (double)g));
        R x = Ht / K.gammaa / hh;
        R Qb = (R)1 - DM<R>::exp(DM<R>::fmax(-DM<R>::pow(x, K.nexp), (R)-100));
        Qb = DM<R>::fmin(Qb, (R)1.0f);
        Dv = Qb * (R)2 * K.alpha / Trep * Eint * Ht / hh;
        R uorb = (R)XBG_PI * Ht / (Trep * DM<R>::sinh(DM<R>::fmin(k * hh, (R)10.0f)));
        Dv = Dv + (R)(0.66666666f / XBG_PI) * rho * fw * uorb * uorb * uorb;
    } else {                   // baldockCPU
        R khh = k * hh;
        R Hb = ((R)0.88f / k) * DM<R>::tanh(K.gammaa * khh / (R)0.88f);
        R Rr = Hb / DM<R>::fmax(Htmp, (R)0.00001f);
        R Qb = DM<R>::exp((R)-1.0f * Rr * Rr);
        Dv = (R)0.25f * K.alpha * Qb * rho * ((R)1.0f / Trep) * g * (Hb * Hb + Htmp * Htmp);
        R uorb = (R)XBG_PI * Htmp / (Trep * DM<R>::sinh(DM<R>::fmin(k * hh, (R)10.0f)));
        Dv = Dv + (R)(0.66666666f / XBG_PI) * rho * fw * uorb * uorb * uorb;
    }
    Dq = Dv / DM<R>::fmax(Eint, (R)0.0000001f);
}

// dissipationCPU's wave-energy part of one bin (wave_CPU.cpp:1258-1295): the
// sanitised advected energy a scaled by 1/idiv, its dissipation dd = e Dq,
// and the new energy max(e - dt dd, 0).  One definition for every kernel
// that forms it, so they round alike.
template <class R>
__device__ __forceinline__ R diss_ee(R a, R ridiv, R Dq, R dtf, R& dd) {
    const R eet = DM<R>::mul(DM<R>::fmax(a, (R)0.0f), ridiv);
    dd = DM<R>::mul(eet, Dq);
    return DM<R>::fmax(DM<R>::fma(-dtf, dd, eet), (R)0.0f);
}
// the roller energy of one bin after the roller's dissipation (rrd, the
// dissipation term) and the wave breaking dissipation dd it gains
template <class R>
__device__ __forceinline__ R diss_rr(R rrt, R rrd, R dd, R dtf) {
    return DM<R>::fmax(DM<R>::fma(dtf, dd - rrd, rrt), (R)0.0f);
}

// radstress (wave_CPU.cpp:1123-1162) of one cell from its bin sums: sum2 =
// sum ee, ec / es / ecs = sum (cos^2, sin^2, sin cos) ee, rc / rs / rcs the
// same for rr, n = cg / c.  Every product and fused product is written out,
// so the rounding is the same in every kernel that stores them.
template <class R>
__device__ __forceinline__ void radstress_of(R n, R sum2, R ec, R es, R ecs, R rc, R rs, R rcs, R dth, R& xx, R& xy,
                                             R& yy) {
    const R half = DM<R>::mul((R)-0.5f, sum2);
    xx = DM<R>::fma(DM<R>::fma(n, sum2 + ec, half), dth, DM<R>::mul(rc, dth));
    yy = DM<R>::fma(DM<R>::fma(n, sum2 + es, half), dth, DM<R>::mul(rs, dth));
    xy = DM<R>::fma(DM<R>::mul(n, ecs), dth, DM<R>::mul(rcs, dth));
}
template <class R>
__device__ __forceinline__ void radstress(R* sxx, R* sxy, R* syy, int i, R n, R sum2, R ec, R es, R ecs, R rc, R rs,
                                          R rcs, R dth) {
    radstress_of(n, sum2, ec, es, ecs, rc, rs, rcs, dth, sxx[i], sxy[i], syy[i]);
}

// Row 0 or ny-1 (iyE), the lateral copy of row iyS = 1 or ny-2
// (rollerlatbnd, wave_CPU.cpp:830-870, around dissipationCPU): its advected
// ee and rr are the source row's times the wet mask, breaking and roller
// dissipation run with the edge cell's own depth and speeds, and after
// dissipation its ee is again the source row's (final) ee times the mask.
// adv_e(t), adv_r(t): the source cell's advected bins; src_final(t): its final
// ee.  Returns the edge cell's WAVEDT.
template <class R, bool ROLLER, bool WCI, class AdvE, class AdvR, class SrcFinal>
__device__ __forceinline__ R wave_edge_cell(const Dev<R>& S, const Konst<R>& K, int ix, int iyE, AdvE&& adv_e,
                                            AdvR&& adv_r, const Dir2<R>* sCS2, const Dir4<R>* sMom, R esum, R sg,
                                            R dtf, R Trep, const R* rro, R* een, R* rrn, SrcFinal&& src_final) {
    const int nx = K.nx, nt = K.nt, C = S.C;
    const int ie = ix + iyE * nx;
    const R dth = K.dtheta, rho = K.rho, g = K.g;
    const R hE = ld(S.f[HH] + ie);
    const bool wet = hE > K.eps;
    const R w = wet ? (R)1.0f : (R)0.0f;
    // WAVEDT: cfl*dtheta over the largest |ctheta| of the edge cell's bins
    const CthCoef<R> ce = cth_coef(S, K, ix, iyE, sg);
    const R P = ce.s * ce.dhdx, Q = -(ce.s * ce.dhdy);
    R cab = (R)0;
    for (int t = 0; t < nt; t++) {
        const Dir2<R> d = sCS2[t];
        R c;
        if (WCI) c = cth_eval(ce, d.c, d.s);
        else c = cmin(cmax(DM<R>::fma(P, d.s, Q * d.c), (R)(-0.25f * ce.sg)), (R)(0.25f * ce.sg));
        cab = DM<R>::fmax(cab, DM<R>::fabs(c));
    }
    const R dtw = DM<R>::fmin(K.cfl * dth / cab, (R)9999999.9f);
    // sum of max(A * w, 0) over the bins: the source's sum, or 0 when dry
    R ridiv, Dv, Dq;
    wave_breaking(K, wet ? esum : (R)0, hE, ld(S.f[WK] + ie), ld(S.f[FWM] + ie), Trep, ridiv, Dv, Dq);
    const R cE = ld(S.f[CC_] + ie);
    const R twogb = (R)2.0f * g * K.beta;
    R uE = (R)0, vE = (R)0;
    if (WCI) {
        const R wc = K.wci * cmin(hE / K.hwci, (R)1.0f);
        uE = ld(S.f[UU] + ie) * wc;
        vE = wc * ld(S.f[VV] + ie);
    }
    const R rcoef = twogb / cE;
    R RR = (R)0, drr = (R)0, rc = (R)0, rs = (R)0, rcs = (R)0;
    for (int t = 0; t < nt; t++) {
        const R eet = DM<R>::fmax(adv_e(t) * w, (R)0.0f) * ridiv;
        R rrt = ROLLER ? adv_r(t) * w : ld(rro + ie + (size_t)t * C);
        const R dd = eet * Dq;
        R rrd;
        if (WCI) {
            const Dir2<R> d = sCS2[t];
            const R cx = cE * d.c + uE, cy = cE * d.s + vE;
            rrd = twogb * rrt / DM<R>::sqrt(cx * cx + cy * cy);
        } else {
            rrd = DM<R>::mul(rrt, rcoef);
        }
        rrt = wet ? diss_rr(rrt, rrd, dd, dtf) : (R)0;
        drr = wet ? drr + rrd : (R)0;
        RR = RR + rrt;
        rrn[ie + (size_t)t * C] = rrt;
        const Dir4<R> m = sMom[t];
        rc = DM<R>::fma(m.c2, rrt, rc);
        rs = DM<R>::fma(m.s2, rrt, rs);
        rcs = DM<R>::fma(m.cs, rrt, rcs);
    }
    // the second copy of ee: the source cell's final bins
    R sume = (R)0, sumethet = (R)0, ec = (R)0, es = (R)0, ecs = (R)0;
    for (int t = 0; t < nt; t++) {
        const R eet = src_final(t) * w;
        een[ie + (size_t)t * C] = eet;
        const Dir4<R> m = sMom[t];
        sume = sume + eet;
        sumethet = DM<R>::fma(eet, m.th, sumethet);
        ec = DM<R>::fma(m.c2, eet, ec);
        es = DM<R>::fma(m.s2, eet, es);
        ecs = DM<R>::fma(m.cs, eet, ecs);
    }
    const R sum2 = sume;
    sume = DM<R>::fmax(sume, (R)0.00001f);
    S.f[THM][ie] = sumethet / sume;
    S.f[E][ie] = sume * dth;
    S.f[H][ie] = DM<R>::sqrt(sume * dth / (rho * g / (R)8));
    S.f[D][ie] = Dv;
    S.f[ROL][ie] = RR * dth;
    S.f[DR][ie] = drr * dth;
    const R n = ld(S.f[CG] + ie) / cE;
    radstress(S.tmp[T_SXX], S.tmp[T_SXY], S.tmp[T_SYY], ie, n, sum2, ec, es, ecs, rc, rs, rcs, dth);
    return dtw;
}

// Plane tile buffers.  At bin t planes t, t+1 and t+2 are resident (the
// stencil of plane t; the cell's own values of planes t+1 and t+2 for the
// theta fluxes) and plane t+3 streams in; it goes into the buffer of plane
// t-2, which every thread finished reading before the previous barrier.  More
// planes in flight did not help: with three, 1203 x 599 x 12 bins 121 against 118
// us and 1001 x 401 x 18 102 against 98; 768 x 384 x 12 with currents the same.
constexpr int WT_LEAD = 1;
constexpr int WT_NB = 4 + WT_LEAD;

template <class R, bool ROLLER, bool WCI>
__device__ __forceinline__ void b_wave_fast(const Dev<R>& S, const Konst<R>& K, const int bix, const int biy) {
    constexpr int NB = WT_NB, LEAD = WT_LEAD;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const Clock* clk = S.clk;
    if (wave_off(clk)) return;
    const int nx = K.nx, ny = K.ny, nt = K.nt, C = S.C;
    const int tid = threadIdx.x + threadIdx.y * WT_X;
    R* tE = (R*)smem_raw;                 // [NB][WT_N] plane tiles of ee
    R* tR = tE + NB * WT_N;            // [NB][WT_N] plane tiles of rr
    R* sA = tR + NB * WT_N;            // [nt][256] advected ee (energy units)
    R* sR = sA + (size_t)nt * 256;        // [nt][256] advected rr
    Dir4<R>* sMom = reinterpret_cast<Dir4<R>*>(sR + (size_t)nt * 256);   // [nt]
    Dir2<R>* sCS2 = reinterpret_cast<Dir2<R>*>(sMom + nt);               // [nt]
    if (tid < nt) {
        const R c = K.cxsth[tid], sn = K.sxnth[tid];
        sCS2[tid] = Dir2<R>{c, sn};
        sMom[tid] = Dir4<R>{c * c, sn * sn, sn * c, K.theta[tid]};
    }
    const int bx0 = bix * WT_X, by0 = 1 + biy * WT_Y;
    const int ix = bx0 + threadIdx.x, iy = by0 + threadIdx.y;
    const bool active = ix < nx && iy <= ny - 2;
    const int par = clk->par;
    const R* eeo = S.ee[par ^ 1];
    const R* rro = S.rr[par ^ 1];
    const R dtf = (R)clk->dt;
    const R taper = (R)cmin((double)(R)clk->totaltime / 100.0, 1.0);
    const R* St = S.St;
    const R dth = K.dtheta;
    const R rdth = (R)1 / dth;
    const R rdx = (R)1 / K.dx;
    // tile elements of this thread (two at most): plane offsets, clamped as
    // mm()/pp()/mm2()/pp2() clamp; column 0 is the offshore boundary St*taper
    int eoff0 = -1, eoff1 = -1, ey0 = 0, ey1 = 0;
    bool ez0 = false, ez1 = false;
    {
        int e = tid, kx = e % WT_TX, ky = e / WT_TX;
        int gx = min(max(bx0 - 2 + kx, 0), nx - 1), gy = min(max(by0 - 2 + ky, 0), ny - 1);
        eoff0 = gx + gy * nx; ey0 = gy; ez0 = gx == 0;
        e = tid + 256;
        if (e < WT_N) {
            kx = e % WT_TX; ky = e / WT_TX;
            gx = min(max(bx0 - 2 + kx, 0), nx - 1); gy = min(max(by0 - 2 + ky, 0), ny - 1);
            eoff1 = gx + gy * nx; ey1 = gy; ez1 = gx == 0;
        }
    }
    // sources of this thread's tile elements in the next plane to issue
    const R* gE0 = eeo + eoff0; const R* gR0 = rro + eoff0; const R* gS0 = St + ey0;
    const R* gE1 = eeo + max(eoff1, 0); const R* gR1 = rro + max(eoff1, 0); const R* gS1 = St + ey1;
    // issue the copies of the next plane into buffer b (boundary column written directly)
    auto issue = [&](int b) {
        R* dE = tE + b * WT_N;
        R* dR = tR + b * WT_N;
        if (ez0) dE[tid] = DM<R>::fmax(*gS0 * taper, (R)0);
        else cp_async<sizeof(R)>(dE + tid, gE0);
        if (ROLLER) cp_async<sizeof(R)>(dR + tid, gR0);
        if (eoff1 >= 0) {
            if (ez1) dE[tid + 256] = DM<R>::fmax(*gS1 * taper, (R)0);
            else cp_async<sizeof(R)>(dE + tid + 256, gE1);
            if (ROLLER) cp_async<sizeof(R)>(dR + tid + 256, gR1);
        }
        cp_async_commit();
        gE0 += C; gR0 += C; gS0 += ny; gE1 += C; gR1 += C; gS1 += ny;
    };
    // sanity (ee = max(ee, 0)) on this thread's copied elements of buffer b
    auto fixup = [&](int b) {
        R* dE = tE + b * WT_N;
        if (!ez0) dE[tid] = DM<R>::fmax(dE[tid], (R)0);
        if (eoff1 >= 0 && !ez1) dE[tid + 256] = DM<R>::fmax(dE[tid + 256], (R)0);
    };
    // the cell's tile slot; the tile is clamped like mm()/pp()/mm2()/pp2(), so
    // its x/y neighbours are at fixed offsets +-1, +-2, +-WT_TX, +-2*WT_TX
    const int ctile = (iy - by0 + 2) * WT_TX + (ix - bx0 + 2);
    int i = 0;
    R hh = 0, uui = 0, vvi = 0;
    // face speeds as ct * A + B (x faces) and st * A + B (y faces), for cg (ee) and c (rr)
    R axp = 0, axm = 0, ayp = 0, aym = 0, rxp = 0, rxm = 0, ryp = 0, rym = 0;
    R bxp = 0, bxm = 0, byp = 0, bym = 0, cgi = 0, cci = 0;
    CthCoef<R> cc{};
    R we1 = 0, we2 = 0, we3 = 0, we4 = 0, wr1 = 0, wr2 = 0, wr3 = 0, wr4 = 0;   // bins t-1 .. t+2
    R c0 = 0, cpp = 0, Etmp = 0, cabs = 0, fte = 0, ftr = 0;
    // ctheta of a bin (propagtheta); without wave-current interaction only the
    // depth-refraction term remains: s (dhdx sin - dhdy cos)
    R cthP = 0, cthQ = 0;
    auto cth = [&](R cx, R sx) -> R {
        if (WCI) return cth_eval(cc, cx, sx);
        const R ctht = DM<R>::fma(cthP, sx, cthQ * cx);
        return cmin(cmax(ctht, (R)(-0.25f * cc.sg)), (R)(0.25f * cc.sg));
    };
    // planes 0 .. LEAD + 1 (empty groups past the last plane)
    for (int k = 0; k < LEAD + 2; k++)
        if (k < nt) issue(k); else cp_async_commit();
    __syncthreads();   // theta tables
    if (active) {
        i = ix + iy * nx;
        const int xm = mm(ix), xp = pp(ix, nx);
        const int ym = mm(iy), yp = pp(iy, ny);
        hh = ld(S.f[HH] + i);
        R sg = (R)clk->sigm;
        cc = cth_coef(S, K, ix, iy, sg);
        const R wci = cc.wci;
        const R* cgp = S.f[CG];
        const R* cp = S.f[CC_];
        cgi = ld(cgp + i); cci = ld(cp + i);
        // without wave-current interaction the face speeds carry dt / dx
        // (flux2kv, euler_k: the arithmetic of the TMA rows pass)
        const R h = WCI ? (R)0.5f : (R)0.5f * (dtf * rdx);
        axp = h * (cgi + ld(cgp + xp + iy * nx)); axm = h * (cgi + ld(cgp + xm + iy * nx));
        ayp = h * (cgi + ld(cgp + ix + yp * nx)); aym = h * (cgi + ld(cgp + ix + ym * nx));
        rxp = h * (cci + ld(cp + xp + iy * nx)); rxm = h * (cci + ld(cp + xm + iy * nx));
        ryp = h * (cci + ld(cp + ix + yp * nx)); rym = h * (cci + ld(cp + ix + ym * nx));
        const R* uu = S.f[UU]; const R* vv = S.f[VV];
        uui = ld(uu + i) * wci; vvi = wci * ld(vv + i);
        bxp = h * (uui + ld(uu + xp + iy * nx) * wci); bxm = h * (uui + ld(uu + xm + iy * nx) * wci);
        byp = h * (vvi + wci * ld(vv + ix + yp * nx)); bym = h * (vvi + wci * ld(vv + ix + ym * nx));
        auto cl = [&](int t) { return t < 0 ? 0 : (t >= nt ? nt - 1 : t); };
        if (!WCI) { cthP = cc.s * cc.dhdx; cthQ = -(cc.s * cc.dhdy); }
        c0 = cth(sCS2[0].c, sCS2[0].s);
        cpp = cth(sCS2[cl(1)].c, sCS2[cl(1)].s);
    }
    cp_async_wait<LEAD>();   // planes 0 and 1 have landed (this thread's copies)
    fixup(0);
    if (nt > 1) fixup(1);
    R* oA = sA + tid;
    R* oR = sR + tid;
    const R* oldR = rro + i;   // without the roller pass rr is carried unchanged
#pragma unroll 1
    for (int t = 0; t < nt; t++) {
        const int b = t % NB;
        if (t + 2 + LEAD < nt) issue((t + 2 + LEAD) % NB);
        else cp_async_commit();
        cp_async_wait<LEAD>();   // plane t+2 has landed (this thread's copies)
        if (t + 2 < nt) fixup((t + 2) % NB);
        __syncthreads();    // ... and every thread's
        if (active) {
            const R* qE = tE + b * WT_N + ctile;
            const R* qR = tR + b * WT_N + ctile;
            // the cell's own bins t-1 .. t+2 (clamped to the last bin)
            if (t == 0) {
                const int b1 = (nt > 1 ? 1 : 0);
                we2 = qE[0]; we1 = we2; we3 = tE[b1 * WT_N + ctile];
                if (ROLLER) { wr2 = qR[0]; wr1 = wr2; wr3 = tR[b1 * WT_N + ctile]; }
            }
            const int b2 = (t + 2 < nt ? t + 2 : nt - 1) % NB;
            we4 = tE[b2 * WT_N + ctile];
            if (ROLLER) wr4 = tR[b2 * WT_N + ctile];
            const Dir2<R> d = sCS2[t];
            const R ct = d.c, st = d.s;
            const bool last = t == nt - 1;
            cabs = DM<R>::fmax(cabs, DM<R>::fabs(c0));
            // theta flux: upper face computed here, lower face carried from bin t-1
            R fup = last ? (R)0 : theta_face(we1, we2, we3, we4, c0, cpp);
            R ft = fup - fte;
            fte = fup;
            R A;
            const bool px = ct > (R)0, py = st > (R)0;
            if (WCI) {
                R fx = flux2(qE[-2], qE[-1], we2, qE[1], qE[2], DM<R>::fma(ct, axp, bxp), DM<R>::fma(ct, axm, bxm));
                R fy = flux2(qE[-2 * WT_TX], qE[-WT_TX], we2, qE[WT_TX], qE[2 * WT_TX], DM<R>::fma(st, ayp, byp),
                             DM<R>::fma(st, aym, bym));
                A = we2 - dtf * ((fx + fy) * rdx + ft * rdth);
            } else {
                R fx = flux2kv(qE[-2], qE[-1], we2, qE[1], qE[2], px, axp, axm);
                R fy = flux2kv(qE[-2 * WT_TX], qE[-WT_TX], we2, qE[WT_TX], qE[2 * WT_TX], py, ayp, aym);
                A = euler_k(we2, ct, st, fx, fy, ft, dtf * rdth);
            }
            R Ar;
            if (!ROLLER) Ar = ld(oldR + (size_t)t * C);
            if (ROLLER) {
                R rup = last ? (R)0 : theta_face(wr1, wr2, wr3, wr4, c0, cpp);
                R rt = rup - ftr;
                ftr = rup;
                if (WCI) {
                    R rx = flux2(qR[-2], qR[-1], wr2, qR[1], qR[2], DM<R>::fma(ct, rxp, bxp),
                                 DM<R>::fma(ct, rxm, bxm));
                    R ry = flux2(qR[-2 * WT_TX], qR[-WT_TX], wr2, qR[WT_TX], qR[2 * WT_TX],
                                 DM<R>::fma(st, ryp, byp), DM<R>::fma(st, rym, bym));
                    Ar = wr2 - dtf * ((rx + ry) * rdx + rt * rdth);
                } else {
                    R rx = flux2kv(qR[-2], qR[-1], wr2, qR[1], qR[2], px, rxp, rxm);
                    R ry = flux2kv(qR[-2 * WT_TX], qR[-WT_TX], wr2, qR[WT_TX], qR[2 * WT_TX], py, ryp, rym);
                    Ar = euler_k(wr2, ct, st, rx, ry, rt, dtf * rdth);
                }
            }
            *oA = A;
            *oR = Ar;
            oA += 256; oR += 256;
            Etmp = Etmp + DM<R>::fmax(A, (R)0);
            const int t2 = t + 2 < nt ? t + 2 : nt - 1;
            we1 = we2; we2 = we3; we3 = we4;
            wr1 = wr2; wr2 = wr3; wr3 = wr4;
            const Dir2<R> d2 = sCS2[t2];
            c0 = cpp; cpp = cth(d2.c, d2.s);
        }
    }
    R dtw = (R)3.0e38f;
    if (active) {
        // WAVEDT: min over bins of cfl*dtheta/|ctheta| (Wave_kernel.cu:232-249)
        dtw = DM<R>::fmin(K.cfl * dth / cabs, (R)9999999.9f);
        R* een = S.ee[par];
        R* rrn = S.rr[par];
        const R Trep = (R)clk->Trep;
        const R rho = K.rho, g = K.g;
        R ridiv, Dv, Dq;
        wave_breaking(K, Etmp, hh, ld(S.f[WK] + i), ld(S.f[FWM] + i), Trep, ridiv, Dv, Dq);
        // dissipationCPU, meandir, radstress
        const R cc_i = cci;
        const R twogb = (R)2.0f * g * K.beta;
        const R rcoef = twogb / cc_i;   // without wave-current interaction |c (cos, sin)| = c
        const bool wet = hh > K.eps;
        R RR = (R)0.0f, drr = (R)0.0f, sume = (R)0, sumethet = (R)0;
        R ec = 0, es = 0, ecs = 0, rc = 0, rs = 0, rcs = 0;   // sums of cos^2, sin^2, sin cos times e / r
        R* pe_n = een + i;
        R* pr_n = rrn + i;
        if (wet) {
#pragma unroll 2
            for (int t = 0; t < nt; t++) {
                R dd;
                R eet = diss_ee(sA[t * 256 + tid], ridiv, Dq, dtf, dd);
                R rrt = sR[t * 256 + tid];
                R rrd;
                if (WCI) {
                    const Dir2<R> d = sCS2[t];
                    const R cx = cc_i * d.c + uui;
                    const R cy = cc_i * d.s + vvi;
                    rrd = twogb * rrt / DM<R>::sqrt(cx * cx + cy * cy);
                } else {
                    rrd = DM<R>::mul(rrt, rcoef);
                }
                rrt = diss_rr(rrt, rrd, dd, dtf);
                drr = drr + rrd;
                RR = RR + rrt;
                pe_n[(size_t)t * C] = eet;
                pr_n[(size_t)t * C] = rrt;
                const Dir4<R> m = sMom[t];
                sume = sume + eet;
                sumethet = DM<R>::fma(eet, m.th, sumethet);
                ec = DM<R>::fma(m.c2, eet, ec);
                es = DM<R>::fma(m.s2, eet, es);
                ecs = DM<R>::fma(m.cs, eet, ecs);
                rc = DM<R>::fma(m.c2, rrt, rc);
                rs = DM<R>::fma(m.s2, rrt, rs);
                rcs = DM<R>::fma(m.cs, rrt, rcs);
            }
        } else {   // dry: ee, rr and every sum are zero
            for (int t = 0; t < nt; t++) {
                pe_n[(size_t)t * C] = (R)0;
                pr_n[(size_t)t * C] = (R)0;
            }
        }
        const R sum2 = sume;
        sume = DM<R>::fmax(sume, (R)0.00001f);
        S.f[THM][i] = sumethet / sume;
        S.f[E][i] = sume * dth;
        S.f[H][i] = DM<R>::sqrt(sume * dth / (rho * g / (R)8));
        S.f[D][i] = Dv;
        S.f[ROL][i] = RR * dth;
        S.f[DR][i] = drr * dth;
        const R n = cgi / cc_i;
        // radstress: sum (1 + cos^2) e = sum e + sum cos^2 e, ...
        radstress(S.tmp[T_SXX], S.tmp[T_SXY], S.tmp[T_SYY], i, n, sum2, ec, es, ecs, rc, rs, rcs, dth);
        // the lateral rows 0 and ny-1, from rows 1 and ny-2
        const R sg = (R)clk->sigm;
        // the source cell's final bins: this thread's own stores, read back
        auto own = [&](int t) { return een[i + (size_t)t * C]; };
        auto adv_e = [&](int t) { return sA[t * 256 + tid]; };
        auto adv_r = [&](int t) { return sR[t * 256 + tid]; };
        if (iy == 1)
            dtw = DM<R>::fmin(dtw, wave_edge_cell<R, ROLLER, WCI>(S, K, ix, 0, adv_e, adv_r, sCS2, sMom, Etmp, sg, dtf, Trep,
                                                                  rro, een, rrn, own));
        if (iy == ny - 2)
            dtw = DM<R>::fmin(dtw, wave_edge_cell<R, ROLLER, WCI>(S, K, ix, ny - 1, adv_e, adv_r, sCS2, sMom, Etmp, sg, dtf,
                                                                  Trep, rro, een, rrn, own));
    }
    block_min_store<R>(dtw, S.part_wave + bix + biy * ((K.nx + 31) / 32));
}
template <class R, bool ROLLER, bool WCI>
__global__ void __launch_bounds__(256, sizeof(R) == 4 ? 3 : 2) k_wave_fast(Dev<R> S, Konst<R> K) {
    b_wave_fast<R, ROLLER, WCI>(S, K, blockIdx.x, blockIdx.y);
}
template <class R, bool ROLLER, bool WCI>
__global__ void __launch_bounds__(256, sizeof(R) == 4 ? 3 : 2) kb_wave_fast(BatchTab<R> T, const int2* items, int n) {
    batch_items<R>(T, items, n, [&](const Dev<R>& S, const Konst<R>& K, const BatchAux&, int bx, int by) {
        b_wave_fast<R, ROLLER, WCI>(S, K, bx, by);
    });
}
// the four variants (roller on/off, wave-current interaction on/off)
template <class R>
void launch_wave_fast(const Dev<R>& S, const Konst<R>& K, dim3 g, dim3 b, size_t smem, cudaStream_t st) {
    const bool w = K.wci != (R)0;
    if (K.roller == 1) {
        if (w) k_wave_fast<R, true, true><<<g, b, smem, st>>>(S, K);
        else k_wave_fast<R, true, false><<<g, b, smem, st>>>(S, K);
    } else {
        if (w) k_wave_fast<R, false, true><<<g, b, smem, st>>>(S, K);
        else k_wave_fast<R, false, false><<<g, b, smem, st>>>(S, K);
    }
}
template <class R>
void launch_wave_fast_batch(const BatchTab<R>& T, const BatchLaunch& L, int roller, int wci, size_t smem,
                            cudaStream_t st) {
    dim3 b(32, 8);
    const int g = L.grid[BS_WROWS], n = L.n[BS_WROWS];
    const int2* it = L.items[BS_WROWS];
    if (roller == 1) {
        if (wci) kb_wave_fast<R, true, true><<<g, b, smem, st>>>(T, it, n);
        else kb_wave_fast<R, true, false><<<g, b, smem, st>>>(T, it, n);
    } else {
        if (wci) kb_wave_fast<R, false, true><<<g, b, smem, st>>>(T, it, n);
        else kb_wave_fast<R, false, false><<<g, b, smem, st>>>(T, it, n);
    }
}
template <class R>
size_t wave_fast_smem(int nt) { return ((size_t)2 * WT_NB * WT_N + (size_t)2 * nt * 256 + 6 * nt) * sizeof(R); }

// ------------------------------------------------------------------------
// Rows pass with tensor-memory-accelerator (TMA) tiles: the same arithmetic
// as b_wave_fast (identical results), with the data movement moved off the
// threads.
//  - One elected thread loads each bin's ee and rr plane tile with one box copy
//    (cp.async.bulk.tensor, no multicast) into one of six buffers, completion
//    counted on the buffer's mbarrier.  Only the upwind side of a bin is
//    read, and that side is the bin's (the sign of cos and sin), so a box is
//    the block's 32 x 8 cells with four columns on one side (the 16-byte rule
//    on x; two are used) and two rows on one side: 36 x 10 cells, each row in
//    two 128-byte lines where a box with halos on both sides takes three.
//  - The theta window needs planes t .. t+2 at bin t, so of six buffers three
//    are in flight and a copy has three bins' time to land.  (With four, one
//    bin's time: a block then waited for the copy's latency at every bin, and
//    the pass took the same time with a quarter of its arithmetic removed.)
//  - Cells outside the grid arrive as zeros; blocks at the grid's edges rewrite
//    those (and the offshore column, St * taper) with the clamped values the
//    reference reads through mm()/pp().
//  - ee in memory is never negative (every writer stores max(., 0), and
//    xbg_set_field clips what a caller sets), so the tile needs no sanity
//    pass.
//  - Every wait on an mbarrier is bounded; a block that gives up records
//    XBG_ERR_TIMEOUT in the clock, halts the step, waits (bounded) for its
//    copies in flight and leaves.
// Used for wave-current interaction off and nx a multiple of 4 (the row
// pitch of a tensor map is a multiple of 16 bytes); else b_wave_fast.
constexpr int TM_X = 36, TM_Y = 10, TM_NB = 6;
// elements from one buffer to the next (a copy's destination is 128-byte aligned)
template <class R> constexpr int TM_S = (int)((TM_X * TM_Y * sizeof(R) + 127) / 128 * 128 / sizeof(R));
constexpr unsigned TM_WAIT_LIMIT = 1u << 20;   // mbarrier polls before a block gives up (copies land in microseconds)

__device__ __forceinline__ unsigned su32(const void* p) { return (unsigned)__cvta_generic_to_shared(p); }
__device__ __forceinline__ void tm_mbar_init(unsigned a) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;\n" ::"r"(a) : "memory");
}
__device__ __forceinline__ void tm_expect(unsigned a, unsigned bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;\n" ::"r"(a), "r"(bytes) : "memory");
}
__device__ __forceinline__ bool tm_wait(unsigned a, unsigned parity) {
    for (unsigned it = 0; it < TM_WAIT_LIMIT; it++) {
        unsigned ok;
        asm volatile(
            "{\n.reg .pred p;\nmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\nselp.u32 %0, 1, 0, p;\n}\n"
            : "=r"(ok)
            : "r"(a), "r"(parity)
            : "memory");
        if (ok) return true;
    }
    return false;
}
__device__ __forceinline__ void tm_load3(unsigned dst, const CUtensorMap* m, int x, int y, int z, unsigned mbar) {
    asm volatile(
        "cp.async.bulk.tensor.3d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4}], "
        "[%5];\n" ::"r"(dst),
        "l"((unsigned long long)m), "r"(x), "r"(y), "r"(z), "r"(mbar)
        : "memory");
}
__device__ __forceinline__ void tm_fence_async() { asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory"); }

template <class R>
size_t wave_tma_smem(int nt, int roller) {   // the rr tiles and bins only with the roller
    return 128 + ((size_t)(roller ? 2 : 1) * (TM_NB * TM_S<R> + nt * 256) + 6 * nt) * sizeof(R) + nt * sizeof(int);
}

// ---- arithmetic on pairs of neighbouring cells.  FP32 pairs use the packed
// instructions of sm_100 (fma / mul / add .f32x2: one instruction, each lane
// rounded as the scalar operation it replaces), FP64 pairs are two scalars.
template <class R> struct Pair;
template <> struct Pair<float> {
    using T = float2;
    static __device__ __forceinline__ T make(float a, float b) { return make_float2(a, b); }
    static __device__ __forceinline__ T fma(T a, T b, T c) { return __ffma2_rn(a, b, c); }
    static __device__ __forceinline__ T mul(T a, T b) { return __fmul2_rn(a, b); }
    static __device__ __forceinline__ T add(T a, T b) { return __fadd2_rn(a, b); }
};
template <> struct Pair<double> {
    using T = double2;
    static __device__ __forceinline__ T make(double a, double b) { return make_double2(a, b); }
    static __device__ __forceinline__ T fma(T a, T b, T c) { return T{::fma(a.x, b.x, c.x), ::fma(a.y, b.y, c.y)}; }
    static __device__ __forceinline__ T mul(T a, T b) { return T{__dmul_rn(a.x, b.x), __dmul_rn(a.y, b.y)}; }
    static __device__ __forceinline__ T add(T a, T b) { return T{__dadd_rn(a.x, b.x), __dadd_rn(a.y, b.y)}; }
};
template <class R, class T = typename Pair<R>::T>
__device__ __forceinline__ T pair1(R a) { return Pair<R>::make(a, a); }
template <class R, class T = typename Pair<R>::T>
__device__ __forceinline__ T upw2(T a, T b) {   // upw() of two cells
    T v = Pair<R>::fma(pair1<R>((R)1.5), a, Pair<R>::mul(pair1<R>((R)-0.5), b));
    v.x = v.x < (R)0 ? a.x : v.x;
    v.y = v.y < (R)0 ? a.y : v.y;
    return v;
}

// V neighbouring cells of a row as V / 2 pairs, moved in the widest loads
// (8 or 16 bytes; p is aligned to V elements).
template <class R, int V>
struct Cells {
    static constexpr int NP = V / 2;
    using P = typename Pair<R>::T;
    P p[NP];
    __device__ __forceinline__ R operator[](int j) const { return j & 1 ? p[j / 2].y : p[j / 2].x; }
    __device__ __forceinline__ void set(int j, R v) {
        if (j & 1) p[j / 2].y = v;
        else p[j / 2].x = v;
    }
    __device__ __forceinline__ void load(const R* q) {
        if constexpr (V * sizeof(R) == 16 && V == 4) {
            const float4 v = *reinterpret_cast<const float4*>(q);
            p[0] = P{v.x, v.y};
            p[1] = P{v.z, v.w};
        } else {
#pragma unroll
            for (int k = 0; k < NP; k++) p[k] = reinterpret_cast<const P*>(q)[k];
        }
    }
    __device__ __forceinline__ void load_ro(const R* q) {   // through the read-only path
        if constexpr (V * sizeof(R) == 16 && V == 4) {
            const float4 v = __ldg(reinterpret_cast<const float4*>(q));
            p[0] = P{v.x, v.y};
            p[1] = P{v.z, v.w};
        } else {
#pragma unroll
            for (int k = 0; k < NP; k++) p[k] = __ldg(reinterpret_cast<const P*>(q) + k);
        }
    }
    __device__ __forceinline__ void store(R* q) const {
        if constexpr (V * sizeof(R) == 16 && V == 4) {
            *reinterpret_cast<float4*>(q) = make_float4(p[0].x, p[0].y, p[1].x, p[1].y);
        } else {
#pragma unroll
            for (int k = 0; k < NP; k++) reinterpret_cast<P*>(q)[k] = p[k];
        }
    }
    __device__ __forceinline__ void fill(R v) {
#pragma unroll
        for (int k = 0; k < NP; k++) p[k] = P{v, v};
    }
};

// W consecutive values of a field in one access (W a power of two, 16 bytes at most)
template <class R, int W>
__device__ __forceinline__ void load_row(R (&v)[W], const R* p) {
    if constexpr (W == 1) {
        v[0] = ld(p);
    } else if constexpr (W * sizeof(R) == 16 && W == 4) {
        const float4 x = __ldg(reinterpret_cast<const float4*>(p));
        v[0] = x.x; v[1] = x.y; v[2] = x.z; v[3] = x.w;
    } else {
        const typename Pair<R>::T x = __ldg(reinterpret_cast<const typename Pair<R>::T*>(p));
        v[0] = x.x; v[1] = x.y;
    }
}
template <class R, int W>
__device__ __forceinline__ void store_row(R* p, const R (&v)[W]) {
    if constexpr (W == 1) *p = v[0];
    else if constexpr (W * sizeof(R) == 16 && W == 4) *reinterpret_cast<float4*>(p) = make_float4(v[0], v[1], v[2], v[3]);
    else *reinterpret_cast<typename Pair<R>::T*>(p) = typename Pair<R>::T{v[0], v[1]};
}

// Phase 1 constants of a thread's V cells: the V + 1 x-face speeds, the upper
// and the negated lower y-face speeds (both times dt / dx), and the negated
// flux of the theta face below, carried from bin to bin.
template <class R, int V>
struct RowFlux {
    R kx[V + 1];
    typename Pair<R>::T ky[V / 2], kyn[V / 2], fdn[V / 2];
};
// Second-order upwind flux differences in x and y over a thread's V cells on
// the side of the bin's cos / sin (PX, PY).  q: the field's plane tile at the
// first cell (row pitch TM_X), e2 the cells' values there.  Each x face is
// evaluated once for the two cells beside it.
template <class R, int V, bool PX, bool PY>
__device__ __forceinline__ void xy_flux(const R* q, const Cells<R, V>& e2, const RowFlux<R, V>& f, Cells<R, V>& fx,
                                        Cells<R, V>& fy) {
    using PR = Pair<R>;
    R ext[V + 1];   // the extrapolated value at x face j (left of cell j)
    if (PX) {
        const typename PR::T l = *reinterpret_cast<const typename PR::T*>(q - 2);
        ext[0] = upw(l.y, l.x);
        ext[1] = upw(e2[0], l.y);
#pragma unroll
        for (int j = 2; j <= V; j++) ext[j] = upw(e2[j - 1], e2[j - 2]);
    } else {
        const typename PR::T r = *reinterpret_cast<const typename PR::T*>(q + V);
#pragma unroll
        for (int j = 0; j < V - 1; j++) ext[j] = upw(e2[j], e2[j + 1]);
        ext[V - 1] = upw(e2[V - 1], r.x);
        ext[V] = upw(r.x, r.y);
    }
#pragma unroll
    for (int j = 0; j < V; j++) fx.set(j, DM<R>::fma(ext[j + 1], f.kx[j + 1], -(DM<R>::mul(ext[j], f.kx[j]))));
    Cells<R, V> a, b;
    a.load(PY ? q - TM_X : q + TM_X);
    b.load(PY ? q - 2 * TM_X : q + 2 * TM_X);
#pragma unroll
    for (int k = 0; k < V / 2; k++) {
        const auto up = PY ? upw2<R>(e2.p[k], a.p[k]) : upw2<R>(a.p[k], b.p[k]);
        const auto lo = PY ? upw2<R>(a.p[k], b.p[k]) : upw2<R>(e2.p[k], a.p[k]);
        fy.p[k] = PR::fma(up, f.ky[k], PR::mul(lo, f.kyn[k]));
    }
}

// Phase 2 of the rows pass over a thread's W neighbouring cells, the first at
// (ix, iy): breaking, dissipation, mean direction and radiation stresses from
// the advected bins at pA[256 t], pR[256 t]; the new bins go to global memory
// (een, rrn), so that the block has nothing left to wait for at its end.  A
// warp holds W rows of 32 cells (the first row's first cell is column bx0); the
// warp that holds row 1 or ny-2 first finishes row 0 or ny-1, one lateral cell
// per lane.  Every thread of a warp comes here, active or not.  Returns the
// smallest WAVEDT of the lateral cells.
template <class R, bool ROLLER, int W>
__device__ __forceinline__ R wave_phase2(const Dev<R>& S, const Konst<R>& K, int bx0, int ix, int iy, const R* pA,
                                         const R* pR, const R* pSum, const Dir4<R>* sMom, const Dir2<R>* sCS2, R sg, R dtf,
                                         const R* rro, R* een, R* rrn) {
    const int nx = K.nx, ny = K.ny, nt = K.nt, C = S.C, i = ix + iy * nx;
    const bool active = ix < nx && iy <= ny - 2;
    const R Trep = (R)S.clk->Trep, dth = K.dtheta, rho = K.rho, g = K.g;
    const R twogb = (R)2.0f * g * K.beta;
    R dtw = (R)3.0e38f;
    R hh[W], cg[W], cc[W], kk[W], fw[W], ridiv[W], Dv[W], Dq[W], rcoef[W];
    bool wet[W];
    bool allwet = true;
    if (active) {
        load_row<R, W>(hh, S.f[HH] + i);
        load_row<R, W>(cg, S.f[CG] + i);
        load_row<R, W>(cc, S.f[CC_] + i);
        load_row<R, W>(kk, S.f[WK] + i);
        load_row<R, W>(fw, S.f[FWM] + i);
    }
#pragma unroll
    for (int j = 0; j < W; j++) {
        if (active) wave_breaking(K, pSum[j], hh[j], kk[j], fw[j], Trep, ridiv[j], Dv[j], Dq[j]);
        else hh[j] = cg[j] = cc[j] = ridiv[j] = Dv[j] = Dq[j] = (R)1;
        rcoef[j] = twogb / cc[j];
        wet[j] = hh[j] > K.eps;
        allwet = allwet && wet[j];
    }
    // the lateral rows 0 and ny-1; the source cell's new ee is formed as below
    const int lane = (int)threadIdx.x & 31;
    const int y0 = iy - lane * W / 32;   // the warp's first row
    if (y0 <= 1 || y0 + W > ny - 2) {
#pragma unroll 1
        for (int n = 0; n < 2 * W; n++) {
            const int r = n / 2, iyE = n % 2 ? ny - 1 : 0;   // the source row, the lateral row
            if (y0 + r != (n % 2 ? ny - 2 : 1)) continue;    // the same for the whole warp
            // the source cell's thread, and its values there
            const int own = (r * 32 + lane) / W, j = lane % W;
            R a = (R)0, q = (R)0, e = (R)0;
#pragma unroll
            for (int m = 0; m < W; m++) {
                const R am = __shfl_sync(0xffffffffu, ridiv[m], own), qm = __shfl_sync(0xffffffffu, Dq[m], own),
                        em = __shfl_sync(0xffffffffu, hh[m], own);
                if (m == j) { a = am; q = qm; e = em; }
            }
            if (bx0 + lane >= nx) continue;
            const int off = (r - lane * W / 32) * 32 + lane - lane * W % 32;   // from this thread's first cell
            const R* sa = pA + off;
            const R* sr = pR + off;
            const bool w = e > K.eps;
            auto adv_e = [&](int t) { return sa[t * 256]; };
            auto adv_r = [&](int t) { return sr[t * 256]; };
            auto fin = [&](int t) {
                R dd;
                return w ? diss_ee(sa[t * 256], a, q, dtf, dd) : (R)0;
            };
            dtw = DM<R>::fmin(dtw, wave_edge_cell<R, ROLLER, false>(S, K, bx0 + lane, iyE, adv_e, adv_r, sCS2, sMom,
                                                                   pSum[off], sg, dtf, Trep, rro, een, rrn, fin));
        }
    }
    if (!active) return dtw;
    R* pe = een + i;
    R* pr = rrn + i;
    const R* po = rro + i;   // without the roller pass rr is carried unchanged
    R o[9][W];   // thetamean, E, H, R, DR, the radiation stresses, D
    auto finish = [&](int j, R sum2, R RR, R drr, R sumethet, R ec, R es, R ecs, R rc, R rs, R rcs) {
        const R sume = DM<R>::fmax(sum2, (R)0.00001f);
        o[0][j] = sumethet / sume;
        o[1][j] = sume * dth;
        o[2][j] = DM<R>::sqrt(sume * dth / (rho * g / (R)8));
        o[3][j] = RR * dth;
        o[4][j] = drr * dth;
        radstress_of(cg[j] / cc[j], sum2, ec, es, ecs, rc, rs, rcs, dth, o[5][j], o[6][j], o[7][j]);
        o[8][j] = Dv[j];
    };
    using PR = Pair<R>;
    using P = typename PR::T;
    const P zero = pair1<R>((R)0);
    if constexpr (W == 1) {   // (wave energy, roller energy) pairs of the one cell
        P sr = zero, cc2 = zero, ss2 = zero, cs2 = zero;
        R drr = (R)0, sumethet = (R)0;
        if (wet[0]) {
#pragma unroll 2
            for (int t = 0; t < nt; t++) {
                R dd;
                const R eet = diss_ee(pA[t * 256], ridiv[0], Dq[0], dtf, dd);
                R rrt = ROLLER ? pR[t * 256] : ld(po + (size_t)t * C);
                const R rrd = DM<R>::mul(rrt, rcoef[0]);
                rrt = diss_rr(rrt, rrd, dd, dtf);
                drr = drr + rrd;
                pe[(size_t)t * C] = eet;
                pr[(size_t)t * C] = rrt;
                const Dir4<R> m = sMom[t];
                const P er = PR::make(eet, rrt);
                sr = PR::add(sr, er);
                sumethet = DM<R>::fma(eet, m.th, sumethet);
                cc2 = PR::fma(pair1<R>(m.c2), er, cc2);
                ss2 = PR::fma(pair1<R>(m.s2), er, ss2);
                cs2 = PR::fma(pair1<R>(m.cs), er, cs2);
            }
        } else {
            for (int t = 0; t < nt; t++) pe[(size_t)t * C] = pr[(size_t)t * C] = (R)0;
        }
        finish(0, sr.x, sr.y, drr, sumethet, cc2.x, ss2.x, cs2.x, cc2.y, ss2.y, cs2.y);
    } else {                  // pairs of neighbouring cells
        using CW = Cells<R, W>;
        CW drr, se, sr, st, ec, es, ecs, rc, rs, rcs, vi, vq, vc;
        drr.fill((R)0); se = sr = st = ec = es = ecs = rc = rs = rcs = drr;
#pragma unroll
        for (int j = 0; j < W; j++) { vi.set(j, ridiv[j]); vq.set(j, Dq[j]); vc.set(j, rcoef[j]); }
        const P dtp = pair1<R>(dtf), dtn = pair1<R>(-dtf), neg = pair1<R>((R)-1);
        auto sweep = [&](auto mask) {
            constexpr bool MASK = decltype(mask)::value;
            constexpr int AHEAD = 3;   // without the roller: bins of rr in flight
            CW ahead[AHEAD];
            if (!ROLLER)
#pragma unroll
                for (int k = 0; k < AHEAD; k++) ahead[k].load_ro(po + (size_t)min(k, nt - 1) * C);
#pragma unroll 2
            for (int t = 0; t < nt; t++) {
                CW a, r;
                a.load(pA + t * 256);
                if (ROLLER) {
                    r.load(pR + t * 256);
                } else {
                    r = ahead[0];
#pragma unroll
                    for (int k = 0; k + 1 < AHEAD; k++) ahead[k] = ahead[k + 1];
                    ahead[AHEAD - 1].load_ro(po + (size_t)min(t + AHEAD, nt - 1) * C);
                }
                const Dir4<R> m = sMom[t];
#pragma unroll
                for (int k = 0; k < W / 2; k++) {
                    // diss_ee, diss_rr of two cells
                    const P z = PR::make(DM<R>::fmax(a.p[k].x, (R)0), DM<R>::fmax(a.p[k].y, (R)0));
                    const P eet = PR::mul(z, vi.p[k]);
                    const P dd = PR::mul(eet, vq.p[k]);
                    P e = PR::fma(dtn, dd, eet);
                    e.x = DM<R>::fmax(e.x, (R)0); e.y = DM<R>::fmax(e.y, (R)0);
                    P rrd = PR::mul(r.p[k], vc.p[k]);
                    P q = PR::fma(dtp, PR::add(dd, PR::mul(rrd, neg)), r.p[k]);
                    q.x = DM<R>::fmax(q.x, (R)0); q.y = DM<R>::fmax(q.y, (R)0);
                    if (MASK) {
                        if (!wet[2 * k]) { e.x = (R)0; q.x = (R)0; rrd.x = (R)0; }
                        if (!wet[2 * k + 1]) { e.y = (R)0; q.y = (R)0; rrd.y = (R)0; }
                    }
                    a.p[k] = e;
                    r.p[k] = q;
                    drr.p[k] = PR::add(drr.p[k], rrd);
                    se.p[k] = PR::add(se.p[k], e);
                    sr.p[k] = PR::add(sr.p[k], q);
                    st.p[k] = PR::fma(e, pair1<R>(m.th), st.p[k]);
                    ec.p[k] = PR::fma(pair1<R>(m.c2), e, ec.p[k]);
                    es.p[k] = PR::fma(pair1<R>(m.s2), e, es.p[k]);
                    ecs.p[k] = PR::fma(pair1<R>(m.cs), e, ecs.p[k]);
                    rc.p[k] = PR::fma(pair1<R>(m.c2), q, rc.p[k]);
                    rs.p[k] = PR::fma(pair1<R>(m.s2), q, rs.p[k]);
                    rcs.p[k] = PR::fma(pair1<R>(m.cs), q, rcs.p[k]);
                }
                a.store(pe + (size_t)t * C);
                r.store(pr + (size_t)t * C);
            }
        };
        if (allwet) sweep(std::false_type{});
        else sweep(std::true_type{});
#pragma unroll
        for (int j = 0; j < W; j++)
            finish(j, se[j], sr[j], drr[j], st[j], ec[j], es[j], ecs[j], rc[j], rs[j], rcs[j]);
    }
    store_row<R, W>(S.f[THM] + i, o[0]);
    store_row<R, W>(S.f[E] + i, o[1]);
    store_row<R, W>(S.f[H] + i, o[2]);
    store_row<R, W>(S.f[ROL] + i, o[3]);
    store_row<R, W>(S.f[DR] + i, o[4]);
    store_row<R, W>(S.tmp[T_SXX] + i, o[5]);
    store_row<R, W>(S.tmp[T_SXY] + i, o[6]);
    store_row<R, W>(S.tmp[T_SYY] + i, o[7]);
    store_row<R, W>(S.f[D] + i, o[8]);
    return dtw;
}

// propagtheta's clamp of ctheta in [lo, hi] (cmin(cmax(v, lo), hi): a NaN
// stays one), one instruction per side
__device__ __forceinline__ float clamp_nan(float v, float lo, float hi) {
    asm("max.NaN.f32 %0, %0, %1;\n\tmin.NaN.f32 %0, %0, %2;" : "+f"(v) : "f"(lo), "f"(hi));
    return v;
}
__device__ __forceinline__ double clamp_nan(double v, double lo, double hi) { return cmin(cmax(v, lo), hi); }

// The rows pass over a block of 32 x 8 cells in two phases.  What bounds it is
// the time a block spends per bin with four blocks on an SM: plane copies take
// about 2.4 us to land under load whatever the box (108 to 187 cycles per box
// and SM in a pure stream of boxes of 1 to 7 KB), and the arithmetic of a bin
// runs beside the other blocks' waits only.  At 2048 x 1024 x 18 bins the pass
// takes 277 us (2.7 TB/s of its 352 bytes per cell); without any x, y, theta
// and dissipation arithmetic it takes 190.  One cell per thread, four buffers
// and boxes with halos on both sides took 334 us.
//  1. Advection, V neighbouring cells of a row per thread.  One wide
//     shared-memory load brings V cells' taps, each x face is evaluated once
//     for the two cells beside it, y and theta fluxes run in packed arithmetic.
//     SPLIT: half of the block's warps advect the wave energy and half the
//     roller energy (the same code on another plane and other face speeds);
//     else every thread advects both.
//  2. Breaking and dissipation, W cells of both fields per thread, every thread
//     of the block on its own cells; the bin sums of the wave energy pass from
//     phase 1 through shared memory.
template <class R, bool ROLLER, int V, bool SPLIT>
__device__ __forceinline__ void b_wave_tma(const Dev<R>& S, const Konst<R>& K, const WaveMaps& M, const int bix,
                                           const int biy) {
    static_assert(ROLLER || !SPLIT, "one field has no second half");
    constexpr int TXN = WT_X / V, NF = TXN * WT_Y;        // phase 1: threads per cell row and per field
    constexpr int NTH = (SPLIT ? 2 : 1) * NF, W = 256 / NTH;   // the block's threads; phase 2: cells per thread
    constexpr int NP = V / 2, NFLD = ROLLER && !SPLIT ? 2 : 1, PL = TM_S<R>;
    using PR = Pair<R>;
    using P = typename PR::T;
    using CV = Cells<R, V>;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    __shared__ __align__(8) unsigned long long mbar[TM_NB];
    Clock* clk = S.clk;
    // the flags and the clock's values in one round trip to memory
    const bool off = wave_off(clk);
    const int par = clk->par;
    const R dtf = (R)clk->dt;
    const R taper = (R)cmin((double)(R)clk->totaltime / 100.0, 1.0);
    const R sg = (R)clk->sigm;
    loads_before_here();
    if (off) return;
    const int nx = K.nx, ny = K.ny, nt = K.nt;
    const int tid = threadIdx.x;
    const unsigned base = (su32(smem_raw) + 127u) & ~127u;
    R* tE = reinterpret_cast<R*>(smem_raw + (base - su32(smem_raw)));   // [TM_NB][PL] plane tiles of ee
    R* tR = tE + (ROLLER ? TM_NB * PL : 0);                             // [TM_NB][PL] plane tiles of rr
    R* sA = tR + TM_NB * PL;             // [nt][256] advected ee (energy units)
    R* sR = sA + (size_t)nt * 256;       // [nt][256] advected rr (with the roller)
    R* sSum = tE;                        // [256] sum over the bins of max(advected ee, 0), once the tiles are done with
    Dir4<R>* sMom = reinterpret_cast<Dir4<R>*>(sR + (ROLLER ? (size_t)nt * 256 : 0));
    Dir2<R>* sCS2 = reinterpret_cast<Dir2<R>*>(sMom + nt);
    int* sOff = reinterpret_cast<int*>(sCS2 + nt);   // [nt] tile index of the block's first cell in the bin's box
    for (int t = tid; t < nt; t += NTH) {
        const R c = K.cxsth[t], sn = K.sxnth[t];
        sCS2[t] = Dir2<R>{c, sn};
        sMom[t] = Dir4<R>{c * c, sn * sn, sn * c, K.theta[t]};
        sOff[t] = (c > (R)0 ? 4 : 0) + (sn > (R)0 ? 2 * TM_X : 0);
    }
    const int bx0 = bix * WT_X, by0 = 1 + biy * WT_Y;
    if (tid < 2 * WT_Y && by0 + tid / 2 < ny) {   // phase 2's own fields into L2
        const R* p = (tid & 1 ? S.f[FWM] : S.f[WK]) + (size_t)(by0 + tid / 2) * nx + bx0;
        asm volatile("prefetch.global.L2 [%0];\n" ::"l"(p));
    }
    const CUtensorMap* mE = &M.ld_e[par ^ 1];
    const CUtensorMap* mR = &M.ld_r[par ^ 1];
    const R* rro = S.rr[par ^ 1];
    const R dth = K.dtheta;
    const R rdth = (R)1 / dth;
    const R rdx = (R)1 / K.dx;
    const R cmax_ = (R)(0.25f * sg), cmin_ = (R)(-0.25f * sg);   // propagtheta's clamp of ctheta
    const R kxy = dtf * rdx, kth = dtf * rdth;
    constexpr unsigned TBYTES = (ROLLER ? 2u : 1u) * TM_X * TM_Y * sizeof(R);
    if (tid == 0) {
        for (int b = 0; b < TM_NB; b++) tm_mbar_init(su32(&mbar[b]));
        asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
        tm_fence_async();
    }
    __syncthreads();   // barriers initialised, theta tables written
    int issued = 0;             // planes issued so far (elected thread)
    auto issue = [&](int p, int b) {   // elected thread: plane p into buffer b = p % TM_NB
        issued = p + 1;
        const unsigned mb = su32(&mbar[b]);
        const Dir2<R> d = sCS2[p];
        const int x = d.c > (R)0 ? bx0 - 4 : bx0, y = d.s > (R)0 ? by0 - 2 : by0;
        tm_expect(mb, TBYTES);
        tm_load3(su32(tE + b * PL), mE, x, y, p, mb);
        if (ROLLER) tm_load3(su32(tR + b * PL), mR, x, y, p, mb);
    };
    if (tid == 0)
        for (int p = 0; p < nt && p < TM_NB; p++) issue(p, p);
    // The clamped values of the tile's out-of-grid cells and St * taper on
    // column 0 (ee only), over the cells the taps reach (two columns or rows on
    // the bin's upwind sides): every rewritten cell reads an in-grid cell of
    // column >= 1 of the same box, which no thread rewrites.
    const bool edge = bx0 == 0 || bx0 + 33 > nx - 1 || by0 - 2 < 0 || by0 + 9 > ny - 1;
    // The cells to rewrite, one list for the block (a thread's share is looked
    // up once): columns -2, -1, 0 and nx, nx + 1 (10 cells each), rows -1 and
    // ny (36 each).  A column's place in a box moves with the bin's box in x, a
    // row's in y.
    constexpr int NFIX = 5 * TM_Y + 2 * TM_X, NFT = (NFIX + NTH - 1) / NTH;
    int fixx[NFT], fixy[NFT];
    unsigned fixcol = 0, fixrow = 0;   // bit k: entry k is a column's (row's) cell that exists in this block
#pragma unroll
    for (int k = 0; k < NFT; k++) {
        const int e = tid + k * NTH;
        fixx[k] = fixy[k] = 0;
        if (e < 5 * TM_Y) {
            const int c = e / TM_Y;   // column -2, -1, 0 or nx, nx + 1
            fixx[k] = c < 3 ? c - 2 : nx - bx0 + c - 3;
            fixy[k] = e % TM_Y;
            if (c < 3 ? bx0 == 0 : bx0 + 33 > nx - 1) fixcol |= 1u << k;
        } else if (e < NFIX) {
            const int r = e - 5 * TM_Y;
            fixx[k] = r % TM_X;
            fixy[k] = (r < TM_X ? -1 : ny) - by0;
            if (r < TM_X ? by0 - 2 < 0 : by0 + 9 > ny - 1) fixrow |= 1u << k;
        }
    }
    auto fixup = [&](int p, int b) {
        R* dE = tE + b * PL;
        R* dR = tR + b * PL;
        const int o = sOff[p], ox = o & 4, oy = o >= 2 * TM_X ? 2 : 0;
#pragma unroll
        for (int k = 0; k < NFT; k++) {
            if (!((fixcol | fixrow) >> k & 1u)) continue;
            const int kx = fixx[k] + (fixcol >> k & 1u ? ox : 0), ky = fixy[k] + (fixrow >> k & 1u ? oy : 0);
            if (kx < 0 || kx >= TM_X || ky < 0 || ky >= TM_Y) continue;
            const int gx = bx0 - ox + kx, gy = by0 - oy + ky;
            const int cx = min(max(gx, 0), nx - 1), cy = min(max(gy, 0), ny - 1);
            const bool in = cx == gx && cy == gy;
            const int e = kx + ky * TM_X, src = (cx - (bx0 - ox)) + (cy - (by0 - oy)) * TM_X;
            if (!(in && gx != 0)) dE[e] = cx == 0 ? DM<R>::fmax(S.St[cy + p * ny] * taper, (R)0) : dE[src];
            if (ROLLER && !in) dR[e] = dR[src];
        }
        tm_fence_async();   // these writes before the buffer's next box copy
    };
    bool ok = true;
    R dtw = (R)3.0e38f;
    {   // ---- phase 1
        const bool isE = !SPLIT || tid < NF;   // the same for a whole warp
        const int l = SPLIT ? tid % NF : tid, lx = (l % TXN) * V, ly = l / TXN;
        const int ix = bx0 + lx, iy = by0 + ly;                    // the thread's first cell
        const int cid = lx + ly * WT_X;                            // its place in sA, sR
        const bool active = ix < nx && iy <= ny - 2;   // nx is a multiple of 4: all V cells or none
        const R* tX[NFLD];
        R* sX[NFLD];
        RowFlux<R, V> f[NFLD];
        tX[0] = (isE ? tE : tR) + ly * TM_X + lx;
        sX[0] = (isE ? sA : sR) + cid;
        if constexpr (NFLD == 2) { tX[1] = tR + ly * TM_X + lx; sX[1] = sR + cid; }
        Cells<R, V> cP, cQ, c0, cp;   // ctheta = cP sin + cQ cos, clamped; of bins t and t + 1
        cP.fill((R)0); cQ.fill((R)0); c0.fill((R)0); cp.fill((R)0);
#pragma unroll
        for (int k = 0; k < NFLD; k++) f[k] = RowFlux<R, V>{};
        auto ctheta = [&](Cells<R, V>& o, R cx, R sx) {
#pragma unroll
            for (int k = 0; k < NP; k++) {
                P v = PR::fma(cP.p[k], pair1<R>(sx), PR::mul(cQ.p[k], pair1<R>(cx)));
                v.x = clamp_nan(v.x, cmin_, cmax_);
                v.y = clamp_nan(v.y, cmin_, cmax_);
                o.p[k] = v;
            }
        };
        if (active) {
            const int i = ix + iy * nx;
            const int rm = mm(iy) * nx + ix, rp = pp(iy, ny) * nx + ix;
            const int xl = mm(ix) - ix, xr = pp(ix + V - 1, nx) - ix;   // offsets of the cells beside the segment
            const R* hp = S.f[HH];
            CV hh, hm, hq, sig;
            hh.load(hp + i); hm.load(hp + rm); hq.load(hp + rp);
            sig.load(S.tmp[T_SIG] + i);   // sigma / sinh(2 kh), from the dispersion pass
            const R hl = ld(hp + i + xl), hr = ld(hp + i + xr);
            // face speeds times dt / dx: without wave-current interaction the
            // current terms of the face speed are exactly zero
            const R h = (R)0.5f * kxy;
#pragma unroll
            for (int n = 0; n < NFLD; n++) {
                const R* cgp = (NFLD == 2 ? n == 0 : isE) ? S.f[CG] : S.f[CC_];   // the field's propagation speed
                CV cg, gm, gq;
                cg.load(cgp + i); gm.load(cgp + rm); gq.load(cgp + rp);
                const R gl = ld(cgp + i + xl), gr = ld(cgp + i + xr);
#pragma unroll
                for (int j = 0; j <= V; j++)
                    f[n].kx[j] = h * ((j > 0 ? cg[j > 0 ? j - 1 : 0] : gl) + (j < V ? cg[j < V ? j : 0] : gr));
#pragma unroll
                for (int k = 0; k < NP; k++) {
                    const int a = 2 * k, b = a + 1;
                    f[n].ky[k] = PR::make(h * (cg[a] + gq[a]), h * (cg[b] + gq[b]));
                    f[n].kyn[k] = PR::make(-(h * (cg[a] + gm[a])), -(h * (cg[b] + gm[b])));
                }
            }
            const R sy = (R)(pp(iy, ny) - mm(iy)) * K.dx;
#pragma unroll
            for (int j = 0; j < V; j++) {
                // propagtheta's slope terms (cth_coef without currents)
                const R sx = (R)(pp(ix + j, nx) - mm(ix + j)) * K.dx;
                const R dhdx = ((j < V - 1 ? hh[j + 1 < V ? j + 1 : j] : hr) - (j > 0 ? hh[j > 0 ? j - 1 : 0] : hl)) / sx;
                const R dhdy = (hq[j] - hm[j]) / sy;
                cP.set(j, sig[j] * dhdx);
                cQ.set(j, -(sig[j] * dhdy));
            }
            ctheta(c0, sCS2[0].c, sCS2[0].s);
            const int t1 = nt > 1 ? 1 : 0;
            ctheta(cp, sCS2[t1].c, sCS2[t1].s);
        }
        // planes t, t+1, t+2 of the window: their buffers' tile offsets; the
        // buffer and parity of the plane waited for next
        int wb = 0, wpar = 0;
        auto wait_next = [&](int p) {
            ok = ok && tm_wait(su32(&mbar[wb]), (unsigned)wpar);
            if (edge) fixup(p, wb);
            const int o = wb * PL + sOff[p];
            if (++wb == TM_NB) { wb = 0; wpar ^= 1; }
            return o;
        };
        int o2 = wait_next(0), o3 = o2, o4;
        if (nt > 1) o3 = wait_next(1);
        int ib = 0;   // buffer of plane t - 1
        CV e1[NFLD], esum, cabs;
#pragma unroll
        for (int n = 0; n < NFLD; n++) e1[n].fill((R)0);
        esum.fill((R)0); cabs.fill((R)0);
#pragma unroll 1
        for (int t = 0; t < nt; t++) {
            o4 = t + 2 < nt ? wait_next(t + 2) : o3;
            __syncthreads();   // fixups visible; plane t-1 read by all
            // the next plane into plane t-1's buffer.  A copy that never lands
            // leaves its waiters with !ok (they poll no further), the elected
            // thread among them, which then issues no more; nothing is stored
            // from such a block (the check after the loop).
            if (tid == 0 && ok && t >= 1 && t - 1 + TM_NB < nt) issue(t - 1 + TM_NB, ib);
            if (t >= 1 && ++ib == TM_NB) ib = 0;
            if (active) {
                const Dir2<R> d = sCS2[t];
                const R ct = d.c, st = d.s;
                const P ctn = pair1<R>(-ct), stn = pair1<R>(-st), kn = pair1<R>(-kth);
                const bool last = t == nt - 1;
                P cb[NP];
                bool px[NP], py[NP];
#pragma unroll
                for (int k = 0; k < NP; k++) {
                    // the upper theta face's speed (0 at the last bin: no flux)
                    cb[k] = PR::mul(pair1<R>(last ? (R)0 : (R)0.5f), PR::add(c0.p[k], cp.p[k]));
                    px[k] = cb[k].x > (R)0;
                    py[k] = cb[k].y > (R)0;
                }
#pragma unroll
                for (int n = 0; n < NFLD; n++) {
                    const R* q = tX[n] + o2;
                    CV e2, e3, e4, fx, fy, A;
                    e2.load(q);
                    e3.load(tX[n] + o3);
                    e4.load(tX[n] + o4);
                    if (t == 0) e1[n] = e2;
                    using T_ = std::true_type;
                    using F_ = std::false_type;
                    auto xy = [&](auto ax, auto ay) {
                        xy_flux<R, V, decltype(ax)::value, decltype(ay)::value>(q, e2, f[n], fx, fy);
                    };
                    // the upwind side of the bin (the sign of cos and sin is the
                    // same for every cell of the bin)
                    if (ct > (R)0) {
                        if (st > (R)0) xy(T_{}, T_{}); else xy(T_{}, F_{});
                    } else {
                        if (st > (R)0) xy(F_{}, T_{}); else xy(F_{}, F_{});
                    }
#pragma unroll
                    for (int k = 0; k < NP; k++) {
                        // theta flux: upper face computed here, lower face carried from bin t-1
                        const P a = PR::make(px[k] ? e2.p[k].x : e3.p[k].x, py[k] ? e2.p[k].y : e3.p[k].y);
                        const P b = PR::make(px[k] ? e1[n].p[k].x : e4.p[k].x, py[k] ? e1[n].p[k].y : e4.p[k].y);
                        const P fup = PR::mul(cb[k], upw2<R>(a, b));
                        const P ft = PR::add(fup, f[n].fdn[k]);
                        f[n].fdn[k] = PR::mul(fup, pair1<R>((R)-1));
                        A.p[k] = PR::add(e2.p[k], PR::fma(ctn, fx.p[k], PR::fma(stn, fy.p[k], PR::mul(ft, kn))));
                    }
                    A.store(sX[n] + t * 256);
                    if (n == 0 && isE) {
#pragma unroll
                        for (int k = 0; k < NP; k++) {
                            cabs.p[k].x = DM<R>::fmax(cabs.p[k].x, DM<R>::fabs(c0.p[k].x));
                            cabs.p[k].y = DM<R>::fmax(cabs.p[k].y, DM<R>::fabs(c0.p[k].y));
                            esum.p[k] = PR::add(esum.p[k],
                                                PR::make(DM<R>::fmax(A.p[k].x, (R)0), DM<R>::fmax(A.p[k].y, (R)0)));
                        }
                    }
                    e1[n] = e2;
                }
                c0 = cp;
                const Dir2<R> d2 = sCS2[t + 2 < nt ? t + 2 : nt - 1];
                ctheta(cp, d2.c, d2.s);
            }
            o2 = o3; o3 = o4;
        }
        if (__syncthreads_or(!ok)) {   // a copy never completed: record, halt, let the copies in flight land (bounded), leave
            if (tid == 0) {
                atomicExch(&clk->status, XBG_ERR_TIMEOUT);
                atomicExch(&clk->halt, 1);
                for (int p = max(issued - TM_NB, 0); p < issued; p++)   // the last plane issued into each buffer
                    tm_wait(su32(&mbar[p % TM_NB]), (unsigned)(p / TM_NB) & 1u);
            }
            __syncthreads();
            return;
        }
        if (isE && active) {
            esum.store(sSum + cid);
#pragma unroll
            for (int j = 0; j < V; j++)   // WAVEDT (Wave_kernel.cu:232-249)
                dtw = DM<R>::fmin(dtw, DM<R>::fmin(K.cfl * dth / cabs[j], (R)9999999.9f));
        }
        __syncthreads();
    }
    // ---- phase 2
    const int cid = tid * W, ix = bx0 + cid % WT_X, iy = by0 + cid / WT_X;
    dtw = DM<R>::fmin(dtw, wave_phase2<R, ROLLER, W>(S, K, bx0, ix, iy, sA + cid, sR + cid, sSum + cid, sMom, sCS2, sg,
                                                     dtf, rro, S.ee[par], S.rr[par]));
    block_min_store<R>(dtw, S.part_wave + bix + biy * ((K.nx + 31) / 32));
}
// Threads and cells.  FP32 with the roller: two cells and both fields per thread
// (128 threads, 109 registers, four blocks per SM by shared memory at 18 bins);
// four cells of one field on as many threads take 306 against 285 us at
// 2048 x 1024, four cells of both on 64 threads leave too few warps (332 us).
// FP64: two cells (16-byte loads at most) of one field on 256 threads (66
// against 74 us at 512 x 256 for both fields on 128).  Without the roller a
// thread has four (FP64: two) cells.
// Blocks per SM: FP64 without the roller has 128 threads, and with two blocks
// (190 registers) an SM had eight warps; with three (155 registers) the pass takes
// 101 against 128 us at 1024 x 512 x 4 bins and 179 against 223 at 18 (one cell per
// thread: 107 and 231), ten ragged domains of 8 bins 739 against 842 (860).  Four
// (128 registers) are faster still up to 18 bins (93 and 169 us) and slower at 24
// and more (224 against 212, 344 against 320).
template <class R, bool ROLLER> constexpr bool wave_split = ROLLER && sizeof(R) == 8;
template <class R, bool ROLLER> constexpr int wave_v = sizeof(R) == 8 || ROLLER ? 2 : 4;
template <class R, bool ROLLER>
constexpr int wave_threads = (wave_split<R, ROLLER> ? 512 : 256) / wave_v<R, ROLLER>;
template <class R, bool ROLLER> constexpr int wave_min_blocks = sizeof(R) == 4 ? 4 : (ROLLER ? 2 : 3);
template <class R, bool ROLLER>
__global__ void __launch_bounds__(wave_threads<R, ROLLER>, wave_min_blocks<R, ROLLER>)
    k_wave_tma(Dev<R> S, Konst<R> K, const __grid_constant__ WaveMaps M) {
    b_wave_tma<R, ROLLER, wave_v<R, ROLLER>, wave_split<R, ROLLER>>(S, K, M, blockIdx.x, blockIdx.y);
}
// every scenario of a batch: its tensor maps from a device array (written
// by the host before the first launch), one per scenario
template <class R, bool ROLLER>
__global__ void __launch_bounds__(wave_threads<R, ROLLER>, wave_min_blocks<R, ROLLER>)
    kb_wave_tma(BatchTab<R> T, const WaveMaps* __restrict__ maps, const int2* items, int n) {
    batch_items<R>(T, items, n, [&](const Dev<R>& S, const Konst<R>& K, const BatchAux& A, int bx, int by) {
        b_wave_tma<R, ROLLER, wave_v<R, ROLLER>, wave_split<R, ROLLER>>(S, K, maps[A.scen], bx, by);
    });
}

// Tensor maps of the TMA rows pass: ee and rr of both plane sets as 3-D
// arrays [nt][ny][nx], loaded in 36 x 10 x 1 boxes.  Encoded with the driver's
// cuTensorMapEncodeTiled (fetched through the runtime).
template <class R>
int wave_maps_make(const Dev<R>& S, const Konst<R>& K, WaveMaps* M) {
    if (K.nx % 4 != 0 || K.nt > 256) return 1;
    static PFN_cuTensorMapEncodeTiled_v12000 enc = nullptr;
    if (!enc) {
        cudaDriverEntryPointQueryResult q;
        void* fn = nullptr;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &fn, cudaEnableDefault, &q) != cudaSuccess ||
            q != cudaDriverEntryPointSuccess || !fn)
            return 1;
        enc = (PFN_cuTensorMapEncodeTiled_v12000)fn;
    }
    const CUtensorMapDataType dt = sizeof(R) == 4 ? CU_TENSOR_MAP_DATA_TYPE_FLOAT32 : CU_TENSOR_MAP_DATA_TYPE_FLOAT64;
    const cuuint64_t es = sizeof(R);
    const cuuint32_t one[3] = {1, 1, 1};
    auto make = [&](CUtensorMap* m, const R* base, int rows, cuuint32_t bx, cuuint32_t by, cuuint32_t bz) {
        const cuuint64_t dims[3] = {(cuuint64_t)K.nx, (cuuint64_t)rows, (cuuint64_t)K.nt};
        const cuuint64_t strides[2] = {(cuuint64_t)K.nx * es, (cuuint64_t)K.nx * K.ny * es};
        const cuuint32_t box[3] = {bx, by, bz};
        return enc(m, dt, 3, (void*)base, dims, strides, box, one, CU_TENSOR_MAP_INTERLEAVE_NONE,
                   CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    };
    for (int k = 0; k < 2; k++) {
        if (make(&M->ld_e[k], S.ee[k], K.ny, TM_X, TM_Y, 1) != CUDA_SUCCESS ||
            make(&M->ld_r[k], S.rr[k], K.ny, TM_X, TM_Y, 1) != CUDA_SUCCESS)
            return 1;
    }
    return 0;
}

// wavforce (wave_CPU.cpp:1164-1238) from the radiation stresses around a
// cell (r: the right neighbour, t: the upper, b: the lower, l: the left, tr,
// br, tl: the diagonals), before the boundary copies
template <class R>
__device__ __forceinline__ void force_of(R dxf, R Sxxi, R Sxxr, R Sxyt, R Sxytr, R Sxyb, R Sxybr, R Syyi, R Syyt,
                                         R Sxyr, R Sxyl, R Sxytl, R& Fx, R& Fy) {
    Fx = (R)-1 * (Sxxr - Sxxi) / dxf - (R)0.5f * (Sxyt + Sxytr - Sxyb - Sxybr) / ((R)2.0f * dxf);
    Fy = (R)-1 * (Syyt - Syyi) / dxf - (R)0.5f * (Sxyr + Sxytr - Sxyl - Sxytl) / ((R)2.0f * dxf);
}
// ... at cell (ix, iy)
template <class R>
__device__ __forceinline__ void force_raw(const Dev<R>& S, const Konst<R>& K, int ix, int iy, R& Fx, R& Fy) {
    const int nx = K.nx, ny = K.ny;
    const R* Sxx = S.tmp[T_SXX]; const R* Sxy = S.tmp[T_SXY]; const R* Syy = S.tmp[T_SYY];
    int xm = mm(ix), xp = pp(ix, nx), ym = mm(iy), yp = pp(iy, ny);
    int i = ix + iy * nx;
    force_of(K.dx, ld(Sxx + i), ld(Sxx + xp + iy * nx), ld(Sxy + ix + yp * nx), ld(Sxy + xp + yp * nx),
             ld(Sxy + ix + ym * nx), ld(Sxy + xp + ym * nx), ld(Syy + i), ld(Syy + ix + yp * nx), ld(Sxy + xp + iy * nx),
             ld(Sxy + xm + iy * nx), ld(Sxy + xm + yp * nx), Fx, Fy);
}

// breakerdelayCPU (wave_CPU.cpp:1333-1368) from a cell's H, k, depth, c,
// roller energy and E
template <class R>
__device__ __forceinline__ void breaker_of(const Konst<R>& K, R Trep, R Hi, R ki, R hh, R c, R Rl, R Ei, R& urms,
                                           R& ust) {
    R hmin = (R)0.2;
    R g = K.g, rho = K.rho;
    R hhi = cmax(hh, hmin);
    R ci = cmax(c, DM<R>::sqrt(hmin * g));
    R uorb = (R)(XBG_PI * (double)Hi / (double)Trep / (double)DM<R>::sinh(cmin(cmax(ki, (R)0.01f) * hhi, (R)10.0f)));
    urms = uorb / (DM<R>::sqrt((R)2.0f));
    R ustw = Ei / ci / rho / hhi;
    R ustr = (R)2.0f * Rl / ci / rho / hhi;
    ust = ustw + ustr;
}
// ... at cell j
template <class R>
__device__ __forceinline__ void breaker_raw(const Dev<R>& S, const Konst<R>& K, int j, R Trep, R& urms, R& ust) {
    breaker_of(K, Trep, ld(S.f[H] + j), ld(S.f[WK] + j), ld(S.f[HH] + j), ld(S.f[CC_] + j), ld(S.f[ROL] + j),
               ld(S.f[E] + j), urms, ust);
}

template <class R>
__device__ __forceinline__ void b_wave_force(const Dev<R>& S, const Konst<R>& K, const int bix, const int biy) {
    const Clock* clk = S.clk;
    if (wave_off(clk)) return;
    const int nx = K.nx, ny = K.ny;
    int ix = bix * blockDim.x + threadIdx.x;
    int iy = biy * blockDim.y + threadIdx.y;
    if (ix >= nx || iy >= ny) return;
    int i = ix + iy * nx;
    R Trep = (R)clk->Trep;
    R w = ld(S.f[HH] + i) > K.eps ? (R)1.0f : (R)0.0f;
    // twodimbndnoixCPU(Fx): rows only; twodimbndCPU(Fy, ust): rows then ix = 0
    int sy = iy;
    if (iy == 0) sy = pp(0, ny);
    if (iy == ny - 1) sy = mm(ny - 1);
    int fx_src_x = ix, fx_src_y = sy;
    int fy_src_x = (ix == 0) ? pp(0, nx) : ix;
    int fy_src_y = (ix == 0) ? iy : sy;
    bool rowb = (iy == 0 || iy == ny - 1);
    bool anyb = rowb || ix == 0;
    R Fx, Fy, tmp;
    force_raw(S, K, fx_src_x, fx_src_y, Fx, tmp);
    if (rowb) Fx = Fx * w;
    force_raw(S, K, fy_src_x, fy_src_y, tmp, Fy);
    if (anyb) Fy = Fy * w;
    S.f[FX][i] = Fx;
    S.f[FY][i] = Fy;
    R urms, ust, u2;
    breaker_raw(S, K, i, Trep, urms, ust);
    if (anyb) {
        breaker_raw(S, K, fy_src_x + fy_src_y * nx, Trep, u2, ust);
        ust = ust * w;
    }
    S.f[URMS][i] = urms;
    S.f[UST][i] = ust;
}
XBG_KERNELS(wave_force)

// ---------------------------------------------------------------- launchers
template <class R>
int wave_parts(const Konst<R>& K) {
    return ((K.nx + 31) / 32) * ((K.ny - 2 + 7) / 8);
}

// join: an event of a concurrent branch (the boundary kernels) that the
// rows pass waits for after the dispersion kernel; null when sequential.
// maps: the tensor maps of the TMA rows pass, or null for the thread-copied
// tiles (b_wave_fast); the TMA pass has no wave-current interaction variant.
template <class R>
int launch_wave(const Dev<R>& S, const Konst<R>& K, cudaStream_t st, Prof* pf, cudaEvent_t join,
                const WaveMaps* maps, bool wide) {
    int n = 0;
    k_disp<R><<<(S.C + 255) / 256, 256, 0, st>>>(S, K); n++;
    PMARK(pf, "k_disp");
    if (join) cudaStreamWaitEvent(st, join, 0);
    {
        dim3 b(32, 8), g((K.nx + 31) / 32, (K.ny - 2 + 7) / 8);
        if (maps && K.wci == (R)0) {
            const size_t smem = wave_tma_smem<R>(K.nt, K.roller);
            if (K.roller == 1) k_wave_tma<R, true><<<g, wave_threads<R, true>, smem, st>>>(S, K, *maps);
            else k_wave_tma<R, false><<<g, wave_threads<R, false>, smem, st>>>(S, K, *maps);
            n++;
            PMARK(pf, "k_wave_tma");
        } else {
            launch_wave_fast(S, K, g, b, wave_fast_smem<R>(K.nt), st); n++;
            PMARK(pf, "k_wave_fast");
        }
    }
    // the force pass is pointwise: 32 x 8 or (wide) 64 x 4 blocks (a row-segment
    // form measured slower: 37.0 against 32.8 us at 2048 x 1024, 94 registers)
    if (wide) k_wave_force<R><<<dim3((K.nx + 63) / 64, (K.ny + 3) / 4), dim3(64, 4), 0, st>>>(S, K);
    else k_wave_force<R><<<dim3((K.nx + 31) / 32, (K.ny + 7) / 8), dim3(32, 8), 0, st>>>(S, K);
    n++;
    PMARK(pf, "k_wave_force");
    return n;
}

// the wave kernels over every scenario of a batch (one ntheta and roller
// setting for the whole batch)
// maps: the scenarios' tensor maps (device array) for the TMA rows pass, or
// null for the thread-copied tiles
template <class R>
int launch_wave_batch(const BatchTab<R>& T, const BatchLaunch& L, int nt, int roller, int wci, cudaStream_t st,
                      Prof* pf, cudaEvent_t join, const WaveMaps* maps, bool wide) {
    kb_disp<R><<<L.grid[BS_LIN], 256, 0, st>>>(T, L.items[BS_LIN], L.n[BS_LIN]);
    PMARK(pf, "k_disp");
    if (join) cudaStreamWaitEvent(st, join, 0);
    if (maps && !wci) {
        const int g = L.grid[BS_WROWS], n = L.n[BS_WROWS];
        const int2* it = L.items[BS_WROWS];
        const size_t smem = wave_tma_smem<R>(nt, roller);
        if (roller == 1) kb_wave_tma<R, true><<<g, wave_threads<R, true>, smem, st>>>(T, maps, it, n);
        else kb_wave_tma<R, false><<<g, wave_threads<R, false>, smem, st>>>(T, maps, it, n);
        PMARK(pf, "k_wave_tma");
    } else {
        launch_wave_fast_batch(T, L, roller, wci, wave_fast_smem<R>(nt), st);
        PMARK(pf, "k_wave_fast");
    }
    const int sf = wide ? BS_WIDE : BS_TILE;
    kb_wave_force<R><<<L.grid[sf], wide ? dim3(64, 4) : dim3(32, 8), 0, st>>>(T, L.items[sf], L.n[sf]);
    PMARK(pf, "k_wave_force");
    return 3;
}
template int launch_wave_batch<float>(const BatchTab<float>&, const BatchLaunch&, int, int, int, cudaStream_t, Prof*,
                                      cudaEvent_t, const WaveMaps*, bool);
template int launch_wave_batch<double>(const BatchTab<double>&, const BatchLaunch&, int, int, int, cudaStream_t, Prof*,
                                       cudaEvent_t, const WaveMaps*, bool);

// One-time kernel attributes (dynamic shared memory above 48 KB for wide
// theta sets in FP64).
template <class R>
int wave_prepare(const Konst<R>&) {
    // the limits of the widest theta set: the attribute belongs to the kernel,
    // not to this handle, and another handle's launches rely on it too
    const int smem = (int)wave_fast_smem<R>(XBG_MAX_THETA);
    const int smem_tma = (int)wave_tma_smem<R>(XBG_MAX_THETA, 1);
    const cudaFuncAttribute a = cudaFuncAttributeMaxDynamicSharedMemorySize;
    if (cudaFuncSetAttribute(k_wave_tma<R, true>, a, smem_tma) != cudaSuccess ||
        cudaFuncSetAttribute(k_wave_tma<R, false>, a, smem_tma) != cudaSuccess ||
        cudaFuncSetAttribute(kb_wave_tma<R, true>, a, smem_tma) != cudaSuccess ||
        cudaFuncSetAttribute(kb_wave_tma<R, false>, a, smem_tma) != cudaSuccess)
        return 1;
    cudaError_t e[8] = {
        cudaFuncSetAttribute(k_wave_fast<R, true, true>, a, smem), cudaFuncSetAttribute(k_wave_fast<R, true, false>, a, smem),
        cudaFuncSetAttribute(k_wave_fast<R, false, true>, a, smem), cudaFuncSetAttribute(k_wave_fast<R, false, false>, a, smem),
        cudaFuncSetAttribute(kb_wave_fast<R, true, true>, a, smem), cudaFuncSetAttribute(kb_wave_fast<R, true, false>, a, smem),
        cudaFuncSetAttribute(kb_wave_fast<R, false, true>, a, smem), cudaFuncSetAttribute(kb_wave_fast<R, false, false>, a, smem)};
    for (auto x : e)
        if (x != cudaSuccess) return 1;
    return 0;
}
template int wave_prepare<float>(const Konst<float>&);
template int wave_prepare<double>(const Konst<double>&);

template int launch_wave<float>(const Dev<float>&, const Konst<float>&, cudaStream_t, Prof*, cudaEvent_t,
                                const WaveMaps*, bool);
template int launch_wave<double>(const Dev<double>&, const Konst<double>&, cudaStream_t, Prof*, cudaEvent_t,
                                 const WaveMaps*, bool);
template int wave_maps_make<float>(const Dev<float>&, const Konst<float>&, WaveMaps*);
template int wave_maps_make<double>(const Dev<double>&, const Konst<double>&, WaveMaps*);
template int wave_parts<float>(const Konst<float>&);
template int wave_parts<double>(const Konst<double>&);

}  // namespace xbg
