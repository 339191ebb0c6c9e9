// Per-cell part of a stage, two x-adjacent cells per thread and iteration (included by stage.cuh, beside
// the one-cell form of stage_cells, which serves the rows staged in shared memory).
//
// What bounds it: instruction issue and load latency, not DRAM. One packed x element holds exactly the two
// cells, so the demag field arrives and the new M leaves as one shared-memory access per component, every
// row is read and written as 8-byte (FP64 16-byte) pairs, and the arithmetic is packed: half the loads,
// addresses and issue slots per cell. The stencil sums the neighbours' differences from the cell, which are exact
// where M varies little, and a boundary cell takes the Neumann term -+ h bd in place of the missing one (the
// one-sided differences of axis_stencil), so no second copy of it is needed and lanes at the x ends do not diverge.
// A sum of two neighbours minus 2 m rounds at the size of M: relative FP32 error of the exchange field of a
// smooth 200 x 150 film 1.0e-4 that way, 6e-8 with differences (97 x 61 x 23 box 1.1e-5, 7e-8).
// Measured (stage launch of the 512 x 512 x 16 film, radix-16 x transforms): 198 -> 188 us in FP32, 407 -> 366 us in
// FP64 (380 with the stencil in differences); 128 x 64 film 15.2 -> 13.4 us. Differences taken separately for the two
// cells, with the one between them formed once, cost FP32 nothing (168.6 us with butterfly pairs; all by pairs 171.4,
// sums 169.2); in FP64 every form of them takes 379 to 381 us, the sums only inside too.
//
// ODD: nx may be odd, so rows start on any value (pairs are read and written as two scalars) and the last
// pair of a row may have one cell: its second lane repeats the first and is never stored (zero in the x line).
#pragma once
#include "pair.cuh"

// pair access of a row: one vector access, or two scalars for odd nx (o2: offset of the second lane, 1, or
// 0 where the pair has one cell; two: whether it has two)
template <bool ODD, typename T> __device__ __forceinline__ cpx<T> prow_ld(const T *p, int o2)
{
    if constexpr (ODD) return mk<T>(p[0], p[o2]);
    else return pk_ld<T>(p);
}
template <bool ODD, typename T> __device__ __forceinline__ void prow_st(T *p, cpx<T> v, bool two)
{
    if constexpr (ODD) {
        p[0] = v.x;
        if (two) p[1] = v.y;
    } else {
        pk_st<T>(p, v);
    }
}

// sum[c] += sum_{i < NEV} cev[i] * ev_i[c], i ascending
template <int NEV, bool ODD, typename T>
__device__ __forceinline__ void ev_acc2(const StageArgs<T> &a, const T *cev, long long cell, int o2, cpx<T> sum[3])
{
    cpx<T> e[NEV][3];
#pragma unroll
    for (int i = 0; i < NEV; i++)
#pragma unroll
        for (int c = 0; c < 3; c++) e[i][c] = prow_ld<ODD>(a.ev[i] + c * a.n + cell, o2);
#pragma unroll
    for (int i = 0; i < NEV; i++)
#pragma unroll
        for (int c = 0; c < 3; c++) sum[c] = pk_fma(pk_bc<T>(cev[i]), e[i][c], sum[c]);
}

// the RKDP54 error estimate of one cell (component values of the pair's lane k), as the one-cell form
template <typename T>
__device__ __forceinline__ void lte_cell(const StageArgs<T> &a, long long cell, const T m[3], const T rhs[3], T Ms, double dT,
                                         double &lmax)
{
    const long long n = a.n;
    double d2 = 0.0, m2 = 0.0, sb[3] = {0, 0, 0}, sa[3] = {0, 0, 0}, mb[3];
#pragma unroll
    for (int c = 0; c < 3; c++) mb[c] = (double)a.Mbase[c * n + cell];
    for (int i = 0; i < a.nev; i++) {
        const T *e = a.ev[i] + cell;
#pragma unroll
        for (int c = 0; c < 3; c++) {
            const double v = (double)e[c * n];
            sb[c] += a.cev[i] * v;
            if (a.lte_embedded) sa[c] += a.cev5[i] * v;
        }
    }
    if (a.lte_embedded) {
        double m5[3], n5 = 0.0;
#pragma unroll
        for (int c = 0; c < 3; c++) {
            m5[c] = mb[c] + dT * sa[c];
            n5 += m5[c] * m5[c];
        }
        const double f = (double)Ms / sqrt(n5);
#pragma unroll
        for (int c = 0; c < 3; c++) {
            const double d = m5[c] * f - (mb[c] + dT * (sb[c] + a.crhs * (double)rhs[c]));
            d2 += d * d;
            m2 += (double)m[c] * (double)m[c];
        }
    } else {
#pragma unroll
        for (int c = 0; c < 3; c++) {
            const double d = (double)m[c] - (mb[c] + dT * (sb[c] + a.crhs * (double)rhs[c]));
            d2 += d * d;
            m2 += (double)m[c] * (double)m[c];
        }
    }
    if (!isfinite(m[0] + m[1] + m[2] + rhs[0] + rhs[1] + rhs[2])) atomicOr(&a.st->error, BM_ERR_NONFINITE);
    double l = sqrt(d2) / sqrt(m2);
    if (!(l <= 1e300)) l = 1e300;
    if (l > lmax) lmax = l;
}

// SPEC 1: the plain stage update (stage_plain on the host): mode, the outputs written and the demag
// and exchange terms are compile-time, so their run-time checks leave the per-cell loop; SPEC 2 the
// plain RKDP54 error estimate (stage_lte_plain), SPEC 3 the plain advance of the base state
// (stage_adv_plain), likewise
template <typename T, int SPEC, bool ODD, typename AddrF>
__device__ __forceinline__ void stage_pairs(const StageArgs<T> &a, cpx<T> *sm, int LSP, AddrF addr, int r0, double &lmax)
{
    constexpr bool PS = SPEC == 1, PL = SPEC == 2, PA = SPEC == 3, SP = SPEC != 0;
    const int nx = a.nx, ny = a.ny, nz = a.nz, rpb = a.rpb, half = ODD ? (nx + 1) >> 1 : nx >> 1;
    const int nrows = ny * nz;
    const int tid = threadIdx.x, nt = blockDim.x;
    const long long n = a.n;
    const int mode = PS ? BM_MODE_STAGE : PL ? BM_MODE_LTE : PA ? BM_MODE_UPDATE : a.mode;
    const T *Hd = SP ? nullptr : a.Hd;
    T *Hsave = SP ? nullptr : a.Hsave;
    T *Ysave = SP ? nullptr : a.Ysave;
    T *copy_to = (PS || PL) ? nullptr : a.copy_to;
    const bool has_ev_out = (PS || PL) || (!PA && a.ev_out), has_Mout = (PS || PA) || (!PL && a.Mout);
    const bool do_xfwd = (PS || PA) || (!PL && a.do_xfwd);
    const bool fields = (PS || PL) || (!PA && mode != BM_MODE_UPDATE);
    const bool demag = (PS || PL) || (!PA && fields && (a.modules & BM_MOD_DEMAG));
    const double dT = a.st ? *((volatile double *)&a.st->dT) : 0.0;
    T Ha[3] = {0, 0, 0};
    if (fields && (a.modules & BM_MOD_ZEEMAN) && a.Ha && a.nHa > 0) {
        double tm = a.st ? *((volatile double *)&a.st->stagetime) : 0.0;
        int hi = 0;
        if (a.nHa > 1 && a.Ha_tspan > 0.0) {
            // one FP64 division per warp, broadcast (every launch runs whole warps)
            if ((threadIdx.x & 31) == 0) {
                hi = (int)floor(tm / a.Ha_tspan * a.nHa);
                hi = hi < 0 ? 0 : (hi >= a.nHa ? a.nHa - 1 : hi);
            }
            hi = __shfl_sync(0xffffffffu, hi, 0);
        }
        Ha[0] = (T)a.Ha[3 * hi]; Ha[1] = (T)a.Ha[3 * hi + 1]; Ha[2] = (T)a.Ha[3 * hi + 2];
    }
    const bool exch = (PS || PL) || (!PA && fields && (a.modules & (BM_MOD_EXCH | BM_MOD_IDMI)));
    const bool idmi = (a.modules & BM_MOD_IDMI) != 0;
    const bool zflat = (nz == 1);
    const int dg = (a.grel != (T)0) ? stage_diag_active(a) : 0;
    unsigned long long *dslot = stage_diag_slots();
    if (stage_diag_active(a)) {
        if (tid == 0) { dslot[0] = 0ull; dslot[1] = 0ull; }
        __syncthreads();
    }
    const int nev = a.nev;
    T cev[6];
#pragma unroll
    for (int i = 0; i < 6; i++) cev[i] = (T)(a.cev[i] * dT);
    const T crhs = (T)(a.crhs * dT);
    const int cs = rpb * LSP;   // elements between the component lines of one row
    // (r, p) of pair index r * half + p, advanced by nt per iteration without divisions
    int dr = 0, dp = nt, r = 0, p = tid;
    if (nt > half) {
        dr = nt / half; dp = nt - dr * half;
        r = tid / half; p = tid - r * half;
    }
    int yrow = -1, y = 0, z = 0;
    for (; r < rpb; p += dp, r += dr) {
        if (p >= half) { p -= half; r++; if (r >= rpb) break; }
        const int row = r0 + r;
        if (row >= nrows) break;
        if (row != yrow) { yrow = row; z = row / ny; y = row - z * ny; }
        const long long cell = (long long)row * nx + 2 * p;
        cpx<T> *sp = &sm[r * LSP + addr(p)];
        const T *Mc = a.Min + cell;
        const bool two = !ODD || 2 * p + 1 < nx;
        const int o2 = two ? 1 : 0;
        cpx<T> m[3];
#pragma unroll
        for (int c = 0; c < 3; c++) m[c] = prow_ld<ODD>(Mc + c * n, o2);
        const cpx<T> Ms = a.Ms_map ? prow_ld<ODD>(a.Ms_map + cell, o2) : pk_bc<T>(a.Ms);
        const cpx<T> iMs = a.Ms_map ? mk<T>((T)1 / Ms.x, (T)1 / Ms.y) : pk_bc<T>(a.iMs);
        cpx<T> rhs[3] = {pk_bc<T>(0), pk_bc<T>(0), pk_bc<T>(0)};
        if (fields) {
            cpx<T> H[3] = {pk_bc<T>(Ha[0]), pk_bc<T>(Ha[1]), pk_bc<T>(Ha[2])};
            if (demag) {
#pragma unroll
                for (int c = 0; c < 3; c++) H[c] = pk_fma(pk_bc<T>(a.scale), sp[c * cs], H[c]);
            }
            if (Hd) {
#pragma unroll
                for (int c = 0; c < 3; c++) H[c] = pk_add(H[c], prow_ld<ODD>(Hd + c * n + cell, o2));
            }
            if (exch) {
                // a missing neighbour is the far side times the axis' sign (periodic) or leaves the boundary term
                // -+ h bd (bd = 0 on a one-cell axis) in place of its difference
                const bool px = a.pbc[0] && nx > 1, py = a.pbc[1] && ny > 1, pz = a.pbc[2] && nz > 1;
                const bool ex0 = p == 0, ex1 = p == half - 1, ey0 = y == 0, ey1 = y == ny - 1, ez0 = z == 0, ez1 = z == nz - 1;
                // the left neighbour of the pair's first cell, the right one of its last
                const int oxm = ex0 ? (px ? nx - 1 : 0) : -1, oxp = ex1 ? (px ? (two ? 2 : 1) - nx : 0) : 2;
                const long long wy = (long long)(ny - 1) * nx, nxy = (long long)nx * ny, wz = (long long)(nz - 1) * nxy;
                const long long oym = ey0 ? (py ? wy : 0) : -nx, oyp = ey1 ? (py ? -wy : 0) : nx;
                const long long ozm = ez0 ? (pz ? wz : 0) : -nxy, ozp = ez1 ? (pz ? -wz : 0) : nxy;
                const T rr = idmi ? a.rrD : (T)0;
                const T bhx = nx > 1 ? rr * a.hh[0] : (T)0, bhy = ny > 1 ? rr * a.hh[1] : (T)0;
                const cpx<T> iMs2 = pk_mul(iMs, iMs);
                const cpx<T> Ac = pk_mul(pk_bc<T>(a.exA), iMs2);
                cpx<T> gx[3], gy[3];
#pragma unroll
                for (int c = 0; c < 3; c++) {
                    const T *q = Mc + c * n;
                    T xl = q[oxm], xr = q[oxp];
                    cpx<T> ym = prow_ld<ODD>(q + oym, o2), yp = prow_ld<ODD>(q + oyp, o2);
                    if (ex0 && px) xl *= (T)a.pbc[0];
                    if (ex1 && px) xr *= (T)a.pbc[0];
                    if (ey0 && py) ym = pk_mul(pk_bc<T>((T)a.pbc[1]), ym);
                    if (ey1 && py) yp = pk_mul(pk_bc<T>((T)a.pbc[1]), yp);
                    // the neighbours minus the cell; at an open side the boundary term -+ h bd instead, with h bd
                    // x (rr m2, 0, -rr m0), y (0, rr m2, -rr m1)
                    T dl = xl - m[c].x, dr = xr - m[c].y;
                    const T e = m[c].y - m[c].x;   // between the two cells; zero where there is one
                    if (ex0 && !px) dl = c == 0 ? -bhx * m[2].x : c == 1 ? (T)0 : bhx * m[0].x;
                    if (ex1 && !px) dr = c == 0 ? bhx * m[2].y : c == 1 ? (T)0 : -bhx * m[0].y;
                    const cpx<T> dxm = mk<T>(dl, -e), dxp = mk<T>(two ? e : dr, dr);
                    cpx<T> dym = pk_sub(ym, m[c]), dyp = pk_sub(yp, m[c]);
                    const cpx<T> b = c == 1 ? m[2] : m[1];
                    const T sb = c == 0 ? (T)0 : c == 1 ? bhy : -bhy;
                    if (ey0 && !py) dym = pk_mul(pk_bc<T>(-sb), b);
                    if (ey1 && !py) dyp = pk_mul(pk_bc<T>(sb), b);
                    cpx<T> lap = pk_mul(pk_add(dxp, dxm), pk_bc<T>(a.ih2[0]));
                    lap = pk_fma(pk_add(dyp, dym), pk_bc<T>(a.ih2[1]), lap);
                    if (!zflat) {
                        // no boundary term along z: the missing neighbour is the cell itself
                        cpx<T> zm = prow_ld<ODD>(q + ozm, o2), zp = prow_ld<ODD>(q + ozp, o2);
                        if (pz) {
                            if (ez0) zm = pk_mul(pk_bc<T>((T)a.pbc[2]), zm);
                            if (ez1) zp = pk_mul(pk_bc<T>((T)a.pbc[2]), zp);
                        }
                        lap = pk_fma(pk_add(pk_sub(zp, m[c]), pk_sub(zm, m[c])), pk_bc<T>(a.ih2[2]), lap);
                    }
                    H[c] = pk_fma(Ac, lap, H[c]);
                    if (idmi) {
                        if (c != 1) gx[c] = pk_sub(dxp, dxm);
                        if (c != 0) gy[c] = pk_sub(dyp, dym);
                    }
                }
                if (idmi) {
                    const cpx<T> Dc = pk_mul(pk_bc<T>(a.exD * (T)0.5), iMs2);
                    const cpx<T> ihx = pk_bc<T>(a.ih[0]), ihy = pk_bc<T>(ny > 1 ? a.ih[1] : (T)0);
                    H[0] = pk_fma(Dc, pk_mul(gx[2], ihx), H[0]);
                    H[1] = pk_fma(Dc, pk_mul(gy[2], ihy), H[1]);
                    H[2] = pk_sub(H[2], pk_mul(Dc, pk_fma(gx[0], ihx, pk_mul(gy[1], ihy))));
                }
            }
            if (a.modules & BM_MOD_ANIUNI) {
                const cpx<T> K1 = a.K1_map ? prow_ld<ODD>(a.K1_map + cell, o2) : pk_bc<T>(a.K1);
                const cpx<T> e0 = pk_bc<T>(a.ea[0]), e1 = pk_bc<T>(a.ea[1]), e2 = pk_bc<T>(a.ea[2]);
                const cpx<T> d = pk_mul(pk_fma(m[2], e2, pk_fma(m[1], e1, pk_mul(m[0], e0))), iMs);
                const cpx<T> k2 = pk_bc<T>(2 * a.K2);
                const cpx<T> w = pk_fma(k2, pk_fma(pk_neg(d), d, pk_bc<T>(1)), K1);
                const cpx<T> s = pk_mul(pk_mul(pk_mul(pk_bc<T>(a.two_mu0), iMs), d), w);
                H[0] = pk_fma(s, e0, H[0]);
                H[1] = pk_fma(s, e1, H[1]);
                H[2] = pk_fma(s, e2, H[2]);
            }
            if (mode == BM_MODE_HEFF) {
#pragma unroll
                for (int c = 0; c < 3; c++) prow_st<ODD>(a.Hout + c * n + cell, H[c], two);
                continue;
            }
            if (Hsave) {
#pragma unroll
                for (int c = 0; c < 3; c++) prow_st<ODD>(Hsave + c * n + cell, H[c], two);
            }
            cpx<T> x[3], nm[3] = {pk_neg(m[0]), pk_neg(m[1]), pk_neg(m[2])};
            x[0] = pk_fma(nm[2], H[1], pk_mul(m[1], H[2]));
            x[1] = pk_fma(nm[0], H[2], pk_mul(m[2], H[0]));
            x[2] = pk_fma(nm[1], H[0], pk_mul(m[0], H[1]));
            if (dg & BM_DIAG_MXH) {
                // |M x Heff| / |M|^2, in the stage's precision as the one-cell form
                const cpx<T> x2 = pk_fma(x[2], x[2], pk_fma(x[1], x[1], pk_mul(x[0], x[0])));
                const cpx<T> mm = pk_fma(m[2], m[2], pk_fma(m[1], m[1], pk_mul(m[0], m[0])));
                const double v0 = (double)(sqrt(x2.x) / mm.x), v1 = (double)(sqrt(x2.y) / mm.y);
                atomicMax(&dslot[0], (unsigned long long)__double_as_longlong(v0));
                if (two) atomicMax(&dslot[0], (unsigned long long)__double_as_longlong(v1));
            }
            const cpx<T> al = pk_mul(pk_bc<T>(a.alpha), iMs), pre = pk_bc<T>(a.llg_pre);
            rhs[0] = pk_mul(pre, pk_fma(al, pk_fma(nm[2], x[1], pk_mul(m[1], x[2])), x[0]));
            rhs[1] = pk_mul(pre, pk_fma(al, pk_fma(nm[0], x[2], pk_mul(m[2], x[0])), x[1]));
            rhs[2] = pk_mul(pre, pk_fma(al, pk_fma(nm[1], x[0], pk_mul(m[0], x[1])), x[2]));
        }
        if (mode == BM_MODE_LTE) {
            const T ma[3] = {m[0].x, m[1].x, m[2].x}, mb[3] = {m[0].y, m[1].y, m[2].y};
            const T ra[3] = {rhs[0].x, rhs[1].x, rhs[2].x}, rb[3] = {rhs[0].y, rhs[1].y, rhs[2].y};
            lte_cell<T>(a, cell, ma, ra, Ms.x, dT, lmax);
            if (two) lte_cell<T>(a, cell + 1, mb, rb, Ms.y, dT, lmax);
#pragma unroll
            for (int c = 0; c < 3; c++) prow_st<ODD>(a.ev_out + c * n + cell, rhs[c], two);
            continue;
        }
        cpx<T> mn[3];
        {
            cpx<T> sum[3];
#pragma unroll
            for (int c = 0; c < 3; c++) sum[c] = pk_mul(pk_bc<T>(crhs), rhs[c]);
            switch (nev) {   // block-uniform: unrolled sums without predicated loads
            case 6: ev_acc2<6, ODD>(a, cev, cell, o2, sum); break;
            case 5: ev_acc2<5, ODD>(a, cev, cell, o2, sum); break;
            case 4: ev_acc2<4, ODD>(a, cev, cell, o2, sum); break;
            case 3: ev_acc2<3, ODD>(a, cev, cell, o2, sum); break;
            case 2: ev_acc2<2, ODD>(a, cev, cell, o2, sum); break;
            case 1: ev_acc2<1, ODD>(a, cev, cell, o2, sum); break;
            default: break;
            }
#pragma unroll
            for (int c = 0; c < 3; c++) mn[c] = pk_add(prow_ld<ODD>(a.Mbase + c * n + cell, o2), sum[c]);
        }
        if (Ysave) {
#pragma unroll
            for (int c = 0; c < 3; c++) prow_st<ODD>(Ysave + c * n + cell, mn[c], two);
        }
        if (!PA && a.renorm) {
            const cpx<T> q = pk_fma(mn[2], mn[2], pk_fma(mn[1], mn[1], pk_mul(mn[0], mn[0])));
            const cpx<T> f = mk<T>(Ms.x / sqrt(q.x), Ms.y / sqrt(q.y));
#pragma unroll
            for (int c = 0; c < 3; c++) mn[c] = pk_mul(mn[c], f);
            // the step's new state must be finite (the sum is non-finite if any component is)
            const cpx<T> s = pk_add(pk_add(mn[0], mn[1]), mn[2]);
            if (!(isfinite(s.x) && (!two || isfinite(s.y))) && a.st) atomicOr(&a.st->error, BM_ERR_NONFINITE);
        }
        if (dg & BM_DIAG_DMDT) {
            // |M - M_start| / (dT GAMMA |M|^2) after the last stage; the base is read before M is written
            cpx<T> d2 = pk_bc<T>(0), mm = pk_bc<T>(0);
#pragma unroll
            for (int c = 0; c < 3; c++) {
                const cpx<T> d = pk_sub(mn[c], prow_ld<ODD>(a.Mbase + c * n + cell, o2));
                d2 = pk_fma(d, d, d2);
                mm = pk_fma(mn[c], mn[c], mm);
            }
            const double v0 = (double)sqrt(d2.x) / (dT * BM_GAMMA * (double)mm.x);
            const double v1 = (double)sqrt(d2.y) / (dT * BM_GAMMA * (double)mm.y);
            atomicMax(&dslot[1], (unsigned long long)__double_as_longlong(v0));
            if (two) atomicMax(&dslot[1], (unsigned long long)__double_as_longlong(v1));
        }
#pragma unroll
        for (int c = 0; c < 3; c++) {
            if (has_ev_out) prow_st<ODD>(a.ev_out + c * n + cell, rhs[c], two);
            if (copy_to) prow_st<ODD>(copy_to + c * n + cell, m[c], two);
            if (has_Mout) prow_st<ODD>(a.Mout + c * n + cell, mn[c], two);
            if (do_xfwd) sp[c * cs] = two ? mn[c] : mk<T>(mn[c].x, (T)0);
        }
    }
}
