// FP64 sweep of the collapsed sum in blocks of four terms, the columns taken in pairs.
//
// Two digits u, v of radix 2 and multiplicity 1 (two output modes chosen once each) are taken out of the Gray
// walk; every walked term then stands for the four sign choices of u and v around the column sums s at
// u = v = 0.  With du = -2 B[u], dv = -2 B[v] a column's sum at digit values (x, y) is s + x du + y dv, so
// for a pair of columns a, b
//
//   product   q(0,0) = s_a s_b,  q(1,0) = q(0,0) + L_u,  q(1,1) = q(1,0) + L_v + C,  q(0,1) = q(1,1) - L_u - C
//             L_u = s_a du_b + s_b du_a + du_a du_b  (L_v alike),  C = du_a dv_b + du_b dv_a
//   cofactor  sum_xy w_xy Y_xy (s_b + x du_b + y dv_b) = S s_b + du_b X_u + dv_b X_v
//             Y = the product of every other pair, S = sum w Y, X_u / X_v = the terms with x = 1 / y = 1
//
// L_u and L_v are affine in the column sums, so they are walked by Gray updates like the sums themselves (the
// table G holds their steps); S multiplies the column sums once per block, X_u and X_v only once per sweep.
// Per pair and term that is 5 FP64 instructions for the products, 12 for the all-but-one products over the
// pairs (prefix, suffix, accumulation) and 4 for the rest: 21, against 28 for two columns taken one by one.
// Bound by the FP64 pipe (68-69 % busy inside the sweep).  Lanes of two threads with ten columns each at 20 columns
// (eleven doubles of state per column pair and thread: 255 registers with a few spills to L1), of four threads with
// six to eight beyond.  Measured against the term-by-term sweep: n = 20, m = 400, 2 000 streams 18.3 -> 14.2 ms;
// n = 24, m = 576, 600 streams 128 -> 97 ms; cofactors at 28 columns (148 blocks) 329 -> 274 ms, at 32 columns
// (16 blocks) 6.2 -> 4.9 s.
// A thread with an odd number of columns keeps the last one as an item of its own (sum walked through the four
// terms, 14 instructions).
//
// Reference: the sum itself is photonic_engines/clifford/cuda_cofactors.py:35-151 (term by term).
#pragma once

namespace pe {

// A step that runs the pair sweep keeps column h KH + r of B (thread h of a lane, its r-th column) at position
// r TPL + h of the row, so that the lane's threads read neighbouring 16-byte words: with the columns in order the
// threads of a lane are KH 16 bytes apart, which for KH = 8 is the same banks (K = 29-32: 1.4x slower than the
// term-by-term sweep instead of faster).

// Step tables of the pair walk, in the same positions.  They take the place of the draw's weights, which are not
// alive during a sweep.
template <int NK>
struct PairTables {
    double2 G[NK][NK];         // per digit and pair (a, b): change of L_u (at a) and L_v (at b) when the sums move by B[kd]
    double2 C[NK];             // C of the pair, at a
};
template <class SM>
__device__ __forceinline__ PairTables<SM::NKMAX>& pair_tables(const SM& sm) {
    constexpr size_t at = (sizeof(SM) + 15) & ~(size_t)15;             // smem_fixed_bytes of the layout
    return *reinterpret_cast<PairTables<SM::NKMAX>*>(reinterpret_cast<unsigned char*>(const_cast<SM*>(&sm)) + at);
}

// All threads, after B is complete: kh columns per thread of a lane of 1 << tl threads.  Columns past K are zero in B.
template <class SM>
static __device__ void prepare_pairs(SM& sm, int kh, int tl) {
    const auto& pl = sm.plan;
    auto& pt = pair_tables(sm);
    const int tid = threadIdx.x, T = blockDim.x, tpl = 1 << tl, kp = kh << tl;
    const int nd = max(1, pl.nin + pl.nmid);               // row 0 is read (times zero) at a lane's first term
    for (int idx = tid; idx < nd * kp; idx += T) {
        const int kd = idx / kp, pos = idx % kp, r = pos >> tl;
        if (r == kh - 1 && (kh & 1)) continue;             // the thread's single column
        const int a = (r & 1) ? pos - tpl : pos, b = a + tpl, d = (r & 1) ? pl.pv : pl.pu;
        const double2 ba = sm.B[kd][a], bb = sm.B[kd][b], da = sm.B[d][a], db = sm.B[d][b];
        const double re = fma(ba.x, db.x, -(ba.y * db.y)) + fma(bb.x, da.x, -(bb.y * da.y));
        const double im = fma(ba.x, db.y, ba.y * db.x) + fma(bb.x, da.y, bb.y * da.x);
        pt.G[kd][pos] = make_double2(-2.0 * re, -2.0 * im);
    }
    for (int a = tid; a < kp; a += T) {
        const int r = a >> tl;
        if ((r & 1) || r == kh - 1) continue;              // the first columns of the pairs only
        const int b = a + tpl;
        const double2 ua = sm.B[pl.pu][a], ub = sm.B[pl.pu][b], va = sm.B[pl.pv][a], vb = sm.B[pl.pv][b];
        const double re = fma(ua.x, vb.x, -(ua.y * vb.y)) + fma(ub.x, va.x, -(ub.y * va.y));
        const double im = fma(ua.x, vb.y, ua.y * vb.x) + fma(ub.x, va.y, ub.y * va.x);
        pt.C[a] = make_double2(4.0 * re, 4.0 * im);
    }
}

// The sweep's values: double (FP64 form), or float2 (plain mixed form: two column groups of a thread side by side on
// paired FP32 instructions).
__device__ __forceinline__ double vfma(double a, double b, double c) { return fma(a, b, c); }
__device__ __forceinline__ double vmul(double a, double b) { return a * b; }
__device__ __forceinline__ double vadd(double a, double b) { return a + b; }
__device__ __forceinline__ double vneg(double a) { return -a; }
__device__ __forceinline__ float2 vfma(float2 a, float2 b, float2 c) { return __ffma2_rn(a, b, c); }
__device__ __forceinline__ float2 vmul(float2 a, float2 b) { return __fmul2_rn(a, b); }
__device__ __forceinline__ float2 vadd(float2 a, float2 b) { return __fadd2_rn(a, b); }
__device__ __forceinline__ float2 vneg(float2 a) { return make_float2(-a.x, -a.y); }

// The product of the other threads' totals of a lane (TPL 2: the partner's; TPL 4: two butterfly exchanges).
template <int TPL>
__device__ __forceinline__ void lane_others(double xr, double xi, double& yr, double& yi) {
    if constexpr (TPL == 1) {
        yr = 1.0; yi = 0.0;
    } else {
        yr = __shfl_xor_sync(0xffffffffu, xr, 1);
        yi = __shfl_xor_sync(0xffffffffu, xi, 1);
        if constexpr (TPL == 4) {
            const double gr = fma(xr, yr, -(xi * yi)), gi = fma(xr, yi, xi * yr);
            const double br = __shfl_xor_sync(0xffffffffu, gr, 2), bi = __shfl_xor_sync(0xffffffffu, gi, 2);
            const double nr = fma(yr, br, -(yi * bi));
            yi = fma(yr, bi, yi * br);
            yr = nr;
        }
    }
}

// The same for paired values, each half counting as a thread of its own.
template <int TPL>
__device__ __forceinline__ void lane_others(float2 xr, float2 xi, float2& yr, float2& yi) {
    yr = make_float2(xr.y, xr.x);
    yi = make_float2(xi.y, xi.x);
    if constexpr (TPL == 2) {
        const float tr = fmaf(xr.x, xr.y, -(xi.x * xi.y)), ti = fmaf(xr.x, xi.y, xi.x * xr.y);
        const float Tr = __shfl_xor_sync(0xffffffffu, tr, 1), Ti = __shfl_xor_sync(0xffffffffu, ti, 1);
        const float2 R = make_float2(Tr, Tr), I = make_float2(Ti, Ti);
        const float2 nr = vfma(yr, R, vneg(vmul(yi, I)));
        yi = vfma(yr, I, vmul(yi, R));
        yr = nr;
    }
}

// P (+)= x y, complex (FIRST: P = x y).
template <bool FIRST, typename V>
__device__ __forceinline__ void cacc(V xr, V xi, V yr, V yi, V& Pr, V& Pi) {
    if (FIRST) {
        Pr = vfma(xr, yr, vneg(vmul(xi, yi)));
        Pi = vfma(xr, yi, vmul(xi, yr));
    } else {
        Pr = vfma(xr, yr, Pr);
        Pr = vfma(vneg(xi), yi, Pr);
        Pi = vfma(xr, yi, Pi);
        Pi = vfma(xi, yr, Pi);
    }
}
template <typename V>
__device__ __forceinline__ void cmul_by(V& xr, V& xi, V yr, V yi) {
    const V nr = vfma(xr, yr, vneg(vmul(xi, yi)));
    xi = vfma(xr, yi, vmul(xi, yr));
    xr = nr;
}

// The items [LO, HI) of one half, y = the product of everything else: P[p] += y prod of the half's other items.
template <int LO, int HI, int NP, int NI, bool FIRST, typename V>
__device__ __forceinline__ void half_items(const V (&qr)[NI], const V (&qi)[NI], const V (&pr)[NI], const V (&pi)[NI],
                                           V yr, V yi, V (&Pr)[NP], V (&Pi)[NP], V& ar, V& ai) {
#pragma unroll
    for (int p = HI - 1; p >= LO; --p) {
        // below p: pr (the prefix); above p: already in y.  The first item's factor above is its neighbour times y
        const bool single = p >= NP;
        V& tr = single ? ar : Pr[p < NP ? p : 0];
        V& ti = single ? ai : Pi[p < NP ? p : 0];
        if (p > LO) {
            if (FIRST && !single) cacc<true>(pr[p], pi[p], yr, yi, tr, ti);
            else cacc<false>(pr[p], pi[p], yr, yi, tr, ti);
            if (p > LO + 1) cmul_by(yr, yi, qr[p], qi[p]);
        } else if (HI - LO > 1) {
            if (FIRST && !single) cacc<true>(qr[LO + 1], qi[LO + 1], yr, yi, tr, ti);
            else cacc<false>(qr[LO + 1], qi[LO + 1], yr, yi, tr, ti);
        } else if (FIRST && !single) {
            tr = yr;
            ti = yi;
        } else {
            tr = vadd(tr, yr);
            ti = vadd(ti, yi);
        }
    }
}

// One term: P[p] += w prod of the other items (FIRST: P[p] = ...), over the lane's items.  The thread's NI items
// are two halves whose prefix and suffix chains run side by side (two complex chains keep the FP64 pipe busy
// where one leaves it waiting), at the same number of multiplications as one chain.  The single item of an odd
// column count is item NI - 1 and accumulates straight into its cofactor.
template <int NP, bool ODD, int TPL, bool FIRST, typename V>
__device__ __forceinline__ void pair_term(const V (&qr)[NP + ODD], const V (&qi)[NP + ODD], V w, V (&Pr)[NP],
                                          V (&Pi)[NP], V& ar, V& ai) {
    constexpr int NI = NP + ODD, NA = NI > 2 ? (NI + 1) / 2 : NI;
    V pr[NI], pi[NI];
    V ur = qr[0], ui = qi[0], vr = qr[NA < NI ? NA : 0], vi = qi[NA < NI ? NA : 0];
#pragma unroll
    for (int p = 1; p < NA; ++p) {
        pr[p] = ur;
        pi[p] = ui;
        cmul_by(ur, ui, qr[p], qi[p]);
        if (NA + p < NI) {
            pr[NA + p < NI ? NA + p : 0] = vr;
            pi[NA + p < NI ? NA + p : 0] = vi;
            cmul_by(vr, vi, qr[NA + p < NI ? NA + p : 0], qi[NA + p < NI ? NA + p : 0]);
        }
    }
    V yr, yi;
    if constexpr (NA < NI) {
        V tr = ur, ti = ui;
        cmul_by(tr, ti, vr, vi);
        lane_others<TPL>(tr, ti, yr, yi);
        yr = vmul(yr, w);
        yi = vmul(yi, w);
        cmul_by(vr, vi, yr, yi);
        cmul_by(ur, ui, yr, yi);
        half_items<NA, NI, NP, NI, FIRST, V>(qr, qi, pr, pi, ur, ui, Pr, Pi, ar, ai);
        half_items<0, NA, NP, NI, FIRST, V>(qr, qi, pr, pi, vr, vi, Pr, Pi, ar, ai);
    } else {
        lane_others<TPL>(ur, ui, yr, yi);
        yr = vmul(yr, w);
        yi = vmul(yi, w);
        half_items<0, NI, NP, NI, FIRST, V>(qr, qi, pr, pi, yr, yi, Pr, Pi, ar, ai);
    }
}

// The four terms of one block from the column sums s at u = v = 0 and the walked L_u, L_v + C: products of the
// pairs, all-but-one sums P, and their shares of the cofactors (a) and of X_u, X_v (x1, x2).  getc(p): C of pair p;
// getd(d): step of the single column's sum when u (d = 0) or v (d = 1) moves to 1.
template <int KH, int TPL, typename V, class GetC, class GetD>
__device__ __forceinline__ void pair_block(const V (&sr)[KH], const V (&si)[KH], const V (&Lur)[KH / 2],
                                           const V (&Lui)[KH / 2], const V (&Lvr)[KH / 2], const V (&Lvi)[KH / 2], V w,
                                           V (&ar)[KH], V (&ai)[KH], V (&x1r)[KH / 2], V (&x1i)[KH / 2],
                                           V (&x2r)[KH / 2], V (&x2i)[KH / 2], GetC getc, GetD getd) {
    constexpr int NP = KH / 2, ODD = KH & 1, NI = NP + ODD;
    V qr[NI], qi[NI], Pr[NP], Pi[NP], cr, ci;
#pragma unroll
    for (int p = 0; p < NP; ++p) {
        qr[p] = vfma(sr[2 * p], sr[2 * p + 1], vneg(vmul(si[2 * p], si[2 * p + 1])));
        qi[p] = vfma(sr[2 * p], si[2 * p + 1], vmul(si[2 * p], sr[2 * p + 1]));
    }
    if (ODD) { qr[NI - 1] = sr[KH - 1]; qi[NI - 1] = si[KH - 1]; }
    pair_term<NP, ODD, TPL, true, V>(qr, qi, w, Pr, Pi, ar[KH - 1], ai[KH - 1]);                // (0, 0)
#pragma unroll
    for (int p = 0; p < NP; ++p) {
        x1r[p] = vadd(x1r[p], vneg(Pr[p]));
        x1i[p] = vadd(x1i[p], vneg(Pi[p]));
        qr[p] = vadd(qr[p], Lur[p]);
        qi[p] = vadd(qi[p], Lui[p]);
    }
    if (ODD) {
        getd(0, cr, ci);
        qr[NI - 1] = vadd(qr[NI - 1], cr);
        qi[NI - 1] = vadd(qi[NI - 1], ci);
    }
    pair_term<NP, ODD, TPL, false, V>(qr, qi, vneg(w), Pr, Pi, ar[KH - 1], ai[KH - 1]);         // (1, 0)
#pragma unroll
    for (int p = 0; p < NP; ++p) {
        x2r[p] = vadd(x2r[p], vneg(Pr[p]));
        x2i[p] = vadd(x2i[p], vneg(Pi[p]));
        qr[p] = vadd(qr[p], Lvr[p]);
        qi[p] = vadd(qi[p], Lvi[p]);
    }
    if (ODD) {
        getd(1, cr, ci);
        qr[NI - 1] = vadd(qr[NI - 1], cr);
        qi[NI - 1] = vadd(qi[NI - 1], ci);
    }
    pair_term<NP, ODD, TPL, false, V>(qr, qi, w, Pr, Pi, ar[KH - 1], ai[KH - 1]);               // (1, 1)
#pragma unroll
    for (int p = 0; p < NP; ++p) {
        getc(p, cr, ci);
        x1r[p] = vadd(x1r[p], Pr[p]);
        x1i[p] = vadd(x1i[p], Pi[p]);
        qr[p] = vadd(qr[p], vneg(vadd(Lur[p], cr)));
        qi[p] = vadd(qi[p], vneg(vadd(Lui[p], ci)));
    }
    if (ODD) {
        getd(0, cr, ci);
        qr[NI - 1] = vadd(qr[NI - 1], vneg(cr));
        qi[NI - 1] = vadd(qi[NI - 1], vneg(ci));
    }
    pair_term<NP, ODD, TPL, false, V>(qr, qi, vneg(w), Pr, Pi, ar[KH - 1], ai[KH - 1]);         // (0, 1)
#pragma unroll
    for (int p = 0; p < NP; ++p) {
        x2r[p] = vadd(x2r[p], Pr[p]);
        x2i[p] = vadd(x2i[p], Pi[p]);
        const int a = 2 * p, b = 2 * p + 1;
        ar[a] = vfma(Pr[p], sr[b], vfma(vneg(Pi[p]), si[b], ar[a]));
        ai[a] = vfma(Pr[p], si[b], vfma(Pi[p], sr[b], ai[a]));
        ar[b] = vfma(Pr[p], sr[a], vfma(vneg(Pi[p]), si[a], ar[b]));
        ai[b] = vfma(Pr[p], si[a], vfma(Pi[p], sr[a], ai[b]));
    }
}

// KH columns per thread, lanes of TPL threads (tier KP = KH TPL); the plan has pair digits.  The sweeps are functions
// of their own, so that their registers are not shared with the chain loop's: at ten columns per thread 520 bytes of
// spill traffic become 212, at eight or fewer none are left (n = 20, m = 400, 2 000 streams 14.19 -> 13.84 ms).
template <int KH, int TPL, class SM>
__device__ __noinline__ void sweep_pairs_f64() {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    SM& sm = *reinterpret_cast<SM*>(smem_raw);
    constexpr int NP = KH / 2;
    const auto& pl = sm.plan;
    const auto& pt = pair_tables(sm);
    const int tid = threadIdx.x;
    const int lanes = blockDim.x / TPL, lane = tid / TPL, h = tid % TPL, c0 = h * KH;
    const int wl0 = (tid & ~31) / TPL;                     // first lane of this warp: its lanes walk in lockstep
    const int K = pl.K, Lin = pl.Lin, Lmid = pl.Lmid, nin = pl.nin;
    const int64_t H = pl.H;
    double ar[KH], ai[KH], x1r[NP], x1i[NP], x2r[NP], x2i[NP];
#pragma unroll
    for (int j = 0; j < KH; ++j) { ar[j] = 0.0; ai[j] = 0.0; }
#pragma unroll
    for (int p = 0; p < NP; ++p) { x1r[p] = 0.0; x1i[p] = 0.0; x2r[p] = 0.0; x2i[p] = 0.0; }
    for (int64_t hw = sm.chunk * lanes + wl0; hw < H; hw += (int64_t)lanes * sm.lane_mult) {
        double sr[KH], si[KH], Lur[NP], Lui[NP], Lvr[NP], Lvi[NP], wh;
        int64_t hl = hw + (lane - wl0);
        const bool live = hl < H;                          // a lane past the end repeats lane H - 1 at weight 0
        if (!live) hl = H - 1;
        const uint64_t hpack = lane_digits(pl, hl, &wh);
        if (!live) wh = 0.0;
        lane_sums<KH, TPL>(sm, h, false, 0, hl, hpack, sr, si);
#pragma unroll
        for (int j = 0; j < KH; ++j) if (c0 + j >= K) { sr[j] = 1.0; si[j] = 0.0; }
        {
            const double2* bu = &sm.B[pl.pu][h];
            const double2* bv = &sm.B[pl.pv][h];
#pragma unroll
            for (int p = 0; p < NP; ++p) {
                const int a = 2 * p, b = 2 * p + 1;
                // L = -2 (s_a d_b + s_b d_a) + 4 d_a d_b = -2 (s_a d_b + (s_b - 2 d_b) d_a) for the row d of u or v
                auto lin = [&](double2 da, double2 db, double& re, double& im) {
                    const double tr = fma(-2.0, db.x, sr[b]), ti = fma(-2.0, db.y, si[b]);
                    re = fma(sr[a], db.x, fma(-si[a], db.y, fma(tr, da.x, -(ti * da.y))));
                    im = fma(sr[a], db.y, fma(si[a], db.x, fma(tr, da.y, ti * da.x)));
                    re *= -2.0;
                    im *= -2.0;
                };
                lin(bu[a * TPL], bu[b * TPL], Lur[p], Lui[p]);
                lin(bv[a * TPL], bv[b * TPL], Lvr[p], Lvi[p]);
                const double2 c = pt.C[2 * p * TPL + h];
                Lvr[p] += c.x;                             // L_v + C: the step from (1, 0) to (1, 1)
                Lvi[p] += c.y;
            }
        }
        for (int pm = 0; pm < Lmid; ++pm) {
            const double wmh = wh * sm.tab_wm[pm];
            const bool fwd = !(pm & 1);
            // the transition into the block's first term: the middle digit's (none at the lane's first term)
            unsigned e = pm > 0 ? (unsigned)sm.tab_fm[pm] : 0u;
            double f = pm > 0 ? ((e & 0x80u) ? -2.0 : 2.0) : 0.0;
            int kd = pm > 0 ? nin + (int)(e & 63u) : 0;
            for (int i = 0;;) {
                const int t = fwd ? i : Lin - 1 - i;
                const double2* b = &sm.B[kd][h];
                const double2* g = &pt.G[kd][h];
#pragma unroll
                for (int j = 0; j < KH; ++j) { sr[j] = fma(f, b[j * TPL].x, sr[j]); si[j] = fma(f, b[j * TPL].y, si[j]); }
#pragma unroll
                for (int p = 0; p < NP; ++p) {
                    Lur[p] = fma(f, g[2 * p * TPL].x, Lur[p]);
                    Lui[p] = fma(f, g[2 * p * TPL].y, Lui[p]);
                    Lvr[p] = fma(f, g[(2 * p + 1) * TPL].x, Lvr[p]);
                    Lvi[p] = fma(f, g[(2 * p + 1) * TPL].y, Lvi[p]);
                }
                const double w = wmh * sm.tab_w[t];
                pair_block<KH, TPL, double>(
                    sr, si, Lur, Lui, Lvr, Lvi, w, ar, ai, x1r, x1i, x2r, x2i,
                    [&](int p, double& re, double& im) {
                        const double2 c = pt.C[2 * p * TPL + h];
                        re = c.x;
                        im = c.y;
                    },
                    [&](int d, double& re, double& im) {
                        const double2 x = sm.B[d ? pl.pv : pl.pu][(KH - 1) * TPL + h];
                        re = -2.0 * x.x;
                        im = -2.0 * x.y;
                    });
                if (++i == Lin) break;
                e = sm.tab_f[fwd ? i : Lin - i];           // backward: the transition into t + 1, undone
                kd = (int)(e & 63u);
                f = (((e & 0x80u) != 0u) == fwd) ? -2.0 : 2.0;
            }
        }
    }
    {
        const double2* bu = &sm.B[pl.pu][h];
        const double2* bv = &sm.B[pl.pv][h];
#pragma unroll
        for (int j = 0; j < 2 * NP; ++j) {
            const int p = j / 2;
            const double2 du = bu[(j ^ 1) * TPL], dv = bv[(j ^ 1) * TPL];
            const double tr = fma(du.x, x1r[p], fma(-du.y, x1i[p], fma(dv.x, x2r[p], -(dv.y * x2i[p]))));
            const double ti = fma(du.x, x1i[p], fma(du.y, x1r[p], fma(dv.x, x2i[p], dv.y * x2r[p])));
            ar[j] = fma(-2.0, tr, ar[j]);
            ai[j] = fma(-2.0, ti, ai[j]);
        }
    }
    reduce_to_P<KH, TPL>(ar, ai, sm, c0);
}

// ---------------------------------------------------------------------------------------- mixed form
// Step tables of the mixed form's pair walk, in the slots of B32: slot h KQ + r holds column h 2 KQ + r in .x / .z and
// column h 2 KQ + KQ + r in .y / .w (real, imaginary).  Only the inner digits are walked in FP32.
template <int NK>
struct PairTables32 {
    float4 G[NK][NK / 2];      // change of L_u (even r) and L_v (odd r) of the slot's pairs when the sums move by 2 B[kd]
    float4 C[NK / 2];          // C of the pairs, at their even slot
};
template <class SM>
__device__ __forceinline__ PairTables32<SM::NKMAX>& pair_tables32(const SM& sm) {
    constexpr size_t at = (sizeof(SM) + 15) & ~(size_t)15;
    return *reinterpret_cast<PairTables32<SM::NKMAX>*>(reinterpret_cast<unsigned char*>(const_cast<SM*>(&sm)) + at);
}

// x_a y_b + x_b y_a, complex: the mixed difference of the products of two columns.
static __device__ __forceinline__ double2 cross(double2 xa, double2 xb, double2 ya, double2 yb) {
    return make_double2(fma(xa.x, yb.x, -(xa.y * yb.y)) + fma(xb.x, ya.x, -(xb.y * ya.y)),
                        fma(xa.x, yb.y, xa.y * yb.x) + fma(xb.x, ya.y, xb.y * ya.x));
}

// All threads, after B is complete (columns in order): kq columns per half thread, tpl threads per lane.
template <class SM>
static __device__ void prepare_pairs32(SM& sm, int kq, int tpl) {
    const auto& pl = sm.plan;
    auto& pt = pair_tables32(sm);
    const int tid = threadIdx.x, T = blockDim.x, ns = kq * tpl;
    const int nd = max(1, pl.nin);                         // row 0 is read (times zero) at a block's first term
    for (int idx = tid; idx < nd * ns; idx += T) {
        const int kd = idx / ns, q = idx % ns, r = q % kq;
        if (r == kq - 1 && (kq & 1)) continue;
        const int a = (q / kq) * 2 * kq + (r & ~1), d = (r & 1) ? pl.pv : pl.pu;
        const double2 x = cross(sm.B[kd][a], sm.B[kd][a + 1], sm.B[d][a], sm.B[d][a + 1]);
        const double2 y = cross(sm.B[kd][a + kq], sm.B[kd][a + kq + 1], sm.B[d][a + kq], sm.B[d][a + kq + 1]);
        pt.G[kd][q] = make_float4((float)(-4.0 * x.x), (float)(-4.0 * y.x), (float)(-4.0 * x.y), (float)(-4.0 * y.y));
    }
    for (int q = tid; q < ns; q += T) {
        const int r = q % kq;
        if ((r & 1) || r == kq - 1) continue;
        const int a = (q / kq) * 2 * kq + r;
        const double2 x = cross(sm.B[pl.pu][a], sm.B[pl.pu][a + 1], sm.B[pl.pv][a], sm.B[pl.pv][a + 1]);
        const double2 y = cross(sm.B[pl.pu][a + kq], sm.B[pl.pu][a + kq + 1], sm.B[pl.pv][a + kq], sm.B[pl.pv][a + kq + 1]);
        pt.C[q] = make_float4((float)(4.0 * x.x), (float)(4.0 * y.x), (float)(4.0 * x.y), (float)(4.0 * y.y));
    }
}

// The mixed form's pair sweep: as sweep_mixed, every inner block starts from column sums (and L_u, L_v) formed in
// FP64 and rounded once, runs in complex FP32 on paired instructions (the thread's 2 KQ columns as two halves side by
// side), and its shares of the cofactors, X_u and X_v are folded into FP64 accumulators.  A block walks a quarter of
// the updates for the same terms, so its column sums drift less: largest marginal error against FP64 3.4e-5 -> 1.2e-5
// at n = 20, m = 400 (256 chains), 9.3e-5 -> 4.5e-5 at n = 28, m = 784, largest CDF error halved.  n = 20, m = 400,
// 2 000 streams 12.6 -> 9.9 ms; n = 24, m = 576, 600 streams 87 -> 70 ms; n = 28, m = 784, 148 streams 874 -> 768 ms.
template <int KQ, int TPL, class SM>
__device__ __noinline__ void sweep_pairs_mixed() {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    SM& sm = *reinterpret_cast<SM*>(smem_raw);
    constexpr int NP = KQ / 2, KH = 2 * KQ;
    const auto& pl = sm.plan;
    const auto& pt = pair_tables32(sm);
    const int tid = threadIdx.x;
    const int lanes = blockDim.x / TPL, lane = tid / TPL, h = tid % TPL, c0 = h * KH;
    const int wl0 = (tid & ~31) / TPL;
    const int K = pl.K, Lin = pl.Lin, Lmid = pl.Lmid;
    const int64_t H = pl.H;
    double ar[KH], ai[KH];
#pragma unroll
    for (int j = 0; j < KH; ++j) { ar[j] = 0.0; ai[j] = 0.0; }
    for (int64_t hw = sm.chunk * lanes + wl0; hw < H; hw += (int64_t)lanes * sm.lane_mult) {
        double wh;
        int64_t hl = hw + (lane - wl0);
        const bool live = hl < H;
        if (!live) hl = H - 1;
        const uint64_t hpack = lane_digits(pl, hl, &wh);
        if (!live) wh = 0.0;
        for (int pm = 0; pm < Lmid; ++pm) {
            const bool fwd = !(pm & 1);
            float2 sr[KQ], si[KQ], Lur[NP], Lui[NP], Lvr[NP], Lvi[NP];
            {
                double xr[KH], xi[KH];
                lane_sums<KH>(sm, c0, !fwd, pm, hl, hpack, xr, xi);
#pragma unroll
                for (int j = 0; j < KH; ++j) if (c0 + j >= K) { xr[j] = 1.0; xi[j] = 0.0; }
#pragma unroll
                for (int r = 0; r < KQ; ++r) {
                    sr[r] = make_float2((float)xr[r], (float)xr[KQ + r]);
                    si[r] = make_float2((float)xi[r], (float)xi[KQ + r]);
                }
                // L = -2 (s_a d_b + s_b d_a) + 4 d_a d_b = -2 ((s_b - d_b) d_a + (s_a - d_a) d_b) for the row d of u
                // or v, and C = 4 (u_a v_b + u_b v_a) added to L_v
                auto lin = [&](int d, int a, bool withc) {
                    const double2 da = sm.B[d][c0 + a], db = sm.B[d][c0 + a + 1];
                    const double2 x = cross(make_double2(xr[a] - da.x, xi[a] - da.y),
                                            make_double2(xr[a + 1] - db.x, xi[a + 1] - db.y), da, db);
                    double2 l = make_double2(-2.0 * x.x, -2.0 * x.y);
                    if (withc) {
                        const double2 c = cross(sm.B[pl.pu][c0 + a], sm.B[pl.pu][c0 + a + 1], da, db);
                        l = make_double2(fma(4.0, c.x, l.x), fma(4.0, c.y, l.y));
                    }
                    return l;
                };
#pragma unroll
                for (int p = 0; p < NP; ++p) {
                    const double2 ux = lin(pl.pu, 2 * p, false), uy = lin(pl.pu, KQ + 2 * p, false);
                    const double2 vx = lin(pl.pv, 2 * p, true), vy = lin(pl.pv, KQ + 2 * p, true);
                    Lur[p] = make_float2((float)ux.x, (float)uy.x);
                    Lui[p] = make_float2((float)ux.y, (float)uy.y);
                    Lvr[p] = make_float2((float)vx.x, (float)vy.x);
                    Lvi[p] = make_float2((float)vx.y, (float)vy.y);
                }
            }
            float2 a2r[KQ], a2i[KQ], x1r[NP], x1i[NP], x2r[NP], x2i[NP];
#pragma unroll
            for (int r = 0; r < KQ; ++r) { a2r[r] = make_float2(0.0f, 0.0f); a2i[r] = make_float2(0.0f, 0.0f); }
#pragma unroll
            for (int p = 0; p < NP; ++p) {
                x1r[p] = make_float2(0.0f, 0.0f); x1i[p] = make_float2(0.0f, 0.0f);
                x2r[p] = make_float2(0.0f, 0.0f); x2i[p] = make_float2(0.0f, 0.0f);
            }
            unsigned e = 0u;
            float f = 0.0f;                                // no transition into the block's first term
            int kd = 0;
            for (int i = 0;;) {
                const int t = fwd ? i : Lin - 1 - i;
                const float4* b = reinterpret_cast<const float4*>(&sm.B32[kd][0]) + h * KQ;
                const float4* g = &pt.G[kd][h * KQ];
                const float2 ff = make_float2(f, f);
#pragma unroll
                for (int r = 0; r < KQ; ++r) {
                    const float4 v = b[r];
                    sr[r] = vfma(ff, make_float2(v.x, v.y), sr[r]);
                    si[r] = vfma(ff, make_float2(v.z, v.w), si[r]);
                }
#pragma unroll
                for (int p = 0; p < NP; ++p) {
                    const float4 u = g[2 * p], v = g[2 * p + 1];
                    Lur[p] = vfma(ff, make_float2(u.x, u.y), Lur[p]);
                    Lui[p] = vfma(ff, make_float2(u.z, u.w), Lui[p]);
                    Lvr[p] = vfma(ff, make_float2(v.x, v.y), Lvr[p]);
                    Lvi[p] = vfma(ff, make_float2(v.z, v.w), Lvi[p]);
                }
                const float w = sm.tab_w32[t];
                pair_block<KQ, TPL, float2>(
                    sr, si, Lur, Lui, Lvr, Lvi, make_float2(w, w), a2r, a2i, x1r, x1i, x2r, x2i,
                    [&](int p, float2& re, float2& im) {
                        const float4 c = pt.C[h * KQ + 2 * p];
                        re = make_float2(c.x, c.y);
                        im = make_float2(c.z, c.w);
                    },
                    [&](int d, float2& re, float2& im) {
                        const float4 x = reinterpret_cast<const float4*>(&sm.B32[d ? pl.pv : pl.pu][0])[h * KQ + KQ - 1];
                        re = make_float2(-x.x, -x.y);
                        im = make_float2(-x.z, -x.w);
                    });
                if (++i == Lin) break;
                e = sm.tab_f[fwd ? i : Lin - i];
                kd = (int)(e & 63u);
                f = (((e & 0x80u) != 0u) == fwd) ? -1.0f : 1.0f;
            }
            const double wmh = wh * sm.tab_wm[pm];
#pragma unroll
            for (int r = 0; r < KQ; ++r) {
                ar[r] = fma(wmh, (double)a2r[r].x, ar[r]);
                ai[r] = fma(wmh, (double)a2i[r].x, ai[r]);
                ar[KQ + r] = fma(wmh, (double)a2r[r].y, ar[KQ + r]);
                ai[KQ + r] = fma(wmh, (double)a2i[r].y, ai[KQ + r]);
            }
#pragma unroll
            for (int r = 0; r < 2 * NP; ++r) {
                const int p = r / 2;
#pragma unroll
                for (int y = 0; y < 2; ++y) {
                    const double2 u = sm.B[pl.pu][c0 + y * KQ + (r ^ 1)], v = sm.B[pl.pv][c0 + y * KQ + (r ^ 1)];
                    const double Xr = y ? x1r[p].y : x1r[p].x, Xi = y ? x1i[p].y : x1i[p].x;
                    const double Yr = y ? x2r[p].y : x2r[p].x, Yi = y ? x2i[p].y : x2i[p].x;
                    const double tr = fma(u.x, Xr, fma(-u.y, Xi, fma(v.x, Yr, -(v.y * Yi))));
                    const double ti = fma(u.x, Xi, fma(u.y, Xr, fma(v.x, Yi, v.y * Yr)));
                    ar[y * KQ + r] = fma(-2.0 * wmh, tr, ar[y * KQ + r]);
                    ai[y * KQ + r] = fma(-2.0 * wmh, ti, ai[y * KQ + r]);
                }
            }
        }
    }
    reduce_to_P<KH, TPL>(ar, ai, sm, c0);
}

// Shared memory a variant's kernels with a sweep set aside for the tables, over the draw's weights.
template <int TPL, int KPM, int PREC>
constexpr size_t pair_table_bytes() {
    if (PREC == PREC_COMP || !has_pairs<TPL, KPM>()) return 0;
    return PREC == PREC_MIXED ? sizeof(PairTables32<NARROW>) : sizeof(PairTables<NARROW>);
}

}  // namespace pe
