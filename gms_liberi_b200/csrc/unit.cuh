// unit.cuh -- quartet classes of small builds: warp tasks whose lanes share a
// quartet's primitive loop (included by k_u*.cu).
//
// A class of a small molecule has fewer quartets than the GPU has lanes, so
// the thread-per-quartet class kernels (quartet.cuh) last as long as one
// thread's primitive loop (36 x 36 primitive quartets in (ss|ss): 400 us) or
// one thread's passes ((dd|pd): 185 us for one primitive quartet), and every
// class is its own launch.  Here a warp takes 1..32 kets of one row pair and
// its 32 lanes are split three ways: kets, passes over the components of
// shells A and B (PG lanes, compile-time per class), and the primitive
// quartets and Rys roots of one quartet (UG lanes, whatever is left).  The UG
// partial blocks are summed with shuffles, then the quartet is digested by
// the DIRFCK rules as in quartet.cuh.  All classes of a register budget share
// one launch: a block looks its class up and calls that class's function.
// Bound by the latency of one lane's chain, not by a pipe (FP64 pipe 6 to 18%):
// a lane's share of the primitive loop is cut to a few microseconds by the
// host's choice of kets per task.  Whole builds through the host call: 7
// functions 350 -> 75 us, 42 functions 752 -> 106 us; the Obara-Saika classes on
// Boys rows instead of one recurrence a root took 10 atoms in the mixed tier from
// 153 to 141 us.
#pragma once
#include "quartet.cuh"

namespace liberi {

struct UnitClass {
    const int *bra_ids;
    const double4 *ket_rec;
    const int *bra_orig, *ket_orig;
    const int4 *tasks;      // (bra position, first ket position, ket count, -)
    const int *ntasks_dev;  // device task count (mixed builds) or null
    int ntasks;             // static count, or capacity of a per-build list
    int first_block;        // first block of the class in the launch
    double cut, thr;
    int k, strict, swapped;
    RankSplit rs;
};
struct UnitArgs {
    DevBasis b;
    const double *tab;
    const float *tabf;
    const double *Dm;
    const float *Dmf;
    double *F, *F2;   // open-shell builds: F_alpha, F_beta
    size_t k_offset;  // open-shell builds: the alpha and beta exchange densities at D + k_offset, D + 2 k_offset
    const unsigned long long *maxd;
    double prim_cut;
    int nbf, ncls;
    UnitClass cls[NKERN];
};

// components of A and B per pass (bounds the block a lane holds; the classes
// of few components take one pass, the largest one A and half of B per pass)
constexpr int unit_nmu(int key) {
    switch (key) {
        case 1111: case 2210: case 1120: case 2211: case 2121: case 2120: case 2111: case 2220: case 2221:
        case 2222: return 1;
        case 2110: case 2200: case 2020: return 3;
        default: return 6;
    }
}
constexpr int unit_nbu(int key) { return key == 2221 || key == 2222 ? 3 : 6; }
constexpr int pow2ceil(int x) { return x <= 1 ? 1 : 2 * pow2ceil((x + 1) / 2); }

template <int LA, int LB, int LC, int LD>
struct UShape {
    static constexpr int KEY = class_key(LA, LB, LC, LD);
    static constexpr int NA = ncart(LA), NB = ncart(LB);
    static constexpr int NMU = unit_nmu(KEY) < NA ? unit_nmu(KEY) : NA;
    static constexpr int NBU = unit_nbu(KEY) < NB ? unit_nbu(KEY) : NB;
    static constexpr int NPB = (NB + NBU - 1) / NBU;
    static constexpr int NPASS = (NA + NMU - 1) / NMU * NPB;
    static constexpr int PG = pow2ceil(NPASS);
    static_assert(PG <= 32 && NA % NMU == 0 && NB % NBU == 0, "passes are lanes of one warp");
};

// one root and weight of the N-root rule (rys_eval's tables and limits)
template <int N>
__device__ __forceinline__ void rys_root(int r, double T, double thr, bool strict, const double *__restrict__ tab,
                                         double &u, double &w) {
    if (strict ? (T > thr) : (T >= thr)) {
        const double it = 1.0 / T;
        const double *hr = tab + rys_herm_off(N);
        u = __ldg(hr + r) * it;
        w = __ldg(hr + MAXROOT + r) * sqrt(it);
        return;
    }
    const double t4 = T * (double)RYS_PER_UNIT;
    const int k = (int)t4;
    const double x = 2.0 * (t4 - (double)k) - 1.0, x2 = x * x, x4 = x2 * x2;
    const double *base = tab + rys_table_off(N) + (size_t)k * (2 * N * RYS_NCOEF) + r * RYS_NCOEF;
    double v[2];
#pragma unroll
    for (int h = 0; h < 2; h++) {
        double c0, c1, c2, c3, c4, c5, c6, c7;
        ldg_v4f64(base + h * (N * RYS_NCOEF), c0, c1, c2, c3);
        ldg_v4f64(base + h * (N * RYS_NCOEF) + 4, c4, c5, c6, c7);
        const double a0 = fma(c1, x, c0), a1 = fma(c3, x, c2);
        const double a2 = fma(c5, x, c4), a3 = fma(c7, x, c6);
        v[h] = fma(fma(a3, x2, a2), x4, fma(a1, x2, a0));
    }
    u = v[0];
    w = v[1];
}
template <int N>
__device__ __forceinline__ void rys_root(int r, float T, float thr, bool strict, const float *__restrict__ tab,
                                         float &u, float &w) {
    if (strict ? (T > thr) : (T >= thr)) {
        const float sq = rsqrtf(T);
        const float *hr = tab + rysf_herm_off(N);
        u = __ldg(hr + r) * (sq * sq);
        w = __ldg(hr + MAXROOT + r) * sq;
        return;
    }
    const float t8 = T * (float)RYSF_PER_UNIT;
    const int k = (int)t8;
    const float x = 2.0f * (t8 - (float)k) - 1.0f, x2 = x * x;
    const float *base = tab + rysf_table_off(N) + (size_t)k * (2 * N * RYSF_NCOEF) + r * RYSF_NCOEF;
    const float4 cu = __ldg(reinterpret_cast<const float4 *>(base));
    const float4 cw = __ldg(reinterpret_cast<const float4 *>(base + N * RYSF_NCOEF));
    u = fmaf(fmaf(cu.w, x, cu.z), x2, fmaf(cu.y, x, cu.x));
    w = fmaf(fmaf(cw.w, x, cw.z), x2, fmaf(cw.y, x, cw.x));
}

// One root's products for NMU components of A (exponents ex..) and NBU of B.
template <int LA, int LB, int LC, int LD, typename R, int NMU, int NBU>
__device__ __forceinline__ void contract_unit(const R (&gx)[LA + LB + 1][LC + LD + 1],
                                              const R (&gy)[LA + LB + 1][LC + LD + 1],
                                              const R (&gz)[LA + LB + 1][LC + LD + 1], R abx, R aby, R abz, R cdx,
                                              R cdy, R cdz, const int (&ex)[NMU], const int (&ey)[NMU],
                                              const int (&ez)[NMU], int nu0,
                                              R (&acc)[NMU][NBU][ncart(LC)][ncart(LD)]) {
    if constexpr (NBU == ncart(LB)) {
        contract_root<LA, LB, LC, LD, R, NMU>(gx, gy, gz, abx, aby, abz, cdx, cdy, cdz, ex, ey, ez, acc);
    } else {
#pragma unroll
        for (int m = 0; m < NMU; m++) {
            R sx[LB + 1][LC + 1][LD + 1], sy[LB + 1][LC + 1][LD + 1], sz[LB + 1][LC + 1][LD + 1];
            hrr_slice<LA, LB, LC, LD, R>(gx, ex[m], abx, cdx, sx);
            hrr_slice<LA, LB, LC, LD, R>(gy, ey[m], aby, cdy, sy);
            hrr_slice<LA, LB, LC, LD, R>(gz, ez[m], abz, cdz, sz);
#pragma unroll
            for (int n = 0; n < NBU; n++) {
                const int bx = cx_rt(LB, nu0 + n), by = cy_rt(LB, nu0 + n), bz = cz_rt(LB, nu0 + n);
                R tx[LC + 1][LD + 1], ty[LC + 1][LD + 1], tz[LC + 1][LD + 1];
#pragma unroll
                for (int c = 0; c <= LC; c++)
#pragma unroll
                    for (int d = 0; d <= LD; d++) {
                        R x = sx[0][c][d], y = sy[0][c][d], z = sz[0][c][d];
#pragma unroll
                        for (int e = 1; e <= LB; e++) {
                            x = bx == e ? sx[e][c][d] : x;
                            y = by == e ? sy[e][c][d] : y;
                            z = bz == e ? sz[e][c][d] : z;
                        }
                        tx[c][d] = x;
                        ty[c][d] = y;
                        tz[c][d] = z;
                    }
#pragma unroll
                for (int ic = 0; ic < ncart(LC); ic++)
#pragma unroll
                    for (int id = 0; id < ncart(LD); id++)
                        acc[m][n][ic][id] += tx[cxp(LC, ic)][cxp(LD, id)] * ty[cyp(LC, ic)][cyp(LD, id)] *
                                             tz[czp(LC, ic)][czp(LD, id)];
            }
        }
    }
}

// The unique-component loops and 0.5 factors of a quartet with coinciding
// shells (int0000.F90:241-292): 0 for a component those loops skip.
template <int LA, int LB, int LC, int LD, typename R>
__device__ __forceinline__ R unit_factor(const QuartetCtx<R> &qc, int ia, int ib, int ic, int id) {
    constexpr int NB = ncart(LB), ND = ncart(LD);
    if (LA == LB && qc.iandj && ib > ia) return R(0);
    if (LC == LD && qc.kandl && id > ic) return R(0);
    if (LA == LC && LB == LD && qc.same) {
        const int oij = qc.iandj ? ia * (ia + 1) / 2 + ib : ia * NB + ib;
        const int okl = qc.kandl ? ic * (ic + 1) / 2 + id : ic * ND + id;
        if (okl > oij) return R(0);
    }
    const int mu = qc.bfA + ia, nu = qc.bfB + ib, la = qc.bfC + ic, si = qc.bfD + id;
    R f = R(1);
    if (mu == nu) f *= R(0.5);
    if (la == si) f *= R(0.5);
    if ((mu == la && nu == si) || (mu == si && nu == la)) f *= R(0.5);
    return f;
}

template <typename R>
__device__ __forceinline__ void f_add(double *F, unsigned i, unsigned j, R v) {
    if (v != R(0)) atomicAdd(F + tri0(i, j), (double)v);
}

// Digestion of NMU x NBU components of (A, B) from (mu0, nu0): the six
// updates, K and ket J sums added as soon as they are complete; jab is left
// for the warp sum.  NS exchange densities (two in an open-shell build, whose
// integrals then serve both spins), each with its own F; the Coulomb updates
// go to all of them.
template <int LA, int LB, int LC, int LD, typename R, int NMU, int NBU, int NS>
__device__ __forceinline__ void digest_unit(const R (&acc)[NMU][NBU][ncart(LC)][ncart(LD)], int mu0, int nu0,
                                            const QuartetCtx<R> &qc, size_t k_offset, double *const (&F)[NS],
                                            R (&jab)[NMU][NBU]) {
    constexpr int NC = ncart(LC), ND = ncart(LD);
    const bool distinct = !qc.iandj && !qc.kandl && !qc.same;
    R sab[NMU][NBU], dAB[NMU][NBU], dAD[NS][NMU][ND], dBD[NS][NBU][ND], kad[NS][NMU][ND], kbd[NS][NBU][ND];
#pragma unroll
    for (int m = 0; m < NMU; m++)
#pragma unroll
        for (int n = 0; n < NBU; n++) {
            sab[m][n] = R(s3pow(cs3_rt(LA, mu0 + m) + cs3_rt(LB, nu0 + n)));
            dAB[m][n] = R(4) * dget(qc.Dm, qc.ld, qc.bfA + mu0 + m, qc.bfB + nu0 + n);
        }
#pragma unroll
    for (int s = 0; s < NS; s++)
#pragma unroll
        for (int id = 0; id < ND; id++) {
#pragma unroll
            for (int m = 0; m < NMU; m++) {
                dAD[s][m][id] = dget(qc.DmK + s * k_offset, qc.ld, qc.bfA + mu0 + m, qc.bfD + id);
                kad[s][m][id] = R(0);
            }
#pragma unroll
            for (int n = 0; n < NBU; n++) {
                dBD[s][n][id] = dget(qc.DmK + s * k_offset, qc.ld, qc.bfB + nu0 + n, qc.bfD + id);
                kbd[s][n][id] = R(0);
            }
        }
#pragma unroll
    for (int ic = 0; ic < NC; ic++) {
        R dAC[NS][NMU], dBC[NS][NBU], kac[NS][NMU], kbc[NS][NBU];
#pragma unroll
        for (int s = 0; s < NS; s++) {
#pragma unroll
            for (int m = 0; m < NMU; m++) {
                dAC[s][m] = dget(qc.DmK + s * k_offset, qc.ld, qc.bfA + mu0 + m, qc.bfC + ic);
                kac[s][m] = R(0);
            }
#pragma unroll
            for (int n = 0; n < NBU; n++) {
                dBC[s][n] = dget(qc.DmK + s * k_offset, qc.ld, qc.bfB + nu0 + n, qc.bfC + ic);
                kbc[s][n] = R(0);
            }
        }
#pragma unroll
        for (int id = 0; id < ND; id++) {
            const R dCD = dget(qc.Dm, qc.ld, qc.bfC + ic, qc.bfD + id);
            R jcd = R(0);
#pragma unroll
            for (int m = 0; m < NMU; m++)
#pragma unroll
                for (int n = 0; n < NBU; n++) {
                    R v = acc[m][n][ic][id] * (sab[m][n] * R(s3pow(cs3(LC, ic) + cs3(LD, id))));
                    v = fabs(v) < qc.cut ? R(0) : v;
                    if (!distinct) v *= unit_factor<LA, LB, LC, LD, R>(qc, mu0 + m, nu0 + n, ic, id);
                    jab[m][n] = fma(v, dCD, jab[m][n]);
                    jcd = fma(v, dAB[m][n], jcd);
#pragma unroll
                    for (int s = 0; s < NS; s++) {
                        kac[s][m] = fma(v, dBD[s][n][id], kac[s][m]);
                        kad[s][m][id] = fma(v, dBC[s][n], kad[s][m][id]);
                        kbc[s][n] = fma(v, dAD[s][m][id], kbc[s][n]);
                        kbd[s][n][id] = fma(v, dAC[s][m], kbd[s][n][id]);
                    }
                }
#pragma unroll
            for (int s = 0; s < NS; s++) f_add(F[s], qc.bfC + ic, qc.bfD + id, jcd);
        }
#pragma unroll
        for (int s = 0; s < NS; s++) {
#pragma unroll
            for (int m = 0; m < NMU; m++) f_add(F[s], qc.bfA + mu0 + m, qc.bfC + ic, -kac[s][m]);
#pragma unroll
            for (int n = 0; n < NBU; n++) f_add(F[s], qc.bfB + nu0 + n, qc.bfC + ic, -kbc[s][n]);
        }
    }
#pragma unroll
    for (int s = 0; s < NS; s++)
#pragma unroll
        for (int id = 0; id < ND; id++) {
#pragma unroll
            for (int m = 0; m < NMU; m++) f_add(F[s], qc.bfA + mu0 + m, qc.bfD + id, -kad[s][m][id]);
#pragma unroll
            for (int n = 0; n < NBU; n++) f_add(F[s], qc.bfB + nu0 + n, qc.bfD + id, -kbd[s][n][id]);
        }
}

// Obara-Saika contribution of one primitive quartet to (e0|c0) (os_add): c the
// Boys values, hp = 1/2p, pq = P-Q, pa = P-A, qc = Q-C.
template <int LA, int LB, int LC, typename R>
__device__ __forceinline__ void unit_os(R (&c)[LA + LB + LC + 1], R pref, R p, R q, R ipq, R hp, R pqx, R pqy, R pqz,
                                        R pax, R pay, R paz, R qcx, R qcy, R qcz,
                                        R (&acc)[nrange(LA, LA + LB)][ncart(LC)][1]) {
    const R rq = q * ipq, rp = p * ipq;
#pragma unroll
    for (int m = 0; m <= LA + LB + LC; m++) c[m] *= pref;
    const R pa[3] = {pax, pay, paz}, qc[3] = {qcx, qcy, qcz};
    const R wp[3] = {-rq * pqx, -rq * pqy, -rq * pqz}, wq[3] = {rp * pqx, rp * pqy, rp * pqz};
    os_add<LA, LB, LC>(c, pa, qc, wp, wq, hp, rq, R(0.5) * ipq, R(0), rp,  // (LC <= 1 here)
                       [&](int e, int ic, R x, R y) { acc[e][ic][0] = fma(x, y, acc[e][ic][0]); });
}

// One warp task: row pair t.x against kets t.y .. t.y+t.z-1, t.z * PG <= 32.
template <int LA, int LB, int LC, int LD, typename R, int NS>
__device__ __noinline__ void unit_task(const UnitArgs &a, const UnitClass &u, int4 t) {
    using S = UShape<LA, LB, LC, LD>;
    constexpr int NC = ncart(LC), ND = ncart(LD), NMU = S::NMU, NBU = S::NBU, PG = S::PG;
    constexpr int LAB = LA + LB, LCD = LC + LD, NR = (LAB + LCD) / 2 + 1;
    const int lane = (int)(threadIdx.x & 31);
    const int qslots = t.z <= 1 ? 1 : 1 << (32 - __clz(t.z - 1));
    const int UG = 32 / (PG * qslots);
    const int psub = lane & (PG - 1), usub = (lane / PG) & (UG - 1), qi = lane / (PG * UG);
    const bool live = psub < S::NPASS;
    const int pass = live ? psub : 0;
    const int mu0 = pass / S::NPB * NMU, nu0 = pass % S::NPB * NBU;

    const DevBasis &b = a.b;
    const int P = __ldg(u.bra_ids + t.x);
    const int2 sab = b.pair_shell[P];
    const double4 A = b.shell_xyz[sab.x], B = b.shell_xyz[sab.y];
    const R abx = R(A.x - B.x), aby = R(A.y - B.y), abz = R(A.z - B.z);
    const int p0 = b.pair_prim0[P], np = b.pair_nprim[P];
    bool act = qi < t.z && live;
    const int j = t.y + (qi < t.z ? qi : 0);
    if (act && u.rs.nsize > 1) {
        ClassArgs ca;
        ca.rs = u.rs;
        ca.bra_orig = u.bra_orig;
        ca.ket_orig = u.ket_orig;
        ca.swapped = u.swapped;
        act = quartet_owned(ca, t.x, j);
    }
    const double4 *krec = u.ket_rec + KET_REC * j;
    const double4 r0 = ldg_double4(krec), r1 = ldg_double4(krec + 1);
    const double4 C = make_double4(r0.w, r1.x, r1.y, 0.0);
    const R cdx = R(r0.x), cdy = R(r0.y), cdz = R(r0.z);
    const unsigned long long kbf = (unsigned long long)__double_as_longlong(r1.z);
    const unsigned long long kpr = (unsigned long long)__double_as_longlong(r1.w);
    const int q0 = (int)(unsigned)kpr, nprim = act ? np * (int)(unsigned)(kpr >> 32) : 0;

    // The Obara-Saika classes sum (e0|c0) (contract as in quartet.cuh, no roots
    // to share out), the others the (ab|cd) block of this pass.
    constexpr bool OS = os_class<LA, LB, LC, LD>() && NMU == S::NA && NBU == S::NB;
    constexpr int NE = OS ? nrange(LA, LAB) : NMU * NBU;
    R acc[NE][NC][ND];
#pragma unroll
    for (int e = 0; e < NE; e++)
#pragma unroll
        for (int ic = 0; ic < NC; ic++)
#pragma unroll
            for (int id = 0; id < ND; id++) acc[e][ic][id] = R(0);
    int ex[NMU], ey[NMU], ez[NMU];
#pragma unroll
    for (int m = 0; m < NMU; m++) {
        ex[m] = cx_rt(LA, mu0 + m);
        ey[m] = cy_rt(LA, mu0 + m);
        ez[m] = cz_rt(LA, mu0 + m);
    }
    // the quartet's UG lanes: over its primitive quartets first, over the
    // roots where there are more lanes than primitive quartets
    int up = UG;
    while (!OS && up > 1 && up > nprim) up >>= 1;
    const int ur = UG / up;
#pragma unroll 1
    for (int i = usub & (up - 1); i < nprim; i += up) {
        const int iq = i / np, kq = q0 + iq, kp = p0 + i - iq * np;
        if constexpr (std::is_same<R, double>::value) {
            const double4 Qp = ldg_double4(b.prim_P + kq), Pp = ldg_double4(b.prim_P + kp);
            const double2 Qx = b.prim_X[kq], Px = b.prim_X[kp];
            const double p = Pp.w, q = Qp.w, hp = Px.y, hq = Qx.y;
            const double pqx = Pp.x - Qp.x, pqy = Pp.y - Qp.y, pqz = Pp.z - Qp.z;
            const double rs = rsqrt(p + q), ipq = rs * rs;
            const double T = p * q * ipq * (pqx * pqx + pqy * pqy + pqz * pqz);
            const double pref = Px.x * Qx.x * rs;
            if constexpr (OS) {
                double c[LAB + LCD + 1];
                boys_eval<LAB + LCD>(T, a.tab, c);
                unit_os<LA, LB, LC>(c, pref, p, q, ipq, hp, pqx, pqy, pqz, Pp.x - A.x, Pp.y - A.y, Pp.z - A.z,
                                    Qp.x - C.x, Qp.y - C.y, Qp.z - C.z, acc);
            } else {
#pragma unroll 1
            for (int r = usub / up; r < NR; r += ur) {
                double ui, wr;
                rys_root<NR>(r, T, u.thr, u.strict != 0, a.tab, ui, wr);
                ui *= ipq;
                wr *= pref;
                const double fq = q * ui, fp = p * ui;
                const double b00 = 0.5 * ui, b10 = hp * (1.0 - fq), b01 = hq * (1.0 - fp);
                double gx[LAB + 1][LCD + 1], gy[LAB + 1][LCD + 1], gz[LAB + 1][LCD + 1];
                vrr<LAB, LCD, double>(gx, (Pp.x - A.x) - fq * pqx, (Qp.x - C.x) + fp * pqx, b10, b01, b00, 1.0);
                vrr<LAB, LCD, double>(gy, (Pp.y - A.y) - fq * pqy, (Qp.y - C.y) + fp * pqy, b10, b01, b00, 1.0);
                vrr<LAB, LCD, double>(gz, (Pp.z - A.z) - fq * pqz, (Qp.z - C.z) + fp * pqz, b10, b01, b00, wr);
                contract_unit<LA, LB, LC, LD, double, NMU, NBU>(gx, gy, gz, abx, aby, abz, cdx, cdy, cdz, ex, ey, ez, nu0,
                                                                reinterpret_cast<double(&)[NMU][NBU][NC][ND]>(acc));
            }
            }
        } else {
            // primitive screening of the FP32 tier (eval_block)
            if (a.prim_cut > 0.0 && a.maxd && b.prim_bound) {
                const double md = __longlong_as_double((long long)a.maxd[0]);
                if (md > 0.0 && __ldg(b.prim_bound + kp) * __ldg(b.prim_bound + kq) < (float)(a.prim_cut / md))
                    continue;
            }
            const float *__restrict__ PAf = reinterpret_cast<const float *>(b.prim_PAf);
            float4 Qp, Qa, Pp, Pa;
            ldg_v8f32(PAf + 8 * (size_t)kq, Qp, Qa);
            ldg_v8f32(PAf + 8 * (size_t)kp, Pp, Pa);
            const float p = Pp.w, q = Qp.w, hp = __fdividef(0.5f, p), hq = __fdividef(0.5f, q);
            const float pqx = Pp.x - Qp.x, pqy = Pp.y - Qp.y, pqz = Pp.z - Qp.z;
            const float rs = rsqrtf(p + q), ipq = rs * rs;
            const float T = p * q * ipq * (pqx * pqx + pqy * pqy + pqz * pqz);
            const float pref = Pa.w * Qa.w * rs;
            if constexpr (OS) {
                float c[LAB + LCD + 1];
                boys_eval<LAB + LCD>(T, a.tabf, c);
                unit_os<LA, LB, LC>(c, pref, p, q, ipq, hp, pqx, pqy, pqz, Pa.x, Pa.y, Pa.z, Qa.x, Qa.y, Qa.z, acc);
            } else {
#pragma unroll 1
            for (int r = usub / up; r < NR; r += ur) {
                float ui, wr;
                rys_root<NR>(r, T, (float)u.thr, u.strict != 0, a.tabf, ui, wr);
                ui *= ipq;
                wr *= pref;
                const float fq = q * ui, fp = p * ui;
                const float b00 = 0.5f * ui, b10 = hp * (1.0f - fq), b01 = hq * (1.0f - fp);
                float gx[LAB + 1][LCD + 1], gy[LAB + 1][LCD + 1], gz[LAB + 1][LCD + 1];
                vrr<LAB, LCD, float>(gx, Pa.x - fq * pqx, Qa.x + fp * pqx, b10, b01, b00, 1.0f);
                vrr<LAB, LCD, float>(gy, Pa.y - fq * pqy, Qa.y + fp * pqy, b10, b01, b00, 1.0f);
                vrr<LAB, LCD, float>(gz, Pa.z - fq * pqz, Qa.z + fp * pqz, b10, b01, b00, wr);
                contract_unit<LA, LB, LC, LD, float, NMU, NBU>(gx, gy, gz, abx, aby, abz, cdx, cdy, cdz, ex, ey, ez, nu0,
                                                               reinterpret_cast<float(&)[NMU][NBU][NC][ND]>(acc));
            }
            }
        }
    }
    __syncwarp();
#pragma unroll 1
    for (int o = PG; o < PG * UG; o <<= 1) {
#pragma unroll
        for (int e = 0; e < NE; e++)
#pragma unroll
            for (int ic = 0; ic < NC; ic++)
#pragma unroll
                for (int id = 0; id < ND; id++) acc[e][ic][id] += __shfl_xor_sync(0xffffffffu, acc[e][ic][id], o);
    }
    R blk[NMU][NBU][NC][ND];
#pragma unroll
    for (int m = 0; m < NMU; m++) {
        R sl[NBU][NC][1];
        if constexpr (OS && LB > 0) bra_transfer<LA, LB, LC, R>(reinterpret_cast<R(&)[NE][NC]>(acc), m, abx, aby, abz, sl);
#pragma unroll
        for (int n = 0; n < NBU; n++)
#pragma unroll
            for (int ic = 0; ic < NC; ic++)
#pragma unroll
                for (int id = 0; id < ND; id++) {
                    if constexpr (OS && LB > 0) blk[m][n][ic][id] = sl[n][ic][0];
                    else blk[m][n][ic][id] = acc[m * NBU + n][ic][id];
                }
    }
    QuartetCtx<R> qc;
    qc.bfA = b.shell_bf0[sab.x];
    qc.bfB = b.shell_bf0[sab.y];
    qc.bfC = (int)(unsigned)kbf;
    qc.bfD = (int)(unsigned)(kbf >> 32);
    qc.iandj = sab.x == sab.y;
    qc.kandl = qc.bfC == qc.bfD;
    qc.same = qc.bfA == qc.bfC && qc.bfB == qc.bfD;
    qc.cut = R(u.cut);
    if constexpr (std::is_same<R, double>::value) qc.Dm = a.Dm;
    else qc.Dm = a.Dmf;
    qc.DmK = qc.Dm + a.k_offset;
    qc.ld = (unsigned)a.nbf;
    R jab[NMU][NBU];
#pragma unroll
    for (int m = 0; m < NMU; m++)
#pragma unroll
        for (int n = 0; n < NBU; n++) jab[m][n] = R(0);
    double *F[NS];
    F[0] = a.F;
    if constexpr (NS > 1) F[1] = a.F2;
    if (act && usub == 0) digest_unit<LA, LB, LC, LD, R, NMU, NBU, NS>(blk, mu0, nu0, qc, a.k_offset, F, jab);
    __syncwarp();
    // the row pair's J: lanes of equal psub hold the same components
#pragma unroll
    for (int m = 0; m < NMU; m++)
#pragma unroll
        for (int n = 0; n < NBU; n++) {
            const R v = R(4) * warp_sum_strided<PG>(jab[m][n]);
            if (lane < PG && live)
#pragma unroll
                for (int s = 0; s < NS; s++) f_add(F[s], qc.bfA + mu0 + m, qc.bfB + nu0 + n, v);
        }
}

// The two register budgets of the merged launches: classes of at most two
// roots and small blocks (16 resident warps per SM), and the rest.
constexpr int UNIT_WARPS = 4;

template <bool LOW, typename R, int NS>
__global__ void __launch_bounds__(32 * UNIT_WARPS, LOW ? 4 : 2) unit_kernel(const __grid_constant__ UnitArgs a) {
    int c = 0;
    while (c + 1 < a.ncls && (int)blockIdx.x >= a.cls[c + 1].first_block) c++;
    const UnitClass &u = a.cls[c];
    const int task = ((int)blockIdx.x - u.first_block) * UNIT_WARPS + (int)(threadIdx.x >> 5);
    if (task >= (u.ntasks_dev ? *u.ntasks_dev : u.ntasks)) return;  // whole warps
    const int4 t = u.tasks[task];
#define LIBERI_U(kk, A, B, C, D) \
    case kk: \
        static_assert(UShape<A, B, C, D>::PG == UNIT_PG[kk], "the host plans with the kernel's pass lanes"); \
        if constexpr (unit_low(kk) == LOW) unit_task<A, B, C, D, R, NS>(a, u, t); \
        break;
    switch (u.k) {
        LIBERI_U(0, 0, 0, 0, 0) LIBERI_U(1, 1, 0, 0, 0) LIBERI_U(2, 1, 1, 0, 0) LIBERI_U(3, 1, 1, 1, 0)
        LIBERI_U(4, 1, 0, 1, 0) LIBERI_U(5, 1, 1, 1, 1) LIBERI_U(6, 2, 0, 0, 0) LIBERI_U(7, 2, 1, 0, 0)
        LIBERI_U(8, 2, 0, 1, 0) LIBERI_U(9, 2, 1, 1, 0) LIBERI_U(10, 2, 2, 0, 0) LIBERI_U(11, 2, 2, 1, 0)
        LIBERI_U(12, 1, 1, 2, 0) LIBERI_U(13, 2, 0, 2, 0) LIBERI_U(14, 2, 2, 1, 1) LIBERI_U(15, 2, 1, 2, 1)
        LIBERI_U(16, 2, 1, 2, 0) LIBERI_U(17, 2, 1, 1, 1) LIBERI_U(18, 2, 2, 2, 0) LIBERI_U(19, 2, 2, 2, 1)
        LIBERI_U(20, 2, 2, 2, 2)
        default: break;
    }
#undef LIBERI_U
}

template <bool LOW, typename R>
cudaError_t launch_unit_t(const UnitArgs &a, int blocks, cudaStream_t st) {
    if (a.F2) unit_kernel<LOW, R, 2><<<(unsigned)blocks, 32 * UNIT_WARPS, 0, st>>>(a);
    else unit_kernel<LOW, R, 1><<<(unsigned)blocks, 32 * UNIT_WARPS, 0, st>>>(a);
    return cudaGetLastError();
}

}  // namespace liberi
