// k_f.cu -- the 34 f-shell quartet classes of the reference's ENABLE_F block
// (src/liberi_driver.F90:103-160: the ERIC kernels int0030/0031/0032/1030 and
// the generated Rys kernels, src/rhf/eric, src/rhf/rys).
//
// An f quartet is too large for the thread-per-quartet class kernels ((ff|ff)
// holds 10,000 integrals and 7 roots), so a group of warps evaluates one
// shell quartet, with the class's angular momenta as compile-time parameters.
// Every class has a pair with an f shell; that pair (the larger one where
// both have) gives the rows: a lane owns one component (a, b) of it and holds
// that row's integrals over all components (c, d) of the other pair in
// registers.  Units of work are (primitive quartet, root):
//   1. one thread per (unit, axis): root and weight from the 7-root table, the
//      2D vertical recurrence and the transfer to shell B in registers, the
//      result h[a][b][f], f <= lc+ld, to shared memory;
//   2. every row lane reads its three h rows, transfers them to (c, d) in
//      registers and adds the products: two FMAs an integral and root and
//      3 (lc+ld+1) shared loads a root, where one thread per component read
//      three tables an integral and root.
// Digestion (DIRFCK rules, src/rhf/rys/int3011_rysgen.F90 digestion) runs on
// the same registers: a lane forms its sums for all six updates, those that
// several rows share are added up over the group (shuffles for the ket pair's
// J, shared memory for the K rows), and one FP64 atomic per function pair goes
// to F, about one for eight integrals instead of six each.  The six atomics
// an integral (4e9 a build of a 30-atom cluster, 187 G/s) and the tables' shared
// loads bounded the earlier form.  FP64 only: a mixed-precision build runs its
// f classes in FP64.
#include "quartet.cuh"

namespace liberi {

__host__ __device__ constexpr int fnc(int l) { return (l + 1) * (l + 2) / 2; }

// Shape of one class: rows (f, LB), kets (LC, LD).
//   SL  a ten-row class puts three slots of rows into a warp, each taking
//       every third unit
//   KS  a ket pair of more than 60 components ((ff|ff) alone) is split over
//       two sets of row lanes, so that a lane's block stays in registers
template <int LB_, int LC_, int LD_>
struct FR {
    static constexpr int LB = LB_, LC = LC_, LD = LD_;
    static constexpr int NB = fnc(LB), NC = fnc(LC), ND = fnc(LD), NROW = 10 * NB;
    static constexpr int NR = (3 + LB + LC + LD) / 2 + 1;
    static constexpr int F1 = LC + LD + 1, F1P = F1 | 1;  // odd row stride: no bank conflicts
    static constexpr int KS = NC * ND > 60 ? 2 : 1, NCS = NC / KS;
    static constexpr int SL = NROW == 10 ? 3 : 1;
    static constexpr int RT = (NROW + 31) / 32 * 32;  // row lanes of one split
    static constexpr int GT = RT * KS;                // threads per quartet
    static constexpr int BLOCK = GT == 32 ? 128 : GT, GROUPS = BLOCK / GT;
    static constexpr int UNIT = 3 * 4 * (LB + 1) * F1P;  // doubles of one unit's h rows
    static constexpr int UFIT = (GT == 32 ? 1280 : 5120) / UNIT;  // 10 KB a warp group, 40 KB a CTA group
    static constexpr int U = UFIT < 1 ? 1 : (UFIT < GT / 3 ? UFIT : GT / 3);  // units per round
    static constexpr int NK = 2 * (NCS + ND);            // K sums of a row
    static constexpr int KBUF = KS * NK * NROW;
    static constexpr int SMEM = U * UNIT > KBUF ? U * UNIT : KBUF;  // doubles per group
    // resident CTAs from what a lane holds: its block and two of the three 2D
    // tables, or the vertical recurrence of step 1
    static constexpr int HOLD_B = NCS * ND + 2 * (LC + 1) * (LD + 1), HOLD_A = (4 + LB) * F1;
    static constexpr int REGS_ = 2 * (HOLD_A > HOLD_B ? HOLD_A : HOLD_B) + 72;
    static constexpr int REGS = REGS_ > 255 ? 255 : REGS_;
    static constexpr int MINB_ = 65536 / (REGS * BLOCK);
    static constexpr int MINB = MINB_ < 1 ? 1 : MINB_;
};

namespace {

// Cartesian exponents of component i of a shell of angular momentum l (GAMESS
// order: p x,y,z; d xx,yy,zz,xy,xz,yz; f xxx,yyy,zzz,xxy,xxz,xyy,yyz,xzz,yzz,xyz)
__constant__ unsigned char c_cart[4][10][3] = {
    {{0, 0, 0}},
    {{1, 0, 0}, {0, 1, 0}, {0, 0, 1}},
    {{2, 0, 0}, {0, 2, 0}, {0, 0, 2}, {1, 1, 0}, {1, 0, 1}, {0, 1, 1}},
    {{3, 0, 0}, {0, 3, 0}, {0, 0, 3}, {2, 1, 0}, {2, 0, 1}, {1, 2, 0}, {0, 2, 1}, {1, 0, 2}, {0, 1, 2}, {1, 1, 1}}};
// the same as compile-time tables (digits x y of the f components)
__host__ __device__ constexpr int fx3(int i) {
    return i == 0 ? 3 : (i == 3 || i == 4) ? 2 : (i == 5 || i == 7 || i == 9) ? 1 : 0;
}
__host__ __device__ constexpr int fy3(int i) {
    return i == 1 ? 3 : (i == 5 || i == 6) ? 2 : (i == 3 || i == 8 || i == 9) ? 1 : 0;
}
__host__ __device__ constexpr int fcx(int l, int i) { return l == 3 ? fx3(i) : cxp(l, i); }
__host__ __device__ constexpr int fcy(int l, int i) { return l == 3 ? fy3(i) : cyp(l, i); }
__host__ __device__ constexpr int fcz(int l, int i) { return l - fcx(l, i) - fcy(l, i); }

// per-component normalisation relative to the axial component: sqrt3 on the
// mixed d, sqrt5 on the six mixed f and sqrt15 on xyz (int3011_rysgen.F90 d03bra)
__host__ __device__ constexpr double cnorm(int l, int i) {
    return l == 2 ? (i >= 3 ? 1.7320508075688772935 : 1.0)
         : l == 3 ? (i == 9 ? 3.8729833462074168852 : (i >= 3 ? 2.2360679774997896964 : 1.0))
                  : 1.0;
}

// root r and weight of the N-root Rys rule at T (large-T limit above thr,
// strict: T > thr, else T >= thr; always at and above the table's end)
template <int N>
__device__ __forceinline__ void rys7_root(int r, double T, double thr, bool strict, const double *tab, double &u,
                                          double &w) {
    const bool asym = (strict ? (T > thr) : (T >= thr)) || T >= RYS7_TMAX;
    if (asym) {
        const double it = 1.0 / T;
        const double *hr = tab + rys7_herm_off(N);
        u = __ldg(hr + r) * it;
        w = __ldg(hr + MAXROOT7 + r) * sqrt(it);
        return;
    }
    const double t4 = T * (double)RYS_PER_UNIT;
    const int k = (int)t4;
    const double x = 2.0 * (t4 - (double)k) - 1.0, x2 = x * x, x4 = x2 * x2;
    const double *base = tab + rys7_table_off(N) + (size_t)k * (2 * N * RYS_NCOEF) + r * RYS_NCOEF;
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

template <int GT>
__device__ __forceinline__ void group_sync() {
    if constexpr (GT == 32) __syncwarp();
    else __syncthreads();
}

// The shell quartet of pairs P (rows) and Q (kets).
struct FQuartet {
    double4 A, C;
    double AB[3], CD[3];
    int p0, np, q0, nq;
};
__device__ __forceinline__ FQuartet fquartet(const DevBasis &b, int P, int Q) {
    FQuartet f;
    const int2 sab = b.pair_shell[P], scd = b.pair_shell[Q];
    f.A = b.shell_xyz[sab.x];
    f.C = b.shell_xyz[scd.x];
    const double4 B = b.shell_xyz[sab.y], D = b.shell_xyz[scd.y];
    f.AB[0] = f.A.x - B.x, f.AB[1] = f.A.y - B.y, f.AB[2] = f.A.z - B.z;
    f.CD[0] = f.C.x - D.x, f.CD[1] = f.C.y - D.y, f.CD[2] = f.C.z - D.z;
    f.p0 = b.pair_prim0[P], f.np = b.pair_nprim[P];
    f.q0 = b.pair_prim0[Q], f.nq = b.pair_nprim[Q];
    return f;
}

// Step 1 for one (unit, axis): h[a][b][f] to hs (rows of F1P doubles).
template <typename S>
__device__ __forceinline__ void fstage(const DevBasis &b, const FQuartet &f, int unit, int x, double thr, bool strict,
                                       const double *__restrict__ tab7, double *hs) {
    constexpr int LB = S::LB, F1 = S::F1, E1 = 4 + LB;
    const int pq = unit / S::NR, r = unit - pq * S::NR;
    const int ip = pq / f.nq, iq = pq - ip * f.nq;
    const double4 Pp = ldg_double4(b.prim_P + f.p0 + ip), Qp = ldg_double4(b.prim_P + f.q0 + iq);
    const double2 Xp = b.prim_X[f.p0 + ip], Xq = b.prim_X[f.q0 + iq];
    const double p = Pp.w, q = Qp.w, rs = rsqrt(p + q), ipq = rs * rs;
    const double dx = Pp.x - Qp.x, dy = Pp.y - Qp.y, dz = Pp.z - Qp.z;
    const double T = p * q * ipq * (dx * dx + dy * dy + dz * dz);
    double u, w;
    rys7_root<S::NR>(r, T, thr, strict, tab7, u, w);
    u *= ipq;
    const double fq = q * u, fp = p * u;
    const double PA = x == 0 ? Pp.x - f.A.x : (x == 1 ? Pp.y - f.A.y : Pp.z - f.A.z);
    const double QC = x == 0 ? Qp.x - f.C.x : (x == 1 ? Qp.y - f.C.y : Qp.z - f.C.z);
    const double PQ = x == 0 ? dx : (x == 1 ? dy : dz);
    const double ab = x == 0 ? f.AB[0] : (x == 1 ? f.AB[1] : f.AB[2]);
    double g[E1][F1];
    vrr<E1 - 1, F1 - 1, double>(g, PA - fq * PQ, QC + fp * PQ, Xp.y * (1.0 - fq), Xq.y * (1.0 - fp), 0.5 * u,
                                x == 0 ? Xp.x * Xq.x * rs * w : 1.0);
#pragma unroll
    for (int k = 0; k < F1; k++) {
        double t[E1];
#pragma unroll
        for (int e = 0; e < E1; e++) t[e] = g[e][k];
#pragma unroll
        for (int bb = 0; bb <= LB; bb++) {
#pragma unroll
            for (int a = 0; a < 4; a++) hs[(a * (LB + 1) + bb) * S::F1P + k] = t[a];
#pragma unroll
            for (int e = 0; e + 1 < E1 - bb; e++) t[e] = fma(ab, t[e], t[e + 1]);
        }
    }
}

// the 2D integrals of one axis over (c, d) from a row of h
template <typename S>
__device__ __forceinline__ void fket(const double *hs, double cd, double (&I)[S::LC + 1][S::LD + 1]) {
    double t[S::F1];
#pragma unroll
    for (int k = 0; k < S::F1; k++) t[k] = hs[k];
#pragma unroll
    for (int d = 0; d <= S::LD; d++) {
#pragma unroll
        for (int c = 0; c <= S::LC; c++) I[c][d] = t[c];
#pragma unroll
        for (int k = 0; k + 1 < S::F1 - d; k++) t[k] = fma(cd, t[k], t[k + 1]);
    }
}

// Step 2 for one unit: the row's products for components C of split H.
template <typename S, int H>
__device__ __forceinline__ void fassemble(const double *h, int ox, int oy, int oz, const double (&CD)[3],
                                          double (&acc)[S::NCS][S::ND]) {
    constexpr int PL = S::UNIT / 3;
    double ix[S::LC + 1][S::LD + 1], iy[S::LC + 1][S::LD + 1], iz[S::LC + 1][S::LD + 1];
    fket<S>(h + ox, CD[0], ix);
    fket<S>(h + PL + oy, CD[1], iy);
    fket<S>(h + 2 * PL + oz, CD[2], iz);
#pragma unroll
    for (int c = 0; c < S::NCS; c++)
#pragma unroll
        for (int d = 0; d < S::ND; d++) {
            const int ic = H * S::NCS + c;
            acc[c][d] = fma(ix[fcx(S::LC, ic)][fcx(S::LD, d)] * iy[fcy(S::LC, ic)][fcy(S::LD, d)],
                            iz[fcz(S::LC, ic)][fcz(S::LD, d)], acc[c][d]);
        }
}

struct FShells {
    int bfA, bfB, bfC, bfD;
    bool iandj, kandl, same;
};

// unique-component loops and 0.5 factors (0: skipped) of coinciding shells
template <typename S>
__device__ __forceinline__ double ffactor(const FShells &s, int ia, int ib, int ic, int id) {
    if (S::LB == 3 && s.iandj && ib > ia) return 0.0;
    if (S::LC == S::LD && s.kandl && id > ic) return 0.0;
    if (S::LC == 3 && S::LD == S::LB && s.same) {
        const int pij = s.iandj ? ia * (ia + 1) / 2 + ib : ia * S::NB + ib;
        const int pkl = s.kandl ? ic * (ic + 1) / 2 + id : ic * S::ND + id;
        if (pkl > pij) return 0.0;
    }
    const int mu = s.bfA + ia, nu = s.bfB + ib, la = s.bfC + ic, si = s.bfD + id;
    double f = 1.0;
    if (mu == nu) f *= 0.5;
    if (la == si) f *= 0.5;
    if ((mu == la && nu == si) || (mu == si && nu == la)) f *= 0.5;
    return f;
}

__device__ __forceinline__ void fadd(double *F, unsigned i, unsigned j, double v) {
    if (v != 0.0) atomicAdd(F + tri0(i, j), v);
}

// Sums v[0..N-1] over the warp; the total of value i arrives at lane i (mod
// the padded length).  31 exchanges for 32 values.
template <int N>
__device__ __forceinline__ double warp_scatter_sum(double (&v)[N], int lane) {
    static_assert(N <= 32 && (N & (N - 1)) == 0, "padded to a power of two");
#pragma unroll
    for (int s = 16; s >= N; s >>= 1)
#pragma unroll
        for (int i = 0; i < N; i++) v[i] += __shfl_xor_sync(0xffffffffu, v[i], s);
#pragma unroll
    for (int s = N / 2; s >= 1; s >>= 1)
#pragma unroll
        for (int i = 0; i < s; i++) {
            const bool up = (lane & s) != 0;
            const double keep = up ? v[i + s] : v[i], send = up ? v[i] : v[i + s];
            v[i] = keep + __shfl_xor_sync(0xffffffffu, send, s);
        }
    return v[0];
}
constexpr int fpow2(int x) { return x <= 1 ? 1 : 2 * fpow2((x + 1) / 2); }

// Digestion of a lane's row over split H: the row pair's J at once, the ket
// pair's J over the warp, the row's K sums to kb[value][row].
template <typename S, int H>
__device__ __forceinline__ void fdigest(double (&acc)[S::NCS][S::ND], bool rowok, int row, int lane,
                                        const FShells &s, const ClassArgs &a, double *kb) {
    constexpr int NCS = S::NCS, ND = S::ND;
    const double *__restrict__ Dm = a.Dm, *__restrict__ Dk = a.Dm + a.k_offset;
    const unsigned n = (unsigned)a.nbf;
    const bool distinct = !s.iandj && !s.kandl && !s.same;
    const int ia = rowok ? row / S::NB : 0, ib = rowok ? row % S::NB : 0;
    const unsigned mu = s.bfA + ia, nu = s.bfB + ib;
    const double nab = cnorm(3, ia) * cnorm(S::LB, ib);
    const double dAB = 4.0 * dget(Dm, n, mu, nu);
    double jab = 0.0, dAD[ND], dBD[ND], kad[ND], kbd[ND];
#pragma unroll
    for (int d = 0; d < ND; d++) {
        dAD[d] = dget(Dk, n, mu, s.bfD + d);
        dBD[d] = dget(Dk, n, nu, s.bfD + d);
        kad[d] = kbd[d] = 0.0;
    }
#pragma unroll
    for (int c = 0; c < NCS; c++) {
        const int ic = H * NCS + c;
        const double dAC = dget(Dk, n, mu, s.bfC + ic), dBC = dget(Dk, n, nu, s.bfC + ic);
        double kac = 0.0, kbc = 0.0;
#pragma unroll
        for (int d = 0; d < ND; d++) {
            double v = acc[c][d] * (nab * (cnorm(S::LC, ic) * cnorm(S::LD, d)));
            v = !rowok || fabs(v) < a.cut ? 0.0 : v;
            if (!distinct) v *= ffactor<S>(s, ia, ib, ic, d);
            jab = fma(v, dget(Dm, n, s.bfC + ic, s.bfD + d), jab);
            kac = fma(v, dBD[d], kac);
            kad[d] = fma(v, dBC, kad[d]);
            kbc = fma(v, dAD[d], kbc);
            kbd[d] = fma(v, dAC, kbd[d]);
            acc[c][d] = v * dAB;
        }
        if (rowok) {
            kb[c * S::NROW + row] = kac;
            kb[(NCS + ND + c) * S::NROW + row] = kbc;
        }
    }
    if (rowok) {
#pragma unroll
        for (int d = 0; d < ND; d++) {
            kb[(NCS + d) * S::NROW + row] = kad[d];
            kb[(2 * NCS + ND + d) * S::NROW + row] = kbd[d];
        }
        fadd(a.F, mu, nu, 4.0 * jab);
    }
    constexpr int NV = NCS * ND;
#pragma unroll
    for (int v0 = 0; v0 < NV; v0 += 32) {
        constexpr int W = NV >= 32 ? 32 : fpow2(NV);
        double v[W];
#pragma unroll
        for (int i = 0; i < W; i++) v[i] = v0 + i < NV ? acc[(v0 + i) / ND][(v0 + i) % ND] : 0.0;
        const double t = warp_scatter_sum<W>(v, lane);
        const int i = v0 + lane;
        if (lane < W && i < NV) fadd(a.F, s.bfC + H * NCS + i / ND, s.bfD + i % ND, t);
    }
}

}  // namespace

// Task `task` of a group (CTA or warp).  SWAP: the class's ket pair holds the f
// shell and gives the rows.
template <typename S, bool SWAP>
__device__ __forceinline__ void fclass_task(const ClassArgs &a, const double *__restrict__ tab7, int block) {
    constexpr int GT = S::GT, NROW = S::NROW;
    const int grp = S::GROUPS > 1 ? (int)(threadIdx.x >> 5) : 0;
    const int task = block * S::GROUPS + grp;
    if (task >= a.ntasks) return;  // the whole group (only warp barriers follow where a CTA holds several)
    extern __shared__ __align__(16) double fsm[];
    double *sm = fsm + (size_t)grp * S::SMEM;
    const int tid = S::GROUPS > 1 ? (int)(threadIdx.x & 31) : (int)threadIdx.x, lane = tid & 31;
    const int half = S::KS > 1 ? tid / S::RT : 0, rt = tid - half * S::RT;
    const int slot = S::SL > 1 ? rt / NROW : 0, row = S::SL > 1 ? rt % NROW : rt;
    const bool rowok = S::SL > 1 ? rt < S::SL * NROW : rt < NROW;
    const int ia = rowok ? row / S::NB : 0, ib = rowok ? row % S::NB : 0;
    const int ox = (c_cart[3][ia][0] * (S::LB + 1) + c_cart[S::LB][ib][0]) * S::F1P;
    const int oy = (c_cart[3][ia][1] * (S::LB + 1) + c_cart[S::LB][ib][1]) * S::F1P;
    const int oz = (c_cart[3][ia][2] * (S::LB + 1) + c_cart[S::LB][ib][2]) * S::F1P;
    const int4 t = a.tasks[task];
    const DevBasis &b = a.b;

    for (int qi = 0; qi < t.z; qi++) {
        const int j = t.y + qi;
        if (a.rs.nsize > 1 && !quartet_owned(a, t.x, j)) continue;  // uniform over the group
        const int pb = a.bra_ids[t.x], pk = a.ket_ids[j];
        const int P = SWAP ? pk : pb, Q = SWAP ? pb : pk;
        const FQuartet f = fquartet(b, P, Q);
        double acc[S::NCS][S::ND];
#pragma unroll
        for (int c = 0; c < S::NCS; c++)
#pragma unroll
            for (int d = 0; d < S::ND; d++) acc[c][d] = 0.0;
        const int nunit = f.np * f.nq * S::NR;
#pragma unroll 1
        for (int u0 = 0; u0 < nunit; u0 += S::U) {
            const int nu = min(S::U, nunit - u0);
            if (tid < 3 * nu) {
                const int uu = tid / 3, x = tid - 3 * uu;
                fstage<S>(b, f, u0 + uu, x, a.thr, a.strict, tab7, sm + uu * S::UNIT + x * (S::UNIT / 3));
            }
            group_sync<GT>();
            if (rowok) {
#pragma unroll 1
                for (int u = slot; u < nu; u += S::SL) {
                    const double *h = sm + u * S::UNIT;
                    if (S::KS == 1 || half == 0) fassemble<S, 0>(h, ox, oy, oz, f.CD, acc);
                    else fassemble<S, S::KS - 1>(h, ox, oy, oz, f.CD, acc);
                }
            }
            group_sync<GT>();
        }
        if constexpr (S::SL > 1) {  // the slots' partial rows
            static_assert(S::SL == 3, "lanes row, row + NROW, row + 2 NROW");
#pragma unroll
            for (int c = 0; c < S::NCS; c++)
#pragma unroll
                for (int d = 0; d < S::ND; d++) {
                    const double v = acc[c][d];
                    acc[c][d] = v + __shfl_down_sync(0xffffffffu, v, NROW) + __shfl_down_sync(0xffffffffu, v, 2 * NROW);
                }
        }
        const int2 sab = b.pair_shell[P], scd = b.pair_shell[Q];
        FShells s;
        s.bfA = b.shell_bf0[sab.x], s.bfB = b.shell_bf0[sab.y];
        s.bfC = b.shell_bf0[scd.x], s.bfD = b.shell_bf0[scd.y];
        s.iandj = sab.x == sab.y;
        s.kandl = scd.x == scd.y;
        s.same = sab.x == scd.x && sab.y == scd.y;
        const bool own = rowok && slot == 0;
        double *kb = sm + half * (S::NK * NROW);
        if (S::KS == 1 || half == 0) fdigest<S, 0>(acc, own, row, lane, s, a, kb);
        else fdigest<S, S::KS - 1>(acc, own, row, lane, s, a, kb);
        group_sync<GT>();
        // the K sums over B (rows of A) and over A (rows of B)
        constexpr int NV = S::NCS + S::ND, RT = S::RT;
        for (int i = rt; i < 10 * NV; i += RT) {
            const int v = i / 10, r = i - 10 * v;
            double sum = 0.0;
            for (int k = 0; k < S::NB; k++) sum += kb[v * NROW + r * S::NB + k];
            const int col = v < S::NCS ? s.bfC + half * S::NCS + v : s.bfD + v - S::NCS;
            fadd(a.F, s.bfA + r, col, -sum);
        }
        for (int i = rt; i < S::NB * NV; i += RT) {
            const int v = i / S::NB, r = i - S::NB * v;
            double sum = 0.0;
            for (int k = 0; k < 10; k++) sum += kb[(NV + v) * NROW + k * S::NB + r];
            const int col = v < S::NCS ? s.bfC + half * S::NCS + v : s.bfD + v - S::NCS;
            fadd(a.F, s.bfB + r, col, -sum);
        }
        if (t.z > 1) group_sync<GT>();
    }
}

template <typename S, bool SWAP>
__global__ void __launch_bounds__(S::BLOCK, S::MINB) fclass_kernel(const __grid_constant__ ClassArgs a,
                                                                   const double *__restrict__ tab7) {
    fclass_task<S, SWAP>(a, tab7, (int)blockIdx.x);
}

// shape of a class by its engine orientation: the rows are the bra pair where
// that holds an f shell, else the ket pair
template <int LA, int LB, int LC, int LD>
struct FShape {
    static constexpr bool SWAP = LA < 3;
    static_assert(SWAP ? LC == 3 : LB >= LD || LC < 3, "rows: the larger f pair");
    using S = typename std::conditional<SWAP, FR<LD, LA, LB>, FR<LB, LC, LD>>::type;
};
#define LIBERI_FCLASSES(X)                                                                                          \
    X(21, 3, 3, 3, 3) X(22, 0, 0, 3, 0) X(23, 0, 0, 3, 1) X(24, 0, 0, 3, 2) X(25, 1, 0, 3, 0) X(26, 3, 3, 3, 0)         \
    X(27, 3, 0, 1, 1) X(28, 3, 0, 2, 0) X(29, 2, 1, 3, 0) X(30, 2, 2, 3, 0) X(31, 3, 0, 3, 0) X(32, 3, 1, 1, 0)         \
    X(33, 3, 1, 1, 1) X(34, 3, 1, 2, 0) X(35, 3, 1, 2, 1) X(36, 2, 2, 3, 1) X(37, 3, 1, 3, 0) X(38, 3, 1, 3, 1)         \
    X(39, 3, 2, 1, 0) X(40, 3, 3, 3, 1) X(41, 3, 2, 1, 1) X(42, 3, 2, 2, 0) X(43, 3, 2, 2, 1) X(44, 3, 2, 2, 2)         \
    X(45, 3, 2, 3, 0) X(46, 3, 2, 3, 1) X(47, 3, 2, 3, 2) X(48, 3, 3, 0, 0) X(49, 3, 3, 1, 0) X(50, 3, 3, 1, 1)         \
    X(51, 3, 3, 2, 0) X(52, 3, 3, 2, 1) X(53, 3, 3, 2, 2) X(54, 3, 3, 3, 2)

// Small builds: all classes of one CTA size (128 threads of warp groups, or
// one group of 64, 128 or 256) in one launch; 34 launches of a few quartets
// each were mostly launch time.
struct FGroup {
    const double *tab7;
    int n;
    int k[NKERN_F], first_block[NKERN_F];
    ClassArgs a[NKERN_F];
};
template <typename S, bool SWAP>
__device__ __noinline__ void fgroup_task(const ClassArgs &a, const double *tab7, int block) {
    fclass_task<S, SWAP>(a, tab7, block);
}
template <int GT>
__global__ void __launch_bounds__(GT == 32 ? 128 : GT) fgroup_kernel(const __grid_constant__ FGroup g) {
    int c = 0;
    while (c + 1 < g.n && (int)blockIdx.x >= g.first_block[c + 1]) c++;
    const int block = (int)blockIdx.x - g.first_block[c];
#define LIBERI_F(kk, A, B, C, D)                                                                     \
    case kk:                                                                                        \
        if constexpr (FShape<A, B, C, D>::S::GT == GT)                                               \
            fgroup_task<typename FShape<A, B, C, D>::S, FShape<A, B, C, D>::SWAP>(g.a[c], g.tab7, block); \
        break;
    switch (g.k[c]) { LIBERI_FCLASSES(LIBERI_F) }
#undef LIBERI_F
}

// Schwarz values of f pairs: one group per pair P of one class, the diagonal
// (ab|ab) of the (P|P) block (one value a row lane), then sqrt(max over
// components |(ab|ab)|) of the normalised integrals into out[P].
template <typename S>
__global__ void __launch_bounds__(S::BLOCK) fschwarz_kernel(DevBasis b, int pair_off, int npairs,
                                                            const double *__restrict__ tab7, double *out) {
    constexpr int GT = S::GT, NROW = S::NROW, PL = S::UNIT / 3;
    const int grp = S::GROUPS > 1 ? (int)(threadIdx.x >> 5) : 0;
    const int item = (int)blockIdx.x * S::GROUPS + grp;
    if (item >= npairs) return;
    extern __shared__ __align__(16) double fsm[];
    __shared__ double wmax[S::BLOCK / 32];
    double *sm = fsm + (size_t)grp * S::SMEM;
    const int tid = S::GROUPS > 1 ? (int)(threadIdx.x & 31) : (int)threadIdx.x;
    // (the ket splits of the block's shape are more slots here)
    constexpr int SLOTS = S::SL > 1 ? S::SL : S::KS, STRIDE = S::SL > 1 ? NROW : S::RT;
    const int slot = tid / STRIDE, row = tid % STRIDE;
    const bool rowok = slot < SLOTS && row < NROW;
    int e[3][2] = {};
    if (rowok)
        for (int x = 0; x < 3; x++) {
            e[x][0] = c_cart[3][row / S::NB][x];
            e[x][1] = c_cart[S::LB][row % S::NB][x];
        }
    const int P = pair_off + item;
    const FQuartet f = fquartet(b, P, P);
    double acc = 0.0;
    const int nunit = f.np * f.nq * S::NR;
    for (int u0 = 0; u0 < nunit; u0 += S::U) {
        const int nu = min(S::U, nunit - u0);
        if (tid < 3 * nu) {
            const int uu = tid / 3, x = tid - 3 * uu;
            fstage<S>(b, f, u0 + uu, x, RYS7_TMAX, false, tab7, sm + uu * S::UNIT + x * PL);
        }
        group_sync<GT>();
        if (rowok)
            for (int u = slot; u < nu; u += SLOTS) {
                double prod = 1.0;
                for (int x = 0; x < 3; x++) {
                    const double *h = sm + u * S::UNIT + x * PL + (e[x][0] * (S::LB + 1) + e[x][1]) * S::F1P + e[x][0];
                    double t[4] = {0.0, 0.0, 0.0, 0.0};
                    for (int k = 0; k <= e[x][1]; k++) t[k] = h[k];
                    for (int d = e[x][1]; d > 0; d--)
                        for (int k = 0; k < d; k++) t[k] = fma(f.CD[x], t[k], t[k + 1]);
                    prod *= t[0];
                }
                acc += prod;
            }
        group_sync<GT>();
    }
    // the slots' partial sums through shared memory, then the maximum
    if (rowok) sm[slot * NROW + row] = acc;
    group_sync<GT>();
    double mx = 0.0;
    if (rowok && slot == 0) {
        for (int k = 1; k < SLOTS; k++) acc += sm[k * NROW + row];
        const double nrm = cnorm(3, row / S::NB) * cnorm(S::LB, row % S::NB);
        mx = fabs(acc) * nrm * nrm;
    }
    for (int o = 16; o > 0; o >>= 1) mx = fmax(mx, __shfl_xor_sync(0xffffffffu, mx, o));
    if constexpr (GT > 32) {
        if ((threadIdx.x & 31) == 0) wmax[threadIdx.x >> 5] = mx;
        __syncthreads();
        for (int w = 0; w < GT / 32; w++) mx = fmax(mx, wmax[w]);
    }
    if (tid == 0) out[P] = sqrt(mx);
}

template <int LF>
static cudaError_t fschwarz_t(int npairs, int pair_off, const DevBasis &b, const double *tab7, double *out,
                              cudaStream_t stream) {
    using S = FR<LF, 3, LF>;
    const size_t smem = (size_t)S::GROUPS * S::SMEM * sizeof(double);
    static FuncAttrs attrs;
    cudaError_t e = attrs.set((const void *)fschwarz_kernel<S>, (int)smem, -1);
    if (e != cudaSuccess) return e;
    fschwarz_kernel<S><<<(unsigned)((npairs + S::GROUPS - 1) / S::GROUPS), S::BLOCK, smem, stream>>>(b, pair_off, npairs,
                                                                                                   tab7, out);
    return cudaGetLastError();
}

cudaError_t launch_fschwarz(int pair_class, int npairs, int pair_off, const DevBasis &b, const double *rys_tab7,
                            double *out, cudaStream_t stream) {
    if (npairs <= 0) return cudaSuccess;
    if (!rys_tab7) return cudaErrorInvalidValue;
    switch (pair_class) {  // sf, pf, df, ff: the lower-L shell s, p, d, f
        case SF: return fschwarz_t<0>(npairs, pair_off, b, rys_tab7, out, stream);
        case PF: return fschwarz_t<1>(npairs, pair_off, b, rys_tab7, out, stream);
        case DF: return fschwarz_t<2>(npairs, pair_off, b, rys_tab7, out, stream);
        case FF: return fschwarz_t<3>(npairs, pair_off, b, rys_tab7, out, stream);
        default: return cudaErrorInvalidValue;
    }
}

// one class
template <int LA, int LB, int LC, int LD>
static cudaError_t fclass_t(const ClassArgs &a, const double *tab7, cudaStream_t stream) {
    using S = typename FShape<LA, LB, LC, LD>::S;
    constexpr bool SWAP = FShape<LA, LB, LC, LD>::SWAP;
    const size_t smem = (size_t)S::GROUPS * S::SMEM * sizeof(double);
    static FuncAttrs attrs;
    cudaError_t e = attrs.set((const void *)fclass_kernel<S, SWAP>, (int)smem, -1);
    if (e != cudaSuccess) return e;
    const unsigned grid = (unsigned)((a.ntasks + S::GROUPS - 1) / S::GROUPS);
    fclass_kernel<S, SWAP><<<grid, S::BLOCK, smem, stream>>>(a, tab7);
    return cudaGetLastError();
}

static ClassArgs fclass_args(int k, const LaunchCtx &ctx, const DevPlan &plan, const RankSplit &rs, int nbf) {
    const KernelDesc &kd = KDESC[k];
    ClassArgs a{};
    a.b = ctx.basis;
    a.Dm = ctx.D;
    a.F = ctx.F;
    a.cut = kd.digest_schwarz ? ctx.schwarz_cut : ctx.eri_cut;
    a.thr = kd.asym;
    a.strict = !kd.rys;
    a.tasks = plan.tasks;
    a.ntasks = plan.ntasks;
    a.nbf = nbf;
    a.bra_ids = plan.bra_ids;
    a.ket_ids = plan.ket_ids;
    a.bra_orig = plan.bra_orig;
    a.ket_orig = plan.ket_orig;
    a.ket_rec = plan.ket_rec;
    a.swapped = plan.swapped;
    a.rs = rs;
    a.k_offset = ctx.k_offset;
    return a;
}

cudaError_t launch_fclass(int k, const LaunchCtx &ctx, const DevPlan &plan, const RankSplit &rs, int nbf) {
    if (plan.ntasks <= 0) return cudaSuccess;
    const ClassArgs a = fclass_args(k, ctx, plan, rs, nbf);
#define LIBERI_F(kk, A, B, C, D) \
    case kk: return fclass_t<A, B, C, D>(a, ctx.rys_tab7, ctx.stream);
    switch (k) {
        LIBERI_FCLASSES(LIBERI_F)
        default: return cudaErrorInvalidValue;
    }
#undef LIBERI_F
}

// CTA size, groups per CTA and shared bytes of class k
static void fclass_shape(int k, int &gt, int &groups, size_t &smem) {
#define LIBERI_F(kk, A, B, C, D)                                                      \
    case kk:                                                                         \
        gt = FShape<A, B, C, D>::S::GT;                                               \
        groups = FShape<A, B, C, D>::S::GROUPS;                                       \
        smem = sizeof(double) * (size_t)groups * FShape<A, B, C, D>::S::SMEM;         \
        break;
    switch (k) {
        LIBERI_FCLASSES(LIBERI_F)
        default: gt = 0; groups = 1; smem = 0;
    }
#undef LIBERI_F
}

template <int GT>
static cudaError_t fgroup_t(const FGroup &g, int blocks, size_t smem, cudaStream_t stream) {
    static FuncAttrs attrs;
    cudaError_t e = attrs.set((const void *)fgroup_kernel<GT>, 96 * 1024, -1);  // above every class's need
    if (e != cudaSuccess) return e;
    fgroup_kernel<GT><<<(unsigned)blocks, GT == 32 ? 128 : GT, smem, stream>>>(g);
    return cudaGetLastError();
}

int fclass_threads(int k) {
    int gt, groups;
    size_t bytes;
    fclass_shape(k, gt, groups, bytes);
    return gt;
}

cudaError_t launch_fgroup(int gt, int n, const int *ks, const LaunchCtx &ctx, const DevPlan *plans,
                          const RankSplit *rs, int nbf) {
    FGroup g{};
    g.tab7 = ctx.rys_tab7;
    int blocks = 0;
    size_t smem = 0;
    for (int i = 0; i < n; i++) {
        int t, groups;
        size_t bytes;
        fclass_shape(ks[i], t, groups, bytes);
        if (t != gt) return cudaErrorInvalidValue;
        if (plans[i].ntasks <= 0) continue;
        g.k[g.n] = ks[i];
        g.first_block[g.n] = blocks;
        g.a[g.n++] = fclass_args(ks[i], ctx, plans[i], rs[i], nbf);
        blocks += (plans[i].ntasks + groups - 1) / groups;
        smem = bytes > smem ? bytes : smem;
    }
    if (blocks == 0) return cudaSuccess;
    switch (gt) {
        case 32: return fgroup_t<32>(g, blocks, smem, ctx.stream);
        case 64: return fgroup_t<64>(g, blocks, smem, ctx.stream);
        case 128: return fgroup_t<128>(g, blocks, smem, ctx.stream);
        case 256: return fgroup_t<256>(g, blocks, smem, ctx.stream);
        default: return cudaErrorInvalidValue;
    }
}

}  // namespace liberi
