// k_s.cu -- Schwarz values and primitive bounds of the s/p/d shell pairs.
//
// One warp per pair, all six pair classes in one launch.  The lanes share the
// pair's primitive quartets (np^2 of them, up to 1,296 for two six-primitive
// s shells) and each adds the diagonal components (ab|ab) only, so of the
// transfer's 2D integrals just I[a][b][a][b] are formed; the warp sums the
// components and takes the largest.  A thread per pair, one pass per
// component of A and six launches, left the table of a 40-atom molecule
// waiting for single threads (400 us for the costliest (ss|ss) pair).
#include "unit.cuh"

namespace liberi {

// one primitive quartet of a pair (primitive pairs (Pp, Px) and (Qp, Qx)): its
// roots' diagonal products
template <int LA, int LB>
__device__ __forceinline__ void diag_add(const double4 &Pp, const double2 &Px, const double4 &Qp, const double2 &Qx,
                                         const double4 &A, double abx, double aby, double abz,
                                         const double *__restrict__ tab, double (&acc)[ncart(LA)][ncart(LB)]) {
    constexpr int L = LA + LB, NR = L + 1;
    const double p = Pp.w, q = Qp.w, rs = rsqrt(p + q), ipq = rs * rs;
    const double pqx = Pp.x - Qp.x, pqy = Pp.y - Qp.y, pqz = Pp.z - Qp.z;
    const double T = p * q * ipq * (pqx * pqx + pqy * pqy + pqz * pqz);
    const double pref = Px.x * Qx.x * rs;
#pragma unroll 1
    for (int r = 0; r < NR; r++) {
        double u, w;
        rys_root<NR>(r, T, RYS_TMAX, false, tab, u, w);
        u *= ipq;
        const double fq = q * u, fp = p * u, b00 = 0.5 * u, b10 = Px.y * (1.0 - fq), b01 = Qx.y * (1.0 - fp);
        double g[L + 1][L + 1], ix[LA + 1][LB + 1][LA + 1][LB + 1], iy[LA + 1][LB + 1][LA + 1][LB + 1],
            iz[LA + 1][LB + 1][LA + 1][LB + 1];
        vrr<L, L, double>(g, (Pp.x - A.x) - fq * pqx, (Qp.x - A.x) + fp * pqx, b10, b01, b00, 1.0);
        hrr<LA, LB, LA, LB, double>(g, abx, abx, ix);
        vrr<L, L, double>(g, (Pp.y - A.y) - fq * pqy, (Qp.y - A.y) + fp * pqy, b10, b01, b00, 1.0);
        hrr<LA, LB, LA, LB, double>(g, aby, aby, iy);
        vrr<L, L, double>(g, (Pp.z - A.z) - fq * pqz, (Qp.z - A.z) + fp * pqz, b10, b01, b00, w * pref);
        hrr<LA, LB, LA, LB, double>(g, abz, abz, iz);
#pragma unroll
        for (int ia = 0; ia < ncart(LA); ia++)
#pragma unroll
            for (int ib = 0; ib < ncart(LB); ib++) {
                const int ax = cxp(LA, ia), ay = cyp(LA, ia), az = czp(LA, ia);
                const int bx = cxp(LB, ib), by = cyp(LB, ib), bz = czp(LB, ib);
                acc[ia][ib] += ix[ax][bx][ax][bx] * iy[ay][by][ay][by] * iz[az][bz][az][bz];
            }
    }
}

// The largest normalised diagonal component of the warp's summed block.
template <int LA, int LB>
__device__ __forceinline__ double diag_max(const double (&acc)[ncart(LA)][ncart(LB)]) {
    __syncwarp();
    double m = 0.0;
#pragma unroll
    for (int ia = 0; ia < ncart(LA); ia++)
#pragma unroll
        for (int ib = 0; ib < ncart(LB); ib++)
            m = fmax(m, fabs(warp_sum(acc[ia][ib])) * s3pow(2 * (cs3(LA, ia) + cs3(LB, ib))));
    return m;
}

// BOUND: out[k] for every primitive pair k, the bound of that primitive alone
// rounded up to float; else out[P], the pair's Schwarz value.
template <int LA, int LB, bool BOUND>
__device__ __noinline__ void schwarz_pair(const DevBasis &b, int P, const double *__restrict__ tab, double *out,
                                          float *outf) {
    constexpr int NA = ncart(LA), NB = ncart(LB);
    const int lane = (int)(threadIdx.x & 31);
    const int2 sab = b.pair_shell[P];
    const double4 A = b.shell_xyz[sab.x], B = b.shell_xyz[sab.y];
    const double abx = A.x - B.x, aby = A.y - B.y, abz = A.z - B.z;
    const int p0 = b.pair_prim0[P], np = b.pair_nprim[P], n = BOUND ? np : np * np;
    double acc[NA][NB];
#pragma unroll
    for (int ia = 0; ia < NA; ia++)
#pragma unroll
        for (int ib = 0; ib < NB; ib++) acc[ia][ib] = 0.0;
#pragma unroll 1
    for (int i = lane; i < n; i += 32) {
        const int iq = BOUND ? i : i / np, ip = BOUND ? i : i - iq * np;
        diag_add<LA, LB>(ldg_double4(b.prim_P + p0 + ip), b.prim_X[p0 + ip], ldg_double4(b.prim_P + p0 + iq),
                         b.prim_X[p0 + iq], A, abx, aby, abz, tab, acc);
        if (BOUND) {
            double m = 0.0;
#pragma unroll
            for (int ia = 0; ia < NA; ia++)
#pragma unroll
                for (int ib = 0; ib < NB; ib++) {
                    m = fmax(m, fabs(acc[ia][ib]) * s3pow(2 * (cs3(LA, ia) + cs3(LB, ib))));
                    acc[ia][ib] = 0.0;
                }
            outf[p0 + i] = __double2float_ru(sqrt(m) * (1.0 + 1e-6));
        }
    }
    if (BOUND) return;
    const double m = diag_max<LA, LB>(acc);
    if (lane == 0) out[P] = sqrt(m);
}

struct PairClasses {
    int off[NPC_SPD + 1];  // global pair index of each class's first pair
};

template <bool BOUND>
__global__ void __launch_bounds__(128) schwarz_kernel(const __grid_constant__ DevBasis b, PairClasses pc, const double *__restrict__ tab,
                                                      double *out, float *outf) {
    // the costliest classes (high L, one warp's longest chains) first
    const int P = pc.off[NPC_SPD] - 1 - ((int)blockIdx.x * 4 + (int)(threadIdx.x >> 5));
    if (P < 0) return;  // whole warps
    if (P >= pc.off[DD]) schwarz_pair<2, 2, BOUND>(b, P, tab, out, outf);
    else if (P >= pc.off[PD]) schwarz_pair<2, 1, BOUND>(b, P, tab, out, outf);
    else if (P >= pc.off[SD]) schwarz_pair<2, 0, BOUND>(b, P, tab, out, outf);
    else if (P >= pc.off[PP]) schwarz_pair<1, 1, BOUND>(b, P, tab, out, outf);
    else if (P >= pc.off[SP]) schwarz_pair<1, 0, BOUND>(b, P, tab, out, outf);
    else schwarz_pair<0, 0, BOUND>(b, P, tab, out, outf);
}

// Schwarz values straight from the shells, for a table without a handle: the
// warp forms its pair's primitive pairs itself (the host's pair construction
// and the upload of its arrays, 80,000 primitive pairs for 40 atoms, took most
// of such a call).  Primitives are staged in shared memory 32 at a time, the
// dropped ones (mu R^2 > cux) left out.
constexpr int SZ_WARPS = 4;
struct PrimTile {
    double4 P[32];
    double2 X[32];
};
template <int LA, int LB>
__device__ __forceinline__ int prim_tile(const ShellTable &t, const int4 &sa, const int4 &sb, const double4 &A,
                                         const double4 &B, int k0, double r2, PrimTile &pt) {
    const int lane = (int)(threadIdx.x & 31), k = k0 + lane;
    bool keep = k < sa.y * sb.y;
    double4 P = make_double4(0.0, 0.0, 0.0, 1.0);
    double2 X = make_double2(0.0, 0.0);
    if (keep) {
        const int i = k / sb.y, j = k - i * sb.y;
        const double a = t.exps[sa.z + i], b = t.exps[sb.z + j], p = a + b, ip = 1.0 / p;
        const double mur2 = r2 * (a * ip) * b;
        keep = mur2 <= t.cux;
        P = make_double4((a * A.x + b * B.x) * ip, (a * A.y + b * B.y) * ip, (a * A.z + b * B.z) * ip, p);
        X = make_double2(t.pref * t.coefs[sa.z + i] * t.coefs[sb.z + j] * exp(-mur2) * ip, 0.5 * ip);
    }
    const unsigned mask = __ballot_sync(0xffffffffu, keep);
    __syncwarp();
    if (keep) {
        const int o = __popc(mask & ((1u << lane) - 1u));
        pt.P[o] = P;
        pt.X[o] = X;
    }
    __syncwarp();
    return __popc(mask);
}
template <int LA, int LB>
__device__ __noinline__ double schwarz_shells(const ShellTable &t, int s1, int s2, PrimTile *pt) {
    const int4 sa = t.shell[s1], sb = t.shell[s2];
    const double4 A = t.xyz[s1], B = t.xyz[s2];
    const double abx = A.x - B.x, aby = A.y - B.y, abz = A.z - B.z;
    const double r2 = abx * abx + aby * aby + abz * abz;
    double acc[ncart(LA)][ncart(LB)];
#pragma unroll
    for (int ia = 0; ia < ncart(LA); ia++)
#pragma unroll
        for (int ib = 0; ib < ncart(LB); ib++) acc[ia][ib] = 0.0;
    const int n = sa.y * sb.y;
    for (int kq = 0; kq < n; kq += 32) {
        const int nq = prim_tile<LA, LB>(t, sa, sb, A, B, kq, r2, pt[0]);
        for (int kp = 0; kp < n; kp += 32) {
            const int np = kp == kq ? nq : prim_tile<LA, LB>(t, sa, sb, A, B, kp, r2, pt[1]);
            const PrimTile &tp = kp == kq ? pt[0] : pt[1];
#pragma unroll 1
            for (int i = (int)(threadIdx.x & 31); i < np * nq; i += 32) {
                const int iq = i / np, ip = i - iq * np;
                diag_add<LA, LB>(tp.P[ip], tp.X[ip], pt[0].P[iq], pt[0].X[iq], A, abx, aby, abz, t.tab, acc);
            }
        }
    }
    return diag_max<LA, LB>(acc);
}
__global__ void __launch_bounds__(32 * SZ_WARPS) schwarz_shells_kernel(const __grid_constant__ ShellTable t, int npairs,
                                                                       double *out) {
    __shared__ PrimTile tiles[SZ_WARPS][2];
    const int w = (int)(threadIdx.x >> 5), pair = (int)blockIdx.x * SZ_WARPS + w;
    if (pair >= npairs) return;  // whole warps
    int i = (int)((sqrt(8.0 * pair + 1.0) - 1.0) * 0.5);  // pair = i (i + 1) / 2 + j
    while ((long long)i * (i + 1) / 2 > pair) i--;
    while ((long long)(i + 1) * (i + 2) / 2 <= pair) i++;
    const int j = pair - (int)((long long)i * (i + 1) / 2);
    const int li = t.shell[i].x, lj = t.shell[j].x;
    const int s1 = li >= lj ? i : j, s2 = li >= lj ? j : i;  // higher L first
    double m = 0.0;
    switch (t.shell[s1].x * 3 + t.shell[s2].x) {
        case 0: m = schwarz_shells<0, 0>(t, s1, s2, tiles[w]); break;
        case 3: m = schwarz_shells<1, 0>(t, s1, s2, tiles[w]); break;
        case 4: m = schwarz_shells<1, 1>(t, s1, s2, tiles[w]); break;
        case 6: m = schwarz_shells<2, 0>(t, s1, s2, tiles[w]); break;
        case 7: m = schwarz_shells<2, 1>(t, s1, s2, tiles[w]); break;
        case 8: m = schwarz_shells<2, 2>(t, s1, s2, tiles[w]); break;
        default: break;
    }
    if ((threadIdx.x & 31) == 0) out[pair] = sqrt(m);
}
cudaError_t launch_schwarz_shells(const ShellTable &t, int nsh, double *out, cudaStream_t st) {
    const long long npairs = (long long)nsh * (nsh + 1) / 2;
    if (npairs <= 0) return cudaSuccess;
    schwarz_shells_kernel<<<(unsigned)((npairs + SZ_WARPS - 1) / SZ_WARPS), 32 * SZ_WARPS, 0, st>>>(t, (int)npairs, out);
    return cudaGetLastError();
}

static PairClasses pair_classes(const int *class_off) {
    PairClasses pc;
    for (int c = 0; c <= NPC_SPD; c++) pc.off[c] = class_off[c];
    return pc;
}

cudaError_t launch_schwarz(const int *class_off, const DevBasis &b, const double *tab, double *out, cudaStream_t st) {
    const int npairs = class_off[NPC_SPD];
    if (npairs <= 0) return cudaSuccess;
    schwarz_kernel<false><<<(unsigned)((npairs + 3) / 4), 128, 0, st>>>(b, pair_classes(class_off), tab, out, nullptr);
    return cudaGetLastError();
}

cudaError_t launch_prim_bound(const int *class_off, const DevBasis &b, const double *tab, float *out, cudaStream_t st) {
    const int npairs = class_off[NPC_SPD];
    if (npairs <= 0) return cudaSuccess;
    schwarz_kernel<true><<<(unsigned)((npairs + 3) / 4), 128, 0, st>>>(b, pair_classes(class_off), tab, nullptr, out);
    return cudaGetLastError();
}

}  // namespace liberi
