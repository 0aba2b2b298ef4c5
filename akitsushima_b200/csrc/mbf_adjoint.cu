// Tersoff adjoint: the vector-Jacobian product of (E, F, virial) with
// respect to the dense parameter tables, for fitting.
//
// With upstream gradients gE (per structure), gF (per atom) and gW (per
// structure, 3x3), the pull-back onto a parameter theta is
//
//   sum_s gE_s dE_s/dtheta + sum_a gF_a . dF_a/dtheta + sum_s gW_s : dW_s/dtheta
//     = d/dtheta [ sum_s gE_s E_s + D_t E ],
//
// because F_a = -dE/dr_a and W_ab = -dE/deps_ab (the virial of a homogeneous
// strain r -> (I + eps) r, compressive-positive stress times volume).  D_t E
// is the derivative of the energy along the tangent field that moves every
// pair vector d_ij (minimum image, j - i) by t_ij = gF_i - gF_j - gW d_ij.
//
// The energy is a sum of directed bond terms, each evaluated from centre i:
//   V_ij = 1/2 fc(r_ij) [fR(r_ij) + b_ij(zeta_ij) fA(r_ij)],
// summing to sum_{i<j} fc (fR + (b_ij + b_ji)/2 fA) (engine/tersoff.py:6-19,
// :1399-1414, with the multi-species gating and table reads of
// :1518-1711).  Every directed bond is re-evaluated here -- zeta included,
// nothing per triplet is stored -- with one infinitesimal along the tangent t
// and the derivatives in the parameters a bond reads at its "sites" written
// out, so each site gives d/dtheta (gE V + D_t V).  Sites are reduced onto
// the table entries they read in a fixed order (deterministic).
//
// A bond's kind is (s_i, s_j, i < j): the records it reads.  Passes: the legs
// of every row, compacted to its front (8 lanes per atom); the bonds
// partitioned into one list per kind (counts per tile of slots, a scan, a
// stable scatter); the pair and bond-order sites of each list
// (adj_pair_sites, which also leaves each bond's two zeta coefficients); the
// leg sites of each list per species of the third atom (adj_leg_sites); the
// final reduction.  Sites:
//   pair: 0..5   A, B, lambda1, lambda2, R, D of the pair record tb[lo, hi]
//         6, 7   beta, n of the centre's record tb[s_i, s_j]
//   leg:  0..4   c, d, h, lambda3, gamma of tri[s_i, s_j, s_k]
//         5, 6   R, D of tb[s_i, s_k] (the cutoff of leg i-k)
#include "mbf_hd.cuh"
#include "mbf_rows.cuh"

namespace mbf {

constexpr int ADJ_PB = 64;           // threads of a bond block
constexpr int ADJ_PG = 148 * 6;      // bond blocks per list at most
constexpr int ADJ_FB = 128;          // threads per table entry of the final sums
constexpr int ADJ_LPA = 8;           // lanes per atom of the row pass
constexpr double ADJ_HALF_PI = 0.5 * 3.14159265358979323846;

struct AdjTab {
    int ns;
    const double *tb;   // (ns*ns, 10): valid A B l1 l2 R D beta n -
    const double *tri;  // (ns^3, 8):   valid c d h l3 m gam -
    double rc;
};

// A leg: displacement from the centre, its tangent, length and the length's
// tangent.  Its meta word: the neighbour's species, LEG, BOND where the pair
// record is valid, and the bond's kind from bit 16 on; 0 behind a row's legs.
struct __align__(16) AdjLeg {
    double d[3], t[3], r, rt;
};
constexpr int ADJ_LEG = 1 << 9, ADJ_BOND = 1 << 8;
constexpr int ADJ_KINDS = 2 * 8 * 8;   // kinds of up to eight species
constexpr int ADJ_TILE = 1024;         // slots per block of the partition
constexpr int ADJ_TB = 256;

// The cutoff function at r (engine/tersoff.py:48-54) and its first and second
// derivatives.
__device__ __forceinline__ void adj_cut(double r, double R, double D, double &f, double &f1, double &f2, double &x) {
    f = 1.0;
    f1 = f2 = x = 0.0;
    if (r < R - D) return;
    f = 0.0;
    if (r > R + D) return;
    const double iD = 1.0 / D, w = ADJ_HALF_PI * iD;
    x = (r - R) * iD;
    double sn, cs;
    sincospi(0.5 * x, &sn, &cs);
    f = 0.5 - 0.5 * sn;
    f1 = -0.5 * w * cs;
    f2 = 0.5 * w * w * sn;
}

// exp clamped as the reference's _nb_exp (engine/_numba_common.py:12-33):
// constant outside [-500, 500]; e1 is the derivative.
__device__ __forceinline__ void adj_exp(double x, double &e, double &e1) {
    e = clamped_exp<double>(x);
    e1 = x > 500.0 || x < -500.0 ? 0.0 : e;
}

// Row pass, ADJ_LPA lanes per atom: the legs inside their pair's reach at the
// front of the row's stretch of `legs`, every slot's meta word, and each
// bond's centre.
__global__ void __launch_bounds__(128) te_adjoint_rows(SysView S, const int *__restrict__ row_off,
                                                       const int *__restrict__ nbr, AdjTab P, AdjIn G,
                                                       AdjLeg *__restrict__ legs, int *__restrict__ meta,
                                                       int *__restrict__ centre) {
    constexpr int LPA = ADJ_LPA;
    const int i = (blockIdx.x * blockDim.x + threadIdx.x) / LPA, sub = threadIdx.x & (LPA - 1);
    if (i >= S.n_atoms) return;  // whole groups leave together
    const int gl = threadIdx.x & 31 & ~(LPA - 1);
    const unsigned gones = (1u << LPA) - 1u, gmask = gones << gl;
    const int ns = P.ns, si = S.types[i], beg = row_off[i], n = row_off[i + 1] - beg;
    const int sst = S.n_struct > 1 ? S.atom_struct[i] : 0;
    RowCell cell;
    cell.load(S, i);
    double xi[3], fi[3], w[9];
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        xi[k] = S.pos[3 * (size_t)i + k];
        fi[k] = G.gF ? G.gF[3 * (size_t)i + k] : 0.0;
    }
#pragma unroll
    for (int k = 0; k < 9; ++k) w[k] = G.gW ? G.gW[9 * (size_t)sst + k] : 0.0;
    const double rc2 = P.rc * P.rc;
    int found = 0;
    for (int s0 = 0; s0 < n; s0 += LPA) {
        const int s = s0 + sub;
        bool lv = false;
        AdjLeg L;
        int m = 0;
        if (s < n) {
            const int j = nbr[beg + s];
            const double *pj = S.pos + 3 * (size_t)j;
            cell.mic(pj[0] - xi[0], pj[1] - xi[1], pj[2] - xi[2], L.d[0], L.d[1], L.d[2]);
            const double r2 = L.d[0] * L.d[0] + L.d[1] * L.d[1] + L.d[2] * L.d[2];
            if (r2 < rc2 && r2 > 1e-24) {
                const int sj = S.types[j];
                const double *t1 = P.tb + 10 * (si * ns + sj), *t2 = P.tb + 10 * (sj * ns + si);
                const double reach = fmax(t1[0] != 0.0 ? t1[5] + t1[6] : -1.0, t2[0] != 0.0 ? t2[5] + t2[6] : -1.0);
                lv = reach > 0.0 && r2 <= reach * reach;
                if (lv) {
                    const bool lower = i < j, bond = (lower ? t1 : t2)[0] != 0.0;
                    m = sj | ADJ_LEG | (bond ? ADJ_BOND : 0) | ((si * ns + sj) * 2 + (lower ? 1 : 0)) << 16;
                    L.r = sqrt(r2);
#pragma unroll
                    for (int k = 0; k < 3; ++k)
                        L.t[k] = fi[k] - (G.gF ? G.gF[3 * (size_t)j + k] : 0.0) -
                                 (w[3 * k] * L.d[0] + w[3 * k + 1] * L.d[1] + w[3 * k + 2] * L.d[2]);
                    L.rt = (L.d[0] * L.t[0] + L.d[1] * L.t[1] + L.d[2] * L.t[2]) / L.r;
                }
            }
        }
        const unsigned b = (__ballot_sync(gmask, lv) >> gl) & gones;
        if (lv) {
            const int q = beg + found + __popc(b & ((1u << sub) - 1u));
            legs[q] = L;
            meta[q] = m;
            centre[q] = i;
        }
        found += __popc(b);
    }
    for (int q = found + sub; q < n; q += LPA) meta[beg + q] = 0;
}

// A slot's kind, or -1.
__device__ __forceinline__ int adj_kind(const int *__restrict__ meta, int s, int n_used) {
    if (s >= n_used) return -1;
    const int m = meta[s];
    return m & ADJ_BOND ? m >> 16 : -1;
}

// Bonds of each kind per tile of slots: counts[kind * n_tiles + tile].
__global__ void __launch_bounds__(ADJ_TB) te_adjoint_count(const int *__restrict__ row_off, int n_atoms, int kinds,
                                                           const int *__restrict__ meta, int *__restrict__ counts) {
    __shared__ int cnt[ADJ_KINDS];
    for (int k = threadIdx.x; k < kinds; k += ADJ_TB) cnt[k] = 0;
    __syncthreads();
    const int used = row_off[n_atoms];
    for (int s = threadIdx.x; s < ADJ_TILE; s += ADJ_TB) {
        const int k = adj_kind(meta, blockIdx.x * ADJ_TILE + s, used);
        if (k >= 0) atomicAdd(cnt + k, 1);
    }
    __syncthreads();
    for (int k = threadIdx.x; k < kinds; k += ADJ_TB) counts[(size_t)k * gridDim.x + blockIdx.x] = cnt[k];
}

// The tile's bonds into the lists, in slot order: (centre, slot).
__global__ void __launch_bounds__(ADJ_TB) te_adjoint_scatter(const int *__restrict__ row_off, int n_atoms, int kinds,
                                                             const int *__restrict__ meta,
                                                             const int *__restrict__ centre,
                                                             const int *__restrict__ pos, int2 *__restrict__ bonds) {
    constexpr int NW = ADJ_TB / 32;
    __shared__ int next[ADJ_KINDS], wcnt[NW][ADJ_KINDS];
    for (int k = threadIdx.x; k < kinds; k += ADJ_TB) next[k] = pos[(size_t)k * gridDim.x + blockIdx.x];
    for (int k = threadIdx.x; k < NW * ADJ_KINDS; k += ADJ_TB) (&wcnt[0][0])[k] = 0;
    __syncthreads();
    const int used = row_off[n_atoms], w = threadIdx.x >> 5, lane = threadIdx.x & 31;
    for (int s0 = 0; s0 < ADJ_TILE; s0 += ADJ_TB) {
        const int s = blockIdx.x * ADJ_TILE + s0 + threadIdx.x;
        const int k = adj_kind(meta, s, used);
        const unsigned same = __match_any_sync(MBF_FULL, k);
        const int rank = __popc(same & ((1u << lane) - 1u));
        if (k >= 0 && rank == 0) wcnt[w][k] = __popc(same);
        __syncthreads();
        if (k >= 0) {
            int o = next[k] + rank;
            for (int q = 0; q < w; ++q) o += wcnt[q][k];
            bonds[o] = make_int2(centre[s], s);
        }
        __syncthreads();
        for (int q = threadIdx.x; q < kinds; q += ADJ_TB) {
            int t = 0;
            for (int v = 0; v < NW; ++v) {
                t += wcnt[v][q];
                wcnt[v][q] = 0;
            }
            next[q] += t;
        }
        __syncthreads();
    }
}

// The kind blockIdx.y stands for and its block's share of the list.
// Bonds per block of a list of np over at most g blocks, whole rounds of a
// block (a share of 46 bonds for 64 threads took 72 us in the pair pass, of
// 64 or 128 it takes 51); the blocks behind the list's end do nothing and
// leave no sums.
__device__ __forceinline__ int adj_per(int np, int g) { return ((np + g - 1) / g + ADJ_PB - 1) / ADJ_PB * ADJ_PB; }

struct AdjShare {
    int si, sj, lower, first, end;
    __device__ __forceinline__ void load(const AdjTab &P, int n_tiles, const int *__restrict__ pos) {
        const int c = blockIdx.y, k = c % (2 * P.ns);
        si = c / (2 * P.ns);
        sj = k >> 1;
        lower = k & 1;
        const int p0 = pos[(size_t)c * n_tiles], np = pos[(size_t)(c + 1) * n_tiles] - p0;
        const int per = adj_per(np, gridDim.x);
        first = p0 + min(np, (int)blockIdx.x * per);
        end = p0 + min(np, ((int)blockIdx.x + 1) * per);
    }
};

// A zeta term's angle: cos between leg k and the bond's leg, and its tangent.
__device__ __forceinline__ void adj_cos(const AdjLeg &a, const AdjLeg &b, double ira, double &c, double &ct) {
    const double irb = 1.0 / b.r, ii = ira * irb;
    c = (a.d[0] * b.d[0] + a.d[1] * b.d[1] + a.d[2] * b.d[2]) * ii;
    const double dt = a.t[0] * b.d[0] + a.t[1] * b.d[1] + a.t[2] * b.d[2] + a.d[0] * b.t[0] + a.d[1] * b.t[1] +
                      a.d[2] * b.t[2];
    ct = dt * ii - c * (a.rt * ira + b.rt * irb);
}

// The exponential of a zeta term, exp((l3 u)^m) clamped, with u's tangent ut:
// value, tangent, l3-derivative and its tangent.
__device__ __forceinline__ void adj_expo(double l3, double m, double u, double ut, double &ex, double &ext, double &el,
                                         double &elt) {
    double w, wu, wl, wlt;
    if (m == 3.0) {
        w = (l3 * l3 * l3) * (u * u * u);
        wu = 3.0 * (l3 * l3 * l3) * (u * u);
        wl = 3.0 * (l3 * l3) * (u * u * u);
        wlt = 9.0 * (l3 * l3) * (u * u) * ut;
    } else if (m == 1.0) {
        w = l3 * u;
        wu = l3;
        wl = u;
        wlt = ut;
    } else {
        const double lm = pow(l3, m), um = pow(u, m), l1 = pow(l3, m - 1.0), u1 = pow(u, m - 1.0);
        w = lm * um;
        wu = m * lm * u1;
        wl = m * l1 * um;
        wlt = m * m * l1 * u1 * ut;
    }
    double e1;
    adj_exp(w, ex, e1);
    ext = e1 * wu * ut;
    el = e1 * wl;
    elt = (e1 == 0.0 ? 0.0 : ext * wl) + e1 * wlt;
}

// Block sums of each thread's NV site sums into (site, block) rows.
template <int NV>
__device__ __forceinline__ void adj_block_sums(double (&o)[NV], double *__restrict__ out) {
    __shared__ double sums[ADJ_PB / 32][NV];
    const int w = threadIdx.x >> 5, l = threadIdx.x & 31;
#pragma unroll
    for (int k = 0; k < NV; ++k) {
        double x = o[k];
#pragma unroll
        for (int d = 16; d > 0; d >>= 1) x += __shfl_xor_sync(MBF_FULL, x, d);
        if (l == 0) sums[w][k] = x;
    }
    __syncthreads();
    for (int k = threadIdx.x; k < NV; k += blockDim.x) {
        double x = 0.0;
        for (int q = 0; q < ADJ_PB / 32; ++q) x += sums[q][k];
        out[(size_t)k * gridDim.x + blockIdx.x] = x;
    }
}

// The pair and bond-order sites of one list: zeta and its tangent over the
// centre's legs, then with V = 1/2 f (fR + b fA) the eight parameters'
// derivatives and tangents; zc = {gE V_z + (V_z)_t, V_z}, through which every
// leg parameter acts on this bond.  Bound by FP64 latency: a thread per bond,
// site sums in registers over the block's share of the list.  220,000 bonds of
// 38,600 SiC atoms: 50 us, the leg pass 74 (at the 140 and 165 registers the
// compiler takes by itself, 7 and 6 blocks an SM, 61 and 101; at 12 blocks an
// SM 64 and 90); one kernel in generic hyper-dual arithmetic that staged every
// bond's sites in shared memory and summed them there by table entry took 329.
__global__ void __launch_bounds__(ADJ_PB, 9) adj_pair_sites(SysView S, const int *__restrict__ row_off, AdjTab P, AdjIn G,
                                                         const AdjLeg *__restrict__ legs, const int *__restrict__ meta,
                                                         int n_tiles, const int *__restrict__ pos,
                                                         const int2 *__restrict__ bonds, double2 *__restrict__ zc,
                                                         double *__restrict__ partial) {
    const int ns = P.ns;
    AdjShare sh;
    sh.load(P, n_tiles, pos);
    if (sh.first >= sh.end) return;  // uniform over the block
    const double *tp = P.tb + 10 * (sh.lower ? sh.si * ns + sh.sj : sh.sj * ns + sh.si);
    const double *tij = P.tb + 10 * (sh.si * ns + sh.sj);
    const double A = __ldg(tp + 1), B = __ldg(tp + 2), l1 = __ldg(tp + 3), l2 = __ldg(tp + 4), R = __ldg(tp + 5),
                 D = __ldg(tp + 6), beta = __ldg(tij + 7), nn = __ldg(tij + 8);
    double o[8];
#pragma unroll
    for (int k = 0; k < 8; ++k) o[k] = 0.0;
    for (int m = sh.first + threadIdx.x; m < sh.end; m += ADJ_PB) {
        const int2 iq = bonds[m];
        const int beg = row_off[iq.x], end = row_off[iq.x + 1];
        const int sst = S.n_struct > 1 ? __ldg(S.atom_struct + iq.x) : 0;
        const double gE = G.gE ? __ldg(G.gE + sst) : 0.0;
        const AdjLeg b = legs[iq.y];
        const double ir = 1.0 / b.r, r = b.r, rt = b.rt;
        double z = 0.0, zt = 0.0;
        for (int k = beg; k < end; ++k) {
            const int mk = meta[k];
            if (!(mk & ADJ_LEG)) break;
            if (k == iq.y) continue;
            const int sk = mk & 0xff;
            const double *tk = P.tb + 10 * (sh.si * ns + sk), *t3 = P.tri + 8 * ((sh.si * ns + sh.sj) * ns + sk);
            if (__ldg(tk) == 0.0 || __ldg(t3) == 0.0) continue;
            const AdjLeg q = legs[k];
            double f, f1, f2, x, c, ct, ex, ext, el, elt;
            adj_cut(q.r, __ldg(tk + 5), __ldg(tk + 6), f, f1, f2, x);
            if (f == 0.0) continue;
            adj_cos(b, q, ir, c, ct);
            const double pc = __ldg(t3 + 1), pd = __ldg(t3 + 2), hc = __ldg(t3 + 3) - c, d2 = pd * pd;
            const double iq2 = 1.0 / (d2 + hc * hc), c2 = pc * pc;
            const double g = 1.0 + c2 * hc * hc * iq2 / d2, gt = -2.0 * c2 * hc * iq2 * iq2 * ct;
            adj_expo(__ldg(t3 + 4), __ldg(t3 + 5), r - q.r, rt - q.rt, ex, ext, el, elt);
            const double gam = __ldg(t3 + 6);
            z += gam * f * g * ex;
            zt += gam * (f1 * q.rt * g * ex + f * gt * ex + f * g * ext);
        }
        // the bond order and its derivatives in z, beta and n
        double bo = 1.0, bz = 0.0, bzz = 0.0, bb = 0.0, bbt = 0.0, bn = 0.0, bnt = 0.0;
        if (z > 0.0 && beta != 0.0) {
            const double iz = 1.0 / z, l = log(beta * z), u = exp(nn * l), L = log(1.0 + u), in = 1.0 / nn;
            const double s = u / (1.0 + u), st = nn * s * (1.0 - s) * iz * zt;
            bo = exp(-0.5 * in * L);
            bz = -0.5 * bo * s * iz;
            bzz = -0.5 * iz * (bz * s + bo * s * iz * (nn * (1.0 - s) - 1.0));
            const double bt = bz * zt, ib = 1.0 / beta;
            bb = -0.5 * bo * s * ib;
            bbt = -0.5 * ib * (bt * s + bo * st);
            const double k = 0.5 * in * (L * in - s * l);
            bn = bo * k;
            bnt = bt * k + bo * 0.5 * in * (s * iz * zt - st * l - s * iz * zt);
        }
        const double bt = bz * zt;
        double f, f1, f2, x, e1, e1d, e2, e2d;
        adj_cut(r, R, D, f, f1, f2, x);
        adj_exp(-l1 * r, e1, e1d);
        adj_exp(-l2 * r, e2, e2d);
        const double ft = f1 * rt, iD = x == 0.0 && f1 == 0.0 ? 0.0 : 1.0 / D;
        const double fR = A * e1, fA = -B * e2, fRt = -l1 * rt * A * e1d, fAt = l2 * rt * B * e2d;
        const double s = fR + bo * fA, st = fRt + bt * fA + bo * fAt;
        const double e1t = -l1 * rt * e1d, e2t = -l2 * rt * e2d;
        const double fr = -f1, frt = -f2 * rt, fd = -f1 * x, fdt = -(f2 * x + f1 * iD) * rt;
        o[0] += 0.5 * (gE * f * e1 + ft * e1 + f * e1t);
        o[1] -= 0.5 * (gE * f * bo * e2 + ft * bo * e2 + f * bt * e2 + f * bo * e2t);
        const double e1x = e1d, e1xt = -l1 * rt * e1d, e2x = e2d, e2xt = -l2 * rt * e2d;
        o[2] -= 0.5 * A * (gE * f * r * e1x + ft * r * e1x + f * rt * e1x + f * r * e1xt);
        o[3] += 0.5 * B * (gE * f * bo * r * e2x + ft * bo * r * e2x + f * bt * r * e2x + f * bo * rt * e2x + f * bo * r * e2xt);
        o[4] += 0.5 * (gE * fr * s + frt * s + fr * st);
        o[5] += 0.5 * (gE * fd * s + fdt * s + fd * st);
        o[6] += 0.5 * (gE * f * bb * fA + ft * bb * fA + f * bbt * fA + f * bb * fAt);
        o[7] += 0.5 * (gE * f * bn * fA + ft * bn * fA + f * bnt * fA + f * bn * fAt);
        const double vz = 0.5 * f * fA * bz;
        zc[m] = make_double2(gE * vz + 0.5 * (ft * fA * bz + f * fAt * bz + f * fA * bzz * zt), vz);
    }
    adj_block_sums<8>(o, partial + (size_t)blockIdx.y * 8 * gridDim.x);
}

// The leg sites of one list for third atoms of species blockIdx.z: each term
// z = gamma f g ex once more, with its derivatives in c, d, h, lambda3, gamma,
// R, D and their tangents, weighted by the bond's coefficients.
__global__ void __launch_bounds__(ADJ_PB, 8) adj_leg_sites(const int *__restrict__ row_off, AdjTab P,
                                                        const AdjLeg *__restrict__ legs, const int *__restrict__ meta,
                                                        int n_tiles, const int *__restrict__ pos,
                                                        const int2 *__restrict__ bonds, const double2 *__restrict__ zc,
                                                        double *__restrict__ partial) {
    const int ns = P.ns, sk = blockIdx.z;
    AdjShare sh;
    sh.load(P, n_tiles, pos);
    if (sh.first >= sh.end) return;  // uniform over the block
    const double *tk = P.tb + 10 * (sh.si * ns + sk), *t3 = P.tri + 8 * ((sh.si * ns + sh.sj) * ns + sk);
    const bool valid = __ldg(tk) != 0.0 && __ldg(t3) != 0.0;
    const double pc = __ldg(t3 + 1), pd = __ldg(t3 + 2), ph = __ldg(t3 + 3), l3 = __ldg(t3 + 4), pm = __ldg(t3 + 5),
                 gam = __ldg(t3 + 6), R = __ldg(tk + 5), D = __ldg(tk + 6);
    const double d2 = pd * pd, c2 = pc * pc, id2 = 1.0 / d2, id3 = id2 / pd;
    const double iD = D != 0.0 ? 1.0 / D : 0.0;  // a sharp cutoff has no slope to scale
    double o[7];
#pragma unroll
    for (int k = 0; k < 7; ++k) o[k] = 0.0;
    if (valid) {
        for (int m = sh.first + threadIdx.x; m < sh.end; m += ADJ_PB) {
            const double2 w = zc[m];
            if (w.x == 0.0 && w.y == 0.0) continue;
            const int2 iq = bonds[m];
            const int beg = row_off[iq.x], end = row_off[iq.x + 1];
            const AdjLeg b = legs[iq.y];
            const double ir = 1.0 / b.r;
            for (int k = beg; k < end; ++k) {
                const int mk = meta[k];
                if (!(mk & ADJ_LEG)) break;
                if (k == iq.y || (mk & 0xff) != sk) continue;
                const AdjLeg q = legs[k];
                double f, f1, f2, x, c, ct, ex, ext, el, elt;
                adj_cut(q.r, R, D, f, f1, f2, x);
                if (f == 0.0) continue;
                adj_cos(b, q, ir, c, ct);
                adj_expo(l3, pm, b.r - q.r, b.rt - q.rt, ex, ext, el, elt);
                const double hc = ph - c, hct = -ct, hc2 = hc * hc, iq2 = 1.0 / (d2 + hc2), iq4 = iq2 * iq2;
                const double g = 1.0 + c2 * hc2 * iq2 * id2;
                const double gh = 2.0 * c2 * hc * iq4, ght = 2.0 * c2 * iq4 * (1.0 - 4.0 * hc2 * iq2) * hct;
                const double ft = f1 * q.rt, gt = gh * hct;
                // derivative y and tangent yt of each factor's parameter, the
                // other two factors a, b: w.x y a b + w.y (y a b)_t
                auto add = [&](double y, double yt, double a, double at, double e, double et) {
                    return w.x * y * a * e + w.y * (yt * a * e + y * at * e + y * a * et);
                };
                const double gc = 2.0 * pc * hc2 * iq2 * id2, gct = 4.0 * pc * hc * iq4 * hct;
                // (the difference 2 d / q^2 - 2 / d^3, written without it: q = d^2
                // + (h - cos)^2 is d^2 to a part in 1e3 to 1e5 for silicon)
                const double gd = -2.0 * c2 * hc2 * (2.0 * d2 + hc2) * iq4 * id3;
                const double gdt = -8.0 * c2 * pd * hc * iq4 * iq2 * hct;
                o[0] += gam * add(gc, gct, f, ft, ex, ext);
                o[1] += gam * add(gd, gdt, f, ft, ex, ext);
                o[2] += gam * add(gh, ght, f, ft, ex, ext);
                o[3] += gam * add(el, elt, f, ft, g, gt);
                o[4] += add(f, ft, g, gt, ex, ext);
                o[5] += gam * add(-f1, -f2 * q.rt, g, gt, ex, ext);
                o[6] += gam * add(-f1 * x, -(f2 * x + f1 * iD) * q.rt, g, gt, ex, ext);
            }
        }
    }
    adj_block_sums<7>(o, partial + ((size_t)blockIdx.y * ns + sk) * 7 * gridDim.x);
}

// One block per table entry (tb (ns*ns, 10), then tri (ns^3, 8)): the block
// values of every (kind, site) row that reads the entry, then a fixed tree.
__global__ void __launch_bounds__(ADJ_FB) te_adjoint_final(int ns, int gP, int n_tiles, const int *__restrict__ pos,
                                 const double *__restrict__ pair, const double *__restrict__ leg,
                                 double *__restrict__ d_tb, double *__restrict__ d_tri) {
    const int e = blockIdx.x, l = threadIdx.x;
    __shared__ double sums[ADJ_FB / 32];
    double acc = 0.0;
    auto kind = [&](int si, int sj, int lower) { return (si * ns + sj) * 2 + lower; };
    // the block sums of one site of a list: four loads in flight a lane
    auto add_row = [&](int c, const double *p) {
        const int np = pos[(size_t)(c + 1) * n_tiles] - pos[(size_t)c * n_tiles];
        if (np <= 0) return;
        const int per = adj_per(np, gP), busy = (np + per - 1) / per;
        double x[4] = {0.0, 0.0, 0.0, 0.0};
        for (int b = l; b < busy; b += 4 * ADJ_FB) {
#pragma unroll
            for (int k = 0; k < 4; ++k)
                if (b + ADJ_FB * k < busy) x[k] += p[b + ADJ_FB * k];
        }
        acc += (x[0] + x[1]) + (x[2] + x[3]);
    };
    auto add_pair = [&](int c, int site) { add_row(c, pair + ((size_t)c * 8 + site) * gP); };
    auto add_leg = [&](int c, int k, int site) { add_row(c, leg + (((size_t)c * ns + k) * 7 + site) * gP); };
    if (e < 10 * ns * ns) {
        const int ra = e / 10 / ns, rb = e / 10 % ns, col = e % 10;
        if (col >= 1 && col <= 6) {  // the pair record: read with lo = ra, hi = rb
            add_pair(kind(ra, rb, 1), col - 1);
            add_pair(kind(rb, ra, 0), col - 1);
        }
        if (col == 7 || col == 8)
            for (int o = 0; o < 2; ++o) add_pair(kind(ra, rb, o), col - 1);
        if (col == 5 || col == 6)
            for (int sj = 0; sj < ns; ++sj)
                for (int o = 0; o < 2; ++o) add_leg(kind(ra, sj, o), rb, col);
    } else {
        const int e3 = e - 10 * ns * ns, row = e3 / 8, col = e3 % 8;
        const int ra = row / (ns * ns), rb = row / ns % ns, k = row % ns;
        const int site = col >= 1 && col <= 4 ? col - 1 : (col == 6 ? 4 : -1);
        if (site >= 0)
            for (int o = 0; o < 2; ++o) add_leg(kind(ra, rb, o), k, site);
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) acc += __shfl_xor_sync(MBF_FULL, acc, o);
    if ((l & 31) == 0) sums[l >> 5] = acc;
    __syncthreads();
    if (l == 0) {
        for (int w = 1; w < ADJ_FB / 32; ++w) acc += sums[w];
        if (e < 10 * ns * ns) d_tb[e] = acc;
        else d_tri[e - 10 * ns * ns] = acc;
    }
}

struct AdjLayout {
    size_t pair, leg, legs, meta, centre, bonds, zc, cnt, pos, scan, total;
    int ne, kinds, gP, n_tiles;
};

static AdjLayout adj_layout(long long n_slots, int ns) {
    AdjLayout L;
    const size_t sl = (size_t)(n_slots > 0 ? n_slots : 1);
    L.ne = 10 * ns * ns + 8 * ns * ns * ns;
    L.kinds = 2 * ns * ns;
    L.n_tiles = (int)((sl + ADJ_TILE - 1) / ADJ_TILE);
    const size_t tiles = (sl + ADJ_PB - 1) / ADJ_PB;
    L.gP = (int)(tiles < (size_t)ADJ_PG ? tiles : (size_t)ADJ_PG);
    size_t o = 0;
    L.pair = o;
    o = align256(o + sizeof(double) * (size_t)L.kinds * 8 * L.gP);
    L.leg = o;
    o = align256(o + sizeof(double) * (size_t)L.kinds * ns * 7 * L.gP);
    L.legs = o;
    o = align256(o + sizeof(AdjLeg) * sl);
    L.meta = o;
    o = align256(o + sizeof(int) * sl);
    L.centre = o;
    o = align256(o + sizeof(int) * sl);
    L.bonds = o;
    o = align256(o + sizeof(int2) * sl);
    L.zc = o;
    o = align256(o + sizeof(double2) * sl);
    L.cnt = o;
    o = align256(o + sizeof(int) * (size_t)L.kinds * L.n_tiles);
    L.pos = o;
    o = align256(o + sizeof(int) * ((size_t)L.kinds * L.n_tiles + 1));
    L.scan = o;
    o = align256(o + sizeof(int) * scan_workspace_ints(L.kinds * L.n_tiles));
    L.total = o + 16;  // the layout starts at the workspace's first 16-byte boundary
    return L;
}

}  // namespace mbf

using namespace mbf;

extern "C" {

size_t mbf_tersoff_adjoint_workspace_bytes(long long n_slots, int ns) {
    if (ns <= 0 || n_slots < 0) return 0;
    return adj_layout(n_slots, ns).total;
}

int mbf_tersoff_adjoint(const mbf_system *sys, const mbf_nlist *nl, const mbf_tersoff_tables *tab,
                        const double *g_energy, const double *g_forces, const double *g_virial, void *workspace,
                        size_t workspace_bytes, double *d_tb, double *d_tri, void *stream) {
    if (!sys || !nl || !tab || !workspace || !d_tb || !d_tri || tab->ns <= 0 || tab->ns > 8)
        return MBF_ERR_ARGUMENT;
    if (nl->n_atoms != sys->n_atoms) return MBF_ERR_ARGUMENT;
    AdjLayout L = adj_layout(nl->n_slots, tab->ns);
    if (workspace_bytes < L.total) return MBF_ERR_WORKSPACE;
    workspace = align16(workspace);
    cudaStream_t st = (cudaStream_t)stream;
    int ns = tab->ns;
    if (sys->n_atoms == 0 || nl->n_slots == 0) {
        if (cudaMemsetAsync(d_tb, 0, sizeof(double) * 10 * ns * ns, st) != cudaSuccess ||
            cudaMemsetAsync(d_tri, 0, sizeof(double) * 8 * ns * ns * ns, st) != cudaSuccess)
            return MBF_ERR_CUDA;
        return MBF_OK;
    }
    SysView S = make_view(sys);
    AdjTab P;
    P.ns = ns;
    P.tb = tab->tb;
    P.tri = tab->tri;
    P.rc = tab->r_cut;
    AdjIn G;
    G.gE = g_energy;
    G.gF = g_forces;
    G.gW = g_virial;
    double *pair = ws_at<double>(workspace, L.pair), *leg = ws_at<double>(workspace, L.leg);
    AdjLeg *legs = ws_at<AdjLeg>(workspace, L.legs);
    int *meta = ws_at<int>(workspace, L.meta);
    int *centre = ws_at<int>(workspace, L.centre);
    int2 *bonds = ws_at<int2>(workspace, L.bonds);
    double2 *zc = ws_at<double2>(workspace, L.zc);
    int *cnt = ws_at<int>(workspace, L.cnt);
    int *pos = ws_at<int>(workspace, L.pos);
    const int N = sys->n_atoms;
    PROF_BEGIN("te_adjoint_rows", st);
    te_adjoint_rows<<<(int)(((long long)N * ADJ_LPA + 127) / 128), 128, 0, st>>>(S, nl->row_off, nl->nbr, P, G, legs, meta,
                                                                                 centre);
    PROF_END("te_adjoint_rows", st);
    MBF_CHECK_LAUNCH();
    PROF_BEGIN("te_adjoint_lists", st);
    te_adjoint_count<<<L.n_tiles, ADJ_TB, 0, st>>>(nl->row_off, N, L.kinds, meta, cnt);
    MBF_CHECK_LAUNCH();
    int rc = exclusive_scan(cnt, pos, L.kinds * L.n_tiles, ws_at<int>(workspace, L.scan), st);
    if (rc != MBF_OK) return rc;
    te_adjoint_scatter<<<L.n_tiles, ADJ_TB, 0, st>>>(nl->row_off, N, L.kinds, meta, centre, pos, bonds);
    PROF_END("te_adjoint_lists", st);
    MBF_CHECK_LAUNCH();
    PROF_BEGIN("te_adjoint_pair", st);
    adj_pair_sites<<<dim3(L.gP, L.kinds), ADJ_PB, 0, st>>>(S, nl->row_off, P, G, legs, meta, L.n_tiles, pos, bonds, zc,
                                                           pair);
    PROF_END("te_adjoint_pair", st);
    MBF_CHECK_LAUNCH();
    PROF_BEGIN("te_adjoint_leg", st);
    adj_leg_sites<<<dim3(L.gP, L.kinds, ns), ADJ_PB, 0, st>>>(nl->row_off, P, legs, meta, L.n_tiles, pos, bonds, zc,
                                                              leg);
    PROF_END("te_adjoint_leg", st);
    MBF_CHECK_LAUNCH();
    PROF_BEGIN("te_adjoint_reduce", st);
    te_adjoint_final<<<L.ne, ADJ_FB, 0, st>>>(ns, L.gP, L.n_tiles, pos, pair, leg, d_tb, d_tri);
    PROF_END("te_adjoint_reduce", st);
    MBF_CHECK_LAUNCH();
    return MBF_OK;
}

}  // extern "C"
