// Tersoff bond-order potential: one kernel per evaluation over the centres
// (zeta, bond orders, energies, the force of every centre's own terms on its
// neighbours), then the gather of the slots.
//
// Replaces engine/tersoff.py:1208-1711 (single-species :1233-1513 with m = 3
// and gamma = 1, multi-species :1518-1711 with its dense species tables
// :1606-1653).  The energy sum_{i<j} fc (fR + b_avg fA), b_avg the mean of the
// two bond orders (engine/tersoff.py:6-19), is the sum over centres of
//   U_i = 1/2 sum_j fc_ij (fR_ij + b_ij fA_ij),
// which needs the centre's own bond orders only.
//
// Owner computes, no atomics: the lane group of centre i evaluates every
// term of U_i, keeps the force on i and writes -dU_i/dr_x into x's own slot
// (x -> i); atom a later sums its own row of slots (gather_live).
#include "mbf_rows.cuh"

namespace mbf {

// Lanes per atom (LPA) is a template parameter chosen by the host (the
// autotuner): LPA lanes stage a centre's row, and LPA / 4 lanes share the
// angle loops of a leg.  A block takes GPB centres (about 30 KB of staged legs
// in float64) with at least two warps for the leg passes.
template <int MAXN, int LPA> struct TeGeom {
    static constexpr int GPB = 256 / MAXN;
    static constexpr int BLOCK = GPB * LPA < 64 ? 64 : GPB * LPA;
    static constexpr int KS = LPA / 4;
    // Resident threads per SM the kernel is compiled for (its registers):
    // with the gather, 32,768-atom SiC float64 at 384 / 512 threads 66 / 62 us,
    // 64,000-atom Si mixed at 512 / 640 55 / 53.
    static constexpr int min_blocks(int size) { return (size == 8 ? 512 : 640) / BLOCK; }
};

struct TeDev {
    int ns;
    const double *tb;   // (ns*ns, 10): valid A B l1 l2 R D beta n -
    const double *tri;  // (ns^3, 8):   valid c d h l3 m gam -
    double rc;
};

__device__ __forceinline__ void te_sincospi(double x, double &s, double &c) { sincospi(x, &s, &c); }
__device__ __forceinline__ void te_sincospi(float x, float &s, float &c) { sincospif(x, &s, &c); }

// The cutoff function fc and its derivative (engine/tersoff.py:48-60).
template <typename T>
__device__ __forceinline__ void te_cut(T r, T R, T D, T &fc, T &dfc) {
    fc = T(1);
    dfc = T(0);
    if (r < R - D) return;
    fc = T(0);
    if (r > R + D) return;
    T s, c;
    te_sincospi(T(0.5) * (r - R) / D, s, c);
    fc = T(0.5) - T(0.5) * s;
    dfc = T(-0.25) * T(3.14159265358979323846) / D * c;
}

// (l3 u)^m for m = 1 or 3 by multiplication, pow otherwise.
template <typename T>
__device__ __forceinline__ T te_arg(T l3, T u, T m) {
    if (m == T(3)) return (l3 * l3 * l3) * (u * u * u);
    if (m == T(1)) return l3 * u;
    return RT<T>::pw(l3, m) * RT<T>::pw(u, m);
}

// The angular function g = 1 + c^2/d^2 - c^2/(d^2 + (h - cos)^2), written as
// 1 + c^2 (h - cos)^2 / (d^2 (d^2 + (h - cos)^2)): the same value without
// the cancellation of two ~c^2/d^2 terms (c^2/d^2 ~ 4e7 for silicon), which
// float32 cannot afford.
template <typename T>
__device__ __forceinline__ T te_g(T c2, T d2, T hc) {
    const T hc2 = hc * hc;
    return T(1) + c2 * hc2 / (d2 * (d2 + hc2));
}

// g and dg/dcos from one reciprocal, cd = c^2/d^2 with the record (for the
// forces alone: a rounded cd would put the same error on every zeta).
template <typename T>
__device__ __forceinline__ void te_gdg(T c2, T cd, T d2, T hc, T &g, T &dg) {
    const T hc2 = hc * hc, q = T(1) / (d2 + hc2);
    g = T(1) + cd * (hc2 * q);
    dg = T(-2) * c2 * hc * (q * q);
}

// An (i, j, k) record as the angle loops read it.
template <typename T>
struct TeTri {
    T c2, d2, h, gam, l3, m, valid, cd;
};

template <typename T>
__device__ __forceinline__ TeTri<T> te_tri_row(const double *__restrict__ t) {
    TeTri<T> q;
    const T c = (T)__ldg(t + 1), d = (T)__ldg(t + 2);
    q.c2 = c * c;
    q.d2 = d * d;
    q.h = (T)__ldg(t + 3);
    q.gam = (T)__ldg(t + 6);
    q.l3 = (T)__ldg(t + 4);
    q.m = (T)__ldg(t + 5);
    q.valid = __ldg(t) != 0.0 ? T(1) : T(0);
    q.cd = q.c2 / q.d2;
    return q;
}

// The tables of up to TE_SH species in shared memory: the pair rows, the
// squared reach of every pair, the triplet records in T, and per centre
// species whether its records are all the same, valid and without lambda3
// (one element, or the Tersoff-1989 mixing rules): then one record serves
// every angle of the centre.
constexpr int TE_SH = 3;
template <typename T>
struct TeTab {
    double tb[TE_SH * TE_SH * 10];
    double reach2[TE_SH * TE_SH];
    TeTri<T> tri[TE_SH * TE_SH * TE_SH];
    int plain[TE_SH];
};

// The square of the largest r at which the pair (a, b) takes part in any
// term, from either atom (negative: none): a leg beyond it contributes
// nothing to its centre or to its neighbour's terms, and both atoms of the
// pair agree on it.
__device__ __forceinline__ double te_reach2(const TeDev &P, int a, int b) {
    const double *t = P.tb + 10 * (a * P.ns + b), *u = P.tb + 10 * (b * P.ns + a);
    const double x = __ldg(t) != 0.0 ? __ldg(t + 5) + __ldg(t + 6) : -1.0;
    const double y = __ldg(u) != 0.0 ? __ldg(u + 5) + __ldg(u + 6) : -1.0;
    const double r = x > y ? x : y;
    return r > 0.0 ? r * r : -1.0;
}

template <typename T>
__device__ __forceinline__ void te_load_tab(const TeDev &P, TeTab<T> &B) {
    const int ns = P.ns;
    if (ns > TE_SH) return;
    for (int q = threadIdx.x; q < 10 * ns * ns; q += blockDim.x) B.tb[q] = P.tb[q];
    for (int q = threadIdx.x; q < ns * ns; q += blockDim.x) B.reach2[q] = te_reach2(P, q / ns, q % ns);
    for (int q = threadIdx.x; q < ns * ns * ns; q += blockDim.x) {
        const double c = P.tri[8 * q + 1], d = P.tri[8 * q + 2];
        B.tri[q] = te_tri_row<T>(P.tri + 8 * q);
        B.tri[q].cd = (T)((c * c) / (d * d));
    }
    __syncthreads();
    for (int a = threadIdx.x; a < ns; a += blockDim.x) {
        const TeTri<T> *t = B.tri + a * ns * ns;
        bool same = t[0].valid != T(0) && t[0].l3 == T(0) && (t[0].m == T(3) || t[0].m == T(1));
        for (int q = 1; q < ns * ns; ++q)
            same = same && t[q].valid != T(0) && t[q].l3 == T(0) && (t[q].m == T(3) || t[q].m == T(1)) &&
                   t[q].c2 == t[0].c2 && t[q].d2 == t[0].d2 && t[q].h == t[0].h && t[q].gam == t[0].gam;
        B.plain[a] = same ? 1 : 0;
    }
    __syncthreads();
}

// r in float64 (the two-body part is float64 in both precisions): a column
// of its own beside float32 rows only.
template <typename T, int MAXN> struct TeDist { double rd[MAXN]; };
template <int MAXN> struct TeDist<double, MAXN> {};

// One centre's legs (neighbours inside their pair's cutoff) in shared
// memory, compacted in slot order: displacement, length and its inverse, the
// cutoff function of the leg as a zeta term's third atom (record (i, k)) and
// its derivative, the bond's zeta, then zeta-gradient coefficient, its pair
// part and energy, and the leg's gradient dU_i/dr.  Rows lie 32 bytes apart
// modulo the banks' 128.
template <typename T, int MAXN>
struct TeRow {
    double gx[MAXN], gy[MAXN], gz[MAXN];
    double e[MAXN];  // r^2, then the pair part's slope, at last the energy (in gx until then)
    T x[MAXN], y[MAXN], z[MAXN], r[MAXN], ir[MAXN], fk[MAXN], dfk[MAXN], coef[MAXN];
    TeDist<T, MAXN> dist;
    int rev[MAXN];    // the leg's reverse slot
    int meta[MAXN];   // slot in the row | (i < j) << 8 | species << 9
    int beg, nl, si, pad[5];
};

template <int MAXN> __device__ __forceinline__ void te_put_r(TeRow<double, MAXN> &R, int q, double r) { R.r[q] = r; }
template <int MAXN> __device__ __forceinline__ double te_get_r(const TeRow<double, MAXN> &R, int q) { return R.r[q]; }
template <int MAXN> __device__ __forceinline__ void te_put_r(TeRow<float, MAXN> &R, int q, double r) {
    R.r[q] = (float)r;
    R.dist.rd[q] = r;
}
template <int MAXN> __device__ __forceinline__ double te_get_r(const TeRow<float, MAXN> &R, int q) { return R.dist.rd[q]; }

// The (l3 u)^m exponential of a zeta term and its derivative in u; 1 and 0
// without lambda3.
template <typename T>
__device__ __forceinline__ void te_expo(T l3, T m, T u, T &ex, T &dex) {
    ex = T(1);
    dex = T(0);
    if (l3 == T(0) && (m == T(3) || m == T(1))) return;
    ex = clamped_exp<T>(te_arg<T>(l3, u, m));
    if (m == T(3)) dex = ex * T(3) * (l3 * l3 * l3) * (u * u);
    else if (m == T(1)) dex = ex * l3;
    else dex = ex * m * RT<T>::pw(l3, m) * RT<T>::pw(u, m - T(1));
}

// Every term of a block's centres.  The bound is instruction issue and
// latency, not memory (32,768-atom SiC, float64: 0.6 % of DRAM bandwidth), so
// the work is cut to what the terms need: legs beyond their own pair's cutoff
// are dropped before any loop, the passes over legs run over the block's legs
// as one list, the cutoff functions are evaluated once per leg and not per
// angle, one angle gives zeta_j's term k and zeta_k's term j one common
// geometry, and g and g' take one reciprocal.  Blocks are persistent: the
// tables are loaded once, and the next row's loads are in flight during the
// current one.  With the gather, SiC above: 60 us (80 with a lane group per
// centre in every pass and one-shot blocks), against 415 us for a zeta and a
// force kernel of a lane per bond that evaluated the cutoff functions per
// angle, each gradient from both of its bonds, and a bond order for the
// partner atom to read.
template <typename T, int MAXN, int LPA>
__global__ void __launch_bounds__(TeGeom<MAXN, LPA>::BLOCK, TeGeom<MAXN, LPA>::min_blocks(sizeof(T)))
    te_center(SysView S, const int *__restrict__ row_off, const int *__restrict__ nbr, const int *__restrict__ rev,
              TeDev P, double *__restrict__ slot_G, double *__restrict__ f_local, double *__restrict__ per_atom,
              unsigned *__restrict__ live_mask, int n_slots, ClearWords clr, SiteOut so) {
    typedef TeGeom<MAXN, LPA> G;
    constexpr int GPB = G::GPB, BLOCK = G::BLOCK, KS = G::KS;
    __shared__ TeRow<T, MAXN> rows[GPB];
    __shared__ TeTab<T> B;
    __shared__ BlockLegs<GPB, MAXN> F;
    const int g = threadIdx.x / LPA, sub = threadIdx.x & (LPA - 1);
    RowHead next;
    next.load(S, row_off, g < GPB ? blockIdx.x * GPB + g : S.n_atoms);
    clr.run();
    te_load_tab<T>(P, B);
    const int ns = P.ns;
    const bool small = ns <= TE_SH;
    const double *const tb = small ? B.tb : P.tb;
    auto tri_row = [&](int q) { return small ? B.tri[q] : te_tri_row<T>(P.tri + 8 * (size_t)q); };
    TeRow<T, MAXN> &mine = rows[g < GPB ? g : 0];
    next.slots<LPA>(nbr, rev, n_slots, ns, MAXN);
    for (int base = blockIdx.x * GPB; base < S.n_atoms; base += gridDim.x * GPB) {  // uniform over the block
    const int i = g < GPB ? base + g : S.n_atoms;
    const RowHead head = next;
    const int i_next = g < GPB ? i + gridDim.x * GPB : S.n_atoms;
    next.load(S, row_off, i_next);
    const RowStage st = stage_row<LPA>(
        S, head, nbr, rev, n_slots, ns, P.rc, i, live_mask, so.vec,
        [&](int a, int b) { return small ? B.reach2[a * ns + b] : te_reach2(P, a, b); },
        [&](int q, int s, int j, int sj, int rs, double dx, double dy, double dz, double r2) {
            mine.x[q] = (T)dx;
            mine.y[q] = (T)dy;
            mine.z[q] = (T)dz;
            mine.e[q] = r2;
            mine.rev[q] = rs;
            mine.meta[q] = s | (i < j ? 1 << 8 : 0) | sj << 9;
        });
    if (sub == 0 && g < GPB) {
        mine.beg = st.beg;
        mine.nl = st.nl;
        mine.si = st.si;
    }
    const int total = flatten_legs<GPB, MAXN, LPA>(F, g, sub, st.nl);
    // a lane per leg: length (float64 in both precisions: the two-body part's)
    // and cutoff function
    for (int q = threadIdx.x; q < total; q += BLOCK) {
        const int m = F.map[q], t = m & (MAXN - 1);
        TeRow<T, MAXN> &R = rows[m / MAXN];
        const double r = sqrt(R.e[t]);
        const double *tk = tb + 10 * (R.si * ns + (R.meta[t] >> 9));
        T fk = T(0), dfk = T(0);
        if (tk[0] != 0.0) te_cut<T>((T)r, (T)tk[5], (T)tk[6], fk, dfk);
        te_put_r(R, t, r);
        R.ir[t] = (T)(1.0 / r);
        R.fk[t] = fk;
        R.dfk[t] = dfk;
    }
    __syncthreads();
    next.slots<LPA>(nbr, rev, n_slots, ns, MAXN);
    // KS lanes per leg: zeta of the bond
    const int ks = threadIdx.x & (KS - 1);
    const unsigned share = ((1u << KS) - 1u) << (threadIdx.x & 31 & ~(KS - 1));
    for (int q = threadIdx.x / KS; q < total; q += BLOCK / KS) {
        const int m = F.map[q], t = m & (MAXN - 1);
        TeRow<T, MAXN> &R = rows[m / MAXN];
        const int nl = R.nl, si = R.si;
        T zeta = T(0);
        const T xs = R.x[t], ys = R.y[t], zs = R.z[t], irs = R.ir[t];
        if (small && B.plain[si]) {
            const TeTri<T> own = B.tri[si * ns * ns];
            for (int k = ks; k < nl; k += KS) {
                const T fk = R.fk[k];
                if (k == t || fk == T(0)) continue;
                const T cs = (xs * R.x[k] + ys * R.y[k] + zs * R.z[k]) * (irs * R.ir[k]);
                zeta += own.gam * fk * te_g<T>(own.c2, own.d2, own.h - cs);
            }
        } else {
            const T rs = R.r[t];
            const int row = (si * ns + (R.meta[t] >> 9)) * ns;
            for (int k = ks; k < nl; k += KS) {
                const T fk = R.fk[k];
                if (k == t || fk == T(0)) continue;
                const TeTri<T> w = tri_row(row + (R.meta[k] >> 9));
                if (w.valid == T(0)) continue;
                const T cs = (xs * R.x[k] + ys * R.y[k] + zs * R.z[k]) * (irs * R.ir[k]);
                T ex, dex;
                te_expo<T>(w.l3, w.m, rs - R.r[k], ex, dex);
                zeta += w.gam * fk * te_g<T>(w.c2, w.d2, w.h - cs) * ex;
            }
        }
        zeta = share_sum<KS>(share, zeta);
        if (ks == 0) R.coef[t] = zeta;
    }
    __syncthreads();
    // a lane per bond: bond order, energy, pair part and the coefficient of
    // zeta's gradient; the two-body part is per bond, not per angle, and
    // float64 in both precisions
    for (int q = threadIdx.x; q < total; q += BLOCK) {
        const int m = F.map[q], t = m & (MAXN - 1);
        TeRow<T, MAXN> &R = rows[m / MAXN];
        const int mt = R.meta[t], sj = mt >> 9, si = R.si;
        const double *tij = tb + 10 * (si * ns + sj);
        const double *tp = mt & 256 ? tij : tb + 10 * (sj * ns + si);
        const double z = (double)R.coef[t];
        T coef = T(0);
        double cx = 0.0, e = 0.0;
        if (tp[0] != 0.0) {
            const double r = te_get_r(R, t);
            double fc, dfc;
            te_cut<double>(r, tp[5], tp[6], fc, dfc);
            if (fc != 0.0 || dfc != 0.0) {
                // b = (1 + (beta zeta)^n)^(-1 / (2 n)) by logarithms (beta
                // zeta > 0): half the cost of two pow()
                const double beta = tij[7], nn = tij[8];
                double b = 1.0, db = 0.0;
                if (z > 0.0 && beta != 0.0) {
                    double bz;
                    if (beta > 0.0) {
                        bz = exp(nn * log(beta * z));
                        b = exp(-0.5 / nn * log(1.0 + bz));
                    } else {
                        bz = pow(beta * z, nn);
                        b = pow(1.0 + bz, -0.5 / nn);
                    }
                    db = -0.5 * b * bz / (z * (1.0 + bz));
                }
                const double l1 = tp[3], l2 = tp[4];
                const double fr = tp[1] * clamped_exp<double>(-l1 * r);
                const double fa = -tp[2] * clamped_exp<double>(-l2 * r);
                e = 0.5 * (fc * (fr + b * fa));
                cx = 0.5 * (dfc * (fr + b * fa) + fc * (-l1 * fr - l2 * b * fa)) / r;
                if (fabs(db) > 1e-30) coef = (T)(0.5 * fc * fa * db);
            }
        }
        R.coef[t] = coef;
        R.e[t] = cx;
        R.gx[t] = e;
    }
    __syncthreads();
    // dU_i / dr of every leg, KS lanes each: t as the bond partner of zeta_t's
    // terms and as the third atom of the other bonds' terms.  With c =
    // cos(t, k), both parts point along d_k and d_t:
    //   d = A (d_k / (r_t r_k) - c d_t / r_t^2) + B d_t
    for (int q = threadIdx.x / KS; q < total; q += BLOCK / KS) {
        const int m = F.map[q], t = m & (MAXN - 1);
        TeRow<T, MAXN> &R = rows[m / MAXN];
        const int nl = R.nl, si = R.si;
        double gx = 0, gy = 0, gz = 0, gs = 0;
        const T xs = R.x[t], ys = R.y[t], zs = R.z[t];
        const T irs = R.ir[t], ct = R.coef[t], ft = R.fk[t], dft = R.dfk[t], ir2 = irs * irs;
        auto add = [&](T A, T B_, T c, T ii, T xk, T yk, T zk) {
            const T Ai = A * ii;
            gx += (double)(Ai * xk);
            gy += (double)(Ai * yk);
            gz += (double)(Ai * zk);
            gs += (double)(B_ - A * c * ir2);
        };
        if (small && B.plain[si]) {
            const TeTri<T> own = B.tri[si * ns * ns];
            for (int k = ks; k < nl; k += KS) {
                const T ck = R.coef[k], w = ct * R.fk[k] + ck * ft;
                if (k == t || (w == T(0) && ck == T(0))) continue;
                const T xk = R.x[k], yk = R.y[k], zk = R.z[k], ii = irs * R.ir[k];
                const T c = (xs * xk + ys * yk + zs * zk) * ii;
                T gg, dg;
                te_gdg<T>(own.c2, own.cd, own.d2, own.h - c, gg, dg);
                add(own.gam * w * dg, own.gam * ck * dft * gg * irs, c, ii, xk, yk, zk);
            }
        } else {
            const T rs = R.r[t];
            const int s_t = R.meta[t] >> 9;
            for (int k = ks; k < nl; k += KS) {
                const T fk = R.fk[k], ck = R.coef[k];
                const bool as_j = ct != T(0) && fk != T(0), as_k = ck != T(0) && ft != T(0);
                if (k == t || !(as_j || as_k)) continue;
                const int s_k = R.meta[k] >> 9;
                const T xk = R.x[k], yk = R.y[k], zk = R.z[k], ii = irs * R.ir[k];
                const T c = (xs * xk + ys * yk + zs * zk) * ii;
                T A = T(0), B_ = T(0), gg, dg, ex, dex;
                if (as_j) {
                    const TeTri<T> u = tri_row((si * ns + s_t) * ns + s_k);
                    if (u.valid != T(0)) {
                        te_gdg<T>(u.c2, u.cd, u.d2, u.h - c, gg, dg);
                        te_expo<T>(u.l3, u.m, rs - R.r[k], ex, dex);
                        const T w = ct * u.gam * fk;
                        A += w * dg * ex;
                        B_ += w * gg * dex * irs;
                    }
                }
                if (as_k) {
                    const TeTri<T> u = tri_row((si * ns + s_k) * ns + s_t);
                    if (u.valid != T(0)) {
                        te_gdg<T>(u.c2, u.cd, u.d2, u.h - c, gg, dg);
                        te_expo<T>(u.l3, u.m, R.r[k] - rs, ex, dex);
                        const T w = ck * u.gam;
                        A += w * ft * dg * ex;
                        B_ += w * gg * (dft * ex - ft * dex) * irs;
                    }
                }
                add(A, B_, c, ii, xk, yk, zk);
            }
        }
        gx = share_sum<KS>(share, gx);
        gy = share_sum<KS>(share, gy);
        gz = share_sum<KS>(share, gz);
        gs = share_sum<KS>(share, gs);
        if (ks == 0) {
            gs += R.e[t];
            R.e[t] = R.gx[t];
            const double Dx = gx + gs * (double)xs, Dy = gy + gs * (double)ys, Dz = gz + gs * (double)zs;
            R.gx[t] = Dx;
            R.gy[t] = Dy;
            R.gz[t] = Dz;
            if (so.dudv) {  // engine/site_terms.py:312-437: own bond order
                const size_t os = 3 * (size_t)(R.beg + (R.meta[t] & 255));
                so.dudv[os] = Dx;
                so.dudv[os + 1] = Dy;
                so.dudv[os + 2] = Dz;
            }
            // the force on neighbour x goes to x's own slot (x -> i)
            const size_t o = 3 * (size_t)R.rev[t];
            slot_G[o] = -Dx;
            slot_G[o + 1] = -Dy;
            slot_G[o + 2] = -Dz;
        }
    }
    __syncthreads();
    sum_legs<LPA>(mine, st, g < GPB && i < S.n_atoms ? i : -1, per_atom, f_local, so.e);
    }
}

// Everything one launch needs besides the shape.
struct TeArgs {
    SysView S;
    const mbf_nlist *nl;
    TeDev P;
    double *slot_G, *f_local, *per_atom;
    unsigned *live_mask;
    ClearWords clr;
    SiteOut so;
};

template <typename T, int MAXN, int LPA>
static int te_launch(const TeArgs &A, cudaStream_t st) {
    constexpr int GPB = TeGeom<MAXN, LPA>::GPB, BLOCK = TeGeom<MAXN, LPA>::BLOCK;
    const int blocks = persistent_grid((A.S.n_atoms + GPB - 1) / GPB, BLOCK, (const void *)te_center<T, MAXN, LPA>);
    PROF_BEGIN("te_center", st);
    te_center<T, MAXN, LPA><<<blocks, BLOCK, 0, st>>>(A.S, A.nl->row_off, A.nl->nbr, A.nl->rev, A.P, A.slot_G, A.f_local,
                                                      A.per_atom, A.live_mask,
                                                      (int)A.nl->n_slots, A.clr, A.so);
    PROF_END("te_center", st);
    MBF_CHECK_LAUNCH();
    return MBF_OK;   // the eval's gather_live adds the slot forces
}

template <typename T, int MAXN>
static int te_lpa(int lpa, const TeArgs &A, cudaStream_t st) {
    switch (lpa) {
        case 4: return te_launch<T, MAXN, 4>(A, st);
        case 8: return te_launch<T, MAXN, 8>(A, st);
        case 16: return te_launch<T, MAXN, 16>(A, st);
        default: return MBF_ERR_ARGUMENT;
    }
}

template <typename T>
static int te_rows(int mr, int lpa, const TeArgs &A, cudaStream_t st) {
    if (mr <= 32) return te_lpa<T, 32>(lpa, A, st);
    if (mr <= 64) return te_lpa<T, 64>(lpa, A, st);
    return te_lpa<T, 128>(lpa, A, st);
}

// The longest row te_rows' choice for `mr` stages.
static int te_row_limit(int mr) { return mr <= 32 ? 32 : (mr <= 64 ? 64 : 128); }

}  // namespace mbf

using namespace mbf;

static int tersoff_eval(const mbf_system *sys, const mbf_nlist *nl, const mbf_tersoff_tables *tab,
                        const mbf_reduce_plan *plan, int precision, int lanes_per_atom, void *workspace,
                        size_t workspace_bytes, double *forces, double *energy, double *virial, const SiteOut &so,
                        void *stream) {
    if (!sys || !nl || !tab || !plan || !workspace || !forces || !energy || !virial) return MBF_ERR_ARGUMENT;
    if (precision != MBF_FP64 && precision != MBF_MIXED) return MBF_ERR_ARGUMENT;
    if (nl->n_atoms != sys->n_atoms || tab->ns <= 0) return MBF_ERR_ARGUMENT;
    EvalLayout L = eval_layout(sys->n_atoms, nl->n_slots, plan->n_chunks);
    if (workspace_bytes < L.total) return MBF_ERR_WORKSPACE;
    cudaStream_t st = (cudaStream_t)stream;
    if (sys->n_atoms == 0) {
        if (cudaMemsetAsync(energy, 0, sizeof(double) * sys->n_struct, st) != cudaSuccess) return MBF_ERR_CUDA;
        if (cudaMemsetAsync(virial, 0, sizeof(double) * 9 * sys->n_struct, st) != cudaSuccess) return MBF_ERR_CUDA;
        return MBF_OK;
    }
    if (nl->n_slots < 0 || nl->n_slots > 0x7fffff00LL) return MBF_ERR_ARGUMENT;
    if (nl->max_row > 128) return MBF_ERR_ROW_TOO_LONG;
    // the per-structure completion counters live in a region of n_chunks
    // words; every structure owns at least one chunk
    if (plan->n_chunks <= 0 || sys->n_struct <= 0 || plan->n_chunks < sys->n_struct) return MBF_ERR_ARGUMENT;
    TeArgs A;
    A.S = make_view(sys);
    A.nl = nl;
    A.P.ns = tab->ns;
    A.P.tb = tab->tb;
    A.P.tri = tab->tri;
    A.P.rc = tab->r_cut;
    A.slot_G = ws_at<double>(workspace, L.slot);
    A.f_local = ws_at<double>(workspace, L.f_local);
    A.per_atom = ws_at<double>(workspace, L.per_atom);
    A.live_mask = live_mask_at(workspace, L);
    unsigned *sdone = ws_at<unsigned>(workspace, L.sdone);
    int *err = ws_at<int>(workspace, L.err);
    A.clr = {(unsigned *)err, ERR_CLEAR_BYTES / 4, sdone, sys->n_struct};
    A.so = so;
    const int lpa = lanes_per_atom > 0 ? lanes_per_atom : 8;
    int rc = precision == MBF_FP64 ? te_rows<double>(nl->max_row, lpa, A, st) : te_rows<float>(nl->max_row, lpa, A, st);
    if (rc != MBF_OK) return rc;
    return gather_live(sys->n_struct, sys->n_atoms, nl->row_off, (int)nl->n_slots, A.slot_G, A.live_mask,
                       te_row_limit(nl->max_row), err, A.f_local, forces, A.per_atom, plan,
                       ws_at<double>(workspace, L.partial), energy, virial, sdone, st);
}

extern "C" int mbf_tersoff_eval(const mbf_system *sys, const mbf_nlist *nl, const mbf_tersoff_tables *tab,
                                const mbf_reduce_plan *plan, int precision, int lanes_per_atom, void *workspace,
                                size_t workspace_bytes, double *forces, double *energy, double *virial,
                                void *stream) {
    SiteOut none = {nullptr, nullptr, nullptr};
    return tersoff_eval(sys, nl, tab, plan, precision, lanes_per_atom, workspace, workspace_bytes, forces, energy,
                        virial, none, stream);
}

extern "C" int mbf_tersoff_eval_sites(const mbf_system *sys, const mbf_nlist *nl, const mbf_tersoff_tables *tab,
                                      const mbf_reduce_plan *plan, int precision, int lanes_per_atom,
                                      void *workspace, size_t workspace_bytes, double *forces, double *energy,
                                      double *virial, double *site_e, double *site_dudv, double *site_vec,
                                      void *stream) {
    if (!site_e || !site_dudv || !site_vec) return MBF_ERR_ARGUMENT;
    if (nl && nl->n_slots > 0 &&
        cudaMemsetAsync(site_dudv, 0, sizeof(double) * 3 * (size_t)nl->n_slots, (cudaStream_t)stream) != cudaSuccess)
        return MBF_ERR_CUDA;
    SiteOut so = {site_e, site_dudv, site_vec};
    return tersoff_eval(sys, nl, tab, plan, precision, lanes_per_atom, workspace, workspace_bytes, forces, energy,
                        virial, so, stream);
}
