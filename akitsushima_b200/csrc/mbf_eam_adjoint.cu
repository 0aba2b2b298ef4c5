// Zhou EAM adjoint: the vector-Jacobian product of (E, F, virial) with
// respect to the function rows P (nf, 43) of an analytic Zhou (2004) table,
// for fitting.
//
// As for the Tersoff adjoint, the pull-back of upstream gradients gE, gF, gW
// onto a parameter theta is d/dtheta [sum_s gE_s E_s + D_t E], D_t the
// derivative along the tangent field t_ij = gF_i - gF_j - gW d_ij of the pair
// vectors.  The energy is a sum of site terms
//
//   U_i = F_{s_i}(rho-bar_i) + 1/2 sum_j phi_{s_i s_j}(r_ij),
//   rho-bar_i = sum_j rho_{s_j}(r_ij)      (engine/eam.py:174-256),
//
// with the Zhou forms of engine/eam_zhou.py:20-115 (density and pair
// functions times the quintic switch, the cross pair
// 1/2 k (f_b/f_a phi_aa + f_a/f_b phi_bb), embedding eqs. (A6)-(A8)).
// Per atom, in float64 hyper-dual arithmetic (one tangent, K parameter
// directions):
//   Q_i = gE F(rho-bar) + F'(rho-bar) D_t rho-bar + 1/2 sum_j (gE phi + D_t phi).
// The embedding's 12 parameters and rho-bar itself are the 13 directions of
// one evaluation of F; with c1 = gE F' + F'' D_t rho-bar and c2 = F', a
// density parameter's site value is c1 d(rho)/dtheta + c2 d(D_t rho)/dtheta.
// Density and pair functions are built from decays
// g(r; r_e, exponent, shift), whose parameter derivatives and tangents are
// written out from d ln g; an element's eight parameters and the cross pair's
// (f_a, u_a, f_b, u_b) dependence are chained by hand from those.
//
// Passes: rho-bar and its tangent (8 lanes per atom), which also marks and
// counts the live pairs above the diagonal by unordered species pair; the
// embedding sites (a thread per atom); a scan and a compaction into one list
// per species pair; one pass over each list with the site sums in registers;
// a final reduction onto the table entries.
//
// Sites of a species pair (a, b), a <= b (PAIR_SITES values):
//   0..7    the pair row phi_f[a, b]: the earlier species' r_e, f_e, alpha,
//           beta, A, B, kappa, lambda (columns 0, 1, 4..9)
//   8..15   the later species' (columns 20, 21, 24..29; a < b only)
//   16      the factor k (column 42; a < b only)
//   17..20  r_e, f_e, beta, lambda of row rho_f[b] (columns 0, 1, 5, 9), from
//           the a atom's density; for a = b, from both atoms'
//   21..24  the same of row rho_f[a], from the b atom's density (a < b only)
// and 12 per centre species: rho_e, rho_s, Fn0..Fn3, F0..F3, eta, F_e of row
// F_f[s] (columns 2, 3, 10..19).  Columns 40, 41 (switch radius and width) are
// not differentiated: the cutoff is fixed during a fit.  The gradient is with
// respect to the rows the generic Zhou evaluation reads (rho_f, F_f, phi_f);
// the fused path reads the same element parameters from the density rows,
// which the table builders fill identically.  Sites are reduced onto the
// entries in a fixed order: deterministic.
#include "mbf_hd.cuh"

namespace mbf {

constexpr int EADJ_NCOL = 43;
constexpr int EADJ_NZ = 20;

struct EamAdjTab {
    int ns, nf;
    const double *P;
    const int *rho_f, *F_f, *phi_f;
    double rc;
};

// g = exp(-expo (x - 1)) / (1 + (x - shift)^20), x = r / re, the decay every
// Zhou function is built from (engine/eam_zhou.py:20-45; ire = 1 / re): value,
// tangent (r's is rt), and for (re, expo, shift) the derivatives p and their tangents q.
// With w = 20 u^19 / (1 + u^20), u = x - shift: d ln g / dx = -(expo + w),
// / d expo = -(x - 1), / d shift = w, and w' = 380 u^18 / (1 + u^20) - w^2;
// p_k = g l_k and q_k = g_t l_k + g (l_k)_t.
struct Decay {
    double v, t, p[3], q[3];
};

__device__ __forceinline__ Decay zdecay3(double r, double rt, double ire, double expo, double shift) {
    const double x = r * ire, xt = rt * ire, u = x - shift;
    const double u2 = u * u, u4 = u2 * u2, u8 = u4 * u4, u16 = u8 * u8, u18 = u16 * u2;
    const double id = 1.0 / fma(u18, u2, 1.0);
    const double w = 20.0 * u18 * u * id, wx = 380.0 * u18 * id - w * w, lx = -(expo + w);
    Decay g;
    g.v = exp(-expo * (x - 1.0)) * id;
    g.t = g.v * lx * xt;
    const double l0 = -lx * x * ire, l0t = (wx * x - lx) * ire * xt;
    g.p[0] = g.v * l0;
    g.p[1] = -g.v * (x - 1.0);
    g.p[2] = g.v * w;
    g.q[0] = fma(g.t, l0, g.v * l0t);
    g.q[1] = -fma(g.t, x - 1.0, g.v * xt);
    g.q[2] = fma(g.t, w, g.v * wx * xt);
    return g;
}

// The quintic switch (columns 40, 41 of a row) at r, from its start r0 = rc -
// width and iw = 1 / width: value and tangent.
struct Switch {
    double r0, iw;
};
__device__ __forceinline__ Switch switch_of(const double *row) {
    return {row[2 * EADJ_NZ] - row[2 * EADJ_NZ + 1], 1.0 / row[2 * EADJ_NZ + 1]};
}
__device__ __forceinline__ void hz_switch(const Switch &w, double r, double rt, double &S, double &St) {
    double s = (r - w.r0) * w.iw;
    s = s < 0.0 ? 0.0 : (s > 1.0 ? 1.0 : s);
    S = 1.0 - s * s * s * (10.0 - 15.0 * s + 6.0 * s * s);
    St = -30.0 * s * s * (1.0 - s) * (1.0 - s) * w.iw * rt;
}

// One element's density f = f_e gB and pair u = A gA - B gB (unswitched),
// gA = g(r; r_e, alpha, kappa), gB = g(r; r_e, beta, lambda), enter a site
// value through their parameter derivatives (p) and the tangent of those
// (q): site_k += af f.p_k + bf f.q_k + au u.p_k + bu u.q_k, for the 8
// element parameters r_e, f_e, alpha, beta, A, B, kappa, lambda (columns 0,
// 1, 4..9 of p).
__device__ __forceinline__ void hz_species_sites(double *o, const Decay &gA, const Decay &gB, const double *p,
                                                 double af, double bf, double au, double bu) {
    double fe = p[1], A = p[6], B = p[7];
    o[0] += fe * (af * gB.p[0] + bf * gB.q[0]) + au * (A * gA.p[0] - B * gB.p[0]) + bu * (A * gA.q[0] - B * gB.q[0]);
    o[1] += af * gB.v + bf * gB.t;
    o[2] += A * (au * gA.p[1] + bu * gA.q[1]);
    o[3] += (fe * af - B * au) * gB.p[1] + (fe * bf - B * bu) * gB.q[1];
    o[4] += au * gA.v + bu * gA.t;
    o[5] -= au * gB.v + bu * gB.t;
    o[6] += A * (au * gA.p[2] + bu * gA.q[2]);
    o[7] += (fe * af - B * au) * gB.p[2] + (fe * bf - B * bu) * gB.q[2];
}

// Zhou embedding F(rho), eqs. (A6)-(A8) (engine/eam_zhou.py:66-115), with
// rho_e, rho_s, Fn0..3, F0..3, eta, F_e (columns 2, 3, 10..19) as directions
// 0..11 and rho itself as direction 12.
__device__ __forceinline__ HD<13> hz_embed(const double *p, double rho, double rho_t) {
    HD<13> q[12];
    const int col[12] = {2, 3, 10, 11, 12, 13, 14, 15, 16, 17, 18, 19};
#pragma unroll
    for (int k = 0; k < 12; ++k) q[k] = hd_param<13>(p[col[k]], k, 0);
    HD<13> x = hd_param<13>(rho, 12, 0);
    x.t = rho_t;
    const HD<13> &re = q[0], &rs = q[1], &eta = q[10], &Fe = q[11];
    if (rho < 0.85 * re.v) {
        HD<13> z = x / (0.85 * re) + (-1.0);
        return q[2] + z * (q[3] + z * (q[4] + z * q[5]));
    }
    if (rho >= 1.15 * re.v) {
        HD<13> lt = hd_log<13>(x / rs);
        HD<13> el = eta * lt;
        return Fe * ((1.0 + (-1.0) * el) * hd_exp<13>(el));
    }
    HD<13> z = x / re + (-1.0);
    return q[6] + z * (q[7] + z * (q[8] + z * q[9]));
}

__device__ __forceinline__ const double *row_of(const EamAdjTab &T, int f) { return T.P + (size_t)f * EADJ_NCOL; }

// A density row's constants for pass 1, and value and r-tangent of
// f_e g(r; r_e, beta, lambda) S(r).
struct DensRow {
    double ire, fe, beta, lam;
    Switch sw;
};
__device__ __forceinline__ void dens_value(const DensRow &p, double r, double rt, double &v, double &vt) {
    const double x = r * p.ire, u = x - p.lam;
    const double u2 = u * u, u4 = u2 * u2, u8 = u4 * u4, u16 = u8 * u8, u19 = u16 * u2 * u;
    const double id = 1.0 / fma(u19, u, 1.0);
    const double g = p.fe * exp(-p.beta * (x - 1.0)) * id;
    double Sw, St;
    hz_switch(p.sw, r, rt, Sw, St);
    v = g * Sw;
    vt = g * (St - (p.beta + 20.0 * u19 * id) * p.ire * rt * Sw);
}

constexpr int EADJ_TA = 128;         // atoms per block of the embedding pass
constexpr int EADJ_LPA = 8;          // lanes per atom of the row passes
constexpr int EADJ_PS = 25;          // sites of a species pair
constexpr int EADJ_PB = 128;         // threads of a pair block
constexpr int EADJ_PG = 148 * 4;     // pair blocks per species pair at most

// Index of the unordered species pair (a, b).
__device__ __forceinline__ int pair_code(int a, int b, int ns) {
    const int lo = min(a, b), hi = max(a, b);
    return lo * ns - lo * (lo - 1) / 2 + hi - lo;
}

// Position and upstream force gradient of an atom.
struct PairAtom {
    double x[3], f[3];
    __device__ __forceinline__ void load(const SysView &S, const AdjIn &G, int a) {
#pragma unroll
        for (int k = 0; k < 3; ++k) {
            x[k] = __ldg(S.pos + 3 * (size_t)a + k);
            f[k] = G.gF ? __ldg(G.gF + 3 * (size_t)a + k) : 0.0;
        }
    }
};

// What a structure contributes to its pairs' geometry: the cell, and the
// upstream virial gradient's symmetric part (only d . gW d enters).
struct PairCell {
    RowCell cell;
    double w[6];  // xx yy zz 2xy 2xz 2yz of the symmetric part
    __device__ __forceinline__ void load(const SysView &S, const AdjIn &G, int atom, int sst) {
        cell.load(S, atom);
        if (G.gW) {
            const double *g = G.gW + 9 * (size_t)sst;
            w[0] = __ldg(g);
            w[1] = __ldg(g + 4);
            w[2] = __ldg(g + 8);
            w[3] = __ldg(g + 1) + __ldg(g + 3);
            w[4] = __ldg(g + 2) + __ldg(g + 6);
            w[5] = __ldg(g + 5) + __ldg(g + 7);
        } else {
#pragma unroll
            for (int k = 0; k < 6; ++k) w[k] = 0.0;
        }
    }
    // r^2, r and the tangent of r of the pair (i, j): t_ij = gF_i - gF_j - gW d
    // enters only through d . t / r.
    __device__ __forceinline__ void pair(const PairAtom &i, const PairAtom &j, double &r2, double &r, double &rt) const {
        double x, y, z;
        cell.mic(j.x[0] - i.x[0], j.x[1] - i.x[1], j.x[2] - i.x[2], x, y, z);
        r2 = x * x + y * y + z * z;
        const double ir = rsqrt(r2);
        r = r2 * ir;
        rt = ir * (x * (i.f[0] - j.f[0]) + y * (i.f[1] - j.f[1]) + z * (i.f[2] - j.f[2]) -
                   (x * (w[0] * x + w[3] * y + w[4] * z) + y * (w[1] * y + w[5] * z) + z * (w[2] * z)));
    }
};

// Pass 1, EADJ_LPA lanes per atom over its full row: rho-bar and its tangent
// into rr.  Slots above the diagonal get a mark (1 + the neighbour's species
// where the pair is inside the cutoff, else 0), and cnt[c * n_atoms + i]
// counts them by species pair.  Bound by FP64 issue and the scattered loads
// of the neighbours: 170 us for 101,000 atoms of 134 slots (a thread per atom,
// with the embedding at its end, took 340).
__global__ void __launch_bounds__(128) eam_adjoint_density(SysView S, const int *__restrict__ row_off,
                                                           const int *__restrict__ upper, const int *__restrict__ nbr,
                                                           EamAdjTab T, AdjIn G, double2 *__restrict__ rr,
                                                           unsigned char *__restrict__ mark, int *__restrict__ cnt) {
    constexpr int LPA = EADJ_LPA;
    __shared__ DensRow dens[8];
    const int i = (blockIdx.x * blockDim.x + threadIdx.x) / LPA, sub = threadIdx.x & (LPA - 1);
    const bool in = i < S.n_atoms;
    const int ns = T.ns;
    for (int k = threadIdx.x; k < ns; k += blockDim.x) {
        const double *p = row_of(T, T.rho_f[k]);
        dens[k] = {1.0 / p[0], p[1], p[5], p[9], switch_of(p)};
    }
    __syncthreads();
    const double rc2 = T.rc * T.rc;
    double rho = 0.0, rho_t = 0.0;
    unsigned long long c0 = 0ull, c1 = 0ull;  // marked slots by species, 16 bits each (species 0-3, 4-7)
    int si = 0;
    if (in) {
        si = S.types[i];
        const int sst = S.n_struct > 1 ? S.atom_struct[i] : 0, up = upper[i], end = row_off[i + 1];
        PairCell pc;
        pc.load(S, G, i, sst);
        // slot indices two iterations ahead, the neighbour's data one ahead
        int s = row_off[i] + sub, j1 = s + LPA < end ? nbr[s + LPA] : i, tn = 0;
        PairAtom me, nx;
        me.load(S, G, i);
        if (s < end) {
            const int j0 = nbr[s];
            nx.load(S, G, j0);
            tn = S.types[j0];
        }
        for (; s < end; s += LPA) {
            const PairAtom at = nx;
            const int sj = tn;
            if (s + LPA < end) {
                nx.load(S, G, j1);
                tn = S.types[j1];
            }
            if (s + 2 * LPA < end) j1 = nbr[s + 2 * LPA];
            double r2, r, rt;
            pc.pair(me, at, r2, r, rt);
            const bool live = r2 < rc2 && r2 > 1e-24;
            if (live) {
                double v, vt;
                dens_value(dens[sj], r, rt, v, vt);
                rho += v;
                rho_t += vt;
            }
            if (s >= up) {
                mark[s] = live ? (unsigned char)(1 + sj) : 0;
                if (live) (sj < 4 ? c0 : c1) += 1ull << (16 * (sj & 3));
            }
        }
    }
    rho = group_sum<LPA>(rho);
    rho_t = group_sum<LPA>(rho_t);
    c0 = group_sum<LPA>(c0);
    c1 = group_sum<LPA>(c1);
    if (!in) return;
    if (sub == 0) rr[i] = make_double2(rho, rho_t);
    for (int c = sub, a = 0, first = 0; c < ns * (ns + 1) / 2; c += LPA) {
        while (c >= first + ns - a) first += ns - a++;  // c = pair_code(a, b)
        const int b = a + c - first, o = a == si ? b : (b == si ? a : -1);
        cnt[(size_t)c * S.n_atoms + i] = o < 0 ? 0 : (int)((o < 4 ? c0 : c1) >> (16 * (o & 3)) & 0xffffull);
    }
}

// Pass 2, a thread per atom: the embedding sites (12; summed per species of
// the centre into the block's partialF row) and the coefficients c1 = gE F' +
// F'' D_t rho-bar, c2 = F' through which every density parameter acts on this
// atom's site term (cc, in place of rr).
__global__ void __launch_bounds__(EADJ_TA) eam_adjoint_embed(SysView S, EamAdjTab T, AdjIn G, double2 *__restrict__ cc,
                                                             double *__restrict__ partialF) {
    __shared__ double sf[EADJ_TA * 13];  // 12 sites per atom, odd stride
    __shared__ int scode[EADJ_TA];
    const int nf = 12 * T.ns;
    const int i = blockIdx.x * EADJ_TA + threadIdx.x;
    int code = -1;
    double *o = sf + 13 * threadIdx.x;
    if (i < S.n_atoms) {
        const int si = S.types[i];
        const int sst = S.n_struct > 1 ? S.atom_struct[i] : 0;
        const double gE = G.gE ? G.gE[sst] : 0.0;
        const double2 rr = cc[i];
        // the embedding, rho-bar clamped at 0 as the evaluation does
        const double rb = rr.x > 0.0 ? rr.x : 0.0;
        HD<13> F = hz_embed(row_of(T, T.F_f[si]), rb, rr.y);
#pragma unroll
        for (int k = 0; k < 12; ++k) o[k] = gE * F.p[k] + F.q[k];
        cc[i] = make_double2(rr.x > 0.0 ? gE * F.p[12] + F.q[12] : 0.0, F.p[12]);
        code = si;
    }
    scode[threadIdx.x] = code;
    __syncthreads();
    const int cnt = min(EADJ_TA, S.n_atoms - (int)blockIdx.x * EADJ_TA);
    for (int item = threadIdx.x; item < nf; item += blockDim.x) {
        const int sp = item / 12, k = item % 12;
        double a = 0.0;
        for (int q = 0; q < cnt; ++q)
            if (scode[q] == sp) a += sf[13 * q + k];
        partialF[(size_t)item * gridDim.x + blockIdx.x] = a;  // (site, block)
    }
}

// Compaction, a warp per atom: the marked slots of its upper half as pairs
// (atom of the earlier species, atom of the later) at the scanned offsets,
// each list in atom then slot order.  A chain of loads: with 8 lanes an atom,
// nine rounds over a half row of 67, it took 65 us with its scan for the 6.8 M
// slots of 101,000 Ni3Al atoms, with 16 lanes 49, with 32 41.
__global__ void __launch_bounds__(128) eam_adjoint_compact(int n_atoms, int ns, const int *__restrict__ types,
                                                           const int *__restrict__ row_off,
                                                           const int *__restrict__ upper, const int *__restrict__ nbr,
                                                           const unsigned char *__restrict__ mark,
                                                           const int *__restrict__ pos, int2 *__restrict__ pairs) {
    const int i = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, sub = threadIdx.x & 31;
    if (i >= n_atoms) return;  // whole warps leave together
    const int si = types[i], beg = upper[i], end = row_off[i + 1];
    // lane b keeps the next position in species b's list
    int next = sub < ns ? pos[(size_t)pair_code(si, sub, ns) * n_atoms + i] : 0;
    int mn = 0, jn = 0;
    if (beg + sub < end) {
        mn = mark[beg + sub];
        jn = nbr[beg + sub];
    }
    for (int s0 = beg; s0 < end; s0 += 32) {
        const int m = mn, j = jn, s1 = s0 + 32 + sub;
        mn = 0;
        if (s1 < end) {
            mn = mark[s1];
            jn = nbr[s1];
        }
        int o = -1;
        for (int b = 0; b < ns; ++b) {
            const unsigned hit = __ballot_sync(MBF_FULL, m == 1 + b);
            const int base = __shfl_sync(MBF_FULL, next, b);
            if (m == 1 + b) o = base + __popc(hit & ((1u << sub) - 1u));
            if (sub == b) next += __popc(hit);
        }
        if (o >= 0) pairs[o] = si <= m - 1 ? make_int2(i, j) : make_int2(j, i);
    }
}

// Density sites of a neighbour species' row at r: f_e gB S, contributing
// c1 d(rho)/dtheta + c2 d(D_t rho)/dtheta to r_e, f_e, beta, lambda (o[0..3]).
__device__ __forceinline__ void dens_sites(double *o, const Decay &gB, const double *row, double Sw, double St,
                                           double c1, double c2) {
    const double a = c1 * Sw + c2 * St, bq = c2 * Sw, af = a * row[1], bf = bq * row[1];
    o[0] += af * gB.p[0] + bf * gB.q[0];
    o[1] += a * gB.v + bq * gB.t;
    o[2] += af * gB.p[1] + bf * gB.q[1];
    o[3] += af * gB.p[2] + bf * gB.q[2];
}

// A block's constants of its species pair: 1 / r_e and the switches of the
// pair row and of the density rows, and whether a density row's decay and
// switch are those of the pair row's element (they are in a table built from
// one set of element parameters, and are then evaluated once).
struct PairConst {
    double ire_a, ire_b, ire_da, ire_db;
    Switch sw, sw_a, sw_b;
    int same_a, same_b;
};
__device__ __forceinline__ bool same_decay(const double *dr, const double *blk) {
    return dr[0] == blk[0] && dr[5] == blk[5] && dr[9] == blk[9];
}

// Pass 3, one species pair per blockIdx.y: a thread takes every
// EADJ_PB-th pair of its block's contiguous share of the list and keeps the
// site sums in registers; the block's sums go to its row of `partial`.  Sites
// staged in shared memory per tile of pairs and summed there by entry, with
// the decays in generic hyper-dual arithmetic, took 714 us for the 4.9 M
// pairs of 101,000 Ni3Al atoms; this pass takes 228.  Bound by FP64 issue and
// its latency (38-45 % of the FP64 pipe).
// Resident blocks: 4 of 128 registers for the like pairs, 2 of 202 for the
// cross pairs (101,000 atoms, both: 228 us; 5 spills: 259; 3 cross blocks: 241).
template <bool LIKE>
__global__ void __launch_bounds__(EADJ_PB, LIKE ? 4 : 2) eam_adjoint_pairs(SysView S, EamAdjTab T, AdjIn G,
                                                             const double2 *__restrict__ cc,
                                                             const int2 *__restrict__ pairs,
                                                             const int *__restrict__ pos,
                                                             double *__restrict__ partial) {
    constexpr int NV = LIKE ? 12 : EADJ_PS;
    __shared__ double rows[4][EADJ_NCOL];   // pair row, the two density rows
    __shared__ double sums[EADJ_PB / 32][NV];
    __shared__ PairConst K;
    const int ns = T.ns;
    int a = blockIdx.y, b = blockIdx.y;
    if (!LIKE) {  // the blockIdx.y-th pair a < b
        a = 0;
        int q = blockIdx.y;
        while (q >= ns - 1 - a) q -= ns - 1 - a++;
        b = a + 1 + q;
    }
    const int c = pair_code(a, b, ns);
    for (int k = threadIdx.x; k < EADJ_NCOL; k += blockDim.x) {
        rows[0][k] = row_of(T, T.phi_f[a * ns + b])[k];
        rows[1][k] = row_of(T, T.rho_f[a])[k];
        rows[2][k] = row_of(T, T.rho_f[b])[k];
    }
    __syncthreads();
    const double *row = rows[0], *rho_a = rows[1], *rho_b = rows[2], *pb = LIKE ? row : row + EADJ_NZ;
    if (threadIdx.x == 0) {
        K.ire_a = 1.0 / row[0];
        K.ire_b = 1.0 / pb[0];
        K.ire_da = 1.0 / rho_a[0];
        K.ire_db = 1.0 / rho_b[0];
        K.sw = switch_of(row);
        K.sw_a = switch_of(rho_a);
        K.sw_b = switch_of(rho_b);
        const bool w_a = row[40] == rho_a[40] && row[41] == rho_a[41], w_b = row[40] == rho_b[40] && row[41] == rho_b[41];
        K.same_a = same_decay(rho_a, row) && w_a;
        K.same_b = same_decay(rho_b, pb) && w_b;
    }
    __syncthreads();
    double o[NV];
#pragma unroll
    for (int k = 0; k < NV; ++k) o[k] = 0.0;
    const int p0 = pos[(size_t)c * S.n_atoms], np = pos[(size_t)(c + 1) * S.n_atoms] - p0;
    const int per = (np + gridDim.x - 1) / gridDim.x;
    const int m1 = min(np, ((int)blockIdx.x + 1) * per);
    for (int m = (int)blockIdx.x * per + threadIdx.x; m < m1; m += EADJ_PB) {
        const int2 pq = pairs[p0 + m];
        const int sst = S.n_struct > 1 ? __ldg(S.atom_struct + pq.x) : 0;
        const double gE = G.gE ? __ldg(G.gE + sst) : 0.0;
        const double2 cp = cc[pq.x], cq = cc[pq.y];
        double r2, r, rt;
        PairCell pc;
        pc.load(S, G, pq.x, sst);
        PairAtom ap, aq;
        ap.load(S, G, pq.x);
        aq.load(S, G, pq.y);
        pc.pair(ap, aq, r2, r, rt);
        double Sw, St;
        hz_switch(K.sw, r, rt, Sw, St);
        const Decay gA = zdecay3(r, rt, K.ire_a, row[4], row[8]);
        const Decay gB = zdecay3(r, rt, K.ire_a, row[5], row[9]);
        // the density sites of row rho (decay gD, or its own) with the
        // coefficients c of the atom that sees it
        auto density = [&](double *od, int same, const Decay &gD, const double *rho, double ire, const Switch &sw,
                           double cx, double cy) {
            if (same) {
                dens_sites(od, gD, rho, Sw, St, cx, cy);
            } else {
                double Dw, Dt;
                hz_switch(sw, r, rt, Dw, Dt);
                dens_sites(od, zdecay3(r, rt, ire, rho[5], rho[9]), rho, Dw, Dt, cx, cy);
            }
        };
        if constexpr (LIKE) {
            // phi = u S; the two atoms' densities are of the same row
            hz_species_sites(o, gA, gB, row, 0.0, 0.0, gE * Sw + St, Sw);
            density(o + 8, K.same_b, gB, rho_b, K.ire_db, K.sw_b, cp.x + cq.x, cp.y + cq.y);
        } else {
            // phi = k psi, psi = 1/2 S (A + B), A = q u_a, B = u_b / q, q =
            // f_b / f_a: psi's derivatives in (f_a, u_a, f_b, u_b) and their
            // tangents, then each element's chain
            const Decay hA = zdecay3(r, rt, K.ire_b, pb[4], pb[8]);
            const Decay hB = zdecay3(r, rt, K.ire_b, pb[5], pb[9]);
            const double fa = row[1] * gB.v, fat = row[1] * gB.t, fb = pb[1] * hB.v, fbt = pb[1] * hB.t;
            const double ua = row[6] * gA.v - row[7] * gB.v, uat = row[6] * gA.t - row[7] * gB.t;
            const double ub = pb[6] * hA.v - pb[7] * hB.v, ubt = pb[6] * hA.t - pb[7] * hB.t;
            const double inv = 1.0 / (fa * fb), ifa = fb * inv, ifb = fa * inv, q = fb * ifa, iq = fa * ifb;
            const double mt = fbt * ifb - fat * ifa;  // (ln q)_t
            const double A = q * ua, B = ub * iq, At = A * mt + q * uat, Bt = ubt * iq - B * mt;
            const double h = row[2 * EADJ_NZ + 2], hS = 0.5 * h * Sw, hSt = 0.5 * h * St;
            const double E = A - B, Et = At - Bt;
            const double wq = hS * q, wqt = q * (hSt + hS * mt), wi = hS * iq, wit = iq * (hSt - hS * mt);
            const double eb = hS * E * ifb, ebt = (hSt * E + hS * Et) * ifb - eb * (fbt * ifb);
            const double ea = -hS * E * ifa, eat = -(hSt * E + hS * Et) * ifa - ea * (fat * ifa);
            o[16] += 0.5 * (gE * Sw * (A + B) + St * (A + B) + Sw * (At + Bt));
            hz_species_sites(o, gA, gB, row, gE * ea + eat, ea, gE * wq + wqt, wq);
            density(o + 21, K.same_a, gB, rho_a, K.ire_da, K.sw_a, cq.x, cq.y);
            hz_species_sites(o + 8, hA, hB, pb, gE * eb + ebt, eb, gE * wi + wit, wi);
            density(o + 17, K.same_b, hB, rho_b, K.ire_db, K.sw_b, cp.x, cp.y);
        }
    }
    const int w = threadIdx.x >> 5, l = threadIdx.x & 31;
#pragma unroll
    for (int k = 0; k < NV; ++k) {
        double x = o[k];
#pragma unroll
        for (int d = 16; d > 0; d >>= 1) x += __shfl_xor_sync(MBF_FULL, x, d);
        if (l == 0) sums[w][k] = x;
    }
    __syncthreads();
    double *out = partial + (size_t)c * EADJ_PS * gridDim.x + blockIdx.x;  // (list, site, block)
    for (int k = threadIdx.x; k < EADJ_PS; k += blockDim.x) {
        const int v = !LIKE ? k : (k < 8 ? k : (k >= 17 && k < 21 ? k - 9 : -1));
        double x = 0.0;
        if (v >= 0)
            for (int q = 0; q < EADJ_PB / 32; ++q) x += sums[q][v];
        out[(size_t)k * gridDim.x] = x;
    }
}

// Column -> site of a role (-1: not differentiated).
__device__ __forceinline__ int f_site(int c) { return c == 2 ? 0 : (c == 3 ? 1 : (c >= 10 && c <= 19 ? c - 8 : -1)); }
__device__ __forceinline__ int d_site(int c) { return c == 0 ? 0 : (c == 1 ? 1 : (c == 5 ? 2 : (c == 9 ? 3 : -1))); }
__device__ __forceinline__ int p_site(int c) {
    if (c == 0 || c == 1) return c;
    if (c >= 4 && c <= 9) return c - 2;
    if (c == 20 || c == 21) return c - 12;
    if (c >= 24 && c <= 29) return c - 14;
    return c == 42 ? 16 : -1;
}

// One warp per entry (row f, column c) of d_P: the block partials that feed
// it -- the embedding sums of the row's species, the density sites of every
// pair with that species, the pair sites of the row's pair -- summed over
// blocks by lanes, then a fixed shuffle tree.
__global__ void eam_adjoint_final(EamAdjTab T, int gA, const double *__restrict__ partialF, int gP,
                                  const double *__restrict__ partial, double *__restrict__ d_P) {
    const int ns = T.ns;
    int e = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, l = threadIdx.x & 31;
    if (e >= T.nf * EADJ_NCOL) return;  // whole warps leave together
    int f = e / EADJ_NCOL, c = e % EADJ_NCOL;
    // one row of n block values: four loads in flight a lane
    double acc = 0.0;
    auto add_row = [&](const double *p, int n) {
        double x[4] = {0.0, 0.0, 0.0, 0.0};
        for (int b = l; b < n; b += 128) {
#pragma unroll
            for (int k = 0; k < 4; ++k)
                if (b + 32 * k < n) x[k] += p[b + 32 * k];
        }
        acc += (x[0] + x[1]) + (x[2] + x[3]);
    };
    for (int s = 0; s < ns; ++s)
        if (T.F_f[s] == f && f_site(c) >= 0) add_row(partialF + (size_t)(12 * s + f_site(c)) * gA, gA);
    const int k = p_site(c), d = d_site(c);
    for (int x = 0; x < ns; ++x)
        for (int y = x; y < ns; ++y) {
            const double *pp = partial + (size_t)pair_code(x, y, ns) * gP * EADJ_PS;
            if (T.phi_f[x * ns + y] == f && k >= 0 && (x != y || k < 8)) add_row(pp + (size_t)k * gP, gP);
            if (T.rho_f[y] == f && d >= 0) add_row(pp + (size_t)(17 + d) * gP, gP);
            if (x != y && T.rho_f[x] == f && d >= 0) add_row(pp + (size_t)(21 + d) * gP, gP);
        }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) acc += __shfl_xor_sync(MBF_FULL, acc, o);
    if (l == 0) d_P[e] = acc;
}

// Workspace of one call.
struct EadjLayout {
    size_t partialF, partial, cc, cnt, pos, mark, pairs, scan, total;
    int gA, gP, nc;
};

static EadjLayout eadj_layout(int n_atoms, long long n_slots, int ns) {
    EadjLayout L;
    const long long ns2 = n_slots > 0 ? n_slots : 1;
    const size_t na = (size_t)(n_atoms > 0 ? n_atoms : 1);
    L.nc = ns * (ns + 1) / 2;
    L.gA = (int)((na + EADJ_TA - 1) / EADJ_TA);
    // pair blocks per list: at least a few hundred pairs each
    const long long tiles = (ns2 / 2 + 4 * EADJ_PB - 1) / (4 * EADJ_PB);
    L.gP = (int)(tiles < 1 ? 1 : (tiles < EADJ_PG ? tiles : EADJ_PG));
    size_t o = 0;
    L.partialF = o;
    o = align256(o + sizeof(double) * (size_t)L.gA * 12 * ns);
    L.partial = o;
    o = align256(o + sizeof(double) * (size_t)L.nc * L.gP * EADJ_PS);
    L.cc = o;
    o = align256(o + sizeof(double2) * na);
    L.cnt = o;
    o = align256(o + sizeof(int) * L.nc * na);
    L.pos = o;
    o = align256(o + sizeof(int) * (L.nc * na + 1));
    L.mark = o;
    o = align256(o + (size_t)ns2);
    L.pairs = o;
    o = align256(o + sizeof(int2) * (size_t)(ns2 / 2 + 1));
    L.scan = o;
    o = align256(o + sizeof(int) * scan_workspace_ints((int)(L.nc * na)));
    L.total = o;
    return L;
}

}  // namespace mbf

using namespace mbf;

extern "C" {

size_t mbf_eam_adjoint_workspace_bytes(int n_atoms, long long n_slots, int ns) {
    if (n_atoms < 0 || n_slots < 0 || ns <= 0 || ns > 8 || n_slots > 0x7fffffffLL) return 0;
    return eadj_layout(n_atoms, n_slots, ns).total;
}

int mbf_eam_adjoint(const mbf_system *sys, const mbf_nlist *nl, const mbf_eam_tables *tab, const double *g_energy,
                    const double *g_forces, const double *g_virial, void *workspace, size_t workspace_bytes,
                    double *d_P, void *stream) {
    if (!sys || !nl || !tab || !workspace || !d_P || tab->ns <= 0 || tab->ns > 8 || tab->nf <= 0)
        return MBF_ERR_ARGUMENT;
    if (nl->n_atoms != sys->n_atoms || !nl->upper || nl->n_slots > 0x7fffffffLL) return MBF_ERR_ARGUMENT;
    EadjLayout L = eadj_layout(sys->n_atoms, nl->n_slots, tab->ns);
    if (workspace_bytes < L.total) return MBF_ERR_WORKSPACE;
    cudaStream_t st = (cudaStream_t)stream;
    int ne = tab->nf * EADJ_NCOL;
    if (sys->n_atoms == 0) {
        if (cudaMemsetAsync(d_P, 0, sizeof(double) * ne, st) != cudaSuccess) return MBF_ERR_CUDA;
        return MBF_OK;
    }
    if ((long long)L.nc * sys->n_atoms > 0x7fffff00LL) return MBF_ERR_ARGUMENT;  // the scan's integers
    SysView S = make_view(sys);
    EamAdjTab T;
    T.ns = tab->ns;
    T.nf = tab->nf;
    T.P = tab->P;
    T.rho_f = tab->rho_f;
    T.F_f = tab->F_f;
    T.phi_f = tab->phi_f;
    T.rc = tab->r_cut;
    AdjIn G;
    G.gE = g_energy;
    G.gF = g_forces;
    G.gW = g_virial;
    double *partialF = ws_at<double>(workspace, L.partialF);
    double *partial = ws_at<double>(workspace, L.partial);
    double2 *cc = ws_at<double2>(workspace, L.cc);
    int *cnt = ws_at<int>(workspace, L.cnt);
    int *pos = ws_at<int>(workspace, L.pos);
    unsigned char *mark = ws_at<unsigned char>(workspace, L.mark);
    int2 *pairs = ws_at<int2>(workspace, L.pairs);
    const int N = sys->n_atoms, ns = T.ns;
    const int rows = (int)(((long long)N * EADJ_LPA + 127) / 128);
    PROF_BEGIN("eam_adjoint_density", st);
    eam_adjoint_density<<<rows, 128, 0, st>>>(S, nl->row_off, nl->upper, nl->nbr, T, G, cc, mark, cnt);
    PROF_END("eam_adjoint_density", st);
    MBF_CHECK_LAUNCH();
    PROF_BEGIN("eam_adjoint_embed", st);
    eam_adjoint_embed<<<L.gA, EADJ_TA, 0, st>>>(S, T, G, cc, partialF);
    PROF_END("eam_adjoint_embed", st);
    MBF_CHECK_LAUNCH();
    PROF_BEGIN("eam_adjoint_compact", st);
    int rc = exclusive_scan(cnt, pos, L.nc * N, ws_at<int>(workspace, L.scan), st);
    if (rc != MBF_OK) return rc;
    eam_adjoint_compact<<<(N + 3) / 4, 128, 0, st>>>(N, ns, S.types, nl->row_off, nl->upper, nl->nbr, mark, pos, pairs);
    PROF_END("eam_adjoint_compact", st);
    MBF_CHECK_LAUNCH();
    PROF_BEGIN("eam_adjoint_pairs", st);
    eam_adjoint_pairs<true><<<dim3(L.gP, ns), EADJ_PB, 0, st>>>(S, T, G, cc, pairs, pos, partial);
    MBF_CHECK_LAUNCH();
    if (ns > 1) {
        eam_adjoint_pairs<false><<<dim3(L.gP, ns * (ns - 1) / 2), EADJ_PB, 0, st>>>(S, T, G, cc, pairs, pos, partial);
        MBF_CHECK_LAUNCH();
    }
    PROF_END("eam_adjoint_pairs", st);
    PROF_BEGIN("eam_adjoint_reduce", st);
    eam_adjoint_final<<<(ne * 32 + 127) / 128, 128, 0, st>>>(T, L.gA, partialF, L.gP, partial, d_P);
    PROF_END("eam_adjoint_reduce", st);
    MBF_CHECK_LAUNCH();
    return MBF_OK;
}

}  // extern "C"
