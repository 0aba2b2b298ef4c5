// Stillinger-Weber: one kernel for the two-body term and the three-body
// angles of each centre (per-slot forces on the neighbours), then the gather
// through the reverse-slot index.
//
// Replaces engine/stillinger_weber.py:900-1451: single species (:927-1159,
// each unordered neighbour pair once with lambda) and multi species
// (:1165-1451, both orders with lambda/2 of their own (i, j, k) record, legs
// from the pair records (i, j, j)).  The two-body term of a pair reads the
// record of the lower-indexed atom (:714-762).
#include "mbf_rows.cuh"

namespace mbf {

// Lanes per atom (LPA) is a template parameter chosen by the host (the
// autotuner); GPB lane groups per block keep the staged rows near 15 KB, so
// that registers and not shared memory bound the resident warps.  A block is
// whole warps: where shared memory holds the rows of half a warp's groups
// only, the other groups have no row.
template <int MAXN, int LPA> struct SwGeom {
    static constexpr int WIDE = 512 / MAXN < 32 / LPA ? 512 / MAXN : 32 / LPA;  // a whole warp, if 48 KB hold it
    static constexpr int GPB = 256 / MAXN > WIDE ? 256 / MAXN : WIDE;
    static constexpr int BLOCK = GPB * LPA < 32 ? 32 : GPB * LPA;
    static_assert(BLOCK % 32 == 0, "the record sums are over whole warps");
    // Resident threads per SM the kernel is compiled for (its registers):
    // with the gather, 64,000-atom Ge-Sn mixed at 640 / 768 / 896 threads 103 /
    // 98 / 96 us, 32,768-atom Ge-Sn float64 at 512 / 640 78 / 83.
    static constexpr int min_blocks(int size) { return (size == 8 ? 512 : 896) / BLOCK; }
};

struct SwDev {
    int ns;
    const double *tb;   // (ns*ns, 8): valid eps sigma a A B p q
    const double *leg;  // (ns*ns, 4): sigma a gamma -
    const double *tri;  // (ns^3, 4):  valid eps*lambda/2 costheta0 -
    double rc;
};

// Records as the kernel reads them, in T.
template <typename T> struct SwPair { T valid, eps, sig, a, A, B, p, q; };
template <typename T> struct SwLeg { T sig, a, gam, pad; };
template <typename T> struct SwTri { T c, cos0; };  // c = 0: no such angle

template <typename T>
__device__ __forceinline__ SwPair<T> sw_pair_row(const double *__restrict__ t) {
    return {(T)__ldg(t), (T)__ldg(t + 1), (T)__ldg(t + 2), (T)__ldg(t + 3),
            (T)__ldg(t + 4), (T)__ldg(t + 5), (T)__ldg(t + 6), (T)__ldg(t + 7)};
}
template <typename T>
__device__ __forceinline__ SwLeg<T> sw_leg_row(const double *__restrict__ t) {
    return {(T)__ldg(t), (T)__ldg(t + 1), (T)__ldg(t + 2), T(0)};
}
template <typename T>
__device__ __forceinline__ SwTri<T> sw_tri_row(const double *__restrict__ t) {
    return {__ldg(t) != 0.0 ? (T)__ldg(t + 1) : T(0), (T)__ldg(t + 2)};
}

// The square of the distance beyond which the pair (a, b) takes part in no
// term, from either atom (a little beyond: the terms test their own cutoff).
// Both atoms of a pair agree on it.
__device__ __forceinline__ double sw_reach2(const SwDev &P, int a, int b) {
    double r = 0.0;
    for (int o = 0; o < 2; ++o) {
        const int ab = o == 0 ? a * P.ns + b : b * P.ns + a;
        const double *t = P.tb + 8 * ab, *l = P.leg + 4 * ab;
        if (__ldg(t) != 0.0) r = fmax(r, __ldg(t + 2) * __ldg(t + 3));
        r = fmax(r, __ldg(l) * __ldg(l + 1));
    }
    return r * r * (1.0 + 1e-6);
}

// The records of an evaluation: of up to SW_SH species staged in shared
// memory in T, of more read from the tables.  The kernel is compiled for
// either, so every access is to one address space.
constexpr int SW_SH = 3;
template <typename T, bool STAGED>
struct SwTab {
    __device__ __forceinline__ void load(const SwDev &) {}
    __device__ __forceinline__ SwPair<T> pair(const SwDev &P, int q) const { return sw_pair_row<T>(P.tb + 8 * q); }
    __device__ __forceinline__ SwLeg<T> leg(const SwDev &P, int q) const { return sw_leg_row<T>(P.leg + 4 * q); }
    __device__ __forceinline__ SwTri<T> tri(const SwDev &P, int q) const { return sw_tri_row<T>(P.tri + 4 * q); }
    __device__ __forceinline__ double reach2(const SwDev &P, int a, int b) const { return sw_reach2(P, a, b); }
};

template <typename T>
struct SwTab<T, true> {
    SwPair<T> pairs[SW_SH * SW_SH];
    SwLeg<T> legs[SW_SH * SW_SH];
    SwTri<T> tris[SW_SH * SW_SH * SW_SH];
    double reach[SW_SH * SW_SH];
    __device__ __forceinline__ SwPair<T> pair(const SwDev &, int q) const { return pairs[q]; }
    __device__ __forceinline__ SwLeg<T> leg(const SwDev &, int q) const { return legs[q]; }
    __device__ __forceinline__ SwTri<T> tri(const SwDev &, int q) const { return tris[q]; }
    __device__ __forceinline__ double reach2(const SwDev &P, int a, int b) const { return reach[a * P.ns + b]; }
    // By the whole block; ends in a barrier.
    __device__ __forceinline__ void load(const SwDev &P) {
        const int ns = P.ns;
        for (int q = threadIdx.x; q < ns * ns; q += blockDim.x) {
            pairs[q] = sw_pair_row<T>(P.tb + 8 * q);
            legs[q] = sw_leg_row<T>(P.leg + 4 * q);
            reach[q] = sw_reach2(P, q / ns, q % ns);
        }
        for (int q = threadIdx.x; q < ns * ns * ns; q += blockDim.x) tris[q] = sw_tri_row<T>(P.tri + 4 * q);
        __syncthreads();
    }
};

// Per-leg factors of the three-body term (engine/stillinger_weber.py:96-154):
// h(i, j, k) = c3 E_j E_k (cos theta_jik - cos0)^2 with E_x = exp(gamma_x /
// (r_ix / sigma_x - a_x)) and dE_x/dr_ix = E_x D_x, D_x = -gamma_x /
// (sigma_x (r_ix / sigma_x - a_x)^2).  A leg at or beyond a_x sigma_x has
// E = D = 0, which zeroes every angle it takes part in (the reference's
// early return).  The legs depend only on (centre, neighbour), so they are
// evaluated once per slot, not once per angle.
template <typename T>
__device__ __forceinline__ void sw_leg(T r, const SwLeg<T> &l, T &E, T &D) {
    E = T(0);
    D = T(0);
    const T x = r / l.sig;
    if (!(x < l.a)) return;
    const T d = x - l.a;
    E = clamped_exp<T>(l.gam / d);
    if (E != T(0)) D = -l.gam / (l.sig * d * d);
}

// x^-4 as accurate as pow(): in float64 for a float32 evaluation (once per
// leg), with the square's rounding carried along in float64.
__device__ __forceinline__ float sw_inv4(float x) {
    const double x2 = (double)x * (double)x;
    return (float)(1.0 / (x2 * x2));
}
__device__ __forceinline__ double sw_inv4(double x) {
    const double x2 = x * x, e = fma(x, x, -x2);
    return 1.0 / fma(x2, x2, 2.0 * x2 * e);
}

// Two-body energy and its r-derivative (engine/stillinger_weber.py:23-52).
template <typename T>
__device__ __forceinline__ void sw_two(T r, const SwPair<T> &t, T &V2, T &dV2) {
    V2 = T(0);
    dV2 = T(0);
    const T x = r / t.sig;
    if (t.valid == T(0) || !(x < t.a)) return;
    const T tt = T(1) / (x - t.a), ex = clamped_exp<T>(tt);
    T xp, xq;
    if (t.p == T(4)) xp = sw_inv4(x);  // the published silicon exponents need no pow
    else xp = RT<T>::pw(x, -t.p);
    xq = t.q == T(0) ? T(1) : RT<T>::pw(x, -t.q);
    const T w = t.eps * t.A * ex, u = t.B * xp - xq;
    V2 = w * u;
    dV2 = w * ((-t.p * t.B * xp + t.q * xq) / x - u * (tt * tt)) / t.sig;
}

// One centre's legs in shared memory, compacted in slot order: displacement
// and unit vector, length and leg factors.  Groups of a warp lie 32 bytes
// apart modulo the banks' 128.
template <typename T, int MAXN>
struct SwRow {
    T ux[MAXN], uy[MAXN], uz[MAXN], E[MAXN], D[MAXN], x[MAXN], y[MAXN], z[MAXN], r[MAXN];
    int sp[MAXN], rev[MAXN];
    int meta[MAXN];  // slot in the row | (i < j) << 8
    char pad[32];
};

// SYM: one species, so every angle has one coefficient and cos0.  Otherwise
// both orders of an angle, each with its own record (lambda/2 of (i, j, k)
// and of (i, k, j)).
//
// For leg s and partner k with P = E_s E_k, cos = u_s . u_k, dc_o = cos -
// cos0_o over the orders o:
//   energy booked on leg s:  c_1 P dc_1^2        (order (i, s, k))
//   dh/dr_s = P [D_s A u_s + (B / r_s)(u_k - cos u_s)],
//   A = sum_o c_o dc_o^2,  B = 2 sum_o c_o dc_o,
// so each ordered triple's energy is booked once and each leg collects the
// whole gradient of every angle on it; the sums over k are a vector
// (P B u_k) and two scalars (P A and P B cos).  With half of the leg's pair
// term that is D_s = dU_i/dr_s, kept on i and left negated in the neighbour's
// own slot.
//
// Bound by instruction issue and latency: 16 legs and 240 ordered angles a
// centre in 64,000-atom Ge-Sn.  The record tables are staged in T (an angle's
// records were six float64 loads and conversions), legs beyond their own
// pair's reach are dropped before the angle loop, and the sums over k are in
// unit vectors: 136 -> 92 us there with the gather, mixed.  (The legs of a
// block as one list, as the Tersoff kernel has them, took 104: its 23 KB of
// staged legs leave fewer warps resident than the fuller lanes gain.)
template <typename T, int MAXN, bool SYM, bool STAGED, int LPA>
__global__ void __launch_bounds__(SwGeom<MAXN, LPA>::BLOCK, SwGeom<MAXN, LPA>::min_blocks(sizeof(T)))
    sw_center(SysView S, const int *__restrict__ row_off, const int *__restrict__ nbr, const int *__restrict__ rev,
              SwDev P, double *__restrict__ slot_G, double *__restrict__ f_local, double *__restrict__ per_atom,
              unsigned *__restrict__ live_mask, int n_slots, ClearWords clr, SiteOut so) {
    constexpr int GPB = SwGeom<MAXN, LPA>::GPB;
    constexpr int NB = LPA < 8 ? LPA : 8, KS = LPA / NB;
    __shared__ SwRow<T, MAXN> rows[GPB];
    __shared__ SwTab<T, STAGED> B;
    const int g = threadIdx.x / LPA, i = g < GPB ? blockIdx.x * GPB + g : S.n_atoms;
    RowHead head;
    head.load(S, row_off, i);
    clr.run();
    B.load(P);
    const int sub = threadIdx.x & (LPA - 1), gl = threadIdx.x & 31 & ~(LPA - 1);
    const unsigned gmask = ((1u << LPA) - 1u) << gl;
    const int lt = sub & (NB - 1), ks = sub / NB;
    SwRow<T, MAXN> &R = rows[g < GPB ? g : 0];
    const int ns = P.ns;
    double fx = 0, fy = 0, fz = 0, e = 0;
    double v[9] = {0, 0, 0, 0, 0, 0, 0, 0, 0};
    head.slots<LPA>(nbr, rev, n_slots, ns, MAXN);
    const RowStage st = stage_row<LPA>(
        S, head, nbr, rev, n_slots, ns, P.rc, i, live_mask, so.vec,
        [&](int a, int b) { return B.reach2(P, a, b); },
        [&](int q, int s, int j, int sj, int rs, double dx, double dy, double dz, double r2) {
            R.x[q] = (T)dx;
            R.y[q] = (T)dy;
            R.z[q] = (T)dz;
            // unit vector and length rounded once, from float64
            double r, ir;
            leg_dist<T>(r2, r, ir);
            R.r[q] = (T)r;
            R.ux[q] = (T)(dx * ir);
            R.uy[q] = (T)(dy * ir);
            R.uz[q] = (T)(dz * ir);
            R.sp[q] = sj;
            R.rev[q] = rs;
            R.meta[q] = s | (i < j ? 1 << 8 : 0);
        });
    const int nl = st.nl, beg = st.beg, si = st.si;
    __syncwarp(gmask);
    for (int q = sub; q < nl; q += LPA) {
        const int ij = si * ns + R.sp[q];
        T E, D;
        sw_leg<T>(R.r[q], B.leg(P, ij), E, D);
        R.E[q] = E;
        R.D[q] = D;
    }
    __syncwarp(gmask);
    SwTri<T> own = {T(0), T(0)};
    if (SYM) own = B.tri(P, 0);
    for (int t0 = 0; t0 < nl; t0 += NB) {
        const int t = t0 + lt;
        const bool act = t < nl;
        // sums over k: P B u_k, P A, P B cos, and the energy
        T wx = T(0), wy = T(0), wz = T(0), sA = T(0), sB = T(0);
        double e3 = 0.0;
        T uxs = T(0), uys = T(0), uzs = T(0);
        if (act) {
            uxs = R.ux[t];
            uys = R.uy[t];
            uzs = R.uz[t];
            const T Es = R.E[t];
            const int rowj = (si * ns + R.sp[t]) * ns;
            if (Es != T(0)) {
                for (int k = ks; k < nl; k += KS) {
                    if (k == t) continue;
                    const T uxk = R.ux[k], uyk = R.uy[k], uzk = R.uz[k];
                    const T cs = uxs * uxk + uys * uyk + uzs * uzk, Pp = Es * R.E[k];
                    T A, Bc, eh;
                    if (SYM) {
                        const T dc = cs - own.cos0;
                        eh = own.c * dc * dc;
                        A = T(2) * eh;
                        Bc = T(4) * own.c * dc;
                    } else {
                        const int sk = R.sp[k], ra = rowj + sk, rb = (si * ns + sk) * ns + R.sp[t];
                        const SwTri<T> q1 = B.tri(P, ra);
                        const SwTri<T> q2 = B.tri(P, rb);
                        const T dc1 = cs - q1.cos0, dc2 = cs - q2.cos0;
                        const T b1 = q1.c * dc1, b2 = q2.c * dc2;
                        eh = b1 * dc1;
                        A = eh + b2 * dc2;
                        Bc = T(2) * (b1 + b2);
                    }
                    const T w = Pp * Bc;
                    wx += w * uxk;
                    wy += w * uyk;
                    wz += w * uzk;
                    sA += Pp * A;
                    sB += w * cs;
                    e3 += (double)(Pp * eh);
                }
            }
        }
#pragma unroll
        for (int o = NB; o < LPA; o <<= 1) {
            wx += __shfl_xor_sync(gmask, wx, o, LPA);
            wy += __shfl_xor_sync(gmask, wy, o, LPA);
            wz += __shfl_xor_sync(gmask, wz, o, LPA);
            sA += __shfl_xor_sync(gmask, sA, o, LPA);
            sB += __shfl_xor_sync(gmask, sB, o, LPA);
        }
        e += e3;
        if (act && ks == 0) {
            const T r = R.r[t], ir = T(1) / r;
            const int mt = R.meta[t], sj = R.sp[t];
            // the pair record of the lower-indexed atom's species order
            const int pr = mt & 256 ? si * ns + sj : sj * ns + si;
            T V2, dV2;
            sw_two<T>(r, B.pair(P, pr), V2, dV2);
            e += 0.5 * (double)V2;
            const double hx = 0.5 * (double)(dV2 * ir);
            const T su = R.D[t] * sA - sB * ir;
            const double dx = (double)R.x[t], dy = (double)R.y[t], dz = (double)R.z[t];
            const double Dx = hx * dx + (double)(su * uxs + wx * ir), Dy = hx * dy + (double)(su * uys + wy * ir),
                         Dz = hx * dz + (double)(su * uzs + wz * ir);
            fx += Dx;
            fy += Dy;
            fz += Dz;
            v[0] -= Dx * dx;
            v[1] -= Dx * dy;
            v[2] -= Dx * dz;
            v[3] -= Dy * dx;
            v[4] -= Dy * dy;
            v[5] -= Dy * dz;
            v[6] -= Dz * dx;
            v[7] -= Dz * dy;
            v[8] -= Dz * dz;
            if (so.dudv) {  // U_i = 1/2 sum V2 + angles at i (engine/site_terms.py:179-300)
                const size_t os = 3 * (size_t)(beg + (mt & 255));
                so.dudv[os] = Dx;
                so.dudv[os + 1] = Dy;
                so.dudv[os + 2] = Dz;
            }
            // the force on neighbour j goes to j's own slot (j -> i)
            const size_t o = 3 * (size_t)R.rev[t];
            slot_G[o] = -Dx;
            slot_G[o + 1] = -Dy;
            slot_G[o + 2] = -Dz;
        }
    }
    __syncwarp();
    put_atom<LPA>(per_atom, f_local, so.e, i < S.n_atoms ? i : -1, e, v, fx, fy, fz, st.nok, st.bad);
}

// Everything one launch needs besides the shape.
struct SwArgs {
    SysView S;
    const mbf_nlist *nl;
    SwDev P;
    double *slot_G, *f_local, *per_atom;
    unsigned *live_mask;
    ClearWords clr;
    SiteOut so;
};

template <typename T, int MAXN, bool SYM, bool STAGED, int LPA>
static int sw_launch(const SwArgs &A, cudaStream_t st) {
    constexpr int GPB = SwGeom<MAXN, LPA>::GPB, BLOCK = SwGeom<MAXN, LPA>::BLOCK;
    const int blocks = (A.S.n_atoms + GPB - 1) / GPB;
    PROF_BEGIN("sw_center", st);
    sw_center<T, MAXN, SYM, STAGED, LPA><<<blocks, BLOCK, 0, st>>>(
        A.S, A.nl->row_off, A.nl->nbr, A.nl->rev, A.P, A.slot_G, A.f_local, A.per_atom, A.live_mask,
        (int)A.nl->n_slots, A.clr, A.so);
    PROF_END("sw_center", st);
    MBF_CHECK_LAUNCH();
    return MBF_OK;   // the eval's gather_live adds the slot forces
}

template <typename T, int MAXN, bool SYM, bool STAGED>
static int sw_lpa(int lpa, const SwArgs &A, cudaStream_t st) {
    switch (lpa) {
        case 4: return sw_launch<T, MAXN, SYM, STAGED, 4>(A, st);
        case 8: return sw_launch<T, MAXN, SYM, STAGED, 8>(A, st);
        case 16: return sw_launch<T, MAXN, SYM, STAGED, 16>(A, st);
        default: return MBF_ERR_ARGUMENT;
    }
}

template <typename T, bool SYM, bool STAGED>
static int sw_dispatch(int mr, int lpa, const SwArgs &A, cudaStream_t st) {
    if (mr <= 32) return sw_lpa<T, 32, SYM, STAGED>(lpa, A, st);
    if (mr <= 64) return sw_lpa<T, 64, SYM, STAGED>(lpa, A, st);
    return sw_lpa<T, 128, SYM, STAGED>(lpa, A, st);
}

// One species: every angle has one record; up to SW_SH: staged.
template <typename T>
static int sw_tables(int mr, int lpa, const SwArgs &A, cudaStream_t st) {
    if (A.P.ns == 1) return sw_dispatch<T, true, true>(mr, lpa, A, st);
    return A.P.ns <= SW_SH ? sw_dispatch<T, false, true>(mr, lpa, A, st) : sw_dispatch<T, false, false>(mr, lpa, A, st);
}

// The longest row sw_dispatch's choice for `mr` stages.
static int sw_row_limit(int mr) { return mr <= 32 ? 32 : (mr <= 64 ? 64 : 128); }

}  // namespace mbf

using namespace mbf;

static int sw_eval(const mbf_system *sys, const mbf_nlist *nl, const mbf_sw_tables *tab,
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
    SwArgs A;
    A.S = make_view(sys);
    A.nl = nl;
    A.P.ns = tab->ns;
    A.P.tb = tab->tb;
    A.P.leg = tab->leg;
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
    const int lpa = lanes_per_atom > 0 ? lanes_per_atom : 8, mr = nl->max_row;
    const int rc = precision == MBF_FP64 ? sw_tables<double>(mr, lpa, A, st) : sw_tables<float>(mr, lpa, A, st);
    if (rc != MBF_OK) return rc;
    return gather_live(sys->n_struct, sys->n_atoms, nl->row_off, (int)nl->n_slots, A.slot_G, A.live_mask,
                       sw_row_limit(mr), err, A.f_local, forces, A.per_atom, plan,
                       ws_at<double>(workspace, L.partial), energy, virial, sdone, st);
}

extern "C" int mbf_sw_eval(const mbf_system *sys, const mbf_nlist *nl, const mbf_sw_tables *tab,
                           const mbf_reduce_plan *plan, int precision, int lanes_per_atom, void *workspace,
                           size_t workspace_bytes, double *forces, double *energy, double *virial, void *stream) {
    SiteOut none = {nullptr, nullptr, nullptr};
    return sw_eval(sys, nl, tab, plan, precision, lanes_per_atom, workspace, workspace_bytes, forces, energy, virial,
                   none, stream);
}

extern "C" int mbf_sw_eval_sites(const mbf_system *sys, const mbf_nlist *nl, const mbf_sw_tables *tab,
                                 const mbf_reduce_plan *plan, int precision, int lanes_per_atom, void *workspace,
                                 size_t workspace_bytes, double *forces, double *energy, double *virial,
                                 double *site_e, double *site_dudv, double *site_vec, void *stream) {
    if (!site_e || !site_dudv || !site_vec) return MBF_ERR_ARGUMENT;
    if (nl && nl->n_slots > 0 &&
        cudaMemsetAsync(site_dudv, 0, sizeof(double) * 3 * (size_t)nl->n_slots, (cudaStream_t)stream) != cudaSuccess)
        return MBF_ERR_CUDA;
    SiteOut so = {site_e, site_dudv, site_vec};
    return sw_eval(sys, nl, tab, plan, precision, lanes_per_atom, workspace, workspace_bytes, forces, energy, virial,
                   so, stream);
}
