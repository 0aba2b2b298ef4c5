// Staging of one centre's row by a lane group, shared by the three-body
// kernels (Tersoff, Stillinger-Weber): the neighbours inside the pair's reach
// are compacted in slot order, and a live bit per slot tells the gather which
// slots will hold a force.
#pragma once

#include "mbf_util.cuh"

namespace mbf {

// What staging found.
struct RowStage {
    int beg;   // first slot of the row
    int nl;    // legs: neighbours within their pair's reach
    int nok;   // neighbours within the cutoff
    int si;    // the centre's species
    bool bad;  // this lane met an index outside its array (skipped)
};

// The loads a row's staging starts from, in two steps so a persistent block
// can issue them for its next row while it works on the current one: the
// row's bounds, species and position, then its first slots (ROW_U a lane; two
// or four cost registers and gave nothing).
constexpr int ROW_U = 1;
struct RowHead {
    int beg, n, si;
    bool bad;  // an index outside its array: the row is skipped
    double x, y, z;
    int j[ROW_U], rs[ROW_U];
    __device__ __forceinline__ void load(const SysView &S, const int *__restrict__ row_off, int i) {
        beg = n = si = 0;
        bad = false;
        x = y = z = 0.0;
        if (i < S.n_atoms) {
            beg = __ldg(row_off + i);
            n = __ldg(row_off + i + 1);
            si = __ldg(S.types + i);
            const double *p = S.pos + 3 * (size_t)i;
            x = __ldg(p);
            y = __ldg(p + 1);
            z = __ldg(p + 2);
        }
    }
    // After load: checks the bounds (a row of more than max_row slots is left
    // to the gather to report) and loads this lane's first slots.
    template <int LPA>
    __device__ __forceinline__ void slots(const int *__restrict__ nbr, const int *__restrict__ rev, int n_slots, int ns,
                                          int max_row) {
        n -= beg;
        if ((unsigned)beg > (unsigned)n_slots || (unsigned)n > (unsigned)(n_slots - beg) ||
            (unsigned)si >= (unsigned)ns) {
            bad = true;
            beg = n = si = 0;
        }
        if (n > max_row) n = 0;
        const int sub = threadIdx.x & (LPA - 1);
#pragma unroll
        for (int u = 0; u < ROW_U; ++u) {
            const int s = u * LPA + sub;
            j[u] = rs[u] = 0;
            if (s < n) {
                j[u] = __ldg(nbr + beg + s);
                rs[u] = __ldg(rev + beg + s);
            }
        }
    }
};

// LPA lanes stage the row of atom i (i >= n_atoms: an empty row).  All lanes
// of a group call it with the same i and take the same number of trips, so
// the group's ballots are complete.  reach2(si, sj): squared distance beyond
// which the pair takes part in no term, the same from both atoms, so both
// find the same live bit (the displacement is odd in the pair and r^2 the
// same double).  put(q, s, j, sj, rs, dx, dy, dz, r2) stores leg q: slot s of
// the row, neighbour j of species sj, reverse slot rs.  Every index read from
// memory is checked by one unsigned comparison before it is used as an
// address.
template <int LPA, class Reach, class Put>
__device__ __forceinline__ RowStage stage_row(const SysView &S, const RowHead &h, const int *__restrict__ nbr,
                                              const int *__restrict__ rev, int n_slots, int ns, double rc, int i,
                                              unsigned *__restrict__ live_mask, double *__restrict__ vec, Reach reach2,
                                              Put put) {
    constexpr int U = ROW_U;
    const int sub = threadIdx.x & (LPA - 1), gl = threadIdx.x & 31 & ~(LPA - 1);
    const unsigned gones = (1u << LPA) - 1u, gmask = gones << gl;
    RowStage o = {h.beg, 0, 0, h.si, h.bad};
    const int n = h.n;
    if (n == 0) {
        // a rejected row (bad bounds or species) has no live slot
        if (h.bad && sub < 4) live_mask[4 * (size_t)i + sub] = 0u;
        return o;
    }
    RowCell cell;
    cell.load(S, i);
    const double rc2 = rc * rc;
    unsigned word = 0;
    for (int c0 = 0; c0 < n; c0 += U * LPA) {
        int j[U], rs[U], sj[U];
        double px[U], py[U], pz[U];
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const int s = c0 + u * LPA + sub;
            j[u] = i;  // at distance 0: no leg
            rs[u] = 0;
            if (s < n) {
                j[u] = c0 == 0 ? h.j[u] : __ldg(nbr + o.beg + s);
                rs[u] = c0 == 0 ? h.rs[u] : __ldg(rev + o.beg + s);
            }
        }
#pragma unroll
        for (int u = 0; u < U; ++u) {
            if ((unsigned)j[u] >= (unsigned)S.n_atoms) {
                o.bad = true;
                j[u] = i;
            }
            const double *p = S.pos + 3 * (size_t)j[u];
            px[u] = __ldg(p);
            py[u] = __ldg(p + 1);
            pz[u] = __ldg(p + 2);
            sj[u] = __ldg(S.types + j[u]);
        }
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const int s0 = c0 + u * LPA, s = s0 + sub;
            if (s0 >= n) break;  // the same over the group
            double dx, dy, dz;
            cell.mic(px[u] - h.x, py[u] - h.y, pz[u] - h.z, dx, dy, dz);
            const double r2 = dx * dx + dy * dy + dz * dz;
            bool ok = s < n && r2 < rc2 && r2 > 1e-24;
            if (s < n && ((unsigned)rs[u] >= (unsigned)n_slots || (unsigned)sj[u] >= (unsigned)ns)) {
                o.bad = true;
                ok = false;
            }
            const bool lv = ok && r2 <= reach2(o.si, sj[u]);
            if (vec && s < n) {
                const size_t os = 3 * (size_t)(o.beg + s);
                vec[os] = dx;
                vec[os + 1] = dy;
                vec[os + 2] = dz;
            }
            const unsigned b = (__ballot_sync(gmask, lv) >> gl) & gones;
            o.nok += __popc((__ballot_sync(gmask, ok) >> gl) & gones);
            if (lv) put(o.nl + __popc(b & ((1u << sub) - 1u)), s, j[u], sj[u], rs[u], dx, dy, dz, r2);
            o.nl += __popc(b);
            word |= b << (s0 & 31);
            if (((s0 + LPA) & 31) == 0 || s0 + LPA >= n) {
                if (sub == 0) live_mask[4 * (size_t)i + (s0 >> 5)] = word;
                word = 0;
            }
        }
    }
    return o;
}

// The legs of a block's rows as one list, so that the passes over legs fill
// every lane whatever each centre's leg count is (a lane group per centre
// left 14 of 32 lanes idle where centres have 13 to 19 legs).  map holds
// row * MAXN + leg, rows in order.
template <int GPB, int MAXN>
struct BlockLegs {
    int cnt[GPB];
    unsigned short map[GPB * MAXN];
};

// Fills F from every group's nl (group g, lane sub of LPA; g >= GPB: none);
// returns the number of legs.  Two block barriers, the last after the fill.
template <int GPB, int MAXN, int LPA>
__device__ __forceinline__ int flatten_legs(BlockLegs<GPB, MAXN> &F, int g, int sub, int nl) {
    if (sub == 0 && g < GPB) F.cnt[g] = nl;
    __syncthreads();
    int off = 0, total = 0;
#pragma unroll
    for (int q = 0; q < GPB; ++q) {
        const int c = F.cnt[q];
        off += q < g ? c : 0;
        total += c;
    }
    if (g < GPB)
        for (int q = sub; q < nl; q += LPA) F.map[off + q] = (unsigned short)(g * MAXN + q);
    __syncthreads();
    return total;
}

// Sum over the KS lanes that share a leg.
template <int KS, typename T>
__device__ __forceinline__ T share_sum(unsigned mask, T v) {
#pragma unroll
    for (int o = 1; o < KS; o <<= 1) v += __shfl_xor_sync(mask, v, o, KS);
    return v;
}

// The sums of an atom's group into its record and force: e, the virial v and
// the force f are each lane's part, nok and bad the row's.  Fourteen values
// over LPA lanes by halving: at each step a lane keeps one half of its values
// and sends the other, so LPA = 8 takes 14 exchanges instead of 3 x 13 and
// the results end spread over the lanes, which store them side by side (two
// store instructions instead of fourteen by one lane).  The order is fixed.
// A pair count of -1 stands for a row with a bad index, which the gather
// turns into MBF_DEV_BAD_INDEX.  All 32 lanes call it; i < 0: no atom.
template <int LPA>
__device__ __forceinline__ void put_atom(double *__restrict__ per_atom, double *__restrict__ f_local,
                                         double *__restrict__ site_e, int i, double e, const double (&v)[9],
                                         double fx, double fy, double fz, int nok, bool bad) {
    const int sub = threadIdx.x & (LPA - 1), gl = threadIdx.x & 31 & ~(LPA - 1);
    const bool any = ((__ballot_sync(MBF_FULL, bad) >> gl) & ((1u << LPA) - 1u)) != 0;
    double w[16] = {e,    v[0], v[1], v[2], v[3], v[4], v[5], v[6], v[7], v[8], sub == 0 ? (any ? -1.0 : (double)nok) : 0.0,
                    fx,   fy,   fz,   0.0,  0.0};
    int first = 0;
#pragma unroll
    for (int o = LPA / 2, half = 8; o > 0; o >>= 1, half >>= 1) {
        const bool up = (sub & o) != 0;
#pragma unroll
        for (int k = 0; k < half; ++k) {
            const double send = up ? w[k] : w[k + half];
            const double keep = up ? w[k + half] : w[k];
            w[k] = keep + __shfl_xor_sync(MBF_FULL, send, o, LPA);
        }
        first += up ? half : 0;
    }
    if (i < 0) return;
#pragma unroll
    for (int k = 0; k < 16 / LPA; ++k) {
        const int q = first + k;
        if (q < ATOM_ACC) per_atom[(size_t)i * ATOM_ACC + q] = w[k];
        else if (q < ATOM_ACC + 3) f_local[3 * (size_t)i + q - ATOM_ACC] = w[k];
        if (q == 0 && site_e) site_e[i] = w[k];
    }
}

// The sums over a centre's legs (row R: displacement x, y, z, gradient gx, gy,
// gz and energy e per leg) into its record: f = sum D, virial -D (x) d.
template <int LPA, class Row>
__device__ __forceinline__ void sum_legs(const Row &R, const RowStage &st, int i, double *__restrict__ per_atom,
                                         double *__restrict__ f_local, double *__restrict__ site_e) {
    const int sub = threadIdx.x & (LPA - 1);
    double fx = 0, fy = 0, fz = 0, e = 0;
    double v[9] = {0, 0, 0, 0, 0, 0, 0, 0, 0};
    for (int q = sub; q < st.nl; q += LPA) {
        const double dx = (double)R.x[q], dy = (double)R.y[q], dz = (double)R.z[q];
        const double Dx = R.gx[q], Dy = R.gy[q], Dz = R.gz[q];
        e += R.e[q];
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
    }
    __syncwarp();
    put_atom<LPA>(per_atom, f_local, site_e, i, e, v, fx, fy, fz, st.nok, st.bad);
}

}  // namespace mbf
