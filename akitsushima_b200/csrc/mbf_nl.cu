// Cell-list neighbour list: binning by integer counting sort, two-way CSR
// by count -> scan -> fill, rows sorted ascending, reverse-slot index.
//
// Replaces engine/neighborlist.py:935-1024 (_build_cell_linked), :312-373
// (_cell_linked_pairs_numpy), :1166-1181 (_canonical_pair_order) and the
// two-way CSR of engine/tersoff.py:1297-1307.  The pair test reproduces the
// reference's rounding exactly (mic_exact), so the pair set is bit-exact.
#include <type_traits>

#include "mbf_util.cuh"

namespace mbf {

constexpr int NL_WARPS = 4;        // warps per block in the search kernels
constexpr int NL_MAXROW = 1024;    // longest row the sort stages in shared memory

struct NlLayout {
    size_t err, atom_cell, cell_count, cell_start, cursor, cell_atoms, row_cnt, maxrow, scan, total;
};

static NlLayout nl_layout(int n_atoms, int n_cells) {
    NlLayout L;
    size_t o = 0;
    L.err = o;
    o = align256(o + 64);
    L.atom_cell = o;
    o = align256(o + sizeof(int) * (size_t)n_atoms);
    L.cell_count = o;
    o = align256(o + sizeof(int) * (size_t)n_cells);
    L.cell_start = o;
    o = align256(o + sizeof(int) * ((size_t)n_cells + 1));
    L.cursor = o;
    o = align256(o + sizeof(int) * (size_t)n_cells);
    L.cell_atoms = o;
    o = align256(o + sizeof(int) * (size_t)n_atoms);
    L.row_cnt = o;
    o = align256(o + sizeof(int) * (size_t)n_atoms);
    L.maxrow = o;
    o = align256(o + 64);
    L.scan = o;
    int nmax = n_atoms > n_cells ? n_atoms : n_cells;
    o = align256(o + sizeof(int) * scan_workspace_ints(nmax + 1));
    L.total = o;
    return L;
}

// Behind the layout, where the workspace has room: the block search's local
// coordinates (a float4 per atom), then the staging rows (n_atoms x
// max_row_limit ints).
static size_t nl_local_bytes(int n_atoms) { return align256(sizeof(float4) * (size_t)n_atoms); }

static bool nl_local_ok(const void *workspace) { return ((size_t)workspace & (sizeof(float4) - 1)) == 0; }

static size_t nl_staged_bytes(const NlLayout &L, int n_atoms, int max_row_limit) {
    return L.total + nl_local_bytes(n_atoms) + align256(sizeof(int) * (size_t)n_atoms * (size_t)max_row_limit);
}

// Bin every atom: fractional coordinate wrapped to [0, 1), sub-cell index
// floor(frac * nc) clipped to [0, nc - 1] (engine/neighborlist.py:982-989).
__global__ void nl_assign(SysView S, const int *__restrict__ grids, int *__restrict__ atom_cell,
                          int *__restrict__ cell_count) {
    int a = blockIdx.x * blockDim.x + threadIdx.x;
    if (a >= S.n_atoms) return;
    int s = S.n_struct > 1 ? S.atom_struct[a] : 0;
    const int *g = grids + 8 * s;
    const double *inv = S.cells + 18 * (size_t)s + 9;
    double x = S.pos[3 * (size_t)a], y = S.pos[3 * (size_t)a + 1], z = S.pos[3 * (size_t)a + 2];
    int ci[3];
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        double f = x * inv[k] + y * inv[3 + k] + z * inv[6 + k];
        f = f - floor(f);
        int c = (int)floor(f * (double)g[k]);
        c = c < 0 ? 0 : (c > g[k] - 1 ? g[k] - 1 : c);
        ci[k] = c;
    }
    int cell = g[3] + (ci[0] * g[1] + ci[1]) * g[2] + ci[2];
    atom_cell[a] = cell;
    atomicAdd(cell_count + cell, 1);
}

__global__ void nl_fill_cells(int n_atoms, const int *__restrict__ atom_cell, int *__restrict__ cursor,
                              int *__restrict__ cell_atoms) {
    int a = blockIdx.x * blockDim.x + threadIdx.x;
    if (a >= n_atoms) return;
    int p = atomicAdd(cursor + atom_cell[a], 1);
    cell_atoms[p] = a;
}

// Stencil of atom a's cell: up to 27 neighbour cells (per-axis offsets
// {0} for nc = 1, {0, 1} for nc = 2, {-1, 0, 1} otherwise -- the reference's
// _axis_offsets, engine/neighborlist.py:270-299), visited in (da, db, dc)
// order.  Lane k < K describes cell k; returns the warp-wide candidate count.
struct Stencil {
    int start[32];
    int pre[33];
};

__device__ int build_stencil_of_cell(const int *__restrict__ grids, const int *__restrict__ cell_start,
                                     int s, int cell_id, Stencil &st) {
    int lane = threadIdx.x & 31;
    const int *g = grids + 8 * s;
    int nc0 = g[0], nc1 = g[1], nc2 = g[2], first = g[3];
    int w0 = g[4], w1 = g[5], w2 = g[6];
    int local = cell_id - first;
    int c2 = local % nc2, c1 = (local / nc2) % nc1, c0 = local / (nc1 * nc2);
    int K = w0 * w1 * w2;
    int len = 0, start = 0;
    if (lane < K) {
        int i0 = lane / (w1 * w2), i1 = (lane / w2) % w1, i2 = lane % w2;
        int o0 = w0 == 3 ? i0 - 1 : i0, o1 = w1 == 3 ? i1 - 1 : i1, o2 = w2 == 3 ? i2 - 1 : i2;
        int j0 = (c0 + o0 + nc0) % nc0, j1 = (c1 + o1 + nc1) % nc1, j2 = (c2 + o2 + nc2) % nc2;
        int cell = first + (j0 * nc1 + j1) * nc2 + j2;
        start = cell_start[cell];
        len = cell_start[cell + 1] - start;
    }
    int inc = len;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        int t = __shfl_up_sync(MBF_FULL, inc, o);
        if (lane >= o) inc += t;
    }
    st.start[lane] = start;
    st.pre[lane] = inc - len;
    int total = __shfl_sync(MBF_FULL, inc, 31);
    if (lane == 0) st.pre[32] = total;
    __syncwarp();
    return total;
}

// Candidate t of the stencil -> atom index (binary search over the prefix).
__device__ __forceinline__ int stencil_atom(const Stencil &st, const int *__restrict__ cell_atoms, int t) {
    int lo = 0, hi = 31;
    while (lo < hi) {  // largest k with pre[k] <= t
        int mid = (lo + hi + 1) >> 1;
        if (st.pre[mid] <= t) lo = mid; else hi = mid - 1;
    }
    // skip empty cells that share the same prefix value
    return cell_atoms[st.start[lo] + (t - st.pre[lo])];
}

// ---- warp per cell -----------------------------------------------------------
// The atoms of one cell share their stencil: a warp builds it once, each lane
// loads one candidate's position per round, and the cell's atoms (32 at a
// time, one per lane) are broadcast by shuffles and tested against every
// lane's candidate.  A pair (a, b != a) is listed iff r2 < r_list^2 and
// r2 > 1e-20, r2 from mic_exact of r_b - r_a: the reference's test in its
// own operation order (engine/neighborlist.py:350-363).
__device__ __forceinline__ bool pair_hit(const double *__restrict__ cell, double xa, double ya, double za,
                                         double xb, double yb, double zb, double rl2) {
    double dx, dy, dz;
    mic_exact(cell, xb - xa, yb - ya, zb - za, dx, dy, dz);
    double r2 = r2_exact(dx, dy, dz);
    return r2 < rl2 && r2 > 1e-20;
}

// A cell whose lattice and inverse have exact zeros off the diagonal.
__device__ __forceinline__ bool cell_is_diagonal(const double *__restrict__ c) {
    bool z = true;
#pragma unroll
    for (int m = 0; m < 2; ++m) {
        const double *q = c + 9 * m;
        z = z && q[1] == 0.0 && q[2] == 0.0 && q[3] == 0.0 && q[5] == 0.0 && q[6] == 0.0 && q[7] == 0.0;
    }
    return z;
}

// pair_hit for a diagonal cell (d = inverse diagonal, l = lattice
// diagonal).  Each dropped term of mic_exact's dot products is a product
// with an exact zero, i.e. +-0, and x + (+-0) == x for every x != 0, so
// every component equals mic_exact's up to the sign of a zero, and r2 --
// a sum of squares -- is the same double bit for bit.
__device__ __forceinline__ bool pair_hit_diag(double d0, double d1, double d2, double l0, double l1, double l2,
                                              double xa, double ya, double za, double xb, double yb, double zb,
                                              double rl2) {
    double sx = __dmul_rn(__dsub_rn(xb, xa), d0);
    double sy = __dmul_rn(__dsub_rn(yb, ya), d1);
    double sz = __dmul_rn(__dsub_rn(zb, za), d2);
    sx = __dsub_rn(sx, rint_shift(sx));
    sy = __dsub_rn(sy, rint_shift(sy));
    sz = __dsub_rn(sz, rint_shift(sz));
    double r2 = r2_exact(__dmul_rn(sx, l0), __dmul_rn(sy, l1), __dmul_rn(sz, l2));
    return r2 < rl2 && r2 > 1e-20;
}

// The rows of atoms [q_begin, q_end) of one cell by one warp, with the exact
// test on every candidate of the stencil.  MODE 0 counts each atom's
// neighbours (row_cnt); MODE 1 writes them into the CSR rows (row_off, nbr);
// MODE 2 counts and writes them at a fixed stride into a staging array
// (`nbr` = stage, row a at a * stride, at most stride entries kept), so one
// pass serves a list of known row bound.  Returns the longest row it counted
// (per lane).
template <int MODE>
__device__ __forceinline__ int cell_rows_exact(const SysView &S, const double *__restrict__ cell, const Stencil &st,
                                               int total, const int *__restrict__ cell_atoms, int cs, int q_begin,
                                               int q_end, double rl2, int *__restrict__ row_cnt,
                                               const int *__restrict__ row_off, int *__restrict__ nbr, int stride) {
    constexpr bool FILL = MODE != 0, COUNT = MODE != 1;
    const int lane = threadIdx.x & 31;
    const bool diag = cell_is_diagonal(cell);
    const double d0 = cell[9], d1 = cell[13], d2 = cell[17], l0 = cell[0], l1 = cell[4], l2 = cell[8];
    int longest = 0;
    for (int q0 = q_begin; q0 < q_end; q0 += 32) {
        int nq = min(32, q_end - q0);
        int a_l = lane < nq ? cell_atoms[cs + q0 + lane] : 0;
        double xa_l = S.pos[3 * (size_t)a_l], ya_l = S.pos[3 * (size_t)a_l + 1], za_l = S.pos[3 * (size_t)a_l + 2];
        int cnt = 0;       // lane q: neighbours of atom q found so far
        int beg_l = 0, len_l = 0;
        if (FILL && lane < nq) {
            beg_l = MODE == 1 ? row_off[a_l] : a_l * stride;
            len_l = MODE == 1 ? row_off[a_l + 1] - beg_l : stride;
        }
        for (int t0 = 0; t0 < total; t0 += 32) {
            int t = t0 + lane;
            int b = -1;
            double xb = 0, yb = 0, zb = 0;
            if (t < total) {
                b = stencil_atom(st, cell_atoms, t);
                xb = S.pos[3 * (size_t)b];
                yb = S.pos[3 * (size_t)b + 1];
                zb = S.pos[3 * (size_t)b + 2];
            }
            // the cell's atoms against this round's candidates, with
            // the test specialised once per cell (warp-uniform)
            auto rounds = [&](auto diag_tag) {
                constexpr bool DIAG = decltype(diag_tag)::value;
                for (int q = 0; q < nq; ++q) {
                    int a = __shfl_sync(MBF_FULL, a_l, q);
                    double xa = __shfl_sync(MBF_FULL, xa_l, q), ya = __shfl_sync(MBF_FULL, ya_l, q),
                           za = __shfl_sync(MBF_FULL, za_l, q);
                    bool hit = b >= 0 && b != a &&
                               (DIAG ? pair_hit_diag(d0, d1, d2, l0, l1, l2, xa, ya, za, xb, yb, zb, rl2)
                                     : pair_hit(cell, xa, ya, za, xb, yb, zb, rl2));
                    unsigned m = __ballot_sync(MBF_FULL, hit);
                    if (FILL) {
                        int w = __shfl_sync(MBF_FULL, cnt, q);
                        int beg = __shfl_sync(MBF_FULL, beg_l, q), len = __shfl_sync(MBF_FULL, len_l, q);
                        if (hit) {
                            int pos = w + __popc(m & ((1u << lane) - 1u));
                            if (pos < len) nbr[beg + pos] = b;
                        }
                    }
                    if (lane == q) cnt += __popc(m);
                }
            };
            if (diag)
                rounds(std::true_type{});
            else
                rounds(std::false_type{});
        }
        if (COUNT && lane < nq) {
            row_cnt[a_l] = cnt;
            longest = max(longest, cnt);
        }
    }
    return longest;
}

// A warp per cell: cells of few atoms, and those the block search left.
template <int MODE>
__global__ void nl_cells(SysView S, const int *__restrict__ grids, const int *__restrict__ cell_start,
                         const int *__restrict__ cell_atoms, int n_cells, double rl2, int *__restrict__ row_cnt,
                         int *__restrict__ max_row, const int *__restrict__ row_off, int *__restrict__ nbr,
                         int stride, const int *__restrict__ done) {
    __shared__ Stencil sst[NL_WARPS];
    int wid = threadIdx.x >> 5, lane = threadIdx.x & 31;
    Stencil &st = sst[wid];
    int longest = 0;
    for (int c = blockIdx.x * NL_WARPS + wid; c < n_cells; c += gridDim.x * NL_WARPS) {
        int cs = cell_start[c], na = cell_start[c + 1] - cs;
        if (na == 0 || (done && done[c])) continue;  // uniform over the warp
        int sidx = S.n_struct > 1 ? S.atom_struct[cell_atoms[cs]] : 0;
        int total = build_stencil_of_cell(grids, cell_start, sidx, c, st);
        longest = max(longest, cell_rows_exact<MODE>(S, S.cells + 18 * (size_t)sidx, st, total, cell_atoms, cs, 0, na,
                                                     rl2, row_cnt, row_off, nbr, stride));
    }
    if (MODE != 1) {
        longest = __reduce_max_sync(MBF_FULL, longest);
        if (lane == 0) atomicMax(max_row, longest);
    }
}

// A block per cell, for cells of many atoms: counts and stages as MODE 2.
// The stencil's candidates are put into ascending atom index once per cell, so
// every row comes out ascending: each sets its bit in a map of the index range
// that they span, and its rank is the number of bits below its own.  The range
// is taken around the end of the index (modulo n_atoms), so a stencil over the
// periodic boundary spans no more of a lattice-ordered structure than one
// inside it.
// They are tested in float32 against the cell's atoms, up to NL_NA atoms a
// warp at a time, in coordinates relative to the cell's middle (`local`, each
// atom relative to the middle of its own cell, plus the stencil offset).  A
// squared distance within `margin` of r_list^2 or of 0 is decided by the exact
// test, so the pair set is the same.  Coordinates are below
// M = 1.5 sum_k |L_k|_1 / nc_k and off by less than 2^-23 M, so the squared
// distance of a pair near r = r_list is off by less than
// 2 sqrt(3) r (2^-22 M + 2^-24 r) + 4 * 2^-24 r^2 < r (M + r) 2^-20; the
// margin is four times that.  From five cells on each axis two atoms of a
// stencil are at most 0.4 of the box apart, so the offset's image is the one
// the minimum image rounds to.  Other cells, cells of more than NL_CAP
// candidates or a range beyond NL_BITS, and cells near an atom more than 4096
// boxes away (where the wrap itself loses digits) are left to nl_cells
// (done = 0).
//
// Issue-bound, the rank and the tests about half each: 256,000 Cu-Ni atoms at
// 80 neighbours (21 atoms a cell, 27 x 21 candidates, 62 % of them kept) take
// 275 us and leave 60 for the rows' copy into the CSR; a warp per cell with
// the exact test on every candidate took 463 and left 198 for the rows'
// sorts.  Merging the 27 runs in shared memory instead of ranking by bits
// took 240 us alone.  Atoms a warp: 3 as 4 (279), 2 worse (the candidates are
// read once for all); 128 threads 316, 512 threads 315; at 5 blocks an SM the
// registers spill (320).
constexpr int NL_T = 256, NL_NW = NL_T / 32;
constexpr int NL_CAP = 1024;   // candidates a block ranks
constexpr int NL_BITS = 1 << 17;   // index range they may span: 32 x 32 groups of 128 bits
constexpr int NL_NA = 4;       // atoms a warp tests at a time

__device__ __forceinline__ bool grid_is_wide(const int *__restrict__ g) {
    return g[0] >= 5 && g[1] >= 5 && g[2] >= 5 && g[4] == 3 && g[5] == 3 && g[6] == 3;
}

// The rows of NA atoms (cand[own[0]], cand[own[NL_NW]], ...) by one warp, every
// candidate against each; returns the longest.
template <int NA>
__device__ __forceinline__ int test_rows(const SysView &S, const double *__restrict__ cell, const float4 *cand,
                                         const unsigned short *own, int total, float lo2, float hi2, double r_list,
                                         int *__restrict__ row_cnt, int *__restrict__ stage, int stride) {
    const int lane = threadIdx.x & 31;
    const unsigned below = (1u << lane) - 1u;
    const float tiny = 0.5f * (hi2 - lo2);
    float ax[NA], ay[NA], az[NA];
    int a[NA], cnt[NA];
    int *out[NA];
#pragma unroll
    for (int i = 0; i < NA; ++i) {
        const float4 v = cand[own[i * NL_NW]];
        ax[i] = v.x;
        ay[i] = v.y;
        az[i] = v.z;
        a[i] = __float_as_int(v.w);
        cnt[i] = 0;
        out[i] = stage + (size_t)a[i] * stride;
    }
    for (int t = lane; t < total + lane; t += 32) {  // the last round reads padding
        const float4 v = cand[t];
        const int b = __float_as_int(v.w);
        bool hit[NA], near[NA], any = false;
#pragma unroll
        for (int i = 0; i < NA; ++i) {
            const float dx = v.x - ax[i], dy = v.y - ay[i], dz = v.z - az[i];
            const float r2 = dx * dx + dy * dy + dz * dz;
            hit[i] = r2 < lo2 && r2 > tiny;
            near[i] = r2 < hi2 && !hit[i] && b != a[i];
            any = any || near[i];
        }
        if (any) {  // seldom
            const double *pb = S.pos + 3 * (size_t)b;
#pragma unroll
            for (int i = 0; i < NA; ++i)
                if (near[i]) {
                    const double *pa = S.pos + 3 * (size_t)a[i];
                    hit[i] = pair_hit(cell, pa[0], pa[1], pa[2], pb[0], pb[1], pb[2], r_list * r_list);
                }
        }
#pragma unroll
        for (int i = 0; i < NA; ++i) {
            const unsigned m = __ballot_sync(MBF_FULL, hit[i]);
            const int p = cnt[i] + __popc(m & below);
            if (hit[i] && p < stride) out[i][p] = b;
            cnt[i] += __popc(m);
        }
    }
    int longest = 0;
#pragma unroll
    for (int i = 0; i < NA; ++i) {
        if (lane == 0) row_cnt[a[i]] = cnt[i];
        longest = max(longest, cnt[i]);
    }
    return longest;
}

__global__ void __launch_bounds__(NL_T, 4) nl_search(SysView S, const int *__restrict__ grids,
                                                  const int *__restrict__ cell_start,
                                                  const float4 *__restrict__ local, int n_cells, double r_list,
                                                  int *__restrict__ row_cnt, int *__restrict__ max_row,
                                                  int *__restrict__ stage, int stride, int *__restrict__ done,
                                                  const int *__restrict__ searched) {
    if (*searched == 0) return;  // no cell to try
    __shared__ Stencil st;
    __shared__ float4 cand[NL_CAP];             // x, y, z, atom; ascending
    __shared__ uint4 bits[NL_BITS / 128];       // all zero between cells
    __shared__ ushort4 before[NL_BITS / 128];   // bits set before each word, in its chunk of 128 words
    __shared__ int chunk[32], ahead_w[NL_NW][32];  // bits set in a chunk, and before it (each warp's copy)
    __shared__ unsigned short own[NL_CAP];      // place in cand of the cell's atoms
    __shared__ float3 offset[27];               // of the stencil's cells
    __shared__ float bound[2];                  // lower and upper squared radius
    __shared__ float box[6];                    // of the cell's atoms
    __shared__ int base_sh, range_sh;
    const int tid = threadIdx.x, wid = tid >> 5, lane = tid & 31;
    const int N = S.n_atoms;
    unsigned *word = (unsigned *)bits;
    const unsigned short *word_before = (const unsigned short *)before;
    for (int k = tid; k < NL_BITS / 128; k += NL_T) bits[k] = make_uint4(0, 0, 0, 0);
    int longest = 0;
    for (int c = blockIdx.x; c < n_cells; c += gridDim.x) {
        const int cs = cell_start[c], na = cell_start[c + 1] - cs;
        if (na == 0 || !done[c]) continue;  // uniform over the block
        const int mid = __float_as_int(local[cs + na / 2].w);
        const int sidx = S.n_struct > 1 ? S.atom_struct[mid] : 0;
        const double *cell = S.cells + 18 * (size_t)sidx;
        const int *g = grids + 8 * sidx;
        __syncthreads();  // the previous cell's readers are done
        if (wid == 0) {
            build_stencil_of_cell(grids, cell_start, sidx, c, st);
            // the range of atom indices, counted from half an index below the
            // cell's middle atom; in a (sorted) cell the indices from there
            // to the end of the index come first
            int base = mid - N / 2;
            base += base < 0 ? N : 0;
            const int beg = st.start[lane], len = st.pre[lane + 1] - st.pre[lane];
            int lo = 0, hi = len;  // entries below base
            if (len && __float_as_int(local[beg].w) >= base) hi = 0;
            if (len && __float_as_int(local[beg + len - 1].w) < base) lo = len;
            while (lo < hi) {
                const int m = (lo + hi) >> 1;
                if (__float_as_int(local[beg + m].w) < base) lo = m + 1; else hi = m;
            }
            int low = N, high = 0;
            if (len) {
                low = __float_as_int(local[beg + (lo < len ? lo : 0)].w) - base;
                high = __float_as_int(local[beg + (lo > 0 ? lo : len) - 1].w) - base;
                low += low < 0 ? N : 0;
                high += high < 0 ? N : 0;
            }
            low = __reduce_min_sync(MBF_FULL, low);
            high = __reduce_max_sync(MBF_FULL, high);
            if (lane == 0) {
                base += low;
                base_sh = base - (base >= N ? N : 0);
                range_sh = high - low;
            }
        }
        if (wid == 1) {
            const double s = lane < 9 ? cell[lane] / (double)g[lane / 3] : 0.0;
            double M = 1.5 * fabs(s);
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) M += __shfl_xor_sync(MBF_FULL, M, o);
            const float margin = (float)(r_list * (M + r_list) * 0x1p-18);
            if (lane < 2) bound[lane] = (float)(r_list * r_list) + (lane ? margin : -margin);
            const float sf = (float)s;
            float o[3];
#pragma unroll
            for (int k = 0; k < 3; ++k)
                o[k] = (float)(lane / 9 - 1) * __shfl_sync(MBF_FULL, sf, k) +
                       (float)((lane / 3) % 3 - 1) * __shfl_sync(MBF_FULL, sf, 3 + k) +
                       (float)(lane % 3 - 1) * __shfl_sync(MBF_FULL, sf, 6 + k);
            if (lane < 27) offset[lane] = make_float3(o[0], o[1], o[2]);
        }
        if (wid == 2) {
            float lo[3] = {1e30f, 1e30f, 1e30f}, hi[3] = {-1e30f, -1e30f, -1e30f};
            for (int k = lane; k < na; k += 32) {
                const float4 q = local[cs + k];
                lo[0] = fminf(lo[0], q.x), hi[0] = fmaxf(hi[0], q.x);
                lo[1] = fminf(lo[1], q.y), hi[1] = fmaxf(hi[1], q.y);
                lo[2] = fminf(lo[2], q.z), hi[2] = fmaxf(hi[2], q.z);
            }
#pragma unroll
            for (int o = 16; o > 0; o >>= 1)
#pragma unroll
                for (int k = 0; k < 3; ++k) {
                    lo[k] = fminf(lo[k], __shfl_xor_sync(MBF_FULL, lo[k], o));
                    hi[k] = fmaxf(hi[k], __shfl_xor_sync(MBF_FULL, hi[k], o));
                }
            if (lane == 0)
#pragma unroll
                for (int k = 0; k < 3; ++k) {
                    box[k] = lo[k];
                    box[3 + k] = hi[k];
                }
        }
        __syncthreads();
        const int base = base_sh, range = range_sh;
        int total = 0;
        bool wide = range < NL_BITS && bound[0] > 0.0f && bound[1] < 1e30f;
        if (wide) {
            // candidates within r_list of the box of the cell's atoms
            bool far = false;
            const float reach = bound[1];
            for (int run = wid; run < 27; run += NL_NW) {
                const int beg = st.start[run], len = st.pre[run + 1] - st.pre[run];
                const float3 o = offset[run];
                for (int k = lane; k < len; k += 32) {
                    const float4 q = local[beg + k];
                    const float x0 = q.x + o.x, x1 = q.y + o.y, x2 = q.z + o.z;
                    const float e0 = fmaxf(fmaxf(box[0] - x0, x0 - box[3]), 0.0f);
                    const float e1 = fmaxf(fmaxf(box[1] - x1, x1 - box[4]), 0.0f);
                    const float e2 = fmaxf(fmaxf(box[2] - x2, x2 - box[5]), 0.0f);
                    far = far || q.x != q.x;
                    if (e0 * e0 + e1 * e1 + e2 * e2 >= reach) continue;
                    const int v = __float_as_int(q.w), x = v - base + (v < base ? N : 0);
                    atomicOr(word + (x >> 5), 1u << (x & 31));
                }
            }
            wide = !__syncthreads_or(far);
            for (int k = wid; k < 32; k += NL_NW) {
                int sum = 0;
                if (k << 12 <= range) {
                    const uint4 w = bits[k * 32 + lane];
                    const int n0 = __popc(w.x), n1 = n0 + __popc(w.y), n2 = n1 + __popc(w.z), n = n2 + __popc(w.w);
                    sum = n;
#pragma unroll
                    for (int o = 1; o < 32; o <<= 1) {
                        const int t = __shfl_up_sync(MBF_FULL, sum, o);
                        if (lane >= o) sum += t;
                    }
                    const int b = sum - n;
                    before[k * 32 + lane] = make_ushort4(b, b + n0, b + n1, b + n2);
                }
                if (lane == 31) chunk[k] = sum;
            }
            __syncthreads();
            int ahead = chunk[lane];  // lane k: bits set before chunk k
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const int t = __shfl_up_sync(MBF_FULL, ahead, o);
                if (lane >= o) ahead += t;
            }
            ahead_w[wid][lane] = ahead - chunk[lane];
            __syncwarp();  // rank() below reads the other lanes' entries
            total = __shfl_sync(MBF_FULL, ahead, 31);
            wide = wide && total <= NL_CAP;
        }
        if (!wide) {  // uniform over the block
            if (tid == 0) done[c] = 0;
            if (range < NL_BITS)
                for (int k = tid; k <= range >> 7; k += NL_T) bits[k] = make_uint4(0, 0, 0, 0);
            continue;
        }
        {
            // bits set below place x of the range
            auto rank = [&](int x) {
                return ahead_w[wid][x >> 12] + word_before[x >> 5] + __popc(word[x >> 5] & ((1u << (x & 31)) - 1u));
            };
            // the atoms below the base, at the range's far end, come first
            const int front = N - base <= range ? total - rank(N - base) : 0;
            for (int run = wid; run < 27; run += NL_NW) {
                const int beg = st.start[run], len = st.pre[run + 1] - st.pre[run];
                const float3 o = offset[run];
                for (int k = lane; k < len; k += 32) {
                    const float4 q = local[beg + k];
                    const int v = __float_as_int(q.w), x = v - base + (v < base ? N : 0);
                    if (!(word[x >> 5] >> (x & 31) & 1u)) continue;
                    const int at = rank(x) + (v < base ? front - total : front);
                    cand[at] = make_float4(q.x + o.x, q.y + o.y, q.z + o.z, q.w);
                    if (run == 13) own[k] = (unsigned short)at;
                }
            }
            if (tid < (-total & 31)) cand[total + tid] = make_float4(1e30f, 1e30f, 1e30f, 0.0f);
            __syncthreads();
            for (int k = tid; k < total; k += NL_T) {
                const int v = __float_as_int(cand[k].w), x = v - base + (v < base ? N : 0);
                word[x >> 5] = 0;
            }
        }
        const float lo2 = bound[0], hi2 = bound[1];
        for (int q = wid; q < na; q += NL_NW * NL_NA) {
            const int n = min(NL_NA, (na - q + NL_NW - 1) / NL_NW);
            int most = 0;
            if (n == 4)
                most = test_rows<4>(S, cell, cand, own + q, total, lo2, hi2, r_list, row_cnt, stage, stride);
            else if (n == 3)
                most = test_rows<3>(S, cell, cand, own + q, total, lo2, hi2, r_list, row_cnt, stage, stride);
            else if (n == 2)
                most = test_rows<2>(S, cell, cand, own + q, total, lo2, hi2, r_list, row_cnt, stage, stride);
            else
                most = test_rows<1>(S, cell, cand, own + q, total, lo2, hi2, r_list, row_cnt, stage, stride);
            longest = max(longest, most);
        }
    }
    if (lane == 0) atomicMax(max_row, longest);
}

// The search: with room for the staging rows and the local coordinates a block
// per cell from NL_BLOCK_ATOMS atoms a cell; the cells that leaves, and all
// others, a warp each.  A block pays about 12 ns a cell for its ranking, a
// warp for every candidate again with each atom and for the row sorts later:
// lists of 64,000 diamond atoms take 374 us by blocks and 102 by warps at 2
// atoms a cell, 190 and 138 at 7, 167 and 178 at 11, 171 and 256 at 19; of
// 4,000 atoms the lines cross at 6 a cell.
constexpr int NL_BLOCK_ATOMS = 10;

// A structure with five cells on each axis, which nl_search needs, has at least
// NL_WIDE_CELLS; with fewer than that on average its launch is spared (4 cells
// on an axis, 2048 atoms: 8 us).
constexpr int NL_WIDE_CELLS = 100;

static bool nl_blocks(const SysView &S, int n_cells, const float4 *local) {
    return local && (long long)S.n_atoms >= (long long)NL_BLOCK_ATOMS * n_cells &&
           (long long)n_cells >= (long long)NL_WIDE_CELLS * S.n_struct;
}

template <int MODE>
static int nl_rows(const SysView &S, const int *grids, const int *cell_start, const int *cell_atoms,
                   const float4 *local, int n_cells, double r_list, int *row_cnt, int *max_row, const int *row_off,
                   int *nbr, int stride, int *done, cudaStream_t st) {
    if (MODE == 2 && nl_blocks(S, n_cells, local)) {
        const int g = persistent_grid(n_cells, NL_T, (const void *)nl_search);
        nl_search<<<g, NL_T, 0, st>>>(S, grids, cell_start, local, n_cells, r_list, row_cnt, max_row, nbr, stride,
                                      done, max_row + 1);
    } else {
        done = nullptr;
    }
    const int g = persistent_grid((n_cells + NL_WARPS - 1) / NL_WARPS, 32 * NL_WARPS, (const void *)nl_cells<MODE>);
    nl_cells<MODE><<<g, 32 * NL_WARPS, 0, st>>>(S, grids, cell_start, cell_atoms, n_cells, r_list * r_list, row_cnt,
                                                max_row, row_off, nbr, stride, done);
    MBF_CHECK_LAUNCH();
    return MBF_OK;
}

// ---- row sorts -----------------------------------------------------------------
// Rows come out of nl_cells in traversal order; the CSR keeps them ascending
// (nl_search's are).  By length n: up to 32 entries one per lane, ranked by
// shuffles; up to 64 or 128 a bitonic network in registers over J = 2 or 4
// entries a lane (entry e = J lane + j, padded with INT_MAX, which sorts
// last since atom indices are smaller); longer rows by rank in shared
// memory.  Entries of a row are distinct.
constexpr int NL_PAD = 0x7fffffff;

__device__ __forceinline__ void cmp_swap(int &lo, int &hi, bool asc) {
    int mn = min(lo, hi), mx = max(lo, hi);
    lo = asc ? mn : mx;
    hi = asc ? mx : mn;
}

template <int J>
__device__ __forceinline__ void bitonic_sort(int (&v)[J]) {
    int lane = threadIdx.x & 31;
#pragma unroll
    for (int k = 2; k <= 32 * J; k <<= 1) {
#pragma unroll
        for (int d = k >> 1; d > 0; d >>= 1) {
            if (d >= J) {  // partner in lane ^ (d / J), same register
                bool low = (lane & (d / J)) == 0;
#pragma unroll
                for (int j = 0; j < J; ++j) {
                    int o = __shfl_xor_sync(MBF_FULL, v[j], d / J);
                    bool asc = ((J * lane + j) & k) == 0;
                    v[j] = (low == asc) ? min(v[j], o) : max(v[j], o);
                }
            } else {  // partner in register j ^ d of this lane
#pragma unroll
                for (int j = 0; j < J; ++j)
                    if ((j & d) == 0) cmp_swap(v[j], v[j ^ d], ((J * lane + j) & k) == 0);
            }
        }
    }
}

// Sorts n <= 32 J entries src[0..n) into out[0..n); returns this lane's
// count of entries below `a`.
template <int J>
__device__ __forceinline__ int sort_row_bitonic(const int *src, int n, int *out, int a) {
    int lane = threadIdx.x & 31;
    int v[J];
#pragma unroll
    for (int j = 0; j < J; ++j) v[j] = J * lane + j < n ? src[J * lane + j] : NL_PAD;
    __syncwarp();
    bitonic_sort<J>(v);
    int lower = 0;
#pragma unroll
    for (int j = 0; j < J; ++j)
        if (J * lane + j < n) {
            out[J * lane + j] = v[j];
            lower += v[j] < a ? 1 : 0;
        }
    return lower;
}

// Sorts the n entries src[0..n) (n <= NL_MAXROW) ascending into out[0..n)
// (src and out may be the same row: every entry is read before any is
// written) and returns how many are below `a` (warp-uniform).  `row` is
// the warp's shared scratch of NL_MAXROW ints.  COPIED: a row that is
// ascending already (the block search's) is only copied.
template <bool COPIED>
__device__ __forceinline__ int sort_row(const int *src, int n, int *out, int a, int *row) {
    int lane = threadIdx.x & 31;
    int lower = 0;
    if (COPIED && n <= 128) {
        int v[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const int k = 32 * j + lane;
            v[j] = k < n ? src[k] : NL_PAD;
        }
        bool asc = true;
        int prev = -1;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const int u = __shfl_up_sync(MBF_FULL, v[j], 1);
            asc = asc && (32 * j + lane >= n || (lane ? u : prev) < v[j]);
            prev = __shfl_sync(MBF_FULL, v[j], 31);
        }
        if (__all_sync(MBF_FULL, asc)) {
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const int k = 32 * j + lane;
                if (k < n && src != out) out[k] = v[j];
                lower += k < n && v[j] < a ? 1 : 0;
            }
            return __reduce_add_sync(MBF_FULL, lower);
        }
    } else if (COPIED) {
        bool asc = true;
        for (int k = lane; k < n - 1; k += 32) asc = asc && src[k] < src[k + 1];
        if (__all_sync(MBF_FULL, asc)) {
            for (int k = lane; k < n; k += 32) {
                const int v = src[k];
                if (src != out) out[k] = v;
                lower += v < a ? 1 : 0;
            }
            return __reduce_add_sync(MBF_FULL, lower);
        }
    }
    if (n <= 32) {
        int v = lane < n ? src[lane] : NL_PAD, rank = 0;
        for (int q = 0; q < n; ++q) rank += __shfl_sync(MBF_FULL, v, q) < v ? 1 : 0;
        if (lane < n) {
            out[rank] = v;
            lower = v < a ? 1 : 0;
        }
    } else if (n <= 64) {
        lower = sort_row_bitonic<2>(src, n, out, a);
    } else if (n <= 128) {
        lower = sort_row_bitonic<4>(src, n, out, a);
    } else {
        for (int k = lane; k < n; k += 32) row[k] = src[k];
        __syncwarp();
        for (int k = lane; k < n; k += 32) {
            int v = row[k], rank = 0;
            for (int q = 0; q < n; ++q) rank += row[q] < v ? 1 : 0;
            out[rank] = v;
            lower += v < a ? 1 : 0;
        }
        __syncwarp();
    }
    return __reduce_add_sync(MBF_FULL, lower);
}

// Each cell's atoms in ascending index order, so the traversal (and the
// rows it produces) do not depend on the order of nl_fill_cells's atomics:
// a warp per cell, the row sort above (a cell beyond NL_MAXROW atoms, which
// no physical density reaches, by insertion on one lane).
// With `local`, each atom's position relative to the middle of its cell, in
// float32, beside its index, in the cells' order (NaN for an atom whose cell
// coordinate lies beyond 4096 boxes): the periodic image next to the cell
// that nl_assign chose, whatever side of a cell face or of the box's own face
// the rounding here puts the atom on.  Then too which cells nl_search is to try
// (done), and whether any: not those of a structure with too few cells on an
// axis, nor those whose own atoms span nearly all of the index that its map
// reaches, as in a large structure whose atoms are in no spatial order (the
// stencil spans more still).  Left to nl_search itself that cost 50 us for
// 256,000 such atoms.
__global__ void nl_sort_cells(SysView S, const int *__restrict__ grids, int n_cells,
                              const int *__restrict__ cell_start, int *__restrict__ cell_atoms,
                              float4 *__restrict__ local, int *__restrict__ done, int *__restrict__ searched) {
    __shared__ int srow[NL_WARPS][NL_MAXROW];
    int wid = threadIdx.x >> 5, lane = threadIdx.x & 31;
    bool any = false;
    for (int c = blockIdx.x * NL_WARPS + wid; c < n_cells; c += gridDim.x * NL_WARPS) {
        int b = cell_start[c], n = cell_start[c + 1] - b;
        if (n <= NL_MAXROW) {
            sort_row<false>(cell_atoms + b, n, cell_atoms + b, NL_PAD, srow[wid]);
        } else if (lane == 0) {
            for (int i = b + 1; i < b + n; ++i) {
                int v = cell_atoms[i];
                int j = i - 1;
                while (j >= b && cell_atoms[j] > v) {
                    cell_atoms[j + 1] = cell_atoms[j];
                    --j;
                }
                cell_atoms[j + 1] = v;
            }
        }
        __syncwarp();
        if (!local || n == 0) continue;
        const int sidx = S.n_struct > 1 ? S.atom_struct[cell_atoms[b]] : 0;
        const int *g = grids + 8 * sidx;
        const double *L = S.cells + 18 * (size_t)sidx;
        const bool wide = grid_is_wide(g);
        bool take = wide && n <= NL_CAP;
        if (take && S.n_atoms > NL_BITS) {  // the cell's span as nl_search counts its range
            const int N = S.n_atoms, mid = cell_atoms[b + n / 2] - N / 2, base = mid + (mid < 0 ? N : 0);
            int low = N, high = 0;
            for (int k = lane; k < n; k += 32) {
                const int v = cell_atoms[b + k], x = v - base + (v < base ? N : 0);
                low = min(low, x);
                high = max(high, x);
            }
            take = __reduce_max_sync(MBF_FULL, high) - __reduce_min_sync(MBF_FULL, low) < NL_BITS - NL_BITS / 8;
        }
        if (lane == 0) done[c] = take ? 1 : 0;
        any = any || take;
        if (!wide) continue;  // no cell of the structure is searched by a block
        const int place = c - g[3];
        const double m0 = ((double)(place / (g[1] * g[2])) + 0.5) / (double)g[0];
        const double m1 = ((double)((place / g[2]) % g[1]) + 0.5) / (double)g[1];
        const double m2 = ((double)(place % g[2]) + 0.5) / (double)g[2];
        for (int k = lane; k < n; k += 32) {
            const int a = cell_atoms[b + k];
            const double *p = S.pos + 3 * (size_t)a;
            double f[3];
            bool far = false;
#pragma unroll
            for (int q = 0; q < 3; ++q) {
                const double s = p[0] * L[9 + q] + p[1] * L[12 + q] + p[2] * L[15 + q];
                if (!(fabs(s) <= 4096.0)) far = true;
                f[q] = s - floor(s) - (q == 0 ? m0 : q == 1 ? m1 : m2);
                f[q] -= rint(f[q]);
            }
            const float x = (float)(f[0] * L[0] + f[1] * L[3] + f[2] * L[6]);
            local[b + k] = make_float4(far ? __int_as_float(0x7fffffff) : x,
                                       (float)(f[0] * L[1] + f[1] * L[4] + f[2] * L[7]),
                                       (float)(f[0] * L[2] + f[1] * L[5] + f[2] * L[8]), __int_as_float(a));
        }
    }
    if (any && lane == 0) *searched = 1;
}

// Rows written in traversal order by nl_cells<1>: sorted in place, and
// each row's first upper slot recorded.
__global__ void nl_sort_rows(int n_atoms, const int *__restrict__ row_off, int *__restrict__ nbr,
                             int *__restrict__ upper, int *__restrict__ err) {
    __shared__ int srow[NL_WARPS][NL_MAXROW];
    int wid = threadIdx.x >> 5, lane = threadIdx.x & 31;
    for (int a = blockIdx.x * NL_WARPS + wid; a < n_atoms; a += gridDim.x * NL_WARPS) {
        int beg = row_off[a], n = row_off[a + 1] - beg;
        if (n > NL_MAXROW) {
            if (lane == 0) {
                atomicOr(err, MBF_DEV_ROW_TOO_LONG);
                upper[a] = beg;
            }
            continue;
        }
        int lower = sort_row<false>(nbr + beg, n, nbr + beg, a, srow[wid]);
        if (lane == 0) upper[a] = beg + lower;
    }
}

// The staged rows (nl_cells<2>, nl_search) into the CSR: each row read from its
// stride-spaced staging slot, sorted where it is not, and written at its scanned
// offset; its first upper slot recorded.  Rows longer than the stride were
// refused by the guard (their rows are empty by then).  COPIED where nl_search
// was launched, *searched whether it had cells: a look at rows that it did not
// leave costs a tenth of their sorts (256,000 atoms in no order: 229 against 209
// us, 198 in the kernel without that choice).
template <bool COPIED>
__device__ __forceinline__ void unstage_rows(int n_atoms, const int *__restrict__ row_off, const int *__restrict__ stage,
                                             int stride, int *__restrict__ nbr, int *__restrict__ upper,
                                             int *__restrict__ err, int *row) {
    int wid = threadIdx.x >> 5, lane = threadIdx.x & 31;
    for (int a = blockIdx.x * NL_WARPS + wid; a < n_atoms; a += gridDim.x * NL_WARPS) {
        int beg = row_off[a], n = row_off[a + 1] - beg;
        if (n > stride || n > NL_MAXROW) {
            if (lane == 0) {
                atomicOr(err, MBF_DEV_ROW_TOO_LONG);
                upper[a] = beg;
            }
            continue;
        }
        int lower = sort_row<COPIED>(stage + (size_t)a * stride, n, nbr + beg, a, row);
        if (lane == 0) upper[a] = beg + lower;
    }
}

template <bool COPIED>
__global__ void __launch_bounds__(32 * NL_WARPS, COPIED ? 10 : 1)
    nl_unstage_rows(int n_atoms, const int *__restrict__ row_off, const int *__restrict__ stage, int stride,
                    const int *__restrict__ searched, int *__restrict__ nbr, int *__restrict__ upper,
                    int *__restrict__ err) {
    __shared__ int srow[NL_WARPS][NL_MAXROW];
    int *row = srow[threadIdx.x >> 5];
    if (COPIED && *searched) unstage_rows<true>(n_atoms, row_off, stage, stride, nbr, upper, err, row);
    else unstage_rows<false>(n_atoms, row_off, stage, stride, nbr, upper, err, row);
}

// Reverse slot of every slot.  rev is an involution, so only the upper
// slots (a -> b, b > a) search: a lies in the lower part of b's sorted row,
// [row_off[b], upper[b]); the slot t found there gets rev[t] = s, so every
// slot is written once.  Eight lanes per row: an upper part holds about
// half a row, so short rows keep the lanes busy.
constexpr int NL_REV_LANES = 8;

__global__ void nl_reverse(int n_atoms, const int *__restrict__ row_off, const int *__restrict__ upper,
                           const int *__restrict__ nbr, int *__restrict__ rev, int *__restrict__ err) {
    const int grp = threadIdx.x / NL_REV_LANES, sub = threadIdx.x % NL_REV_LANES;
    const int per_block = 32 * NL_WARPS / NL_REV_LANES;
    for (int a = blockIdx.x * per_block + grp; a < n_atoms; a += gridDim.x * per_block) {
        for (int s = upper[a] + sub; s < row_off[a + 1]; s += NL_REV_LANES) {
            int b = nbr[s];
            int lo = row_off[b], hi = upper[b] - 1, found = -1;
            while (lo <= hi) {
                int mid = (lo + hi) >> 1;
                int v = nbr[mid];
                if (v == a) { found = mid; break; }
                if (v < a) lo = mid + 1; else hi = mid - 1;
            }
            if (found < 0) {
                atomicOr(err, MBF_DEV_BAD_INDEX);
                rev[s] = s;
                continue;
            }
            rev[s] = found;
            rev[found] = s;
        }
    }
}

// Per-structure largest minimum-image displacement from the reference
// positions mapped by the lattice change (engine/neighborlist.py:661-668).
__global__ void nl_max_disp(SysView S, const double *__restrict__ ref, const double *__restrict__ maps,
                            unsigned long long *__restrict__ dmax_bits) {
    int a = blockIdx.x * blockDim.x + threadIdx.x;
    if (a >= S.n_atoms) return;
    int s = S.n_struct > 1 ? S.atom_struct[a] : 0;
    const double *r0 = ref + 3 * (size_t)a;
    double ax = r0[0], ay = r0[1], az = r0[2];
    if (maps) {  // null: lattice unchanged, M = I
        const double *M = maps + 9 * (size_t)s;
        ax = r0[0] * M[0] + r0[1] * M[3] + r0[2] * M[6];
        ay = r0[0] * M[1] + r0[1] * M[4] + r0[2] * M[7];
        az = r0[0] * M[2] + r0[1] * M[5] + r0[2] * M[8];
    }
    double dx, dy, dz;
    mic_exact(S.cells + 18 * (size_t)s, S.pos[3 * (size_t)a] - ax, S.pos[3 * (size_t)a + 1] - ay,
              S.pos[3 * (size_t)a + 2] - az, dx, dy, dz);
    double d = sqrt(dx * dx + dy * dy + dz * dz);
    atomicMax(dmax_bits + s, (unsigned long long)__double_as_longlong(d));
}

__global__ void nl_upper_count(int n_atoms, const int *__restrict__ row_off, const int *__restrict__ nbr,
                               int *__restrict__ up) {
    int a = blockIdx.x * blockDim.x + threadIdx.x;
    if (a >= n_atoms) return;
    int c = 0;
    for (int s = row_off[a]; s < row_off[a + 1]; ++s) c += nbr[s] > a ? 1 : 0;
    up[a] = c;
}

__global__ void nl_upper_write(int n_atoms, const int *__restrict__ row_off, const int *__restrict__ nbr,
                               const int *__restrict__ up_off, int *__restrict__ pi, int *__restrict__ pj) {
    int a = blockIdx.x * blockDim.x + threadIdx.x;
    if (a >= n_atoms) return;
    int o = up_off[a];
    for (int s = row_off[a]; s < row_off[a + 1]; ++s) {
        int b = nbr[s];
        if (b > a) {
            pi[o] = a;
            pj[o] = b;
            ++o;
        }
    }
}

// Device-side checks of the graph-capturable rebuild: a list that would not
// fit its buffers or a row beyond the caller's staging limit sets a status
// bit and leaves every row empty (no slot is written), so later kernels of a
// captured sequence read nothing out of bounds.
__global__ void nl_guard(int n_atoms, const int *__restrict__ row_off, const int *__restrict__ mrow,
                         long long cap, int limit, int *__restrict__ status, int *__restrict__ skip) {
    if (threadIdx.x != 0) return;
    int bad = 0;
    if ((long long)row_off[n_atoms] > cap) bad |= MBF_STATUS_CAPACITY;
    if (*mrow > limit) bad |= MBF_STATUS_ROW_TOO_LONG;
    *skip = bad;
    if (bad) atomicOr(status, bad);
}

__global__ void nl_clear_if(int n_atoms, const int *__restrict__ skip, int *__restrict__ row_off,
                            int *__restrict__ upper) {
    if (*skip == 0) return;
    int a = blockIdx.x * blockDim.x + threadIdx.x;
    if (a <= n_atoms) row_off[a] = 0;
    if (a < n_atoms) upper[a] = 0;
}

// Records d (this step's largest displacement since the last rebuild) and
// the reference's rebuild decision r_list - 2 d <= r_cut (any structure,
// engine/neighborlist.py:653-673 with the lattice unchanged); sets the
// graph conditional that gates the rebuild branch when one is given, and
// flags MBF_STATUS_SKIN when a status word is given (fixed-interval runs,
// where the decision is an assertion).
__global__ void nl_skin_record(int n_struct, const double *__restrict__ d, double r_list, double r_cut,
                               double *__restrict__ d_log,
                               int rows, int *__restrict__ counter, int *__restrict__ gate, int *__restrict__ status,
                               unsigned long long cond) {
    if (threadIdx.x != 0) return;
    int row = *counter % rows;
    int need = 0;
    for (int s = 0; s < n_struct; ++s) {
        d_log[(size_t)row * n_struct + s] = d[s];
        if (r_list - 2.0 * d[s] <= r_cut) need = 1;
    }
    *gate = need;
    if (need && status) atomicOr(status, MBF_STATUS_SKIN);
    if (cond) cudaGraphSetConditional((cudaGraphConditionalHandle)cond, need ? 1u : 0u);
    *counter += 1;
}

__global__ void nl_count_rebuild(int *__restrict__ n) {
    if (threadIdx.x == 0) *n += 1;
}

__global__ void nl_status_merge(const int *__restrict__ err, int *__restrict__ status) {
    if (threadIdx.x != 0) return;
    int e = err[0];
    if (e & MBF_DEV_ROW_TOO_LONG) atomicOr(status, MBF_STATUS_ROW_TOO_LONG);
    if (e & ~MBF_DEV_ROW_TOO_LONG) atomicOr(status, MBF_STATUS_BAD_INDEX);
}

}  // namespace mbf

using namespace mbf;

extern "C" {

size_t mbf_nl_workspace_bytes(int n_atoms, int n_cells_total) {
    return nl_layout(n_atoms, n_cells_total).total;
}

size_t mbf_nl_rebuild_workspace_bytes(int n_atoms, int n_cells_total, int max_row_limit) {
    if (n_atoms < 0 || n_cells_total <= 0 || max_row_limit <= 0) return 0;
    return nl_staged_bytes(nl_layout(n_atoms, n_cells_total), n_atoms, max_row_limit);
}

static int nl_prepare(const SysView &S, const int *grids, int n_cells_total, double r_list, void *workspace,
                      const NlLayout &L, int *row_off, cudaStream_t st, int *stage = nullptr, int stride = 0,
                      float4 *local = nullptr) {
    int N = S.n_atoms;
    int *err = ws_at<int>(workspace, L.err);
    int *atom_cell = ws_at<int>(workspace, L.atom_cell);
    int *cell_count = ws_at<int>(workspace, L.cell_count);
    int *cell_start = ws_at<int>(workspace, L.cell_start);
    int *cursor = ws_at<int>(workspace, L.cursor);
    int *cell_atoms = ws_at<int>(workspace, L.cell_atoms);
    int *row_cnt = ws_at<int>(workspace, L.row_cnt);
    int *mrow = ws_at<int>(workspace, L.maxrow);
    int *scan_ws = ws_at<int>(workspace, L.scan);
    if (cudaMemsetAsync(err, 0, 64, st) != cudaSuccess) return MBF_ERR_CUDA;
    // the longest row, and whether nl_search has cells
    if (cudaMemsetAsync(mrow, 0, 2 * sizeof(int), st) != cudaSuccess) return MBF_ERR_CUDA;
    if (cudaMemsetAsync(cell_count, 0, sizeof(int) * (size_t)n_cells_total, st) != cudaSuccess)
        return MBF_ERR_CUDA;
    PROF_BEGIN("nl_assign", st);
    nl_assign<<<(N + 255) / 256, 256, 0, st>>>(S, grids, atom_cell, cell_count);
    PROF_END("nl_assign", st);
    MBF_CHECK_LAUNCH();
    int rc = exclusive_scan(cell_count, cell_start, n_cells_total, scan_ws, st);
    if (rc != MBF_OK) return rc;
    if (cudaMemcpyAsync(cursor, cell_start, sizeof(int) * (size_t)n_cells_total,
                        cudaMemcpyDeviceToDevice, st) != cudaSuccess)
        return MBF_ERR_CUDA;
    PROF_BEGIN("nl_fill_cells", st);
    nl_fill_cells<<<(N + 255) / 256, 256, 0, st>>>(N, atom_cell, cursor, cell_atoms);
    nl_sort_cells<<<persistent_grid((n_cells_total + NL_WARPS - 1) / NL_WARPS, 32 * NL_WARPS,
                                    (const void *)nl_sort_cells),
                    32 * NL_WARPS, 0, st>>>(S, grids, n_cells_total, cell_start, cell_atoms,
                                            nl_blocks(S, n_cells_total, local) ? local : nullptr, cursor, mrow + 1);
    PROF_END("nl_fill_cells", st);
    MBF_CHECK_LAUNCH();
    PROF_BEGIN("nl_count", st);
    rc = stage ? nl_rows<2>(S, grids, cell_start, cell_atoms, local, n_cells_total, r_list, row_cnt, mrow, nullptr,
                            stage, stride, cursor, st)
               : nl_rows<0>(S, grids, cell_start, cell_atoms, nullptr, n_cells_total, r_list, row_cnt, mrow, nullptr,
                            nullptr, 0, nullptr, st);
    PROF_END("nl_count", st);
    if (rc != MBF_OK) return rc;
    return exclusive_scan(row_cnt, row_off, N, scan_ws, st);
}

static int nl_finish(const SysView &S, const int *grids, int n_cells_total, double r_list, void *workspace,
                     const NlLayout &L, const int *row_off, int *nbr, int *rev, int *upper, cudaStream_t st,
                     const int *stage, int stride, const float4 *local) {
    int N = S.n_atoms;
    int *err = ws_at<int>(workspace, L.err);
    int blocks = (N + NL_WARPS - 1) / NL_WARPS;
    const bool copied = nl_blocks(S, n_cells_total, local);
    int g = persistent_grid(blocks, 32 * NL_WARPS, !stage   ? (const void *)nl_sort_rows
                                                   : copied ? (const void *)nl_unstage_rows<true>
                                                            : (const void *)nl_unstage_rows<false>);
    PROF_BEGIN("nl_fill", st);
    if (stage) {
        const int *searched = ws_at<int>(workspace, L.maxrow) + 1;
        if (copied)
            nl_unstage_rows<true><<<g, 32 * NL_WARPS, 0, st>>>(N, row_off, stage, stride, searched, nbr, upper, err);
        else
            nl_unstage_rows<false><<<g, 32 * NL_WARPS, 0, st>>>(N, row_off, stage, stride, searched, nbr, upper, err);
    } else {
        int rc = nl_rows<1>(S, grids, ws_at<int>(workspace, L.cell_start), ws_at<int>(workspace, L.cell_atoms),
                            nullptr, n_cells_total, r_list, nullptr, nullptr, row_off, nbr, 0, nullptr, st);
        if (rc != MBF_OK) return rc;
        nl_sort_rows<<<g, 32 * NL_WARPS, 0, st>>>(N, row_off, nbr, upper, err);
    }
    PROF_END("nl_fill", st);
    MBF_CHECK_LAUNCH();
    g = persistent_grid((N + 32 * NL_WARPS / NL_REV_LANES - 1) / (32 * NL_WARPS / NL_REV_LANES), 32 * NL_WARPS,
                        (const void *)nl_reverse);
    PROF_BEGIN("nl_reverse", st);
    nl_reverse<<<g, 32 * NL_WARPS, 0, st>>>(N, row_off, upper, nbr, rev, err);
    PROF_END("nl_reverse", st);
    MBF_CHECK_LAUNCH();
    return MBF_OK;
}

int mbf_nl_build(const mbf_system *sys, const int *grids, int n_cells_total, double r_list,
                 void *workspace, size_t workspace_bytes, int *row_off, int *nbr, int *rev, int *upper,
                 long long nbr_capacity, long long *n_slots, int *max_row, void *stream) {
    if (!sys || !grids || !workspace || !row_off || !n_slots || !max_row || sys->n_atoms < 0 ||
        n_cells_total <= 0 || !(r_list > 0.0))
        return MBF_ERR_ARGUMENT;
    cudaStream_t st = (cudaStream_t)stream;
    int N = sys->n_atoms;
    NlLayout L = nl_layout(N, n_cells_total);
    if (workspace_bytes < L.total) return MBF_ERR_WORKSPACE;
    SysView S = make_view(sys);
    if (N == 0) {
        if (cudaMemsetAsync(row_off, 0, sizeof(int), st) != cudaSuccess) return MBF_ERR_CUDA;
        *n_slots = 0;
        *max_row = 0;
        return MBF_OK;
    }
    // workspace beyond the layout holds staging rows at the stride it allows:
    // if no row is longer, the search runs once (count and stage, then sort
    // into the CSR), else the rows are searched again (fill); where it has
    // room for both, the local coordinates of the block search come first
    int stride = 0;
    float4 *local = nullptr;
    size_t room = workspace_bytes - L.total, front = 0;
    if (room >= 256) {
        front = nl_local_bytes(N);
        if (room >= front + sizeof(int) * (size_t)N && nl_local_ok(workspace))
            local = ws_at<float4>(workspace, L.total);
        else
            front = 0;
        size_t per = (room - front) / (sizeof(int) * (size_t)N);
        stride = (int)(per < (size_t)NL_MAXROW ? per : (size_t)NL_MAXROW);
        if ((long long)N * stride >= 0x7fffffffLL) stride = (int)(0x7ffffffeLL / N);
    }
    int *stage = stride > 0 ? ws_at<int>(workspace, L.total + front) : nullptr;
    int rc = nl_prepare(S, grids, n_cells_total, r_list, workspace, L, row_off, st, stage, stride, local);
    if (rc != MBF_OK) return rc;
    int host[2];
    if (cudaMemcpyAsync(&host[0], row_off + N, sizeof(int), cudaMemcpyDeviceToHost, st) != cudaSuccess ||
        cudaMemcpyAsync(&host[1], ws_at<int>(workspace, L.maxrow), sizeof(int), cudaMemcpyDeviceToHost, st) !=
            cudaSuccess ||
        cudaStreamSynchronize(st) != cudaSuccess)
        return MBF_ERR_CUDA;
    *n_slots = host[0];
    *max_row = host[1];
    if ((long long)host[0] > nbr_capacity || !nbr || !rev) return MBF_ERR_CAPACITY;
    if (!upper) return MBF_ERR_ARGUMENT;
    if (host[1] > NL_MAXROW) return MBF_ERR_ROW_TOO_LONG;
    if (host[1] > stride) stage = nullptr;
    rc = nl_finish(S, grids, n_cells_total, r_list, workspace, L, row_off, nbr, rev, upper, st, stage,
                   stage ? stride : 0, local);
    if (rc != MBF_OK) return rc;
    int herr = 0;
    if (cudaMemcpyAsync(&herr, ws_at<int>(workspace, L.err), sizeof(int), cudaMemcpyDeviceToHost, st) !=
            cudaSuccess ||
        cudaStreamSynchronize(st) != cudaSuccess)
        return MBF_ERR_CUDA;
    if (herr & MBF_DEV_ROW_TOO_LONG) return MBF_ERR_ROW_TOO_LONG;
    if (herr) return MBF_ERR_ARGUMENT;
    return MBF_OK;
}

int mbf_nl_rebuild_async(const mbf_system *sys, const int *grids, int n_cells_total, double r_list,
                         void *workspace, size_t workspace_bytes, int *row_off, int *nbr, int *rev, int *upper,
                         long long nbr_capacity, int max_row_limit, int *status, void *stream) {
    if (!sys || !grids || !workspace || !row_off || !nbr || !rev || !upper || !status || sys->n_atoms <= 0 ||
        n_cells_total <= 0 || !(r_list > 0.0) || nbr_capacity < 0 || max_row_limit <= 0 ||
        max_row_limit > NL_MAXROW)
        return MBF_ERR_ARGUMENT;
    cudaStream_t st = (cudaStream_t)stream;
    int N = sys->n_atoms;
    NlLayout L = nl_layout(N, n_cells_total);
    if (workspace_bytes < L.total) return MBF_ERR_WORKSPACE;
    SysView S = make_view(sys);
    // with room for the staging rows the search runs once (count and stage),
    // with room for the local coordinates too by blocks; else it counts, then
    // fills
    int *stage = nullptr;
    float4 *local = nullptr;
    size_t rows = align256(sizeof(int) * (size_t)N * (size_t)max_row_limit);
    if (workspace_bytes >= L.total + rows && (long long)N * max_row_limit < 0x7fffffffLL) {
        stage = ws_at<int>(workspace, L.total);
        if (workspace_bytes >= nl_staged_bytes(L, N, max_row_limit) && nl_local_ok(workspace)) {
            local = ws_at<float4>(workspace, L.total);
            stage = ws_at<int>(workspace, L.total + nl_local_bytes(N));
        }
    }
    int rc = nl_prepare(S, grids, n_cells_total, r_list, workspace, L, row_off, st, stage, max_row_limit, local);
    if (rc != MBF_OK) return rc;
    int *err = ws_at<int>(workspace, L.err);
    nl_guard<<<1, 32, 0, st>>>(N, row_off, ws_at<int>(workspace, L.maxrow), nbr_capacity, max_row_limit, status,
                               err + 4);
    nl_clear_if<<<(N + 256) / 256, 256, 0, st>>>(N, err + 4, row_off, upper);
    MBF_CHECK_LAUNCH();
    rc = nl_finish(S, grids, n_cells_total, r_list, workspace, L, row_off, nbr, rev, upper, st, stage, max_row_limit, local);
    if (rc != MBF_OK) return rc;
    nl_status_merge<<<1, 32, 0, st>>>(err, status);
    MBF_CHECK_LAUNCH();
    return MBF_OK;
}

int mbf_nl_max_displacement(const mbf_system *sys, const double *ref_positions, const double *maps,
                            double *d_max, void *stream) {
    if (!sys || !ref_positions || !maps || !d_max) return MBF_ERR_ARGUMENT;
    cudaStream_t st = (cudaStream_t)stream;
    SysView S = make_view(sys);
    if (cudaMemsetAsync(d_max, 0, sizeof(double) * (size_t)sys->n_struct, st) != cudaSuccess)
        return MBF_ERR_CUDA;
    if (sys->n_atoms == 0) return MBF_OK;
    nl_max_disp<<<(sys->n_atoms + 255) / 256, 256, 0, st>>>(S, ref_positions, maps,
                                                            (unsigned long long *)d_max);
    MBF_CHECK_LAUNCH();
    return MBF_OK;
}

int mbf_md_skin_check(const mbf_system *sys, const double *ref_positions, double r_list, double r_cut,
                      double *d_scratch, double *d_log, int rows, int *counter, int *gate, int *status,
                      unsigned long long cond_handle, void *stream) {
    if (!sys || !ref_positions || !d_scratch || !d_log || !counter || !gate || rows <= 0 || !(r_list > r_cut) ||
        !(r_cut > 0.0) || sys->n_struct <= 0)
        return MBF_ERR_ARGUMENT;
    cudaStream_t st = (cudaStream_t)stream;
    SysView S = make_view(sys);
    if (cudaMemsetAsync(d_scratch, 0, sizeof(double) * (size_t)sys->n_struct, st) != cudaSuccess)
        return MBF_ERR_CUDA;
    if (sys->n_atoms > 0) {
        nl_max_disp<<<(sys->n_atoms + 255) / 256, 256, 0, st>>>(S, ref_positions, nullptr,
                                                                (unsigned long long *)d_scratch);
        MBF_CHECK_LAUNCH();
    }
    nl_skin_record<<<1, 32, 0, st>>>(sys->n_struct, d_scratch, r_list, r_cut, d_log, rows, counter, gate,
                                     status, cond_handle);
    MBF_CHECK_LAUNCH();
    return MBF_OK;
}

int mbf_md_rebuild_done(const mbf_system *sys, double *ref_positions, int *rebuild_count, void *stream) {
    if (!sys || !ref_positions || !rebuild_count) return MBF_ERR_ARGUMENT;
    cudaStream_t st = (cudaStream_t)stream;
    if (sys->n_atoms > 0 &&
        cudaMemcpyAsync(ref_positions, sys->positions, sizeof(double) * 3 * (size_t)sys->n_atoms,
                        cudaMemcpyDeviceToDevice, st) != cudaSuccess)
        return MBF_ERR_CUDA;
    nl_count_rebuild<<<1, 32, 0, st>>>(rebuild_count);
    MBF_CHECK_LAUNCH();
    return MBF_OK;
}

size_t mbf_nl_half_workspace_bytes(int n_atoms) {
    return sizeof(int) * ((size_t)2 * n_atoms + 2 + scan_workspace_ints(n_atoms + 1)) + 256;
}

int mbf_nl_half_pairs(const mbf_nlist *nl, int *pair_i, int *pair_j, void *workspace,
                      size_t workspace_bytes, void *stream) {
    if (!nl || !pair_i || !pair_j || !workspace) return MBF_ERR_ARGUMENT;
    int N = nl->n_atoms;
    if (workspace_bytes < mbf_nl_half_workspace_bytes(N)) return MBF_ERR_WORKSPACE;
    if (N == 0) return MBF_OK;
    cudaStream_t st = (cudaStream_t)stream;
    int *up = (int *)workspace;
    int *up_off = up + N;
    int *scan_ws = up_off + N + 2;
    nl_upper_count<<<(N + 255) / 256, 256, 0, st>>>(N, nl->row_off, nl->nbr, up);
    MBF_CHECK_LAUNCH();
    int rc = exclusive_scan(up, up_off, N, scan_ws, st);
    if (rc != MBF_OK) return rc;
    nl_upper_write<<<(N + 255) / 256, 256, 0, st>>>(N, nl->row_off, nl->nbr, up_off, pair_i, pair_j);
    MBF_CHECK_LAUNCH();
    return MBF_OK;
}

}  // extern "C"
