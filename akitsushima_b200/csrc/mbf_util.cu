// Scan, per-structure reduction and small utilities shared by the kernels.
#include "mbf_util.cuh"

namespace mbf {

int persistent_grid(int blocks_needed, int block, const void *kernel, size_t smem) {
    static int n_sm = 0;
    if (n_sm == 0) {
        int dev = 0;
        cudaGetDevice(&dev);
        cudaDeviceGetAttribute(&n_sm, cudaDevAttrMultiProcessorCount, dev);
        if (n_sm <= 0) n_sm = 148;
    }
    int per_sm = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, block, smem) != cudaSuccess ||
        per_sm <= 0)
        per_sm = 1;
    int g = n_sm * per_sm;
    if (blocks_needed < g) g = blocks_needed;
    return g > 0 ? g : 1;
}

// ---- exclusive scan of int32 (n + 1 outputs: out[n] = total) -------------

constexpr int SCAN_BLOCK = 1024;
constexpr int SCAN_ITEMS = 4;
constexpr int SCAN_TILE = SCAN_BLOCK * SCAN_ITEMS;

__device__ __forceinline__ int warp_incl_scan(int v) {
    int lane = threadIdx.x & 31;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        int t = __shfl_up_sync(MBF_FULL, v, o);
        if (lane >= o) v += t;
    }
    return v;
}

// Block-wide exclusive scan of one value per thread; returns the block total.
__device__ int block_excl_scan(int v, int &excl) {
    __shared__ int warp_tot[32];
    __shared__ int block_tot;
    int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    int inc = warp_incl_scan(v);
    if (lane == 31) warp_tot[wid] = inc;
    __syncthreads();
    if (wid == 0) {
        int nw = blockDim.x >> 5;
        int t = lane < nw ? warp_tot[lane] : 0;
        int ti = warp_incl_scan(t);
        if (lane < nw) warp_tot[lane] = ti - t;
        if (lane == 31) block_tot = ti;  // nw <= 32
    }
    __syncthreads();
    excl = inc - v + warp_tot[wid];
    int total = block_tot;
    __syncthreads();
    return total;
}

__global__ void scan_tiles(const int *__restrict__ in, int *__restrict__ out, int n,
                           int *__restrict__ tile_sums) {
    int base = blockIdx.x * SCAN_TILE + threadIdx.x * SCAN_ITEMS;
    int v[SCAN_ITEMS];
    int s = 0;
#pragma unroll
    for (int k = 0; k < SCAN_ITEMS; ++k) {
        v[k] = (base + k < n) ? in[base + k] : 0;
        s += v[k];
    }
    int excl;
    int total = block_excl_scan(s, excl);
#pragma unroll
    for (int k = 0; k < SCAN_ITEMS; ++k) {
        if (base + k < n) out[base + k] = excl;
        excl += v[k];
    }
    if (threadIdx.x == 0) tile_sums[blockIdx.x] = total;
}

// Adds to each tile the sum of the tiles before it, which every block forms
// for itself from the tile sums (at most a few thousand, in cache), so the
// scan is two launches; the last block writes the grand total.
__global__ void __launch_bounds__(SCAN_BLOCK) scan_add(int *__restrict__ out, int n, const int *__restrict__ tile_sums,
                                                       int n_tiles) {
    __shared__ int warp_sum[32];
    __shared__ int before;
    int v = 0;
    for (int k = threadIdx.x; k < blockIdx.x; k += SCAN_BLOCK) v += tile_sums[k];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(MBF_FULL, v, o);
    if ((threadIdx.x & 31) == 0) warp_sum[threadIdx.x >> 5] = v;
    __syncthreads();
    if (threadIdx.x < 32) {
        int t = warp_sum[threadIdx.x];
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) t += __shfl_xor_sync(MBF_FULL, t, o);
        if (threadIdx.x == 0) before = t;
    }
    __syncthreads();
    const int add = before;
    const int base = blockIdx.x * SCAN_TILE + threadIdx.x;
#pragma unroll
    for (int k = 0; k < SCAN_ITEMS; ++k) {
        const int i = base + k * SCAN_BLOCK;
        if (i < n) out[i] += add;
    }
    if ((int)blockIdx.x == n_tiles - 1 && threadIdx.x == 0) out[n] = add + tile_sums[n_tiles - 1];
}

size_t scan_workspace_ints(int n) { return (size_t)(n + SCAN_TILE - 1) / SCAN_TILE + 2; }

int exclusive_scan(const int *in, int *out, int n, int *ws, cudaStream_t st) {
    int n_tiles = (n + SCAN_TILE - 1) / SCAN_TILE;
    if (n_tiles == 0) n_tiles = 1;
    scan_tiles<<<n_tiles, SCAN_BLOCK, 0, st>>>(in, out, n, ws);
    scan_add<<<n_tiles, SCAN_BLOCK, 0, st>>>(out, n, ws, n_tiles);
    MBF_CHECK_LAUNCH();
    return MBF_OK;
}

// ---- force gather and per-structure sums -----------------------------------

// Gather the three-body forces the centres left on atom a: every centre x
// wrote the force its terms put on a into a's own slot (a -> x), so the row
// is read contiguously, 8 lanes per atom; fused with the per-structure sums
// (ChunkSums): a block per chunk of the reduction plan, each group also
// adding its atom's record (entries sub and sub + 8).  Only the slots whose
// live bit is set are read: a list radius of cutoff + skin holds two to three
// times the slots that carry a force (32,768-atom SiC: 15.5 listed, 6 live),
// and the others are never written.  Bound by latency, hence by how many
// groups are resident and how much of a row each has in flight: 16 slots of a
// row at a time take 22.9 us for the 512 uneven silicon cells and 16.1 for
// 64,000 GeSn atoms, 32 at a time 28.6 and 18.9, 8 at a time 24.7 and 18.8;
// two atoms a group at once 31 and 20.7; at 1536 threads an SM the registers
// spill (30 and 20.9).
constexpr int GATHER_K = 2;

template <int NT>
__global__ void __launch_bounds__(NT, 1024 / NT) gather_live_rows(const int *__restrict__ row_off, int n_slots,
                                                       const double *__restrict__ G,
                                                       const uint4 *__restrict__ live_mask, int row_limit,
                                                       int *__restrict__ err, const double *__restrict__ f_local,
                                                       double *__restrict__ forces, ChunkSums cs) {
    constexpr int LPA = 8, NG = NT / LPA;
    const int c = blockIdx.x;
    const int s = cs.chunk[3 * c], a0 = cs.chunk[3 * c + 1], a1 = cs.chunk[3 * c + 2];
    const int sub = threadIdx.x & (LPA - 1), grp = threadIdx.x / LPA;
    double r0 = 0.0, r1 = 0.0;
    // the next atom's bounds and mask one iteration ahead: a slot's load then
    // waits on nothing
    int nb = 0, ne = 0;
    uint4 nm = make_uint4(0u, 0u, 0u, 0u);
    if (a0 + grp < a1) {
        nb = row_off[a0 + grp];
        ne = row_off[a0 + grp + 1];
        nm = live_mask[a0 + grp];
    }
    for (int base = a0; base < a1; base += NG) {  // uniform over the block
        const int a = base + grp, beg = nb;
        int n = ne - nb;
        const uint4 m4 = nm;
        if (a + NG < a1) {
            nb = row_off[a + NG];
            ne = row_off[a + NG + 1];
            nm = live_mask[a + NG];
        }
        double ra = 0.0, rb = 0.0, fl = 0.0, f[3] = {0.0, 0.0, 0.0};
        if (a < a1) {
            const double *pa = cs.per_atom + (size_t)a * ATOM_ACC;
            ra = pa[sub];
            if (sub < ATOM_ACC - LPA) rb = pa[LPA + sub];
            if (sub < 3) fl = f_local[3 * (size_t)a + sub];
        } else {
            n = 0;
        }
        if ((unsigned)beg > (unsigned)n_slots || (unsigned)n > (unsigned)(n_slots - beg)) {
            if (sub == 0) atomicOr(err, MBF_DEV_BAD_INDEX);
            n = 0;
        } else if (n > row_limit) {
            if (sub == 0) atomicOr(err, MBF_DEV_ROW_TOO_LONG);
            n = 0;
        }
        for (int w = 0; w < n; w += GATHER_K * LPA) {
            const unsigned m = w < 32 ? m4.x : (w < 64 ? m4.y : (w < 96 ? m4.z : m4.w));
            double x[GATHER_K][3];
#pragma unroll
            for (int k = 0; k < GATHER_K; ++k) {
                x[k][0] = x[k][1] = x[k][2] = 0.0;
                if (m >> ((w & 31) + sub + LPA * k) & 1u) {
                    const double *g = G + 3 * (size_t)(beg + w + sub + LPA * k);
#pragma unroll
                    for (int q = 0; q < 3; ++q) x[k][q] = __ldcs(g + q);
                }
            }
#pragma unroll
            for (int k = 0; k < GATHER_K; ++k)
#pragma unroll
                for (int q = 0; q < 3; ++q) f[q] += x[k][q];
        }
        if (sub == 10 - LPA && rb < 0.0) {  // a bad index in the row (put_atom)
            atomicOr(err, MBF_DEV_BAD_INDEX);
            rb = 0.0;
        }
        r0 += ra;
        r1 += rb;
#pragma unroll
        for (int q = 0; q < 3; ++q) f[q] = group_sum<LPA>(f[q]);
        // lane k (k < 3) of the group writes component k
        const double g = sub == 0 ? f[0] : (sub == 1 ? f[1] : f[2]);
        if (sub < 3 && a < a1) forces[3 * (size_t)a + sub] = fl + g;
    }
    chunk_sums_finish<NT>(cs, c, s, r0, r1);
}

int gather_live(int n_struct, int n_atoms, const int *row_off, int n_slots, const double *G, const unsigned *live_mask,
                int row_limit, int *err, const double *f_local, double *forces, const double *per_atom,
                const mbf_reduce_plan *plan, double *partial, double *energy, double *virial, unsigned *sdone,
                cudaStream_t st) {
    if (plan->n_chunks <= 0 || n_struct <= 0 || plan->n_chunks < n_struct || !sdone) return MBF_ERR_ARGUMENT;
    ChunkSums cs = {plan->chunk, plan->chunk_first, per_atom, partial, energy, virial, sdone};
    const uint4 *mask = reinterpret_cast<const uint4 *>(live_mask);
    PROF_BEGIN("gather_live", st);
    const int nt = chunk_block(n_atoms, plan->n_chunks);
    if (nt == 128)
        gather_live_rows<128><<<plan->n_chunks, 128, 0, st>>>(row_off, n_slots, G, mask, row_limit, err, f_local,
                                                              forces, cs);
    else if (nt == 256)
        gather_live_rows<256><<<plan->n_chunks, 256, 0, st>>>(row_off, n_slots, G, mask, row_limit, err, f_local,
                                                              forces, cs);
    else
        gather_live_rows<512><<<plan->n_chunks, 512, 0, st>>>(row_off, n_slots, G, mask, row_limit, err, f_local,
                                                              forces, cs);
    PROF_END("gather_live", st);
    MBF_CHECK_LAUNCH();
    return MBF_OK;
}

}  // namespace mbf

extern "C" {

const char *mbf_error_string(int code) {
    switch (code) {
        case MBF_OK: return "ok";
        case MBF_ERR_ARGUMENT: return "invalid argument";
        case MBF_ERR_CUDA: return "CUDA runtime error";
        case MBF_ERR_CAPACITY: return "neighbour capacity too small";
        case MBF_ERR_ROW_TOO_LONG: return "neighbour row longer than the kernel's staging limit";
        case MBF_ERR_WORKSPACE: return "workspace too small";
        case MBF_ERR_SCRATCH_LIMIT: return "size beyond the no-allocation entry point's limit";
        default: return "unknown error";
    }
}

int mbf_version(void) { return 10000; }

size_t mbf_eval_workspace_bytes(int n_atoms, long long n_slots, int n_chunks) {
    return mbf::eval_layout(n_atoms, n_slots, n_chunks).total;
}

int mbf_eval_status(const void *workspace, int *host_words, void *stream) {
    if (!workspace || !host_words) return MBF_ERR_ARGUMENT;
    cudaStream_t st = (cudaStream_t)stream;
    if (cudaMemcpyAsync(host_words, workspace, 4 * sizeof(int), cudaMemcpyDeviceToHost, st) != cudaSuccess ||
        cudaStreamSynchronize(st) != cudaSuccess)
        return MBF_ERR_CUDA;
    return MBF_OK;
}

}  // extern "C"
