// ssp_pcg.cu -- a8: preconditioned conjugate gradients on all k right-hand sides at once.
//
// Reference: example_pcg_solver (custom_cg.hpp:96-274), called once per sketch column
// (example.cc:552-569).  Per column: b = rhs - mean(rhs) (:132), x0 = 0 (:140), PCG with the
// preconditioner M^{-1} r = L^{-T} D^+ L^{-1} r (:224-235, zero pivots skipped), stop once
// ||r|| <= max(abs_tol, tol ||b||) (the reference's own rule is ||r||^2 <= 2e-7, :159,213), at most
// max_iters iterations (:153), and success iff ||b - A x|| / ||b|| < 0.01 (:251-258).
//
// Layout ("tile-major", tile_off): an n x k block is stored as slabs of n x SSP_TILE values.  Every
// kernel works on one tile at a time across all rows, so the rows it gathers (one slab) stay resident
// in L2 while the sparse matrix streams.  Column reductions are two-stage with a fixed order
// (deterministic run to run) and always accumulate in FP64.
//
// Precision.  SSP_PRECISION_FP64 runs the whole iteration in FP64.  SSP_PRECISION_MIXED runs FP64
// iterative refinement around FP32 inner PCG solves: the inner SpMM, triangular solves and vector
// updates read and write FP32 (half the bytes of every gather and stream), the inner dot products
// accumulate in FP64, and after each inner solve the true residual b - A x is recomputed with the FP64
// matrix and FP64 x, so the stopping rule is checked on the same FP64 residual as in the FP64 mode.
// An inner solve stops at a fixed relative reduction (or at half the outer threshold); once a round
// fails to contract the FP64 residual by a large factor, the remaining rounds use an FP64 inner solve
// that goes straight to the outer threshold.
#include <algorithm>
#include <cmath>
#include <cstdlib>

#include <functional>
#include <optional>
#include <type_traits>

#include "ssp_internal.cuh"

namespace ssp {

constexpr int TILE = SSP_TILE;    // columns per tile
constexpr int RED_BLOCKS = 6;     // ... resident per SM: one wave of them is the grid
constexpr int RED_THREADS = 256;  // column reductions: (256 / TILE) row lanes x TILE columns

// mixed precision: relative reduction asked of one FP32 inner solve, and the round limit
constexpr double MIXED_INNER_REDUCTION = 1e-4;
constexpr int MIXED_MAX_ROUNDS = 40;
// a round whose FP64 residual shrinks by less than this factor (max over columns) switches the remaining
// rounds to FP64 inner solves
constexpr double MIXED_MIN_CONTRACTION = 1e-2;
// FP32 rounds after the first may take at most this many times the first round's iterations (at least
// MIXED_MIN_ROUND_ITERS); on ill-conditioned systems the FP32 recurrence stalls short of its target, and a
// round that runs into the cap hands the rest to FP64
constexpr int MIXED_ROUND_ITER_FACTOR = 2;
constexpr int MIXED_MIN_ROUND_ITERS = 20;
// the first FP32 round may take at most max_iters / MIXED_FIRST_ROUND_DIV iterations (at least
// MIXED_MIN_ROUND_ITERS): an FP32 recurrence that stalls above its target (3-D grid, n = 64^3, weights over
// six decades: still at relative residual 0.26 after 400 iterations) then leaves the rest to FP64 rounds
constexpr int MIXED_FIRST_ROUND_DIV = 4;

__host__ __device__ __forceinline__ int64_t tm_off(int64_t n, int64_t r, int64_t c) { return tile_off(n, r, c); }

// ---------------------------------------------------------------- layout conversion
__global__ void k_rm_to_tm(int64_t n, int32_t k, int64_t ldr, const double* __restrict__ src, double* __restrict__ dst,
                           int64_t ld) {
    const int64_t total = n * ld;
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < total; i += (int64_t)gridDim.x * blockDim.x) {
        const int64_t t = i / (n * TILE), rem = i - t * n * TILE, r = rem / TILE, c = t * TILE + (rem % TILE);
        dst[i] = c < k ? src[r * ldr + c] : 0.0;
    }
}
__global__ void k_tm_to_rm(int64_t n, int32_t k, const double* __restrict__ src, double* __restrict__ dst, int64_t ldr) {
    const int64_t total = n * (int64_t)k;
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < total; i += (int64_t)gridDim.x * blockDim.x) {
        const int64_t r = i / k, c = i - r * k;
        dst[r * ldr + c] = src[tm_off(n, r, c)];
    }
}

void rowmajor_to_tiles(Context& C, int64_t n, int32_t k, int64_t ldr, const double* src, double* dst) {
    const int64_t ld = ((int64_t)k + TILE - 1) / TILE * TILE;
    k_rm_to_tm<<<grid_for(n * ld, 256, 148 * 16), 256, 0, C.stream>>>(n, k, ldr, src, dst, ld);
    SSP_CHECK_LAUNCH();
    C.kernels_launched++;
}
void tiles_to_rowmajor(Context& C, int64_t n, int32_t k, const double* src, double* dst, int64_t ldr) {
    k_tm_to_rm<<<grid_for(n * (int64_t)k, 256, 148 * 16), 256, 0, C.stream>>>(n, k, src, dst, ldr);
    SSP_CHECK_LAUNCH();
    C.kernels_launched++;
}

// ---------------------------------------------------------------- segments (several graphs in one solve)
// A batch of graphs is solved as the disjoint union of their Laplacians: rows [row0_s, row0_{s+1}) belong to
// segment s, which owns columns [0, k_s) of the n x k block (the rest of its columns stay zero and inactive).
// Every per-column scalar (norms, thresholds, alpha, beta, activity) is per (segment, column), at index
// s * ld + c, so each graph's iterates are its own; reductions use blocks that never straddle two segments.
// A single graph is one segment with null tables, and every kernel then does exactly what it did before.
struct SegDev {
    int32_t nseg = 1;
    const int32_t* rowseg = nullptr;    // [n] segment of each row
    const int32_t* kseg = nullptr;      // [nseg] columns of each segment
    const int64_t* segrows = nullptr;   // [nseg] rows of each segment
    const int64_t* blk_row = nullptr;   // [nparts + 1] row boundaries of the reduction blocks
    const int32_t* blk_seg = nullptr;   // [nparts] segment of each reduction block
    const int32_t* part_start = nullptr;  // [nseg + 1] first reduction block of each segment
};
__device__ __forceinline__ int64_t seg_of_row(const SegDev& G, int64_t row) { return G.rowseg ? G.rowseg[row] : 0; }
// rows of reduction block blockIdx.x and the state offset (segment * ld) of its segment
__device__ __forceinline__ void red_block(const SegDev& G, int64_t n, int64_t rows_per_blk, int64_t ld, int64_t& r0,
                                          int64_t& r1, int64_t& sbase) {
    if (G.blk_row) {
        r0 = G.blk_row[blockIdx.x];
        r1 = G.blk_row[blockIdx.x + 1];
        sbase = (int64_t)G.blk_seg[blockIdx.x] * ld;
    } else {
        r0 = (int64_t)blockIdx.x * rows_per_blk;
        r1 = min(n, r0 + rows_per_blk);
        sbase = 0;
    }
}

// Rows of converged graphs (several graphs at once): act[s * ntiles + t] says whether graph s still has an
// active column in tile t; the SpMM and the triangular solves skip the rows of inactive (graph, tile) pairs,
// whose values no active column reads (alpha is 0 there).  A null act (one graph) skips nothing.
struct RowAct {
    const int32_t* act = nullptr;
    const int32_t* rowseg = nullptr;  // graph of each vertex
    int32_t ntiles = 0;
};
__device__ __forceinline__ bool row_on(const RowAct& A, int64_t vertex, int64_t tile) {
    return !A.act || A.act[(int64_t)A.rowseg[vertex] * A.ntiles + tile];
}
__global__ void k_seg_tile_active(int32_t nseg, int32_t ntiles, int64_t ld, const int32_t* __restrict__ active,
                                  int32_t* __restrict__ act) {
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < (int64_t)nseg * ntiles;
         i += (int64_t)gridDim.x * blockDim.x) {
        const int64_t sg = i / ntiles, t = i - sg * ntiles;
        int32_t a = 0;
        for (int c = 0; c < TILE; c++) a |= active[sg * ld + t * TILE + c];
        act[i] = a;
    }
}

// ---------------------------------------------------------------- column reductions
enum ColOp { OP_SUM = 0, OP_DOT = 1, OP_SQ = 2, OP_SQDIFF_CENTERED = 3 };

// 16 bytes of a tile's row: a thread of the vector kernels below has these columns of every RROWS<T>-th row of its block.
template <class T>
struct alignas(16) Vec {
    static constexpr int V = 16 / sizeof(T);
    T v[V];
};
template <class T>
__device__ __forceinline__ Vec<T> vec_at(const T* p) {
    return *reinterpret_cast<const Vec<T>*>(p);
}
template <class T>
__device__ __forceinline__ void vec_to(T* p, const Vec<T>& x) {
    *reinterpret_cast<Vec<T>*>(p) = x;
}
template <class T>
constexpr int RROWS = RED_THREADS * Vec<T>::V / TILE;

// the block's per-column sums of acc (thread: columns c ..), row lanes in order
template <class T>
__device__ __forceinline__ void block_part(const double (&acc)[Vec<T>::V], int64_t t, int64_t ld, double* part) {
    __shared__ double s[RED_THREADS * Vec<T>::V];
#pragma unroll
    for (int u = 0; u < Vec<T>::V; u++) s[threadIdx.x * Vec<T>::V + u] = acc[u];
    __syncthreads();
    if (threadIdx.x < TILE) {
        double tt = s[threadIdx.x];
        for (int i = 1; i < RROWS<T>; i++) tt += s[i * TILE + threadIdx.x];
        part[(int64_t)blockIdx.x * ld + t * TILE + threadIdx.x] = tt;
    }
}

// Grid (nparts, ntiles); part[blk][col].  These stream their operands once, so the bound is DRAM: 16-byte loads, two rows of a
// thread in flight, and a grid of one wave (148 x RED_BLOCKS; a few blocks more, as before, ran alone afterwards).
// Measured on B200 with a lane per value -> here, over 1185-1194 columns: r.z at ER n = 250,000 FP64 868 -> 671 us (7.1 TB/s),
// at n = 229,373 FP32 553 -> 339 (6.4); r -= alpha q 1.29 -> 1.19 ms (6.0) and 653 -> 600 us (5.4).  The rows of a block stay
// contiguous: taken in turn by all blocks, r -= alpha q took 1.31 ms.
template <int OP, class T>
__global__ void __launch_bounds__(RED_THREADS, RED_BLOCKS) k_colred_partial(int64_t n, const T* __restrict__ a,
                                                                const T* __restrict__ b,
                                                                const double* __restrict__ mean, int64_t rows_per_blk,
                                                                int64_t ld, double* __restrict__ part, SegDev G) {
    constexpr int V = Vec<T>::V;
    const int64_t t = blockIdx.y;
    const int c = threadIdx.x * V % TILE, rl = threadIdx.x * V / TILE;
    int64_t r0, r1, sb;
    red_block(G, n, rows_per_blk, ld, r0, r1, sb);
    const T* at = a + t * n * TILE + c;
    const T* bt = b ? b + t * n * TILE + c : nullptr;
    double mu[V], acc[V];
#pragma unroll
    for (int u = 0; u < V; u++) {
        mu[u] = (OP == OP_SQDIFF_CENTERED) ? mean[sb + t * TILE + c + u] : 0.0;
        acc[u] = 0.0;
    }
#pragma unroll 2
    for (int64_t r = r0 + rl; r < r1; r += RROWS<T>) {
        const Vec<T> x = vec_at(at + r * TILE);
        Vec<T> y;
        if (OP == OP_DOT || OP == OP_SQDIFF_CENTERED) y = vec_at(bt + r * TILE);
#pragma unroll
        for (int u = 0; u < V; u++) {
            if (OP == OP_SUM) acc[u] += (double)x.v[u];
            else if (OP == OP_DOT) acc[u] += (double)x.v[u] * (double)y.v[u];
            else if (OP == OP_SQ) acc[u] += (double)x.v[u] * (double)x.v[u];
            else {
                const double d = ((double)x.v[u] - mu[u]) - (double)y.v[u];  // (Y - mean) - A x
                acc[u] += d * d;
            }
        }
    }
    block_part<T>(acc, t, ld, part);
}

// out[c] = sum over parts of part[i][c]: a block per 32 columns, warp w sums the parts i = w (mod FIN_WARPS) two
// at a time, then the warps' sums are added in warp order (fixed order: deterministic).  Hundreds of parts per
// column (the SpMM's p.q partials) are then 16-way parallel instead of one thread's dependent chain.
constexpr int FIN_WARPS = 16;
// With segments, out[s * ld + c] sums the parts of segment s's blocks, in the same order.
__global__ void __launch_bounds__(FIN_WARPS * 32) k_colred_final(int64_t ld, int nparts, const double* __restrict__ part,
                                                                  double* __restrict__ out, SegDev G) {
    __shared__ double s[FIN_WARPS][32];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const int64_t o = (int64_t)blockIdx.x * 32 + lane;
    const int64_t seg = o / ld, c = o - seg * ld;
    const bool in = o < (int64_t)G.nseg * ld;
    const int p0 = G.part_start && in ? G.part_start[seg] : 0;
    const int np = G.part_start && in ? G.part_start[seg + 1] - p0 : nparts;
    double a0 = 0.0, a1 = 0.0;
    if (in) {
        int i = w;
        for (; i + FIN_WARPS < np; i += 2 * FIN_WARPS) {
            a0 += part[(int64_t)(p0 + i) * ld + c];
            a1 += part[(int64_t)(p0 + i + FIN_WARPS) * ld + c];
        }
        if (i < np) a0 += part[(int64_t)(p0 + i) * ld + c];
    }
    s[w][lane] = a0 + a1;
    __syncthreads();
    if (w == 0 && in) {
        double t = 0.0;
        for (int j = 0; j < FIN_WARPS; j++) t += s[j][lane];
        out[o] = t;
    }
}
static void colred_final(Context& C, int64_t ld, int nparts, const double* part, double* out,
                         const SegDev& G = SegDev()) {
    k_colred_final<<<(unsigned)ceil_div<int64_t>((int64_t)G.nseg * ld, 32), FIN_WARPS * 32, 0, C.stream>>>(
        ld, nparts, part, out, G);
}

struct Reducer {
    Context* C;
    int64_t n, ld;
    int nparts;
    int64_t rows_per_blk;
    double* part;
    SegDev G;  // segment tables (the block tables are filled in by init when there are several segments)
    // row0: nseg + 1 segment row starts on the host (empty: one segment); G's rowseg/kseg/segrows are the
    // caller's
    void init(Context& c, int64_t n_, int64_t ld_, const char* tag = "pcg_red_part", const SegDev& segs = SegDev(),
              const std::vector<int64_t>* row0 = nullptr) {
        C = &c;
        n = n_;
        ld = ld_;
        G = segs;
        const int64_t ntiles = ld / TILE;
        int64_t target = std::max<int64_t>(8, std::min<int64_t>(148 * RED_BLOCKS / std::max<int64_t>(1, ntiles), 1024));
        rows_per_blk = std::max<int64_t>(RED_THREADS / TILE, ceil_div<int64_t>(n, target));
        if (G.nseg <= 1 || !row0) {
            nparts = (int)ceil_div<int64_t>(n, rows_per_blk);
        } else {
            // blocks of at most rows_per_blk rows inside each segment
            std::vector<int64_t> brow;
            std::vector<int32_t> bseg, pstart;
            for (int32_t sg = 0; sg < G.nseg; sg++) {
                pstart.push_back((int32_t)bseg.size());
                for (int64_t r = (*row0)[sg]; r < (*row0)[sg + 1]; r += rows_per_blk) {
                    brow.push_back(r);
                    bseg.push_back(sg);
                }
            }
            pstart.push_back((int32_t)bseg.size());
            brow.push_back(n);
            nparts = (int)bseg.size();
            int64_t* d_brow = c.ws.get_t<int64_t>(std::string(tag) + "_brow", brow.size());
            int32_t* d_bseg = c.ws.get_t<int32_t>(std::string(tag) + "_bseg", bseg.size() + 1);
            int32_t* d_pst = c.ws.get_t<int32_t>(std::string(tag) + "_pstart", pstart.size());
            SSP_CUDA(cudaMemcpyAsync(d_brow, brow.data(), sizeof(int64_t) * brow.size(), cudaMemcpyHostToDevice,
                                     c.stream));
            SSP_CUDA(cudaMemcpyAsync(d_bseg, bseg.data(), sizeof(int32_t) * bseg.size(), cudaMemcpyHostToDevice,
                                     c.stream));
            SSP_CUDA(cudaMemcpyAsync(d_pst, pstart.data(), sizeof(int32_t) * pstart.size(), cudaMemcpyHostToDevice,
                                     c.stream));
            SSP_CUDA(cudaStreamSynchronize(c.stream));
            G.blk_row = d_brow;
            G.blk_seg = d_bseg;
            G.part_start = d_pst;
        }
        part = c.ws.get_t<double>(tag, (size_t)nparts * ld);
    }
    template <int OP, class T>
    void run(const T* a, const T* b, double* out, const double* mean = nullptr) {
        dim3 grid((unsigned)nparts, (unsigned)(ld / TILE));
        k_colred_partial<OP, T><<<grid, RED_THREADS, 0, C->stream>>>(n, a, b, mean, rows_per_blk, ld, part, G);
        colred_final(*C, ld, nparts, part, out, G);
        SSP_CHECK_LAUNCH();
        C->kernels_launched += 2;
    }
    void finish(double* out) {
        colred_final(*C, ld, nparts, part, out, G);
        SSP_CHECK_LAUNCH();
        C->kernels_launched++;
    }
};

// ---------------------------------------------------------------- elementwise (grid.y = tile)
// r = Y - mean(Y) over each segment's rows for its columns (0 elsewhere), x = 0, mean per (segment, column)
__global__ void k_center(int64_t n, int32_t k, int64_t ld, const double* __restrict__ Y,
                         const double* __restrict__ colsum, double* __restrict__ r, double* __restrict__ x,
                         double* __restrict__ mean, SegDev G) {
    const int64_t t = blockIdx.y;
    const int64_t cnt = n * TILE;
    if (blockIdx.x == 0 && threadIdx.x < TILE)
        for (int32_t sg = 0; sg < G.nseg; sg++) {
            const int64_t c = t * TILE + threadIdx.x;
            const int32_t kk = G.kseg ? G.kseg[sg] : k;
            const int64_t nr = G.segrows ? G.segrows[sg] : n;
            mean[sg * ld + c] = c < kk ? colsum[sg * ld + c] / (double)nr : 0.0;
        }
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < cnt; i += (int64_t)gridDim.x * blockDim.x) {
        const int64_t c = t * TILE + (i % TILE);
        const int64_t o = t * cnt + i;
        const int64_t sg = seg_of_row(G, i / TILE);
        const int32_t kk = G.kseg ? G.kseg[sg] : k;
        const int64_t nr = G.segrows ? G.segrows[sg] : n;
        const double mu = c < kk ? colsum[sg * ld + c] / (double)nr : 0.0;
        r[o] = c < kk ? Y[o] - mu : 0.0;
        x[o] = 0.0;
    }
}

// r -= alpha q ; partial ||r||^2 per column (FP64 accumulation).  The matching x += alpha p is deferred to
// the next p update (k_update_xp), which reads p anyway, or to k_axpy_x after the last iteration: x gets
// the same additions in the same order, one n x k stream fewer per iteration.
template <class T>
__global__ void __launch_bounds__(RED_THREADS, RED_BLOCKS) k_axpy_r_rr(int64_t n, const double* __restrict__ alpha,
                                                           const T* __restrict__ q, T* __restrict__ r,
                                                           int64_t rows_per_blk, int64_t ld, double* __restrict__ part,
                                                           SegDev G) {
    constexpr int V = Vec<T>::V;
    const int64_t t = blockIdx.y;
    const int c = threadIdx.x * V % TILE, rl = threadIdx.x * V / TILE;
    int64_t r0, r1, sb;
    red_block(G, n, rows_per_blk, ld, r0, r1, sb);
    double a64[V], acc[V];
    bool any = false;
#pragma unroll
    for (int u = 0; u < V; u++) {
        a64[u] = alpha[sb + t * TILE + c + u];
        any |= a64[u] != 0.0;
        acc[u] = 0.0;
    }
    const int64_t base = t * n * TILE + c;
    auto row_done = [&](Vec<T> rv, const Vec<T>& qv, int64_t o) {
        if (any) {
#pragma unroll
            for (int u = 0; u < V; u++)
                if (a64[u] != 0.0) rv.v[u] -= (T)a64[u] * qv.v[u];
            vec_to(r + o, rv);
        }
#pragma unroll
        for (int u = 0; u < V; u++) acc[u] += (double)rv.v[u] * (double)rv.v[u];
    };
    int64_t row = r0 + rl;
    for (; row + RROWS<T> < r1; row += 2 * RROWS<T>) {  // both rows' loads before the first store
        const int64_t o0 = base + row * TILE, o1 = o0 + RROWS<T> * TILE;
        const Vec<T> ra = vec_at(r + o0), rb = vec_at(r + o1);
        Vec<T> qa = {}, qb = {};
        if (any) {
            qa = vec_at(q + o0);
            qb = vec_at(q + o1);
        }
        row_done(ra, qa, o0);
        row_done(rb, qb, o1);
    }
    if (row < r1) {
        const int64_t o = base + row * TILE;
        const Vec<T> ra = vec_at(r + o);
        row_done(ra, any ? vec_at(q + o) : Vec<T>{}, o);
    }
    block_part<T>(acc, t, ld, part);
}

// x += alpha p (the previous step's alpha and p), then p = z + beta p.  Five streams in 16-byte pieces (FP32 5.4 GB:
// 1.09 -> 0.94 ms; FP64 stays at 6.7 TB/s)
template <class T>
__global__ void k_update_xp(int64_t n, int64_t ld, const double* __restrict__ alpha, const double* __restrict__ beta,
                            const T* __restrict__ z, T* __restrict__ p, T* __restrict__ x, SegDev G) {
    constexpr int V = Vec<T>::V;
    const int64_t t = blockIdx.y;
    const int64_t cnt = n * TILE;
    for (int64_t i = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) * V; i < cnt;
         i += (int64_t)gridDim.x * blockDim.x * V) {
        const int64_t o = t * cnt + i;
        const int64_t c = seg_of_row(G, i / TILE) * ld + t * TILE + (i % TILE);
        double a64[V];
        bool any = false;
#pragma unroll
        for (int u = 0; u < V; u++) {
            a64[u] = alpha[c + u];
            any |= a64[u] != 0.0;
        }
        Vec<T> pv = vec_at(p + o), zv = vec_at(z + o);
        if (any) {
            Vec<T> xv = vec_at(x + o);
#pragma unroll
            for (int u = 0; u < V; u++)
                if (a64[u] != 0.0) xv.v[u] += (T)a64[u] * pv.v[u];
            vec_to(x + o, xv);
        }
#pragma unroll
        for (int u = 0; u < V; u++) pv.v[u] = zv.v[u] + (T)beta[c + u] * pv.v[u];
        vec_to(p + o, pv);
    }
}

// the last step's x += alpha p
template <class T>
__global__ void k_axpy_x(int64_t n, int64_t ld, const double* __restrict__ alpha, const T* __restrict__ p,
                         T* __restrict__ x, SegDev G) {
    const int64_t t = blockIdx.y;
    const int64_t cnt = n * TILE;
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < cnt; i += (int64_t)gridDim.x * blockDim.x) {
        const int64_t o = t * cnt + i;
        const double a64 = alpha[seg_of_row(G, i / TILE) * ld + t * TILE + (i % TILE)];
        if (a64 != 0.0) x[o] += (T)a64 * p[o];
    }
}

// ---------------------------------------------------------------- mixed-precision helpers
__global__ void k_d2f(int64_t count, const double* __restrict__ src, float* __restrict__ dst) {
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < count; i += (int64_t)gridDim.x * blockDim.x)
        dst[i] = (float)src[i];
}
__global__ void k_f2d(int64_t count, const float* __restrict__ src, double* __restrict__ dst) {
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < count; i += (int64_t)gridDim.x * blockDim.x)
        dst[i] = (double)src[i];
}

__global__ void k_ent_f32(int64_t count, const FactorEnt<double>* __restrict__ src, FactorEnt<float>* __restrict__ dst) {
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < count; i += (int64_t)gridDim.x * blockDim.x) {
        const FactorEnt<double> e = src[i];
        dst[i] = FactorEnt<float>{(float)e.v, e.idx};
    }
}

// inner right-hand side: the FP64 residual of the columns still active, rounded to T; zero elsewhere
// (runs in place when T is double)
template <class T>
__global__ void k_rhs_masked(int64_t n, int64_t ld, const double* r64, const int32_t* __restrict__ active, T* rin,
                             SegDev G) {
    const int64_t t = blockIdx.y;
    const int64_t cnt = n * TILE;
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < cnt; i += (int64_t)gridDim.x * blockDim.x) {
        const int64_t o = t * cnt + i;
        rin[o] = active[seg_of_row(G, i / TILE) * ld + t * TILE + (i % TILE)] ? (T)r64[o] : (T)0;
    }
}

template <class T>
__global__ void k_add_into(int64_t count, const T* __restrict__ e, double* __restrict__ x) {
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < count; i += (int64_t)gridDim.x * blockDim.x)
        x[i] += (double)e[i];
}

// r = (Y - mean) - q with partial ||r||^2 per column: the true FP64 residual after a refinement round
__global__ void __launch_bounds__(RED_THREADS, RED_BLOCKS) k_true_resid(int64_t n, int32_t k, const double* __restrict__ Y,
                                                            const double* __restrict__ mean,
                                                            const double* __restrict__ q, double* __restrict__ r,
                                                            int64_t rows_per_blk, int64_t ld, double* __restrict__ part,
                                                            SegDev G) {
    constexpr int V = Vec<double>::V;
    const int64_t t = blockIdx.y;
    const int c = threadIdx.x * V % TILE, rl = threadIdx.x * V / TILE;
    int64_t r0, r1, sb;
    red_block(G, n, rows_per_blk, ld, r0, r1, sb);
    const int64_t col = t * TILE + c;
    if (G.kseg) k = G.kseg[sb / ld];
    double mu[V], acc[V];
#pragma unroll
    for (int u = 0; u < V; u++) {
        mu[u] = mean[sb + col + u];
        acc[u] = 0.0;
    }
    const int64_t base = t * n * TILE + c;
#pragma unroll 2
    for (int64_t row = r0 + rl; row < r1; row += RROWS<double>) {
        const int64_t o = base + row * TILE;
        const Vec<double> yv = vec_at(Y + o), qv = vec_at(q + o);
        Vec<double> rv;
#pragma unroll
        for (int u = 0; u < V; u++) {
            rv.v[u] = col + u < k ? (yv.v[u] - mu[u]) - qv.v[u] : 0.0;
            acc[u] += rv.v[u] * rv.v[u];
        }
        vec_to(r + o, rv);
    }
    block_part<double>(acc, t, ld, part);
}

// ---------------------------------------------------------------- per-column scalars
struct ColState {
    double* bnorm2;
    double* thr;
    double* rz;
    double* rz_new;
    double* pq;
    double* rr;
    double* alpha;
    double* beta;
    int32_t* active;
    int32_t* iters;
    int64_t* nactive;
};

static ColState make_colstate(Context& C, int64_t ld, const std::string& tag) {
    double* v = C.ws.get_t<double>(tag + "_cols", 8 * ld);
    int32_t* iv = C.ws.get_t<int32_t>(tag + "_coli", 2 * ld);
    int64_t* na = C.ws.get_t<int64_t>(tag + "_nactive", 1);
    return ColState{v, v + ld, v + 2 * ld, v + 3 * ld, v + 4 * ld, v + 5 * ld, v + 6 * ld, v + 7 * ld, iv, iv + ld, na};
}

// state entries c = segment * ld + column; a column past its segment's k_s is inactive
__global__ void k_cols_init(int64_t ld, int32_t k, double tol, double abs_tol, ColState S, SegDev G) {
    for (int64_t c = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; c < (int64_t)G.nseg * ld;
         c += (int64_t)gridDim.x * blockDim.x) {
        const int32_t kk = G.kseg ? G.kseg[c / ld] : k;
        double bn = sqrt(S.bnorm2[c]);
        double thr = tol * bn;
        if (abs_tol > thr) thr = abs_tol;
        S.thr[c] = thr;
        S.rr[c] = S.bnorm2[c];
        int act = (c % ld < kk) && (bn > thr);
        S.active[c] = act;
        S.iters[c] = 0;
        S.alpha[c] = 0.0;
        S.beta[c] = 0.0;
        if (act) atomicAdd((unsigned long long*)S.nactive, 1ull);
    }
}

// inner solve of a refinement round: stop at a relative reduction `reduction` of its right-hand side, or
// once below half the outer threshold of the column (no point solving past what the outer test needs)
__global__ void k_cols_init_inner(int64_t ld, int32_t k, double reduction, const double* __restrict__ thr_out,
                                  ColState S, SegDev G) {
    for (int64_t c = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; c < (int64_t)G.nseg * ld;
         c += (int64_t)gridDim.x * blockDim.x) {
        const int32_t kk = G.kseg ? G.kseg[c / ld] : k;
        const double bn = sqrt(S.bnorm2[c]);
        double thr = reduction * bn;
        const double half_out = 0.5 * thr_out[c];
        if (half_out > thr) thr = half_out;
        S.thr[c] = thr;
        S.rr[c] = S.bnorm2[c];
        const int act = (c % ld < kk) && (bn > thr);
        S.active[c] = act;
        S.iters[c] = 0;
        S.alpha[c] = 0.0;
        S.beta[c] = 0.0;
        if (act) atomicAdd((unsigned long long*)S.nactive, 1ull);
    }
}

__global__ void k_cols_alpha(int64_t cnt, ColState S) {
    for (int64_t c = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; c < cnt; c += (int64_t)gridDim.x * blockDim.x)
        S.alpha[c] = S.active[c] ? S.rz[c] / S.pq[c] : 0.0;
}

__global__ void k_cols_check(int64_t cnt, int32_t it, ColState S) {
    for (int64_t c = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; c < cnt; c += (int64_t)gridDim.x * blockDim.x) {
        if (!S.active[c]) continue;
        S.iters[c] = it;
        if (sqrt(S.rr[c]) <= S.thr[c]) S.active[c] = 0;
        else atomicAdd((unsigned long long*)S.nactive, 1ull);
    }
}

// One iteration's entry of the residual history: per segment (block) the largest ||r|| / ||b|| of its columns, then the
// columns still active.  Kept on the device so that a probe's iterations are launched without waiting: reading them back
// after each took 60-80 us an iteration.
__global__ void __launch_bounds__(32) k_hist(int64_t ld, ColState S, double* __restrict__ hist) {
    const int64_t sg = blockIdx.x;
    double m = 0.0;
    for (int64_t j = threadIdx.x; j < ld; j += 32) {
        const double b = S.bnorm2[sg * ld + j];
        if (b > 0) {
            const double q = sqrt(S.rr[sg * ld + j] / b);
            if (m < q) m = q;
        }
    }
    for (int o = 16; o > 0; o >>= 1) {
        const double q = __shfl_xor_sync(0xffffffffu, m, o);
        if (m < q) m = q;
    }
    if (threadIdx.x) return;
    hist[sg] = m;
    if (sg == 0) hist[gridDim.x] = (double)*S.nactive;
}

__global__ void k_cols_beta(int64_t cnt, ColState S) {
    for (int64_t c = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; c < cnt; c += (int64_t)gridDim.x * blockDim.x) {
        double b = 0.0;
        if (S.active[c]) b = S.rz_new[c] / S.rz[c];
        S.beta[c] = b;
        S.rz[c] = S.rz_new[c];
    }
}

// outer test of a refinement round on the true residual: adds the round's inner iterations to the
// column's count, deactivates converged columns, and records the largest residual ratio new/old
__global__ void k_cols_outer(int64_t cnt, const int32_t* __restrict__ inner_iters, const double* __restrict__ rr_new,
                             ColState S, double* __restrict__ worst_ratio) {
    for (int64_t c = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; c < cnt; c += (int64_t)gridDim.x * blockDim.x) {
        if (!S.active[c]) continue;
        S.iters[c] += inner_iters[c];
        const double before = S.rr[c], after = rr_new[c];
        S.rr[c] = after;
        if (sqrt(after) <= S.thr[c]) {
            S.active[c] = 0;
        } else {
            atomicAdd((unsigned long long*)S.nactive, 1ull);
            const double ratio = before > 0 ? sqrt(after / before) : 1.0;
            // ratios are non-negative: their IEEE bit patterns order like the values
            atomicMax((unsigned long long*)worst_ratio, (unsigned long long)__double_as_longlong(ratio));
        }
    }
}

// ---------------------------------------------------------------- the iteration loop on the device
// The PCG iterations after the first run as the body of a CUDA-graph WHILE node: the body advances the
// iteration counter on the device, runs the convergence check, and k_loop_ctl keeps the loop going only while
// some column is active and fewer than max_iters iterations have run, so the loop ends by itself without a
// host round trip per iteration.
__global__ void k_it_set(int32_t* it, int32_t v) { *it = v; }
__global__ void k_it_next(int32_t* it) { *it += 1; }

__global__ void k_cols_check_at(int64_t cnt, const int32_t* __restrict__ it, ColState S) {
    const int32_t i = *it;
    for (int64_t c = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; c < cnt; c += (int64_t)gridDim.x * blockDim.x) {
        if (!S.active[c]) continue;
        S.iters[c] = i;
        if (sqrt(S.rr[c]) <= S.thr[c]) S.active[c] = 0;
        else atomicAdd((unsigned long long*)S.nactive, 1ull);
    }
}

__global__ void k_loop_ctl(cudaGraphConditionalHandle h, const int64_t* __restrict__ nactive,
                           const int32_t* __restrict__ it, int32_t max_iters) {
    cudaGraphSetConditional(h, (*nactive > 0 && *it < max_iters) ? 1u : 0u);
}

struct LoopGraph {
    cudaGraph_t graph = nullptr;
    cudaGraphExec_t exec = nullptr;
    ~LoopGraph() {
        if (exec) cudaGraphExecDestroy(exec);
        if (graph) cudaGraphDestroy(graph);
    }
};

// ---------------------------------------------------------------- SpMM and triangular solves
// Warp per row; lane = slot * W + column, W = the columns handled (TILE, or 8 when at most 8 are real).
// ---------------------------------------------------------------- chunked gather (SpMM-shaped work)
// A chunk is a run of consecutive stored rows with at most CHUNK_CAP entries and CHUNK_ROWS rows (or
// one longer row).  Each warp owns whole chunks: it stages the chunk's (index, value) pairs in its own
// shared-memory slice with coalesced streaming loads (the matrix is read once per tile and should not
// evict the gathered slab from L2), then every (row, column) lane pair sums its row with independent
// gathers from the tile slab.  Warps never wait for each other.  The Laplacian product (k_spmm) works on such
// chunks too; the modes here are the forward solve, the backward solve, and the forward solve of the last level with that
// level's backward step.
enum { M_FWD = 1, M_BWD = 2, M_FWD_LAST = 4 };
constexpr int CH_THREADS = 256;
constexpr int CH_WARPS = CH_THREADS / 32;
constexpr int MINB_FWD = 6, MINB_BWD = 5, MINB_WIDE64 = 4;

template <int MODE, class T>
__device__ __forceinline__ void chunk_epilogue(T* out, const T* aux, int64_t toff, int64_t v, int col, T acc,
                                               const T* dlast) {
    const int64_t o = toff + v * TILE + col;
    if (MODE == M_FWD) {
        out[o] = aux[o] - acc;
    } else if (MODE == M_FWD_LAST) {
        // the forward value, then the backward solve's step for a row with an empty column
        const T yu = aux[o] - acc;
        const T d = dlast[v];
        out[o] = (d != (T)0 ? yu / d : yu) - (T)0;
    } else {
        const T d = aux[v];
        const T yu = out[o];
        out[o] = (d != (T)0 ? yu / d : yu) - acc;
    }
}

// two columns
template <class T>
struct ColPair;
template <>
struct ColPair<double> {
    using V = double2;
};
template <>
struct ColPair<float> {
    using V = float2;
};

// the epilogue of two columns
template <int MODE, class T, class V>
__device__ __forceinline__ void chunk_epilogue2(T* out, const T* aux, int64_t toff, int64_t v, int col, V acc,
                                                const T* dlast) {
    const int64_t o = toff + v * TILE + col;
    V y = *reinterpret_cast<const V*>((MODE == M_BWD ? out : aux) + o);
    if (MODE != M_BWD) y = {y.x - acc.x, y.y - acc.y};
    if (MODE != M_FWD) {
        const T d = MODE == M_BWD ? aux[v] : dlast[v];
        if (d != (T)0) y = {y.x / d, y.y / d};
        if (MODE == M_BWD) y = {y.x - acc.x, y.y - acc.y};
    }
    *reinterpret_cast<V*>(out + o) = y;
}

// Row sums of the triangular solves.  A row's entries are summed in segments of ROW_SEG: entry i of a segment goes to
// accumulator i mod 4 (in entry order), the four are combined as (a0 + a1) + (a2 + a3), and the segments' sums are
// added in order.  Every launch width forms a row this way -- one lane per (row, column), or the entry slots of a warp
// for a row longer than a chunk -- so the values do not depend on it.
constexpr int ROW_SEG = 64;

// one lane, entries [q0, q1) of staged or global index and value arrays.  The last entries of a row are loaded under
// predicates, all at once: a row of three entries costs one gather latency, not three.
template <class T, class I>
__device__ __forceinline__ T row_sum_lane(const int32_t* si, const T* sv, I q0, I q1, const T* xt) {
    T tot = 0;
    for (I s = q0; s < q1; s += ROW_SEG) {
        const I e = min(s + (I)ROW_SEG, q1);
        T a[4] = {0, 0, 0, 0};
        I q = s;
        for (; q + 3 < e; q += 4) {
#pragma unroll
            for (int u = 0; u < 4; u++) a[u] += sv[q + u] * xt[(int64_t)si[q + u] * TILE];
        }
        if (q < e) {
            T x[3];
#pragma unroll
            for (int u = 0; u < 3; u++) x[u] = q + u < e ? xt[(int64_t)si[q + u] * TILE] : (T)0;
#pragma unroll
            for (int u = 0; u < 3; u++)
                if (q + u < e) a[u] += sv[q + u] * x[u];
        }
        tot += (a[0] + a[1]) + (a[2] + a[3]);
    }
    return tot;
}

// The same for two columns of a lane, half the load instructions for a row.  On B200 an FP32 application at ER n =
// 229,373, 1185 columns: the truncated level 1.28 -> 0.92 ms, the backward levels 0.79 -> 0.56.  FP64 (four blocks per SM: at
// five and six the 16-byte gathers spill), ER n = 250,000, 1194 columns: 3.10 -> 2.95 ms in all.
template <class T>
__device__ __forceinline__ typename ColPair<T>::V row_sum_lane2(const int32_t* si, const T* sv, int q0, int q1,
                                                                  const T* xt) {
    using V = typename ColPair<T>::V;
    V tot = {0, 0};
    auto at = [&](int q) { return *reinterpret_cast<const V*>(xt + (int64_t)si[q] * TILE); };
    for (int s = q0; s < q1; s += ROW_SEG) {
        const int e = min(s + ROW_SEG, q1);
        V a[4] = {{0, 0}, {0, 0}, {0, 0}, {0, 0}};
        auto add = [&](int u, T v, const V& x) {
            a[u].x += v * x.x;
            a[u].y += v * x.y;
        };
        int q = s;
        for (; q + 3 < e; q += 4) {
            V x[4];
#pragma unroll
            for (int u = 0; u < 4; u++) x[u] = at(q + u);
#pragma unroll
            for (int u = 0; u < 4; u++) add(u, sv[q + u], x[u]);
        }
        if (q < e) {
            V x[3];
#pragma unroll
            for (int u = 0; u < 3; u++)
                if (q + u < e) x[u] = at(q + u);
#pragma unroll
            for (int u = 0; u < 3; u++)
                if (q + u < e) add(u, sv[q + u], x[u]);
        }
        tot.x += (a[0].x + a[1].x) + (a[2].x + a[3].x);
        tot.y += (a[0].y + a[1].y) + (a[2].y + a[3].y);
    }
    return tot;
}

// one segment [s, e) of staged entries by the 32 / W slots of a full warp (W = 8, 16 or 32); every lane of a column
// gets the sum
template <class T, int W>
__device__ __forceinline__ T seg_sum_slots(const int32_t* si, const T* sv, int s, int e, const T* xt, int slot) {
    constexpr int SLOTS = 32 / W, NA = 4 / SLOTS, U = NA == 1 ? 4 : 4 / NA;
    static_assert(SLOTS <= 4, "columns per row below 8");
    T a[NA];
#pragma unroll
    for (int j = 0; j < NA; j++) a[j] = 0;
    for (int q = s + slot; q < e; q += 4 * U) {
        T x[U * NA];
#pragma unroll
        for (int u = 0; u < U * NA; u++) {
            const int p = q + SLOTS * u;
            x[u] = p < e ? xt[(int64_t)si[p] * TILE] : (T)0;
        }
#pragma unroll
        for (int u = 0; u < U * NA; u++) {
            const int p = q + SLOTS * u;
            if (p < e) a[u % NA] += sv[p] * x[u];
        }
    }
#pragma unroll
    for (int o = W; o < 32; o <<= 1)
#pragma unroll
        for (int j = 0; j < NA; j++) a[j] += __shfl_xor_sync(0xffffffffu, a[j], o);
    if constexpr (NA == 4) return (a[0] + a[1]) + (a[2] + a[3]);
    else if constexpr (NA == 2) return a[0] + a[1];
    else return a[0];
}

// Grid: x over chunks, y over (tile, sub-tile): a tile's TILE columns are covered by nsub = TILE / W warps'
// column ranges (nsub = 1 for the full-width layout, or for the narrow one when only W columns are real).
// MINB: resident blocks per SM asked of the compiler, what each direction's own register choice gives (forward 6,
// backward 5; forcing six on the backward solve cost the preconditioner 7 %), or 4 at full width in FP64 (row_sum_lane2).
template <int MODE, class T, int W, int MINB>
__global__ void __launch_bounds__(CH_THREADS, MINB)
    k_chunked(int64_t n, const int32_t* __restrict__ cstart, int32_t nchunks, const int64_t* __restrict__ ptr,
              const int32_t* __restrict__ idx, const T* __restrict__ val, const int32_t* __restrict__ rowmap,
              const T* xsrc, T* out, const T* __restrict__ aux, int32_t kcols, int nsub,
              const T* __restrict__ dlast = nullptr, RowAct ra = RowAct()) {
    __shared__ int32_t s_idx[CH_WARPS][CHUNK_CAP];
    __shared__ T s_val[CH_WARPS][CHUNK_CAP];
    __shared__ int32_t s_ptr[CH_WARPS][CHUNK_ROWS + 1];
    __shared__ int32_t s_row[CH_WARPS][CHUNK_ROWS];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const int64_t t = blockIdx.y / nsub;
    const int c0 = (int)(blockIdx.y % nsub) * W;  // first column of this block's sub-tile
    const int64_t toff = t * n * TILE;
    const T* xt = xsrc + toff;
    int32_t* si = s_idx[w];
    T* sv = s_val[w];
    int32_t* sp = s_ptr[w];
    int32_t* sr = s_row[w];
    for (int32_t c = blockIdx.x * CH_WARPS + w; c < nchunks; c += gridDim.x * CH_WARPS) {
        const int32_t r0 = cstart[c], r1 = cstart[c + 1];
        const int64_t e0 = ptr[r0], e1 = ptr[r1];
        const int64_t ne = e1 - e0;
        if (ne <= CHUNK_CAP) {
            for (int64_t i = lane; i < ne; i += 32) {
                si[i] = __ldcs(idx + e0 + i);
                sv[i] = __ldcs(val + e0 + i);
            }
            // the chunk's row pointers and vertex ids staged together
            for (int32_t i = lane; i <= r1 - r0; i += 32) {
                sp[i] = (int32_t)(ptr[r0 + i] - e0);
                if (i < r1 - r0) sr[i] = rowmap[r0 + i];
            }
            __syncwarp();
            if constexpr (W == TILE) {
                // a lane has two columns of a row, a half-warp the row
                for (int32_t pr = lane; pr < (r1 - r0) * (W / 2); pr += 32) {
                    const int32_t rr = pr / (W / 2), col = pr % (W / 2) * 2;
                    const int64_t vrow = sr[rr];
                    if (!row_on(ra, vrow, t)) continue;
                    const int32_t q0 = sp[rr], q1 = t * TILE + col < kcols ? sp[rr + 1] : q0;
                    const auto sum = row_sum_lane2<T>(si, sv, q0, q1, xt + col);
                    chunk_epilogue2<MODE, T>(out, aux, toff, vrow, col, sum, dlast);
                }
                __syncwarp();
                continue;
            }
            const int32_t pairs = (r1 - r0) * W;
            for (int32_t pr = lane; pr < pairs; pr += 32) {
                const int32_t rr = pr / W, col = c0 + pr % W;
                const int64_t vrow = sr[rr];
                const bool on = row_on(ra, vrow, t);
                const bool live = on && t * TILE + col < kcols;
                const int32_t q0 = sp[rr], q1 = live ? sp[rr + 1] : q0;
                const T sum = row_sum_lane<T>(si, sv, q0, q1, xt + col);
                if (on) chunk_epilogue<MODE, T>(out, aux, toff, vrow, col, sum, dlast);
            }
            __syncwarp();
        } else {
            // one long row: (32 / W) entry slots x W columns
            const int slot = lane / W, col = c0 + lane % W;
            const int64_t vr0 = rowmap[r0];
            const bool on = row_on(ra, vr0, t);
            const bool live = t * TILE + col < kcols;
            T acc = 0;
            for (int64_t base = e0; on && base < e1; base += CHUNK_CAP) {  // warp-uniform
                const int m = (int)min((int64_t)CHUNK_CAP, e1 - base);
                for (int i = lane; i < m; i += 32) {
                    si[i] = __ldcs(idx + base + i);
                    sv[i] = __ldcs(val + base + i);
                }
                __syncwarp();
                for (int q = 0; q < m; q += ROW_SEG)
                    acc += seg_sum_slots<T, W>(si, sv, q, live ? min(q + ROW_SEG, m) : q, xt + col, slot);
                __syncwarp();
            }
            if (lane < W && on) chunk_epilogue<MODE, T>(out, aux, toff, vr0, col, acc, dlast);
        }
    }
}

// ---------------------------------------------------------------- q = A p
// A warp's item is a chunk (as above) or a segment of CHUNK_CAP entries of a longer row.  A segment's sums go to
// lpart[segment][column], and k_spmm_long adds a row's segments up: a hub's row, walked by one warp, kept a whole launch
// waiting.  Where most rows are that long, lpart holds some tiles' columns only and a product is launched in groups of
// tiles (SpmmPlan::group).  The lanes of a row have eight gathers in flight, its last entries (under predicates) among them,
// in four accumulators: a grid's row of seven entries costs one gather latency, where a loop over the last three added three.
// Bound by random 256-byte row gathers through L2 (51 GB in 5.1 ms at ER n = 250,000).  Measured on B200, one FP64 product,
// with the long rows walked whole and serial last entries -> here: R-MAT n = 24,281, 883K entries, 2693 columns 4.21 ->
// 1.78 ms; 3-D grid n = 80,840, 1085 columns 1.05 -> 0.58; ER n = 250,000, degree 20, 1194 columns 6.4 -> 5.1; ER n = 1M, 80
// columns 2.70 -> 2.10.  FP32 (spmm_row_pair) 2.98 -> 2.45 ms at ER n = 229,373, 1185 columns.  Slower: 16-column halves of a
// tile, whose gathered rows then fit L2 (2.89 against 2.75 ms at ER n = 1M); FP64 in 16-byte pieces the same way (6.2 ms
// against 5.06 at ER n = 250,000); FP32 with 3, 5 or 6 pairs in flight (2.67, 2.90, 2.98 against 2.37 with one chain a
// half-warp) and a half-warp per row (3.83).
// Six resident blocks per SM (five ran slower: FP32 29.7 against 22.6 ms at ER n = 1M, 1327 columns).
struct SpmmItems {
    const int32_t* chunks = nullptr;  // nchunks + 1 row starts (a row of more than CHUNK_CAP entries is skipped there)
    int32_t nchunks = 0;
    int32_t nseg = 0;
    const int64_t* seg = nullptr;     // first entry of each segment (its end: CHUNK_CAP further, or the row's)
    const int32_t* segrow = nullptr;  // row of each segment
    int32_t nlong = 0;
    const int32_t* lrow = nullptr;    // rows of more than CHUNK_CAP entries
    const int32_t* lseg = nullptr;    // nlong + 1 first segments
};
// Up to SPMM_SEG entries of a row are summed in four chains; where rows are longer on average (SpmmPlan::segs), segment by
// segment.  Rows of 100 to 256 entries in four chains throughout (FP32: two) were rounded 1.2 to 1.3 (1.6 to 1.8) times worse
// than in the eight of a lane per value; in segments it is 0.86 to 0.97 (1.02 to 1.04) times, and shorter rows are the same.
// The products take 1.65 -> 1.78 ms (R-MAT as above) and 2.05 -> 2.13 (ER n = 20,000, degree 200); with segments on ER n = 1M,
// degree 20, 1327 columns, one took 32.5 ms instead of 30.7.  Eight chains, whose registers cost gathers in flight, made a
// whole call on ER n = 250,000 230 ms instead of 189.
constexpr int SPMM_SEG = 32;
template <class T>
__device__ __forceinline__ T spmm_seg(const int32_t* si, const T* sv, int32_t q, int32_t q1, const T* xt) {
    T a[4] = {0, 0, 0, 0};
    for (; q + 7 < q1; q += 8) {
        T x[8];
#pragma unroll
        for (int u = 0; u < 8; u++) x[u] = xt[(int64_t)si[q + u] * TILE];
#pragma unroll
        for (int u = 0; u < 8; u++) a[u & 3] += sv[q + u] * x[u];
    }
    if (q < q1) {
        T x[7];
#pragma unroll
        for (int u = 0; u < 7; u++) x[u] = q + u < q1 ? xt[(int64_t)si[q + u] * TILE] : (T)0;
#pragma unroll
        for (int u = 0; u < 7; u++)
            if (q + u < q1) a[u & 3] += sv[q + u] * x[u];
    }
    return (a[0] + a[1]) + (a[2] + a[3]);
}
template <class T, bool SEGS>
__device__ __forceinline__ T spmm_row(const int32_t* si, const T* sv, int32_t q, int32_t q1, const T* xt) {
    if (!SEGS || q1 - q <= SPMM_SEG) return spmm_seg<T>(si, sv, q, q1, xt);
    T tot = 0;
    for (; q < q1; q += SPMM_SEG) tot += spmm_seg<T>(si, sv, q, min(q + SPMM_SEG, q1), xt);
    return tot;
}

// The same sums of an FP32 row by a whole warp: a lane has two columns, and the half-warps take every second entry, so that
// a load instruction moves 256 bytes as in FP64.  Both halves return the row's sums; a half adds up
// four entries before they join its chain.  (q0, q1: the row's entries; xt: at the lane's first column)
__device__ __forceinline__ float2 spmm_row_pair(const int32_t* si, const float* sv, int32_t q0, int32_t q1,
                                                const float* xt, int half) {
    constexpr int U = 4;
    float2 a = {0, 0};
    int32_t q = q0 + half;
    for (; q + 2 * (U - 1) < q1; q += 2 * U) {
        float2 x[U];
#pragma unroll
        for (int u = 0; u < U; u++) x[u] = *reinterpret_cast<const float2*>(xt + (int64_t)si[q + 2 * u] * TILE);
        const float v0 = sv[q], v1 = sv[q + 2], v2 = sv[q + 4], v3 = sv[q + 6];
        a.x += (v0 * x[0].x + v1 * x[1].x) + (v2 * x[2].x + v3 * x[3].x);
        a.y += (v0 * x[0].y + v1 * x[1].y) + (v2 * x[2].y + v3 * x[3].y);
    }
    if (q < q1) {
        float2 x[U - 1], t = {0, 0};
#pragma unroll
        for (int u = 0; u < U - 1; u++)
            if (q + 2 * u < q1) x[u] = *reinterpret_cast<const float2*>(xt + (int64_t)si[q + 2 * u] * TILE);
#pragma unroll
        for (int u = 0; u < U - 1; u++)
            if (q + 2 * u < q1) {
                t.x += sv[q + 2 * u] * x[u].x;
                t.y += sv[q + 2 * u] * x[u].y;
            }
        a.x += t.x;
        a.y += t.y;
    }
    __syncwarp();
    a.x += __shfl_xor_sync(0xffffffffu, a.x, 16);
    a.y += __shfl_xor_sync(0xffffffffu, a.y, 16);
    return a;
}

// W: columns per warp row (TILE, or 8 when at most 8 are real); ACC adds into q (the second and later column slabs); SEGS: rows
// are summed in segments
template <class T, int W, bool ACC, bool SEGS>
__global__ void __launch_bounds__(CH_THREADS, 6)
    k_spmm(int64_t n, SpmmItems S, const int64_t* __restrict__ ptr, const int32_t* __restrict__ idx,
           const T* __restrict__ val, const T* __restrict__ p, T* __restrict__ q, int64_t ld, T* __restrict__ lpart,
           int64_t lld, double* __restrict__ part, int32_t kcols, RowAct ra) {
    __shared__ int32_t s_idx[CH_WARPS][CHUNK_CAP];
    __shared__ T s_val[CH_WARPS][CHUNK_CAP];
    __shared__ int32_t s_ptr[CH_WARPS][CHUNK_ROWS + 1];
    __shared__ double s_red[CH_THREADS];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const int64_t t = blockIdx.y;
    const int64_t toff = t * n * TILE;
    const T* xt = p + toff;
    int32_t* si = s_idx[w];
    T* sv = s_val[w];
    int32_t* sp = s_ptr[w];
    constexpr bool PAIR = W == TILE && sizeof(T) == 4;
    double dot = 0.0, dot1 = 0.0;  // per-lane partials of p.q for column (lane % W), or for the lane's two columns
    for (int32_t c = blockIdx.x * CH_WARPS + w; c < S.nseg + S.nchunks; c += gridDim.x * CH_WARPS) {
        const bool seg = c < S.nseg;  // segments, the larger items, first
        const int32_t r0 = seg ? S.segrow[c] : S.chunks[c - S.nseg], r1 = seg ? r0 + 1 : S.chunks[c - S.nseg + 1];
        const int64_t e0 = seg ? S.seg[c] : ptr[r0];
        const int64_t e1 = seg ? min(e0 + CHUNK_CAP, ptr[r1]) : ptr[r1];
        const int32_t ne = (int32_t)(e1 - e0);
        if (ne > CHUNK_CAP) continue;  // a long row: its segments
        for (int32_t i = lane; i < ne; i += 32) {
            si[i] = __ldcs(idx + e0 + i);
            sv[i] = __ldcs(val + e0 + i);
        }
        for (int32_t i = lane; i <= r1 - r0; i += 32) sp[i] = seg ? i * ne : (int32_t)(ptr[r0 + i] - e0);
        __syncwarp();
        if constexpr (PAIR) {
            const int half = lane >> 4, col = (lane & 15) * 2;
            for (int32_t rr = 0; rr < r1 - r0; rr++) {
                const int64_t row = r0 + rr;
                if (!row_on(ra, row, t)) continue;  // warp-uniform
                float2 acc = spmm_row_pair(si, sv, sp[rr], t * TILE + col < kcols ? sp[rr + 1] : 0, xt + col, half);
                if (half) continue;
                if (seg) {
                    *reinterpret_cast<float2*>(lpart + (int64_t)c * lld + t * TILE + col) = acc;
                    continue;
                }
                const int64_t o = toff + row * TILE + col;
                if (ACC) {
                    const float2 old = __ldcs(reinterpret_cast<const float2*>(q + o));
                    acc.x += old.x;
                    acc.y += old.y;
                }
                __stcs(reinterpret_cast<float2*>(q + o), acc);
                if (part) {
                    const float2 pv = *reinterpret_cast<const float2*>(xt + row * TILE + col);
                    dot += (double)acc.x * (double)pv.x;
                    dot1 += (double)acc.y * (double)pv.y;
                }
            }
            __syncwarp();
            continue;
        }
        const int32_t pairs = (r1 - r0) * W;
        for (int32_t pr = lane; pr < pairs; pr += 32) {
            const int32_t rr = pr / W, col = pr % W;
            const int64_t row = r0 + rr;
            const bool on = row_on(ra, row, t);
            const int32_t q0 = sp[rr], q1 = on && t * TILE + col < kcols ? sp[rr + 1] : q0;
            T acc = spmm_row<T, SEGS>(si, sv, q0, q1, xt + col);
            if (!on) continue;
            if (seg) {
                lpart[(int64_t)c * lld + t * TILE + col] = acc;
            } else {
                // q streams out (evict-first), so it does not push the gathered slab out of L2
                const int64_t o = toff + row * TILE + col;
                if (ACC) acc += __ldcs(q + o);
                __stcs(q + o, acc);
                if (part) dot += (double)acc * (double)xt[row * TILE + col];
            }
        }
        __syncwarp();
    }
    if (part) {
        if (!PAIR) {
            s_red[threadIdx.x] = dot;
        } else if (lane < 16) {
            s_red[w * TILE + 2 * lane] = dot;
            s_red[w * TILE + 2 * lane + 1] = dot1;
        }
        __syncthreads();
        if (threadIdx.x < TILE) {
            double tt = 0.0;
            if (threadIdx.x < W)
                for (int i = 0; i < CH_THREADS / W; i++) tt += s_red[i * W + threadIdx.x];
            part[(int64_t)blockIdx.x * ld + t * TILE + threadIdx.x] = tt;
        }
    }
}

// the long rows: their segments' sums in order into q, and their share of p.q (grid: x over rows, y over the group's tiles)
template <class T, bool ACC>
__global__ void __launch_bounds__(CH_THREADS) k_spmm_long(int64_t n, SpmmItems S, const T* __restrict__ lpart, int64_t lld,
                                                          const T* __restrict__ p, T* __restrict__ q, int64_t ld,
                                                          double* __restrict__ part, int32_t kcols, RowAct ra) {
    __shared__ double s_red[CH_THREADS];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const int64_t t = blockIdx.y, toff = t * n * TILE;
    const bool live = t * TILE + lane < kcols;  // a narrow product leaves the other columns' partials unset
    double dot = 0.0;
    for (int32_t i = blockIdx.x * CH_WARPS + w; i < S.nlong; i += gridDim.x * CH_WARPS) {
        const int64_t row = S.lrow[i];
        if (!row_on(ra, row, t)) continue;
        T acc = 0;
#pragma unroll 4
        for (int32_t g = S.lseg[i]; g < S.lseg[i + 1] && live; g++) acc += lpart[(int64_t)g * lld + t * TILE + lane];
        const int64_t o = toff + row * TILE + lane;
        if (ACC) acc += q[o];
        q[o] = acc;
        dot += (double)acc * (double)p[o];
    }
    if (part) {
        s_red[threadIdx.x] = dot;
        __syncthreads();
        if (threadIdx.x < TILE) {
            double tt = 0.0;
            for (int i = 0; i < CH_WARPS; i++) tt += s_red[i * 32 + threadIdx.x];
            part[(int64_t)blockIdx.x * ld + t * TILE + threadIdx.x] = tt;
        }
    }
}

// Four squared differences' sums over a warp, each as the xor butterfly over offsets 16, 8, 4, 2, 1 would form it (the
// same operands added in the same order), in 6 shuffles of a double instead of 20: the first two steps hand half
// of the values to the other half of the lanes.  Lane 8 v gets value v.
__device__ __forceinline__ double warp_sum4(double s0, double s1, double s2, double s3, int lane) {
    const bool h = lane & 16, g = lane & 8;
    const double a = __dadd_rn(h ? s2 : s0, __shfl_xor_sync(0xffffffffu, h ? s0 : s2, 16));
    const double b = __dadd_rn(h ? s3 : s1, __shfl_xor_sync(0xffffffffu, h ? s1 : s3, 16));
    double c = __dadd_rn(g ? b : a, __shfl_xor_sync(0xffffffffu, g ? a : b, 8));
#pragma unroll
    for (int o = 4; o >= 1; o >>= 1) c = __dadd_rn(c, __shfl_xor_sync(0xffffffffu, c, o));
    return c;
}

// The final product of a solve, one tile per launch, also forming the squared diff norms of the edges from
// the rows it gathers: the edge of an entry with row < column (eid >= 0) gets, per tile, the xor-butterfly
// sum over the tile's 32 columns of (x[row] - x[col])^2 (0 for columns past k), added to d2 in tile order
// (first: stored) -- diff_norms_device's order.  All 32 lanes of a warp walk the same row, eight gathers in flight; a
// group of four entries without an edge skips the sums.  Long rows are cut into segments as in k_spmm.  With four gathers
// in flight, 20 shuffles per edge and whole rows a launch took 0.38 ms at ER n = 250,000, 1.38 at ER n = 1M and 1.15 on
// k_spmm's R-MAT graph (its hubs); here 0.32, 1.25 and 0.08.
__global__ void __launch_bounds__(CH_THREADS) k_spmm_diff(int64_t n, SpmmItems S, const int64_t* __restrict__ ptr,
                                                          const int32_t* __restrict__ idx,
                                                          const double* __restrict__ val,
                                                          const int32_t* __restrict__ eid, const double* xt,
                                                          double* qt, int32_t kcols, double* __restrict__ d2,
                                                          int first, double* __restrict__ lpart, int64_t lld) {
    __shared__ int32_t s_idx[CH_WARPS][CHUNK_CAP];
    __shared__ double s_val[CH_WARPS][CHUNK_CAP];
    __shared__ int32_t s_eid[CH_WARPS][CHUNK_CAP];
    __shared__ int32_t s_ptr[CH_WARPS][CHUNK_ROWS + 1];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const bool live = lane < kcols;
    int32_t* si = s_idx[w];
    double* sv = s_val[w];
    int32_t* se = s_eid[w];
    int32_t* sp = s_ptr[w];
    for (int32_t c = blockIdx.x * CH_WARPS + w; c < S.nseg + S.nchunks; c += gridDim.x * CH_WARPS) {
        const bool seg = c < S.nseg;
        const int32_t r0 = seg ? S.segrow[c] : S.chunks[c - S.nseg], r1 = seg ? r0 + 1 : S.chunks[c - S.nseg + 1];
        const int64_t e0 = seg ? S.seg[c] : ptr[r0];
        const int64_t e1 = seg ? min(e0 + CHUNK_CAP, ptr[r1]) : ptr[r1];
        const int32_t ne = (int32_t)(e1 - e0);
        if (ne > CHUNK_CAP) continue;
        for (int32_t i = lane; i < ne; i += 32) {
            si[i] = __ldcs(idx + e0 + i);
            sv[i] = __ldcs(val + e0 + i);
            se[i] = __ldcs(eid + e0 + i);
        }
        for (int32_t i = lane; i <= r1 - r0; i += 32) sp[i] = seg ? i * ne : (int32_t)(ptr[r0 + i] - e0);
        __syncwarp();
        for (int32_t rr = 0; rr < r1 - r0; rr++) {
            const int64_t row = r0 + rr;
            const double xo = live ? xt[row * TILE + lane] : 0.0;
            const int32_t q0 = sp[rr], q1 = sp[rr + 1];
            double a[4] = {0, 0, 0, 0};
            for (int32_t q = q0; q < q1; q += 8) {
                double g[8];
#pragma unroll
                for (int u = 0; u < 8; u++) g[u] = live && q + u < q1 ? xt[(int64_t)si[q + u] * TILE + lane] : 0.0;
#pragma unroll
                for (int h = 0; h < 8; h += 4) {
                    int32_t any = -1;
#pragma unroll
                    for (int u = h; u < h + 4; u++)
                        if (q + u < q1) {
                            a[u & 3] += sv[q + u] * g[u];
                            any = max(any, se[q + u]);
                        }
                    if (any < 0) continue;  // warp-uniform
                    double sq[4];
#pragma unroll
                    for (int u = 0; u < 4; u++) {
                        const double dx = live ? __dsub_rn(xo, g[h + u]) : 0.0;
                        sq[u] = __dmul_rn(dx, dx);
                    }
                    const double sum = warp_sum4(sq[0], sq[1], sq[2], sq[3], lane);
                    const int v = h + (lane >> 3);
                    const int32_t e = (lane & 7) == 0 && q + v < q1 ? se[q + v] : -1;
                    if (e >= 0) d2[e] = first ? sum : __dadd_rn(d2[e], sum);
                }
            }
            const double sum = (a[0] + a[1]) + (a[2] + a[3]);
            if (seg) lpart[(int64_t)c * lld + lane] = sum;
            else __stcs(qt + row * TILE + lane, sum);
        }
        __syncwarp();
    }
}

// blocks per tile: about one wave of resident blocks, so the gathered slab of the tile being worked
// on is the only one live in L2
static int chunk_blocks(int32_t nchunks) {
    return std::max(1, std::min((nchunks + CH_WARPS - 1) / CH_WARPS, 148 * 6));
}

// Levels walked inside one launch: the k columns are independent, so one block per sub-tile of W columns goes through
// consecutive levels on its own, with only block barriers between them (it reads back nothing but its own writes).
// A level then costs the chain barrier -> gather -> sum -> store instead of a launch.  Its rows, ordered by length, are
// taken in rounds (TrsvPlan): a slot of W / 2 lanes (two columns each, 16-byte gathers) works on a row, or 2^lg slots of a
// warp share it.  The next round's rows, their own values and first entries are loaded while the current one is
// summed, across level boundaries too.  y is read and written in place: no read-only cache path.
// What bounds it is the issue of one SM per sub-tile (a round costs every warp about a hundred instructions, however few
// columns it carries: the time is the same with 4 blocks and with 112) and the latency of its chain, not bandwidth.
// Measured on B200, one FP64 application, all levels launched one by one with the thin ones in dependency runs -> here:
// 2-D grid n = 10,000, 885 columns 1.34 -> 0.42 ms; geometric graph n = 20,011, 2642 columns 6.7 -> 4.2 ms; 3-D grid
// n = 80,840, 1085 columns 9.2 -> 4.6 ms; union of 20 graphs, n = 29K, 726 columns 3.5 -> 1.5 ms; ER n = 20,000, degree
// 200, 951 columns 2.0 -> 0.68 ms; geometric graph n = 30,011, 60 columns 9.7 -> 1.8 ms.
// Slower: a row per lane without ordering rows by length (1.3x to 1.6x); rows and entries staged through shared memory
// by cp.async, by warp or by block (1.3x to 2.2x: more instructions per round than the latency they hide).
// Rows row .. row + nr of the storage order, 2^lg slots per row; last: the level's last round
struct WalkRound {
    int32_t row;
    uint16_t nr;
    uint8_t lg, last;
};
constexpr int WALK_MAX_ROUNDS = 4096;  // of one launch (kept in shared memory)

template <class T, int W, int NT, bool FWD, bool CLUSTER>
__global__ void __launch_bounds__(NT, 1024 / NT)
    k_trsv_walk(int64_t n, const WalkRound* __restrict__ rounds, int32_t nrounds, const FactorRow* __restrict__ rows,
                const FactorEnt<T>* __restrict__ ent, const T* __restrict__ aux, T* y, int32_t kcols, int nsub, int cl,
                RowAct ra) {
    using V = typename ColPair<T>::V;
    constexpr int LPS = W / 2, B = 4;
    extern __shared__ WalkRound s_rounds[];
    for (int i = threadIdx.x; i < nrounds; i += NT) s_rounds[i] = rounds[i];
    __syncthreads();
    // a cluster of cl blocks shares a sub-tile's rows
    const int sub = CLUSTER ? blockIdx.x / cl : blockIdx.x;
    const int slot = (CLUSTER ? blockIdx.x % cl : 0) * (NT / LPS) + threadIdx.x / LPS;
    const int64_t t = sub / nsub;
    const int c0 = sub % nsub * W;
    // a block of padding columns only keeps them at zero (r is zero there): no gathers
    const bool dead = t * TILE + c0 >= kcols;
    T* yt = y + t * n * TILE + c0 + 2 * (threadIdx.x % LPS);
    const T* rt = FWD ? aux + t * n * TILE + c0 + 2 * (threadIdx.x % LPS) : nullptr;
    auto at = [](const T* p, int32_t u) -> V { return *reinterpret_cast<const V*>(p + (int64_t)u * TILE); };
    // this slot's share of a row: vertex u (-1: none), cnt entries from e on, stride 2^lg
    int32_t u, cnt;
    const FactorEnt<T>* e;
    FactorEnt<T> en[B];
    V o;
    T d = (T)0;
    auto load_row = [&](const WalkRound& w) -> FactorRow {
        FactorRow r;
        r.u = -1;
        const int q = slot >> w.lg;
        if (q < w.nr) r = rows[w.row + q];
        return r;
    };
    auto take = [&](const FactorRow& r, int lg) {
        u = r.u;
        cnt = 0;
        if (u >= 0) {
            if (!row_on(ra, u, t)) {
                u = -1;
            } else {
                const int g = slot & ((1 << lg) - 1);
                if (!dead) cnt = (r.cnt - g + (1 << lg) - 1) >> lg;
                e = ent + r.e0 + g;
                o = at(FWD ? rt : yt, u);
                if (!FWD) d = aux[u];
#pragma unroll
                for (int k = 0; k < B; k++)
                    if (k < cnt) en[k] = e[k << lg];
            }
        }
    };
    WalkRound w = s_rounds[0];
    take(load_row(w), w.lg);
    for (int32_t i = 0; i < nrounds; i++) {
        WalkRound nw = s_rounds[min(i + 1, nrounds - 1)];
        if (i + 1 == nrounds) nw.nr = 0;
        if (!__any_sync(0xffffffffu, u >= 0)) {
            take(load_row(nw), nw.lg);
        } else {
            V acc{(T)0, (T)0}, x[B];
#pragma unroll
            for (int k = 0; k < B; k++)
                if (k < cnt) x[k] = at(yt, en[k].idx);
            const FactorRow nr = load_row(nw);
#pragma unroll
            for (int k = 0; k < B; k++)
                if (k < cnt) {
                    acc.x += en[k].v * x[k].x;
                    acc.y += en[k].v * x[k].y;
                }
            for (int done = B; done < cnt; done += B) {
                e += B << w.lg;
#pragma unroll
                for (int k = 0; k < B; k++)
                    if (done + k < cnt) en[k] = e[k << w.lg];
#pragma unroll
                for (int k = 0; k < B; k++)
                    if (done + k < cnt) x[k] = at(yt, en[k].idx);
#pragma unroll
                for (int k = 0; k < B; k++)
                    if (done + k < cnt) {
                        acc.x += en[k].v * x[k].x;
                        acc.y += en[k].v * x[k].y;
                    }
            }
            __syncwarp();
            for (int f = LPS; f < (LPS << w.lg); f <<= 1) {
                acc.x += __shfl_xor_sync(0xffffffffu, acc.x, f);
                acc.y += __shfl_xor_sync(0xffffffffu, acc.y, f);
            }
            if (u >= 0 && (slot & ((1 << w.lg) - 1)) == 0) {
                // FWD: y_u = r_u - L[u, :] y.  BWD: y_u = y_u / D_u (D_u != 0) - L[:, u]^T y.
                if (!FWD && d != (T)0) {
                    o.x /= d;
                    o.y /= d;
                }
                o.x -= acc.x;
                o.y -= acc.y;
                *reinterpret_cast<V*>(yt + (int64_t)u * TILE) = o;
            }
            take(nr, nw.lg);
        }
        if (w.last) {
            // the level's rows are written, for this block or, released and acquired, for the cluster's others
            if (!CLUSTER) __syncthreads();
            else asm volatile("barrier.cluster.arrive.release;\nbarrier.cluster.wait.acquire;" ::: "memory");
        }
        w = nw;
    }
}

// ---------------------------------------------------------------- the last forward level, finished
// The rows of a factor's last level are read by no later forward level, and their columns of L are empty
// (nothing is eliminated after them; a level's rows never reference each other), so the backward solve's
// whole work on them is z_u = y_u / D_u - 0.  When there is no dense tail, the last level is a launch of its own and
// its forward launch (M_FWD_LAST) does this too and its backward launch is skipped; each
// value is formed by the same operations in the same order as in the two launches.  At ER n = 1M the
// truncated factor's last level holds 855K of the 1M rows, and its backward launch took 5.5 ms of a 21 ms
// application.  (A kernel that gave each warp several of these short rows at once, with all their loads
// issued first, ran slower than this chunk walk: 28.8 against 20.8 ms per application.)

// ---------------------------------------------------------------- preconditioner as a CUDA graph
// values of the factor in the precision of the solve (the structure is shared)
template <class T>
struct FactorVals {
    const T* prow_val;
    const T* pcol_val;
    const T* D;
    // null where the memory does not allow them:
    const T* tin_val = nullptr;  // the dense tail's entries in earlier levels, and its inverse
    const T* linv = nullptr;
    T* tail_tmp = nullptr;       // tail rows x ld scratch
    const FactorEnt<T>* fent = nullptr;  // the entries of both forms with their values beside them (walked levels)
    const FactorEnt<T>* bent = nullptr;
};

// Column layouts of the triangular-solve launches.  A level launch gives each warp row a width of W columns
// (8, 16 or 32; TILE / W blocks per column tile): with W = 32 a warp's lanes cover a tile's columns of one row
// (256-byte gathers); with W = 8 a warp works on four rows at once, with four times the blocks, which suits
// latency-bound levels of few rows.  Every width gives the same values bit for bit (each (row, column) sum is
// formed the same way, see k_chunked), so the width is a pure launch-shape choice: the fixed rule below, or
// widths measured level by level (tune_trsv_shapes).  Walked levels have their own layout (WalkShape).  With no more
// than 8 real columns (the factor autotuner's probe) every launch uses 8 columns and one sub-tile; the padding
// columns of y must then be zero.
constexpr int NARROW_W = 8;
constexpr int SPLIT_LEVEL_ROWS = 28 * 1024;
constexpr int TRSV_NWIDTH = TILE >= 32 ? 3 : TILE >= 16 ? 2 : 1;  // widths 8, 16, 32 that fit a tile
static inline int trsv_width(int code) { return 8 << code; }
// The fixed rule: 8 columns per warp row up to SPLIT_LEVEL_ROWS (row, column tile) pairs -- 1024 rows at 900 columns --
// and 32 above: a small solve's levels need the four times as many warps up to more rows.
static int rule_code(const DevFactor& F, int32_t l, int ntiles, bool narrow) {
    if (narrow) return 0;
    const int64_t rows = F.level_ptr[l + 1] - F.level_ptr[l];
    return std::min(rows * ntiles <= SPLIT_LEVEL_ROWS ? 0 : 2, TRSV_NWIDTH - 1);
}

// CUDA events around each level launch of a preconditioner application (measurement only)
struct LevelEvents {
    std::vector<cudaEvent_t> ev;        // pairs: before, after
    std::vector<std::pair<bool, int32_t>> tag;  // (forward, level) of each pair
    size_t used = 0;
    ~LevelEvents() {
        for (auto e : ev) cudaEventDestroy(e);
    }
    void begin(cudaStream_t s, bool fwd, int32_t l) {
        if (2 * used == ev.size()) {
            for (int i = 0; i < 2; i++) {
                cudaEvent_t e;
                SSP_CUDA(cudaEventCreate(&e));
                ev.push_back(e);
            }
            tag.push_back({fwd, l});
        }
        tag[used] = {fwd, l};
        SSP_CUDA(cudaEventRecord(ev[2 * used], s));
    }
    void end(cudaStream_t s) {
        SSP_CUDA(cudaEventRecord(ev[2 * used + 1], s));
        used++;
    }
};

template <int MODE, class T, int MINB>
static void launch_level_w(int code, dim3 grid, cudaStream_t s, int64_t n, const int32_t* ch, int32_t nc,
                           const int64_t* ptr, const int32_t* idx, const T* val, const int32_t* rowmap, T* y,
                           const T* aux, int32_t kcols, int nsub, const T* dlast, const RowAct& ra) {
    switch (code) {
    case 0:
        k_chunked<MODE, T, 8, MINB><<<grid, CH_THREADS, 0, s>>>(n, ch, nc, ptr, idx, val, rowmap, y, y, aux, kcols,
                                                                nsub, dlast, ra);
        break;
    case 1:
        k_chunked<MODE, T, (TILE >= 16 ? 16 : 8), MINB><<<grid, CH_THREADS, 0, s>>>(
            n, ch, nc, ptr, idx, val, rowmap, y, y, aux, kcols,
                                                                nsub, dlast, ra);
        break;
    default:
        k_chunked<MODE, T, TILE, (sizeof(T) == 8 ? MINB_WIDE64 : MINB)><<<grid, CH_THREADS, 0, s>>>(
            n, ch, nc, ptr, idx, val, rowmap, y, y, aux, kcols, nsub, dlast, ra);
        break;
    }
}

// ---------------------------------------------------------------- which levels are walked
// A walk's blocks: W columns and NT threads each, one of 1024 threads per SM, or smaller ones so that all of them are
// resident at once.  Where the columns leave SMs idle, a cluster of cl blocks shares a sub-tile's rows.
struct WalkShape {
    int W = 8, NT = 1024, nsub = 1, cl = 1;  // nsub sub-tiles per column tile
    int64_t blocks = 0;
    int slots() const { return 2 * NT / W * cl; }
};
static WalkShape walk_shape(int ntiles, bool narrow, int cl) {
    const int64_t cols = narrow ? NARROW_W : (int64_t)ntiles * TILE;
    WalkShape w;
    w.W = narrow ? 2 : 8;
    w.nsub = (narrow ? NARROW_W : TILE) / w.W;
    w.cl = cl;
    w.blocks = cols / w.W * cl;
    w.NT = w.blocks <= 148 ? 1024 : w.blocks <= 2 * 148 ? 512 : 256;
    return w;
}
// One direction's segments [l0, l1) of the levels before the dense tail, in level order.
struct TrsvSeg {
    int32_t l0, l1;
    const WalkRound* rounds = nullptr;  // device; null: a launch of its own
    int32_t nrounds = 0;
    size_t at = 0;                      // the first of them in the plan's list
};
struct TrsvPlan {
    std::vector<TrsvSeg> fw, bw;
    bool fuse_last = false;
    bool tail = false;  // the dense tail as a product with its inverse; else its levels like the others
    WalkShape walk;
};

template <class T, int W, int NT, bool CLUSTER>
static void launch_walk_fb(Context& C, bool fwd, const TrsvPlan& P, const TrsvSeg& S, const DevFactor& F,
                           const FactorVals<T>& V, int64_t n, const T* r, T* y, int32_t kcols, const RowAct& ra) {
    auto kern = fwd ? k_trsv_walk<T, W, NT, true, CLUSTER> : k_trsv_walk<T, W, NT, false, CLUSTER>;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)P.walk.blocks);
    cfg.blockDim = dim3(NT);
    cfg.dynamicSmemBytes = sizeof(WalkRound) * S.nrounds;  // at most 32 KB
    cfg.stream = C.stream;
    cudaLaunchAttribute cluster;
    cluster.id = cudaLaunchAttributeClusterDimension;
    cluster.val.clusterDim.x = (unsigned)P.walk.cl;
    cluster.val.clusterDim.y = cluster.val.clusterDim.z = 1;
    cfg.attrs = &cluster;
    cfg.numAttrs = CLUSTER ? 1 : 0;
    const WalkRound* rounds = S.rounds;
    const FactorRow* rows = fwd ? F.frow : F.brow;
    const FactorEnt<T>* ent = fwd ? V.fent : V.bent;
    const T* aux = fwd ? r : V.D;
    SSP_CUDA(cudaLaunchKernelEx(&cfg, kern, n, rounds, S.nrounds, rows, ent, aux, y, kcols, P.walk.nsub, P.walk.cl, ra));
}
template <class T>
static void launch_walk(Context& C, bool fwd, const TrsvPlan& P, const TrsvSeg& S, const DevFactor& F,
                        const FactorVals<T>& V, int64_t n, const T* r, T* y, int32_t kcols, const RowAct& ra) {
    const WalkShape& w = P.walk;
    auto launch = w.W == 2 ? (w.cl > 1 ? launch_walk_fb<T, 2, 1024, true> : launch_walk_fb<T, 2, 1024, false>)
                  : w.cl > 1 ? launch_walk_fb<T, 8, 1024, true>
                  : w.NT == 1024 ? launch_walk_fb<T, 8, 1024, false>
                  : w.NT == 512 ? launch_walk_fb<T, 8, 512, false> : launch_walk_fb<T, 8, 256, false>;
    launch(C, fwd, P, S, F, V, n, r, y, kcols, ra);
}

// The plan for a solve's columns; the rounds go to workspace buffers named after tag.  Without the copies of the factor's
// entries no level is walked.
template <class T>
static TrsvPlan make_trsv_plan(Context& C, const DevFactor& F, const FactorVals<T>& V, int ntiles, bool narrow,
                               const std::string& tag) {
    TrsvPlan P;
    constexpr size_t elem = sizeof(T);
    P.tail = F.tail_rows && V.linv && V.tail_tmp;
    // SSP_TRSV_WALK=0 launches every level, =1 walks every one that can be; SSP_TRSV_CLUSTER=1|2|4|8 sets the blocks of a
    // cluster (as far as they are resident at once).  For comparisons.
    const char* walk_env = getenv("SSP_TRSV_WALK");
    const char* cl_env = getenv("SSP_TRSV_CLUSTER");
    const bool walk_all = walk_env && walk_env[0] == '1';
    const int set_cl = cl_env ? atoi(cl_env) : 0;
    const bool walks = V.fent && V.bent && !(walk_env && walk_env[0] == '0');
    const int32_t NL = P.tail ? F.tail_l0 : F.num_levels;
    // the last level finished by its forward launch (M_FWD_LAST); SSP_PRECOND_FUSE_LAST=0 keeps the level's two
    // launches (the same values, bit for bit; for comparisons)
    const char* fuse_env = getenv("SSP_PRECOND_FUSE_LAST");
    P.fuse_last = !(fuse_env && fuse_env[0] == '0') && !P.tail && F.num_levels > 0 && F.last_bwd_nnz == 0;
    const double cols = narrow ? NARROW_W : (double)ntiles * TILE;
    // The costs (us, bytes per us) that decide between a launch and a walk, fitted on B200 to the graphs above.  A
    // level's launch takes 13-18 us where it is small (five dependent loads per chunk, most blocks with one chunk) and
    // moves gathered rows at 5.5 TB/s where it is large; a walk costs a round's issue, a cycle of its SM's cache tags per
    // gathered row, or its traffic in 64-byte pieces, whichever is most.
    const double c_launch = 20.0, bw_launch = 5.5e6;
    const double c_round = 0.6, bw_walk = 3.9e6, c_level = 0.5, c_cluster = 0.9;
    const double per_slot = 16.0;
    // The rounds of level l in storage-row order (longest rows first).  2^lg slots share a row: per_slot entries of the
    // round's longest row each, or all the slots there are.
    auto level_rounds = [&](const std::vector<int64_t>& ptr, const WalkShape& w, int32_t l, std::vector<WalkRound>& out) {
        const int slots = w.slots(), max_lg = w.W == 8 ? 3 : 5;  // slots of a warp
        const int64_t a = F.level_ptr[l], b = F.level_ptr[l + 1];
        for (int64_t r = a; r < b;) {
            const int64_t len = ptr[r + 1] - ptr[r];
            int lg = 0;
            while (lg < max_lg && (((b - r) << (lg + 1)) <= slots || (double)len > per_slot * (double)(1 << lg))) lg++;
            const int64_t e = std::min(b, r + (slots >> lg));
            out.push_back(WalkRound{(int32_t)r, (uint16_t)(e - r), (uint8_t)lg, (uint8_t)(e == b)});
            r = e;
        }
    };
    // us of level l walked (rounds: how many) and launched
    auto walk_us = [&](const std::vector<int64_t>& ptr, const WalkShape& w, int32_t l, size_t rounds) {
        const double E = (double)(ptr[F.level_ptr[l + 1]] - ptr[F.level_ptr[l]]), R = F.level_ptr[l + 1] - F.level_ptr[l];
        const double per_sm = (double)ceil_div<int64_t>(w.blocks, 148);
        return c_level + (w.cl > 1 ? c_cluster : 0.0) +
               std::max({per_sm * c_round * rounds, per_sm * E / w.cl / 1900.0, (E + 2 * R) * cols * elem / bw_walk});
    };
    auto launch_us = [&](const std::vector<int64_t>& ptr, int32_t l) {
        const double E = (double)(ptr[F.level_ptr[l + 1]] - ptr[F.level_ptr[l]]), R = F.level_ptr[l + 1] - F.level_ptr[l];
        return c_launch + (E + 2 * R) * cols * elem / bw_launch;
    };
    // the factor's last level is a launch of its own (M_FWD_LAST when it can be)
    const int32_t alone = !walks ? 0 : P.tail ? NL : NL - 1;
    std::vector<WalkRound> tmp;
    double best = 0;
    for (int cl = 1; cl <= 8; cl *= 2) {
        const WalkShape w = walk_shape(ntiles, narrow, cl);
        if (cl > 1 && (w.blocks > 128 || (set_cl && cl > set_cl))) break;
        double us = 0;
        for (int32_t l = 0; l < alone; l++)
            for (const auto* ptr : {&F.hfptr, &F.hbptr}) {
                tmp.clear();
                level_rounds(*ptr, w, l, tmp);
                us += std::min(launch_us(*ptr, l), walk_us(*ptr, w, l, tmp.size()));
            }
        if (cl == 1 || us < best || set_cl) {
            best = us;
            P.walk = w;
        }
    }
    std::vector<WalkRound> all;
    auto plan = [&](bool fwd) {
        const std::vector<int64_t>& ptr = fwd ? F.hfptr : F.hbptr;
        std::vector<TrsvSeg> seg;
        std::vector<double> gain(NL, -1.0);
        std::vector<size_t> cnt(NL, 0);
        for (int32_t l = 0; l < alone; l++) {
            tmp.clear();
            level_rounds(ptr, P.walk, l, tmp);
            cnt[l] = tmp.size();
            gain[l] = walk_all ? c_launch : launch_us(ptr, l) - walk_us(ptr, P.walk, l, tmp.size());
        }
        for (int32_t l = 0; l < NL;) {
            int32_t r = l;
            double g = -c_launch;
            size_t nrd = 0;
            while (r < NL && gain[r] > 0 && nrd + cnt[r] <= WALK_MAX_ROUNDS) nrd += cnt[r], g += gain[r++];
            if (r - l >= 2 && g > 0) {
                const size_t at = all.size();
                for (int32_t i = 0; i < r - l; i++) level_rounds(ptr, P.walk, fwd ? l + i : r - 1 - i, all);
                seg.push_back(TrsvSeg{l, r, nullptr, (int32_t)(all.size() - at), at});
                l = r;
            } else {
                for (r = std::max(r, l + 1); l < r; l++) seg.push_back(TrsvSeg{l, l + 1});
            }
        }
        return seg;
    };
    P.fw = plan(true);
    P.bw = plan(false);
    if (all.empty()) return P;
    WalkRound* d = C.ws.get_optional_t<WalkRound>(tag + "_rounds", all.size());
    if (!d) {
        FactorVals<T> launched = V;
        launched.fent = nullptr;
        return make_trsv_plan<T>(C, F, launched, ntiles, narrow, tag);
    }
    SSP_CUDA(cudaMemcpyAsync(d, all.data(), sizeof(WalkRound) * all.size(), cudaMemcpyHostToDevice, C.stream));
    SSP_CUDA(cudaStreamSynchronize(C.stream));
    for (auto* v : {&P.fw, &P.bw})
        for (TrsvSeg& g : *v) g.rounds = g.nrounds ? d + g.at : nullptr;
    return P;
}

// sh: per-level widths (nullptr: the fixed rule); lev: events around each level launch (nullptr: none)
template <class T>
static int64_t launch_precond(Context& C, const DevFactor& F, const TrsvPlan& P, const FactorVals<T>& V, int64_t n,
                              const T* r, T* y, int64_t ld, int32_t kcols, const RowAct& ra = RowAct(),
                              const TrsvShapes* sh = nullptr, LevelEvents* lev = nullptr) {
    const int ntiles = (int)(ld / TILE);
    const bool narrow = TILE > NARROW_W && kcols <= NARROW_W;
    int64_t launches = 0;
    const int32_t L_last = F.num_levels - 1;
    auto width_code = [&](bool fwd, int32_t l) -> int {
        if (narrow) return 0;
        int c = rule_code(F, l, ntiles, narrow);
        if (sh) {
            const auto& v = fwd ? sh->fw : sh->bw;
            if ((size_t)l < v.size()) c = v[l];
        }
        return std::min(c, TRSV_NWIDTH - 1);
    };
    auto level = [&](bool fwd, int32_t l) {
        const auto& lvl = fwd ? F.fchunk_lvl : F.bchunk_lvl;
        const int32_t c0 = lvl[l], nc = lvl[l + 1] - c0;
        if (nc == 0) return;
        const int code = width_code(fwd, l);
        const int ns = narrow ? 1 : TILE / trsv_width(code);
        const dim3 grid((unsigned)chunk_blocks(nc), (unsigned)(ntiles * ns));
        const int32_t* ch = (fwd ? F.fchunk : F.bchunk) + c0;
        const bool last = fwd && P.fuse_last && l == L_last;
        if (lev) lev->begin(C.stream, fwd, l);
        if (last)
            launch_level_w<M_FWD_LAST, T, MINB_FWD>(code, grid, C.stream, n, ch, nc, F.prow_ptr, F.prow_idx,
                                                    V.prow_val, F.level_rows, y, r, kcols, ns, V.D, ra);
        else if (fwd)
            launch_level_w<M_FWD, T, MINB_FWD>(code, grid, C.stream, n, ch, nc, F.prow_ptr, F.prow_idx, V.prow_val,
                                               F.level_rows, y, r, kcols, ns, nullptr, ra);
        else
            launch_level_w<M_BWD, T, MINB_BWD>(code, grid, C.stream, n, ch, nc, F.pcol_ptr, F.pcol_idx, V.pcol_val,
                                               F.level_cols, y, V.D, kcols, ns, nullptr, ra);
        if (lev) lev->end(C.stream);
        launches++;
    };
    for (const auto& s : P.fw) {
        if (!s.rounds) {
            level(true, s.l0);
            continue;
        }
        launch_walk<T>(C, true, P, s, F, V, n, r, y, kcols, ra);
        launches++;
    }
    if (P.tail) {
        // the tail's rows less their entries in earlier levels (one launch, as a level), then its block
        const int code = width_code(true, F.tail_l0);
        const int ns = narrow ? 1 : TILE / trsv_width(code);
        launch_level_w<M_FWD, T, MINB_FWD>(code, dim3((unsigned)chunk_blocks(F.ntchunk), (unsigned)(ntiles * ns)),
                                           C.stream, n, F.tchunk, F.ntchunk, F.tin_ptr, F.tin_idx, V.tin_val,
                                           F.level_rows + (F.n - F.tail_rows), y, r, kcols, ns, nullptr, ra);
        launches += 1 + launch_tail<T>(C, F, V.linv, V.D, y, V.tail_tmp, ntiles);
    }
    for (size_t i = P.bw.size(); i-- > 0;) {
        const auto& s = P.bw[i];
        if (P.fuse_last && s.l1 == F.num_levels) continue;  // finished by its forward launch (M_FWD_LAST)
        if (!s.rounds) {
            level(false, s.l0);
            continue;
        }
        launch_walk<T>(C, false, P, s, F, V, n, r, y, kcols, ra);
        launches++;
    }
    SSP_CHECK_LAUNCH();
    return launches;
}

// Level-launch shapes by measurement.  Each width is timed on every level launch of one preconditioner
// application (CUDA events around each launch), and each level and direction keeps its fastest width.  In a PCG
// solve the measured applications are the solve's own first three (one per width): the values are the same
// whatever the widths, so they are real iterations and nothing is applied twice; the preconditioner's graph is
// then rebuilt with the result.  The shapes are kept per context under a signature of the factor's level
// structure and the solve's shape, so repeated solves on the same graph measure once.  Small solves (n * ld
// below SSP_TRSV_TUNE_MIN elements, 2^26 unless the environment variable of that name says otherwise) keep the
// rule.  SSP_TRSV_TUNE=0 keeps the rule everywhere; SSP_TRSV_WIDTH=8|16|32 forces one width.
#ifndef SSP_TRSV_TUNE_MIN
#define SSP_TRSV_TUNE_MIN (int64_t(1) << 26)
#endif
constexpr int TRSV_CACHE_MAX = 8;
static int64_t trsv_tune_min() {
    const char* e = getenv("SSP_TRSV_TUNE_MIN");  // elements n * ld from which to measure
    return e && e[0] ? atoll(e) : (int64_t)SSP_TRSV_TUNE_MIN;
}

static uint64_t trsv_signature(const DevFactor& F, int64_t n, int64_t ld, int32_t kcols, size_t elem,
                               bool segmented) {
    uint64_t h = 1469598103934665603ull;
    auto mix = [&](uint64_t v) {
        for (int i = 0; i < 8; i++) {
            h ^= (v >> (8 * i)) & 0xff;
            h *= 1099511628211ull;
        }
    };
    mix((uint64_t)n);
    mix((uint64_t)ld);
    mix((uint64_t)kcols);
    mix((uint64_t)elem);
    mix((uint64_t)segmented);
    // the level sizes, entry counts and runs: fixed by the factor (the order of the rows inside a level, and so
    // the chunk boundaries, may differ from one factorization to the next; the widths are chosen per level)
    mix((uint64_t)F.nnz);
    mix((uint64_t)F.num_levels);
    mix((uint64_t)F.last_fwd_nnz);
    mix((uint64_t)F.last_bwd_nnz);
    for (int32_t v : F.level_ptr) mix((uint64_t)(uint32_t)v);
    mix((uint64_t)F.tail_rows);
    return h;
}

static void count_trsv_widths(const DevFactor& F, const TrsvShapes& sh, const TrsvPlan& P, PcgReport& rep) {
    for (int i = 0; i < 3; i++) rep.trsv_levels[i] = 0;
    for (const auto& s : P.fw)
        if (!s.rounds && F.fchunk_lvl[s.l1] > F.fchunk_lvl[s.l0]) rep.trsv_levels[sh.fw[s.l0]]++;
    for (const auto& s : P.bw)
        if (!s.rounds && F.bchunk_lvl[s.l1] > F.bchunk_lvl[s.l0]) rep.trsv_levels[sh.bw[s.l0]]++;
}

static TrsvShapes rule_shapes(const DevFactor& F, int ntiles, bool narrow) {
    TrsvShapes s;
    s.fw.resize(F.num_levels);
    for (int32_t l = 0; l < F.num_levels; l++) s.fw[l] = (uint8_t)rule_code(F, l, ntiles, narrow);
    s.bw = s.fw;
    return s;
}
static TrsvShapes forced_shapes(const DevFactor& F, int code) {
    TrsvShapes s;
    s.fw.assign(F.num_levels, (uint8_t)std::min(code, TRSV_NWIDTH - 1));
    s.bw = s.fw;
    return s;
}

// per level and direction, the width with the smallest time in ev[c] (one measured application per width
// code c); the rule's width unless another is faster
static void shapes_from_events(const DevFactor& F, int ntiles, const LevelEvents* ev, int nw, TrsvShapes& out) {
    const float INF = 3.0e38f;
    std::vector<float> best(2 * (size_t)F.num_levels * nw, INF);
    for (int c = 0; c < nw; c++) {
        const LevelEvents& L = ev[c];
        for (size_t i = 0; i < L.used; i++) {
            float t = 0;
            SSP_CUDA(cudaEventElapsedTime(&t, L.ev[2 * i], L.ev[2 * i + 1]));
            const size_t o = ((size_t)(L.tag[i].first ? 0 : 1) * F.num_levels + L.tag[i].second) * nw + c;
            best[o] = std::min(best[o], t);
        }
    }
    out.fw.assign(F.num_levels, 0);
    out.bw.assign(F.num_levels, 0);
    for (int dir = 0; dir < 2; dir++)
        for (int32_t l = 0; l < F.num_levels; l++) {
            const float* b = &best[((size_t)dir * F.num_levels + l) * nw];
            int pick = rule_code(F, l, ntiles, false);
            for (int c = 0; c < nw; c++)
                if (b[c] < b[pick]) pick = c;
            (dir == 0 ? out.fw : out.bw)[l] = (uint8_t)pick;
        }
}

// how a solve's level shapes are chosen: Forced and Cached fill store; Measure returns the cache key
enum class ShapeSource { Rule, Forced, Cached, Measure };
static ShapeSource trsv_shape_source(Context& C, const DevFactor& F, int64_t n, int64_t ld, int32_t kcols,
                                     size_t elem, bool segmented, TrsvShapes& store, uint64_t& key) {
    const bool narrow = TILE > NARROW_W && kcols <= NARROW_W;
    if (narrow || F.num_levels == 0) return ShapeSource::Rule;  // one width for all (8 columns)
    const char* fw = getenv("SSP_TRSV_WIDTH");
    if (fw && fw[0]) {
        const int w = atoi(fw);
        store = forced_shapes(F, w >= 32 ? 2 : w >= 16 ? 1 : 0);
        return ShapeSource::Forced;
    }
    const char* tn = getenv("SSP_TRSV_TUNE");
    if ((tn && tn[0] == '0') || n * ld < trsv_tune_min()) return ShapeSource::Rule;
    key = trsv_signature(F, n, ld, kcols, elem, segmented);
    for (auto& e : C.trsv_cache.entries)
        if (e.first == key) {
            store = e.second;
            return ShapeSource::Cached;
        }
    return ShapeSource::Measure;
}

static void cache_shapes(Context& C, uint64_t key, const TrsvShapes& s) {
    auto& E = C.trsv_cache.entries;
    if ((int)E.size() >= TRSV_CACHE_MAX) E.erase(E.begin());
    E.push_back({key, s});
}

static void report_shapes(PcgReport& rep, int32_t source, const DevFactor& F, const TrsvShapes& s, const TrsvPlan& P) {
    rep.trsv_shapes = source;
    count_trsv_widths(F, s, P, rep);
}

// Three applications, one per width, then the per-level choice (the stage entry point's measurement).
template <class T>
static void tune_trsv_shapes(Context& C, const DevFactor& F, const TrsvPlan& P, const FactorVals<T>& V, int64_t n,
                             const T* r, T* y, int64_t ld, int32_t kcols, const RowAct& ra, TrsvShapes& out) {
    LevelEvents ev[3];
    for (int c = 0; c < TRSV_NWIDTH; c++) {
        const TrsvShapes f = forced_shapes(F, c);
        C.kernels_launched += launch_precond<T>(C, F, P, V, n, r, y, ld, kcols, ra, &f, &ev[c]);
    }
    SSP_CUDA(cudaStreamSynchronize(C.stream));
    shapes_from_events(F, (int)(ld / TILE), ev, TRSV_NWIDTH, out);
}

// The preconditioner application as a CUDA graph, with its level shapes.  measure: the shapes are still to be
// measured by the solve's next applications (pcg_solve), after which the graph is captured anew.
struct Precond {
    cudaGraph_t graph = nullptr;
    cudaGraphExec_t exec = nullptr;
    TrsvShapes shapes;
    bool planned = false;
    bool has_shapes = false;
    bool measure = false;
    uint64_t key = 0;
    TrsvPlan plan;                 // which levels are walked
    int mstep = 0;                 // widths measured so far
    LevelEvents mev[3];            // their level launches
    cudaEvent_t m0 = nullptr, m1 = nullptr;  // around the measured applications
    void drop_graph() {
        if (exec) cudaGraphExecDestroy(exec);
        if (graph) cudaGraphDestroy(graph);
        exec = nullptr;
        graph = nullptr;
    }
    ~Precond() {
        drop_graph();
        if (m0) cudaEventDestroy(m0);
        if (m1) cudaEventDestroy(m1);
    }
};

// ---------------------------------------------------------------- SpMM plan
// The Laplacian as the SpMM reads it.  When one tile of the gathered operand (n rows of TILE values) is
// far larger than L2 and the matrix has no locality to exploit (random graphs: a row's neighbours are
// anywhere), the columns are cut into nslabs equal ranges and the entries stored slab-major: slab b,
// row i holds row i's entries with a column in slab b, in their stored order, at ptr[b n + i] ..
// ptr[b n + i + 1].  The SpMM then makes one pass per slab (the first writes q, the others add into it),
// and each pass gathers from a 1/nslabs share of the tile that stays resident in L2; the price is
// 2 nslabs - 1 streaming passes over q instead of 1.  Measured on B200 (ER n = 1M, average degree 20,
// 1327 columns, FP64): one pass 39.5 ms; 3, 4, 6, 8, 11 slabs 48.0, 52.6, 63.4, 75.4, 93.7 ms -- the extra q
// passes cost more than the L2 hits save, so slabs are off unless SSP_SPMM_SLAB_MB (the L2 share of one
// slab, MB) asks for them.
constexpr int MAX_SLABS = 16;

double spmm_slab_mb() {
    const char* e = getenv("SSP_SPMM_SLAB_MB");
    return e ? atof(e) : 0.0;
}

struct SpmmPlan {
    int32_t nslabs = 1;
    int64_t nnz = 0;
    const int64_t* ptr = nullptr;  // nslabs * n + 1 row pointers
    const int32_t* idx = nullptr;
    const double* val = nullptr;  // FP64 values in this entry order
    SpmmItems items[MAX_SLABS];   // of each slab
    dim3 grid;                    // of k_spmm
    unsigned long_blocks = 0;     // x blocks of k_spmm_long for the last slab (p.q partials follow the grid's)
    int nparts = 0;               // partials of p.q per column
    int launches = 0;             // of one product
    bool segs = false;            // rows (their share of a slab) hold more than SPMM_SEG entries on average
    // Sums of the long rows' segments (both precisions), for `group` tiles at a time: as many as fit half an n x ld block,
    // one at least.  At 1000 entries a row the segments of all columns would be five blocks beside the solve's six.
    double* lpart = nullptr;
    int group = 1;
    double* part = nullptr;
};

// entries farther than `window` from the diagonal, summed per block into *far
__global__ void k_far_count(int64_t n, const int64_t* __restrict__ ptr, const int32_t* __restrict__ idx,
                            int64_t window, unsigned long long* far) {
    __shared__ unsigned long long s_far;
    if (threadIdx.x == 0) s_far = 0;
    __syncthreads();
    const int lane = threadIdx.x & 31;
    const int64_t i = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    unsigned c = 0;
    if (i < n)
        for (int64_t e = ptr[i] + lane; e < ptr[i + 1]; e += 32) c += llabs((int64_t)idx[e] - i) > window;
    for (int o = 16; o > 0; o >>= 1) c += __shfl_xor_sync(0xffffffffu, c, o);
    if (lane == 0 && c) atomicAdd(&s_far, (unsigned long long)c);
    __syncthreads();
    if (threadIdx.x == 0 && s_far) atomicAdd(far, s_far);
}

// per (slab, row) entry counts; one warp per row, lane b keeps slab b's count
__global__ void k_slab_count(int64_t n, const int64_t* __restrict__ ptr, const int32_t* __restrict__ idx,
                             int64_t slab_rows, int32_t nslabs, int32_t* __restrict__ cnt) {
    const int lane = threadIdx.x & 31;
    const int64_t i = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    if (i >= n) return;
    int32_t mine = 0;
    for (int64_t e0 = ptr[i]; e0 < ptr[i + 1]; e0 += 32) {
        const int64_t e = e0 + lane;
        const int b = e < ptr[i + 1] ? (int)(idx[e] / slab_rows) : -1;
        for (int s = 0; s < nslabs; s++) {
            const int c = __popc(__ballot_sync(0xffffffffu, b == s));
            if (lane == s) mine += c;
        }
    }
    if (lane < nslabs) cnt[(int64_t)lane * n + i] = mine;
}

// stable partition of each row's entries into the slab-major copy
__global__ void k_slab_fill(int64_t n, const int64_t* __restrict__ ptr, const int32_t* __restrict__ idx,
                            const double* __restrict__ val, int64_t slab_rows, int32_t nslabs,
                            const int64_t* __restrict__ sptr, int32_t* __restrict__ sidx,
                            double* __restrict__ sval) {
    const int lane = threadIdx.x & 31;
    const int64_t i = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    if (i >= n) return;
    int64_t base = lane < nslabs ? sptr[(int64_t)lane * n + i] : 0;  // lane b: next free slot of slab b
    const unsigned lt = (1u << lane) - 1u;
    for (int64_t e0 = ptr[i]; e0 < ptr[i + 1]; e0 += 32) {
        const int64_t e = e0 + lane;
        const bool in = e < ptr[i + 1];
        const int b = in ? (int)(idx[e] / slab_rows) : -1;
        for (int s = 0; s < nslabs; s++) {
            const unsigned bal = __ballot_sync(0xffffffffu, b == s);
            const int64_t at = __shfl_sync(0xffffffffu, base, s);
            if (b == s) {
                const int64_t pos = at + __popc(bal & lt);
                sidx[pos] = idx[e];
                sval[pos] = val[e];
            }
            if (lane == s) base += __popc(bal);
        }
    }
}

static int32_t spmm_slab_count(Context& C, int64_t n, const int64_t* ptr, const int32_t* idx, int64_t nnz) {
    const double mb = spmm_slab_mb();
    if (!(mb > 0) || nnz == 0) return 1;
    // slabs are cut for the FP64 operand (TILE doubles per row); FP32 solves use the same cut
    const int64_t slab_rows = std::max<int64_t>(1, (int64_t)(mb * 1048576.0 / (TILE * sizeof(double))));
    if (n <= slab_rows) return 1;
    unsigned long long* far = C.ws.get_t<unsigned long long>("pcg_slab_far", 1);
    SSP_CUDA(cudaMemsetAsync(far, 0, sizeof(unsigned long long), C.stream));
    k_far_count<<<(unsigned)ceil_div<int64_t>(n * 32, 256), 256, 0, C.stream>>>(n, ptr, idx, slab_rows / 2, far);
    SSP_CHECK_LAUNCH();
    C.kernels_launched++;
    // a matrix whose entries mostly sit near the diagonal already reuses L2 in a row sweep
    if (read_i64(C, reinterpret_cast<const int64_t*>(far)) * 4 < nnz) return 1;
    return (int32_t)std::min<int64_t>(MAX_SLABS, ceil_div<int64_t>(n, slab_rows));
}

static SpmmPlan make_spmm_plan(Context& C, int64_t n, const int64_t* lap_ptr, const int32_t* lap_idx,
                               const double* lap_val, int64_t ld) {
    Workspace& W = C.ws;
    SpmmPlan A;
    A.nnz = read_i64(C, lap_ptr + n);
    A.nslabs = spmm_slab_count(C, n, lap_ptr, lap_idx, A.nnz);
    const int32_t m = A.nslabs;
    if (m == 1) {
        A.ptr = lap_ptr;
        A.idx = lap_idx;
        A.val = lap_val;
    } else {
        const int64_t slab_rows = ceil_div<int64_t>(n, m);
        int32_t* cnt = W.get_t<int32_t>("pcg_slab_cnt", (size_t)m * n);
        int64_t* sptr = W.get_t<int64_t>("pcg_slab_ptr", (size_t)m * n + 1);
        int32_t* sidx = W.get_t<int32_t>("pcg_slab_idx", A.nnz + 1);
        double* sval = W.get_t<double>("pcg_slab_val", A.nnz + 1);
        const unsigned blocks = (unsigned)ceil_div<int64_t>(n * 32, 256);
        k_slab_count<<<blocks, 256, 0, C.stream>>>(n, lap_ptr, lap_idx, slab_rows, m, cnt);
        SSP_CHECK_LAUNCH();
        exclusive_scan_i32_to_i64(C, cnt, sptr, (int64_t)m * n, sptr + (int64_t)m * n);
        k_slab_fill<<<blocks, 256, 0, C.stream>>>(n, lap_ptr, lap_idx, lap_val, slab_rows, m, sptr, sidx, sval);
        SSP_CHECK_LAUNCH();
        C.kernels_launched += 2;
        A.ptr = sptr;
        A.idx = sidx;
        A.val = sval;
    }
    // per slab: the chunks, and the segments of the rows longer than one
    int32_t most = 0, most_seg = 0;
    for (int32_t b = 0; b < m; b++) {
        const DevChunks D = device_chunks(C, A.ptr + (int64_t)b * n, 0, (int32_t)n, "pcg_a" + std::to_string(b));
        SpmmItems& I = A.items[b];
        I.chunks = D.starts;
        I.nchunks = D.nchunks;
        I.nseg = D.nseg;
        I.seg = D.seg;
        I.segrow = D.segrow;
        I.nlong = D.nlong;
        I.lrow = D.lrow;
        I.lseg = D.lseg;
        most = std::max(most, I.nchunks + I.nseg);
        most_seg = std::max(most_seg, I.nseg);
    }
    const int bx = chunk_blocks(most);
    A.grid = dim3((unsigned)bx, (unsigned)(ld / TILE));
    const int32_t nl = A.items[m - 1].nlong;
    A.long_blocks = nl ? (unsigned)std::min(ceil_div(nl, CH_WARPS), 64) : 0;
    A.nparts = bx + (int)A.long_blocks;
    A.segs = A.nnz > (int64_t)SPMM_SEG * n * m;
    const int ntiles = (int)(ld / TILE);
    A.group = ntiles;
    if (most_seg) {
        A.group = (int)std::max<int64_t>(1, std::min<int64_t>(ntiles, n * ld / 2 / ((int64_t)most_seg * TILE)));
        A.lpart = W.get_t<double>("pcg_lpart", (size_t)most_seg * A.group * TILE);
    }
    for (int32_t b = 0; b < m; b++) A.launches += A.items[b].nlong > 0 ? 2 * ceil_div(ntiles, A.group) : 1;
    A.part = W.get_t<double>("pcg_spmm_part", (size_t)A.nparts * ld);
    return A;
}

// SpMM q = A p over the plan's slabs (+ p.q partials into A.part when dot)
template <class T>
static void launch_spmm(Context& C, int64_t n, const SpmmPlan& A, const T* aval, const T* p, T* q, int64_t ld,
                        bool dot, int32_t kcols, const RowAct& ra = RowAct()) {
    const bool narrow = TILE > NARROW_W && kcols <= NARROW_W;
    T* lpart = reinterpret_cast<T*>(A.lpart);
    for (int32_t b = 0; b < A.nslabs; b++) {
        const SpmmItems& I = A.items[b];
        const int64_t* ptr = A.ptr + (int64_t)b * n;
        double* part = dot && b == A.nslabs - 1 ? A.part : nullptr;
        auto pick = [&](auto segs) {
            constexpr bool S = decltype(segs)::value;
            return narrow ? (b == 0 ? k_spmm<T, NARROW_W, false, S> : k_spmm<T, NARROW_W, true, S>)
                          : (b == 0 ? k_spmm<T, TILE, false, S> : k_spmm<T, TILE, true, S>);
        };
        auto kern = A.segs ? pick(std::true_type()) : pick(std::false_type());
        const int ntiles = (int)A.grid.y, group = I.nlong ? A.group : ntiles;
        const int64_t lld = (int64_t)A.group * TILE;
        const unsigned lx = part ? A.long_blocks : (unsigned)std::min(ceil_div(I.nlong, CH_WARPS), 64);
        auto fin = b == 0 ? k_spmm_long<T, false> : k_spmm_long<T, true>;
        for (int t0 = 0; t0 < ntiles; t0 += group) {
            // the kernels count tiles and columns from the group's first
            const unsigned nt = (unsigned)std::min(group, ntiles - t0);
            const int64_t o = (int64_t)t0 * n * TILE;
            const int32_t kc = kcols - t0 * TILE;
            RowAct rg = ra;
            if (rg.act) rg.act += t0;
            double* pt = part ? part + t0 * TILE : nullptr;
            kern<<<dim3(A.grid.x, nt), CH_THREADS, 0, C.stream>>>(n, I, ptr, A.idx, aval, p + o, q + o, ld, lpart, lld, pt, kc, rg);
            if (I.nlong == 0) continue;
            fin<<<dim3(lx, nt), CH_THREADS, 0, C.stream>>>(n, I, lpart, lld, p + o, q + o, ld,
                                                           pt ? pt + (int64_t)A.grid.x * ld : nullptr, kc, rg);
        }
    }
}

// One preconditioner application from the solve's r into its z with the given level shapes (nullptr: the rule)
// and optional events around each level launch; returns the kernels it launched.
using PcApply = std::function<int64_t(const TrsvShapes*, LevelEvents*)>;

// P's graph: one application with P's shapes (the rule when it has none)
static void capture_precond(Context& C, Precond& P, int64_t& launches, const PcApply& pc) {
    P.drop_graph();
    SSP_CUDA(cudaStreamBeginCapture(C.stream, cudaStreamCaptureModeThreadLocal));
    try {
        launches = pc(P.has_shapes ? &P.shapes : nullptr, nullptr);
    } catch (...) {
        cudaGraph_t g;
        cudaStreamEndCapture(C.stream, &g);
        if (g) cudaGraphDestroy(g);
        throw;
    }
    SSP_CUDA(cudaStreamEndCapture(C.stream, &P.graph));
    SSP_CUDA(cudaGraphInstantiate(&P.exec, P.graph, 0));
}

// The solve's preconditioner: its level shapes (forced, cached, the rule, or the rule until the solve's first
// applications have measured them).  Its graph is captured by the first application that launches one (pcg_solve).
template <class T>
static void plan_precond(Context& C, const DevFactor& F, const FactorVals<T>& V, int64_t n, int64_t ld, int32_t kcols,
                         Precond& P, PcgReport& rep, const RowAct& ra, int verbose) {
    TrsvShapes store;
    uint64_t key = 0;
    const bool narrow = TILE > NARROW_W && kcols <= NARROW_W;
    const ShapeSource src = trsv_shape_source(C, F, n, ld, kcols, sizeof(T), ra.act != nullptr, store, key);
    P.plan = make_trsv_plan<T>(C, F, V, (int)(ld / TILE), narrow, sizeof(T) == sizeof(float) ? "pcg32" : "pcg");
    P.measure = false;
    P.has_shapes = src == ShapeSource::Forced || src == ShapeSource::Cached;
    if (P.has_shapes) {
        P.shapes = store;
        report_shapes(rep, src == ShapeSource::Forced ? SSP_TRSV_FORCED : SSP_TRSV_CACHED, F, store, P.plan);
    } else {
        report_shapes(rep, SSP_TRSV_RULE, F, rule_shapes(F, (int)(ld / TILE), narrow), P.plan);
        if (src == ShapeSource::Measure) {
            P.measure = true;
            P.key = key;
            P.mstep = 0;
        }
    }
    if (verbose) {
        int32_t walked = 0, launched = 0;
        for (const auto* v : {&P.plan.fw, &P.plan.bw})
            for (const TrsvSeg& g : *v) (g.rounds ? walked : launched) += g.l1 - g.l0;
        const WalkShape& w = P.plan.walk;
        fprintf(stderr, "[ssp] triangular solves%s: %d levels walked (%d columns, %d threads, clusters of %d), %d launched, "
                "dense tail of %d\n", sizeof(T) == 4 ? " (fp32)" : "", walked, w.W, w.NT, w.cl, launched,
                P.plan.tail ? F.tail_rows : 0);
    }
    P.planned = true;
    P.drop_graph();
}

static FactorVals<double> fp64_vals(Context& C, const DevFactor& F, int64_t ld) {
    FactorVals<double> V{F.prow_val, F.pcol_val, F.D};
    if (F.extras(C) && F.tail_rows) {
        V.tin_val = F.tin_val;
        V.linv = F.linv;
        V.tail_tmp = C.ws.get_optional_t<double>("pcg_tail", (size_t)F.tail_rows * ld);
    }
    if (F.extras(C) && F.frow && F.brow) {
        V.fent = F.fent;
        V.bent = F.bent;
    }
    return V;
}
// The factor's values rounded to FP32, in workspace buffers named after tag: the caller gets the first 2 nnz + n (f32_base)
// before it needs the memory for anything optional.
static float* f32_base(Context& C, const DevFactor& F, int64_t n, const std::string& tag) {
    return C.ws.get_t<float>(tag + "_fval", 2 * F.nnz + n + 1);
}
static FactorVals<float> fp32_vals(Context& C, const DevFactor& F, int64_t n, int64_t ld, float* base,
                                   const std::string& tag) {
    auto put = [&](int64_t cnt, const double* src, float* dst) {
        if (cnt <= 0) return;
        k_d2f<<<grid_for(cnt, 256, 148 * 16), 256, 0, C.stream>>>(cnt, src, dst);
        SSP_CHECK_LAUNCH();
        C.kernels_launched++;
    };
    FactorVals<float> V{base, base + F.nnz, base + 2 * F.nnz};
    put(F.nnz, F.prow_val, base);
    put(F.nnz, F.pcol_val, base + F.nnz);
    put(n, F.D, base + 2 * F.nnz);
    if (F.extras(C) && F.tail_rows) {
        const int64_t T = F.tail_rows;
        float* f = C.ws.get_optional_t<float>(tag + "_ftail", F.tin_nnz + T * T + 1);
        float* tmp = f ? C.ws.get_optional_t<float>(tag + "_tail", (size_t)T * ld) : nullptr;
        if (tmp) {
            put(F.tin_nnz, F.tin_val, f);
            put(T * T, F.linv, f + F.tin_nnz);
            V.tin_val = f;
            V.linv = f + F.tin_nnz;
            V.tail_tmp = tmp;
        }
    }
    const bool ents = F.extras(C) && F.frow && F.brow && F.fent && F.bent;
    FactorEnt<float>* e = ents ? C.ws.get_optional_t<FactorEnt<float>>(tag + "_ent", 2 * F.nnz + 1) : nullptr;
    if (e) {
        if (F.nnz > 0) {
            const int g = grid_for(F.nnz, 256, 148 * 16);
            k_ent_f32<<<g, 256, 0, C.stream>>>(F.nnz, F.fent, e);
            k_ent_f32<<<g, 256, 0, C.stream>>>(F.nnz, F.bent, e + F.nnz);
            SSP_CHECK_LAUNCH();
            C.kernels_launched += 2;
        }
        V.fent = e;
        V.bent = e + F.nnz;
    }
    return V;
}

// apply M^{-1} to R into Z once (tile-major n x ld blocks; stage entry point).  When the shapes are to be
// measured, one application per width measures them first (each writes the same Z).
void precond_apply_device(Context& C, const DevFactor& F, const double* R, double* Z, int64_t ld) {
    TrsvShapes store;
    uint64_t key = 0;
    const ShapeSource src = trsv_shape_source(C, F, F.n, ld, (int32_t)ld, sizeof(double), false, store, key);
    const FactorVals<double> V = fp64_vals(C, F, ld);
    const Workspace::KeepOptional keep(C.ws);
    const TrsvPlan P = make_trsv_plan<double>(C, F, V, (int)(ld / TILE), TILE > NARROW_W && ld <= NARROW_W, "pcg");
    const TrsvShapes* sh = nullptr;
    if (src == ShapeSource::Forced || src == ShapeSource::Cached) {
        sh = &store;
    } else if (src == ShapeSource::Measure) {
        tune_trsv_shapes<double>(C, F, P, V, F.n, R, Z, ld, (int32_t)ld, RowAct(), store);
        cache_shapes(C, key, store);
        sh = &store;
    }
    int64_t l = launch_precond<double>(C, F, P, V, F.n, R, Z, ld, (int32_t)ld, RowAct(), sh);
    C.kernels_launched += l;
}

// ---------------------------------------------------------------- per-kernel event timing
struct EventPairs {
    std::vector<cudaEvent_t> a, b;
    size_t used = 0;
    ~EventPairs() {
        for (auto e : a) cudaEventDestroy(e);
        for (auto e : b) cudaEventDestroy(e);
    }
    void begin(cudaStream_t s) {
        if (used == a.size()) {
            cudaEvent_t x, y;
            SSP_CUDA(cudaEventCreate(&x));
            SSP_CUDA(cudaEventCreate(&y));
            a.push_back(x);
            b.push_back(y);
        }
        SSP_CUDA(cudaEventRecord(a[used], s));
    }
    void end(cudaStream_t s) { SSP_CUDA(cudaEventRecord(b[used++], s)); }
    double total_ms() {
        double t = 0;
        for (size_t i = 0; i < used; i++) {
            float x = 0;
            cudaEventElapsedTime(&x, a[i], b[i]);
            t += x;
        }
        return t;
    }
};

// ---------------------------------------------------------------- one PCG solve in one precision
template <class T>
struct PcgBufs {
    T* e;  // solution increment (zero on entry)
    T* r;  // right-hand side on entry, residual on exit
    T* z;
    T* p;
    T* q;
};

struct PcgTimers {
    EventPairs spmm, pc, loop;
};

// Runs PCG on A e = r for every column that S marks active (S.thr, S.active, S.nactive set by the
// caller; e zero).  Returns the iterations of the loop.
template <class T>
static int32_t pcg_solve(Context& C, int64_t n, int32_t k, int64_t ld, const SpmmPlan& A, const T* aval,
                         const DevFactor& F, const PcApply& pc,
                         Precond& P, int64_t& pc_launches, PcgBufs<T> B, ColState& S, Reducer& R,
                         int32_t max_iters, const PcgOptions& opt, PcgTimers& tm, PcgReport& rep,
                         const RowAct& ra = RowAct()) {
    // without a residual history or progress output the iterations after the first run on the device
    // SSP_PCG_HOST_LOOP=1 keeps every iteration on the host loop (the same kernels, launched one by one), for
    // profilers that do not look inside conditional graph nodes
    static const bool host_loop = [] {
        const char* e = getenv("SSP_PCG_HOST_LOOP");
        return e && e[0] == '1';
    }();
    const bool seg_history = opt.segs && opt.segs->record_history;
    const bool device_loop = !opt.history && !seg_history && !opt.verbose && !host_loop;
    const int64_t ntiles = ld / TILE;
    const int64_t total = n * ld;
    const dim3 egrid((unsigned)std::max<int64_t>(1, std::min<int64_t>(ceil_div<int64_t>(n * TILE, 256),
                                                                      2048 / std::max<int64_t>(1, ntiles) + 4)),
                     (unsigned)ntiles);
    const dim3 vgrid((unsigned)std::max<int64_t>(1, std::min<int64_t>(ceil_div<int64_t>(n * TILE, 256 * Vec<T>::V),
                                                                      2048 / std::max<int64_t>(1, ntiles) + 4)),
                     (unsigned)ntiles);
    const SegDev& G = R.G;
    const int64_t ns = (int64_t)G.nseg * ld;  // per-(graph, column) state entries
    const int cg = grid_for(ns, 256);
    // with several graphs the SpMM's blocks straddle graphs, so p.q is a segmented reduction of its own
    auto pq_dot = [&]() {
        if (G.nseg > 1) R.run<OP_DOT, T>(B.p, B.q, S.pq);
        else colred_final(C, ld, A.nparts, A.part, S.pq);
    };
    // which (graph, tile) pairs still have an active column: the row kernels skip the others
    auto update_act = [&]() {
        if (!ra.act) return;
        k_seg_tile_active<<<grid_for((int64_t)G.nseg * ntiles, 256), 256, 0, C.stream>>>(G.nseg, (int32_t)ntiles, ld,
                                                                                        S.active, (int32_t*)ra.act);
        C.kernels_launched++;
    };
    // one preconditioner application: the graph, or while the level shapes are being measured, one width's
    // launches with events around each level (a real application: every width gives the same values)
    auto apply_precond = [&]() {
        tm.pc.begin(C.stream);
        if (P.measure && P.mstep < TRSV_NWIDTH) {
            if (P.mstep == 0) {
                if (!P.m0) SSP_CUDA(cudaEventCreate(&P.m0));
                if (!P.m1) SSP_CUDA(cudaEventCreate(&P.m1));
                SSP_CUDA(cudaEventRecord(P.m0, C.stream));
            }
            const TrsvShapes f = forced_shapes(F, P.mstep);
            C.kernels_launched += pc(&f, &P.mev[P.mstep]);
            if (++P.mstep == TRSV_NWIDTH) SSP_CUDA(cudaEventRecord(P.m1, C.stream));
        } else if (device_loop) {
            // launched once before the loop's own graph takes over: capturing it costs more than its launches
            C.kernels_launched += pc(P.has_shapes ? &P.shapes : nullptr, nullptr);
        } else {
            if (!P.exec) capture_precond(C, P, pc_launches, pc);
            SSP_CUDA(cudaGraphLaunch(P.exec, C.stream));
            C.kernels_launched += pc_launches;
        }
        tm.pc.end(C.stream);
    };
    // after a synchronization that follows the last measured application: keep the fastest width per level,
    // cache it, and drop the graph that lacks it
    auto finish_measure = [&]() {
        if (!P.measure || P.mstep < TRSV_NWIDTH) return;
        shapes_from_events(F, (int)ntiles, P.mev, TRSV_NWIDTH, P.shapes);
        float ms = 0;
        SSP_CUDA(cudaEventElapsedTime(&ms, P.m0, P.m1));
        rep.ms_trsv_tune += ms;
        P.has_shapes = true;
        P.measure = false;
        cache_shapes(C, P.key, P.shapes);
        report_shapes(rep, SSP_TRSV_TUNED, F, P.shapes, P.plan);
        P.drop_graph();
    };
    int64_t active = read_i64(C, S.nactive);
    int32_t it = 0;
    if (active == 0) return 0;
    update_act();
    apply_precond();
    R.run<OP_DOT, T>(B.r, B.z, S.rz);
    SSP_CUDA(cudaMemcpyAsync(B.p, B.z, sizeof(T) * total, cudaMemcpyDeviceToDevice, C.stream));
    const bool history = opt.history || seg_history;
    double* d_hist = history ? C.ws.get_t<double>("pcg_hist", (size_t)max_iters * (G.nseg + 1)) : nullptr;
    tm.loop.begin(C.stream);
    while (it < max_iters) {
        tm.spmm.begin(C.stream);
        launch_spmm<T>(C, n, A, aval, B.p, B.q, ld, G.nseg == 1, k, ra);
        tm.spmm.end(C.stream);
        pq_dot();
        k_cols_alpha<<<cg, 256, 0, C.stream>>>(ns, S);
        k_axpy_r_rr<T><<<dim3((unsigned)R.nparts, (unsigned)ntiles), RED_THREADS, 0, C.stream>>>(
            n, S.alpha, B.q, B.r, R.rows_per_blk, ld, R.part, G);
        SSP_CHECK_LAUNCH();
        C.kernels_launched += 3 + A.launches;
        R.finish(S.rr);
        it++;
        SSP_CUDA(cudaMemsetAsync(S.nactive, 0, sizeof(int64_t), C.stream));
        k_cols_check<<<cg, 256, 0, C.stream>>>(ns, it, S);
        SSP_CHECK_LAUNCH();
        C.kernels_launched++;
        update_act();
        if (history) {
            k_hist<<<(unsigned)G.nseg, 32, 0, C.stream>>>(ld, S, d_hist + (int64_t)(it - 1) * (G.nseg + 1));
            SSP_CHECK_LAUNCH();
            C.kernels_launched++;
        }
        // A history's solve waits only at the end (or while it measures, or reports): iterations after the last column has
        // stopped change nothing (alpha is 0) and are dropped from the history below.
        if (!history || P.measure || opt.verbose) {
            active = read_i64(C, S.nactive);
            finish_measure();
        }
        if (opt.verbose && (it % 10 == 0 || active == 0))
            fprintf(stderr, "[ssp] pcg%s iter %d: %lld columns active\n", sizeof(T) == 4 ? " (fp32 inner)" : "", it,
                    (long long)active);
        if (active == 0) break;
        if (device_loop && !P.measure) break;
        apply_precond();
        R.run<OP_DOT, T>(B.r, B.z, S.rz_new);
        k_cols_beta<<<cg, 256, 0, C.stream>>>(ns, S);
        k_update_xp<T><<<vgrid, 256, 0, C.stream>>>(n, ld, S.alpha, S.beta, B.z, B.p, B.e, G);
        SSP_CHECK_LAUNCH();
        C.kernels_launched += 2;
    }
    if (history && it > 0) {
        std::vector<double> hh((size_t)it * (G.nseg + 1));
        SSP_CUDA(cudaMemcpyAsync(hh.data(), d_hist, sizeof(double) * hh.size(), cudaMemcpyDeviceToHost, C.stream));
        SSP_CUDA(cudaStreamSynchronize(C.stream));
        if (seg_history) opt.segs->history.resize(G.nseg);
        const int32_t ran = it;
        for (it = 0; it < ran;) {
            const double* e = hh.data() + (size_t)it * (G.nseg + 1);
            if (opt.history) opt.history->push_back(*std::max_element(e, e + G.nseg));
            for (int32_t sg = 0; seg_history && sg < G.nseg; sg++) opt.segs->history[sg].push_back(e[sg]);
            it++;
            active = (int64_t)e[G.nseg];
            if (active == 0) break;
        }
    }
    if (device_loop && active > 0 && it < max_iters) {
        // one iteration = preconditioner, r.z, beta, p update, SpMM, alpha, x/r update, check, control
        int32_t* d_it = C.ws.get_t<int32_t>("pcg_loop_it", 1);
        k_it_set<<<1, 1, 0, C.stream>>>(d_it, it);
        SSP_CHECK_LAUNCH();
        LoopGraph L;
        cudaGraphConditionalHandle h;
        const int64_t k_before = C.kernels_launched;
        int64_t body_kernels = 0;
        SSP_CUDA(cudaGraphCreate(&L.graph, 0));
        SSP_CUDA(cudaGraphConditionalHandleCreate(&h, L.graph, 0, cudaGraphCondAssignDefault));
        auto capture = [&](cudaGraph_t g, auto&& fn) {
            SSP_CUDA(cudaStreamBeginCaptureToGraph(C.stream, g, nullptr, nullptr, 0, cudaStreamCaptureModeThreadLocal));
            try {
                fn();
            } catch (...) {
                cudaGraph_t tmp;
                cudaStreamEndCapture(C.stream, &tmp);
                throw;
            }
            SSP_CUDA(cudaStreamEndCapture(C.stream, &g));
        };
        capture(L.graph, [&] {
            k_loop_ctl<<<1, 1, 0, C.stream>>>(h, S.nactive, d_it, max_iters);
            SSP_CHECK_LAUNCH();
        });
        size_t nn = 0;
        SSP_CUDA(cudaGraphGetNodes(L.graph, nullptr, &nn));
        std::vector<cudaGraphNode_t> roots(nn);
        SSP_CUDA(cudaGraphGetNodes(L.graph, roots.data(), &nn));
        cudaGraphNodeParams cp = {};
        cp.type = cudaGraphNodeTypeConditional;
        cp.conditional.handle = h;
        cp.conditional.type = cudaGraphCondTypeWhile;
        cp.conditional.size = 1;
        cudaGraphNode_t wnode;
        SSP_CUDA(cudaGraphAddNode(&wnode, L.graph, roots.data(), nn, &cp));
        capture(cp.conditional.phGraph_out[0], [&] {
            body_kernels += pc(P.has_shapes ? &P.shapes : nullptr, nullptr);
            R.run<OP_DOT, T>(B.r, B.z, S.rz_new);
            k_cols_beta<<<cg, 256, 0, C.stream>>>(ns, S);
            k_update_xp<T><<<vgrid, 256, 0, C.stream>>>(n, ld, S.alpha, S.beta, B.z, B.p, B.e, G);
            launch_spmm<T>(C, n, A, aval, B.p, B.q, ld, G.nseg == 1, k, ra);
            pq_dot();
            k_cols_alpha<<<cg, 256, 0, C.stream>>>(ns, S);
            k_axpy_r_rr<T><<<dim3((unsigned)R.nparts, (unsigned)ntiles), RED_THREADS, 0, C.stream>>>(
                n, S.alpha, B.q, B.r, R.rows_per_blk, ld, R.part, G);
            R.finish(S.rr);
            k_it_next<<<1, 1, 0, C.stream>>>(d_it);
            SSP_CUDA(cudaMemsetAsync(S.nactive, 0, sizeof(int64_t), C.stream));
            k_cols_check_at<<<cg, 256, 0, C.stream>>>(ns, d_it, S);
            update_act();
            k_loop_ctl<<<1, 1, 0, C.stream>>>(h, S.nactive, d_it, max_iters);
            SSP_CHECK_LAUNCH();
        });
        // the helpers count theirs; with several graphs p.q is a reduction (counted) instead of a final pass
        body_kernels += (C.kernels_launched - k_before) + 9 + A.launches - (G.nseg > 1 ? 1 : 0);
        C.kernels_launched = k_before;
        SSP_CUDA(cudaGraphInstantiate(&L.exec, L.graph, 0));
        SSP_CUDA(cudaGraphLaunch(L.exec, C.stream));
        int32_t it_end = it;
        SSP_CUDA(cudaMemcpyAsync(&it_end, d_it, sizeof(int32_t), cudaMemcpyDeviceToHost, C.stream));
        SSP_CUDA(cudaStreamSynchronize(C.stream));
        C.kernels_launched += 1 + body_kernels * (int64_t)(it_end - it);
        it = it_end;
    }
    // the last step's x += alpha p (alpha is 0 for columns that stopped earlier)
    k_axpy_x<T><<<egrid, 256, 0, C.stream>>>(n, ld, S.alpha, B.p, B.e, G);
    SSP_CHECK_LAUNCH();
    C.kernels_launched++;
    tm.loop.end(C.stream);
    return it;
}

// ---------------------------------------------------------------- driver
// Y: tile-major n x ld (ld = round8(k)), read only.  The solution stays in the workspace buffer
// "pcg_x" (tile-major); *x_out points at it.
void pcg_device(Context& C, int64_t n, const int64_t* lap_ptr, const int32_t* lap_idx, const double* lap_val,
                const DevFactor& F, const double* Y, int32_t k, const double** x_out, const PcgOptions& opt,
                PcgReport& rep, int32_t* h_iters, double* h_relres, const int32_t* lap_eid, double* d2,
                bool d2_accumulate) {
    SSP_REQUIRE(k > 0, SSP_ERR_INVALID, "pcg: k must be positive");
    const bool mixed = opt.precision == SSP_PRECISION_MIXED;
    SSP_REQUIRE(mixed || opt.precision == SSP_PRECISION_FP64 || opt.precision == SSP_PRECISION_PC32, SSP_ERR_INVALID,
                "pcg: unknown precision");
    const int64_t ld = ((int64_t)k + TILE - 1) / TILE * TILE;
    const int64_t ntiles = ld / TILE;
    const int64_t total = n * ld;
    Workspace& W = C.ws;
    double* x = W.get_t<double>("pcg_x", total);
    double* r = W.get_t<double>("pcg_r", total);
    double* z = W.get_t<double>("pcg_z", total);
    double* p = W.get_t<double>("pcg_p", total);
    double* q = W.get_t<double>("pcg_q", total);
    // (pcg_solve's small buffers, before the optional ones are in use)
    W.get_t<int32_t>("pcg_loop_it", 1);
    // graphs solved at once (one segment: a single graph)
    SegDev G;
    PcgSegments* segs = opt.segs;
    if (opt.history || (segs && segs->record_history))
        W.get_t<double>("pcg_hist", (size_t)opt.max_iters * ((segs ? segs->k.size() : 1) + 1));
    if (segs) {
        const int32_t nseg = (int32_t)segs->k.size();
        SSP_REQUIRE(nseg >= 1 && (int64_t)segs->row0.size() == nseg + 1 && segs->row0.front() == 0 &&
                        segs->row0.back() == n && segs->rowseg,
                    SSP_ERR_INVALID, "pcg: inconsistent graph segments");
        std::vector<int64_t> rows(nseg);
        for (int32_t i = 0; i < nseg; i++) {
            SSP_REQUIRE(segs->k[i] >= 1 && segs->k[i] <= k && segs->row0[i + 1] > segs->row0[i], SSP_ERR_INVALID,
                        "pcg: a graph segment needs rows and 1..k columns");
            rows[i] = segs->row0[i + 1] - segs->row0[i];
        }
        int32_t* d_k = W.get_t<int32_t>("pcg_seg_k", nseg);
        int64_t* d_rows = W.get_t<int64_t>("pcg_seg_rows", nseg);
        SSP_CUDA(cudaMemcpyAsync(d_k, segs->k.data(), sizeof(int32_t) * nseg, cudaMemcpyHostToDevice, C.stream));
        SSP_CUDA(cudaMemcpyAsync(d_rows, rows.data(), sizeof(int64_t) * nseg, cudaMemcpyHostToDevice, C.stream));
        G.nseg = nseg;
        G.rowseg = segs->rowseg;
        G.kseg = d_k;
        G.segrows = d_rows;
    }
    const int64_t ns = (int64_t)G.nseg * ld;  // per-(graph, column) state entries
    ColState S = make_colstate(C, ns, "pcg");
    double* colv = W.get_t<double>("pcg_aux", 3 * ns);
    double* colsum = colv;
    double* relres = colv + ns;
    double* mean = colv + 2 * ns;
    Reducer R;
    R.init(C, n, ld, "pcg_red_part", G, segs ? &segs->row0 : nullptr);
    // SpMM: row-aligned chunks of the Laplacian (column slabs on large random graphs), about one wave of
    // blocks per tile
    const SpmmPlan A = make_spmm_plan(C, n, lap_ptr, lap_idx, lap_val, ld);
    const int64_t lap_nnz = A.nnz;
    const dim3 egrid((unsigned)std::max<int64_t>(1, std::min<int64_t>(ceil_div<int64_t>(n * TILE, 256),
                                                                      2048 / std::max<int64_t>(1, ntiles) + 4)),
                     (unsigned)ntiles);
    const int cg = grid_for(ns, 256);
    RowAct ra;
    if (G.nseg > 1) {
        ra.act = W.get_t<int32_t>("pcg_act", (size_t)G.nseg * ntiles);
        ra.rowseg = G.rowseg;
        ra.ntiles = (int32_t)ntiles;
    }

    // r = Y - mean(Y); x = 0; ||b||^2
    R.run<OP_SUM, double>(Y, nullptr, colsum);
    k_center<<<egrid, 256, 0, C.stream>>>(n, k, ld, Y, colsum, r, x, mean, R.G);
    SSP_CHECK_LAUNCH();
    C.kernels_launched++;
    R.run<OP_SQ, double>(r, nullptr, S.bnorm2);
    SSP_CUDA(cudaMemsetAsync(S.nactive, 0, sizeof(int64_t), C.stream));
    k_cols_init<<<cg, 256, 0, C.stream>>>(ld, k, opt.tol, opt.abs_tol, S, R.G);
    SSP_CHECK_LAUNCH();
    C.kernels_launched++;

    // a narrow solve leaves the padding columns of its gathered outputs untouched: start them at zero
    if (TILE > NARROW_W && k <= NARROW_W) {
        SSP_CUDA(cudaMemsetAsync(z, 0, sizeof(double) * total, C.stream));
        SSP_CUDA(cudaMemsetAsync(p, 0, sizeof(double) * total, C.stream));
        SSP_CUDA(cudaMemsetAsync(q, 0, sizeof(double) * total, C.stream));
    }
    PcgTimers tm;
    EventPairs ev_resid;
    int32_t it = 0;
    rep = PcgReport();
    if (!mixed) {
        Precond P;
        int64_t pc_launches = 0;
        if (read_i64(C, S.nactive) > 0) {
            PcApply pc;
            std::optional<Workspace::KeepOptional> keep;
            if (opt.precision == SSP_PRECISION_PC32 && !(TILE > NARROW_W && k <= NARROW_W)) {
                // FP64 PCG with the triangular solves in FP32: r rounded on the way in, z widened on the way out
                float* base = f32_base(C, F, n, "pcgp");
                const FactorVals<float> V32 = fp32_vals(C, F, n, ld, base, "pcgp");
                keep.emplace(W);
                // r32 and z32 live in q's memory: q (= A p) is dead from the r update to the next Laplacian
                // product, and the preconditioner runs in between, so this mode needs no more memory than FP64
                float* r32 = reinterpret_cast<float*>(q);
                float* z32 = r32 + total;
                const int cgrid = grid_for(total, 256, 148 * 16);
                pc = [&C, &F, &P, V32, n, r32, z32, r, z, ld, k, ra, total, cgrid](const TrsvShapes* sh, LevelEvents* lev) {
                    k_d2f<<<cgrid, 256, 0, C.stream>>>(total, r, r32);
                    const int64_t l = launch_precond<float>(C, F, P.plan, V32, n, r32, z32, ld, k, ra, sh, lev);
                    k_f2d<<<cgrid, 256, 0, C.stream>>>(total, z32, z);
                    SSP_CHECK_LAUNCH();
                    return l + 2;
                };
                plan_precond<float>(C, F, V32, n, ld, k, P, rep, ra, opt.verbose);
            } else {
                // (its scratch is allocated here: the applications are captured into graphs)
                const FactorVals<double> V64 = fp64_vals(C, F, ld);
                keep.emplace(W);
                pc = [&C, &F, &P, V64, n, r, z, ld, k, ra](const TrsvShapes* sh, LevelEvents* lev) {
                    return launch_precond<double>(C, F, P.plan, V64, n, r, z, ld, k, ra, sh, lev);
                };
                plan_precond<double>(C, F, V64, n, ld, k, P, rep, ra, opt.verbose);
            }
            it = pcg_solve<double>(C, n, k, ld, A, A.val, F, pc, P, pc_launches,
                                   PcgBufs<double>{x, r, z, p, q}, S, R, opt.max_iters, opt, tm, rep, ra);
        }
    } else {
        // FP32 copies of the Laplacian and factor values, and the FP32 inner vectors
        float* aval32 = W.get_t<float>("pcgm_aval", lap_nnz + 1);
        auto to_f32 = [&](int64_t count, const double* src, float* dst) {
            if (count <= 0) return;
            k_d2f<<<grid_for(count, 256, 148 * 16), 256, 0, C.stream>>>(count, src, dst);
            SSP_CHECK_LAUNCH();
            C.kernels_launched++;
        };
        to_f32(lap_nnz, A.val, aval32);
        float* base32 = f32_base(C, F, n, "pcgm");
        float* e32 = W.get_t<float>("pcgm_e", total);
        float* r32 = W.get_t<float>("pcgm_r", total);
        float* z32 = W.get_t<float>("pcgm_z", total);
        float* p32 = W.get_t<float>("pcgm_p", total);
        float* q32 = W.get_t<float>("pcgm_q", total);
        ColState Si = make_colstate(C, ns, "pcgm_in");
        double* worst = W.get_t<double>("pcgm_worst", 1);
        const FactorVals<float> V32 = fp32_vals(C, F, n, ld, base32, "pcgm");
        FactorVals<double> V64{};  // once a round falls back
        std::optional<Workspace::KeepOptional> keep(std::in_place, W);
        double* e64 = nullptr;  // FP64 inner increment, only if a round falls back
        Precond P32, P64;
        int64_t pc32 = 0, pc64 = 0;
        bool use64 = false;
        int32_t first_its = -1;
        int64_t active = read_i64(C, S.nactive);
        while (active > 0 && rep.refinements < MIXED_MAX_ROUNDS && it < opt.max_iters) {
            int32_t its;
            bool hit_cap = false;
            SSP_CUDA(cudaMemsetAsync(Si.nactive, 0, sizeof(int64_t), C.stream));
            if (!use64) {
                k_rhs_masked<float><<<egrid, 256, 0, C.stream>>>(n, ld, r, S.active, r32, R.G);
                SSP_CUDA(cudaMemsetAsync(e32, 0, sizeof(float) * total, C.stream));
                R.run<OP_SQ, float>(r32, nullptr, Si.bnorm2);
                k_cols_init_inner<<<cg, 256, 0, C.stream>>>(ld, k, MIXED_INNER_REDUCTION, S.thr, Si, R.G);
                SSP_CHECK_LAUNCH();
                C.kernels_launched += 2;
                const PcApply pc32f = [&C, &F, &P32, V32, n, r32, z32, ld, k, ra](const TrsvShapes* sh,
                                                                                   LevelEvents* lev) {
                    return launch_precond<float>(C, F, P32.plan, V32, n, r32, z32, ld, k, ra, sh, lev);
                };
                if (!P32.planned) plan_precond<float>(C, F, V32, n, ld, k, P32, rep, ra, opt.verbose);
                int32_t cap = opt.max_iters - it;
                if (first_its >= 0)
                    cap = std::min(cap, std::max(MIXED_MIN_ROUND_ITERS, MIXED_ROUND_ITER_FACTOR * first_its));
                else
                    cap = std::min(cap, std::max(MIXED_MIN_ROUND_ITERS, opt.max_iters / MIXED_FIRST_ROUND_DIV));
                its = pcg_solve<float>(C, n, k, ld, A, aval32, F, pc32f, P32, pc32,
                                       PcgBufs<float>{e32, r32, z32, p32, q32}, Si, R, cap, opt, tm, rep, ra);
                if (first_its < 0) first_its = its;
                hit_cap = its >= cap;
                k_add_into<float><<<grid_for(total, 256, 148 * 16), 256, 0, C.stream>>>(total, e32, x);
            } else {
                if (!e64) {
                    keep.reset();  // no FP32 round follows, so what they used may go
                    e64 = W.get_t<double>("pcgm_e64", total);
                    V64 = fp64_vals(C, F, ld);
                    keep.emplace(W);
                }
                // the FP64 inner solve runs in place on the residual of the active columns and goes straight
                // to (half) the outer threshold
                k_rhs_masked<double><<<egrid, 256, 0, C.stream>>>(n, ld, r, S.active, r, R.G);
                SSP_CUDA(cudaMemsetAsync(e64, 0, sizeof(double) * total, C.stream));
                R.run<OP_SQ, double>(r, nullptr, Si.bnorm2);
                k_cols_init_inner<<<cg, 256, 0, C.stream>>>(ld, k, 0.0, S.thr, Si, R.G);
                SSP_CHECK_LAUNCH();
                C.kernels_launched += 2;
                const PcApply pc64f = [&C, &F, &P64, V64, n, r, z, ld, k, ra](const TrsvShapes* sh, LevelEvents* lev) {
                    return launch_precond<double>(C, F, P64.plan, V64, n, r, z, ld, k, ra, sh, lev);
                };
                if (!P64.planned) plan_precond<double>(C, F, V64, n, ld, k, P64, rep, ra, opt.verbose);
                its = pcg_solve<double>(C, n, k, ld, A, A.val, F, pc64f, P64, pc64,
                                        PcgBufs<double>{e64, r, z, p, q}, Si, R, opt.max_iters - it, opt, tm, rep,
                                        ra);
                k_add_into<double><<<grid_for(total, 256, 148 * 16), 256, 0, C.stream>>>(total, e64, x);
                rep.fp64_rounds++;
            }
            SSP_CHECK_LAUNCH();
            C.kernels_launched++;
            it += its;
            rep.refinements++;
            // true residual with the FP64 matrix and FP64 x
            ev_resid.begin(C.stream);
            launch_spmm<double>(C, n, A, A.val, x, q, ld, false, k);
            ev_resid.end(C.stream);
            k_true_resid<<<dim3((unsigned)R.nparts, (unsigned)ntiles), RED_THREADS, 0, C.stream>>>(
                n, k, Y, mean, q, r, R.rows_per_blk, ld, R.part, R.G);
            SSP_CHECK_LAUNCH();
            C.kernels_launched += 1 + A.launches;
            R.finish(relres);
            SSP_CUDA(cudaMemsetAsync(S.nactive, 0, sizeof(int64_t), C.stream));
            SSP_CUDA(cudaMemsetAsync(worst, 0, sizeof(double), C.stream));
            k_cols_outer<<<cg, 256, 0, C.stream>>>(ns, Si.iters, relres, S, worst);
            SSP_CHECK_LAUNCH();
            C.kernels_launched++;
            active = read_i64(C, S.nactive);
            double hw = 0.0;
            SSP_CUDA(cudaMemcpyAsync(&hw, worst, sizeof(double), cudaMemcpyDeviceToHost, C.stream));
            SSP_CUDA(cudaStreamSynchronize(C.stream));
            if (opt.verbose)
                fprintf(stderr, "[ssp] refinement %d (%s inner, %d iterations): %lld columns active, worst ratio %.3g\n",
                        rep.refinements, use64 ? "fp64" : "fp32", its, (long long)active, hw);
            if (active > 0 && !use64 && (hw > MIXED_MIN_CONTRACTION || its == 0 || hit_cap)) use64 = true;
        }
    }
    // true relative residual ||(Y - mean) - A x|| / ||Y - mean|| (with the edges' squared diff norms when asked)
    if (lap_eid && d2 && A.nslabs == 1) {
        const SpmmItems& I = A.items[0];
        const int64_t lld = (int64_t)A.group * TILE;
        for (int64_t t = 0; t < ntiles; t++) {
            k_spmm_diff<<<dim3(A.grid.x, 1), CH_THREADS, 0, C.stream>>>(
                n, I, A.ptr, A.idx, A.val, lap_eid, x + t * n * TILE, q + t * n * TILE, (int32_t)(k - t * TILE), d2,
                (t == 0 && !d2_accumulate) ? 1 : 0, A.lpart ? A.lpart + t % A.group * TILE : nullptr, lld);
            C.kernels_launched++;
            // the group's long rows, once its last tile's segments are summed
            if (I.nlong == 0 || (t + 1 < ntiles && (t + 1) % A.group)) continue;
            const int64_t t0 = t / A.group * A.group;
            k_spmm_long<double, false><<<dim3(A.long_blocks, (unsigned)(t + 1 - t0)), CH_THREADS, 0, C.stream>>>(
                n, I, A.lpart, lld, x + t0 * n * TILE, q + t0 * n * TILE, ld, nullptr, (int32_t)(k - t0 * TILE), RowAct());
            C.kernels_launched++;
        }
        SSP_CHECK_LAUNCH();
        rep.diff_fused = true;
    } else {
        launch_spmm<double>(C, n, A, A.val, x, q, ld, false, k);
        SSP_CHECK_LAUNCH();
        C.kernels_launched += A.launches;
    }
    R.run<OP_SQDIFF_CENTERED, double>(Y, q, relres, mean);
    std::vector<double> hb(ns), hr(ns);
    std::vector<int32_t> hi(ns);
    SSP_CUDA(cudaMemcpyAsync(hb.data(), S.bnorm2, sizeof(double) * ns, cudaMemcpyDeviceToHost, C.stream));
    SSP_CUDA(cudaMemcpyAsync(hr.data(), relres, sizeof(double) * ns, cudaMemcpyDeviceToHost, C.stream));
    SSP_CUDA(cudaMemcpyAsync(hi.data(), S.iters, sizeof(int32_t) * ns, cudaMemcpyDeviceToHost, C.stream));
    SSP_CUDA(cudaStreamSynchronize(C.stream));
    double sum_it = 0;
    int64_t cols = 0;
    if (segs) {
        segs->iters.assign(ns, 0);
        segs->relres.assign(ns, 0.0);
    }
    for (int32_t sg = 0; sg < G.nseg; sg++) {
        const int32_t kk = segs ? segs->k[sg] : k;
        for (int32_t j = 0; j < kk; j++) {
            const int64_t o = (int64_t)sg * ld + j;
            double rel = hb[o] > 0 ? sqrt(hr[o]) / sqrt(hb[o]) : 0.0;
            if (h_relres && !segs) h_relres[j] = rel;
            if (h_iters && !segs) h_iters[j] = hi[o];
            if (segs) {
                segs->iters[o] = hi[o];
                segs->relres[o] = rel;
            }
            rep.max_iters_used = std::max(rep.max_iters_used, hi[o]);
            sum_it += hi[o];
            cols++;
            rep.max_relres = std::max(rep.max_relres, rel);
            if (!(rel < 0.01)) rep.not_converged++;
        }
    }
    rep.mean_iters = sum_it / std::max<int64_t>(1, cols);
    rep.ms_spmm = tm.spmm.total_ms();
    rep.n_spmm = (int64_t)tm.spmm.used;
    rep.ms_precond = tm.pc.total_ms();
    rep.n_precond = (int64_t)tm.pc.used;
    rep.ms_loop = tm.loop.total_ms();
    rep.ms_resid = ev_resid.total_ms();
    rep.n_resid = (int64_t)ev_resid.used;
    rep.iters_run = it;
    rep.spmm_slabs = A.nslabs;
    if (x_out) *x_out = x;
}

}  // namespace ssp
