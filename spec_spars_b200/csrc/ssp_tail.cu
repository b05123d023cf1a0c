// ssp_tail.cu -- the dense tail of a factor, solved as a dense matrix.
//
// Complete elimination ends in a dense tail: the last T vertices are eliminated one per level (ssp_factor.cu; the
// reference eliminates every vertex one after another, example.cc:332-471).  As a triangular solve that is a chain of
// up to T dependent rows, and however it is scheduled a step costs a few dependent L2 accesses.  The tail's block of
// L is unit lower triangular with -1 <= L <= 0 and column sums of at least -1, so the entries of its inverse are
// probabilities in [0, 1]: it is formed once per factor (T x T doubles) and the tail of every application is two
// dense triangular products, y = Linv r and z = Linv^T (D^+ y), with no chain at all.
//
// The figures of the whole application (tail and walked levels) stand at k_trsv_walk in ssp_pcg.cu; what the exact sums of
// tile_product add to it on B200: 3-D grid n = 80,840 (tail of 1007), 1085 columns, 4.65 -> 4.67 ms.
#include <algorithm>

#include "ssp_internal.cuh"

namespace ssp {

constexpr int TB = 32;            // tile edge of the products and of the inverted diagonal blocks
constexpr int TAIL_THREADS = 128;  // 2 x 4 outputs each

// entries of a tail row (storage rows r0 ..) whose column is eliminated before the tail (level < l0)
__global__ void k_tail_count(int32_t T, const int64_t* __restrict__ ptr, const int32_t* __restrict__ idx,
                             const int32_t* __restrict__ level, int32_t l0, int32_t* __restrict__ cnt) {
    const int lane = threadIdx.x & 31;
    const int64_t t = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    if (t >= T) return;
    int32_t c = 0;
    for (int64_t e = ptr[t] + lane; e < ptr[t + 1]; e += 32) c += level[idx[e]] < l0;
    for (int o = 16; o > 0; o >>= 1) c += __shfl_xor_sync(0xffffffffu, c, o);
    if (lane == 0) cnt[t] = c;
}

// those entries in their stored order, and the rest into the dense block (row t, column level - l0; 1 on the diagonal)
__global__ void k_tail_split(int32_t T, const int64_t* __restrict__ ptr, const int32_t* __restrict__ idx,
                             const double* __restrict__ val, const int32_t* __restrict__ level, int32_t l0,
                             const int64_t* __restrict__ tptr, int32_t* __restrict__ tidx, double* __restrict__ tval,
                             double* __restrict__ M) {
    const int lane = threadIdx.x & 31;
    const int64_t t = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    if (t >= T) return;
    int64_t at = tptr[t];
    for (int64_t e0 = ptr[t]; e0 < ptr[t + 1]; e0 += 32) {
        const int64_t e = e0 + lane;
        const bool in = e < ptr[t + 1];
        const int32_t v = in ? idx[e] : 0;
        const int32_t l = in ? level[v] : 0;
        const bool before = in && l < l0;
        const unsigned bal = __ballot_sync(0xffffffffu, before);
        if (before) {
            const int64_t p = at + __popc(bal & ((1u << lane) - 1u));
            tidx[p] = v;
            tval[p] = val[e];
        } else if (in) {
            M[t * T + (l - l0)] = val[e];
        }
        at += __popc(bal);
    }
    if (lane == 0) M[t * T + t] = 1.0;
}

// inverses of the 32 x 32 diagonal blocks, in place: lane j forms column j by forward substitution
__global__ void __launch_bounds__(32) k_tail_diag(int32_t T, double* __restrict__ M) {
    __shared__ double s[TB][TB + 1];
    const int64_t o = (int64_t)blockIdx.x * TB;
    const int nb = (int)min((int64_t)TB, T - o), j = threadIdx.x;
    for (int i = 0; i < nb; i++) s[i][j] = j < nb ? M[(o + i) * T + o + j] : 0.0;
    __syncwarp();
    double x[TB];
#pragma unroll
    for (int i = 0; i < TB; i++) {
        double a = i == j ? 1.0 : 0.0;
#pragma unroll
        for (int q = 0; q < TB; q++)
            if (q < i) a -= (i < nb ? s[i][q] : 0.0) * x[q];
        x[i] = i < j ? 0.0 : a;
    }
#pragma unroll
    for (int i = 0; i < TB; i++)
        if (i < nb && j < nb && j <= i) M[(o + i) * T + o + j] = x[i];
}

// One 32 x 32 output tile over k in [k0, k1): out = A(i, k) B(k, j), both fetched through the callers' accessors
// into shared memory (zero outside their ranges).  Thread (ti, tj) holds rows 2 ti, 2 ti + 1 and columns 4 tj ..+3.
//
// A sum has up to T terms where a triangular solve's rows have a few, so it is not one chain of additions: chains of
// SUM_CHAIN terms are added up exactly (Knuth's two-sum, its errors kept in lo) and rounded once.  The error against 64-bit
// arithmetic then does not grow with T and is that of a solve row by row; one chain was 3 to 15 times further off
// (tails of 246 and 1110 vertices, FP64 and FP32).
constexpr int SUM_CHAIN = 8;
template <class T, class FA, class FB>
__device__ __forceinline__ void tile_product(int64_t k0, int64_t k1, FA fa, FB fb, T (&out)[2][4]) {
    __shared__ T sa[TB][TB + 2];
    __shared__ __align__(16) T sb[TB][TB];
    const int ti = threadIdx.x / 8, tj = threadIdx.x % 8;
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    T ra[8], rb[8], hi[2][4] = {}, lo[2][4] = {};
    auto fetch = [&](int64_t k) {
#pragma unroll
        for (int u = 0; u < 8; u++) {
            ra[u] = fa(w + 4 * u, lane, k, k1);
            rb[u] = fb(w + 4 * u, lane, k, k1);
        }
    };
    if (k0 < k1) fetch(k0);
    for (int64_t k = k0; k < k1; k += TB) {
        __syncthreads();
#pragma unroll
        for (int u = 0; u < 8; u++) {
            sa[FA::row_of(w + 4 * u, lane)][FA::k_of(w + 4 * u, lane)] = ra[u];
            sb[w + 4 * u][lane] = rb[u];
        }
        __syncthreads();
        if (k + TB < k1) fetch(k + TB);
#pragma unroll 1
        for (int q0 = 0; q0 < TB; q0 += SUM_CHAIN) {
            T c[2][4] = {};
#pragma unroll
            for (int q = q0; q < q0 + SUM_CHAIN; q++) {
                const T a0 = sa[2 * ti][q], a1 = sa[2 * ti + 1][q];
#pragma unroll
                for (int j = 0; j < 4; j++) {
                    const T b = sb[q][4 * tj + j];
                    c[0][j] += a0 * b;
                    c[1][j] += a1 * b;
                }
            }
#pragma unroll
            for (int i = 0; i < 2; i++)
#pragma unroll
                for (int j = 0; j < 4; j++) {
                    const T h = hi[i][j], s = h + c[i][j], d = s - h;
                    lo[i][j] += (h - (s - d)) + (c[i][j] - d);
                    hi[i][j] = s;
                }
        }
    }
#pragma unroll
    for (int i = 0; i < 2; i++)
#pragma unroll
        for (int j = 0; j < 4; j++) out[i][j] = hi[i][j] + lo[i][j];
}

// A accessors: element (u, lane) of the 32 x 32 fetch is row u, column lane of A (row-major) or, transposed, row
// lane, column u -- coalesced along lane either way.
template <class T>
struct RowMajorA {
    const T* p;
    int64_t ld, rows;
    static __device__ __forceinline__ int row_of(int u, int) { return u; }
    static __device__ __forceinline__ int k_of(int, int lane) { return lane; }
    __device__ __forceinline__ T operator()(int u, int lane, int64_t k, int64_t k1) const {
        return u < rows && k + lane < k1 ? p[u * ld + k + lane] : (T)0;
    }
};
template <class T>
struct TransposedA {
    const T* p;
    int64_t ld, rows;
    static __device__ __forceinline__ int row_of(int, int lane) { return lane; }
    static __device__ __forceinline__ int k_of(int u, int) { return u; }
    __device__ __forceinline__ T operator()(int u, int lane, int64_t k, int64_t k1) const {
        return lane < rows && k + u < k1 ? p[(k + u) * ld + lane] : (T)0;
    }
};
template <class T>
struct RowMajorB {
    const T* p;
    int64_t ld, cols;
    __device__ __forceinline__ T operator()(int u, int lane, int64_t k, int64_t k1) const {
        return lane < cols && k + u < k1 ? p[(k + u) * ld + lane] : (T)0;
    }
};

// One doubling step of the inverse: for each pair of blocks of s rows with inverted diagonals Ainv (upper) and Cinv
// (lower), the block between them becomes -Cinv (N Ainv).  STEP 0 forms N Ainv in X, STEP 1 the rest in M.
template <int STEP>
__global__ void __launch_bounds__(TAIL_THREADS) k_tail_double(int64_t T, int64_t s, double* __restrict__ M,
                                                              double* __restrict__ X) {
    const int64_t o = (int64_t)blockIdx.z * 2 * s, c = o + s;  // first row of the upper and of the lower block
    const int64_t sc = min(s, T - c);
    const int64_t i0 = (int64_t)blockIdx.y * TB, j0 = (int64_t)blockIdx.x * TB;
    if (i0 >= sc || j0 >= s) return;
    double acc[2][4] = {};
    if (STEP == 0)
        tile_product<double>(j0, s, RowMajorA<double>{M + (c + i0) * T + o, T, sc - i0},
                             RowMajorB<double>{M + o * T + o + j0, T, s - j0}, acc);
    else
        tile_product<double>(0, min(i0 + TB, sc), RowMajorA<double>{M + (c + i0) * T + c, T, sc - i0},
                             RowMajorB<double>{X + c * T + o + j0, T, s - j0}, acc);
    const int ti = threadIdx.x / 8, tj = threadIdx.x % 8;
#pragma unroll
    for (int a = 0; a < 2; a++)
#pragma unroll
        for (int j = 0; j < 4; j++) {
            const int64_t i = i0 + 2 * ti + a, q = j0 + 4 * tj + j;
            if (i >= sc || q >= s) continue;
            if (STEP == 0) X[(c + i) * T + o + q] = acc[a][j];
            else M[(c + i) * T + o + q] = -acc[a][j];
        }
}

void build_tail(Context& C, DevFactor& F, int64_t T, double* X, const std::string& tag) {
    F.tail_rows = 0;
    if (T <= 0) return;
    Workspace& W = C.ws;
    const int64_t r0 = F.n - T;
    F.tail_l0 = F.num_levels - (int32_t)T;
    // Without the memory for it there is no dense tail: its levels are solved like the others.
    const Workspace::KeepOptional keep(W);
    double* M = W.get_optional_t<double>(tag + "_linv", (size_t)T * T);
    int32_t* cnt = W.get_optional_t<int32_t>(tag + "_tincnt", T + 1);
    F.tin_ptr = W.get_optional_t<int64_t>(tag + "_tinptr", T + 1);
    if (!M || !cnt || !F.tin_ptr) return;
    SSP_CUDA(cudaMemsetAsync(M, 0, sizeof(double) * T * T, C.stream));
    SSP_CUDA(cudaMemsetAsync(cnt + T, 0, sizeof(int32_t), C.stream));
    const unsigned wb = (unsigned)ceil_div<int64_t>(T * 32, 256);
    k_tail_count<<<wb, 256, 0, C.stream>>>((int32_t)T, F.prow_ptr + r0, F.prow_idx, F.level, F.tail_l0, cnt);
    SSP_CHECK_LAUNCH();
    exclusive_scan_i32_to_i64(C, cnt, F.tin_ptr, T + 1, nullptr);
    std::vector<int64_t> hp(T + 1);
    SSP_CUDA(cudaMemcpyAsync(hp.data(), F.tin_ptr, sizeof(int64_t) * (T + 1), cudaMemcpyDeviceToHost, C.stream));
    SSP_CUDA(cudaStreamSynchronize(C.stream));
    F.tin_nnz = hp[T];
    F.tin_idx = W.get_optional_t<int32_t>(tag + "_tinidx", F.tin_nnz + 1);
    F.tin_val = W.get_optional_t<double>(tag + "_tinval", F.tin_nnz + 1);
    if (!F.tin_idx || !F.tin_val) return;
    k_tail_split<<<wb, 256, 0, C.stream>>>((int32_t)T, F.prow_ptr + r0, F.prow_idx, F.prow_val, F.level, F.tail_l0,
                                           F.tin_ptr, F.tin_idx, F.tin_val, M);
    k_tail_diag<<<(unsigned)ceil_div<int64_t>(T, TB), 32, 0, C.stream>>>((int32_t)T, M);
    SSP_CHECK_LAUNCH();
    C.kernels_launched += 3;
    for (int64_t s = TB; s < T; s *= 2) {
        const unsigned b = (unsigned)ceil_div<int64_t>(s, TB);
        const dim3 grid(b, b, (unsigned)ceil_div<int64_t>(T - s, 2 * s));
        k_tail_double<0><<<grid, TAIL_THREADS, 0, C.stream>>>(T, s, M, X);
        k_tail_double<1><<<grid, TAIL_THREADS, 0, C.stream>>>(T, s, M, X);
        SSP_CHECK_LAUNCH();
        C.kernels_launched += 2;
    }
    std::vector<int32_t> ch;
    make_chunks(hp.data(), 0, (int32_t)T, ch);
    F.ntchunk = (int32_t)ch.size();
    ch.push_back((int32_t)T);
    F.tchunk = W.get_optional_t<int32_t>(tag + "_tinchunk", ch.size());
    if (!F.tchunk) return;
    SSP_CUDA(cudaMemcpyAsync(F.tchunk, ch.data(), sizeof(int32_t) * ch.size(), cudaMemcpyHostToDevice, C.stream));
    SSP_CUDA(cudaStreamSynchronize(C.stream));
    F.linv = M;
    F.tail_rows = (int32_t)T;
}

// The tail of one application, one 32-row block of one column tile per thread block.  Forward: tmp = D^+ (Linv y) for
// the tail rows of y (D^+ leaves a row with a zero pivot alone); backward: y = Linv^T tmp.  Grid (row blocks, tiles),
// the longest row blocks first.
template <class T, bool FWD>
__global__ void __launch_bounds__(TAIL_THREADS) k_tail_solve(int64_t n, int64_t nt, const T* __restrict__ Linv,
                                                             const int32_t* __restrict__ rows,
                                                             const T* __restrict__ D, T* __restrict__ y,
                                                             T* __restrict__ tmp) {
    constexpr int TILE = SSP_TILE;
    static_assert(TILE == TB, "one product tile per column tile");
    __shared__ int32_t s_row[TB];
    const int64_t t = blockIdx.y;
    const int64_t i0 = (FWD ? (int64_t)gridDim.x - 1 - blockIdx.x : (int64_t)blockIdx.x) * TB;
    T* yt = y + t * n * TILE;
    T* tt = tmp + t * nt * TILE;
    struct GatherB {
        const T* y;
        const int32_t* rows;
        __device__ __forceinline__ T operator()(int u, int lane, int64_t k, int64_t k1) const {
            return k + u < k1 ? y[(int64_t)rows[k + u] * TILE + lane] : (T)0;
        }
    };
    if (threadIdx.x < TB) s_row[threadIdx.x] = i0 + threadIdx.x < nt ? rows[i0 + threadIdx.x] : 0;
    T acc[2][4] = {};
    if (FWD)
        tile_product<T>(0, min(i0 + TB, nt), RowMajorA<T>{Linv + i0 * nt, nt, nt - i0}, GatherB{yt, rows}, acc);
    else
        tile_product<T>(i0, nt, TransposedA<T>{Linv + i0, nt, nt - i0}, RowMajorB<T>{tt, TILE, TILE}, acc);
    __syncthreads();
    const int ti = threadIdx.x / 8, tj = threadIdx.x % 8;
#pragma unroll
    for (int a = 0; a < 2; a++) {
        const int r = 2 * ti + a;
        if (i0 + r >= nt) continue;
        const int64_t v = s_row[r];
        const T d = FWD ? D[v] : (T)1;
#pragma unroll
        for (int j = 0; j < 4; j++) {
            const T x = acc[a][j];
            if (FWD) tt[(i0 + r) * TILE + 4 * tj + j] = d != (T)0 ? x / d : x;
            else yt[v * TILE + 4 * tj + j] = x;
        }
    }
}

template <class T>
int64_t launch_tail(Context& C, const DevFactor& F, const T* linv, const T* D, T* y, T* tmp, int64_t ntiles) {
    const int64_t nt = F.tail_rows;
    const dim3 grid((unsigned)ceil_div<int64_t>(nt, TB), (unsigned)ntiles);
    const int32_t* rows = F.level_rows + (F.n - nt);
    k_tail_solve<T, true><<<grid, TAIL_THREADS, 0, C.stream>>>(F.n, nt, linv, rows, D, y, tmp);
    k_tail_solve<T, false><<<grid, TAIL_THREADS, 0, C.stream>>>(F.n, nt, linv, rows, D, y, tmp);
    SSP_CHECK_LAUNCH();
    return 2;
}
template int64_t launch_tail<double>(Context&, const DevFactor&, const double*, const double*, double*, double*, int64_t);
template int64_t launch_tail<float>(Context&, const DevFactor&, const float*, const float*, float*, float*, int64_t);

}  // namespace ssp
