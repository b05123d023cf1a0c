// ssp_factor.cu -- a7: randomized approximate Cholesky of a graph Laplacian on the device.
//
// Per-column arithmetic restates perform_factorization_device (example.cc:188-300): the entries
// of the column (original lower entries plus fill) are merged by row (:209-235), sorted by value
// (:243) and prefix-summed (:248-258); every entry but the last picks a partner j > i with
// probability proportional to weight (:264-268) and emits fill (max(r_i,r_j), min(r_i,r_j)) of
// weight v_i (S - c_i) / S (:269-271); L entries are -v_i / S (:293, :437-446), D = S (:441).
//
// Schedule (this build): vertices are eliminated in increasing (Philox priority, id) order.  A
// vertex is ready once every neighbour with a smaller key has been eliminated, which is the
// reference's dependency-count scheme (example.cc:163-168,302-315) with a random instead of the
// natural order.  Every ready vertex of a level is eliminated in parallel; they are pairwise
// non-adjacent, so the factor equals sequential elimination in key order.  Once at most
// `dense_threshold` vertices are live at a level boundary, the live Schur complement is merged into
// a dense matrix and eliminated one vertex per level by a single block.  (The switch also waits for the
// frontier to collapse to at most 8 vertices, so sparse Schur complements stay in the sparse phase.)
//
// Every random draw is Philox(seed, column, slot); merges sort by (row, weight) and sum runs
// left to right; prefix sums are 32-wide Kogge-Stone chunks with a sequential carry.  Compiled
// with -fmad=false, so results are bit-identical to the CPU oracle.
#include "ssp_internal.cuh"
#include "ssp_sort.cuh"

namespace ssp {

enum { C_NEXT = 0, C_LCUR, C_FCUR, C_ERR, C_NB, C_NG, C_MAXLIVE, C_POOL, C_OWNERS, C_REM, C_NFILL, C_NCTR };
enum { FERR_POOL = 1, FERR_OVERFLOW = 2 };
enum { GC_FCUR = 0, GC_NFRONT = 1, GC_NFILL = 2 };

constexpr int BLOCK_TIER_MAX = 4096;    // live entries handled in shared memory
constexpr int DENSE_FRONTIER_MAX = 8;   // dense tail once the frontier has collapsed to this size

struct FDev {
    int64_t n;
    uint64_t seed;
    // several graphs factored at once: vbase[v] is the first vertex of v's graph, and every random draw is keyed
    // by the vertex's id inside its graph, so each graph's factor is the one it gets alone (null: one graph)
    const int32_t* vbase;
    // ... and vseg[v] its graph: per graph, gctr[3 g + GC_*] count the upcoming frontier's live entries and
    // vertices and the fill of the level just eliminated, for the truncation test of each graph
    const int32_t* vseg;
    int64_t* gctr;
    int32_t nseg;
    const uint64_t* prio;
    int32_t* count;
    int32_t* level;
    int64_t* bag_start;
    int32_t* bag_len;
    int32_t* bag_cap;
    int32_t* pool_u;
    double* pool_w;
    int64_t pool_cap;
    int64_t* ctr;
    int64_t* Lstart;
    int32_t* Lcnt;
    int32_t* Lrow;
    double* Lval;
    double* D;
    // per-level frontier data
    int64_t* fstart;  // [frontier idx] fill region start
    int32_t* fcnt;    // [frontier idx] fills emitted
    int32_t* fill_a;
    int32_t* fill_b;
    double* fill_w;
    int32_t* incoming;  // [vertex] fill entries of this level for its bag (0 between levels)
    int32_t* owners;    // the vertices of the level's fill
};

__device__ __forceinline__ bool key_less(const uint64_t* prio, int32_t a, int32_t b) {
    uint64_t pa = prio[a], pb = prio[b];
    return pa != pb ? pa < pb : a < b;
}

// ---------------------------------------------------------------- init
__device__ __forceinline__ int64_t local_vertex(const int32_t* vbase, int64_t v) { return vbase ? v - vbase[v] : v; }

__global__ void k_prio(int64_t n, uint64_t seed, uint64_t* prio, const int32_t* vbase) {
    for (int64_t v = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; v < n; v += (int64_t)gridDim.x * blockDim.x)
        prio[v] = vertex_priority(seed, local_vertex(vbase, v));
}

// lower entries (r > c, |val| != 0) counted for both endpoints
__global__ void k_lower_deg(int64_t n, const int64_t* colptr, const int32_t* rowidx, const double* val, int32_t* deg) {
    for (int64_t c = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; c < n; c += (int64_t)gridDim.x * blockDim.x) {
        int32_t cnt = 0;
        for (int64_t p = colptr[c]; p < colptr[c + 1]; p++) {
            int32_t r = rowidx[p];
            if (r > c && fabs(val[p]) != 0.0) {
                cnt++;
                atomicAdd(&deg[r], 1);
            }
        }
        atomicAdd(&deg[c], cnt);
    }
}

__global__ void k_bag_caps(int64_t n, const int32_t* deg, int32_t* cap) {
    for (int64_t v = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; v < n; v += (int64_t)gridDim.x * blockDim.x)
        cap[v] = 2 * deg[v] + 4;
}

__global__ void k_bag_fill(int64_t n, const int64_t* colptr, const int32_t* rowidx, const double* val, FDev F) {
    for (int64_t c = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; c < n; c += (int64_t)gridDim.x * blockDim.x) {
        for (int64_t p = colptr[c]; p < colptr[c + 1]; p++) {
            int32_t r = rowidx[p];
            double w = fabs(val[p]);
            if (r > c && w != 0.0) {
                int32_t s1 = atomicAdd(&F.bag_len[c], 1);
                F.pool_u[F.bag_start[c] + s1] = r;
                F.pool_w[F.bag_start[c] + s1] = w;
                int32_t s2 = atomicAdd(&F.bag_len[r], 1);
                F.pool_u[F.bag_start[r] + s2] = (int32_t)c;
                F.pool_w[F.bag_start[r] + s2] = w;
            }
        }
    }
}

// warp per vertex: count entries pointing to smaller keys; ready vertices form the first frontier
__global__ void k_init_count(FDev F, int32_t* frontier) {
    int64_t warp = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    int lane = threadIdx.x & 31;
    int64_t nw = ((int64_t)gridDim.x * blockDim.x) >> 5;
    for (int64_t v = warp; v < F.n; v += nw) {
        int32_t cnt = 0;
        int64_t s = F.bag_start[v];
        int32_t len = F.bag_len[v];
        for (int32_t i = lane; i < len; i += 32) cnt += key_less(F.prio, F.pool_u[s + i], (int32_t)v) ? 1 : 0;
        for (int o = 16; o > 0; o >>= 1) cnt += __shfl_xor_sync(0xffffffffu, cnt, o);
        if (lane == 0) {
            F.count[v] = cnt;
            F.level[v] = -1;
            if (cnt == 0) frontier[atomicAdd((unsigned long long*)&F.ctr[C_NEXT], 1ull)] = (int32_t)v;
        }
    }
}

// warp per frontier vertex: live entries, L and fill reservations, tier lists
__device__ void live_count(const FDev& F, const int32_t* frontier, int32_t* live_cnt, int32_t* list_b, int32_t* list_g,
                           int64_t warp, int64_t nw) {
    const int64_t nf = F.ctr[C_NEXT];
    const int lane = threadIdx.x & 31;
    for (int64_t i = warp; i < nf; i += nw) {
        int32_t v = frontier[i];
        int64_t s = F.bag_start[v];
        int32_t len = F.bag_len[v];
        int32_t cnt = 0;
        for (int32_t q = lane; q < len; q += 32) cnt += (F.level[F.pool_u[s + q]] < 0) ? 1 : 0;
        for (int o = 16; o > 0; o >>= 1) cnt += __shfl_xor_sync(0xffffffffu, cnt, o);
        if (lane == 0) {
            live_cnt[i] = cnt;
            if (F.vseg) {
                atomicAdd((unsigned long long*)&F.gctr[3 * F.vseg[v] + GC_FCUR], (unsigned long long)cnt);
                atomicAdd((unsigned long long*)&F.gctr[3 * F.vseg[v] + GC_NFRONT], 1ull);
            }
            F.Lstart[v] = (int64_t)atomicAdd((unsigned long long*)&F.ctr[C_LCUR], (unsigned long long)cnt);
            F.fstart[i] = (int64_t)atomicAdd((unsigned long long*)&F.ctr[C_FCUR], (unsigned long long)cnt);
            atomicMax((unsigned long long*)&F.ctr[C_MAXLIVE], (unsigned long long)cnt);
            if (cnt > 32 && cnt <= BLOCK_TIER_MAX)
                list_b[atomicAdd((unsigned long long*)&F.ctr[C_NB], 1ull)] = (int32_t)i;
            else if (cnt > BLOCK_TIER_MAX)
                list_g[atomicAdd((unsigned long long*)&F.ctr[C_NG], 1ull)] = (int32_t)i;
        }
    }
}

#define SSP_WARP_OF_GRID ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5, ((int64_t)gridDim.x * blockDim.x) >> 5
__global__ void k_live_count(FDev F, const int32_t* frontier, int32_t* live_cnt, int32_t* list_b, int32_t* list_g) {
    live_count(F, frontier, live_cnt, list_b, list_g, SSP_WARP_OF_GRID);
}

// ---------------------------------------------------------------- elimination (shared tail)
// Given merged entries (mu, mw)[0..cnt) sorted by (w, u) and inclusive prefix sums sc, emit one slot.
__device__ __forceinline__ void emit_slot(const FDev& F, int32_t v, int64_t fidx, int32_t i, int32_t cnt,
                                          const int32_t* mu, const double* mw, const double* sc, double S) {
    const int64_t Ls = F.Lstart[v];
    F.Lrow[Ls + i] = mu[i];
    F.Lval[Ls + i] = -(mw[i] / S);
    if (i + 1 < cnt) {
        const double ci = sc[i];
        const double rem = S - ci;
        const double tgt = factor_uniform(F.seed, local_vertex(F.vbase, v), i) * rem;
        int32_t lo = i + 1, hi = cnt;
        while (lo < hi) {
            int32_t mid = lo + ((hi - lo) >> 1);
            if ((sc[mid] - ci) < tgt) lo = mid + 1;
            else hi = mid;
        }
        const int32_t j = lo < cnt ? lo : cnt - 1;
        const int32_t r0 = mu[i], r1 = mu[j];
        const int32_t a = r0 > r1 ? r0 : r1, b = r0 > r1 ? r1 : r0;
        const double wf = (mw[i] * rem) / S;
        if (fidx >= 0) {
            const int64_t fp = F.fstart[fidx] + i;
            F.fill_a[fp] = a;
            F.fill_b[fp] = b;
            F.fill_w[fp] = wf;
            atomicAdd(&F.count[key_less(F.prio, b, a) ? a : b], 1);
            if (atomicAdd(&F.incoming[a], 1) == 0) F.owners[atomicAdd((unsigned long long*)&F.ctr[C_OWNERS], 1ull)] = a;
            if (atomicAdd(&F.incoming[b], 1) == 0) F.owners[atomicAdd((unsigned long long*)&F.ctr[C_OWNERS], 1ull)] = b;
        }
    }
}

// One entry of an eliminated vertex' bag: its live neighbour u loses a predecessor.  A vertex comes here after all of
// its fill is counted, so a count that reaches 0 has seen all of the level's fill at u: u is free.
__device__ __forceinline__ void release_entry(const FDev& F, int32_t u, int32_t* next) {
    if (atomicSub(&F.count[u], 1) == 1) next[atomicAdd((unsigned long long*)&F.ctr[C_NEXT], 1ull)] = u;
}

// Warp tier: <= 32 live entries, all in registers.
// s_mu, s_mw, s_c: 32 slots for each warp of the block.
__device__ void elim_warp(const FDev& F, const int32_t* frontier, int32_t* next, int32_t lvl, const int32_t* live_cnt,
                          int32_t (*s_mu)[32], double (*s_mw)[32], double (*s_c)[32], int64_t warp, int64_t nw) {
    const int64_t nf = F.ctr[C_REM];  // frontier size of this level
    const int lane = threadIdx.x & 31;
    for (int64_t fi = warp; fi < nf; fi += nw) {
        const int32_t L = live_cnt[fi];
        if (L > 32) continue;
        const int32_t v = frontier[fi];
        const int64_t s = F.bag_start[v];
        const int32_t len = F.bag_len[v];
        // gather live entries (order irrelevant: sorted next) through a per-warp staging area
        const int wib = threadIdx.x >> 5;
        int32_t got = 0;
        for (int32_t q0 = 0; q0 < len; q0 += 32) {
            int32_t q = q0 + lane;
            int32_t uu = 0;
            double ww = 0;
            bool live = false;
            if (q < len) {
                uu = F.pool_u[s + q];
                ww = F.pool_w[s + q];
                live = F.level[uu] < 0;
            }
            unsigned mask = __ballot_sync(0xffffffffu, live);
            if (live) {
                int32_t pos = got + __popc(mask & ((1u << lane) - 1u));
                if (pos < 32) {
                    s_mu[wib][pos] = uu;
                    s_mw[wib][pos] = ww;
                } else {
                    atomicOr((unsigned long long*)&F.ctr[C_ERR], (unsigned long long)FERR_OVERFLOW);
                }
            }
            got += __popc(mask);
        }
        got = got < 32 ? got : 32;
        __syncwarp();
        int32_t u = lane < got ? s_mu[wib][lane] : INT32_MAX;
        double w = lane < got ? s_mw[wib][lane] : __longlong_as_double(0x7ff0000000000000ll);
        __syncwarp();
        if (got == 0) {
            if (lane == 0) {
                F.D[v] = 0.0;
                F.Lcnt[v] = 0;
                F.fcnt[fi] = 0;
                F.level[v] = lvl;
            }
            continue;
        }
        warp_bitonic_ent(u, w, lane, EntUW());
        // merge runs of equal u: the head lane sums its run left to right
        const int32_t prev_u = __shfl_up_sync(0xffffffffu, u, 1);
        const bool head = (lane < got) && (lane == 0 || prev_u != u);
        double sum = w;
        bool cont = true;
        for (int t = 1; t < 32; t++) {
            double ow = __shfl_down_sync(0xffffffffu, w, t);
            int32_t ou = __shfl_down_sync(0xffffffffu, u, t);
            if (cont && lane + t < got && ou == u) sum = sum + ow;
            else cont = false;
            if (!__any_sync(0xffffffffu, cont)) break;  // few entries come twice
        }
        const unsigned hmask = __ballot_sync(0xffffffffu, head);
        const int32_t cnt = __popc(hmask);
        if (head) {
            int32_t pos = __popc(hmask & ((1u << lane) - 1u));
            s_mu[wib][pos] = u;
            s_mw[wib][pos] = sum;
        }
        __syncwarp();
        int32_t mu = lane < cnt ? s_mu[wib][lane] : INT32_MAX;
        double mw = lane < cnt ? s_mw[wib][lane] : __longlong_as_double(0x7ff0000000000000ll);
        __syncwarp();
        warp_bitonic_ent(mu, mw, lane, EntWU());
        // 32-wide Kogge-Stone inclusive scan (lanes >= cnt hold 0)
        double c = lane < cnt ? mw : 0.0;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            double t = __shfl_up_sync(0xffffffffu, c, o);
            if (lane >= o) c = t + c;
        }
        const double S = __shfl_sync(0xffffffffu, c, cnt - 1);
        // emission needs random access to (mu, mw, c): stage in shared memory
        s_mu[wib][lane] = mu;
        s_mw[wib][lane] = mw;
        s_c[wib][lane] = c;
        __syncwarp();
        if (lane < cnt) emit_slot(F, v, fi, lane, cnt, s_mu[wib], s_mw[wib], s_c[wib], S);
        if (lane == 0) {
            F.D[v] = S;
            F.Lcnt[v] = cnt;
            F.fcnt[fi] = cnt > 0 ? cnt - 1 : 0;
            if (cnt > 1) atomicAdd((unsigned long long*)&F.ctr[C_NFILL], (unsigned long long)(cnt - 1));
            if (cnt > 1 && F.vseg)
                atomicAdd((unsigned long long*)&F.gctr[3 * F.vseg[v] + GC_NFILL], (unsigned long long)(cnt - 1));
            F.level[v] = lvl;
        }
        __syncwarp();
        if (lane < got) release_entry(F, u, next);
    }
}

__global__ void __launch_bounds__(128)
    k_elim_warp(FDev F, const int32_t* frontier, int32_t* next, int32_t lvl, const int32_t* live_cnt) {
    __shared__ int32_t s_mu[4][32];
    __shared__ double s_mw[4][32];
    __shared__ double s_c[4][32];
    elim_warp(F, frontier, next, lvl, live_cnt, s_mu, s_mw, s_c, SSP_WARP_OF_GRID);
}

// Sorts the entries (mu, mw)[0 .. cnt) into (ou, ow), by (u, w) or by (w, u): 2^lg threads per entry count the entries
// before it, one barrier instead of the bitonic network's one per stage.  Weights compare by their bits, a total order
// (equal entries keep theirs), so the positions are a permutation for NaN too.
constexpr int RANK_SORT_MAX = 512;  // entries; at most one for each thread
template <bool W_FIRST>
__device__ __forceinline__ void block_rank_sort(const int32_t* mu, const double* mw, int32_t cnt, int32_t* ou, double* ow) {
    auto key = [](double w) {
        const long long x = __double_as_longlong(w);
        return x ^ ((x >> 63) & 0x7fffffffffffffffll);
    };
    int lg = 0;
    while (lg < 5 && (cnt << (lg + 1)) <= (int)blockDim.x) lg++;
    const int g = threadIdx.x & ((1 << lg) - 1);
    for (int32_t i0 = 0; i0 < cnt; i0 += (int)blockDim.x >> lg) {  // block-uniform
        const int32_t i = i0 + (int)(threadIdx.x >> lg);
        const bool in = i < cnt;
        const int32_t u = in ? mu[i] : 0;
        const double w = in ? mw[i] : 0.0;
        const long long k = key(w);
        int32_t before = 0;
        if (in)
            for (int32_t j = g; j < cnt; j += 1 << lg) {
                const int32_t uj = mu[j];
                const long long kj = key(mw[j]);
                const bool first = W_FIRST ? kj < k || (kj == k && (uj < u || (uj == u && j < i)))
                                           : uj < u || (uj == u && (kj < k || (kj == k && j < i)));
                before += first ? 1 : 0;
            }
        __syncwarp();
        for (int o = 1; o < 1 << lg; o <<= 1) before += __shfl_xor_sync(0xffffffffu, before, o);
        if (in && g == 0) {
            ou[before] = u;
            ow[before] = w;
        }
    }
}

// Block helpers -----------------------------------------------------------------
// exclusive block scan of an int flag (one per thread), returns the prefix; *total gets the sum.
__device__ __forceinline__ int32_t block_excl_scan(int32_t x, int32_t* s_warp, int32_t* total) {
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, nwarp = blockDim.x >> 5;
    int32_t incl = x;
    for (int o = 1; o < 32; o <<= 1) {
        int32_t t = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += t;
    }
    if (lane == 31) s_warp[wid] = incl;
    __syncthreads();
    if (wid == 0) {
        int32_t t = lane < nwarp ? s_warp[lane] : 0;
        int32_t ti = t;
        for (int o = 1; o < 32; o <<= 1) {
            int32_t u = __shfl_up_sync(0xffffffffu, ti, o);
            if (lane >= o) ti += u;
        }
        if (lane < nwarp) s_warp[lane] = ti - t;
        if (lane == 31) s_warp[32] = ti;
    }
    __syncthreads();
    int32_t r = s_warp[wid] + incl - x;
    *total = s_warp[32];
    __syncthreads();
    return r;
}

// Chunked scan of mw[0..cnt) into sc: 32-wide Kogge-Stone chunks, sequential carry.
__device__ void block_chunk_scan(const double* mw, double* sc, int32_t cnt, double* s_carry) {
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, nwarp = blockDim.x >> 5;
    const int32_t nch = (cnt + 31) >> 5;
    for (int32_t ch = wid; ch < nch; ch += nwarp) {
        int32_t i = ch * 32 + lane;
        double c = i < cnt ? mw[i] : 0.0;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            double t = __shfl_up_sync(0xffffffffu, c, o);
            if (lane >= o) c = t + c;
        }
        if (i < cnt) sc[i] = c;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        double carry = 0.0;
        for (int32_t ch = 1; ch < nch; ch++) {
            int32_t last_prev = min(ch * 32, cnt) - 1;  // last element of chunk ch-1
            double prev_local = sc[last_prev];
            carry = (ch == 1) ? prev_local : carry + prev_local;
            s_carry[ch] = carry;
        }
    }
    __syncthreads();
    for (int32_t i = 32 + threadIdx.x; i < cnt; i += blockDim.x) sc[i] = s_carry[i >> 5] + sc[i];
    __syncthreads();
}

// gather live entries of bag[v], sort by (u,w), merge runs.  Returns merged count in mu/mw.
// Arrays hold P slots (P = pow2 >= L).
__device__ int32_t block_gather_merge(const FDev& F, int32_t v, int32_t L, int32_t cap, int32_t* su, double* sw,
                                      int32_t* mu, double* mw, int32_t* s_warp, int32_t* s_cnt) {
    int P = 2;
    while (P < L) P <<= 1;
    if (threadIdx.x == 0) *s_cnt = 0;
    __syncthreads();
    const int64_t s = F.bag_start[v];
    const int32_t len = F.bag_len[v];
    for (int32_t q = threadIdx.x; q < len; q += blockDim.x) {
        int32_t uu = F.pool_u[s + q];
        if (F.level[uu] < 0) {
            int32_t pos = atomicAdd(s_cnt, 1);
            if (pos < L && pos < cap) {
                su[pos] = uu;
                sw[pos] = F.pool_w[s + q];
            } else {
                atomicOr((unsigned long long*)&F.ctr[C_ERR], (unsigned long long)FERR_OVERFLOW);
            }
        }
    }
    __syncthreads();
    if (L <= min(RANK_SORT_MAX, (int)blockDim.x)) {
        // counted into (mu, mw), which are free until the merged entries go there
        block_rank_sort<false>(su, sw, L, mu, mw);
        __syncthreads();
        for (int32_t i = threadIdx.x; i < L; i += blockDim.x) {
            su[i] = mu[i];
            sw[i] = mw[i];
        }
        __syncthreads();
    } else {
        for (int32_t i = L + threadIdx.x; i < P; i += blockDim.x) {
            su[i] = INT32_MAX;
            sw[i] = __longlong_as_double(0x7ff0000000000000ll);
        }
        __syncthreads();
        block_bitonic_ent(su, sw, P, EntUW());
    }
    // heads and run sums
    int32_t cnt = 0;
    for (int32_t base = 0; base < L; base += blockDim.x) {
        int32_t i = base + threadIdx.x;
        bool head = i < L && (i == 0 || su[i - 1] != su[i]);
        double sum = 0.0;
        if (head) {
            sum = sw[i];
            for (int32_t j = i + 1; j < L && su[j] == su[i]; j++) sum = sum + sw[j];
        }
        int32_t tot;
        int32_t pos = block_excl_scan(head ? 1 : 0, s_warp, &tot);
        if (head) {
            mu[cnt + pos] = su[i];
            mw[cnt + pos] = sum;
        }
        cnt += tot;
    }
    __syncthreads();
    return cnt;
}

// (su, sw): scratch of cnt entries
__device__ void block_finish_column(const FDev& F, int32_t v, int64_t fidx, int32_t cnt, int32_t* mu, double* mw,
                                    double* sc, double* s_carry, int32_t* su, double* sw) {
    if (cnt == 0) {
        if (threadIdx.x == 0) {
            F.D[v] = 0.0;
            F.Lcnt[v] = 0;
            if (fidx >= 0) F.fcnt[fidx] = 0;
        }
        __syncthreads();
        return;
    }
    if (cnt <= min(RANK_SORT_MAX, (int)blockDim.x)) {
        block_rank_sort<true>(mu, mw, cnt, su, sw);
        __syncthreads();
        mu = su;
        mw = sw;
    } else {
        int P = 2;
        while (P < cnt) P <<= 1;
        for (int32_t i = cnt + threadIdx.x; i < P; i += blockDim.x) {
            mu[i] = INT32_MAX;
            mw[i] = __longlong_as_double(0x7ff0000000000000ll);
        }
        __syncthreads();
        block_bitonic_ent(mu, mw, P, EntWU());
    }
    block_chunk_scan(mw, sc, cnt, s_carry);
    const double S = sc[cnt - 1];
    for (int32_t i = threadIdx.x; i < cnt; i += blockDim.x) emit_slot(F, v, fidx, i, cnt, mu, mw, sc, S);
    if (threadIdx.x == 0) {
        F.D[v] = S;
        F.Lcnt[v] = cnt;
        if (fidx >= 0) {
            F.fcnt[fidx] = cnt - 1;
            if (cnt > 1) atomicAdd((unsigned long long*)&F.ctr[C_NFILL], (unsigned long long)(cnt - 1));
            if (cnt > 1 && F.vseg)
                atomicAdd((unsigned long long*)&F.gctr[3 * F.vseg[v] + GC_NFILL], (unsigned long long)(cnt - 1));
        }
    }
    __syncthreads();
}

// One block eliminates frontier vertex fi.
__device__ void elim_block(const FDev& F, int32_t fi, const int32_t* frontier, int32_t* next, int32_t lvl, int32_t L,
                           int32_t cap, int32_t* su, double* sw, int32_t* mu, double* mw, double* sc, double* s_carry,
                           int32_t* s_warp, int32_t* s_cnt) {
    const int32_t v = frontier[fi];
    const int32_t cnt = block_gather_merge(F, v, L, cap, su, sw, mu, mw, s_warp, s_cnt);
    block_finish_column(F, v, fi, cnt, mu, mw, sc, s_carry, su, sw);
    const int64_t s = F.bag_start[v];
    const int32_t len = F.bag_len[v];
    for (int32_t q = threadIdx.x; q < len; q += blockDim.x) {
        const int32_t u = F.pool_u[s + q];
        if (F.level[u] < 0) release_entry(F, u, next);
    }
    if (threadIdx.x == 0) F.level[v] = lvl;
}

// Block tier (shared memory) and global tier (scratch slices), one block per vertex.
__global__ void k_elim_block(FDev F, const int32_t* frontier, int32_t* next, int32_t lvl, const int32_t* live_cnt,
                             const int32_t* list, int64_t nlist_idx, int32_t cap, int32_t* g_u, double* g_w) {
    extern __shared__ __align__(16) unsigned char smem[];
    __shared__ int32_t s_warp[33];
    __shared__ int32_t s_cnt;
    __shared__ double s_carry_static[BLOCK_TIER_MAX / 32 + 1];
    const int64_t nlist = F.ctr[nlist_idx];
    for (int64_t li = blockIdx.x; li < nlist; li += gridDim.x) {
        const int32_t fi = list[li];
        int32_t *su, *mu;
        double *sw, *mw, *sc, *s_carry;
        if (g_u) {  // global scratch: 2 int arrays + 3 double arrays of cap, carry after
            int64_t base = (int64_t)blockIdx.x * cap;
            su = g_u + 2 * base;
            mu = su + cap;
            sw = g_w + 4 * base;
            mw = sw + cap;
            sc = mw + cap;
            s_carry = sc + cap;
        } else {
            sw = (double*)smem;
            mw = sw + cap;
            sc = mw + cap;
            su = (int32_t*)(sc + cap);
            mu = su + cap;
            s_carry = s_carry_static;
        }
        elim_block(F, fi, frontier, next, lvl, live_cnt[fi], cap, su, sw, mu, mw, sc, s_carry, s_warp, &s_cnt);
    }
}

// ---------------------------------------------------------------- fill bookkeeping
// warp per owner: make room for the incoming fill (relocate, dropping stale entries)
__device__ void reserve(const FDev& F, int64_t warp, int64_t nw) {
    const int64_t no = F.ctr[C_OWNERS];
    const int lane = threadIdx.x & 31;
    for (int64_t oi = warp; oi < no; oi += nw) {
        const int32_t a = F.owners[oi];
        const int32_t inc = F.incoming[a];
        const int32_t len = F.bag_len[a];
        if (len + inc > F.bag_cap[a]) {
            const int64_t s = F.bag_start[a];
            int32_t live = 0;
            for (int32_t q = lane; q < len; q += 32) live += (F.level[F.pool_u[s + q]] < 0) ? 1 : 0;
            for (int o = 16; o > 0; o >>= 1) live += __shfl_xor_sync(0xffffffffu, live, o);
            const int32_t ncap = max(2 * (live + inc), 16);
            int64_t ns = 0;
            if (lane == 0) ns = (int64_t)atomicAdd((unsigned long long*)&F.ctr[C_POOL], (unsigned long long)ncap);
            ns = __shfl_sync(0xffffffffu, ns, 0);
            if (ns + ncap > F.pool_cap) {
                if (lane == 0) atomicOr((unsigned long long*)&F.ctr[C_ERR], (unsigned long long)FERR_POOL);
            } else {
                int32_t out = 0;
                for (int32_t q0 = 0; q0 < len; q0 += 32) {
                    int32_t q = q0 + lane;
                    bool lv = false;
                    int32_t uu = 0;
                    double ww = 0;
                    if (q < len) {
                        uu = F.pool_u[s + q];
                        ww = F.pool_w[s + q];
                        lv = F.level[uu] < 0;
                    }
                    unsigned m = __ballot_sync(0xffffffffu, lv);
                    if (lv) {
                        int32_t p = out + __popc(m & ((1u << lane) - 1u));
                        F.pool_u[ns + p] = uu;
                        F.pool_w[ns + p] = ww;
                    }
                    out += __popc(m);
                }
                __syncwarp();
                if (lane == 0) {
                    F.bag_start[a] = ns;
                    F.bag_len[a] = live;
                    F.bag_cap[a] = ncap;
                }
            }
        }
        __syncwarp();
        if (lane == 0) F.incoming[a] = 0;
    }
}
__global__ void k_reserve(FDev F) {
    reserve(F, SSP_WARP_OF_GRID);
}

__device__ void fill_scatter(const FDev& F, int64_t warp, int64_t nw) {
    const int64_t nf = F.ctr[C_REM];
    const int lane = threadIdx.x & 31;
    for (int64_t fi = warp; fi < nf; fi += nw) {
        const int64_t s = F.fstart[fi];
        const int32_t c = F.fcnt[fi];
        for (int32_t q = lane; q < c; q += 32) {
            int32_t a = F.fill_a[s + q], b = F.fill_b[s + q];
            double w = F.fill_w[s + q];
            int32_t sa = atomicAdd(&F.bag_len[a], 1);
            if (sa < F.bag_cap[a]) {
                F.pool_u[F.bag_start[a] + sa] = b;
                F.pool_w[F.bag_start[a] + sa] = w;
            } else {
                atomicOr((unsigned long long*)&F.ctr[C_ERR], (unsigned long long)FERR_OVERFLOW);
            }
            int32_t sb = atomicAdd(&F.bag_len[b], 1);
            if (sb < F.bag_cap[b]) {
                F.pool_u[F.bag_start[b] + sb] = a;
                F.pool_w[F.bag_start[b] + sb] = w;
            } else {
                atomicOr((unsigned long long*)&F.ctr[C_ERR], (unsigned long long)FERR_OVERFLOW);
            }
        }
    }
}
__global__ void k_fill_scatter(FDev F) {
    fill_scatter(F, SSP_WARP_OF_GRID);
}

// ---------------------------------------------------------------- many levels in one launch
// The levels of small frontiers, which are most: latency alone counts there (an elimination of 32 entries is a chain of
// five dependent loads and two sorts; the host loop's launches and its wait for the counters come on top).  One cooperative
// launch, a block per SM, runs level after level with four barriers over its blocks: on B200 30-37 us a level for
// frontiers of 30-320 vertices where launches and a read-back took about 95 (the factors of a 30k-vertex geometric
// graph 32 -> 24.5 ms, of a 40^3 grid 27.5 -> 22).  It starts with a level whose capacities the host has checked, and
// at every level boundary takes the host loop's own decisions on the same numbers; what it does not handle (a
// truncation, the dense tail, a pool to compact, buffers to grow, bags above ELIM_LIVE_MAX, wide frontiers) ends it
// there, and the host loop goes on from the state it leaves.  So does a stream that cannot hold all of its blocks at once: the
// launch is refused, or its blocks give up before the first level (ST_GO).
// ELIM_FRONT_MAX: 3.5 vertices for each warp of the grid; such a level takes 86-90 us here, as in the host loop, and wider
// ones are better spread over the launches' larger grids.  ELIM_LIVE_MAX: what fits the static shared memory.
enum { ST_LIVE = 0, ST_ELIM, ST_LVL, ST_PREV, ST_LUSED, ST_STOP, ST_ERR, ST_GO, ST_N };
enum { GO_ALL = 1, GO_NONE = 2 };  // ST_GO: every block has arrived, or a block has given up waiting for the others
constexpr int ELIM_THREADS = 256, ELIM_LIVE_MAX = 512;
constexpr int64_t ELIM_FRONT_MAX = 4096;

// The launch's blocks (one per SM) and the limit of the wait for them to run; the environment variables make either too
// much for the device, which takes the ways back to the host loop.
static int env_int(const char* name, int value) {
    const char* e = getenv(name);
    return e && e[0] ? atoi(e) : value;
}
static int level_blocks(int sms) { return env_int("SSP_FACTOR_LEVEL_BLOCKS", sms); }
static int level_start_spins() { return env_int("SSP_FACTOR_LEVEL_SPINS", 1 << 20); }

struct ElimArgs {
    FDev F;
    int32_t* front[2];  // frontier of the first level and the other list, in turn
    int32_t *live_cnt, *list_b, *list_g;
    int64_t* st;             // ST_*
    int start_spins;         // limit on the wait for all blocks to run
    unsigned* bar;           // arrivals, releases, blocks that run
    int32_t* log;            // frontier size by level
    int64_t max_degree, dense_threshold, pool_init, pool_cap, Lcap, Fcap;
    // several graphs: per graph its vertices, truncation, and the accounting of ST_LIVE, ST_ELIM, ST_PREV
    const int64_t *g_n, *g_max;
    int64_t *g_live, *g_elim, *g_prev;
};

// Waits until every block of the grid runs, or gives up after some tenths of a second (other work may hold a part of the
// device).  One compare-and-swap decides between the last block to arrive and the first to give up, so all blocks, also
// those that come later, return the same; nothing has been changed when they return false.
__device__ bool all_blocks_run(const ElimArgs& A) {
    __shared__ int s_go;
    if (threadIdx.x == 0) {
        unsigned long long* go = (unsigned long long*)&A.st[ST_GO];
        if (atomicAdd(&A.bar[2], 1u) == gridDim.x - 1) atomicCAS(go, 0ull, (unsigned long long)GO_ALL);
        for (int spins = 0; *(volatile unsigned long long*)go == 0; spins++) {
            if (spins >= A.start_spins) atomicCAS(go, 0ull, (unsigned long long)GO_NONE);
            else if (spins > 1024) __nanosleep(100);
        }
        s_go = *(volatile unsigned long long*)go == GO_ALL;
    }
    __syncthreads();
    return s_go != 0;
}

// Barrier over the grid; the last block to arrive runs ctl (all its threads) before the others go on.  All blocks run
// (all_blocks_run), so the wait is one for a part of a level; it is bounded all the same (some ten seconds), and past that the
// kernel reports ST_ERR and ends.  Returns false then.
template <class Ctl>
__device__ bool grid_barrier(const ElimArgs& A, Ctl ctl) {
    __shared__ unsigned s_ticket;
    __shared__ int s_ok;
    __syncthreads();
    if (threadIdx.x == 0) {
        __threadfence();
        s_ticket = atomicAdd(&A.bar[0], 1u);
        s_ok = 1;
    }
    __syncthreads();
    const unsigned round = s_ticket / gridDim.x;
    if (s_ticket % gridDim.x == gridDim.x - 1) {
        if (threadIdx.x == 0) __threadfence();
        __syncthreads();
        ctl();
        __syncthreads();
        if (threadIdx.x == 0) {
            __threadfence();
            atomicExch(&A.bar[1], round + 1);
        }
    } else if (threadIdx.x == 0) {
        int spins = 0;
        while ((int)(*(volatile unsigned*)&A.bar[1] - (round + 1)) < 0) {
            if (++spins > 1024) __nanosleep(100);
            if (spins > (1 << 26)) {
                atomicExch((unsigned long long*)&A.st[ST_ERR], 1ull);
                s_ok = 0;
                break;
            }
        }
    }
    if (threadIdx.x == 0) __threadfence();
    __syncthreads();
    return s_ok != 0;
}

__global__ void __launch_bounds__(ELIM_THREADS) k_elim_levels(ElimArgs A) {
    constexpr int NWARP = ELIM_THREADS / 32;
    __shared__ int32_t s_mu[NWARP][32];
    __shared__ double s_mw[NWARP][32];
    __shared__ double s_c[NWARP][32];
    __shared__ int32_t b_su[ELIM_LIVE_MAX], b_mu[ELIM_LIVE_MAX];
    __shared__ double b_sw[ELIM_LIVE_MAX], b_mw[ELIM_LIVE_MAX], b_sc[ELIM_LIVE_MAX];
    __shared__ double s_carry[ELIM_LIVE_MAX / 32 + 1];
    __shared__ int32_t s_warp[33];
    __shared__ int32_t s_cnt;
    const FDev& F = A.F;
    const int wib = threadIdx.x >> 5;
    const int64_t warp = (int64_t)blockIdx.x * NWARP + wib, nw = (int64_t)gridDim.x * NWARP;
    int64_t* ctr = F.ctr;
    auto nothing = [] {};
    // the level begins: its frontier is the list just counted
    auto begin = [&] {
        if (threadIdx.x == 0) {
            const int64_t nf = ctr[C_NEXT];
            A.log[A.st[ST_LVL]] = (int32_t)nf;
            A.st[ST_LUSED] = ctr[C_LCUR];
            A.st[ST_PREV] = ctr[C_FCUR];
            A.st[ST_ELIM] += nf;
            ctr[C_REM] = nf;
            ctr[C_NEXT] = 0;
            ctr[C_OWNERS] = 0;
            ctr[C_NFILL] = 0;
        }
        for (int32_t g = threadIdx.x; g < F.nseg; g += ELIM_THREADS) {
            A.g_prev[g] = F.gctr[3 * g + GC_FCUR];
            A.g_elim[g] += F.gctr[3 * g + GC_NFRONT];
            F.gctr[3 * g + GC_NFILL] = 0;
        }
    };
    // the boundary after a level, with the upcoming frontier counted: the host loop's tests in its order
    auto boundary = [&] {
        __shared__ int s_stop;
        if (threadIdx.x == 0) {
            const int64_t nf = ctr[C_NEXT], n = F.n, elim = A.st[ST_ELIM], maxlive = ctr[C_MAXLIVE];
            const int64_t live = A.st[ST_LIVE] + 2 * ctr[C_NFILL] - 2 * A.st[ST_PREV];
            const int64_t reserve = 2 * (A.pool_init + 2 * ctr[C_FCUR]) + 16 * (n - elim) + 1024;
            s_stop = ctr[C_ERR] != 0 || nf == 0 || nf > ELIM_FRONT_MAX || ctr[C_NG] > 0 || maxlive > ELIM_LIVE_MAX ||
                     (F.nseg == 0 && A.max_degree > 0 && live > A.max_degree * (n - elim)) || elim + nf > n ||
                     (A.dense_threshold > 0 && n - elim <= A.dense_threshold && nf <= DENSE_FRONTIER_MAX) ||
                     ctr[C_POOL] + reserve > A.pool_cap || ctr[C_LCUR] > A.Lcap || ctr[C_FCUR] > A.Fcap;
        }
        __syncthreads();
        for (int32_t g = threadIdx.x; g < F.nseg; g += ELIM_THREADS) {
            const int64_t live = A.g_live[g] + (A.g_prev[g] >= 0 ? 2 * F.gctr[3 * g + GC_NFILL] - 2 * A.g_prev[g] : 0);
            if (A.g_max[g] > 0 && F.gctr[3 * g + GC_NFRONT] > 0 && live > A.g_max[g] * (A.g_n[g] - A.g_elim[g])) s_stop = 1;
        }
        __syncthreads();
        if (s_stop) {
            if (threadIdx.x == 0) A.st[ST_STOP] = 1;
            return;
        }
        for (int32_t g = threadIdx.x; g < F.nseg; g += ELIM_THREADS)
            if (A.g_prev[g] >= 0) A.g_live[g] += 2 * F.gctr[3 * g + GC_NFILL] - 2 * A.g_prev[g];
        if (threadIdx.x == 0) A.st[ST_LIVE] += 2 * ctr[C_NFILL] - 2 * A.st[ST_PREV];
        __syncthreads();
        begin();
    };
    if (!all_blocks_run(A)) return;
    if (!grid_barrier(A, begin)) return;
    for (int cur = 0;; cur ^= 1) {
        const int32_t* frontier = A.front[cur];
        int32_t* next = A.front[cur ^ 1];
        const int32_t lvl = (int32_t)A.st[ST_LVL];
        // eliminate: some blocks take the bags above 32 live entries, the others' warps the rest
        const int64_t nlist = ctr[C_NB], nrest = ctr[C_REM] - nlist;
        const int nb = (int)min(nlist, (int64_t)gridDim.x - min((nrest + NWARP - 1) / NWARP, (int64_t)gridDim.x / 2));
        if ((int)blockIdx.x < nb) {
            for (int64_t li = blockIdx.x; li < nlist; li += nb) {
                const int32_t fi = A.list_b[li];
                elim_block(F, fi, frontier, next, lvl, A.live_cnt[fi], ELIM_LIVE_MAX, b_su, b_sw, b_mu, b_mw, b_sc,
                           s_carry, s_warp, &s_cnt);
            }
        } else {
            elim_warp(F, frontier, next, lvl, A.live_cnt, s_mu, s_mw, s_c, warp - (int64_t)nb * NWARP,
                      nw - (int64_t)nb * NWARP);
        }
        if (!grid_barrier(A, nothing)) return;
        reserve(F, warp, nw);
        if (blockIdx.x == 0) {  // (nothing below reads these before the next barrier)
            if (threadIdx.x == 0) {
                ctr[C_FCUR] = 0;
                ctr[C_NB] = 0;
                ctr[C_NG] = 0;
                ctr[C_MAXLIVE] = 0;
                A.st[ST_LVL] = lvl + 1;
            }
            for (int32_t g = threadIdx.x; g < F.nseg; g += ELIM_THREADS)
                F.gctr[3 * g + GC_FCUR] = F.gctr[3 * g + GC_NFRONT] = 0;
        }
        if (!grid_barrier(A, nothing)) return;
        fill_scatter(F, warp, nw);
        if (!grid_barrier(A, nothing)) return;
        live_count(F, next, A.live_cnt, A.list_b, A.list_g, warp, nw);
        if (!grid_barrier(A, boundary)) return;
        if (A.st[ST_STOP]) return;
    }
}

// frontier swap bookkeeping: REM <- NEXT, reset per-level cursors
__global__ void k_level_begin(int64_t* ctr, int64_t* gctr, int32_t nseg) {
    ctr[C_REM] = ctr[C_NEXT];
    ctr[C_NEXT] = 0;
    ctr[C_OWNERS] = 0;
    ctr[C_NFILL] = 0;
    for (int32_t g = 0; g < nseg; g++) gctr[3 * g + GC_NFILL] = 0;
}
__global__ void k_level_prep(int64_t* ctr, int64_t* gctr, int32_t nseg) {
    // the upcoming frontier's counts become the live-count kernel's domain
    ctr[C_FCUR] = 0;
    ctr[C_NB] = 0;
    ctr[C_NG] = 0;
    ctr[C_MAXLIVE] = 0;
    for (int32_t g = 0; g < nseg; g++) gctr[3 * g + GC_FCUR] = gctr[3 * g + GC_NFRONT] = 0;
}
__global__ void k_set_ctr(int64_t* ctr, int idx, int64_t v) { ctr[idx] = v; }
// the frontier without the vertices of stopped graphs (order kept)
__global__ void k_drop_stopped(const int32_t* __restrict__ in, int64_t nin, const int32_t* __restrict__ vseg,
                               const int32_t* __restrict__ stopped, int32_t* __restrict__ out, int64_t* cnt) {
    // one block: order-preserving compaction
    __shared__ int32_t s_base;
    if (threadIdx.x == 0) s_base = 0;
    __syncthreads();
    for (int64_t b0 = 0; b0 < nin; b0 += blockDim.x) {
        const int64_t i = b0 + threadIdx.x;
        const int keep = i < nin && !stopped[vseg[in[i]]];
        const unsigned bal = __ballot_sync(0xffffffffu, keep);
        __shared__ int32_t s_warp[32];
        const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
        if (lane == 0) s_warp[w] = __popc(bal);
        __syncthreads();
        int32_t before = 0;
        for (int j = 0; j < w; j++) before += s_warp[j];
        int32_t tot = 0;
        for (int j = 0; j < (int)(blockDim.x >> 5); j++) tot += s_warp[j];
        if (keep) out[s_base + before + __popc(bal & ((1u << lane) - 1u))] = in[i];
        __syncthreads();
        if (threadIdx.x == 0) s_base += tot;
        __syncthreads();
    }
    if (threadIdx.x == 0) *cnt = s_base;
}
__global__ void k_collect_live_range(int64_t v0, int64_t v1, const int32_t* level, int32_t* rem, int64_t* cnt) {
    for (int64_t v = v0 + (int64_t)blockIdx.x * blockDim.x + threadIdx.x; v < v1; v += (int64_t)gridDim.x * blockDim.x)
        if (level[v] < 0) rem[atomicAdd((unsigned long long*)cnt, 1ull)] = (int32_t)v;
}

// ---------------------------------------------------------------- dense tail
__global__ void k_collect_live(int64_t n, const int32_t* level, int32_t* rem, int64_t* cnt) {
    for (int64_t v = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; v < n; v += (int64_t)gridDim.x * blockDim.x)
        if (level[v] < 0) rem[atomicAdd((unsigned long long*)cnt, 1ull)] = (int32_t)v;
}

struct KeyVLess {
    const uint64_t* prio;
    __device__ bool operator()(const int32_t& a, const int32_t& b) const {
        uint64_t pa = prio[a], pb = prio[b];
        return pa != pb ? pa < pb : a < b;
    }
};

__global__ void k_sort_rem(int32_t* rem, int32_t T, int32_t P, const uint64_t* prio, int32_t* idx) {
    extern __shared__ int32_t s_keys[];
    for (int i = threadIdx.x; i < P; i += blockDim.x) s_keys[i] = i < T ? rem[i] : -1;
    __syncthreads();
    // -1 sentinels must sort last: compare with sentinel handling
    struct L {
        const uint64_t* prio;
        __device__ bool operator()(const int32_t& a, const int32_t& b) const {
            if (a < 0) return false;
            if (b < 0) return true;
            uint64_t pa = prio[a], pb = prio[b];
            return pa != pb ? pa < pb : a < b;
        }
    } less{prio};
    block_bitonic_kv<false, int32_t, int32_t>(s_keys, (int32_t*)nullptr, P, less);
    for (int i = threadIdx.x; i < T; i += blockDim.x) {
        rem[i] = s_keys[i];
        idx[s_keys[i]] = i;
    }
}

// block per remaining vertex: merged live entries into the dense matrix
__global__ void k_dense_build(FDev F, const int32_t* rem, int32_t T, const int32_t* idx, double* W, int32_t cap,
                              int32_t* g_u, double* g_w, int use_global) {
    extern __shared__ __align__(16) unsigned char smem[];
    __shared__ int32_t s_warp[33];
    __shared__ int32_t s_cnt;
    __shared__ int32_t s_live;
    for (int32_t i = blockIdx.x; i < T; i += gridDim.x) {
        const int32_t v = rem[i];
        // live count
        if (threadIdx.x == 0) s_live = 0;
        __syncthreads();
        const int64_t s = F.bag_start[v];
        const int32_t len = F.bag_len[v];
        int32_t c = 0;
        for (int32_t q = threadIdx.x; q < len; q += blockDim.x) c += (F.level[F.pool_u[s + q]] < 0) ? 1 : 0;
        atomicAdd(&s_live, c);
        __syncthreads();
        const int32_t L = s_live;
        int32_t *su, *mu;
        double *sw, *mw;
        if (use_global) {
            int64_t base = (int64_t)blockIdx.x * cap;
            su = g_u + 2 * base;
            mu = su + cap;
            sw = g_w + 4 * base;
            mw = sw + cap;
        } else {
            sw = (double*)smem;
            mw = sw + cap;
            su = (int32_t*)(mw + cap);
            mu = su + cap;
        }
        int32_t cnt = block_gather_merge(F, v, L, cap, su, sw, mu, mw, s_warp, &s_cnt);
        for (int32_t q = threadIdx.x; q < cnt; q += blockDim.x) W[(int64_t)i * T + idx[mu[q]]] = mw[q];
        __syncthreads();
    }
}

// Single block: eliminate the T remaining vertices in key order.  A chain of T columns, so what counts is the latency
// of one: the row's nonzeros are collected in any order (their keys are unique), ranked, scanned in 32-wide chunks
// whose carries every thread adds up for itself, and each fill goes out as two fire-and-forget additions (a pair of
// rows gets at most one fill per column, so the sums are the same in every run) -- six barriers a column.  On B200 the
// tails of 1852 vertices (geometric graph, n = 30,011), 1112 (3-D grid, n = 64,000) and 1007 (n = 80,840) take 7.6, 3.5 and
// 1.9 ms; with an ordered compaction, a bitonic sort and read-modify-write fills they took 23.3, 11.0 and 5.8.  Columns
// longer than RANK_SORT_MAX are still sorted by the network.
__global__ void __launch_bounds__(1024) k_dense_elim(FDev F, const int32_t* rem, int32_t T, int32_t Pmax,
                                                     const int32_t* idx, double* W, int64_t Lbase, int32_t lvl0) {
    extern __shared__ __align__(16) unsigned char smem[];
    __shared__ int32_t s_cnt;
    __shared__ double s_carry2[8192 / 32 + 1];
    __shared__ int32_t s_u[RANK_SORT_MAX];
    __shared__ double s_w[RANK_SORT_MAX];
    double* mw = (double*)smem;
    double* sc = mw + Pmax;
    int32_t* mu = (int32_t*)(sc + Pmax);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    int64_t Lpos = Lbase;
    if (threadIdx.x == 0) s_cnt = 0;
    __syncthreads();
    for (int32_t i = 0; i < T; i++) {
        const int32_t v = rem[i];
        const double* row = W + (int64_t)i * T;
        // the nonzeros q > i
        for (int32_t base = i + 1; base < T; base += blockDim.x) {
            const int32_t q = base + threadIdx.x;
            const double x = q < T ? __ldcg(row + q) : 0.0;
            const bool nz = x != 0.0;
            const unsigned m = __ballot_sync(0xffffffffu, nz);
            int32_t at = 0;
            if (lane == 0 && m) at = atomicAdd(&s_cnt, __popc(m));
            at = __shfl_sync(0xffffffffu, at, 0) + __popc(m & ((1u << lane) - 1u));
            if (nz) {
                mu[at] = rem[q];
                mw[at] = x;
            }
        }
        __syncthreads();
        const int32_t cnt = s_cnt;
        int32_t* su = mu;
        double* sw = mw;
        if (cnt <= RANK_SORT_MAX) {
            block_rank_sort<true>(mu, mw, cnt, s_u, s_w);
            su = s_u;
            sw = s_w;
        } else {
            int P = 2;
            while (P < cnt) P <<= 1;
            for (int32_t q = cnt + threadIdx.x; q < P; q += blockDim.x) {
                mu[q] = INT32_MAX;
                mw[q] = __longlong_as_double(0x7ff0000000000000ll);
            }
            __syncthreads();
            block_bitonic_ent(mu, mw, P, EntWU());
        }
        __syncthreads();
        if (threadIdx.x == 0) s_cnt = 0;  // every thread has read it
        // prefix sums: 32-wide Kogge-Stone chunks, then each thread adds the chunks before its own in order
        const int32_t nch = (cnt + 31) >> 5;
        for (int32_t ch = warp; ch < nch; ch += blockDim.x >> 5) {
            const int32_t q = ch * 32 + lane;
            double c = q < cnt ? sw[q] : 0.0;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const double t = __shfl_up_sync(0xffffffffu, c, o);
                if (lane >= o) c = t + c;
            }
            if (q < cnt) sc[q] = c;
        }
        __syncthreads();
        if (cnt <= RANK_SORT_MAX) {
            // at most 16 chunks: thread q's own carry (its sum so far must not be overwritten before all have read theirs)
            const int32_t q = threadIdx.x, ch = q >> 5;
            double carry = 0.0, mine = 0.0;
            if (q < cnt) {
                for (int32_t j = 1; j <= ch; j++) carry = j == 1 ? sc[31] : carry + sc[j * 32 - 1];
                mine = ch > 0 ? carry + sc[q] : sc[q];
            }
            __syncthreads();
            if (q < cnt) sc[q] = mine;
        } else {
            if (threadIdx.x == 0) {
                double carry = 0.0;
                for (int32_t ch = 1; ch < nch; ch++) {
                    const double prev = sc[ch * 32 - 1];
                    carry = ch == 1 ? prev : carry + prev;
                    s_carry2[ch] = carry;
                }
            }
            __syncthreads();
            for (int32_t q = 32 + threadIdx.x; q < cnt; q += blockDim.x) sc[q] = s_carry2[q >> 5] + sc[q];
        }
        __syncthreads();
        const double S = cnt > 0 ? sc[cnt - 1] : 0.0;
        for (int32_t q = threadIdx.x; q < cnt; q += blockDim.x) {
            F.Lrow[Lpos + q] = su[q];
            F.Lval[Lpos + q] = -(sw[q] / S);
            if (q + 1 < cnt) {
                const double ci = sc[q];
                const double rem_ = S - ci;
                const double tgt = factor_uniform(F.seed, local_vertex(F.vbase, v), q) * rem_;
                int32_t lo = q + 1, hi = cnt;
                while (lo < hi) {
                    int32_t mid = lo + ((hi - lo) >> 1);
                    if ((sc[mid] - ci) < tgt) lo = mid + 1;
                    else hi = mid;
                }
                const int32_t j = lo < cnt ? lo : cnt - 1;
                const int32_t a = su[q], b = su[j];
                const double wf = (sw[q] * rem_) / S;
                const int64_t ia = idx[a], ib = idx[b];
                atomicAdd(&W[ia * T + ib], wf);
                atomicAdd(&W[ib * T + ia], wf);
            }
        }
        if (threadIdx.x == 0) {
            F.Lstart[v] = Lpos;
            F.D[v] = S;
            F.Lcnt[v] = cnt;
            F.level[v] = lvl0 + i;
        }
        Lpos += cnt;
        __syncthreads();
    }
}

// ---------------------------------------------------------------- truncation
// Per remaining vertex: no L entries, D = merged live weights summed in row order.  A warp does a vertex of at most
// 32 live entries in registers; the others go to the block version below.  At ER n = 1M (855,771 vertices) a block each
// took 11.5 ms; here the warps take 1.2 ms and the blocks of the rest 0.9.
__global__ void __launch_bounds__(256) k_trunc_diag_warp(FDev F, const int32_t* rem, int32_t T, int32_t* big) {
    const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
    __shared__ int32_t s_u[8][32];
    __shared__ double s_w[8][32];
    const int64_t nw = ((int64_t)gridDim.x * blockDim.x) >> 5;
    for (int64_t i = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5; i < T; i += nw) {
        const int32_t v = rem[i];
        const int64_t s = F.bag_start[v];
        const int32_t len = F.bag_len[v];
        int32_t got = 0;
        for (int32_t q0 = 0; q0 < len; q0 += 32) {
            const int32_t q = q0 + lane;
            int32_t u = 0;
            bool live = false;
            if (q < len) {
                u = F.pool_u[s + q];
                live = F.level[u] < 0;
            }
            const unsigned m = __ballot_sync(0xffffffffu, live);
            const int32_t pos = got + __popc(m & ((1u << lane) - 1u));
            if (live && pos < 32) {
                s_u[wib][pos] = u;
                s_w[wib][pos] = F.pool_w[s + q];
            }
            got += __popc(m);
        }
        __syncwarp();
        if (got > 32) {
            if (lane == 0) big[atomicAdd((unsigned long long*)&F.ctr[C_NB], 1ull)] = v;
            __syncwarp();
            continue;
        }
        int32_t u = lane < got ? s_u[wib][lane] : INT32_MAX;
        double w = lane < got ? s_w[wib][lane] : __longlong_as_double(0x7ff0000000000000ll);
        __syncwarp();
        warp_bitonic_ent(u, w, lane, EntUW());
        // runs of equal u summed left to right, the runs' sums added in row order
        double d = 0.0, run = 0.0;
        for (int q = 0; q < got; q++) {
            const double wq = __shfl_sync(0xffffffffu, w, q);
            const int32_t uq = __shfl_sync(0xffffffffu, u, q), un = __shfl_sync(0xffffffffu, u, (q + 1) & 31);
            const int32_t up = __shfl_sync(0xffffffffu, u, (q + 31) & 31);
            run = q > 0 && up == uq ? run + wq : wq;
            if (q + 1 == got || un != uq) d = d + run;
        }
        if (lane == 0) {
            F.D[v] = d;
            F.Lcnt[v] = 0;
            F.Lstart[v] = 0;
        }
    }
}
__global__ void k_trunc_diag(FDev F, const int32_t* rem, int32_t lvl, int32_t cap, int32_t* g_u, double* g_w,
                             int use_global) {
    const int32_t T = (int32_t)F.ctr[C_NB];
    extern __shared__ __align__(16) unsigned char smem[];
    __shared__ int32_t s_warp[33];
    __shared__ int32_t s_cnt;
    __shared__ int32_t s_live;
    for (int32_t i = blockIdx.x; i < T; i += gridDim.x) {
        const int32_t v = rem[i];
        if (threadIdx.x == 0) s_live = 0;
        __syncthreads();
        const int64_t s = F.bag_start[v];
        const int32_t len = F.bag_len[v];
        int32_t c = 0;
        for (int32_t q = threadIdx.x; q < len; q += blockDim.x) c += (F.level[F.pool_u[s + q]] < 0) ? 1 : 0;
        atomicAdd(&s_live, c);
        __syncthreads();
        const int32_t L = s_live;
        int32_t *su, *mu;
        double *sw, *mw;
        if (use_global) {
            int64_t base = (int64_t)blockIdx.x * cap;
            su = g_u + 2 * base;
            mu = su + cap;
            sw = g_w + 4 * base;
            mw = sw + cap;
        } else {
            sw = (double*)smem;
            mw = sw + cap;
            su = (int32_t*)(mw + cap);
            mu = su + cap;
        }
        const int32_t cnt = block_gather_merge(F, v, L, cap, su, sw, mu, mw, s_warp, &s_cnt);
        if (threadIdx.x == 0) {
            double d = 0.0;
            for (int32_t q = 0; q < cnt; q++) d = d + mw[q];
            F.D[v] = d;
            F.Lcnt[v] = 0;
            F.Lstart[v] = 0;
        }
        __syncthreads();
    }
}
__global__ void k_set_level(const int32_t* rem, int32_t T, int32_t lvl, int32_t* level) {
    for (int32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < T; i += gridDim.x * blockDim.x) level[rem[i]] = lvl;
}

// ---------------------------------------------------------------- post-processing
__global__ void k_copy_cols(int64_t n, const int64_t* Lstart, const int32_t* Lcnt, const int32_t* Lrow,
                            const double* Lval, const int64_t* col_ptr, int32_t* col_idx, double* col_val) {
    const int lane = threadIdx.x & 31;
    const int64_t nw = ((int64_t)gridDim.x * blockDim.x) >> 5;
    for (int64_t v = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5; v < n; v += nw) {
        const int64_t s = Lstart[v], d = col_ptr[v];
        const int32_t c = Lcnt[v];
        for (int32_t q = lane; q < c; q += 32) {
            col_idx[d + q] = Lrow[s + q];
            col_val[d + q] = Lval[s + q];
        }
    }
}

__global__ void k_row_count(int64_t nnz, const int32_t* col_idx, int32_t* rowcnt) {
    for (int64_t p = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; p < nnz; p += (int64_t)gridDim.x * blockDim.x)
        atomicAdd(&rowcnt[col_idx[p]], 1);
}

__global__ void k_row_scatter(int64_t n, const int64_t* col_ptr, const int32_t* col_idx, const double* col_val,
                              const int64_t* row_ptr, int32_t* cursor, int32_t* row_idx, double* row_val) {
    const int lane = threadIdx.x & 31;
    const int64_t nw = ((int64_t)gridDim.x * blockDim.x) >> 5;
    for (int64_t v = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5; v < n; v += nw) {
        for (int64_t p = col_ptr[v] + lane; p < col_ptr[v + 1]; p += 32) {
            int32_t u = col_idx[p];
            int32_t slot = atomicAdd(&cursor[u], 1);
            row_idx[row_ptr[u] + slot] = (int32_t)v;
            row_val[row_ptr[u] + slot] = col_val[p];
        }
    }
}

__global__ void k_level_count(int64_t n, const int32_t* level, int32_t* lvcnt) {
    for (int64_t v = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; v < n; v += (int64_t)gridDim.x * blockDim.x)
        atomicAdd(&lvcnt[level[v]], 1);
}
// sort key of a vertex: its level, then the length of its row (or column) of L, longest first
__global__ void k_level_keys(int64_t n, const int32_t* level, const int64_t* ptr, uint64_t* key, int32_t* v_out) {
    for (int64_t v = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; v < n; v += (int64_t)gridDim.x * blockDim.x) {
        const int64_t len = ptr[v + 1] - ptr[v];
        key[v] = ((uint64_t)(uint32_t)level[v] << 8) | (uint64_t)(255 - (len < 255 ? len : 255));
        v_out[v] = (int32_t)v;
    }
}
__global__ void k_i64_to_i32(int64_t n, const int64_t* a, int32_t* b) {
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
        b[i] = (int32_t)a[i];
}

// ---------------------------------------------------------------- bag pool compaction
// warp per vertex: live bags get 2*live + 8 slots in a fresh pool; eliminated vertices get none
__global__ void k_compact_caps(FDev F, int32_t* newcap) {
    const int lane = threadIdx.x & 31;
    const int64_t nw = ((int64_t)gridDim.x * blockDim.x) >> 5;
    for (int64_t v = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5; v < F.n; v += nw) {
        int32_t live = 0;
        if (F.level[v] < 0) {
            const int64_t s = F.bag_start[v];
            const int32_t len = F.bag_len[v];
            for (int32_t q = lane; q < len; q += 32) live += (F.level[F.pool_u[s + q]] < 0) ? 1 : 0;
            for (int o = 16; o > 0; o >>= 1) live += __shfl_xor_sync(0xffffffffu, live, o);
        }
        if (lane == 0) newcap[v] = F.level[v] < 0 ? 2 * live + 8 : 0;
    }
}

__global__ void k_compact_copy(FDev F, const int64_t* newstart, const int32_t* newcap, int32_t* nu, double* nw_) {
    const int lane = threadIdx.x & 31;
    const int64_t nw = ((int64_t)gridDim.x * blockDim.x) >> 5;
    for (int64_t v = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5; v < F.n; v += nw) {
        if (F.level[v] >= 0) continue;
        const int64_t s = F.bag_start[v], d = newstart[v];
        const int32_t len = F.bag_len[v];
        int32_t out = 0;
        for (int32_t q0 = 0; q0 < len; q0 += 32) {
            int32_t q = q0 + lane;
            bool lv = false;
            int32_t uu = 0;
            double ww = 0;
            if (q < len) {
                uu = F.pool_u[s + q];
                ww = F.pool_w[s + q];
                lv = F.level[uu] < 0;
            }
            unsigned m = __ballot_sync(0xffffffffu, lv);
            if (lv) {
                int32_t p = out + __popc(m & ((1u << lane) - 1u));
                nu[d + p] = uu;
                nw_[d + p] = ww;
            }
            out += __popc(m);
        }
        __syncwarp();
        if (lane == 0) {
            F.bag_start[v] = d;
            F.bag_len[v] = out;
            F.bag_cap[v] = newcap[v];
        }
    }
}

// storage-order copies of the row and column forms
__global__ void k_perm_count(int64_t n, const int32_t* perm, const int64_t* ptr, int32_t* cnt) {
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
        const int32_t v = perm[i];
        cnt[i] = (int32_t)(ptr[v + 1] - ptr[v]);
    }
}
__global__ void k_perm_copy(int64_t n, const int32_t* perm, const int64_t* ptr, const int32_t* idx, const double* val,
                            const int64_t* pptr, int32_t* pidx, double* pval, FactorRow* prow,
                            FactorEnt<double>* pent) {
    const int lane = threadIdx.x & 31;
    const int64_t nw = ((int64_t)gridDim.x * blockDim.x) >> 5;
    for (int64_t i = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5; i < n; i += nw) {
        const int32_t v = perm[i];
        const int64_t s = ptr[v], d = pptr[i], c = ptr[v + 1] - s;
        if (lane == 0 && prow) prow[i] = FactorRow{v, (int32_t)c, d};
        for (int64_t q = lane; q < c; q += 32) {
            const int32_t u = idx[s + q];
            const double x = val[s + q];
            pidx[d + q] = u;
            pval[d + q] = x;
            if (pent) pent[d + q] = FactorEnt<double>{x, u};
        }
    }
}

// ---------------------------------------------------------------- host driver
// grow a device buffer, keeping its first `keep` bytes
static void* grow_keep(Context& C, const std::string& name, void* old, size_t keep, size_t bytes) {
    (void)old;
    return C.ws.grow(name, keep, bytes, C.stream);
}

void factor_device(Context& C, int64_t n, const int64_t* colptr, const int32_t* rowidx, const double* val,
                   const FactorOptions& opt, DevFactor& out, const std::string& tag) {
    SSP_REQUIRE(n > 0, SSP_ERR_INVALID, "factor: empty matrix");
    SSP_REQUIRE(opt.dense_threshold >= 0 && opt.dense_threshold <= 8192, SSP_ERR_INVALID,
                "factor: dense_threshold must be in [0, 8192]");
    Workspace& W = C.ws;
    auto nm = [&](const char* s) { return tag + "_" + s; };
    FDev F;
    F.n = n;
    F.seed = opt.seed;
    F.vbase = opt.vbase;
    // the dense tail looks at the whole Schur complement and would couple several graphs: a union is
    // eliminated in the sparse phase, and truncated graph by graph (vseg)
    const bool seg_mode = opt.vseg != nullptr;
    const int32_t nseg = seg_mode ? (int32_t)opt.seg_row0.size() - 1 : 0;
    SSP_REQUIRE(!opt.vbase || (opt.dense_threshold == 0 && (opt.max_degree == 0 || seg_mode)), SSP_ERR_INVALID,
                "factor: several graphs at once need dense_threshold = 0 (and the graph of every vertex when "
                "truncating)");
    SSP_REQUIRE(!seg_mode || (nseg >= 1 && opt.seg_row0.front() == 0 && opt.seg_row0.back() == n &&
                              (opt.seg_max_degree.empty() || (int32_t)opt.seg_max_degree.size() == nseg)),
                SSP_ERR_INVALID, "factor: inconsistent graph ranges");
    std::vector<int64_t> g_maxdeg(nseg);
    for (int32_t g = 0; g < nseg; g++) {
        g_maxdeg[g] = opt.seg_max_degree.empty() ? opt.max_degree : opt.seg_max_degree[g];
        SSP_REQUIRE(g_maxdeg[g] >= 0, SSP_ERR_INVALID, "factor: a graph's truncation must be >= 0");
    }
    F.vseg = opt.vseg;
    F.nseg = nseg;
    F.gctr = seg_mode ? W.get_t<int64_t>(nm("gctr"), 3 * (size_t)nseg) : nullptr;
    if (seg_mode) SSP_CUDA(cudaMemsetAsync(F.gctr, 0, sizeof(int64_t) * 3 * nseg, C.stream));
    uint64_t* prio = W.get_t<uint64_t>(nm("prio"), n);
    F.prio = prio;
    F.count = W.get_t<int32_t>(nm("count"), n);
    F.level = W.get_t<int32_t>(nm("level"), n);
    F.bag_start = W.get_t<int64_t>(nm("bag_start"), n + 1);
    F.bag_len = W.get_t<int32_t>(nm("bag_len"), n);
    F.bag_cap = W.get_t<int32_t>(nm("bag_cap"), n + 1);
    F.ctr = W.get_t<int64_t>(nm("ctr"), C_NCTR);
    F.Lstart = W.get_t<int64_t>(nm("Lstart"), n);
    F.Lcnt = W.get_t<int32_t>(nm("Lcnt"), n + 1);
    F.D = W.get_t<double>(nm("D"), n);
    int32_t* deg = W.get_t<int32_t>(nm("deg"), n + 1);
    SSP_CUDA(cudaMemsetAsync(F.ctr, 0, sizeof(int64_t) * C_NCTR, C.stream));
    SSP_CUDA(cudaMemsetAsync(deg, 0, sizeof(int32_t) * (n + 1), C.stream));
    SSP_CUDA(cudaMemsetAsync(F.bag_len, 0, sizeof(int32_t) * n, C.stream));
    SSP_CUDA(cudaMemsetAsync(F.Lcnt, 0, sizeof(int32_t) * (n + 1), C.stream));
    const int T256 = 256;
    k_prio<<<grid_for(n, T256), T256, 0, C.stream>>>(n, opt.seed, prio, opt.vbase);
    k_lower_deg<<<grid_for(n, T256), T256, 0, C.stream>>>(n, colptr, rowidx, val, deg);
    k_bag_caps<<<grid_for(n, T256), T256, 0, C.stream>>>(n, deg, F.bag_cap);
    SSP_CHECK_LAUNCH();
    C.kernels_launched += 3;
    SSP_CUDA(cudaMemsetAsync(F.bag_cap + n, 0, sizeof(int32_t), C.stream));
    int64_t* d_tot = W.get_t<int64_t>(nm("tot"), 2);
    exclusive_scan_i32_to_i64(C, F.bag_cap, F.bag_start, n + 1, d_tot);
    const int64_t pool_init = read_i64(C, d_tot);
    // room for relocations: the live entry count never grows, so 3x the initial layout plus slack
    int64_t pool_cap = pool_init * 4 + 20 * n + 4096;
    F.pool_u = W.get_t<int32_t>(nm("pool_u"), pool_cap);
    F.pool_w = W.get_t<double>(nm("pool_w"), pool_cap);
    F.pool_cap = pool_cap;
    int pool_gen = 0;
    out.frontier_sizes.clear();
    out.compactions = 0;
    out.truncated_rows = 0;
    k_bag_fill<<<grid_for(n, T256), T256, 0, C.stream>>>(n, colptr, rowidx, val, F);
    SSP_CHECK_LAUNCH();
    C.kernels_launched++;
    // pool cursor = pool_init
    SSP_CUDA(cudaMemcpyAsync(F.ctr + C_POOL, d_tot, sizeof(int64_t), cudaMemcpyDeviceToDevice, C.stream));
    int32_t* frontier = W.get_t<int32_t>(nm("frontier"), n);
    int32_t* next = W.get_t<int32_t>(nm("next"), n);
    int32_t* live_cnt = W.get_t<int32_t>(nm("live_cnt"), n);
    int32_t* list_b = W.get_t<int32_t>(nm("list_b"), n);
    int32_t* list_g = W.get_t<int32_t>(nm("list_g"), n);
    F.incoming = W.get_t<int32_t>(nm("incoming"), n);
    F.owners = W.get_t<int32_t>(nm("owners"), n);
    F.fstart = W.get_t<int64_t>(nm("fstart"), n);
    F.fcnt = W.get_t<int32_t>(nm("fcnt"), n);
    SSP_CUDA(cudaMemsetAsync(F.incoming, 0, sizeof(int32_t) * n, C.stream));
    k_init_count<<<grid_for(n * 32, T256, 148 * 64), T256, 0, C.stream>>>(F, next);
    SSP_CHECK_LAUNCH();
    C.kernels_launched++;

    // L pool and fill buffer (grown on demand)
    int64_t Lcap = std::max<int64_t>(pool_init * 2, 1024);
    F.Lrow = W.get_t<int32_t>(nm("Lrow"), Lcap);
    F.Lval = W.get_t<double>(nm("Lval"), Lcap);
    int64_t Fcap = std::max<int64_t>(pool_init, 1024);
    F.fill_a = W.get_t<int32_t>(nm("fill_a"), Fcap);
    F.fill_b = W.get_t<int32_t>(nm("fill_b"), Fcap);
    F.fill_w = W.get_t<double>(nm("fill_w"), Fcap);

    // live counts of the first frontier
    auto live_count = [&](int32_t* fr) {
        k_level_prep<<<1, 1, 0, C.stream>>>(F.ctr, F.gctr, F.nseg);
        k_live_count<<<grid_for(n * 32, T256, 148 * 64), T256, 0, C.stream>>>(F, fr, live_cnt, list_b, list_g);
        SSP_CHECK_LAUNCH();
        C.kernels_launched += 2;
    };
    live_count(next);

    int64_t h[C_NCTR];
    int64_t eliminated = 0;
    int32_t lvl = 0;
    int64_t live_entries = 0;  // live entries of the current Schur complement (both directions)
    {
        SSP_CUDA(cudaMemsetAsync(deg + n, 0, sizeof(int32_t), C.stream));
        int64_t* tmp = W.get_t<int64_t>(nm("degscan"), n + 1);
        exclusive_scan_i32_to_i64(C, deg, tmp, n + 1, d_tot);
        live_entries = read_i64(C, d_tot);
    }
    int64_t prev_fcur = -1;
    bool truncated = false;
    bool many_levels = true;  // small frontiers' levels in one launch, until a stream turns out not to hold it
    int64_t Lused_prev = 0;
    const size_t blk_smem = (size_t)BLOCK_TIER_MAX * (3 * sizeof(double) + 2 * sizeof(int32_t));
    allow_dynamic_smem(C, k_elim_block, blk_smem);
    // several graphs: each graph's own truncation test, with its own live-entry count (the same accounting
    // as the single-graph test below, restricted to its vertices)
    std::vector<int64_t> g_live(nseg, 0), g_elim(nseg, 0), g_prev(nseg, -1), g_cnt(3 * (size_t)nseg + 1, 0);
    std::vector<int32_t> g_stopped(nseg, 0);
    int32_t* d_stopped = seg_mode ? W.get_t<int32_t>(nm("gstop"), nseg) : nullptr;
    int32_t last_trunc_level = -1;
    if (seg_mode) {
        std::vector<int32_t> hdeg(n);
        SSP_CUDA(cudaMemcpyAsync(hdeg.data(), deg, sizeof(int32_t) * n, cudaMemcpyDeviceToHost, C.stream));
        SSP_CUDA(cudaStreamSynchronize(C.stream));
        for (int32_t g = 0; g < nseg; g++)
            for (int64_t v = opt.seg_row0[g]; v < opt.seg_row0[g + 1]; v++) g_live[g] += hdeg[v];
    }
    // D of the R vertices rem (their bags hold at most maxlen entries): warps, then blocks for the larger bags, whose
    // list's length stays on the device
    auto trunc_diag = [&](const int32_t* rem, int64_t R, int32_t at, int32_t maxlen) {
        int32_t* big = list_b;  // (a level's lists are made after its truncations)
        SSP_CUDA(cudaMemsetAsync(F.ctr + C_NB, 0, sizeof(int64_t), C.stream));
        k_trunc_diag_warp<<<grid_for(R * 32, T256, 148 * 64), T256, 0, C.stream>>>(F, rem, (int32_t)R, big);
        SSP_CHECK_LAUNCH();
        C.kernels_launched++;
        if (maxlen <= 32) return;
        int32_t cap = 64;
        while (cap < maxlen) cap <<= 1;
        if (cap <= BLOCK_TIER_MAX) {
            size_t smem = (size_t)cap * (2 * sizeof(double) + 2 * sizeof(int32_t));
            allow_dynamic_smem(C, k_trunc_diag, smem);
            k_trunc_diag<<<(int)std::min<int64_t>(R, 148 * 8), 256, smem, C.stream>>>(F, big, at, cap, nullptr, nullptr, 0);
        } else {
            int blocks = 32;
            int32_t* gu = W.get_t<int32_t>(nm("gscr_u"), (size_t)2 * cap * blocks);
            double* gw = W.get_t<double>(nm("gscr_w"), (size_t)4 * cap * blocks);
            k_trunc_diag<<<blocks, 1024, 0, C.stream>>>(F, big, at, cap, gu, gw, 1);
        }
        SSP_CHECK_LAUNCH();
        C.kernels_launched++;
    };
    // graph g's live vertices become its final, diagonal level `at` (k_trunc_diag), as a lone truncation does
    auto truncate_graph = [&](int32_t g, int32_t at) -> int64_t {
        const int64_t v0 = opt.seg_row0[g], v1 = opt.seg_row0[g + 1];
        int32_t* rem = W.get_t<int32_t>(nm("rem"), n + 1);
        SSP_CUDA(cudaMemsetAsync(F.ctr + C_REM, 0, sizeof(int64_t), C.stream));
        k_collect_live_range<<<grid_for(v1 - v0, T256), T256, 0, C.stream>>>(v0, v1, F.level, rem, F.ctr + C_REM);
        SSP_CHECK_LAUNCH();
        const int64_t R = read_i64(C, F.ctr + C_REM);
        if (R == 0) return 0;
        trunc_diag(rem, R, at, device_max_i32(C, F.bag_len + v0, v1 - v0));
        k_set_level<<<grid_for(R, T256), T256, 0, C.stream>>>(rem, (int32_t)R, at, F.level);
        SSP_CHECK_LAUNCH();
        C.kernels_launched += 2;
        int64_t hh[C_NCTR];
        read_i64s(C, F.ctr, hh, C_NCTR);
        if (hh[C_ERR]) throw Error(SSP_ERR_CAPACITY, "factor: truncation overflow");
        return R;
    };
    while (true) {
        read_i64s(C, F.ctr, h, C_NCTR);
        if (h[C_ERR] & FERR_POOL) throw Error(SSP_ERR_CAPACITY, "factor: bag pool exhausted");
        if (h[C_ERR] & FERR_OVERFLOW) throw Error(SSP_ERR_CAPACITY, "factor: bag overflow");
        if (prev_fcur >= 0) live_entries += 2 * h[C_NFILL] - 2 * prev_fcur;
        int64_t nf = h[C_NEXT];
        if (seg_mode) {
            read_i64s(C, F.gctr, g_cnt.data(), 3 * nseg);
            for (int32_t g = 0; g < nseg; g++)
                if (g_prev[g] >= 0) g_live[g] += 2 * g_cnt[3 * g + GC_NFILL] - 2 * g_prev[g];
        }
        if (nf == 0) break;
        if (seg_mode) {
            std::vector<int32_t> stop;
            for (int32_t g = 0; g < nseg; g++) {
                const int64_t ng = opt.seg_row0[g + 1] - opt.seg_row0[g];
                if (!g_stopped[g] && g_maxdeg[g] > 0 && g_cnt[3 * g + GC_NFRONT] > 0 &&
                    g_live[g] > g_maxdeg[g] * (ng - g_elim[g]))
                    stop.push_back(g);
            }
            if (!stop.empty()) {
                for (int32_t g : stop) {
                    const int64_t R = truncate_graph(g, lvl);
                    g_stopped[g] = 1;
                    eliminated += R;
                    out.truncated_rows += R;
                    last_trunc_level = lvl;
                }
                // the frontier without the stopped graphs, and its reservations made again
                SSP_CUDA(cudaMemcpyAsync(d_stopped, g_stopped.data(), sizeof(int32_t) * nseg, cudaMemcpyHostToDevice,
                                         C.stream));
                k_drop_stopped<<<1, 1024, 0, C.stream>>>(next, nf, F.vseg, d_stopped, frontier, F.ctr + C_NEXT);
                k_set_ctr<<<1, 1, 0, C.stream>>>(F.ctr, C_LCUR, Lused_prev);
                SSP_CHECK_LAUNCH();
                C.kernels_launched += 2;
                std::swap(frontier, next);
                live_count(next);
                read_i64s(C, F.ctr, h, C_NCTR);
                read_i64s(C, F.gctr, g_cnt.data(), 3 * nseg);
                nf = h[C_NEXT];
                if (nf == 0) break;
            }
        }
        if (!seg_mode && opt.max_degree > 0 && live_entries > opt.max_degree * (n - eliminated)) {
            truncated = true;
            break;
        }
        if (eliminated + nf > n || lvl > n)
            throw Error(SSP_ERR_CAPACITY, "factor: frontier accounting inconsistent (eliminated > n)");
        if (opt.dense_threshold > 0 && n - eliminated <= opt.dense_threshold && nf <= DENSE_FRONTIER_MAX) break;
        out.frontier_sizes.push_back(nf);
        // relocations of this level allocate at most 2*(live entries + incoming fill) + 16 per owner
        {
            const int64_t reserve = 2 * (pool_init + 2 * h[C_FCUR]) + 16 * (n - eliminated) + 1024;
            if (h[C_POOL] + reserve > pool_cap) {
                int32_t* newcap = W.get_t<int32_t>(nm("newcap"), n + 1);
                int64_t* newstart = W.get_t<int64_t>(nm("newstart"), n + 1);
                k_compact_caps<<<grid_for(n * 32, T256, 148 * 64), T256, 0, C.stream>>>(F, newcap);
                SSP_CUDA(cudaMemsetAsync(newcap + n, 0, sizeof(int32_t), C.stream));
                exclusive_scan_i32_to_i64(C, newcap, newstart, n + 1, d_tot);
                const int64_t used = read_i64(C, d_tot);
                const int64_t ncap = std::max<int64_t>(pool_cap, used + reserve + used / 2);
                const std::string other = (pool_gen & 1) ? "" : "_b";
                int32_t* nu = W.get_t<int32_t>(nm("pool_u") + other, ncap);
                double* nwp = W.get_t<double>(nm("pool_w") + other, ncap);
                k_compact_copy<<<grid_for(n * 32, T256, 148 * 64), T256, 0, C.stream>>>(F, newstart, newcap, nu, nwp);
                SSP_CHECK_LAUNCH();
                C.kernels_launched += 2;
                F.pool_u = nu;
                F.pool_w = nwp;
                F.pool_cap = pool_cap = ncap;
                SSP_CUDA(cudaMemcpyAsync(F.ctr + C_POOL, d_tot, sizeof(int64_t), cudaMemcpyDeviceToDevice, C.stream));
                pool_gen++;
                out.compactions++;
            }
        }
        // capacities for this level's reservations
        if (h[C_LCUR] > Lcap) {
            int64_t ncap = std::max<int64_t>(h[C_LCUR] + h[C_LCUR] / 2, Lcap * 2);
            F.Lrow = (int32_t*)grow_keep(C, nm("Lrow"), F.Lrow, sizeof(int32_t) * Lused_prev, sizeof(int32_t) * ncap);
            F.Lval = (double*)grow_keep(C, nm("Lval"), F.Lval, sizeof(double) * Lused_prev, sizeof(double) * ncap);
            Lcap = ncap;
        }
        if (h[C_FCUR] > Fcap) {
            Fcap = std::max<int64_t>(h[C_FCUR] + h[C_FCUR] / 2, Fcap * 2);
            F.fill_a = W.get_t<int32_t>(nm("fill_a"), Fcap);
            F.fill_b = W.get_t<int32_t>(nm("fill_b"), Fcap);
            F.fill_w = W.get_t<double>(nm("fill_w"), Fcap);
        }
        if (many_levels && nf <= ELIM_FRONT_MAX && h[C_NG] == 0 && h[C_MAXLIVE] <= ELIM_LIVE_MAX) {
            // this level and those after it, up to one that needs the host
            int64_t st[ST_N] = {live_entries, eliminated, lvl, -1, Lused_prev, 0, 0, 0};
            int64_t* d_st = W.get_t<int64_t>(nm("el_st"), ST_N + 2);
            int64_t* d_g = W.get_t<int64_t>(nm("el_g"), 5 * (size_t)nseg + 1);
            int32_t* d_log = deg;  // (no longer needed)
            std::vector<int64_t> hg;
            for (int32_t g = 0; g < nseg; g++) hg.push_back(opt.seg_row0[g + 1] - opt.seg_row0[g]);
            // a stopped graph has no vertex in a frontier any more, so its test never holds again
            for (const auto* v : {&g_maxdeg, &g_live, &g_elim, &g_prev}) hg.insert(hg.end(), v->begin(), v->end());
            SSP_CUDA(cudaMemcpyAsync(d_st, st, sizeof(st), cudaMemcpyHostToDevice, C.stream));
            SSP_CUDA(cudaMemsetAsync(d_st + ST_N, 0, 2 * sizeof(int64_t), C.stream));
            if (nseg)
                SSP_CUDA(cudaMemcpyAsync(d_g, hg.data(), sizeof(int64_t) * hg.size(), cudaMemcpyHostToDevice, C.stream));
            ElimArgs A;
            A.F = F;
            A.front[0] = next;
            A.front[1] = frontier;
            A.live_cnt = live_cnt;
            A.list_b = list_b;
            A.list_g = list_g;
            A.st = d_st;
            A.start_spins = level_start_spins();
            A.bar = (unsigned*)(d_st + ST_N);
            A.log = d_log;
            A.max_degree = opt.max_degree;
            A.dense_threshold = opt.dense_threshold;
            A.pool_init = pool_init;
            A.pool_cap = pool_cap;
            A.Lcap = Lcap;
            A.Fcap = Fcap;
            A.g_n = d_g;
            A.g_max = d_g + nseg;
            A.g_live = d_g + 2 * nseg;
            A.g_elim = d_g + 3 * nseg;
            A.g_prev = d_g + 4 * nseg;
            int sms = 0;
            SSP_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, C.device));
            void* args[] = {&A};
            const cudaError_t le = cudaLaunchCooperativeKernel((const void*)k_elim_levels, dim3((unsigned)level_blocks(sms)),
                                                               dim3(ELIM_THREADS), args, 0, C.stream);
            if (le == cudaErrorCooperativeLaunchTooLarge || le == cudaErrorLaunchOutOfResources ||
                le == cudaErrorNotSupported) {
                cudaGetLastError();
                many_levels = false;
            } else {
                SSP_CUDA(le);
                C.kernels_launched++;
                read_i64s(C, d_st, st, ST_N);
                if (st[ST_ERR]) throw Error(SSP_ERR_CUDA, "factor: a level's barrier was not reached in time");
                many_levels = st[ST_GO] == GO_ALL;
            }
            if (many_levels) {
                const int32_t done = (int32_t)st[ST_LVL] - lvl;
                std::vector<int32_t> sizes(done);
                SSP_CUDA(cudaMemcpyAsync(sizes.data(), d_log + lvl, sizeof(int32_t) * done, cudaMemcpyDeviceToHost, C.stream));
                if (nseg) {
                    read_i64s(C, A.g_live, g_live.data(), nseg);
                    read_i64s(C, A.g_elim, g_elim.data(), nseg);
                    read_i64s(C, A.g_prev, g_prev.data(), nseg);
                }
                SSP_CUDA(cudaStreamSynchronize(C.stream));
                out.frontier_sizes.pop_back();
                out.frontier_sizes.insert(out.frontier_sizes.end(), sizes.begin(), sizes.end());
                live_entries = st[ST_LIVE];
                eliminated = st[ST_ELIM];
                lvl = (int32_t)st[ST_LVL];
                prev_fcur = st[ST_PREV];
                Lused_prev = st[ST_LUSED];
                if (done & 1) std::swap(frontier, next);
                continue;
            }
        }
        Lused_prev = h[C_LCUR];
        prev_fcur = h[C_FCUR];
        for (int32_t g = 0; g < nseg; g++) {
            g_prev[g] = g_cnt[3 * g + GC_FCUR];
            g_elim[g] += g_cnt[3 * g + GC_NFRONT];
        }
        std::swap(frontier, next);
        k_level_begin<<<1, 1, 0, C.stream>>>(F.ctr, F.gctr, F.nseg);  // REM <- NEXT (frontier size), NEXT <- 0
        k_elim_warp<<<grid_for(nf * 32, 128, 148 * 64), 128, 0, C.stream>>>(F, frontier, next, lvl, live_cnt);
        SSP_CHECK_LAUNCH();
        C.kernels_launched += 2;
        if (h[C_NB] > 0) {
            int32_t cap = 64;
            while (cap < std::min<int64_t>(h[C_MAXLIVE], BLOCK_TIER_MAX)) cap <<= 1;
            size_t smem = (size_t)cap * (3 * sizeof(double) + 2 * sizeof(int32_t));
            int blocks = (int)std::min<int64_t>(h[C_NB], 148 * 4);
            k_elim_block<<<blocks, 256, smem, C.stream>>>(F, frontier, next, lvl, live_cnt, list_b, C_NB, cap, nullptr,
                                                       nullptr);
            SSP_CHECK_LAUNCH();
            C.kernels_launched++;
        }
        if (h[C_NG] > 0) {
            int32_t cap = 64;
            while (cap < h[C_MAXLIVE]) cap <<= 1;
            int blocks = (int)std::min<int64_t>(h[C_NG], 32);
            int32_t* gu = W.get_t<int32_t>(nm("gscr_u"), (size_t)2 * cap * blocks);
            double* gw = W.get_t<double>(nm("gscr_w"), (size_t)4 * cap * blocks);
            k_elim_block<<<blocks, 1024, 0, C.stream>>>(F, frontier, next, lvl, live_cnt, list_g, C_NG, cap, gu, gw);
            SSP_CHECK_LAUNCH();
            C.kernels_launched++;
        }
        const int gw32 = grid_for(nf * 32, T256, 148 * 64);
        k_reserve<<<grid_for(n * 32, T256, 148 * 64), T256, 0, C.stream>>>(F);
        k_fill_scatter<<<gw32, T256, 0, C.stream>>>(F);
        SSP_CHECK_LAUNCH();
        C.kernels_launched += 2;
        eliminated += nf;
        lvl++;
        live_count(next);
    }
    if (seg_mode && last_trunc_level >= lvl) lvl = last_trunc_level + 1;  // a graph truncated after the last level
    const int32_t sparse_levels = lvl;
    const int64_t T = truncated ? 0 : n - eliminated;
    if (truncated) {
        const int64_t R = n - eliminated;
        int32_t* rem = W.get_t<int32_t>(nm("rem"), R + 1);
        SSP_CUDA(cudaMemsetAsync(F.ctr + C_REM, 0, sizeof(int64_t), C.stream));
        k_collect_live<<<grid_for(n, T256), T256, 0, C.stream>>>(n, F.level, rem, F.ctr + C_REM);
        trunc_diag(rem, R, lvl, device_max_i32(C, F.bag_len, n));
        k_set_level<<<grid_for(R, T256), T256, 0, C.stream>>>(rem, (int32_t)R, lvl, F.level);
        SSP_CHECK_LAUNCH();
        C.kernels_launched += 2;
        int64_t hh[C_NCTR];
        read_i64s(C, F.ctr, hh, C_NCTR);
        if (hh[C_ERR]) throw Error(SSP_ERR_CAPACITY, "factor: truncation overflow");
        out.truncated_rows = R;
        lvl++;
    }
    int64_t Lused = Lused_prev;
    // note: Lused_prev covers reservations up to the last processed level
    if (T > 0) {
        // dense tail
        int32_t* rem = W.get_t<int32_t>(nm("rem"), T + 1);
        int32_t* idx = W.get_t<int32_t>(nm("idx"), n);
        SSP_CUDA(cudaMemsetAsync(F.ctr + C_REM, 0, sizeof(int64_t), C.stream));
        k_collect_live<<<grid_for(n, T256), T256, 0, C.stream>>>(n, F.level, rem, F.ctr + C_REM);
        SSP_CHECK_LAUNCH();
        int32_t P = 2;
        while (P < T) P <<= 1;
        allow_dynamic_smem(C, k_sort_rem, (P * sizeof(int32_t)));
        k_sort_rem<<<1, 1024, P * sizeof(int32_t), C.stream>>>(rem, (int32_t)T, P, F.prio, idx);
        SSP_CHECK_LAUNCH();
        double* Wd = W.get_t<double>(nm("W"), (size_t)T * T);
        SSP_CUDA(cudaMemsetAsync(Wd, 0, sizeof(double) * T * T, C.stream));
        // bag sizes bound the build scratch
        const int32_t maxlen = device_max_i32(C, F.bag_len, n);
        int32_t cap = 64;
        while (cap < maxlen) cap <<= 1;
        if (cap <= BLOCK_TIER_MAX) {
            size_t smem = (size_t)cap * (2 * sizeof(double) + 2 * sizeof(int32_t));
            allow_dynamic_smem(C, k_dense_build, smem);
            k_dense_build<<<(int)std::min<int64_t>(T, 148 * 4), 256, smem, C.stream>>>(F, rem, (int32_t)T, idx, Wd,
                                                                                        cap, nullptr, nullptr, 0);
        } else {
            int blocks = 32;
            int32_t* gu = W.get_t<int32_t>(nm("gscr_u"), (size_t)2 * cap * blocks);
            double* gw = W.get_t<double>(nm("gscr_w"), (size_t)4 * cap * blocks);
            k_dense_build<<<blocks, 1024, 0, C.stream>>>(F, rem, (int32_t)T, idx, Wd, cap, gu, gw, 1);
        }
        SSP_CHECK_LAUNCH();
        // L room for the dense phase
        int64_t need = Lused + T * (T - 1) / 2 + 1;
        if (need > Lcap) {
            int64_t ncap = need;
            F.Lrow = (int32_t*)grow_keep(C, nm("Lrow"), F.Lrow, sizeof(int32_t) * Lused, sizeof(int32_t) * ncap);
            F.Lval = (double*)grow_keep(C, nm("Lval"), F.Lval, sizeof(double) * Lused, sizeof(double) * ncap);
            Lcap = ncap;
        }
        // the bitonic sort needs P = pow2 >= T slots per array
        size_t smem = (size_t)P * (2 * sizeof(double) + sizeof(int32_t));
        allow_dynamic_smem(C, k_dense_elim, smem);
        k_dense_elim<<<1, 1024, smem, C.stream>>>(F, rem, (int32_t)T, P, idx, Wd, Lused, sparse_levels);
        SSP_CHECK_LAUNCH();
        C.kernels_launched += 4;
        Lused += T * (T - 1) / 2;
        int64_t hh[C_NCTR];
        read_i64s(C, F.ctr, hh, C_NCTR);
        if (hh[C_ERR]) throw Error(SSP_ERR_CAPACITY, "factor: dense tail overflow");
    }
    out.n = n;
    out.num_levels = lvl + (int32_t)T;
    out.dense_levels = (int32_t)T;
    // compact columns
    out.col_ptr = W.get_t<int64_t>(nm("col_ptr"), n + 1);
    SSP_CUDA(cudaMemsetAsync(F.Lcnt + n, 0, sizeof(int32_t), C.stream));
    exclusive_scan_i32_to_i64(C, F.Lcnt, out.col_ptr, n + 1, d_tot);
    out.nnz = read_i64(C, d_tot);
    out.col_idx = W.get_t<int32_t>(nm("col_idx"), out.nnz + 1);
    out.col_val = W.get_t<double>(nm("col_val"), out.nnz + 1);
    k_copy_cols<<<grid_for(n * 32, T256, 148 * 64), T256, 0, C.stream>>>(n, F.Lstart, F.Lcnt, F.Lrow, F.Lval,
                                                                        out.col_ptr, out.col_idx, out.col_val);
    SSP_CHECK_LAUNCH();
    // row form
    int32_t* rowcnt = W.get_t<int32_t>(nm("rowcnt"), n + 1);
    int32_t* cursor = W.get_t<int32_t>(nm("rcursor"), n + 1);
    SSP_CUDA(cudaMemsetAsync(rowcnt, 0, sizeof(int32_t) * (n + 1), C.stream));
    SSP_CUDA(cudaMemsetAsync(cursor, 0, sizeof(int32_t) * (n + 1), C.stream));
    k_row_count<<<grid_for(out.nnz, T256), T256, 0, C.stream>>>(out.nnz, out.col_idx, rowcnt);
    SSP_CHECK_LAUNCH();
    out.row_ptr = W.get_t<int64_t>(nm("row_ptr"), n + 1);
    exclusive_scan_i32_to_i64(C, rowcnt, out.row_ptr, n + 1, nullptr);
    out.row_idx = W.get_t<int32_t>(nm("row_idx"), out.nnz + 1);
    out.row_val = W.get_t<double>(nm("row_val"), out.nnz + 1);
    k_row_scatter<<<grid_for(n * 32, T256, 148 * 64), T256, 0, C.stream>>>(n, out.col_ptr, out.col_idx, out.col_val,
                                                                          out.row_ptr, cursor, out.row_idx,
                                                                          out.row_val);
    SSP_CHECK_LAUNCH();
    C.kernels_launched += 4;
    // sort each row by column id (deterministic summation order in the forward solve)
    {
        int64_t* seg_start = out.row_ptr;
        const int32_t maxrow = device_max_i32(C, rowcnt, n);
        segsort_pairs_i32_f64(C, out.row_idx, out.row_val, seg_start, rowcnt, n, maxrow);
    }
    out.D = F.D;
    out.level = F.level;
    // level lists
    const int32_t NL = out.num_levels;
    int32_t* lvcnt = W.get_t<int32_t>(nm("lvcnt"), NL + 1);
    SSP_CUDA(cudaMemsetAsync(lvcnt, 0, sizeof(int32_t) * (NL + 1), C.stream));
    k_level_count<<<grid_for(n, T256), T256, 0, C.stream>>>(n, F.level, lvcnt);
    SSP_CHECK_LAUNCH();
    int64_t* lvptr = W.get_t<int64_t>(nm("lvptr64"), NL + 1);
    exclusive_scan_i32_to_i64(C, lvcnt, lvptr, NL + 1, nullptr);
    out.level_rows = W.get_t<int32_t>(nm("level_rows"), n);
    // a level's vertices by the length of their rows (columns) and then by id: neighbours in the order have about as much
    // work, and everything laid out from here on (and the order in which the solves add a row up) is the same in every run
    out.level_cols = W.get_t<int32_t>(nm("level_cols"), n);
    {
        // the elimination's lists are free now
        uint64_t* key = (uint64_t*)F.fstart;
        uint64_t* tkey = (uint64_t*)F.bag_start;
        int32_t* tval = list_b;
        int bits = 9;
        while (bits < 40 && (int64_t(256) << (bits - 8)) < (int64_t)NL * 256) bits++;
        for (int f = 0; f < 2; f++) {
            int32_t* order = f == 0 ? out.level_rows : out.level_cols;
            k_level_keys<<<grid_for(n, T256), T256, 0, C.stream>>>(n, F.level, f == 0 ? out.row_ptr : out.col_ptr, key, order);
            SSP_CHECK_LAUNCH();
            radix_sort_u64(C, key, order, n, bits, tkey, tval);
        }
    }
    out.level_ptr_d = W.get_t<int32_t>(nm("level_ptr"), NL + 1);
    k_i64_to_i32<<<grid_for(NL + 1, T256), T256, 0, C.stream>>>(NL + 1, lvptr, out.level_ptr_d);
    SSP_CHECK_LAUNCH();
    C.kernels_launched += 3;
    std::vector<int64_t> lp(NL + 1);
    SSP_CUDA(cudaMemcpyAsync(lp.data(), lvptr, sizeof(int64_t) * (NL + 1), cudaMemcpyDeviceToHost, C.stream));
    SSP_CUDA(cudaStreamSynchronize(C.stream));
    out.level_ptr.assign(NL + 1, 0);
    out.max_level_rows = 0;
    for (int32_t l = 0; l <= NL; l++) out.level_ptr[l] = (int32_t)lp[l];
    for (int32_t l = 0; l < NL; l++) out.max_level_rows = std::max(out.max_level_rows, (int32_t)(lp[l + 1] - lp[l]));
    // storage-order row and column forms + per-level chunk lists
    const int64_t drops = C.ws.drops();
    {
        int32_t* cnt = W.get_t<int32_t>(nm("permcnt"), n + 1);
        auto build = [&](const int32_t* order, const int64_t* ptr, const int32_t* idx, const double* val, const char* tagp,
                         int64_t** pptr, int32_t** pidx, double** pval, int32_t** chunks,
                         std::vector<int32_t>& chunk_lvl, std::vector<int64_t>& hp, FactorRow** prow, FactorEnt<double>** pent) {
            *pptr = W.get_t<int64_t>(nm(tagp) + "_ptr", n + 1);
            k_perm_count<<<grid_for(n, T256), T256, 0, C.stream>>>(n, order, ptr, cnt);
            SSP_CUDA(cudaMemsetAsync(cnt + n, 0, sizeof(int32_t), C.stream));
            exclusive_scan_i32_to_i64(C, cnt, *pptr, n + 1, nullptr);
            *pidx = W.get_t<int32_t>(nm(tagp) + "_idx", out.nnz + 1);
            *pval = W.get_t<double>(nm(tagp) + "_val", out.nnz + 1);
            *prow = W.get_optional_t<FactorRow>(nm(tagp) + "_row", n);
            *pent = W.get_optional_t<FactorEnt<double>>(nm(tagp) + "_ent", out.nnz + 1);
            k_perm_copy<<<grid_for(n * 32, T256, 148 * 64), T256, 0, C.stream>>>(n, order, ptr, idx, val,
                                                                                *pptr, *pidx, *pval, *prow, *pent);
            SSP_CHECK_LAUNCH();
            C.kernels_launched += 2;
            // a truncation's rows, the last level, are most of a large graph: they are cut into chunks on the device, and the
            // host, whose plans look at the levels before, does not get their pointers.  A last level of one row
            // (a complete elimination's) is not worth the launches and the wait, some 50 us.
            const int64_t last = NL > 0 ? lp[NL - 1] : 0;
            const bool on_dev = n - last > 4096;
            hp.resize((on_dev ? last : n) + 1);
            SSP_CUDA(cudaMemcpyAsync(hp.data(), *pptr, sizeof(int64_t) * hp.size(), cudaMemcpyDeviceToHost, C.stream));
            SSP_CUDA(cudaStreamSynchronize(C.stream));
            const int64_t last_nnz = out.nnz - hp[last];
            if (pptr == &out.prow_ptr) out.last_fwd_nnz = last_nnz;
            else out.last_bwd_nnz = last_nnz;
            std::vector<int32_t> starts;
            chunk_lvl.assign(NL + 1, 0);
            for (int32_t l = 0; l < NL; l++) {
                chunk_lvl[l] = (int32_t)starts.size();
                if (l + 1 < NL || !on_dev) make_chunks(hp, (int32_t)lp[l], (int32_t)lp[l + 1], starts);
            }
            const DevChunks D = device_chunks(C, *pptr, on_dev ? (int32_t)last : (int32_t)n, (int32_t)n, nm(tagp), starts);
            chunk_lvl[NL] = (int32_t)starts.size() + D.nchunks;
            *chunks = D.starts;
        };
        build(out.level_rows, out.row_ptr, out.row_idx, out.row_val, "prow", &out.prow_ptr, &out.prow_idx, &out.prow_val,
              &out.fchunk, out.fchunk_lvl, out.hfptr, &out.frow, &out.fent);
        build(out.level_cols, out.col_ptr, out.col_idx, out.col_val, "pcol", &out.pcol_ptr, &out.pcol_idx, &out.pcol_val,
              &out.bchunk, out.bchunk_lvl, out.hbptr, &out.brow, &out.bent);
    }
    // (a buffer above may have cost the first form's copies)
    out.ws_drops = drops;
    build_tail(C, out, T, T > 0 ? W.get_t<double>(nm("W"), (size_t)T * T) : nullptr, tag);
}

}  // namespace ssp
