// Brute-force kNN on the CUDA cores with a threshold known before the rows
// are read (every metric, fp32 and fp64): the plain path's keys and order.
//
// Keeping a running top-k per query inside the distance kernel costs more
// than the distances: every (query tile, row chunk) block starts with no
// threshold, so that all of its first keys go through merges, and the blocks'
// lists are merged once more.  Here three short passes give every query a
// bound first:
//   * knn_min_kernel: the keys of a sample, one row of every `step`; every
//     thread keeps the smallest of each query's keys that it sees, one value
//     per (query, 32 thread groups, block);
//   * knn_bound_kernel: the k-th smallest of those minima -- k keys of k
//     different rows, so the k-th neighbour's key is at most this bound;
//   * knn_append_kernel: the keys of all rows; those at or below the bound are
//     collected in shared memory and go to the query's list in global memory;
//   * knn_pick_kernel: sorts the list by (key, index) and writes its first k.
// A list that overflows raises the flag; the k-th of the keys that it holds is a
// closer bound, with which the caller runs the last two passes again for its
// query, and running lists (knn_chunk_kernel) where that does not help (ties).
// Fewer than k entries are all keys that are
// numbers: fewer than k finite minima leave the bound at +inf.
//
// The passes are bound by FP32 / FP64 issue (tile_sweep.cuh).  Measured on a
// B200, device time against running lists and their merge: 50,000 x 37 fp32,
// 1,000 queries, manhattan, k = 5: 223 us against 1,072; 10,000 x 32 fp64,
// 2,000 queries, k = 10: 186 against 655; whole calls of 16 queries on 16,000
// x 32 rows, k = 10: 86 us against 1,286; 130 queries on 30,000 x 24, k = 64:
// 0.2 ms against 49.
#include "b200_common.cuh"
#include "b200_kernels.hpp"
#include "tile_sweep.cuh"
#include <algorithm>
#include <cmath>

namespace b200 {

namespace {

B200_DEV float min_num(float a, float b) { return fminf(a, b); }
B200_DEV double min_num(double a, double b) { return fmin(a, b); }

// Block (query tile, part p): the smallest key of each query over 32 disjoint
// sets of the part's sample rows (thread column x two sets of its columns).
template <typename T, int ACC>
__global__ void __launch_bounds__(256, 2)
knn_min_kernel(const T *Q, int nq, const T *X, SampleRows rows, int n_sample, int part_rows, int ld,
               int d, const T *qn, const T *xn, int post, int kc, T p, T invp, T *minima,
               int groups) {
    constexpr int TM = SweepAcc<T, ACC>::TM, TN = SweepAcc<T, ACC>::TN;
    __shared__ SweepStage<T> st[2];
    const int tid = threadIdx.x, tm = tid / 16, tn = tid % 16;
    const int q0 = blockIdx.x * SW_BM;
    const int x_begin = blockIdx.y * part_rows, x_end = min(n_sample, x_begin + part_rows);
    T qv[TM], m[TM][2];
#pragma unroll
    for (int i = 0; i < TM; ++i) {
        const int gq = q0 + tm * 4 + i;
        qv[i] = (qn && gq < nq) ? qn[gq] : T(0);
        m[i][0] = m[i][1] = Lim<T>::inf();
    }
    SweepAcc<T, ACC> acc;
    sweep_tiles<T, ACC>(
        st, Q, nq, q0, X, rows, x_begin, x_end, ld, d, kc, p, acc, tid, [&](int x0) {
            sweep_post<T, ACC>(acc, post, qv, nq - q0 - tm * 4, xn, rows, x0, x_end, tn, invp,
                               [&](int i, T (&key)[TN]) {
#pragma unroll
                                   for (int j = 0; j < TN; ++j) {
                                       T &best = m[i][j & 1];
                                       // a NaN key never counts
                                       if (key[j] < best && x0 + SweepCols<T>::of(j, tn) < x_end)
                                           best = key[j];
                                   }
                               });
        });
#pragma unroll
    for (int i = 0; i < TM; ++i) {
        const int gq = q0 + tm * 4 + i;
        if (gq >= nq) continue;
        T *o = minima + (size_t)gq * groups + blockIdx.y * 32 + tn * 2;
        o[0] = m[i][0];
        o[1] = m[i][1];
    }
}

// Order-preserving bits of a key and back.
template <typename T> struct OrdBits;
template <> struct OrdBits<float> {
    using U = unsigned;
    static B200_DEV U of(float f) {
        const unsigned b = __float_as_uint(f);
        return (b & 0x80000000u) ? ~b : (b | 0x80000000u);
    }
    static B200_DEV float back(U o) {
        return __uint_as_float((o & 0x80000000u) ? (o & 0x7fffffffu) : ~o);
    }
};
template <> struct OrdBits<double> {
    using U = unsigned long long;
    static B200_DEV U of(double f) {
        const U b = (U)__double_as_longlong(f);
        return (b >> 63) ? ~b : (b | (1ull << 63));
    }
    static B200_DEV double back(U o) {
        return __longlong_as_double((long long)((o >> 63) ? (o & ~(1ull << 63)) : ~o));
    }
};

// One warp per query: the k-th smallest of the query's minima, folded to 32 R
// of them (the smaller of several is as good: k keys of k different rows stay
// at or below the k-th); +inf where fewer than k are finite: everything
// passes.  Found bit by bit from the top: the largest value with fewer than k
// below it (counting every value's rank took 256 us for 4,096 queries of 512
// minima, this 14).  Clears the query's list, its redo word and the overflow flag
// (cnt null: none of them).
template <typename T, int R>
__global__ void __launch_bounds__(128)
knn_bound_kernel(const T *minima, int groups, int nq, int k, T *bound, int *cnt, int *flag,
                 int *redo) {
    using O = OrdBits<T>;
    using U = typename O::U;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int q = blockIdx.x * 4 + warp;
    if (q >= nq) return;
    T v[R];
    U u[R];
#pragma unroll
    for (int r = 0; r < R; ++r) v[r] = Lim<T>::inf();
    for (int i = 0; i < groups; i += 32 * R)
#pragma unroll
        for (int r = 0; r < R; ++r) {
            const int e = i + 32 * r + lane;
            const T x = e < groups ? minima[(size_t)q * groups + e] : Lim<T>::inf();
            if (x < v[r]) v[r] = x;
        }
#pragma unroll
    for (int r = 0; r < R; ++r) u[r] = O::of(v[r]);
    U kth = 0;
    for (int bit = 8 * (int)sizeof(T) - 1; bit >= 0; --bit) {
        const U trial = kth | (U(1) << bit);
        int below = 0;
#pragma unroll
        for (int r = 0; r < R; ++r) below += u[r] < trial ? 1 : 0;
        if ((int)__reduce_add_sync(0xffffffffu, below) < k) kth = trial;
    }
    if (lane == 0) {
        bound[q] = O::back(kth);
        if (cnt) {
            cnt[q] = 0;
            redo[q] = 0;
            if (q == 0) *flag = 0;
        }
    }
}
template <typename T>
void bound_pass(const T *minima, int groups, int nq, int k, T *bound, int *cnt, int *flag,
                int *redo, cudaStream_t s) {
    const int nb = (nq + 3) / 4;
    if (k <= 16)
        knn_bound_kernel<T, 2><<<nb, 128, 0, s>>>(minima, groups, nq, k, bound, cnt, flag, redo);
    else if (k <= 64)
        knn_bound_kernel<T, 8><<<nb, 128, 0, s>>>(minima, groups, nq, k, bound, cnt, flag, redo);
    else
        knn_bound_kernel<T, 16><<<nb, 128, 0, s>>>(minima, groups, nq, k, bound, cnt, flag, redo);
}

// Block (query tile, row chunk): appends every (key, row) with key <= the
// query's bound to its list.  Hits wait in shared memory, HITS per query; one
// global reservation per query and block moves them, and what does not fit
// reserves its own slot until the list is full (its query then gets a closer
// bound from what it holds).
template <typename T> struct SelHits;
template <> struct SelHits<float> { static constexpr int N = 24; };
template <> struct SelHits<double> { static constexpr int N = 16; };

template <typename T, int ACC>
__global__ void __launch_bounds__(256, 2)
knn_append_kernel(const T *Q, int nq, const T *X, int nx, int ld, int d, const T *qn,
                  const T *xn, int post, int kc, T p, T invp, int chunk_rows, const T *bound,
                  int *cnt, T *list_key, int *list_idx, int cap) {
    constexpr int TM = SweepAcc<T, ACC>::TM, TN = SweepAcc<T, ACC>::TN, BM = SW_BM;
    constexpr int HITS = SelHits<T>::N;
    __shared__ SweepStage<T> st[2];
    __shared__ T hkey[BM][HITS];
    __shared__ int hidx[BM][HITS];
    __shared__ int hn[BM];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int tm = tid / 16, tn = tid % 16;
    const int q0 = blockIdx.x * BM;
    const int x_begin = blockIdx.y * chunk_rows, x_end = min(nx, x_begin + chunk_rows);
    if (tid < BM) hn[tid] = 0; // visible after the sweep's first barrier
    T qv[TM], thr[TM];
#pragma unroll
    for (int i = 0; i < TM; ++i) {
        const int gq = q0 + tm * 4 + i;
        qv[i] = (qn && gq < nq) ? qn[gq] : T(0);
        thr[i] = gq < nq ? bound[gq] : -Lim<T>::inf();
    }
    SweepAcc<T, ACC> acc;
    sweep_tiles<T, ACC>(
        st, Q, nq, q0, X, AllRows{}, x_begin, x_end, ld, d, kc, p, acc, tid, [&](int x0) {
            sweep_post<T, ACC>(
                acc, post, qv, nq - q0 - tm * 4, xn, AllRows{}, x0, x_end, tn, invp,
                [&](int i, T (&key)[TN]) {
                    // few keys pass: one test for the row first (the minimum
                    // of the keys that are not NaN)
                    T m = key[0];
#pragma unroll
                    for (int j = 1; j < TN; ++j) m = min_num(m, key[j]);
                    if (!(m <= thr[i])) return;
                    const int ql = tm * 4 + i;
                    if (q0 + ql >= nq) return;
#pragma unroll
                    for (int j = 0; j < TN; ++j) {
                        const int gx = x0 + SweepCols<T>::of(j, tn);
                        if (!(key[j] <= thr[i]) || gx >= x_end) continue;
                        const int pos = atomicAdd(&hn[ql], 1);
                        if (pos < HITS) {
                            hkey[ql][pos] = key[j];
                            hidx[ql][pos] = gx;
                        } else {
                            const int gp = atomicAdd(&cnt[q0 + ql], 1);
                            if (gp < cap) {
                                list_key[(size_t)(q0 + ql) * cap + gp] = key[j];
                                list_idx[(size_t)(q0 + ql) * cap + gp] = gx;
                            } else {
                                thr[i] = -Lim<T>::inf(); // full: it takes no more
                            }
                        }
                    }
                });
        });
    __syncthreads();
    for (int ql = warp; ql < BM; ql += 8) {
        const int gq = q0 + ql, h = min(hn[ql], HITS);
        if (gq >= nq || h == 0) continue;
        int base = 0;
        if (lane == 0) base = atomicAdd(&cnt[gq], h);
        base = __shfl_sync(0xffffffffu, base, 0);
        if (lane < h && base + lane < cap) {
            list_key[(size_t)gq * cap + base + lane] = hkey[ql][lane];
            list_idx[(size_t)gq * cap + base + lane] = hidx[ql][lane];
        }
    }
}

// One block per query: the listed entries sorted by (key, index), the first k
// written (tf 1: square root, 2: negated; past the last entry index -1, distance
// +inf).  A list that overflowed: its k-th key at the query's first output, and
// whether that is below the bound (redo 2) or not (1).
template <typename T>
__global__ void __launch_bounds__(128)
knn_pick_kernel(const int *cnt, const T *list_key, const int *list_idx, int cap, int k, int tf,
                const T *bound, T *ok, int *oi, int *flag, int *redo) {
    extern __shared__ __align__(16) unsigned char pick_sm[];
    T *sk = reinterpret_cast<T *>(pick_sm);           // cap
    int *si = reinterpret_cast<int *>(sk + cap);      // cap
    const int q = blockIdx.x;
    const bool over = cnt[q] > cap;
    const int m = min(cnt[q], cap);
    int np2 = 1;
    while (np2 < m) np2 <<= 1; // <= cap, a power of two
    for (int e = threadIdx.x; e < np2; e += 128) {
        sk[e] = e < m ? list_key[(size_t)q * cap + e] : Lim<T>::inf();
        si[e] = e < m ? list_idx[(size_t)q * cap + e] : 0x7fffffff;
    }
    __syncthreads();
    for (int size = 2; size <= np2; size <<= 1)
        for (int stride = size >> 1; stride > 0; stride >>= 1) {
            for (int h = threadIdx.x; h < np2 / 2; h += 128) {
                const int i = 2 * h - (h & (stride - 1)), j = i + stride;
                const bool asc = (i & size) == 0;
                const T ki = sk[i], kj = sk[j];
                const int ii = si[i], ij = si[j];
                if (key_less(kj, ij, ki, ii) == asc) {
                    sk[i] = kj;
                    sk[j] = ki;
                    si[i] = ij;
                    si[j] = ii;
                }
            }
            __syncthreads();
        }
    if (over) {
        if (threadIdx.x == 0) {
            *flag = 1;
            redo[q] = sk[k - 1] < bound[q] ? 2 : 1;
            ok[(size_t)q * k] = sk[k - 1];
        }
        return;
    }
    for (int r = threadIdx.x; r < k; r += 128) {
        T v = r < m ? sk[r] : Lim<T>::inf();
        if (tf == 1) v = sqrt_rn(v);
        else if (tf == 2) v = -v;
        ok[(size_t)q * k + r] = v;
        oi[(size_t)q * k + r] = r < m ? si[r] : -1;
    }
}

template <typename T, int ACC>
cudaError_t select_t(const T *Q, int nq, const T *X, int nx, int ld, int d, const T *qn,
                     const T *xn, const KnnArgs &a, const KnnSelPlan &pl, void *work, int tf,
                     T *ok, int *oi, int *flag, int *redo, const T *given, cudaStream_t s) {
    constexpr int BM = SW_BM, BN = SweepStage<T>::BN;
    const T p = T(a.p), invp = T(1.0 / (double)p);
    T *list_key = static_cast<T *>(work);
    T *minima = list_key + (size_t)nq * pl.cap;
    T *bound = minima + (size_t)nq * pl.groups;
    int *list_idx = reinterpret_cast<int *>(bound + nq);
    int *cnt = list_idx + (size_t)nq * pl.cap;
    const int qt = (nq + BM - 1) / BM;
    cudaError_t e = cudaSuccess;
    if (given) {
        e = cudaMemcpy2DAsync(bound, sizeof(T), given, a.k * sizeof(T), sizeof(T), nq,
                              cudaMemcpyDeviceToDevice, s);
        if (e == cudaSuccess) e = cudaMemsetAsync(cnt, 0, nq * sizeof(int), s);
        if (e == cudaSuccess) e = cudaMemsetAsync(redo, 0, nq * sizeof(int), s);
        if (e == cudaSuccess) e = cudaMemsetAsync(flag, 0, sizeof(int), s);
        if (e != cudaSuccess) return e;
    } else {
        knn_min_kernel<T, ACC><<<dim3(qt, pl.parts), 256, 0, s>>>(
            Q, nq, X, SampleRows{pl.step, nx}, pl.n_sample, pl.part_rows, ld, d, qn, xn, a.post,
            a.kc, p, invp, minima, pl.groups);
        bound_pass(minima, pl.groups, nq, a.k, bound, cnt, flag, redo, s);
    }
    // chunks of whole row tiles: about four blocks per SM slot (two slots per
    // SM), so that the last wave costs little
    const int tiles = (nx + BN - 1) / BN;
    int chunks = std::max(1, std::min(tiles, (148 * 8 + qt - 1) / qt));
    const int chunk_rows = (tiles + chunks - 1) / chunks * BN;
    chunks = (nx + chunk_rows - 1) / chunk_rows;
    knn_append_kernel<T, ACC><<<dim3(qt, chunks), 256, 0, s>>>(
        Q, nq, X, nx, ld, d, qn, xn, a.post, a.kc, p, invp, chunk_rows, bound, cnt, list_key,
        list_idx, pl.cap);
    const size_t smem = (size_t)pl.cap * (sizeof(T) + 4);
    e = ensure_smem_limit(reinterpret_cast<const void *>(knn_pick_kernel<T>), smem);
    if (e != cudaSuccess) return e;
    knn_pick_kernel<T><<<nq, 128, smem, s>>>(cnt, list_key, list_idx, pl.cap, a.k, tf, bound, ok, oi,
                                             flag, redo);
    return cudaGetLastError();
}

} // namespace

cudaError_t launch_knn_bound(const float *minima, int groups, int nq, int k, float *bound,
                             cudaStream_t s) {
    bound_pass<float>(minima, groups, nq, k, bound, nullptr, nullptr, nullptr, s);
    return cudaGetLastError();
}

// Sample, lists and whether the passes apply.  The sample is a sixteenth of
// the rows (1,024 to 16,384 of them), so the first pass adds a sixteenth to
// the work and a query is expected to list about 1.5 x 16 k keys; more rows
// for a large k, so that about 2,000 are listed at most.  At least 2 k minima
// keep their k-th close to the sample's k-th key.  The number listed varies
// like a sum of k exponentials: a list holds x times the expected number with
// k (x - 1 - ln x) above 18, one overflow in 10^7 queries.
bool knn_sel_plan(int n, int nq, int k, bool fp64, KnnSelPlan &pl) {
    const int BN = knn_tile_rows_train(fp64);
    if (nq < 1 || k < 1) return false;
    const double by_k = 1.5 * k * (double)n / 2000.0;
    const int want = (int)std::min<double>(n, std::max({1024.0, std::min(16384.0, n / 16.0), by_k}));
    pl.step = std::max(1, n / want);
    pl.n_sample = (n + pl.step - 1) / pl.step;
    const int tiles = (pl.n_sample + BN - 1) / BN;
    const int need = (2 * k + 31) / 32; // parts of 32 minima
    if (need > tiles || need * 32 > KNN_SEL_GROUPS) return false;
    // enough blocks to fill the SMs twice where the sample has the tiles
    const int qt = (nq + 63) / 64;
    pl.parts = std::min({tiles, KNN_SEL_GROUPS / 32, std::max(need, (148 * 2 + qt - 1) / qt)});
    pl.part_rows = (tiles + pl.parts - 1) / pl.parts * BN;
    pl.parts = (pl.n_sample + pl.part_rows - 1) / pl.part_rows;
    if (pl.parts < need) return false;
    pl.groups = pl.parts * 32;
    const double expected = std::min((double)n, 1.5 * k * ((double)n / pl.n_sample) + 16.0);
    const double room =
        pl.step == 1 ? std::min((double)n, 4.0 * k + 64.0) // the minima are over all rows
                     : std::min((double)n, expected * (1.0 + 6.0 / std::sqrt((double)k) + 15.0 / k));
    pl.cap = 128;
    while (pl.cap < room && pl.cap < KNN_SEL_CAP) pl.cap <<= 1;
    return pl.cap >= room;
}

size_t knn_sel_bytes(const KnnSelPlan &pl, int nq, bool fp64) {
    const size_t e = fp64 ? 8 : 4;
    return (size_t)nq * (pl.cap * (e + 4) + pl.groups * e + e + 4) + 256;
}

template <typename T>
cudaError_t launch_knn_select(const T *Q, int nq, const T *X, int nx, int ld, int d, const T *qn,
                              const T *xn, const KnnArgs &a, const KnnSelPlan &pl, void *work,
                              int tf, T *out_key, int *out_idx, int *flag, int *redo,
                              const T *given, cudaStream_t s) {
    switch (a.acc) {
    case ACC_SQEUC:
        return select_t<T, ACC_SQEUC>(Q, nq, X, nx, ld, d, qn, xn, a, pl, work, tf, out_key,
                                      out_idx, flag, redo, given, s);
    case ACC_DOT:
        return select_t<T, ACC_DOT>(Q, nq, X, nx, ld, d, qn, xn, a, pl, work, tf, out_key, out_idx,
                                    flag, redo, given, s);
    case ACC_MANHATTAN:
        return select_t<T, ACC_MANHATTAN>(Q, nq, X, nx, ld, d, qn, xn, a, pl, work, tf, out_key,
                                          out_idx, flag, redo, given, s);
    default:
        return select_t<T, ACC_MINKOWSKI>(Q, nq, X, nx, ld, d, qn, xn, a, pl, work, tf, out_key,
                                          out_idx, flag, redo, given, s);
    }
}
template cudaError_t launch_knn_select<float>(const float *, int, const float *, int, int, int,
                                              const float *, const float *, const KnnArgs &,
                                              const KnnSelPlan &, void *, int, float *, int *,
                                              int *, int *, const float *, cudaStream_t);
template cudaError_t launch_knn_select<double>(const double *, int, const double *, int, int, int,
                                               const double *, const double *, const KnnArgs &,
                                               const KnnSelPlan &, void *, int, double *, int *,
                                               int *, int *, const double *, cudaStream_t);

} // namespace b200
