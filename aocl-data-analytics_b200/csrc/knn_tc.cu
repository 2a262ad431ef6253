// Brute-force kNN (euclidean / squared euclidean, fp32 data) with a bf16
// tensor-core candidate pass and an exact fp32 re-score.
//
// Ranking value of train row j for query q: v'_j = |x_j|^2 - 2 x_j.q (the
// squared distance minus the query's own |q|^2).  The tcgen05 pass computes
// v'_tc from three bf16 products (x = xh + xl, -2q = qh + ql:
// xh.qh + xh.ql + xl.qh) accumulated in fp32 in TMEM, plus the fp32 |x_j|^2.
// A rigorous bound |v'_tc - v'_plain| <= eps_q (v'_plain: the plain path's
// fp32 squared distance, in the reference's accumulation order, minus |q|^2)
// gives the certificate: every row of the plain top-k has
// v'_tc <= v'_tc(k) + 2 eps_q, where v'_tc(k) is the k-th smallest v'_tc.
//
// Two passes of the same kernel.  The first, over an evenly strided sample of
// the rows, keeps minima of v'_tc over disjoint sets of rows; the k-th smallest
// of a query's minima is at least v'_tc(k), so theta_q = that + 2 eps_q admits
// every candidate (so does the k-th of any values listed, which a query whose list
// overflowed takes for another go).  The second appends every (v'_tc, j) with v'_tc < theta_q to
// the query's list.  The finalize kernel takes the k-th smallest listed v'_tc
// (that is v'_tc(k)), re-scores the listed rows within 2 eps_q of it exactly
// (the plain kernel's formula and order) and keeps the k best by (distance,
// index): the plain path's neighbours.
//
// The queries are the MMA's M side: a TMEM lane, so an epilogue thread, is one
// query.  Its threshold is a register, a value below it goes to the thread's
// own stash in shared memory, and the list costs one global reservation per
// full stash.  With the rows on the lanes every column needed its own
// threshold, its own atomics and a shared, locked refresh of thresholds that
// started loose: at 1M x 128, 4,096 queries, k = 100 that epilogue took 5.5 ms
// for 1.9 ms of tensor work, after 1.0 ms of threshold pre-pass on the CUDA
// cores.  Measured now: see launch_knn_tc.
#include "b200_common.cuh"
#include "b200_kernels.hpp"
#include "tc_common.cuh"
#include <algorithm>
#include <cuda_bf16.h>
#include <cmath>

namespace b200 {

using namespace tc;

namespace {

constexpr int TK_BM = 128;       // queries per M tile (UMMA M, TMEM lanes)
constexpr int TK_KB = 64;        // bf16 elements per 128-byte K block
constexpr int TK_THREADS = 320;  // TMA warp, MMA warp, 8 epilogue warps
constexpr int TK_COLS = 128;     // rows that one epilogue thread sees per tile
constexpr int TK_STASH = 8;      // values below threshold held per thread
constexpr int TK_CAP = 8192;     // listed values per query, at most
constexpr int TK_GROUPS = 512;   // sample minima per query, at most
// Tile: 128 queries x 256 rows (one accumulator set: 256 TMEM columns).  The
// rows' operand is read from shared memory once per MMA, so an MMA of 256 rows
// moves 12 KB for twice the work of the 8 KB of one of 128: 256 queries x 128
// rows per block (half the L2 reads) took 3.04 ms where this takes 2.46 (1M x
// 128, 4,096 queries).
constexpr int TK_ROWS = 256;     // train rows per tile (UMMA N)

struct KnnTcArgs {
    int nx, nq, nkb, stages, n_qtiles, n_xtiles, tiles, n_items, cap, groups;
    int kk_last; // K steps of 16 in the last K block (the rest are zero columns)
    int xstep;   // xnorm elements from one row to the next (sample pass)
    const float *xnorm;  // nx: fp32 |x_j|^2 (cosine: 1 / |x_j|)
    const float *bound;  // list pass: the k-th smallest sample minimum per query
    const float *margin; // per query: 2 eps_q (nudged up)
    float *minima;       // sample pass: nq x groups
    int *cnt;            // list and mask pass: values below the threshold per query
    unsigned *mask;      // mask pass: nq x n_xtiles * 8 words, a bit per train row
    int2 *list;          // nq * cap: (value bits, train row)
    int *err;
};

struct __align__(16) TkShared {
    uint64_t full[8], empty[8], tfull[2], tempty[2], qfull;
    uint32_t tmem_base;
    int abort_flag;
};

__device__ __forceinline__ unsigned ord_bits(float f) {
    const unsigned b = __float_as_uint(f);
    return (b & 0x80000000u) ? ~b : (b | 0x80000000u);
}
__device__ __forceinline__ float ord_float(unsigned o) {
    return __uint_as_float((o & 0x80000000u) ? (o & 0x7fffffffu) : ~o);
}
__device__ __forceinline__ float nudge_up(float t) {
    return t + fabsf(t) * 9.5367431640625e-7f + 1e-30f;
}
__device__ __forceinline__ void tk_raise(int *abort_flag, int *err, int code) {
    *((volatile int *)abort_flag) = 1;
    atomicExch(err, code);
}

// v[u] for a runtime u without dynamic register indexing (a tree of selects).
__device__ __forceinline__ float pick32(const float (&v)[32], int u) {
    float r[16];
#pragma unroll
    for (int i = 0; i < 16; ++i) r[i] = (u & 1) ? v[2 * i + 1] : v[2 * i];
#pragma unroll
    for (int i = 0; i < 8; ++i) r[i] = (u & 2) ? r[2 * i + 1] : r[2 * i];
#pragma unroll
    for (int i = 0; i < 4; ++i) r[i] = (u & 4) ? r[2 * i + 1] : r[2 * i];
    r[0] = (u & 8) ? r[1] : r[0];
    r[1] = (u & 8) ? r[3] : r[2];
    return (u & 16) ? r[1] : r[0];
}

// The ranking value of a train row: squared euclidean |x|^2 - 2 x.q (xs =
// |x|^2), or cosine -2 x.q / |x| with q normalised (xs = 1 / |x|), which is
// 2 (cosine distance - 1); of two neighbouring columns, one packed instruction.
template <bool COS> __device__ __forceinline__ void tk_val2(float &a, float &b, float xa, float xb) {
    unsigned long long v = (unsigned long long)__float_as_uint(a) |
                           ((unsigned long long)__float_as_uint(b) << 32);
    const unsigned long long x = (unsigned long long)__float_as_uint(xa) |
                                 ((unsigned long long)__float_as_uint(xb) << 32);
    if (COS) asm("mul.rn.f32x2 %0, %0, %1;" : "+l"(v) : "l"(x));
    else asm("add.rn.f32x2 %0, %0, %1;" : "+l"(v) : "l"(x));
    a = __uint_as_float((unsigned)v);
    b = __uint_as_float((unsigned)(v >> 32));
}

// What a pass writes: minima, lists, or (radius search) a bit per pair.
enum { TK_SAMPLE, TK_LIST, TK_MASK };

// One work item: query tile qt against `tiles` consecutive row tiles.
template <bool COS, int PASS>
__global__ void __launch_bounds__(TK_THREADS, 1)
knn_tc_kernel(const __grid_constant__ CUtensorMap tmQh, const __grid_constant__ CUtensorMap tmQl,
              const __grid_constant__ CUtensorMap tmXh, const __grid_constant__ CUtensorMap tmXl,
              KnnTcArgs a) {
    extern __shared__ __align__(1024) unsigned char tk_raw[];
    unsigned char *base = reinterpret_cast<unsigned char *>(
        (reinterpret_cast<uintptr_t>(tk_raw) + 1023) & ~uintptr_t(1023));
    const int S = a.stages, nkb = a.nkb;
    constexpr uint32_t kQ = TK_BM * 128u;   // one K block of the query tile (16 KB)
    constexpr uint32_t kX = TK_ROWS * 128u; // of a row tile (32 KB)
    unsigned char *Qh = base;
    unsigned char *Ql = Qh + (size_t)nkb * kQ;
    unsigned char *Xs = Ql + (size_t)nkb * kQ; // S stages of (Xh, Xl) for one K block
    float *xn_w = reinterpret_cast<float *>(Xs + (size_t)S * 2 * kX); // 8 warps x TK_COLS
    int2 *stash_w = reinterpret_cast<int2 *>(xn_w + 8 * TK_COLS);     // TK_STASH x 256 threads
    TkShared *sh = reinterpret_cast<TkShared *>(stash_w + (PASS == TK_LIST ? TK_STASH * 256 : 0));

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (threadIdx.x == 0) {
        for (int s = 0; s < S; ++s) {
            mbar_init(&sh->full[s], 1);
            mbar_init(&sh->empty[s], 1);
        }
        for (int b = 0; b < 2; ++b) {
            mbar_init(&sh->tfull[b], 1);
            mbar_init(&sh->tempty[b], 8 * 32);
        }
        mbar_init(&sh->qfull, 1);
        sh->abort_flag = 0;
        fence_barrier_init();
    }
    if (warp == 1) {
        tmem_alloc(&sh->tmem_base, 512u);
        tmem_relinquish();
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tbase = sh->tmem_base;
    const int xc = blockIdx.x / a.n_qtiles, qt = blockIdx.x % a.n_qtiles;
    const int x0 = xc * a.tiles, nt = min(a.tiles, a.n_xtiles - x0);

    if (warp == 0) {
        // ---------------------------------------------------- TMA producer --
        if (lane == 0) {
            prefetch_tmap(&tmQh);
            prefetch_tmap(&tmXh);
            mbar_arrive_expect_tx(&sh->qfull, (uint32_t)(2 * nkb) * kQ);
            for (int kb = 0; kb < nkb; ++kb) {
                tma_load_2d(&tmQh, &sh->qfull, Qh + (size_t)kb * kQ, kb * TK_KB, qt * TK_BM);
                tma_load_2d(&tmQl, &sh->qfull, Ql + (size_t)kb * kQ, kb * TK_KB, qt * TK_BM);
            }
            int us = 0;
            bool ok = true;
            for (int t = 0; ok && t < nt; ++t) {
                for (int kb = 0; kb < nkb; ++kb, ++us) {
                    const int s = us % S;
                    if (!mbar_wait(&sh->empty[s], (uint32_t)(((us / S) & 1) ^ 1))) {
                        tk_raise(&sh->abort_flag, a.err, 12);
                        ok = false;
                        break;
                    }
                    if (*((volatile int *)&sh->abort_flag)) {
                        ok = false;
                        break;
                    }
                    unsigned char *st = Xs + (size_t)s * 2 * kX;
                    mbar_arrive_expect_tx(&sh->full[s], 2 * kX);
                    tma_load_2d(&tmXh, &sh->full[s], st, kb * TK_KB, (x0 + t) * TK_ROWS);
                    tma_load_2d(&tmXl, &sh->full[s], st + kX, kb * TK_KB, (x0 + t) * TK_ROWS);
                }
            }
            // every issued load must have landed before exit
            mbar_wait(&sh->qfull, 0);
            for (int u = (us > S ? us - S : 0); u < us; ++u)
                mbar_wait(&sh->full[u % S], (uint32_t)((u / S) & 1));
        }
    } else if (warp == 1) {
        // ---------------------------------------------------- MMA issuer ----
        if (lane == 0) {
            const uint32_t idesc = idesc_bf16_f32(TK_BM, TK_ROWS);
            int us = 0, tc = 0;
            bool ok = mbar_wait(&sh->qfull, 0);
            if (!ok) tk_raise(&sh->abort_flag, a.err, 13);
            for (; ok && tc < nt; ++tc) {
                const int b = tc & 1;
                if (!mbar_wait(&sh->tempty[b], (uint32_t)(((tc >> 1) & 1) ^ 1))) {
                    tk_raise(&sh->abort_flag, a.err, 14);
                    ok = false;
                    break;
                }
                const uint32_t tacc = tbase + (uint32_t)(b * 256);
                for (int kb = 0; kb < nkb; ++kb, ++us) {
                    const int s = us % S;
                    if (!mbar_wait(&sh->full[s], (uint32_t)((us / S) & 1))) {
                        tk_raise(&sh->abort_flag, a.err, 15);
                        ok = false;
                        break;
                    }
                    if (*((volatile int *)&sh->abort_flag)) {
                        ok = false;
                        break;
                    }
                    tc_fence_after();
                    const uint32_t xh = smem_u32(Xs + (size_t)s * 2 * kX), xl = xh + kX;
                    const uint32_t qh = smem_u32(Qh + (size_t)kb * kQ);
                    const uint32_t ql = smem_u32(Ql + (size_t)kb * kQ);
                    const int nkk = kb == nkb - 1 ? a.kk_last : TK_KB / 16;
#pragma unroll
                    for (int kk = 0; kk < TK_KB / 16; ++kk) {
                        if (kk >= nkk) break;
                        const uint64_t dqh = desc_k_sw128(qh + kk * 32);
                        const uint64_t dql = desc_k_sw128(ql + kk * 32);
                        const uint64_t dxh = desc_k_sw128(xh + kk * 32);
                        mma_f16_ss(tacc, dqh, dxh, idesc, kb == 0 && kk == 0 ? 0u : 1u);
                        mma_f16_ss(tacc, dql, dxh, idesc, 1);
                        mma_f16_ss(tacc, dqh, desc_k_sw128(xl + kk * 32), idesc, 1);
                    }
                    mma_commit(&sh->empty[s]);
                }
                if (!ok) break;
                mma_commit(&sh->tfull[b]);
            }
            // the accumulators of the last tiles must be complete before the
            // TMEM is released
            for (int u = (tc > 2 ? tc - 2 : 0); u < tc; ++u)
                mbar_wait(&sh->tfull[u & 1], (uint32_t)((u >> 1) & 1));
        }
    } else {
        // ---------------------------------------------------- epilogue ------
        // Warp e reads the lanes of its quarter and the g-th half of the columns.
        const int e = warp - 2, g = e >> 2, quarter = warp & 3;
        const int q = qt * TK_BM + quarter * 32 + lane;
        const int row_off = g * TK_COLS;
        float *xs = xn_w + e * TK_COLS;
        int2 *stash = stash_w + e * 32 + lane; // entries 256 apart: no bank conflicts
        const float inf = __int_as_float(0x7f800000);
        // rows past the end never pass (+inf, or NaN for cosine)
        const float pad = COS ? __int_as_float(0x7fc00000) : inf;
        float theta = -inf, low[4] = {inf, inf, inf, inf};
        if (PASS != TK_SAMPLE && q < a.nq) theta = nudge_up(a.bound[q] + a.margin[q]);
        int ns = 0, found = 0;
        // the stashed values to the query's list; a full one takes no more (its
        // query gets a closer bound from what it holds)
        auto flush = [&]() {
            if (ns > 0) {
                const int at = atomicAdd(&a.cnt[q], ns);
                for (int i = 0; i < ns; ++i)
                    if (at + i < a.cap) a.list[(size_t)q * a.cap + at + i] = stash[i * 256];
                if (at + ns > a.cap) theta = -inf;
                ns = 0;
            }
        };
        auto norms = [&](int t) { // this lane's four of the half tile's 128
            const int r = (x0 + t) * TK_ROWS + row_off + lane * 4;
            float4 v = make_float4(pad, pad, pad, pad);
            if (a.xstep == 1 && r + 3 < a.nx) {
                v = *reinterpret_cast<const float4 *>(a.xnorm + r);
            } else {
                if (r < a.nx) v.x = a.xnorm[(size_t)r * a.xstep];
                if (r + 1 < a.nx) v.y = a.xnorm[(size_t)(r + 1) * a.xstep];
                if (r + 2 < a.nx) v.z = a.xnorm[(size_t)(r + 2) * a.xstep];
                if (r + 3 < a.nx) v.w = a.xnorm[(size_t)(r + 3) * a.xstep];
            }
            return v;
        };
        float4 xv = norms(0);
        for (int t = 0; t < nt; ++t) {
            const int b = t & 1;
            __syncwarp();
            *reinterpret_cast<float4 *>(xs + lane * 4) = xv;
            __syncwarp();
            if (t + 1 < nt) xv = norms(t + 1);
            bool ok = mbar_wait(&sh->tfull[b], (uint32_t)((t >> 1) & 1));
            if (!ok) tk_raise(&sh->abort_flag, a.err, 16);
            ok = ok && !*((volatile int *)&sh->abort_flag);
            if (!__all_sync(0xffffffffu, ok)) break;
            tc_fence_after();
            const uint32_t trow = tbase + ((uint32_t)(quarter * 32) << 16) +
                                  (uint32_t)(b * 256 + row_off);
            // two 32-column loads in flight: the latency of a TMEM load is that
            // of a chunk's arithmetic, and two warps a scheduler do not hide it
            float v[2][32];
            tmem_ld32_issue(trow, v[0]);
#pragma unroll 1
            for (int c2 = 0; c2 < TK_COLS / 32; c2 += 2) {
                unsigned word[2] = {0, 0}; // mask pass
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    const int c = c2 + h;
                    float(&w)[32] = v[h];
                    tmem_ld_wait(w);
                    if (c + 1 < TK_COLS / 32)
                        tmem_ld32_issue(trow + (uint32_t)((c + 1) * 32), v[h ^ 1]);
                    float mp[4] = {inf, inf, inf, inf}; // short chains: latency counts
#pragma unroll
                    for (int u = 0; u < 32; u += 4) {
                        const float4 x = *reinterpret_cast<const float4 *>(xs + c * 32 + u);
                        tk_val2<COS>(w[u], w[u + 1], x.x, x.y);
                        tk_val2<COS>(w[u + 2], w[u + 3], x.z, x.w);
                        float &a0 = mp[(u / 4) & 1], &a1 = mp[2 + ((u / 4) & 1)];
                        a0 = fminf(fminf(a0, w[u]), w[u + 1]);
                        a1 = fminf(fminf(a1, w[u + 2]), w[u + 3]);
                    }
                    const float m = fminf(fminf(mp[0], mp[1]), fminf(mp[2], mp[3]));
                    if (PASS == TK_SAMPLE) {
                        if (c2 == 0) low[h] = fminf(low[h], m);
                        else low[h + 2] = fminf(low[h + 2], m);
                        continue;
                    }
                    if (!__any_sync(0xffffffffu, m < theta)) continue;
                    unsigned part[4] = {0, 0, 0, 0};
#pragma unroll
                    for (int u = 0; u < 32; ++u) part[u & 3] |= (w[u] < theta ? 1u : 0u) << u;
                    unsigned bits = (part[0] | part[1]) | (part[2] | part[3]);
                    if (PASS == TK_MASK) {
                        word[h] = bits;
                        continue;
                    }
                    const int row = (x0 + t) * TK_ROWS + row_off + c * 32;
                    while (bits) {
                        if (ns == TK_STASH) flush();
                        const int u = __ffs(bits) - 1;
                        bits &= bits - 1;
                        stash[ns * 256] = make_int2(__float_as_int(pick32(w, u)), row + u);
                        ++ns;
                    }
                    __syncwarp();
                }
                if (PASS == TK_MASK && q < a.nq) {
                    found += __popc(word[0]) + __popc(word[1]);
                    *reinterpret_cast<uint2 *>(a.mask + ((size_t)q * a.n_xtiles + x0 + t) * 8 +
                                               g * 4 + c2) = make_uint2(word[0], word[1]);
                }
            }
            tc_fence_before();
            mbar_arrive(&sh->tempty[b]);
        }
        if (PASS == TK_MASK) {
            if (found > 0) atomicAdd(&a.cnt[q], found);
        } else if (PASS == TK_SAMPLE) {
            if (q < a.nq) {
                float *o = a.minima + (size_t)q * a.groups + (xc * 2 + g) * 4;
#pragma unroll
                for (int c = 0; c < 4; ++c) o[c] = low[c];
            }
        } else {
            flush();
        }
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 1) {
        tc_fence_after();
        tmem_dealloc(tbase, 512u);
    }
}

// -2q split into bf16 hi / lo (rows nq..nq_pad-1 zero) and the margins 2
// eps_q; the lists' lengths, the fallback flags and the state words cleared.
// Cosine (qnorm: the plain path's query norms): -2 q / |q| instead, and the
// margin 2 e1 for every query.  Radius search (bound): thr - |q|^2 per query, the
// fp32 |q|^2 within eps_q of the exact one; a query whose threshold is not
// finite gets none (NaN) and RADIUS_TC_NO values.
__global__ void knn_tc_prep_queries(const float *Q, int ld, int nq, int d, int nq_pad, int ldo,
                                    __nv_bfloat16 *Qh, __nv_bfloat16 *Ql, float e1, float e2,
                                    const float *xmax, float *margin, int *cnt, int *fallback,
                                    int *state, const float *qnorm, float *bound, float thr) {
    const int qi = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
    const int lane = threadIdx.x & 31;
    if (blockIdx.x == 0 && threadIdx.x < KNN_TC_STATE) state[threadIdx.x] = 0;
    if (qi >= nq_pad) return;
    const float qinv = (qnorm && qi < nq) ? __frcp_rn(qnorm[qi]) : 1.f;
    float s = 0.f;
    for (int f = lane; f < ldo; f += 32) {
        const float x = (qi < nq && f < d) ? Q[(size_t)qi * ld + f] : 0.f;
        s = __fmaf_rn(x, x, s);
        const float y = qnorm ? -2.f * __fmul_rn(x, qinv) : -2.f * x;
        const __nv_bfloat16 h = __float2bfloat16_rn(y);
        Qh[(size_t)qi * ldo + f] = h;
        Ql[(size_t)qi * ldo + f] = __float2bfloat16_rn(y - __bfloat162float(h));
    }
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) s += __shfl_xor_sync(0xffffffffu, s, off);
    if (lane == 0 && qi < nq) {
        const float qn = sqrtf(s) * 1.0001f;
        const float xm = qnorm ? 0.f : *xmax;
        const float eps = qnorm ? e1 : e1 * xm * qn + e2 * (xm * xm + qn * qn);
        margin[qi] = nudge_up(2.f * eps);
        cnt[qi] = 0;
        if (bound) {
            const float b = thr - s;
            const bool finite = isfinite(nudge_up(b + margin[qi]));
            bound[qi] = finite ? b : __int_as_float(0x7fc00000);
            if (!finite) cnt[qi] = RADIUS_TC_NO;
        } else {
            fallback[qi] = 0;
        }
    }
}

// The plain path's squared euclidean distance of one pair, in its exact
// accumulation order: per group of 4 dims, dims 4t, 4t+1 into g1 and
// 4t+2, 4t+3 into g2 (fma of the rounded difference), g1 += g2 at the end of
// every kc-block and of the last full group; remaining dims into g1.
// x: a row of the training set (16-byte aligned); q in shared memory.
__device__ __forceinline__ float sqeuc_ref(const float *x, const float *q, int d, int kc) {
    const int d4 = d & ~3;
    float g1 = 0.f, g2 = 0.f;
#pragma unroll 8
    for (int kg = 0; kg < d4; kg += 4) {
        const float4 xv = __ldg(reinterpret_cast<const float4 *>(x + kg));
        const float4 qv = *reinterpret_cast<const float4 *>(q + kg);
        const float t0 = __fsub_rn(qv.x, xv.x), t1 = __fsub_rn(qv.y, xv.y);
        const float t2 = __fsub_rn(qv.z, xv.z), t3 = __fsub_rn(qv.w, xv.w);
        g1 = __fmaf_rn(t0, t0, g1);
        g1 = __fmaf_rn(t1, t1, g1);
        g2 = __fmaf_rn(t2, t2, g2);
        g2 = __fmaf_rn(t3, t3, g2);
        if (((kg + 4) & (kc - 1)) == 0 || (kg + 4) == d4) { // kc: a power of two
            g1 = __fadd_rn(g1, g2);
            g2 = 0.f;
        }
    }
    for (int f = d4; f < d; ++f) {
        const float t = __fsub_rn(q[f], x[f]);
        g1 = __fmaf_rn(t, t, g1);
    }
    return g1;
}

// The plain path's cosine distance 1 - g / (|x| |q|), g one sequential fma
// chain over the features, the norms the plain path's.
__device__ __forceinline__ float cos_ref(const float *x, const float *q, int d, float xn,
                                         float qn) {
    float g = 0.f;
    for (int f = 0; f < d; ++f) g = __fmaf_rn(x[f], q[f], g);
    return __fsub_rn(1.f, __fdiv_rn(g, __fmul_rn(xn, qn)));
}

// The k-th smallest (1-based) of n keys in shared memory, by a radix select
// on four 8-bit digits, most significant first.  Block-wide (every thread
// gets the result); n >= k >= 1.
__device__ unsigned block_kth(const unsigned *keys, int n, int k, int *hist, int *sel) {
    unsigned prefix = 0, mask = 0;
    int kk = k; // rank of the wanted key among those matching prefix
    for (int shift = 24; shift >= 0; shift -= 8) {
        for (int b = threadIdx.x; b < 256; b += blockDim.x) hist[b] = 0;
        __syncthreads();
        for (int i = threadIdx.x; i < n; i += blockDim.x) {
            const unsigned u = keys[i];
            if ((u & mask) == prefix) atomicAdd(&hist[(u >> shift) & 255u], 1);
        }
        __syncthreads();
        if (threadIdx.x < 32) {
            const int lane = threadIdx.x;
            int c[8], sum = 0;
#pragma unroll
            for (int j = 0; j < 8; ++j) {
                c[j] = hist[lane * 8 + j];
                sum += c[j];
            }
            int inc = sum;
#pragma unroll
            for (int off = 1; off < 32; off <<= 1) {
                const int t = __shfl_up_sync(0xffffffffu, inc, off);
                if (lane >= off) inc += t;
            }
            const int exc = inc - sum;
            if (exc < kk && kk <= inc) { // this lane's 8 digits hold the kk-th key
                int run = exc, b = 7;
                for (int j = 0; j < 8; ++j) {
                    if (run + c[j] >= kk) {
                        b = j;
                        break;
                    }
                    run += c[j];
                }
                sel[0] = lane * 8 + b;
                sel[1] = kk - run;
            }
        }
        __syncthreads();
        prefix |= (unsigned)sel[0] << shift;
        mask |= 0xFFu << shift;
        kk = sel[1];
    }
    return prefix;
}

// One block per query: v'_tc(k) among the listed values, the exact distances of
// the rows within 2 eps_q of it, sorted by (distance, index); the first k are
// written (sqrt for euclidean).  A query whose list overflowed or is short of k
// is flagged, counted at state[0] and by reason at state[2] (overflow) and
// state[4] (short).  The k-th of an overflowed list's values, where it is below
// the query's bound by more than half the margin (which another go keeps), is its
// next one: flag 2, the value at its first output.
__global__ void __launch_bounds__(256)
knn_tc_finalize(const float *X, const float *Q, int ld, int d, int kc, int k, int cap,
                const float *margin, const float *bound, const int *cnt, const int2 *list, int take_sqrt,
                float *out_key, int *out_idx, int *fallback, int *state, const float *xnp,
                const float *qnp) {
    __shared__ int scount;
    __shared__ int hist[256], sel[2];
    extern __shared__ __align__(16) float fin_smem[];
    const int dp = (d + 3) & ~3;
    float *qs = fin_smem;                                    // d, padded
    unsigned *sval = reinterpret_cast<unsigned *>(qs + dp);  // cap: listed values, then keys
    int *srow = reinterpret_cast<int *>(sval + cap);         // cap: listed rows
    int *sidx = srow + cap;                                  // cap: survivors
    float *skey = reinterpret_cast<float *>(sval);
    const int qi = blockIdx.x;
    const bool over = cnt[qi] > cap;
    const int n = min(cnt[qi], cap);
    if (threadIdx.x == 0 && (over || n < k)) {
        fallback[qi] = 1;
        atomicAdd(state, 1);
        atomicAdd(state + (over ? 2 : 4), 1);
    }
    if (n < k) return;
    if (threadIdx.x == 0) scount = 0;
    for (int f = threadIdx.x; f < d; f += blockDim.x) qs[f] = Q[(size_t)qi * ld + f];
    for (int e = threadIdx.x; e < n; e += blockDim.x) {
        const int2 ev = list[(size_t)qi * cap + e];
        sval[e] = ord_bits(__int_as_float(ev.x));
        srow[e] = ev.y;
    }
    __syncthreads();
    const float kth = ord_float(block_kth(sval, n, k, hist, sel));
    if (over) {
        if (threadIdx.x == 0 && kth < bound[qi] - 0.5f * margin[qi]) {
            fallback[qi] = 2;
            out_key[(size_t)qi * k] = kth;
        }
        return;
    }
    const unsigned th = ord_bits(nudge_up(kth + margin[qi]));
    for (int e = threadIdx.x; e < n; e += blockDim.x)
        if (sval[e] < th) sidx[atomicAdd(&scount, 1)] = srow[e];
    __syncthreads();
    const int m = scount; // at least k: theirs are at most kth
    int np2 = 1;
    while (np2 < m) np2 <<= 1; // <= cap, a power of two
    for (int e = threadIdx.x; e < np2; e += blockDim.x) {
        if (e < m) {
            const float *x = X + (size_t)sidx[e] * ld;
            skey[e] = xnp ? cos_ref(x, qs, d, xnp[sidx[e]], qnp[qi]) : sqeuc_ref(x, qs, d, kc);
        } else {
            skey[e] = __int_as_float(0x7f800000);
            sidx[e] = 0x7fffffff;
        }
    }
    __syncthreads();
    // bitonic sort of (key, index) pairs, ascending
    for (int size = 2; size <= np2; size <<= 1) {
        for (int stride = size >> 1; stride > 0; stride >>= 1) {
            for (int h = threadIdx.x; h < np2 / 2; h += blockDim.x) {
                const int i = 2 * h - (h & (stride - 1)), j = i + stride;
                const bool asc = (i & size) == 0;
                const float ki = skey[i], kj = skey[j];
                const int ii = sidx[i], ij = sidx[j];
                if (key_less(kj, ij, ki, ii) == asc) {
                    skey[i] = kj;
                    skey[j] = ki;
                    sidx[i] = ij;
                    sidx[j] = ii;
                }
            }
            __syncthreads();
        }
    }
    for (int r = threadIdx.x; r < k; r += blockDim.x) {
        const float kv = skey[r];
        out_key[(size_t)qi * k + r] = take_sqrt ? __fsqrt_rn(kv) : kv;
        out_idx[(size_t)qi * k + r] = sidx[r];
    }
}

__global__ void max_value_kernel(const float *v, int n, float *out) {
    float m = 0.f;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
        m = fmaxf(m, v[i]);
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, off));
    if ((threadIdx.x & 31) == 0) atomicMax(reinterpret_cast<int *>(out), __float_as_int(m));
}
__global__ void sqrt_inplace_kernel(float *v) { *v = sqrtf(*v) * 1.0001f; }

// |v'_tc - v'_plain| <= e1 |x||q| + e2 (|x|^2 + |q|^2)  (u = 2^-24):
//   bf16 hi/lo split of x and of -2q, dropped lo.lo term: 3.1 2^-16 |x||2q|
//   fp32 accumulation of K_total = 3 Kp products in the tensor core
//   (allowing truncation): 2 K_total u |x||2q|
//   fp32 |x|^2 (Kp-term fma chain) and the final add: (Kp + 2) u |x|^2, u |2xq|
//   the plain path's direct-difference sum: (d + 4) u (|x| + |q|)^2
void sqeuc_error(int nkb, int d, double &e1, double &e2) {
    const double u = std::ldexp(1.0, -24);
    const double kp = (double)nkb * TK_KB, ktot = 3.0 * kp;
    e1 = 1.1 * (3.1 * std::ldexp(1.0, -16) * 2.0 + 2.0 * ktot * u * 2.0 + 2.0 * u +
                (d + 4.0) * u * 2.0);
    e2 = 1.1 * ((kp + 2.0) * u + (d + 4.0) * u * 2.0 + 2.0 * u);
}

size_t tk_smem_bytes(int nkb, int stages) {
    return 1024 + (size_t)nkb * 2 * TK_BM * 128 + (size_t)stages * 2 * TK_ROWS * 128 +
           (size_t)8 * TK_COLS * 4 + (size_t)TK_STASH * 256 * 8 + sizeof(TkShared) + 64;
}
constexpr size_t TK_SMEM = 225 * 1024;

// Row tiles per work item: about 32 (a block's start costs about one tile), in
// whole waves of one block per SM.
int tk_item_tiles(int n_xtiles, int n_qtiles) {
    const long long total = (long long)n_xtiles * n_qtiles, want = 32;
    const long long waves = std::max(1ll, (total + 74 * want) / (148 * want));
    const long long items = std::max(1ll, 148 * waves / n_qtiles);
    return (int)((n_xtiles + items - 1) / items);
}

} // namespace

int knn_tc_supported(int nx, int d, int k) {
    if (k < 1 || k > 256 || nx < k || d < 1) return 0;
    const int nkb = (d + TK_KB - 1) / TK_KB;
    return tk_smem_bytes(nkb, 2) <= TK_SMEM ? 1 : 0;
}

// List entries per query for a sample of every step-th row (see knn_tc_plan).
static int list_cap(int nx, int k, int step) {
    const double expected = 1.5 * 1.2 * k * step + 16.0;
    const double room = std::min((double)nx, expected * (1.0 + 6.0 / std::sqrt((double)k) + 15.0 / k));
    int cap = 512;
    while (cap < room && cap < TK_CAP) cap <<= 1;
    return cap;
}

// Every step-th row: a prime, so that rows in a cyclic order (a customer in turn, an
// hour of the day) are met in all their phases unless the period is a multiple of
// it; not 7, days of the week being common, where 11 does.  The next one up (a
// smaller sample) if the lists stay as long, else the next one down.
static int sample_step(int nx, int k, int want, int most) {
    auto prime = [](int v) {
        for (int q = 2; q * q <= v; ++q)
            if (v % q == 0) return false;
        return true;
    };
    const int s = std::max(1, std::min(want, most));
    if (s == 1) return 1;
    int up = s >= 7 ? std::max(s, 11) : s, down = s;
    while (!prime(up)) ++up;
    while (!prime(down)) --down;
    return up <= most && list_cap(nx, k, up) == list_cap(nx, k, s) ? up : down;
}

// Sample, lists.  A query is expected to list about 1.2 k times the inverse of
// the sampled share: an eighth of the rows at most (the sample pass costs its
// share of the tensor work), about a 20th at least, else the share that lists
// about 512; more where a short set would give fewer than 2 k minima.  A list holds x
// times that with k (x - 1 - ln x) above 18 (the number varies like a sum of k
// exponentials), and half as much again for the margin.
KnnTcPlan knn_tc_plan(int nx, int nq, int k) {
    KnnTcPlan p;
    constexpr int slots = 8, rows = TK_ROWS; // minima of a work item
    const double share = std::min(1.0 / 8.0, std::max(1.0 / 20.0, 1.2 * k / 512.0));
    const int least_rows = (2 * k + slots - 1) / slots * rows;
    p.step = sample_step(nx, k, (int)(1.0 / share), nx / least_rows);
    p.n_sample = (nx + p.step - 1) / p.step;
    const int n_qtiles = (nq + TK_BM - 1) / TK_BM;
    const int tiles = (p.n_sample + rows - 1) / rows;
    // minima: 4 k where the sample has the tiles, at most TK_GROUPS
    const int most = std::min(tiles, TK_GROUPS / slots);
    const int least = std::min(most, (4 * k + slots - 1) / slots);
    const int items = std::max(least, std::min(most, (148 + n_qtiles - 1) / n_qtiles));
    p.sample_tiles = (tiles + items - 1) / items;
    p.groups = (tiles + p.sample_tiles - 1) / p.sample_tiles * slots;
    p.cap = list_cap(nx, k, p.step);
    p.tiles = tk_item_tiles((nx + TK_ROWS - 1) / TK_ROWS, n_qtiles);
    return p;
}

__global__ void recip_kernel(const float *v, int n, float *out) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) out[i] = __frcp_rn(v[i]);
}
cudaError_t launch_recip(const float *v, int n, float *out, cudaStream_t s) {
    if (n <= 0) return cudaSuccess;
    recip_kernel<<<(n + 255) / 256, 256, 0, s>>>(v, n, out);
    return cudaGetLastError();
}

cudaError_t launch_knn_tc_train_prep(const float *X, int ld, int nx, int d, void *Xh, void *Xl,
                                     int ldbf, float *xnorm2, float *xmax, cudaStream_t s) {
    cudaError_t e = launch_split_bf16(X, ld, nx, d, Xh, Xl, ldbf, s);
    if (e != cudaSuccess) return e;
    e = launch_row_sqnorms<float>(X, ld, nx, d, xnorm2, s);
    if (e != cudaSuccess) return e;
    e = cudaMemsetAsync(xmax, 0, sizeof(float), s);
    if (e != cudaSuccess) return e;
    max_value_kernel<<<148 * 4, 256, 0, s>>>(xnorm2, nx, xmax);
    sqrt_inplace_kernel<<<1, 1, 0, s>>>(xmax);
    return cudaGetLastError();
}

// Device time on a B200 at 1M x 128, 4,096 queries, k = 100: 2.83 ms (list pass
// 2.45 under ncu -- 2.05 of it the MMAs, 1.87 at the measured cuBLAS rate --,
// sample pass 0.25, finalize 0.18; 1,296 listed a query), 7.32 ms before (see the
// top); with every 8th row sampled instead of every 11th 0.33 and 0.17, 925 listed,
// the sum the same.  At 1M x 96, one query, k = 10: 109 us (list pass 79, 4.9 TB/s
// of the bf16 rows), 228 before.
// Variants that were slower at the first size (list pass): all warps storing
// hits to global memory as they find them 4.6 ms, a warp handling one query's
// hits together 2.8, hi and lo rows in separate 32 KB stages 3.1, sixteen
// epilogue warps 2.56.
cudaError_t launch_knn_tc(const float *X, const void *Xh, const void *Xl, const float *xnorm2,
                          const float *xmax, int nx, int ld, int ldbf, int d, const float *Q,
                          int nq, int k, int kc, int take_sqrt, const KnnTcPlan &pl, void *qbuf,
                          void *list, int *fallback, int *cnt, int *state, float *out_key,
                          int *out_idx, cudaStream_t s, const KnnTcCosine *cosine,
                          const float *given) {
    // ldbf: the bf16 rows' length (d rounded up to 8, at least 64); the MMA
    // runs nkb K blocks of 64, the last with only the 16-column steps that
    // hold data (the tensor maps zero-fill the columns past ldbf)
    const int nkb = (ldbf + TK_KB - 1) / TK_KB;
    const int n_qtiles = (nq + TK_BM - 1) / TK_BM, nq_pad = n_qtiles * TK_BM;
    unsigned char *p = static_cast<unsigned char *>(qbuf);
    __nv_bfloat16 *Qh = reinterpret_cast<__nv_bfloat16 *>(p);
    __nv_bfloat16 *Ql = Qh + (size_t)nq_pad * ldbf;
    float *margin = reinterpret_cast<float *>(Ql + (size_t)nq_pad * ldbf);
    float *bound = margin + nq_pad;
    float *minima = bound + nq_pad;
    double e1, e2;
    sqeuc_error(nkb, d, e1, e2);
    const double u = std::ldexp(1.0, -24);
    const double kp = (double)nkb * TK_KB, ktot = 3.0 * kp;
    // cosine, r = -2 x.q / (|x| |q|) = 2 (distance - 1), |x|, |q| the plain
    // path's norms: bf16 hi/lo split and fp32 accumulation as above on unit-
    // scale products, the scalings by 1/|q| and 1/|x| (4 u), and twice the
    // plain distance's own error (d fma terms, the product, division and
    // subtraction: (d + 6) u)
    const double ec = 1.1 * (2.0 * (3.1 * std::ldexp(1.0, -16) + 2.0 * ktot * u + 4.0 * u) +
                             2.0 * (d + 6.0) * u);
    const bool cosm = cosine != nullptr;
    const int wpb = 8;
    knn_tc_prep_queries<<<(nq_pad + wpb - 1) / wpb, wpb * 32, 0, s>>>(
        Q, ld, nq, d, nq_pad, ldbf, Qh, Ql, (float)(cosm ? ec : e1), (float)e2, xmax, margin, cnt,
        fallback, state, cosm ? cosine->qnorm : nullptr, nullptr, 0.f);
    KnnTcArgs a;
    a.nq = nq;
    a.nkb = nkb;
    a.kk_last = (d - (nkb - 1) * TK_KB + 15) / 16;
    a.n_qtiles = n_qtiles;
    a.cap = pl.cap;
    a.groups = pl.groups;
    a.xnorm = cosm ? cosine->xinv : xnorm2;
    a.bound = bound;
    a.margin = margin;
    a.minima = minima;
    a.cnt = cnt;
    a.list = static_cast<int2 *>(list);
    a.err = state + 1;
    a.stages = 8;
    while (a.stages > 2 && tk_smem_bytes(nkb, a.stages) > TK_SMEM) --a.stages;
    const size_t smem = tk_smem_bytes(nkb, a.stages);
    CUtensorMap mqh, mql, mxh, mxl;
    if (!make_map_bf16_rows(&mqh, Qh, nq_pad, ldbf, TK_BM) ||
        !make_map_bf16_rows(&mql, Ql, nq_pad, ldbf, TK_BM))
        return cudaErrorInvalidValue;
    if (given) {
        const cudaError_t e = cudaMemcpy2DAsync(bound, sizeof(float), given, k * sizeof(float),
                                                sizeof(float), nq, cudaMemcpyDeviceToDevice, s);
        if (e != cudaSuccess) return e;
    }
    for (int pass = given ? 1 : 0; pass < 2; ++pass) {
        const bool sample = pass == 0;
        a.xstep = sample ? pl.step : 1;
        a.nx = sample ? pl.n_sample : nx;
        a.n_xtiles = (a.nx + TK_ROWS - 1) / TK_ROWS;
        a.tiles = sample ? pl.sample_tiles : pl.tiles;
        a.n_items = n_qtiles * ((a.n_xtiles + a.tiles - 1) / a.tiles);
        if (!make_map_bf16_rows(&mxh, Xh, a.nx, ldbf, TK_ROWS, a.xstep) ||
            !make_map_bf16_rows(&mxl, Xl, a.nx, ldbf, TK_ROWS, a.xstep))
            return cudaErrorInvalidValue;
        using Kern = void (*)(CUtensorMap, CUtensorMap, CUtensorMap, CUtensorMap, KnnTcArgs);
        const Kern kern =
            sample ? (cosm ? knn_tc_kernel<true, TK_SAMPLE> : knn_tc_kernel<false, TK_SAMPLE>)
                   : (cosm ? knn_tc_kernel<true, TK_LIST> : knn_tc_kernel<false, TK_LIST>);
        cudaError_t e = ensure_smem_limit(reinterpret_cast<const void *>(kern), smem);
        if (e != cudaSuccess) return e;
        // one block per work item: blocks end often, so the kernels of a
        // higher-priority stream get SMs within one item's time
        kern<<<a.n_items, TK_THREADS, smem, s>>>(mqh, mql, mxh, mxl, a);
        e = cudaGetLastError();
        if (e != cudaSuccess) return e;
        if (sample) {
            e = launch_knn_bound(minima, pl.groups, nq, k, bound, s);
            if (e != cudaSuccess) return e;
        }
    }
    const size_t fsm = (size_t)((d + 3) & ~3) * sizeof(float) + (size_t)pl.cap * 12;
    cudaError_t e = ensure_smem_limit(reinterpret_cast<const void *>(knn_tc_finalize), fsm);
    if (e != cudaSuccess) return e;
    knn_tc_finalize<<<nq, 256, fsm, s>>>(X, Q, ld, d, kc, k, pl.cap, margin, bound, cnt,
                                         static_cast<const int2 *>(list), cosm ? 0 : take_sqrt,
                                         out_key, out_idx, fallback, state,
                                         cosm ? cosine->xnorm : nullptr,
                                         cosm ? cosine->qnorm : nullptr);
    return cudaGetLastError();
}

// Rows of w words: from rows idx[i] of src to rows i of dst, or the other way.
__global__ void rows_move_kernel(const int *src, int w, const int *idx, int m, int *dst, int gather) {
    const size_t e = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (e >= (size_t)m * w) return;
    const int i = (int)(e / w), c = (int)(e % w);
    const size_t far = (size_t)idx[i] * w + c;
    if (gather) dst[e] = src[far];
    else dst[far] = src[e];
}
static cudaError_t rows_move(const void *src, size_t row_bytes, const int *idx, int m, void *dst,
                             int gather, cudaStream_t s) {
    const size_t w = row_bytes / 4, n = (size_t)m * w;
    if (n == 0) return cudaSuccess;
    rows_move_kernel<<<(unsigned)((n + 255) / 256), 256, 0, s>>>(
        static_cast<const int *>(src), (int)w, idx, m, static_cast<int *>(dst), gather);
    return cudaGetLastError();
}
cudaError_t launch_rows_gather(const void *src, size_t row_bytes, const int *idx, int m, void *dst,
                               cudaStream_t s) {
    return rows_move(src, row_bytes, idx, m, dst, 1, s);
}
cudaError_t launch_rows_scatter(const void *src, size_t row_bytes, const int *idx, int m, void *dst,
                                cudaStream_t s) {
    return rows_move(src, row_bytes, idx, m, dst, 0, s);
}

// ------------------------------------------------------ radius search ---
// The mask pass sets a bit for every pair whose v'_tc is below the query's
// threshold (thr - |q|^2 + 2 eps_q): every row the plain path finds within thr,
// in index order, whatever their number.  The offsets of a query's set bits
// follow, and one block per query computes the plain path's distances of its
// rows, keeping those at most thr.

// off[q] = cnt[0] + .. + cnt[q - 1], *total = all.  One block.
__global__ void __launch_bounds__(1024)
radius_cand_scan(const int *cnt, int nq, long long *off, long long *total) {
    __shared__ long long part[32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    long long before = 0;
    for (int q0 = 0; q0 < nq; q0 += 1024) {
        const int q = q0 + threadIdx.x;
        const long long c = q < nq ? cnt[q] : 0;
        long long inc = c;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const long long t = __shfl_up_sync(0xffffffffu, inc, o);
            if (lane >= o) inc += t;
        }
        if (lane == 31) part[warp] = inc;
        __syncthreads();
        long long add = before, all = 0;
        for (int w = 0; w < 32; ++w) {
            if (w < warp) add += part[w];
            all += part[w];
        }
        if (q < nq) off[q] = add + inc - c;
        before += all;
        __syncthreads();
    }
    if (threadIdx.x == 0) *total = before;
}

// A query's candidates: the set bits of its mask row gather in a shared list
// (the bits are sparse: without it most threads of the distances below would
// idle), RX_LIST at a time.
constexpr int RX_THREADS = 256, RX_LIST = 2048;
__global__ void __launch_bounds__(RX_THREADS)
radius_exact_kernel(const float *X, const float *Q, int ld, int d, int kc, float thr,
                    const unsigned *mask, int words, const int *cnt, const long long *off,
                    int *hits, int *idx, float *val) {
    extern __shared__ __align__(16) float rx_smem[];
    __shared__ int rows[RX_LIST], part[RX_THREADS / 32];
    const int q = blockIdx.x, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    if (cnt[q] == 0) {
        if (tid == 0) hits[q] = 0;
        return;
    }
    for (int f = tid; f < d; f += RX_THREADS) rx_smem[f] = Q[(size_t)q * ld + f];
    // the sum over the block of v before this thread's, and over all
    auto scan = [&](int v, int &all) {
        int inc = v;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int t = __shfl_up_sync(0xffffffffu, inc, o);
            if (lane >= o) inc += t;
        }
        __syncthreads(); // part is free again
        if (lane == 31) part[warp] = inc;
        __syncthreads();
        int add = 0;
        all = 0;
#pragma unroll
        for (int w = 0; w < RX_THREADS / 32; ++w) {
            if (w < warp) add += part[w];
            all += part[w];
        }
        return add + inc - v;
    };
    int have = 0, kept = 0;
    auto emit = [&]() { // the listed rows
        __syncthreads();
        for (int i0 = 0; i0 < have; i0 += RX_THREADS) {
            const int i = i0 + tid;
            float v = 0.f;
            if (i < have) v = sqeuc_ref(X + (size_t)rows[i] * ld, rx_smem, d, kc);
            const bool in = i < have && v <= thr;
            int all;
            const int at = scan(in ? 1 : 0, all);
            if (in) {
                idx[off[q] + kept + at] = rows[i];
                val[off[q] + kept + at] = v;
            }
            kept += all;
        }
        have = 0;
        __syncthreads();
    };
    const uint4 *m4 = reinterpret_cast<const uint4 *>(mask + (size_t)q * words);
    for (int w0 = 0; w0 < words / 4; w0 += RX_THREADS) {
        uint4 m = make_uint4(0, 0, 0, 0);
        if (w0 + tid < words / 4) m = m4[w0 + tid];
        const unsigned wd[4] = {m.x, m.y, m.z, m.w};
        int all;
        const int at = scan(__popc(m.x) + __popc(m.y) + __popc(m.z) + __popc(m.w), all);
        for (int done = 0; done < all;) {
            const int take = min(RX_LIST - have, all - done);
            int p = at - done; // of this thread's first bit, from the window's start
#pragma unroll
            for (int u = 0; u < 4; ++u)
                for (unsigned b = wd[u]; b; b &= b - 1, ++p)
                    if (p >= 0 && p < take)
                        rows[have + p] = (w0 + tid) * 128 + u * 32 + __ffs(b) - 1;
            have += take;
            done += take;
            if (have == RX_LIST) emit();
        }
    }
    emit();
    if (tid == 0) hits[q] = kept;
}

size_t radius_tc_query_bytes(int nq, int ldbf) {
    const size_t nq_pad = ((size_t)nq + TK_BM - 1) / TK_BM * TK_BM;
    return nq_pad * ldbf * 2 * 2 + nq_pad * 8 + 256;
}
int radius_tc_words(int nx) { return (nx + TK_ROWS - 1) / TK_ROWS * 8; }

// Device time at 200,000 x 32, 2,000 queries, 140,000 hits: 185 us (the mask 136), where a
// block of distances written, counted and compacted takes 2.03 ms (1.44 of it
// the distances).  Bound by the epilogue's instructions (1.5 per pair).
cudaError_t launch_radius_tc(const void *Xh, const void *Xl, const float *xnorm2,
                             const float *xmax, int nx, int ld, int ldbf, int d, const float *Q,
                             int nq, float thr, void *qbuf, unsigned *mask, int *cnt, int *state,
                             cudaStream_t s) {
    const int nkb = (ldbf + TK_KB - 1) / TK_KB;
    const int n_qtiles = (nq + TK_BM - 1) / TK_BM, nq_pad = n_qtiles * TK_BM;
    __nv_bfloat16 *Qh = static_cast<__nv_bfloat16 *>(qbuf);
    __nv_bfloat16 *Ql = Qh + (size_t)nq_pad * ldbf;
    float *margin = reinterpret_cast<float *>(Ql + (size_t)nq_pad * ldbf);
    float *bound = margin + nq_pad;
    double e1, e2;
    sqeuc_error(nkb, d, e1, e2);
    const int wpb = 8;
    knn_tc_prep_queries<<<(nq_pad + wpb - 1) / wpb, wpb * 32, 0, s>>>(
        Q, ld, nq, d, nq_pad, ldbf, Qh, Ql, (float)e1, (float)e2, xmax, margin, cnt, nullptr,
        state, nullptr, bound, thr);
    KnnTcArgs a{};
    a.nx = nx;
    a.nq = nq;
    a.nkb = nkb;
    a.kk_last = (d - (nkb - 1) * TK_KB + 15) / 16;
    a.n_qtiles = n_qtiles;
    a.n_xtiles = (nx + TK_ROWS - 1) / TK_ROWS;
    a.tiles = tk_item_tiles(a.n_xtiles, n_qtiles);
    a.n_items = n_qtiles * ((a.n_xtiles + a.tiles - 1) / a.tiles);
    a.xstep = 1;
    a.xnorm = xnorm2;
    a.bound = bound;
    a.margin = margin;
    a.cnt = cnt;
    a.mask = mask;
    a.err = state + 1;
    a.stages = 8;
    while (a.stages > 2 && tk_smem_bytes(nkb, a.stages) > TK_SMEM) --a.stages;
    const size_t smem = tk_smem_bytes(nkb, a.stages);
    CUtensorMap mqh, mql, mxh, mxl;
    if (!make_map_bf16_rows(&mqh, Qh, nq_pad, ldbf, TK_BM) ||
        !make_map_bf16_rows(&mql, Ql, nq_pad, ldbf, TK_BM) ||
        !make_map_bf16_rows(&mxh, Xh, nx, ldbf, TK_ROWS, 1) ||
        !make_map_bf16_rows(&mxl, Xl, nx, ldbf, TK_ROWS, 1))
        return cudaErrorInvalidValue;
    const auto kern = knn_tc_kernel<false, TK_MASK>;
    const cudaError_t e = ensure_smem_limit(reinterpret_cast<const void *>(kern), smem);
    if (e != cudaSuccess) return e;
    kern<<<a.n_items, TK_THREADS, smem, s>>>(mqh, mql, mxh, mxl, a);
    return cudaGetLastError();
}
cudaError_t launch_radius_cand_scan(const int *cnt, int nq, long long *off, long long *total,
                                    cudaStream_t s) {
    radius_cand_scan<<<1, 1024, 0, s>>>(cnt, nq, off, total);
    return cudaGetLastError();
}
cudaError_t launch_radius_exact(const float *X, int nx, int ld, int d, const float *Q, int nq,
                                int kc, float thr, const unsigned *mask, const int *cnt,
                                const long long *off, int *hits, int *idx, float *val,
                                cudaStream_t s) {
    const size_t smem = (size_t)((d + 3) & ~3) * sizeof(float);
    radius_exact_kernel<<<nq, RX_THREADS, smem, s>>>(X, Q, ld, d, kc, thr, mask,
                                                     radius_tc_words(nx), cnt, off, hits, idx, val);
    return cudaGetLastError();
}

size_t knn_tc_query_bytes(int nq, int ldbf, const KnnTcPlan &pl) {
    const size_t nq_pad = ((size_t)nq + TK_BM - 1) / TK_BM * TK_BM;
    return nq_pad * ldbf * 2 * 2 + nq_pad * 8 + (size_t)nq * pl.groups * 4 + 256;
}

} // namespace b200
