// Register-tiled pair values on the CUDA cores, several row tiles in one
// pipeline (pairwise distances, the kNN selection passes, the radius block).
// The values are those of the accumulation-order contract in dist_simt.cu:
// per pair and feature the same operations, in the same order and rounding.
//
// A block of 256 threads holds BM = 64 rows of A against tiles of BN rows of
// B; a thread's micro-tile is 4 x 8 pairs (fp32) or 4 x 4 (fp64).  Bound: the
// FP pipes -- 36 T fp32 (17.6 T fp64) element operations a second on a B200,
// two per pair and feature for differences, one for products.  The packed fp32
// instructions (two columns at a time) do not raise that rate, but they halve
// the issue slots it takes, which the shared-memory loads and the loop need.
// 4,001 x 3,001 x 96 squared euclidean fp32 (64 us at that rate): 126 us;
// scalar code with per-group order checks, operands loaded where they are used
// and one tile per block took 165.  A's values are staged twice over, (x, x),
// so that a packed operand is one part of a 16-byte load.
#pragma once
#include "simt_engine.cuh"

namespace b200 {

using pk2 = unsigned long long; // two fp32: low word first

B200_DEV pk2 pk_sub(pk2 a, pk2 b) {
    pk2 r;
    asm("sub.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
B200_DEV pk2 pk_fma(pk2 a, pk2 b, pk2 c) {
    pk2 r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
    return r;
}
B200_DEV pk2 pk_add(pk2 a, pk2 b) {
    pk2 r;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
B200_DEV float pk_lo(pk2 v) { return __uint_as_float((unsigned)v); }
B200_DEV float pk_hi(pk2 v) { return __uint_as_float((unsigned)(v >> 32)); }
B200_DEV pk2 pk_make(float lo, float hi) {
    return (pk2)__float_as_uint(lo) | ((pk2)__float_as_uint(hi) << 32);
}

constexpr int SW_BM = 64; // rows of A per block
constexpr int SW_BK = 16; // features per slab

// One slab of both operands, feature-major.  Rows padded so that a warp's
// transposing stores hit each bank twice at most.
template <typename T> struct SweepStage;
template <> struct __align__(16) SweepStage<float> {
    static constexpr int BN = 128;
    float a[SW_BK][2 * SW_BM + 4]; // every value twice
    float b[SW_BK][BN + 4];
    B200_DEV void put_a(int k, int r, float v) {
        *reinterpret_cast<float2 *>(&a[k][2 * r]) = make_float2(v, v);
    }
};
template <> struct __align__(16) SweepStage<double> {
    static constexpr int BN = 64;
    double a[SW_BK][SW_BM + 2];
    double b[SW_BK][BN + 2];
    B200_DEV void put_a(int k, int r, double v) { a[k][r] = v; }
};

// Column (within the tile) of a thread's j-th pair: groups of 16 bytes, one
// per thread column, so that a warp's operand loads are contiguous.
template <typename T> struct SweepCols {
    static constexpr int W = 16 / (int)sizeof(T); // columns per group
    static B200_DEV int of(int j, int tn) { return (j / W) * 16 * W + tn * W + (j % W); }
};

// A thread's accumulators.  The squared euclidean sum has two (features 4t,
// 4t + 1 in the first, 4t + 2, 4t + 3 in the second), added at the borders.
template <typename T, int ACC> struct SweepAcc;
template <int ACC> struct SweepAcc<float, ACC> {
    static constexpr int TM = 4, TN = 8;
    pk2 g1[TM][TN / 2], g2[TM][TN / 2];
    B200_DEV void zero() {
#pragma unroll
        for (int i = 0; i < TM; ++i)
#pragma unroll
            for (int j = 0; j < TN / 2; ++j) g1[i][j] = g2[i][j] = 0ull;
    }
    B200_DEV void merge() {
#pragma unroll
        for (int i = 0; i < TM; ++i)
#pragma unroll
            for (int j = 0; j < TN / 2; ++j) {
                g1[i][j] = pk_add(g1[i][j], g2[i][j]);
                g2[i][j] = 0ull;
            }
    }
    // one feature's operands, and their part of the first or second sum
    struct Ops {
        pk2 a[TM], b[TN / 2];
        B200_DEV void load(const SweepStage<float> &st, int u, int tm, int tn) {
            const ulonglong2 *ap = reinterpret_cast<const ulonglong2 *>(&st.a[u][tm * 8]);
            const ulonglong2 a0 = ap[0], a1 = ap[1];
            a[0] = a0.x, a[1] = a0.y, a[2] = a1.x, a[3] = a1.y;
            const ulonglong2 b0 = *reinterpret_cast<const ulonglong2 *>(&st.b[u][tn * 4]);
            const ulonglong2 b1 = *reinterpret_cast<const ulonglong2 *>(&st.b[u][64 + tn * 4]);
            b[0] = b0.x, b[1] = b0.y, b[2] = b1.x, b[3] = b1.y;
        }
    };
    B200_DEV void add(const Ops &o, bool second, float p) {
#pragma unroll
        for (int i = 0; i < TM; ++i)
#pragma unroll
            for (int j = 0; j < TN / 2; ++j) {
                if (ACC == ACC_SQEUC) {
                    const pk2 t = pk_sub(o.a[i], o.b[j]);
                    if (second) g2[i][j] = pk_fma(t, t, g2[i][j]);
                    else g1[i][j] = pk_fma(t, t, g1[i][j]);
                } else if (ACC == ACC_DOT) {
                    g1[i][j] = pk_fma(o.a[i], o.b[j], g1[i][j]);
                } else {
                    const pk2 t = pk_sub(o.a[i], o.b[j]);
                    float x = abs_(pk_lo(t)), y = abs_(pk_hi(t));
                    if (ACC == ACC_MINKOWSKI) {
                        x = pow_(x, p);
                        y = pow_(y, p);
                    }
                    g1[i][j] = pk_make(add_rn(pk_lo(g1[i][j]), x), add_rn(pk_hi(g1[i][j]), y));
                }
            }
    }
    B200_DEV float value(int i, int j) const {
        return (j & 1) ? pk_hi(g1[i][j / 2]) : pk_lo(g1[i][j / 2]);
    }
};
template <int ACC> struct SweepAcc<double, ACC> {
    static constexpr int TM = 4, TN = 4;
    double g1[TM][TN], g2[TM][TN];
    B200_DEV void zero() {
#pragma unroll
        for (int i = 0; i < TM; ++i)
#pragma unroll
            for (int j = 0; j < TN; ++j) g1[i][j] = g2[i][j] = 0.0;
    }
    B200_DEV void merge() {
#pragma unroll
        for (int i = 0; i < TM; ++i)
#pragma unroll
            for (int j = 0; j < TN; ++j) {
                g1[i][j] = add_rn(g1[i][j], g2[i][j]);
                g2[i][j] = 0.0;
            }
    }
    struct Ops {
        double a[TM], b[TN];
        B200_DEV void load(const SweepStage<double> &st, int u, int tm, int tn) {
            const double2 *ap = reinterpret_cast<const double2 *>(&st.a[u][tm * 4]);
            const double2 a0 = ap[0], a1 = ap[1];
            a[0] = a0.x, a[1] = a0.y, a[2] = a1.x, a[3] = a1.y;
            const double2 b0 = *reinterpret_cast<const double2 *>(&st.b[u][tn * 2]);
            const double2 b1 = *reinterpret_cast<const double2 *>(&st.b[u][32 + tn * 2]);
            b[0] = b0.x, b[1] = b0.y, b[2] = b1.x, b[3] = b1.y;
        }
    };
    B200_DEV void add(const Ops &o, bool second, double p) {
#pragma unroll
        for (int i = 0; i < TM; ++i)
#pragma unroll
            for (int j = 0; j < TN; ++j) {
                if (ACC == ACC_SQEUC) {
                    const double t = sub_rn(o.a[i], o.b[j]);
                    if (second) g2[i][j] = fma_rn(t, t, g2[i][j]);
                    else g1[i][j] = fma_rn(t, t, g1[i][j]);
                } else if (ACC == ACC_DOT) {
                    g1[i][j] = fma_rn(o.a[i], o.b[j], g1[i][j]);
                } else if (ACC == ACC_MANHATTAN) {
                    g1[i][j] = add_rn(g1[i][j], abs_(sub_rn(o.a[i], o.b[j])));
                } else {
                    g1[i][j] = add_rn(g1[i][j], pow_(abs_(sub_rn(o.a[i], o.b[j])), p));
                }
            }
    }
    B200_DEV double value(int i, int j) const { return g1[i][j]; }
};

// One slab, features k0 .. k0 + 15 of d.  Every feature's operands are loaded
// while the one before is added (row u + 1 of the last feature is row 0: read,
// not used).  Four features per loop step: fully unrolled, the code of a slab
// ran out of the instruction cache.
template <typename T, int ACC>
B200_DEV void sweep_slab(const SweepStage<T> &st, int k0, int d, int kc, T p, SweepAcc<T, ACC> &acc,
                         int tm, int tn) {
    using Ops = typename SweepAcc<T, ACC>::Ops;
    const int d4 = d & ~3;
    const int n4 = ACC == ACC_MINKOWSKI ? 0 : min(SW_BK, d4 - k0); // whole groups of four
    Ops o[2];
    o[0].load(st, 0, tm, tn);
    if (ACC == ACC_SQEUC || ACC == ACC_DOT || ACC == ACC_MANHATTAN) {
#pragma unroll 1
        for (int g = 0; g < n4; g += 4) {
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                o[(u + 1) & 1].load(st, (g + u + 1) & (SW_BK - 1), tm, tn);
                acc.add(o[u & 1], ACC == ACC_SQEUC && (u & 2), p);
            }
        }
        // kc is a multiple of 16: its borders are slab borders
        if (ACC == ACC_SQEUC && n4 > 0 && (k0 + n4 == d4 || (k0 + n4) % kc == 0)) acc.merge();
    }
    // the last d % 4 features, one at a time; every feature of minkowski's
    // (a pow call per pair: one copy of the code)
    const int n = min(SW_BK, d - k0);
#pragma unroll 1
    for (int u = max(0, n4); u < n; ++u) {
        o[0].load(st, u, tm, tn);
        acc.add(o[0], false, p);
    }
}

// The matrix row that a sweep's row number stands for: itself, or (SampleRows)
// one of every `step` consecutive rows, at a place that varies, so that rows in a
// cyclic order are met in all their phases.
struct AllRows {
    B200_DEV size_t operator()(int r) const { return (size_t)r; }
};
struct SampleRows {
    int step, n;
    B200_DEV size_t operator()(int r) const {
        return (size_t)min(r * step + (int)__umulhi((unsigned)r * 0x9E3779B1u, (unsigned)step), n - 1);
    }
};

// Global loads of one slab of ROWS rows (ld elements apart, all readable; zeros
// elsewhere) into registers.
template <typename T, int ROWS> struct SweepRegs {
    static constexpr int NV = ROWS * (SW_BK / 4) / 256;
    V4<T> v[NV];
    template <typename R>
    B200_DEV void load(const T *M, int ld, R rows, int row0, int nrows, int k0, int tid) {
#pragma unroll
        for (int u = 0; u < NV; ++u) {
            const int e = tid + u * 256;
            const int gr = row0 + e / (SW_BK / 4), gk = k0 + (e % (SW_BK / 4)) * 4;
            if (gr < nrows && gk < ld) {
                v[u] = ld4_global(M + rows(gr) * ld + gk);
            } else {
                v[u].v[0] = v[u].v[1] = v[u].v[2] = v[u].v[3] = T(0);
            }
        }
    }
};

template <typename T>
B200_DEV void sweep_put(SweepStage<T> &st, const SweepRegs<T, SW_BM> &ra,
                        const SweepRegs<T, SweepStage<T>::BN> &rb, int tid) {
#pragma unroll
    for (int u = 0; u < SweepRegs<T, SW_BM>::NV; ++u) {
        const int e = tid + u * 256, r = e / (SW_BK / 4), kq = (e % (SW_BK / 4)) * 4;
#pragma unroll
        for (int w = 0; w < 4; ++w) st.put_a(kq + w, r, ra.v[u].v[w]);
    }
#pragma unroll
    for (int u = 0; u < SweepRegs<T, SweepStage<T>::BN>::NV; ++u) {
        const int e = tid + u * 256, r = e / (SW_BK / 4), kq = (e % (SW_BK / 4)) * 4;
#pragma unroll
        for (int w = 0; w < 4; ++w) st.b[kq + w][r] = rb.v[u].v[w];
    }
}

// The pair values of rows a0 .. a0 + 63 of A (na rows) with rows [b_begin,
// b_end) of B, tile by tile: epi(b0) runs with the accumulators of the tile at
// b0 complete.  One pipeline over all (tile, slab) steps: the next step's
// global loads are in flight while the current slab is consumed, across tile
// borders too.  Rows are ld elements (padded to four, pad readable).  A warp whose
// eight rows of A do not exist only loads: with few rows (300,000 x 64 against 2
// rows) the others' shared-memory reads and arithmetic are what a tile costs.  No
// barrier separates the last epi from what follows.
template <typename T, int ACC, typename R, typename F>
B200_DEV void sweep_tiles(SweepStage<T> *st, const T *A, int na, int a0, const T *B, R brows,
                          int b_begin, int b_end, int ld, int d, int kc, T p,
                          SweepAcc<T, ACC> &acc, int tid, F &&epi) {
    constexpr int BN = SweepStage<T>::BN;
    const int tm = tid / 16, tn = tid % 16;
    const int nslab = (d + SW_BK - 1) / SW_BK;
    SweepRegs<T, SW_BM> ra;
    SweepRegs<T, BN> rb;
    const bool some = a0 + (tid >> 5) * 8 < na; // of the warp's rows of A
    if (b_begin >= b_end) return;
    ra.load(A, ld, AllRows{}, a0, na, 0, tid);
    rb.load(B, ld, brows, b_begin, b_end, 0, tid);
    sweep_put(st[0], ra, rb, tid);
    __syncthreads();
    int cur = 0;
    for (int b0 = b_begin; b0 < b_end; b0 += BN) {
        acc.zero();
        for (int s = 0; s < nslab; ++s) {
            const bool last = s + 1 == nslab;
            const int nb0 = last ? b0 + BN : b0, ns = last ? 0 : s + 1;
            const bool more = nb0 < b_end;
            if (more) {
                ra.load(A, ld, AllRows{}, a0, na, ns * SW_BK, tid);
                rb.load(B, ld, brows, nb0, b_end, ns * SW_BK, tid);
            }
            if (some) sweep_slab<T, ACC>(st[cur], s * SW_BK, d, kc, p, acc, tm, tn);
            if (more) sweep_put(st[cur ^ 1], ra, rb, tid);
            if (last) epi(b0);
            __syncthreads();
            cur ^= 1;
        }
    }
}

// The post-operation over a whole micro-tile (the cases of post_value that the
// accumulation can have: fewer copies of the code), rows in turn to out(i, v).
// xv: A rows' norms, yn: B rows' norms.  rows: how many of the thread's four exist;
// a division or a power is left out for the others.
template <typename T, int ACC, typename R, typename F>
B200_DEV void sweep_post(const SweepAcc<T, ACC> &acc, int post, const T (&xv)[4], int rows,
                         const T *yn, R brows, int b0, int nb, int tn, T invp, F &&out) {
    constexpr int TN = SweepAcc<T, ACC>::TN;
    T yv[TN];
    if (ACC == ACC_DOT && post != POST_NONE && post != POST_NEG) {
#pragma unroll
        for (int j = 0; j < TN; ++j) {
            const int gb = b0 + SweepCols<T>::of(j, tn);
            yv[j] = (yn && gb < nb) ? yn[brows(gb)] : T(0);
        }
    }
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        T v[TN];
#pragma unroll
        for (int j = 0; j < TN; ++j) v[j] = acc.value(i, j);
        auto each = [&](int as) {
            if ((as == POST_COSINE || as == POST_POW) && i >= rows) return;
#pragma unroll
            for (int j = 0; j < TN; ++j) v[j] = post_value<T>(as, v[j], xv[i], yv[j], invp);
        };
        if (ACC == ACC_SQEUC) {
            if (post == POST_SQRT) each(POST_SQRT);
        } else if (ACC == ACC_DOT) {
            if (post == POST_COSINE) each(POST_COSINE);
            else if (post == POST_GEMM_SQ) each(POST_GEMM_SQ);
            else if (post == POST_GEMM_SQRT) each(POST_GEMM_SQRT);
            else if (post == POST_GEMM_SQ_CLAMP) each(POST_GEMM_SQ_CLAMP);
            else if (post == POST_NEG) each(POST_NEG);
        } else if (ACC == ACC_MINKOWSKI) {
            each(POST_POW);
        }
        out(i, v);
    }
}

} // namespace b200
