// k-means++ initialisation on the device (clustering/kmeans/kmeans.cpp:
// 1524-1664) with the reference's random draws.
//
// The reference picks every candidate centre with std::discrete_distribution
// over the current minimum squared distances w: one canonical double u in
// [0, 1) per draw, then the first index i whose cumulative probability
// cp_i >= u, where cp is the sequential double prefix sum of w_j / S and S
// the sequential double sum of w (cp of the last index set to 1).  The host
// draws the u values from the same engine in the same order; the device
// maps them to indices:
//   * kpp_draw_kernel: block sums of w (2,048 weights a block, written by
//     the kernel that last changed w), their prefix, the block holding u S
//     and the index within it -- a parallel prefix whose value P'_i / S'
//     differs from the sequential cp_i by at most
//     bound = 1.2 (2 n + 2 nb + 4200) 2^-53 (first-order rounding of the two
//     sequential sums, the divisions and the parallel sums).  The index is
//     certified when u - P'_{i-1} / S' and P'_i / S' - u both exceed the
//     bound; then the sequential search returns the same index.
//   * exact_draw: the draws that are not certified (about one per
//     k-means++ run on a million rows) are redone with the sequential sums
//     themselves, in the reference's order of operations.
// The candidates' distances are the kpp_dist kernel; their costs are the
// reference's serial sums in the working precision, reproduced exactly by
// kpp_walk_kernel (at a million fp32 rows the rounding of those sums
// decides between candidates whose costs are that close, so an fp64 sum
// would choose differently); kpp_select_update_kernel picks the candidate
// with the smallest finite cost (repeats skipped, first strictly smaller wins), writes it to
// `chosen`, lowers w to the minimum with its distances, zeroes its own
// weight and writes the block sums of the new w.  No host round trip per
// centre.
#include "b200_common.cuh"
#include <algorithm>

namespace b200 {

static constexpr int KPP_THREADS = 256;
static constexpr int KPP_PER_THREAD = 8;
static constexpr int KPP_BLOCK = KPP_THREADS * KPP_PER_THREAD;
static constexpr int KPP_TRIALS = 64; // candidates per centre, at most (2 + ln k)

__device__ __forceinline__ bool finite_(float v) { return isfinite(v); }
__device__ __forceinline__ bool finite_(double v) { return isfinite(v); }

// Block-wide exclusive prefix sum of one double per thread (fixed order);
// `total` receives the block's sum.  sh: KPP_THREADS / 32 + 1 doubles.
__device__ double block_exclusive_scan(double v, double *sh, double &total) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    double x = v;
#pragma unroll
    for (int off = 1; off < 32; off <<= 1) {
        const double y = __shfl_up_sync(0xffffffffu, x, off);
        if (lane >= off) x += y;
    }
    double ex = __shfl_up_sync(0xffffffffu, x, 1);
    if (lane == 0) ex = 0.0;
    __syncthreads();
    if (lane == 31) sh[warp] = x;
    __syncthreads();
    if (threadIdx.x == 0) {
        double a = 0.0;
        for (int w = 0; w < KPP_THREADS / 32; ++w) {
            const double t = sh[w];
            sh[w] = a;
            a += t;
        }
        sh[KPP_THREADS / 32] = a;
    }
    __syncthreads();
    total = sh[KPP_THREADS / 32];
    return sh[warp] + ex;
}

// A centre is six launches, one after another: each is issued as dependent on the
// one before (programmatic stream serialization), so that its blocks come in as
// those of that one end: 1M x 64, k = 256 32.5 -> 29.3 ms, 300,000 x 20, k = 100
// 5.9 -> 4.5, 10,000 x 16, k = 32 1.33 -> 0.92.  step_begin waits for the whole
// of the step before, its writes included; nothing that a step writes is
// touched before.  (Letting the next step in from this one's start: 33 ms, its
// waiting blocks hold the SMs.  Taking the chunks backwards on every other
// pass, to meet those still in the L2 cache: 30.9.)
__device__ __forceinline__ void step_begin() {
    asm volatile("griddepcontrol.wait;" ::: "memory");
}
template <typename... P, typename... A>
static cudaError_t step_launch(void (*kern)(P...), dim3 grid, dim3 block, size_t smem,
                               cudaStream_t s, A... a) {
    cudaLaunchAttribute at{};
    at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at.val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = grid;
    cfg.blockDim = block;
    cfg.dynamicSmemBytes = smem;
    cfg.stream = s;
    cfg.attrs = &at;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, kern, static_cast<P>(a)...);
}

// w_i = 0 where negative or not finite, and at the first centre; block sums
// of w; flag[0] = 1 when some weight is positive (kmeans.cpp:1571-1590).
template <typename T>
__global__ void __launch_bounds__(KPP_THREADS)
kpp_clamp_kernel(T *w, int n, int first, double *bs, int *flag) {
    __shared__ double sh[KPP_THREADS / 32 + 1];
    const size_t base = (size_t)blockIdx.x * KPP_BLOCK + (size_t)threadIdx.x * KPP_PER_THREAD;
    double s = 0.0;
    bool pos = false;
#pragma unroll
    for (int j = 0; j < KPP_PER_THREAD; ++j) {
        const size_t i = base + j;
        if (i < (size_t)n) {
            T v = w[i];
            if (!finite_(v) || v < T(0) || (int)i == first) v = T(0);
            w[i] = v;
            pos = pos || v > T(0);
            s += (double)v;
        }
    }
    double tot;
    block_exclusive_scan(s, sh, tot);
    if (threadIdx.x == 0) bs[blockIdx.x] = tot;
    if (__syncthreads_or(pos) && threadIdx.x == 0) atomicOr(flag, 1);
}

// ------------------------------------------------ serial cost sums ------
// The reference's candidate cost (kmeans.cpp:1624-1636) is the serial sum,
// in the working precision T and index order from 0, of m_i = max(0,
// min(w_i, d_i)).  It is reproduced exactly, not approximated.  While the
// running sum s stays inside one binade [2^E, 2^(E+1)) every addition rounds
// to the grid g = 2^(E - MANT) (s itself lies on it), so fl(s + m_i) =
// s + RN_g(m_i) and a run of additions is one integer sum of the
// independently rounded terms q_i = RN_g(m_i) (a tie, m_i / g exactly half-way,
// rounds by the running sum's last bit) -- until the sum leaves the binade.
// Three passes per candidate set:
//   * kpp_dist_csum_kernel: the candidates' distances and, per 256-row
//     chunk, the fp64 sum of its terms;
//   * kpp_chunk_q_kernel: the fp64 prefix of the chunk sums predicts the
//     binade E_j of the serial sum at each chunk; the chunk's run on that
//     binade's grid as a parity function (Pf: ties need the sum's last bit);
//   * kpp_walk_kernel, one block per candidate: adds runs of chunks whole
//     where the running sum is in their binade and stays there, and the others
//     term by term.  The prediction only chooses what is added whole; every
//     such step is checked, so the result is the reference's T value whatever
//     the fp64 prefix says.
template <typename T> struct FpTraits;
template <> struct FpTraits<float> {
    static constexpr int MANT = 23, EMIN = -126;
    static __device__ __forceinline__ int exponent(float s) {
        return (int)((__float_as_uint(s) >> 23) & 0xFF) - 127;
    }
};
template <> struct FpTraits<double> {
    static constexpr int MANT = 52, EMIN = -1022;
    static __device__ __forceinline__ int exponent(double s) {
        return (int)((__double_as_longlong(s) >> 52) & 0x7FF) - 1023;
    }
};

__host__ __device__ size_t kpp_dist_stride(int n, size_t elem);
static constexpr int CK = 256;           // terms per chunk
static constexpr int WALK_THREADS = 512;
static constexpr int WALK_PER = 4; // chunk records per thread per pass
static constexpr int NO_BINADE = -100000; // chunk record: sum it exactly
static constexpr unsigned long long SC_SAT = 1ull << 62;

__device__ __forceinline__ unsigned long long sat_add(unsigned long long a, unsigned long long b) {
    const unsigned long long r = a + b; // a, b <= 2^62: no wrap
    return r > SC_SAT ? SC_SAT : r;
}

// the reference's works5 element: std::max(0, std::min(w, d))
template <typename T> __device__ __forceinline__ T kpp_term(T wv, T dv) {
    const T mn = (dv < wv) ? dv : wv;
    return (T(0) < mn) ? mn : T(0);
}

// PER consecutive values from row i0 (a multiple of PER; 0 past the end), with
// 16-byte loads where they all exist (v starts on 16 bytes).
template <typename T, int PER>
__device__ __forceinline__ void kpp_load(const T *v, int n, int i0, T (&o)[PER]) {
    constexpr int W = 16 / (int)sizeof(T);
    struct __align__(16) V { T e[W]; };
    if (i0 + PER <= n) {
#pragma unroll
        for (int c = 0; c < PER / W; ++c) {
            const V a = reinterpret_cast<const V *>(v + i0)[c];
#pragma unroll
            for (int u = 0; u < W; ++u) o[c * W + u] = a.e[u];
        }
    } else {
#pragma unroll
        for (int u = 0; u < PER; ++u) o[u] = i0 + u < n ? v[i0 + u] : T(0);
    }
}

// The grid of the binade of s > 0: raw exponent (subnormals: EMIN - 1),
// sh = -log2(g), the binade's end in grid units, s in grid units.
template <typename T> struct Binade {
    int ex, sh;
    unsigned long long limit, s_int;
    __device__ __forceinline__ void set(T s) {
        using F = FpTraits<T>;
        ex = F::exponent(s);
        const bool sub = ex < F::EMIN;
        sh = F::MANT - (sub ? F::EMIN : ex);
        limit = sub ? (1ull << F::MANT) : (2ull << F::MANT);
        s_int = (unsigned long long)ldexp((double)s, sh);
    }
    // t = 2 m / g is exact (power-of-two scaling in double, in two factors so
    // that neither overflows).  q for a term staying inside the binade by
    // itself: RN_g(m) for a
    // non-tie; for a tie (m / g = k + 1/2) k, with *tie set (its rounding
    // depends on the running sum's parity); SC_SAT for a term that leaves
    // the binade by itself
    __device__ __forceinline__ unsigned long long qt(T m, bool &tie) const {
        const int e2 = sh + 1, ea = min(e2, 1000), eb = e2 - ea;
        const double sa = __longlong_as_double((long long)(ea + 1023) << 52);
        const double sb = __longlong_as_double((long long)(eb + 1023) << 52);
        const double tt = ((double)m * sa) * sb;
        tie = false;
        if (!(tt < 2.0 * (double)limit)) return SC_SAT;
        const unsigned long long ti = __double2ull_rz(tt);
        if ((ti & 1ull) && tt == __ull2double_rn(ti)) {
            tie = true;
            return ti >> 1;
        }
        return (ti + 1ull) >> 1;
    }
    __device__ __forceinline__ T value(unsigned long long units) const {
        return (T)ldexp((double)units, -sh);
    }
};

// A run of additions on one grid as a function of the running sum's parity
// (its last bit in grid units) at the run's start: q0 / q1 the run's total
// for start parity 0 / 1, o bit p the parity at its end for start parity p.
// A non-tie term q: (q, q, parity flips with q's last bit).  A tie term
// m / g = k + 1/2 rounds to the even neighbour: k + ((R + k) & 1) for a
// running sum R, after which the sum is even.  Runs compose associatively,
// so a scan over them gives the running sum before every term.
struct Pf {
    unsigned long long q0, q1;
    int o;
};
__device__ __forceinline__ Pf pf_id() { return Pf{0ull, 0ull, 2}; }
__device__ __forceinline__ Pf pf_term(unsigned long long q, bool tie) {
    if (!tie) {
        const int b = (int)(q & 1ull);
        return Pf{q, q, b | ((1 ^ b) << 1)};
    }
    return Pf{q + (q & 1ull), q + ((q + 1ull) & 1ull), 0};
}
__device__ __forceinline__ unsigned long long pf_q(const Pf &f, int p) { return p ? f.q1 : f.q0; }
__device__ __forceinline__ int pf_o(const Pf &f, int p) { return (f.o >> p) & 1; }
// a, then b
__device__ __forceinline__ Pf pf_cat(const Pf &a, const Pf &b) {
    const int a0 = a.o & 1, a1 = (a.o >> 1) & 1;
    return Pf{sat_add(a.q0, pf_q(b, a0)), sat_add(a.q1, pf_q(b, a1)),
              pf_o(b, a0) | (pf_o(b, a1) << 1)};
}
__device__ __forceinline__ Pf pf_shfl_up(const Pf &v, int off) {
    return Pf{__shfl_up_sync(0xffffffffu, v.q0, off), __shfl_up_sync(0xffffffffu, v.q1, off),
              __shfl_up_sync(0xffffffffu, v.o, off)};
}

// Scan of one run per thread over a block of NT threads in thread order:
// the composition of the runs before this thread's (`excl`) and of all
// (`total`).  shm: 2 * (NT / 32) + 1 entries.
template <int NT>
__device__ void block_scan_pf(const Pf &v, Pf *shm, Pf &excl, Pf &total) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    constexpr int NW = NT / 32;
    Pf x = v;
#pragma unroll
    for (int off = 1; off < 32; off <<= 1) {
        const Pf y = pf_shfl_up(x, off);
        if (lane >= off) x = pf_cat(y, x);
    }
    Pf xe = pf_shfl_up(x, 1);
    if (lane == 0) xe = pf_id();
    __syncthreads();
    if (lane == 31) shm[warp] = x;
    __syncthreads();
    if (warp == 0) {
        Pf y = lane < NW ? shm[lane] : pf_id();
#pragma unroll
        for (int off = 1; off < 32; off <<= 1) {
            const Pf z = pf_shfl_up(y, off);
            if (lane >= off) y = pf_cat(z, y);
        }
        Pf ye = pf_shfl_up(y, 1);
        if (lane == 0) ye = pf_id();
        if (lane < NW) shm[NW + lane] = ye;
        if (lane == NW - 1) shm[2 * NW] = y;
    }
    __syncthreads();
    total = shm[2 * NW];
    excl = pf_cat(shm[NW + warp], xe);
}

// The sequential sum in double, from s, of a block's tile of terms in thread
// order (8 consecutive per thread; v: this thread's, cnt in all): by one scan
// of the terms' runs on the grid of s where the sum stays in its binade, else
// by thread 0 term by term.  Every thread returns the new sum.
__device__ double exact_tile(double s, const double (&v)[KPP_PER_THREAD], int cnt, Pf *shm,
                             double *tile, double *out) {
    if (s != 0.0 && isfinite(s)) { // the same for every thread
        Binade<double> b;
        b.set(s);
        Pf loc = pf_id();
        bool sat = false;
#pragma unroll
        for (int u = 0; u < KPP_PER_THREAD; ++u) {
            bool tie;
            const unsigned long long q = b.qt(v[u], tie);
            sat = sat || q == SC_SAT;
            loc = pf_cat(loc, pf_term(q, tie));
        }
        Pf ex, tot;
        block_scan_pf<KPP_THREADS>(loc, shm, ex, tot);
        const unsigned long long R = sat_add(b.s_int, pf_q(tot, (int)(b.s_int & 1ull)));
        if (!__syncthreads_or(sat) && R < b.limit) return b.value(R);
    }
#pragma unroll
    for (int u = 0; u < KPP_PER_THREAD; ++u) tile[threadIdx.x * KPP_PER_THREAD + u] = v[u];
    __syncthreads();
    if (threadIdx.x == 0) {
        for (int j = 0; j < cnt; ++j) s = __dadd_rn(s, tile[j]);
        *out = s;
    }
    __syncthreads();
    s = *out;
    __syncthreads();
    return s;
}

// A draw with the reference's sequential arithmetic: S = sum w (double, index
// order, from 0), p_i = w_i / S, cp_i = cp_{i-1} + p_i, cp_{n-1} = 1, the first
// i with !(cp_i < u) (std::lower_bound).  Block-wide, 2,048 terms at a time;
// the terms that decide the draw are added one by one.  About one draw in a
// k-means++ run on a million rows comes here: 2 ms there, 12 ms when one
// thread added all terms.
template <typename T> __device__ __noinline__ void exact_draw(const T *w, int n, double u, int *out) {
    __shared__ double tile[KPP_BLOCK];
    __shared__ Pf shm[2 * (KPP_THREADS / 32) + 1];
    __shared__ double s_out;
    __shared__ int s_res;
    double v[KPP_PER_THREAD], S = 0.0;
    auto load = [&](int t0) {
        T x[KPP_PER_THREAD];
        kpp_load<T, KPP_PER_THREAD>(w, n, t0 + (int)threadIdx.x * KPP_PER_THREAD, x);
#pragma unroll
        for (int j = 0; j < KPP_PER_THREAD; ++j) v[j] = (double)x[j];
    };
    for (int t0 = 0; t0 < n; t0 += KPP_BLOCK) {
        load(t0);
        S = exact_tile(S, v, min(KPP_BLOCK, n - t0), shm, tile, &s_out);
    }
    if (threadIdx.x == 0) s_res = n - 1;
    double cp = 0.0;
    for (int t0 = 0; t0 < n; t0 += KPP_BLOCK) {
        load(t0);
#pragma unroll
        for (int j = 0; j < KPP_PER_THREAD; ++j) v[j] = __ddiv_rn(v[j], S);
        const double before = cp;
        cp = exact_tile(cp, v, min(KPP_BLOCK, n - t0), shm, tile, &s_out);
        // the tile in which cp reaches u (or the last index, cp = 1), or any
        // when cp is NaN: with all weights zero (S = 0) the test !(cp < u)
        // holds at once
        if (cp < u && t0 + KPP_BLOCK < n) continue;
#pragma unroll
        for (int j = 0; j < KPP_PER_THREAD; ++j) tile[threadIdx.x * KPP_PER_THREAD + j] = v[j];
        __syncthreads();
        if (threadIdx.x == 0) {
            double c = before;
            for (int j = 0; j < KPP_BLOCK && t0 + j < n; ++j) {
                c = __dadd_rn(c, tile[j]);
                if (t0 + j == n - 1) c = 1.0;
                if (!(c < u)) {
                    s_res = t0 + j;
                    break;
                }
            }
        }
        break;
    }
    __syncthreads();
    if (threadIdx.x == 0) *out = s_res;
}

// One block per draw t: the index that std::discrete_distribution gives for
// u = U[t] over the weights w, certified against the bound; a draw that is not
// certified is redone by exact_draw and counted.
template <typename T>
__global__ void __launch_bounds__(KPP_THREADS)
kpp_draw_kernel(const T *w, int n, const double *bs, int nb, const double *U, double bound,
                int force_exact, int *cand, int *exact_count) {
    __shared__ double sh[KPP_THREADS / 32 + 1];
    __shared__ double s_prev;
    __shared__ int s_block, s_idx;
    __shared__ double s_pi, s_pim1;
    const int t = blockIdx.x;
    step_begin();
    const double u = U[t];
    // S: the sum of the block sums (strided per thread, then the scan's total)
    double part = 0.0;
    for (int j = threadIdx.x; j < nb; j += KPP_THREADS) part += bs[j];
    double S;
    block_exclusive_scan(part, sh, S);
    const double target = u * S;
    // the first block whose cumulative sum reaches u S (chunked scan)
    if (threadIdx.x == 0) {
        s_block = 0x7fffffff;
        s_prev = 0.0;
    }
    __syncthreads();
    double carry = 0.0;
    for (int c0 = 0; c0 < nb; c0 += KPP_THREADS) {
        const int j = c0 + (int)threadIdx.x;
        const double v = j < nb ? bs[j] : 0.0;
        double tot;
        const double ex = carry + block_exclusive_scan(v, sh, tot);
        const double in = ex + v;
        // several blocks can qualify only within rounding of u S (then the
        // draw is not certified); the first one is taken
        if (j < nb && in >= target && ex < target) atomicMin(&s_block, j);
        carry += tot;
        __syncthreads();
        if (j == s_block) s_prev = ex;
        __syncthreads();
        if (s_block != 0x7fffffff) break;
    }
    int b = s_block;
    double prev = s_prev;
    const bool found_block = b != 0x7fffffff;
    if (!found_block) {
        b = nb - 1;
        prev = carry - bs[nb - 1];
    }
    // prefix within block b, in index order
    const size_t base = (size_t)b * KPP_BLOCK + (size_t)threadIdx.x * KPP_PER_THREAD;
    T v[KPP_PER_THREAD];
    double s = 0.0;
#pragma unroll
    for (int j = 0; j < KPP_PER_THREAD; ++j) {
        const size_t i = base + j;
        v[j] = i < (size_t)n ? w[i] : T(0);
        s += (double)v[j];
    }
    double tot;
    const double ex = block_exclusive_scan(s, sh, tot);
    if (threadIdx.x == 0) s_idx = 0x7fffffff;
    __syncthreads();
    double run = prev + ex;
    int mine = 0x7fffffff;
    double pi = 0.0, pim1 = 0.0;
#pragma unroll
    for (int j = 0; j < KPP_PER_THREAD; ++j) {
        const size_t i = base + j;
        const double before = run;
        run += (double)v[j];
        if (mine == 0x7fffffff && i < (size_t)n && run >= target) {
            mine = (int)i;
            pi = run;
            pim1 = before;
        }
    }
    if (mine != 0x7fffffff) atomicMin(&s_idx, mine);
    __syncthreads();
    if (mine != 0x7fffffff && mine == s_idx) {
        s_pi = pi;
        s_pim1 = pim1;
    }
    __syncthreads();
    __shared__ int s_certified;
    if (threadIdx.x == 0) {
        int idx = s_idx;
        bool certified = found_block && idx != 0x7fffffff && S > 0.0 && isfinite(S);
        if (idx == 0x7fffffff) idx = n - 1;
        if (certified) {
            const double hi = s_pi / S - u;
            const double lo = u - s_pim1 / S;
            certified = hi > bound && lo > bound;
        }
        cand[t] = idx;
        s_certified = certified && !force_exact;
        if (!s_certified) atomicAdd(exact_count, 1);
    }
    __syncthreads();
    if (!s_certified) exact_draw<T>(w, n, u, &cand[t]);
}

template <typename T> struct SegTraits;
template <> struct SegTraits<float> {
    static constexpr int SEG = 64; // features per register segment (kpp_dist_long_kernel)
    using V = float4;
    static constexpr int W = 4;
    static __device__ __forceinline__ void split(const float4 &v, float (&o)[4]) {
        o[0] = v.x; o[1] = v.y; o[2] = v.z; o[3] = v.w;
    }
};
template <> struct SegTraits<double> {
    static constexpr int SEG = 32;
    using V = double2;
    static constexpr int W = 2;
    static __device__ __forceinline__ void split(const double2 &v, double (&o)[2]) {
        o[0] = v.x; o[1] = v.y;
    }
};

// Distances of 256-row chunks to the candidates, with each chunk's fp64 sum of
// the cost terms per candidate.  Bound: HBM, one read of the rows (256 MB at
// 1M x 64 fp32: 39 us at the measured copy rate).  Three blocks per SM stay for
// the whole pass and take every gridDim-th chunk; the rows come in as 128-byte
// slabs (asynchronous 16-byte copies, the 16-byte parts of a row exchanged by
// the row's low bits so that eight lanes reading eight rows hit all banks), one
// slab ahead of the arithmetic, across chunks too.  A thread carries two rows'
// fma chains (features in order) for G candidates, whose values come from
// shared memory once for both.  At 1M x 64 and seven candidates: 58 us;
// one thread per row with its own strided 16-byte loads took 138 us (a warp's
// load touches 32 lines).
static constexpr int KD_THREADS = 128;
static constexpr int KD_SLAB = 128; // bytes of a row per slab
static constexpr int KD_BLOCKS = 3; // per SM

__device__ __forceinline__ void kd_copy16(void *dst, const void *src) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(
                     (unsigned)__cvta_generic_to_shared(dst)),
                 "l"(src));
}
__device__ __forceinline__ void kd_commit() { asm volatile("cp.async.commit_group;"); }
template <int N> __device__ __forceinline__ void kd_wait() {
    asm volatile("cp.async.wait_group %0;" ::"n"(N));
}

// bytes of shared memory: two slabs of a chunk's rows, the candidates' rows
template <typename T> static size_t kd_smem(int t, int ld) {
    return 2 * (size_t)CK * KD_SLAB + (size_t)t * ld * sizeof(T);
}

template <typename T, int G>
__global__ void __launch_bounds__(KD_THREADS, KD_BLOCKS)
kpp_dist_csum_kernel(const T *X, int ld, int n, const T *xnorm, const int *cand, int c0, int t,
                     const T *w, T *D, size_t nd, double *csum, int nchunks, const T *xinv,
                     int cosine) {
    using S = SegTraits<T>;
    using V = typename S::V;
    extern __shared__ __align__(16) unsigned char sm[];
    __shared__ double red[KD_THREADS / 32][G];
    unsigned char *slab = sm;                                     // [2][CK][KD_SLAB]
    T *cs = reinterpret_cast<T *>(sm + 2 * (size_t)CK * KD_SLAB); // [t][ld]
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int row_bytes = ld * (int)sizeof(T); // a multiple of 16, pad columns zero
    const int nslab = (row_bytes + KD_SLAB - 1) / KD_SLAB;
    const unsigned char *Xb = reinterpret_cast<const unsigned char *>(X);
    auto fetch = [&](int chunk, int k, int buf) {
        const int r0 = chunk * CK;
#pragma unroll
        for (int u = 0; u < CK * 8 / KD_THREADS; ++u) {
            const int e = tid + u * KD_THREADS, r = e >> 3, c = e & 7;
            const int off = k * KD_SLAB + c * 16;
            if (r0 + r < n && off < row_bytes)
                kd_copy16(slab + ((size_t)buf * CK + r) * KD_SLAB + ((c ^ (r & 7)) * 16),
                          Xb + (size_t)(r0 + r) * row_bytes + off);
        }
    };
    int chunk = blockIdx.x;
    if (chunk >= nchunks) return;
    fetch(chunk, 0, 0); // rows: no step before this one writes them
    kd_commit();
    step_begin();
    for (int e = tid; e < t * ld; e += KD_THREADS)
        cs[e] = X[(size_t)cand[c0 + e / ld] * ld + e % ld];
    int cg[G], buf = 0;
    T cn[G];
#pragma unroll
    for (int g = 0; g < G; ++g) {
        cg[g] = min(g, t - 1) * ld;
        cn[g] = xnorm[cand[c0 + min(g, t - 1)]];
    }
    for (; chunk < nchunks; chunk += gridDim.x) {
        const int r0 = chunk * CK;
        T xn[2], wi[2], s[2][G];
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const int i = r0 + tid + h * KD_THREADS;
            xn[h] = i < n ? xnorm[i] : T(0);
            wi[h] = i < n ? w[i] : T(0);
#pragma unroll
            for (int g = 0; g < G; ++g) s[h][g] = T(0);
        }
        for (int k = 0; k < nslab; ++k, buf ^= 1) {
            // the next slab, of this chunk or of the block's next one, into the
            // other buffer (whose readers passed the barrier below)
            if (k + 1 < nslab) fetch(chunk, k + 1, buf ^ 1);
            else if (chunk + (int)gridDim.x < nchunks) fetch(chunk + gridDim.x, 0, buf ^ 1);
            kd_commit();
            kd_wait<1>();
            __syncthreads();
            const unsigned char *row = slab + ((size_t)buf * CK + tid) * KD_SLAB;
            const int nv = min(8, (row_bytes - k * KD_SLAB) / 16);
            const int f0 = k * (KD_SLAB / (int)sizeof(T));
#pragma unroll 2
            for (int v = 0; v < nv; ++v) {
                const int o = (v ^ (tid & 7)) * 16; // rows tid and tid + 128: the same low bits
                T x0[S::W], x1[S::W];
                S::split(*reinterpret_cast<const V *>(row + o), x0);
                S::split(*reinterpret_cast<const V *>(row + KD_THREADS * KD_SLAB + o), x1);
#pragma unroll
                for (int g = 0; g < G; ++g) {
                    T ce[S::W];
                    S::split(*reinterpret_cast<const V *>(cs + cg[g] + f0 + v * S::W), ce);
#pragma unroll
                    for (int u = 0; u < S::W; ++u) {
                        s[0][g] = fma_rn(x0[u], ce[u], s[0][g]);
                        s[1][g] = fma_rn(x1[u], ce[u], s[1][g]);
                    }
                }
            }
            __syncthreads();
        }
        double part[G];
#pragma unroll
        for (int g = 0; g < G; ++g) {
            part[g] = 0.0;
            if (g < t) {
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    const int i = r0 + tid + h * KD_THREADS;
                    if (i >= n) continue;
                    const T dv = cosine ? cos_dist_kpp(s[h][g], xinv, i, cand[c0 + g])
                                        : fma_rn(T(-2), s[h][g], add_rn(xn[h], cn[g]));
                    D[(size_t)(c0 + g) * nd + i] = dv;
                    part[g] += (double)kpp_term(wi[h], dv);
                }
            }
        }
        // sums over the warp: lane bits 4, 3, 2 also split the candidates
        // while there are several (a quarter of the exchanges of G full sums)
#pragma unroll
        for (int off = 16, m = G; off > 0; off >>= 1) {
            if (m % 2 == 0) {
                m /= 2;
                const bool up = lane & off;
#pragma unroll
                for (int g = 0; g < G / 2; ++g)
                    if (g < m) {
                        const double give = up ? part[g] : part[g + m];
                        const double keep = up ? part[g + m] : part[g];
                        part[g] = keep + __shfl_xor_sync(0xffffffffu, give, off);
                    }
            } else {
#pragma unroll
                for (int g = 0; g < G; ++g)
                    if (g < m) part[g] += __shfl_xor_sync(0xffffffffu, part[g], off);
            }
        }
        constexpr int H = G == 8 ? 1 : G == 6 ? 3 : 1; // sums left in a lane
        constexpr int SPLIT = G / H;                   // lane groups of different ones
        if ((lane & (32 / SPLIT - 1)) == 0) {
            // the lane's top bits choose its candidates: bit 4 the upper half
            int g0 = 0, m = G;
#pragma unroll
            for (int off = 16; off >= 32 / SPLIT; off >>= 1) {
                m /= 2;
                g0 += (lane & off) ? m : 0;
            }
#pragma unroll
            for (int h = 0; h < H; ++h) red[warp][g0 + h] = part[h];
        }
        __syncthreads();
        if (tid < G && tid < t) {
            double a = 0.0;
#pragma unroll
            for (int v = 0; v < KD_THREADS / 32; ++v) a += red[v][tid];
            csum[(size_t)(c0 + tid) * nchunks + chunk] = a;
        }
        // red is rewritten after the next chunk's barriers
    }
}

// The same for rows too long for that (candidates beyond 96 KB of shared
// memory): one thread per row, the candidates' values through L1.
template <typename T>
__global__ void __launch_bounds__(CK, 2)
kpp_dist_long_kernel(const T *X, int ld, int n, int d, const T *xnorm, const int *cand, int t,
                     const T *w, T *D, size_t nd, double *csum, int nchunks, const T *xinv, int cosine) {
    using S = SegTraits<T>;
    constexpr int NV = S::SEG / S::W;
    __shared__ double red[CK / 32][8];
    const int i = blockIdx.x * CK + threadIdx.x;
    const bool valid = i < n;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const T *x = X + (size_t)(valid ? i : 0) * ld;
    step_begin();
    const T xn = valid ? xnorm[i] : T(0);
    const T wi = valid ? w[i] : T(0);
    for (int c0 = 0; c0 < t; c0 += 8) {
        T s[8];
#pragma unroll
        for (int g = 0; g < 8; ++g) s[g] = T(0);
        int cg[8];
#pragma unroll
        for (int g = 0; g < 8; ++g) cg[g] = min(c0 + g, t - 1);
        if (valid) {
            for (int f0 = 0; f0 < d; f0 += S::SEG) {
                typename S::V xv[NV];
#pragma unroll
                for (int v = 0; v < NV; ++v)
                    if (f0 + v * S::W < d) // rows are padded to 16 bytes
                        xv[v] = *reinterpret_cast<const typename S::V *>(x + f0 + v * S::W);
#pragma unroll
                for (int v = 0; v < NV; ++v) {
                    const int fb = f0 + v * S::W;
                    if (fb >= d) break;
                    T xe[S::W];
                    S::split(xv[v], xe);
#pragma unroll
                    for (int g = 0; g < 8; ++g) {
                        T ce[S::W];
                        const T *yr = X + (size_t)cand[cg[g]] * ld + fb;
                        S::split(*reinterpret_cast<const typename S::V *>(yr), ce);
#pragma unroll
                        for (int u = 0; u < S::W; ++u)
                            if (fb + u < d) s[g] = fma_rn(xe[u], ce[u], s[g]);
                    }
                }
            }
        }
        double part[8];
#pragma unroll
        for (int g = 0; g < 8; ++g) {
            part[g] = 0.0;
            if (valid && c0 + g < t) {
                const int cc = cand[c0 + g];
                const T dv = cosine ? cos_dist_kpp(s[g], xinv, i, cc)
                                    : fma_rn(T(-2), s[g], add_rn(xn, xnorm[cc]));
                D[(size_t)(c0 + g) * nd + i] = dv;
                part[g] = (double)kpp_term(wi, dv);
            }
#pragma unroll
            for (int off = 16; off > 0; off >>= 1) part[g] += __shfl_xor_sync(0xffffffffu, part[g], off);
        }
        __syncthreads();
        if (lane == 0)
#pragma unroll
            for (int g = 0; g < 8; ++g) red[warp][g] = part[g];
        __syncthreads();
        if (threadIdx.x < 8 && c0 + (int)threadIdx.x < t) {
            double a = 0.0;
            for (int v = 0; v < CK / 32; ++v) a += red[v][threadIdx.x];
            csum[(size_t)(c0 + threadIdx.x) * nchunks + blockIdx.x] = a;
        }
    }
}

// Exclusive fp64 prefix of the chunk sums of candidate blockIdx.x: one range
// of consecutive chunks per thread.
__global__ void __launch_bounds__(1024) kpp_chunk_prefix_kernel(const double *csum, int nchunks,
                                                                double *P) {
    __shared__ double shd[32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const double *cs = csum + (size_t)blockIdx.x * nchunks;
    double *Pt = P + (size_t)blockIdx.x * nchunks;
    const int per = (nchunks + 1023) / 1024;
    const int j0 = min(nchunks, (int)threadIdx.x * per), j1 = min(nchunks, j0 + per);
    step_begin();
    double mine = 0.0;
    for (int j = j0; j < j1; ++j) mine += cs[j];
    double x = mine;
#pragma unroll
    for (int off = 1; off < 32; off <<= 1) {
        const double y = __shfl_up_sync(0xffffffffu, x, off);
        if (lane >= off) x += y;
    }
    if (lane == 31) shd[warp] = x;
    __syncthreads();
    double before = lane < warp ? shd[lane] : 0.0;
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) before += __shfl_xor_sync(0xffffffffu, before, off);
    double run = before + (x - mine);
    for (int j = j0; j < j1; ++j) {
        Pt[j] = run;
        run += cs[j];
    }
}

// The terms of one warp's chunk on one binade's grid, eight consecutive terms a
// lane, in the integer width that the type's grid needs: 32 bits for fp32 (a
// binade holds 2^23 grid steps; totals saturate far above that), 64 for fp64.
// run(): a lane's terms as one parity function; warp_scan(): the runs of the
// lanes before.  SAT marks a run that leaves the binade.
template <typename T> struct Grid;
template <> struct Grid<float> {
    using U = unsigned;
    static constexpr U SAT = 1u << 30;
    U limit, s_int, base; // base: the binade's exponent bits (0: subnormal)
    float sa, sb;         // terms to half grid steps, in two exact factors
    __device__ __forceinline__ void set(float s) {
        const unsigned bits = __float_as_uint(s);
        base = bits & 0x7f800000u;
        limit = base ? 1u << 24 : 1u << 23;
        s_int = (bits & 0x7fffffu) | (base ? 0x800000u : 0u);
        const int e2 = 24 - (max((int)(base >> 23), 1) - 127), ea = min(e2, 100);
        sa = __uint_as_float((unsigned)(ea + 127) << 23);
        sb = __uint_as_float((unsigned)(e2 - ea + 127) << 23);
    }
    // the sum of `steps` grid steps, s_int <= steps < limit
    __device__ __forceinline__ float value(U steps) const {
        return __uint_as_float(base | (steps & 0x7fffffu));
    }
    // RN to the grid of a term that does not tie; k of a tie k + 1/2 (tie set)
    __device__ __forceinline__ U term(float m, bool &tie) const {
        const float t = (m * sa) * sb; // exact, or below half a step
        tie = false;
        if (!(t < 2.0f * __uint2float_rn(limit))) return SAT;
        const U ti = __float2uint_rz(t);
        tie = (ti & 1u) && t == __uint2float_rn(ti);
        return tie ? ti >> 1 : (ti + 1u) >> 1;
    }
    static __device__ __forceinline__ U add(U a, U b) { return min(a + b, SAT); }
    static __device__ __forceinline__ unsigned long long wide(U v) { return v >= SAT ? SC_SAT : v; }
};
template <> struct Grid<double> {
    using U = unsigned long long;
    static constexpr U SAT = SC_SAT;
    U limit, s_int;
    Binade<double> b;
    __device__ __forceinline__ void set(double s) {
        b.set(s);
        limit = b.limit;
        s_int = b.s_int;
    }
    __device__ __forceinline__ double value(U steps) const { return b.value(steps); }
    __device__ __forceinline__ U term(double m, bool &tie) const { return b.qt(m, tie); }
    static __device__ __forceinline__ U add(U a, U b) { return sat_add(a, b); }
    static __device__ __forceinline__ unsigned long long wide(U v) { return v; }
};
// a parity function in the grid's integer width (see Pf)
template <typename T> struct Run {
    using G = Grid<T>;
    using U = typename G::U;
    U q0, q1;
    int o;
    static __device__ __forceinline__ Run id() { return Run{0, 0, 2}; }
    __device__ __forceinline__ U q(int p) const { return p ? q1 : q0; }
    __device__ __forceinline__ int par(int p) const { return (o >> p) & 1; }
    // then one term
    __device__ __forceinline__ void add_term(U k, bool tie) {
        const int a0 = o & 1, a1 = (o >> 1) & 1, b = (int)(k & 1);
        q0 = G::add(q0, tie ? k + (U)(a0 ^ b) : k);
        q1 = G::add(q1, tie ? k + (U)(a1 ^ b) : k);
        o = tie ? 0 : (a0 ^ b) | ((a1 ^ b) << 1);
    }
    static __device__ __forceinline__ Run cat(const Run &a, const Run &b) {
        const int a0 = a.par(0), a1 = a.par(1);
        return Run{G::add(a.q0, b.q(a0)), G::add(a.q1, b.q(a1)), b.par(a0) | (b.par(a1) << 1)};
    }
    __device__ __forceinline__ Run up(int off) const {
        return Run{__shfl_up_sync(0xffffffffu, q0, off), __shfl_up_sync(0xffffffffu, q1, off),
                   __shfl_up_sync(0xffffffffu, o, off)};
    }
};

// Chunk records of candidate blockIdx.y, one warp per chunk: the binade the
// fp64 prefix predicts for the serial sum at the chunk (raw exponent of
// (T)P_j, or NO_BINADE when P_j is 0 or not finite) and the chunk's run on
// that binade's grid as a parity function (saturating totals).
template <typename T>
__global__ void __launch_bounds__(256)
kpp_chunk_q_kernel(const T *w, const T *D, size_t nd, int n, int nchunks, const double *P,
                   unsigned long long *Q0, unsigned long long *Q1, int *Or, int *Er) {
    constexpr int PER = CK / 32;
    const int j = blockIdx.x * 8 + (threadIdx.x >> 5);
    const int lane = threadIdx.x & 31;
    step_begin();
    if (j >= nchunks) return;
    const size_t r = (size_t)blockIdx.y * nchunks + j;
    const int i0 = j * CK + lane * PER;
    T wv[PER], dv[PER];
    kpp_load<T, PER>(w, n, i0, wv);
    kpp_load<T, PER>(D + (size_t)blockIdx.y * nd, n, i0, dv);
    const double Pj = P[r];
    const T Ts = (T)Pj;
    if (!(Pj > 0.0) || !isfinite(Ts) || Ts == T(0)) {
        if (lane == 0) {
            Q0[r] = Q1[r] = 0;
            Or[r] = 2;
            Er[r] = NO_BINADE;
        }
        return;
    }
    Grid<T> g;
    g.set(Ts);
    // each lane composes 8 consecutive terms, then the lanes' runs in lane
    // order (a tree over neighbouring blocks of lanes)
    Run<T> acc = Run<T>::id();
#pragma unroll
    for (int u = 0; u < PER; ++u) {
        bool tie;
        // a term past the end is 0: no change
        const typename Grid<T>::U k = g.term(kpp_term(wv[u], dv[u]), tie);
        acc.add_term(k, tie);
    }
#pragma unroll
    for (int off = 1; off < 32; off <<= 1) {
        const Run<T> y = Run<T>{__shfl_down_sync(0xffffffffu, acc.q0, off),
                                __shfl_down_sync(0xffffffffu, acc.q1, off),
                                __shfl_down_sync(0xffffffffu, acc.o, off)};
        if ((lane & (2 * off - 1)) == 0) acc = Run<T>::cat(acc, y);
    }
    if (lane == 0) {
        Q0[r] = Grid<T>::wide(acc.q0);
        Q1[r] = Grid<T>::wide(acc.q1);
        Or[r] = acc.o;
        Er[r] = FpTraits<T>::exponent(Ts);
    }
}

// The serial sum of candidate blockIdx.x over the chunk records (see above),
// in two parts.  Bound: latency, one block per candidate; the steps below are
// what it waits for.
//
// Fast part.  A chunk whose successor has the same predicted binade is inner:
// the sum is expected to stay in that binade through it.  The others -- about
// one per doubling of the sum -- are borders.  One segmented scan over all
// records gives the composition of the inner chunks before every border; the
// borders' terms are brought to shared memory together.  One thread then steps
// from border to border: the inner chunks in one addition (taken only when the
// running sum is in their binade and stays there), the border chunk's 256
// terms by 256 dependent additions (0.7 us: less than one block-wide scan to
// find where the sum leaves its binade).  At 1M rows and seven candidates:
// 30 us per centre; a block-wide scan per border and per serial step
// took 93 us.
//
// Chunks before the first positive term are left out (their fp64 sums are 0).
//
// General part: from the chunk where the fast part stopped (a check that
// failed, more borders than are kept), block-wide scans from one chunk that
// cannot be added whole to the next, that chunk's terms serially.
static constexpr int WALK_BORDERS = 32; // borders kept

struct SegRun { // runs since the last border
    Pf f;
    int cut; // a border lies in this range
};
__device__ __forceinline__ SegRun seg_cat(const SegRun &a, const SegRun &b) {
    return SegRun{b.cut ? b.f : pf_cat(a.f, b.f), a.cut | b.cut};
}

// s + m[0] + m[1] + ... + m[CK - 1], left to right in T (m in shared memory,
// 16-byte aligned; zero terms change nothing).
template <typename T> __device__ T serial_sum(T s, const T *m) {
    constexpr int W = 16 / (int)sizeof(T);
    struct __align__(16) V { T e[W]; };
    const V *v = reinterpret_cast<const V *>(m);
#pragma unroll 8
    for (int c = 0; c < CK / W; ++c) {
        const V x = v[c];
#pragma unroll
        for (int u = 0; u < W; ++u) s = add_rn(s, x.e[u]);
    }
    return s;
}

template <typename T>
__global__ void __launch_bounds__(WALK_THREADS)
kpp_walk_kernel(const T *w, const T *D, size_t nd, int n, int nchunks,
                const unsigned long long *Q0, const unsigned long long *Q1, const int *Or,
                const int *Er, const double *csum, double *cost) {
    __shared__ Pf shm[2 * (WALK_THREADS / 32) + 1];
    __shared__ int s_f;
    __shared__ T s_val;
    __shared__ int s_border[WALK_BORDERS], s_ex[WALK_BORDERS];
    __shared__ Pf s_run[WALK_BORDERS];
    __shared__ int s_cnt[WALK_THREADS / 32];
    __shared__ SegRun s_seg[WALK_THREADS / 32];
    extern __shared__ __align__(16) unsigned char walk_sm[];
    T *bt = reinterpret_cast<T *>(walk_sm); // [WALK_BORDERS][CK]: the borders' terms
    const int t = blockIdx.x;
    const T *Dt = D + (size_t)t * nd;
    const size_t ro = (size_t)t * nchunks;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    step_begin();
    int first = nchunks; // the first chunk with a positive term
    for (int c = threadIdx.x; c < nchunks; c += WALK_THREADS)
        if (!(csum[ro + c] == 0.0)) {
            first = c;
            break;
        }
    first = __reduce_min_sync(0xffffffffu, first);
    if (lane == 0) s_cnt[warp] = first;
    __syncthreads();
    first = __reduce_min_sync(0xffffffffu, s_cnt[lane & (WALK_THREADS / 32 - 1)]);
    if (first == nchunks) {
        if (threadIdx.x == 0) cost[t] = 0.0;
        return;
    }
    __syncthreads();
    // ---- fast part: borders, in order, and the inner runs before them
    int nb = 0;
    {
        // a thread's range of records, WALK_PER at a time: at(c, border, run)
        const int per = (nchunks - first + WALK_THREADS - 1) / WALK_THREADS;
        const int c0 = min(nchunks, first + (int)threadIdx.x * per), c1 = min(nchunks, c0 + per);
        auto each = [&](auto &&at) {
            for (int c = c0; c < c1; c += WALK_PER) {
                Pf f[WALK_PER];
                int ex[WALK_PER + 1];
#pragma unroll
                for (int u = 0; u < WALK_PER; ++u) {
                    const int r = min(c + u, nchunks - 1);
                    f[u] = Pf{Q0[ro + r], Q1[ro + r], Or[ro + r]};
                    ex[u] = Er[ro + r];
                }
                ex[WALK_PER] = Er[ro + min(c + WALK_PER, nchunks - 1)];
#pragma unroll
                for (int u = 0; u < WALK_PER; ++u)
                    if (c + u < c1)
                        at(c + u, c + u + 1 == nchunks || ex[u] == NO_BINADE || ex[u + 1] != ex[u],
                           f[u], ex[u]);
            }
        };
        SegRun loc{pf_id(), 0};
        int mine = 0;
        each([&](int, bool border, const Pf &f, int) {
            loc = border ? SegRun{pf_id(), 1} : SegRun{pf_cat(loc.f, f), loc.cut};
            mine += border ? 1 : 0;
        });
        SegRun inc = loc;
        int cinc = mine;
#pragma unroll
        for (int off = 1; off < 32; off <<= 1) {
            const SegRun y{pf_shfl_up(inc.f, off), __shfl_up_sync(0xffffffffu, inc.cut, off)};
            const int cy = __shfl_up_sync(0xffffffffu, cinc, off);
            if (lane >= off) {
                inc = seg_cat(y, inc);
                cinc += cy;
            }
        }
        if (lane == 31) {
            s_seg[warp] = inc;
            s_cnt[warp] = cinc;
        }
        SegRun ex{pf_shfl_up(inc.f, 1), __shfl_up_sync(0xffffffffu, inc.cut, 1)};
        if (lane == 0) ex = SegRun{pf_id(), 0};
        __syncthreads();
        SegRun before{pf_id(), 0};
        int rank = cinc - mine;
#pragma unroll
        for (int v = 0; v < WALK_THREADS / 32; ++v) {
            if (v < warp) {
                before = seg_cat(before, s_seg[v]);
                rank += s_cnt[v];
            }
            nb += s_cnt[v];
        }
        Pf run = seg_cat(before, ex).f;
        each([&](int c, bool border, const Pf &f, int e) {
            if (border) {
                if (rank < WALK_BORDERS) {
                    s_border[rank] = c;
                    s_ex[rank] = e; // the inner chunks before c are in its binade
                    s_run[rank] = run;
                }
                ++rank;
                run = pf_id();
            } else {
                run = pf_cat(run, f);
            }
        });
        nb = min(nb, WALK_BORDERS);
        __syncthreads();
        for (int e = threadIdx.x; e < nb * CK; e += WALK_THREADS) {
            const int i = s_border[e / CK] * CK + e % CK;
            bt[e] = i < n ? kpp_term(w[i], Dt[i]) : T(0);
        }
        __syncthreads();
    }
    if (threadIdx.x == 0) {
        T sum = T(0);
        int next = first; // the first chunk not yet added
        for (int b = 0; b < nb && isfinite(sum); ++b) {
            const int c = s_border[b];
            if (c > next) { // inner chunks next .. c - 1, one binade
                if (sum == T(0)) break;
                Binade<T> bn;
                bn.set(sum);
                const unsigned long long R = sat_add(bn.s_int, pf_q(s_run[b], (int)(bn.s_int & 1ull)));
                if (bn.ex != s_ex[b] || R >= bn.limit) break;
                sum = bn.value(R);
            }
            sum = serial_sum<T>(sum, bt + (size_t)b * CK);
            next = c + 1;
        }
        s_val = sum;
        s_f = next;
    }
    __syncthreads();
    // ---- general part
    T s = s_val;
    int j = s_f;
    __syncthreads();
    while (j < nchunks && isfinite(s)) {
        Binade<T> b;
        b.ex = NO_BINADE - 1;
        b.sh = 0;
        b.limit = 0;
        b.s_int = 0;
        if (s != T(0)) b.set(s);
        const int p0 = (int)(b.s_int & 1ull);
        // WALK_PER consecutive records per thread
        const int r0 = j + (int)threadIdx.x * WALK_PER;
        Pf rv[WALK_PER];
        bool okv[WALK_PER];
        Pf loc = pf_id();
#pragma unroll
        for (int u = 0; u < WALK_PER; ++u) {
            const int r = r0 + u;
            const bool valid = r < nchunks;
            rv[u] = valid ? Pf{Q0[ro + r], Q1[ro + r], Or[ro + r]} : pf_id();
            okv[u] = !valid || Er[ro + r] == b.ex;
            loc = pf_cat(loc, rv[u]);
        }
        Pf excl, total;
        block_scan_pf<WALK_THREADS>(loc, shm, excl, total);
        int mine = 0x7fffffff;
        unsigned long long R = b.s_int + pf_q(excl, p0), R_at = 0; // running sum, grid units
        int par = pf_o(excl, p0);
#pragma unroll
        for (int u = 0; u < WALK_PER; ++u) {
            const unsigned long long q = pf_q(rv[u], par);
            if (mine == 0x7fffffff && r0 + u < nchunks && (!okv[u] || R + q >= b.limit)) {
                mine = (int)threadIdx.x * WALK_PER + u;
                R_at = R;
            }
            R = sat_add(R, q);
            par = pf_o(rv[u], par);
        }
        if (threadIdx.x == 0) s_f = 0x7fffffff;
        __syncthreads();
        if (mine != 0x7fffffff) atomicMin(&s_f, mine);
        __syncthreads();
        const int f = s_f;
        if (f == 0x7fffffff) {
            s = b.value(b.s_int + pf_q(total, p0));
            j += WALK_THREADS * WALK_PER;
            continue;
        }
        // the records before f on the grid, then chunk j + f term by term
        if (mine == f) s_val = (f == 0) ? s : b.value(R_at);
        const int c = j + f;
        for (int e = threadIdx.x; e < CK; e += WALK_THREADS) {
            const int i = c * CK + e;
            bt[e] = i < n ? kpp_term(w[i], Dt[i]) : T(0);
        }
        __syncthreads();
        if (threadIdx.x == 0) s_val = serial_sum<T>(s_val, bt);
        __syncthreads();
        s = s_val;
        __syncthreads();
        j = c + 1;
    }
    if (threadIdx.x == 0) cost[t] = (double)s;
}

int kpp_num_chunks(int n) { return (n + CK - 1) / CK; }

template <typename T>
cudaError_t launch_kpp_dist_cost(const T *X, int ldx, int n, int d, const T *xnorm,
                                 const int *cand, int t, const T *w, T *D, double *cost,
                                 void *work, cudaStream_t s, const T *xinv, int cosine) {
    if (ldx % 4 != 0 || (reinterpret_cast<uintptr_t>(X) & 15) != 0) return cudaErrorInvalidValue;
    const int nch = kpp_num_chunks(n);
    double *csum = static_cast<double *>(work);
    double *P = csum + (size_t)t * nch;
    unsigned long long *Q0 = reinterpret_cast<unsigned long long *>(P + (size_t)t * nch);
    unsigned long long *Q1 = Q0 + (size_t)t * nch;
    int *Or = reinterpret_cast<int *>(Q1 + (size_t)t * nch);
    int *Er = Or + (size_t)t * nch;
    const size_t nd = kpp_dist_stride(n, sizeof(T));
    const size_t cand_bytes = (size_t)t * ldx * sizeof(T);
    if (cand_bytes <= 96 * 1024) {
        const int grid = std::min(nch, 148 * KD_BLOCKS);
        for (int c0 = 0; c0 < t; c0 += 8) {
            const int m = std::min(8, t - c0);
            auto kern = m <= 4   ? kpp_dist_csum_kernel<T, 4>
                        : m <= 6 ? kpp_dist_csum_kernel<T, 6>
                                 : kpp_dist_csum_kernel<T, 8>;
            const size_t smem = kd_smem<T>(m, ldx);
            cudaError_t e = ensure_smem_limit(reinterpret_cast<const void *>(kern), smem);
            if (e != cudaSuccess) return e;
            e = step_launch(kern, dim3(grid), dim3(KD_THREADS), smem, s, X, ldx, n, xnorm, cand, c0,
                            m, w, D, nd, csum, nch, xinv, cosine);
            if (e != cudaSuccess) return e;
        }
    } else {
        const cudaError_t e = step_launch(kpp_dist_long_kernel<T>, dim3(nch), dim3(CK), 0, s, X, ldx,
                                          n, d, xnorm, cand, t, w, D, nd, csum, nch, xinv, cosine);
        if (e != cudaSuccess) return e;
    }
    cudaError_t e = step_launch(kpp_chunk_prefix_kernel, dim3(t), dim3(1024), 0, s, csum, nch, P);
    if (e != cudaSuccess) return e;
    e = step_launch(kpp_chunk_q_kernel<T>, dim3((nch + 7) / 8, t), dim3(256), 0, s, w, D, nd, n, nch,
                    P, Q0, Q1, Or, Er);
    if (e != cudaSuccess) return e;
    const size_t wsm = (size_t)WALK_BORDERS * CK * sizeof(T);
    e = ensure_smem_limit(reinterpret_cast<const void *>(kpp_walk_kernel<T>), wsm);
    if (e != cudaSuccess) return e;
    return step_launch(kpp_walk_kernel<T>, dim3(t), dim3(WALK_THREADS), wsm, s, w, D, nd, n, nch, Q0,
                       Q1, Or, Er, csum, cost);
}

// Elements from one candidate's distances to the next: rows start on 16 bytes.
__host__ __device__ size_t kpp_dist_stride(int n, size_t elem) {
    const size_t w = 16 / elem;
    return ((size_t)n + w - 1) / w * w;
}

size_t kpp_cost_work_bytes(int n, int t) {
    return (size_t)kpp_num_chunks(n) * t * (8 + 8 + 8 + 8 + 4 + 4) + 256;
}

// Choose the candidate (kmeans.cpp:1614-1646): repeats skipped, the first
// finite cost strictly below the best so far; none: index 0.  Every block
// makes the same choice; block 0 records it.  Then w_i = max(0, min(w_i,
// D_best,i)), the chosen row's weight 0, and the block sums of the new w.
template <typename T>
__global__ void __launch_bounds__(KPP_THREADS)
kpp_select_update_kernel(T *w, const T *D, int n, const double *cost, const int *cand, int nt,
                         int *chosen, int c, double *bs) {
    __shared__ double sh[KPP_THREADS / 32 + 1];
    __shared__ int s_best_t, s_best;
    __shared__ double s_cost[KPP_TRIALS];
    __shared__ int s_cand[KPP_TRIALS];
    step_begin();
    if ((int)threadIdx.x < nt) {
        s_cost[threadIdx.x] = cost[threadIdx.x];
        s_cand[threadIdx.x] = cand[threadIdx.x];
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        int bt = -1, best = 0;
        double bc = __longlong_as_double(0x7ff0000000000000ULL);
        for (int t = 0; t < nt; ++t) {
            bool rep = false;
            for (int q = 0; q < t; ++q) rep = rep || s_cand[q] == s_cand[t];
            if (rep) continue;
            const double ct = s_cost[t];
            if (isfinite(ct) && ct < bc) {
                bc = ct;
                bt = t;
                best = s_cand[t];
            }
        }
        s_best_t = bt;
        s_best = best;
        if (blockIdx.x == 0) chosen[c] = best;
    }
    __syncthreads();
    const int bt = s_best_t, best = s_best;
    const T *Dc = bt >= 0 ? D + (size_t)bt * kpp_dist_stride(n, sizeof(T)) : nullptr;
    const size_t base = (size_t)blockIdx.x * KPP_BLOCK + (size_t)threadIdx.x * KPP_PER_THREAD;
    double s = 0.0;
    if (Dc && base + KPP_PER_THREAD <= (size_t)n) { // 16-byte loads and stores
        constexpr int W = 16 / (int)sizeof(T);
        struct __align__(16) V { T e[W]; };
        T m[KPP_PER_THREAD], dv[KPP_PER_THREAD];
        kpp_load<T, KPP_PER_THREAD>(w, n, (int)base, m);
        kpp_load<T, KPP_PER_THREAD>(Dc, n, (int)base, dv);
#pragma unroll
        for (int j = 0; j < KPP_PER_THREAD; ++j) {
            m[j] = (int)base + j == best ? T(0) : kpp_term(m[j], dv[j]);
            s += (double)m[j];
        }
#pragma unroll
        for (int v = 0; v < KPP_PER_THREAD / W; ++v) {
            V o;
#pragma unroll
            for (int u = 0; u < W; ++u) o.e[u] = m[v * W + u];
            reinterpret_cast<V *>(w + base)[v] = o;
        }
    } else
#pragma unroll
    for (int j = 0; j < KPP_PER_THREAD; ++j) {
        const size_t i = base + j;
        if (i < (size_t)n) {
            T v = w[i];
            if (Dc) {
                const T dv = Dc[i];
                T m = dv < v ? dv : v;
                if (!(m > T(0))) m = T(0);
                v = m;
            }
            if ((int)i == best) v = T(0);
            w[i] = v;
            s += (double)v;
        }
    }
    double tot;
    block_exclusive_scan(s, sh, tot);
    if (threadIdx.x == 0) bs[blockIdx.x] = tot;
}

int kpp_num_blocks(int n) { return (n + KPP_BLOCK - 1) / KPP_BLOCK; }

double kpp_draw_bound(int n) {
    const double nb = (double)kpp_num_blocks(n);
    return 1.2 * (2.0 * n + 2.0 * nb + 4200.0) * 0x1p-53;
}

template <typename T>
cudaError_t launch_kpp_clamp(T *w, int n, int first, double *bs, int *flag, cudaStream_t s) {
    kpp_clamp_kernel<T><<<kpp_num_blocks(n), KPP_THREADS, 0, s>>>(w, n, first, bs, flag);
    return cudaGetLastError();
}

template <typename T>
cudaError_t launch_kpp_draw(const T *w, int n, const double *bs, const double *U, int nt,
                            int force_exact, int *cand, int *exact_count,
                            cudaStream_t s) {
    const int nb = kpp_num_blocks(n);
    return step_launch(kpp_draw_kernel<T>, dim3(nt), dim3(KPP_THREADS), 0, s, w, n, bs, nb, U,
                       kpp_draw_bound(n), force_exact, cand, exact_count);
}

template <typename T>
cudaError_t launch_kpp_select_update(T *w, const T *D, int n, const double *cost,
                                     const int *cand, int nt, int *chosen, int c, double *bs,
                                     cudaStream_t s) {
    if (nt > KPP_TRIALS) return cudaErrorInvalidValue;
    return step_launch(kpp_select_update_kernel<T>, dim3(kpp_num_blocks(n)), dim3(KPP_THREADS), 0, s,
                       w, D, n, cost, cand, nt, chosen, c, bs);
}

#define B200_KPP_INST(T)                                                                       \
    template cudaError_t launch_kpp_clamp<T>(T *, int, int, double *, int *, cudaStream_t);     \
    template cudaError_t launch_kpp_draw<T>(const T *, int, const double *, const double *,     \
                                            int, int, int *, int *, cudaStream_t);              \
    template cudaError_t launch_kpp_select_update<T>(T *, const T *, int, const double *,       \
                                                     const int *, int, int *, int, double *,    \
                                                     cudaStream_t);                             \
    template cudaError_t launch_kpp_dist_cost<T>(const T *, int, int, int, const T *,           \
                                                 const int *, int, const T *, T *, double *,     \
                                                 void *, cudaStream_t, const T *, int);
B200_KPP_INST(float)
B200_KPP_INST(double)

} // namespace b200
