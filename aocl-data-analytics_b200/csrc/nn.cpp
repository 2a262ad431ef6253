// Brute-force k-nearest-neighbours handle (host side).  Argument checks,
// option semantics and status codes follow
// source/core/nearest_neighbors/nearest_neighbors.cpp; the distance tile and
// the top-k selection run on the GPU (dist_simt.cu).
#include "alg.hpp"
#include <cstdlib>
#include <map>

namespace b200 {

// metric ids of the "metric" option (aoclda_metrics.h:44-59)
enum { M_EUC = 0, M_SQEUC = 1, M_MINK = 2, M_MANH = 3, M_COS = 4, M_EUC_GEMM = 5,
       M_SQEUC_GEMM = 6, M_IP = 7 };
// algorithm ids (nearest_neighbors_types.hpp:29)
enum { A_BRUTE = 0, A_KD = 1, A_BALL = 2, A_AUTO = 3 };
// "outlier handling" ids (nearest_neighbors_types.hpp)
enum { OH_NONE = 0, OH_MANUAL = 1, OH_MOST_FREQUENT = 2 };

template <typename T>
NN<T>::NN(ErrorRecord *e, CudaCtx *c, bool single) {
    err = e;
    cuda = c;
    opts.single = single;
    register_common_options(opts);
    // nearest_neighbors_options.hpp:52-124
    const da_int imax = std::numeric_limits<da_int>::max();
    const da_int imin = std::numeric_limits<da_int>::min();
    const double fmax = (double)std::numeric_limits<T>::max();
    const double flow = (double)std::numeric_limits<T>::lowest();
    opts.add_int("number of neighbors", 1, LB::greaterequal, imax, UB::p_inf, 5);
    opts.add_int("leaf size", 1, LB::greaterequal, imax, UB::p_inf, 30);
    opts.add_int("outlier label", imin, LB::m_inf, imax, UB::p_inf, 0);
    opts.add_real("minkowski parameter", 0.0, LB::greaterthan, fmax, UB::p_inf, 2.0);
    opts.add_real("radius", 0.0, LB::greaterequal, fmax, UB::p_inf, 1.0);
    opts.add_real("outlier target", flow, LB::m_inf, fmax, UB::p_inf, 0.0);
    opts.add_string("algorithm",
                    {{"auto", A_AUTO}, {"brute", A_BRUTE}, {"kd tree", A_KD}, {"ball tree", A_BALL}},
                    "auto");
    opts.add_string("metric",
                    {{"euclidean", M_EUC},
                     {"l2", M_EUC},
                     {"sqeuclidean", M_SQEUC},
                     {"manhattan", M_MANH},
                     {"l1", M_MANH},
                     {"cityblock", M_MANH},
                     {"cosine", M_COS},
                     {"minkowski", M_MINK},
                     {"sqeuclidean_gemm", M_SQEUC_GEMM},
                     {"euclidean_gemm", M_EUC_GEMM},
                     {"inner product", M_IP}},
                    "euclidean");
    opts.add_string("weights", {{"uniform", 0}, {"distance", 1}}, "uniform");
    opts.add_string("outlier handling",
                    {{"none", OH_NONE}, {"manual", OH_MANUAL}, {"most frequent", OH_MOST_FREQUENT}},
                    "none");
    // B200 options (no counterpart in the reference):
    //   "reference isa": which AOCL-DA build's KC blocking the squared-euclidean
    //   summation order reproduces (avx512: KC=256/512, avx2: KC=64/32).
    opts.add_string("reference isa", {{"avx512", 0}, {"avx2", 1}}, "avx512");
    //   "precision mode": "bf16x3" lets large fp32 euclidean searches run a
    //   tensor-core candidate pass with an exact re-score (same neighbours and
    //   distances as "plain", the SIMT fp32 path).
    opts.add_string("precision mode", {{"plain", 0}, {"bf16x3", 3}}, "bf16x3");
}

template <typename T> da_status NN<T>::set_params() {
    n_neighbors = opts.i("number of neighbors");
    algo = opts.key("algorithm");
    metric = opts.key("metric");
    weights = opts.key("weights");
    p = (T)opts.r("minkowski parameter");
    // Tree algorithms reject non-metric distances (nearest_neighbors.cpp:313-330).
    if (algo == A_KD || algo == A_BALL) {
        if (metric == M_COS || metric == M_SQEUC || metric == M_SQEUC_GEMM || metric == M_IP)
            return err->error(da_status_incompatible_options,
                              "The tree algorithms are not compatible with the cosine, squared "
                              "Euclidean, or inner product distances.");
        if (metric == M_MINK && p < T(1))
            return err->error(da_status_incompatible_options,
                              "Tree algorithms are not compatible with the Minkowski metric when "
                              "0 < p < 1.");
    }
    up_to_date = true;
    return da_status_success;
}

// nearest_neighbors.cpp:398-466: after set_data the tree-related options are
// locked.  As in the reference, "number of neighbors", "metric", "weights" and
// "minkowski parameter" are read when the training data are set
// (set_params, nearest_neighbors.cpp:497-499) and not re-read afterwards.
template <typename T> da_status NN<T>::check_options_update() {
    const da_int a = opts.key("algorithm");
    if (a == A_AUTO || a == A_KD || a == A_BALL) {
        if (a != locked_algo || opts.i("leaf size") != locked_leaf)
            return err->error(da_status_option_locked,
                              "Options need to be set before calling set_training_data().");
        if (a == A_AUTO &&
            (opts.key("metric") != locked_metric || (T)opts.r("minkowski parameter") != locked_p))
            return err->error(da_status_option_locked,
                              "Options need to be set before calling set_training_data().");
    }
    return da_status_success;
}

template <typename T>
da_status NN<T>::set_data(da_int n, da_int d, const T *X, da_int ldx) {
    if (n_samples > 0 && n != n_samples)
        return err->error(da_status_invalid_array_dimension,
                          "n_samples = " + std::to_string(n) +
                              " doesn't match the training data size " +
                              std::to_string(n_samples) + ".");
    const da_order ord = order();
    da_status s = check_2d(*err, ord, n, d, X, ldx, "n_samples", "n_features", "X_train",
                           "ldx_train", 1, 1, opts.key("check data") == 1);
    if (s != da_status_success) return s;
    n_samples = n;
    n_features = d;
    X_host = X;
    ldx_host = ldx;
    data_order = ord;
    have_X = true;
    X_on_device = false;
    xn_kind = -1;
    s = set_params();
    if (s != da_status_success) return s;
    locked_algo = algo;
    locked_leaf = opts.i("leaf size");
    locked_metric = metric;
    locked_p = p;
    // Upload now when a device is present (the reference keeps the user's
    // pointer; an eager device copy is a safe superset of that contract).
    if (cuda->init(*err) == da_status_success) {
        s = ensure_device_data();
        if (s != da_status_success) return s;
    } else {
        err->clear();
    }
    return da_status_success;
}

// The training data of `src` (same precision and storage order, same device):
// this handle takes its host pointers (rows, labels, targets) as set_data /
// set_labels / set_targets would, and holds the same device copies of the
// rows -- fp32/fp64 rows, and the tensor-core bf16 pair and norms when src
// has built them -- instead of uploading its own.  Neither handle writes into
// a shared copy: a later set_data on either gives that handle new buffers.
template <typename T> da_status NN<T>::share_data(NN<T> &src) {
    if (!src.have_X)
        return err->error(da_status_no_data, "The source handle holds no training data.");
    if (src.order() != order())
        return err->error(da_status_invalid_input,
                          "The two handles have different storage orders.");
    if (n_samples > 0 && src.n_samples != n_samples)
        return err->error(da_status_invalid_array_dimension,
                          "n_samples = " + std::to_string(src.n_samples) +
                              " doesn't match the training data size " +
                              std::to_string(n_samples) + ".");
    da_status s = cuda->init(*err);
    if (s != da_status_success) return s;
    if (src.cuda->init(*src.err) != da_status_success || src.ensure_device_data() != da_status_success)
        return err->error(da_status_memory_error,
                          "The source handle's training data are not on the device: " +
                              src.err->message);
    if (src.cuda->device != cuda->device)
        return err->error(da_status_invalid_input, "The two handles use different devices.");
    // the source's uploads are complete before this handle's stream reads them
    B200_TRY(cudaStreamSynchronize(src.cuda->stream), "synchronisation with the source handle");
    n_samples = src.n_samples;
    n_features = src.n_features;
    X_host = src.X_host;
    if (!src.X_own.empty()) { // a loaded source owns its rows: keep a copy
        X_own = src.X_own;
        X_host = X_own.data();
    }
    ldx_host = src.ldx_host;
    data_order = src.data_order;
    have_X = true;
    s = set_params();
    if (s != da_status_success) return s;
    locked_algo = algo;
    locked_leaf = opts.i("leaf size");
    locked_metric = metric;
    locked_p = p;
    ld = src.ld;
    dX.share(src.dX);
    X_on_device = true;
    xn_kind = -1;
    tc_train_ready = false;
    if (src.tc_train_ready) {
        // max |x| is the first scalar of the tensor-core state; the rest of
        // that buffer is per call
        if (!dTkScal.ensure(64))
            return err->error(da_status_memory_error, "Device memory allocation failed.");
        B200_TRY(cudaMemcpyAsync(dTkScal.p, src.dTkScal.p, 16, cudaMemcpyDeviceToDevice,
                                 cuda->stream),
                 "copy");
        dXh.share(src.dXh);
        dXl.share(src.dXl);
        dXsq.share(src.dXsq);
        tc_ldbf = src.tc_ldbf;
        tc_train_ready = true;
    }
    if (src.have_labels) {
        const da_int *y = src.y_class;
        if (!src.y_own.empty()) {
            y_own = src.y_own;
            y = y_own.data();
        }
        s = set_labels(src.n_samples, y);
        if (s != da_status_success) return s;
    }
    if (src.have_targets) {
        const T *y = src.y_reg;
        if (!src.t_own.empty()) {
            t_own = src.t_own;
            y = t_own.data();
        }
        s = set_targets(src.n_samples, y);
        if (s != da_status_success) return s;
    }
    return da_status_success;
}

// Model persistence: the training rows in their storage order (dense), then
// the labels and targets when set.  Loading replays set_data / set_labels /
// set_targets on the handle's own copies (the options were loaded first).
template <typename T> da_status NN<T>::save_state(ByteWriter &w) {
    if (!have_X)
        return err->error(da_status_no_data,
                          "No training data have been set. Please call da_nn_set_data_s or "
                          "da_nn_set_data_d before saving the model.");
    const bool rm = data_order == row_major;
    std::vector<T> X((size_t)n_samples * n_features);
    for (da_int i = 0; i < n_samples; ++i)
        for (da_int j = 0; j < n_features; ++j)
            X[rm ? (size_t)i * n_features + j : i + (size_t)j * n_samples] =
                X_host[rm ? (size_t)i * ldx_host + j : i + (size_t)j * ldx_host];
    w.put<int64_t>(n_samples);
    w.put<int64_t>(n_features);
    w.put<int32_t>((int32_t)data_order);
    w.put_vec(X.data(), X.size());
    w.put<int32_t>(have_labels ? 1 : 0);
    if (have_labels) w.put_vec(y_class, (size_t)n_samples);
    w.put<int32_t>(have_targets ? 1 : 0);
    if (have_targets) w.put_vec(y_reg, (size_t)n_samples);
    return da_status_success;
}

template <typename T> da_status NN<T>::load_state(ByteReader &r) {
    const int64_t n = r.get<int64_t>(), d = r.get<int64_t>();
    const int32_t ord = r.get<int32_t>();
    X_own = r.get_vec<T>();
    if (!r.ok || n < 1 || d < 1 || X_own.size() != (size_t)(n * d) || ord != (int32_t)order())
        return err->error(da_status_invalid_file_data, "The model file is corrupted.");
    da_status s = set_data((da_int)n, (da_int)d, X_own.data(),
                           ord == row_major ? (da_int)d : (da_int)n);
    if (s != da_status_success) return s;
    if (r.get<int32_t>()) {
        y_own = r.get_vec<da_int>();
        if (!r.ok || y_own.size() != (size_t)n)
            return err->error(da_status_invalid_file_data, "The model file is corrupted.");
        s = set_labels((da_int)n, y_own.data());
        if (s != da_status_success) return s;
    }
    if (r.get<int32_t>()) {
        t_own = r.get_vec<T>();
        if (!r.ok || t_own.size() != (size_t)n)
            return err->error(da_status_invalid_file_data, "The model file is corrupted.");
        s = set_targets((da_int)n, t_own.data());
        if (s != da_status_success) return s;
    }
    if (!r.ok) return err->error(da_status_invalid_file_data, "The model file is corrupted.");
    return da_status_success;
}

template <typename T> da_status NN<T>::ensure_device_data() {
    da_status s = cuda->init(*err);
    if (s != da_status_success) return s;
    if (X_on_device) return da_status_success;
    ld = pad4(n_features);
    if (!dX.ensure((size_t)n_samples * ld * sizeof(T)))
        return err->error(da_status_memory_error, "Device memory allocation failed.");
    B200_TRY(upload_matrix<T>(data_order, n_samples, n_features, X_host, ldx_host, dX.as<T>(),
                              ld, dStage, cuda->stream),
             "upload of X_train");
    B200_TRY(cuda->leave_in_flight(), "upload of X_train");
    radius_accepted();
    X_on_device = true;
    xn_kind = -1;
    tc_train_ready = false;
    return da_status_success;
}

// The training rows' tensor-core copies: bf16 rows of d rounded up to 8 (at
// least 64): no padded K block is stored or read (the tensor maps zero-fill past
// the row).  cudaErrorMemoryAllocation: nothing was built.
template <typename T> cudaError_t NN<T>::tc_train_copies(da_int d) {
    if constexpr (std::is_same_v<T, float>) {
        const int ldbf = d <= 64 ? 64 : (int)((d + 7) / 8 * 8);
        if (tc_train_ready && tc_ldbf == ldbf) return cudaSuccess;
        const size_t xb = (size_t)n_samples * ldbf * 2;
        tc_train_ready = false;
        tc_ldbf = ldbf;
        if (!dXh.ensure(xb) || !dXl.ensure(xb) || !dXsq.ensure((size_t)n_samples * 4) ||
            !dTkScal.ensure(64))
            return cudaErrorMemoryAllocation;
        const cudaError_t e = launch_knn_tc_train_prep(
            dX.as<float>(), ld, (int)n_samples, (int)d, dXh.p, dXl.p, ldbf, dXsq.as<float>(),
            dTkScal.as<float>(), cuda->stream);
        tc_train_ready = e == cudaSuccess;
        return e;
    } else {
        return cudaErrorNotSupported;
    }
}

// The tensor-core buffers given back: there is no room for all of them, and the
// plain path needs none.
template <typename T> void NN<T>::drop_tc() {
    tc_train_ready = false;
    for (DevBuf *b : {&dXh, &dXl, &dXsq, &dXinv, &dTkQ, &dTkList, &dTkFlag}) b->release();
}

// Tensor-core candidate pass + exact re-score (knn_tc.cu) into dOutK (indices
// after the distances; `done` false where there is no room for its buffers), in
// query batches that bound the candidate lists' memory; n_extra ints of
// state follow the indices, for tc_finish.
static constexpr da_int KNN_TC_BATCH = 16384;
template <typename T>
da_status NN<T>::kneighbors_tc(da_int nq, da_int d, da_int k, const KnnWay &w, size_t &n_extra,
                                bool &done) {
    done = false;
    if constexpr (std::is_same_v<T, float>) {
        cudaStream_t st = cuda->stream;
        const bool cosine = w.post == POST_COSINE;
        if (cosine) {
            // the plain path's norms of the training rows and queries, and the
            // reciprocals of the former
            if (!dQn.ensure((size_t)nq * sizeof(T)) || !dXn.ensure((size_t)n_samples * sizeof(T)) ||
                !dXinv.ensure((size_t)n_samples * sizeof(float))) {
                drop_tc();
                return da_status_success;
            }
            B200_TRY(launch_row_norms_eps1<float>(dQ.as<float>(), ld, (int)nq, (int)d,
                                                  dQn.as<float>(), st), "norms");
            if (xn_kind != 1)
                B200_TRY(launch_row_norms_eps1<float>(dX.as<float>(), ld, (int)n_samples, (int)d,
                                                      dXn.as<float>(), st), "norms");
            xn_kind = 1;
            B200_TRY(launch_recip(dXn.as<float>(), (int)n_samples, dXinv.as<float>(), st),
                     "norms");
        }
        const cudaError_t te = tc_train_copies(d);
        if (te == cudaErrorMemoryAllocation) {
            drop_tc();
            return da_status_success;
        }
        B200_TRY(te, "tensor-core training copies");
        const int ldbf = tc_ldbf;
        // batches of queries; their state words and list lengths follow the
        // indices and come back with them (tc_finish)
        const da_int qb = std::min<da_int>(nq, KNN_TC_BATCH);
        const int batches = (int)((nq + KNN_TC_BATCH - 1) / KNN_TC_BATCH);
        const KnnTcPlan pl = knn_tc_plan((int)n_samples, (int)qb, (int)k);
        n_extra = (size_t)batches * KNN_TC_STATE + (size_t)nq;
        if (!dTkQ.ensure(knn_tc_query_bytes((int)qb, ldbf, pl)) ||
            !dTkList.ensure((size_t)qb * pl.cap * 8) || !dTkFlag.ensure((size_t)nq * sizeof(int)) ||
            !dOutK.ensure(out_bytes((size_t)nq * k, n_extra))) {
            drop_tc();
            return da_status_success;
        }
        int *state = out_idx((size_t)nq * k) + (size_t)nq * k;
        int *counts = state + (size_t)batches * KNN_TC_STATE;
        for (da_int q0 = 0; q0 < nq; q0 += KNN_TC_BATCH, state += KNN_TC_STATE) {
            const da_int nb = std::min<da_int>(KNN_TC_BATCH, nq - q0);
            const KnnTcCosine cs{dXn.as<float>(), dXinv.as<float>(),
                                 cosine ? dQn.as<float>() + q0 : nullptr};
            // a last batch that fits one M tile has its own sizes
            const KnnTcPlan pb = nb == qb ? pl : knn_tc_plan((int)n_samples, (int)nb, (int)k);
            if (!dTkQ.ensure(knn_tc_query_bytes((int)nb, ldbf, pb)) ||
                !dTkList.ensure((size_t)nb * pb.cap * 8)) {
                drop_tc();
                return da_status_success;
            }
            B200_TRY(cuda->timed("knn_tc", [&] {
                return launch_knn_tc(dX.as<float>(), dXh.p, dXl.p, dXsq.as<float>(),
                                     dTkScal.as<float>(), (int)n_samples, ld, tc_ldbf, (int)d,
                                     dQ.as<float>() + (size_t)q0 * ld, (int)nb, (int)k, w.kc,
                                     w.tf, pb, dTkQ.p, dTkList.p,
                                     dTkFlag.as<int>() + q0, counts + q0, state,
                                     dOutK.as<float>() + (size_t)q0 * k,
                                     out_idx((size_t)nq * k) + (size_t)q0 * k, st,
                                     cosine ? &cs : nullptr);
            }), "kNN tensor-core pass");
        }
        cuda->stats["tensor_core"] = 1.0;
        done = true;
    } else {
        (void)nq, (void)d, (void)k, (void)w, (void)n_extra;
    }
    return da_status_success;
}

template <typename T> da_status NN<T>::tc_check(const int *state) {
    if (state[1] == 0) return da_status_success;
    return err->error(da_status_internal_error,
                      "The tensor-core kNN kernel timed out waiting on a pipeline barrier (code " +
                          std::to_string(state[1]) + ").");
}

static constexpr int KNN_ROUNDS = 3; // list passes with closer bounds, at most

// The state words and list lengths of a tensor-core search (`extra`, as
// kneighbors_tc laid them out): statistics, errors, and the flagged queries
// searched again into dOutK (`redone`).
template <typename T>
da_status NN<T>::tc_finish(da_int nq, da_int d, da_int k, const KnnWay &w, const int *extra,
                           bool &redone) {
    redone = false;
    if constexpr (std::is_same_v<T, float>) {
        const int batches = (int)((nq + KNN_TC_BATCH - 1) / KNN_TC_BATCH);
        const int *lens = extra + (size_t)batches * KNN_TC_STATE;
        double mx = 0, sum = 0;
        int flagged = 0;
        for (int b = 0; b < batches; ++b) {
            const int *h = extra + (size_t)b * KNN_TC_STATE;
            const da_status s = tc_check(h);
            if (s != da_status_success) return s;
            flagged += h[0];
            cuda->stats["knn_tc_fallback_list_overflow"] += (double)h[2];
            cuda->stats["knn_tc_fallback_few_survivors"] += (double)h[4];
        }
        for (da_int i = 0; i < nq; ++i) {
            mx = std::max(mx, (double)lens[i]);
            sum += lens[i];
        }
        cuda->stats["knn_tc_max_list"] = std::max(cuda->stats["knn_tc_max_list"], mx);
        cuda->stats["knn_tc_mean_list"] = sum / std::max<double>(1.0, (double)nq);
        if (flagged == 0) return da_status_success;
        // the queries the pass could not certify: again with closer bounds while
        // that helps, the plain path on the rest
        redone = true;
        Redo r;
        da_status s = flagged_queries(dTkFlag.as<int>(), (size_t)nq, nullptr, r);
        cuda->stats["knn_tc_again_queries"] = (double)r.again.size();
        for (int round = 0; s == da_status_success && round < KNN_ROUNDS && !r.again.empty();
             ++round) {
            std::vector<int> idx;
            idx.swap(r.again);
            s = knn_tc_some(nq, d, k, w, idx, r);
        }
        if (s != da_status_success) return s;
        std::vector<int> fresh;
        fresh.swap(r.over);
        fresh.insert(fresh.end(), r.again.begin(), r.again.end());
        r.again.clear();
        cuda->stats["knn_tc_fallback_queries"] = (double)fresh.size();
        return knn_redo(nq, d, k, w, fresh, r);
    } else {
        (void)nq, (void)d, (void)k, (void)w, (void)extra;
    }
    return da_status_success;
}

// The queries whose word is set, by their numbers (null: their places).
template <typename T>
da_status NN<T>::flagged_queries(const int *words, size_t nq, const int *number, Redo &r) {
    std::vector<int> h(nq);
    B200_TRY(cudaMemcpyAsync(h.data(), words, nq * sizeof(int), cudaMemcpyDeviceToHost,
                             cuda->stream), "copy");
    B200_TRY(cudaStreamSynchronize(cuda->stream), "copy");
    for (size_t i = 0; i < nq; ++i)
        if (h[i]) (h[i] == 2 ? r.again : r.over).push_back(number ? number[i] : (int)i);
    return da_status_success;
}

// Queries idx[0 .. m) brought together, with room for their results, in the
// upload's stage (free by the time a search has run).
template <typename T>
cudaError_t NN<T>::gather_queries(const int *idx, size_t m, da_int k, const KnnWay &w, Gathered &g) {
    cudaStream_t st = cuda->stream;
    const size_t mk = m * k;
    if (!dStage.ensure((m * ld + m + mk) * sizeof(T) + (mk + 3 * m + KNN_TC_STATE) * sizeof(int)))
        return cudaErrorMemoryAllocation;
    g.Q = dStage.as<T>();
    g.qn = g.Q + m * ld;
    g.key = g.qn + m;
    g.ind = reinterpret_cast<int *>(g.key + mk);
    g.number = g.ind + mk;
    g.redo = g.number + m;
    g.state = g.redo + m;
    cudaError_t e =
        cudaMemcpyAsync(g.number, idx, m * sizeof(int), cudaMemcpyHostToDevice, st);
    if (e == cudaSuccess)
        e = launch_rows_gather(dQ.p, ld * sizeof(T), g.number, (int)m, g.Q, st);
    if (!w.qn) g.qn = nullptr;
    else if (e == cudaSuccess) e = launch_rows_gather(w.qn, sizeof(T), g.number, (int)m, g.qn, st);
    return e;
}
template <typename T>
da_status NN<T>::scatter_results(da_int nq, da_int k, size_t m, const Gathered &g) {
    cudaStream_t st = cuda->stream;
    B200_TRY(launch_rows_scatter(g.key, k * sizeof(T), g.number, (int)m, dOutK.p, st), "scatter");
    B200_TRY(launch_rows_scatter(g.ind, k * sizeof(int), g.number, (int)m, out_idx((size_t)nq * k),
                                 st), "scatter");
    return da_status_success;
}

// Queries per batch of the selection passes: 256 MB of lists.
template <typename T> size_t NN<T>::sel_batch(const KnnSelPlan &pl) const {
    const size_t per = knn_sel_bytes(pl, 1, sizeof(T) == 8);
    return std::max<size_t>(64, ((size_t)1 << 28) / per / 64 * 64);
}

// Some queries by the selection passes, into dOutK, from their own bounds or
// (given) from those at their first output keys.
template <typename T>
da_status NN<T>::knn_select_some(da_int nq, da_int d, da_int k, const KnnWay &w,
                                 const std::vector<int> &idx, bool given, Redo &r) {
    cudaStream_t st = cuda->stream;
    const bool fp64 = sizeof(T) == 8;
    KnnSelPlan pl{};
    if (!knn_sel_plan((int)n_samples, (int)std::min<size_t>(idx.size(), 65536), (int)k, fp64, pl)) {
        r.over.insert(r.over.end(), idx.begin(), idx.end());
        return da_status_success;
    }
    const KnnArgs a{w.acc, w.post, w.kc, (double)p, (int)k, 0, 0};
    const size_t qb = std::min(idx.size(), sel_batch(pl));
    for (size_t i0 = 0; i0 < idx.size(); i0 += qb) {
        const size_t m = std::min(qb, idx.size() - i0);
        Gathered g;
        const bool room = dPartK.ensure(knn_sel_bytes(pl, (int)m, fp64));
        const cudaError_t e = room ? gather_queries(idx.data() + i0, m, k, w, g)
                                   : cudaErrorMemoryAllocation;
        if (e == cudaErrorMemoryAllocation) {
            r.over.insert(r.over.end(), idx.begin() + i0, idx.end());
            return da_status_success;
        }
        B200_TRY(e, "gather");
        if (given)
            B200_TRY(launch_rows_gather(dOutK.p, k * sizeof(T), g.number, (int)m, g.key, st), "gather");
        B200_TRY(cuda->timed("knn_select", [&] {
            return launch_knn_select<T>(g.Q, (int)m, dX.as<T>(), (int)n_samples, ld, (int)d, g.qn,
                                        w.xn, a, pl, dPartK.p, w.tf, g.key, g.ind, g.state, g.redo,
                                        given ? g.key : nullptr, st);
        }), "kNN selection kernels");
        da_status s = scatter_results(nq, k, m, g);
        if (s == da_status_success) s = flagged_queries(g.redo, m, idx.data() + i0, r);
        if (s != da_status_success) return s;
    }
    return da_status_success;
}

// Some queries by the tensor-core list pass, into dOutK, from the bounds at their
// first output keys.
template <typename T>
da_status NN<T>::knn_tc_some(da_int nq, da_int d, da_int k, const KnnWay &w,
                             const std::vector<int> &idx, Redo &r) {
    if constexpr (std::is_same_v<T, float>) {
        cudaStream_t st = cuda->stream;
        const bool cosine = w.post == POST_COSINE;
        for (size_t i0 = 0; i0 < idx.size(); i0 += KNN_TC_BATCH) {
            const size_t m = std::min<size_t>(KNN_TC_BATCH, idx.size() - i0);
            const KnnTcPlan pl = knn_tc_plan((int)n_samples, (int)m, (int)k);
            Gathered g;
            const bool room = dTkQ.ensure(knn_tc_query_bytes((int)m, tc_ldbf, pl)) &&
                              dTkList.ensure(m * pl.cap * 8);
            const cudaError_t e = room ? gather_queries(idx.data() + i0, m, k, w, g)
                                       : cudaErrorMemoryAllocation;
            if (e == cudaErrorMemoryAllocation) {
                r.over.insert(r.over.end(), idx.begin() + i0, idx.end());
                return da_status_success;
            }
            B200_TRY(e, "gather");
            B200_TRY(launch_rows_gather(dOutK.p, k * sizeof(T), g.number, (int)m, g.key, st), "gather");
            const KnnTcCosine cs{dXn.as<float>(), dXinv.as<float>(), g.qn};
            B200_TRY(cuda->timed("knn_tc", [&] {
                return launch_knn_tc(dX.as<float>(), dXh.p, dXl.p, dXsq.as<float>(),
                                     dTkScal.as<float>(), (int)n_samples, ld, tc_ldbf, (int)d, g.Q,
                                     (int)m, (int)k, w.kc, w.tf, pl, dTkQ.p, dTkList.p, g.redo,
                                     g.state + KNN_TC_STATE, g.state, g.key, g.ind, st,
                                     cosine ? &cs : nullptr, g.key);
            }), "kNN tensor-core pass");
            int state[KNN_TC_STATE];
            B200_TRY(cudaMemcpyAsync(state, g.state, sizeof(state), cudaMemcpyDeviceToHost, st), "copy");
            da_status s = scatter_results(nq, k, m, g);
            if (s == da_status_success) s = flagged_queries(g.redo, m, idx.data() + i0, r);
            if (s == da_status_success) s = tc_check(state);
            if (s != da_status_success) return s;
        }
    } else {
        (void)nq, (void)d, (void)k, (void)w, (void)idx, (void)r;
    }
    return da_status_success;
}

// What a first pass left: `fresh` by the selection passes, again with closer
// bounds while that helps, the rest by running lists.
template <typename T>
da_status NN<T>::knn_redo(da_int nq, da_int d, da_int k, const KnnWay &w, std::vector<int> &fresh,
                          Redo &r) {
    da_status s = da_status_success;
    if (!fresh.empty()) s = knn_select_some(nq, d, k, w, fresh, false, r);
    for (int round = 0; s == da_status_success && round < KNN_ROUNDS && !r.again.empty(); ++round) {
        std::vector<int> idx;
        idx.swap(r.again);
        s = knn_select_some(nq, d, k, w, idx, true, r);
    }
    r.over.insert(r.over.end(), r.again.begin(), r.again.end());
    return s == da_status_success ? knn_lists(nq, d, k, w, &r.over) : s;
}

// Running lists and their merge into dOutK, for all queries or those of `only`
// (all, where there is no room to bring these together).
template <typename T>
da_status NN<T>::knn_lists(da_int nq, da_int d, da_int k, const KnnWay &w,
                           const std::vector<int> *only) {
    cudaStream_t st = cuda->stream;
    const bool fp64 = sizeof(T) == 8;
    const size_t m = only ? only->size() : (size_t)nq;
    if (m == 0) return da_status_success;
    cuda->stats["knn_select_fallback"] = (double)m;
    Gathered g{dQ.as<T>(), const_cast<T *>(w.qn), dOutK.as<T>(), out_idx((size_t)nq * k), nullptr,
               nullptr, nullptr};
    if (m == (size_t)nq) only = nullptr;
    if (only) {
        const cudaError_t e = gather_queries(only->data(), m, k, w, g);
        if (e == cudaErrorMemoryAllocation) return knn_lists(nq, d, k, w, nullptr);
        B200_TRY(e, "gather");
    }
    // chunking of the training rows: enough CTAs to fill 148 SMs several times
    const int BN = knn_tile_rows_train(fp64);
    const int q_tiles = (int)((m + 63) / 64);
    const int max_chunks = std::max(1, (int)((n_samples + BN - 1) / BN));
    // enough CTAs to fill the GPU; but one warp merges a query's lists, in a time
    // that grows with the square of their number (391 lists of 5: 8.3 ms, the rows
    // of as many chunks: 10 us a tile), so for few queries the sum of both is
    // least near the cube root below
    const double merge = (double)k * std::log2(k + 1.0);
    const int balance = std::max(8, (int)std::cbrt(10.0 * (double)n_samples / merge));
    int n_chunks = std::max(1, std::min({max_chunks, (148 * 8 + q_tiles - 1) / q_tiles, balance}));
    int chunk_rows = (int)((n_samples + n_chunks - 1) / n_chunks);
    chunk_rows = ((chunk_rows + BN - 1) / BN) * BN;
    n_chunks = (int)((n_samples + chunk_rows - 1) / chunk_rows);
    const KnnArgs a{w.acc, w.post, w.kc, (double)p, (int)k, chunk_rows, n_chunks};
    const size_t parts = m * k * n_chunks;
    if (!dPartK.ensure(parts * sizeof(T)) || !dPartI.ensure(parts * sizeof(int)))
        return err->error(da_status_memory_error, "Device memory allocation failed.");
    B200_TRY(cuda->timed("knn_chunks", [&] {
        return launch_knn_chunks<T>(g.Q, ld, (int)m, dX.as<T>(), ld, (int)n_samples, (int)d, g.qn,
                                    w.xn, a, dPartK.as<T>(), dPartI.as<int>(), nullptr, st);
    }), "kNN distance kernel");
    B200_TRY(cuda->timed("knn_merge", [&] {
        return launch_knn_merge<T>(dPartK.as<T>(), dPartI.as<int>(), (int)m, n_chunks, (int)k, w.tf,
                                   g.key, g.ind, st);
    }), "kNN merge kernel");
    return only ? scatter_results(nq, k, m, g) : da_status_success;
}

template <typename T> da_status NN<T>::set_labels(da_int n, const da_int *y) {
    if (n_samples > 0 && n != n_samples)
        return err->error(da_status_invalid_array_dimension,
                          "n_samples = " + std::to_string(n) +
                              " doesn't match the training data size " +
                              std::to_string(n_samples) + ".");
    if (n < 1)
        return err->error(da_status_invalid_array_dimension,
                          "The function was called with n_samples = " + std::to_string(n) +
                              ". Constraint: n_samples >= 1.");
    if (y == nullptr) return err->error(da_status_invalid_pointer, "The array y_train_class is null.");
    n_samples = n;
    y_class = y;
    have_labels = true;
    classes_done = false;
    return da_status_success;
}

template <typename T> da_status NN<T>::set_targets(da_int n, const T *y) {
    if (n_samples > 0 && n != n_samples)
        return err->error(da_status_invalid_array_dimension,
                          "n_samples = " + std::to_string(n) +
                              " doesn't match the training data size " +
                              std::to_string(n_samples) + ".");
    if (n < 1)
        return err->error(da_status_invalid_array_dimension,
                          "The function was called with n_samples = " + std::to_string(n) +
                              ". Constraint: n_samples >= 1.");
    if (y == nullptr) return err->error(da_status_invalid_pointer, "The array y_train_reg is null.");
    n_samples = n;
    y_reg = y;
    have_targets = true;
    return da_status_success;
}

template <typename T>
da_status NN<T>::validate_queries(da_int nq, da_int d, const T *Xt, da_int ldt) {
    if (Xt == nullptr) return err->error(da_status_invalid_pointer, "X_test is not a valid pointer.");
    if (d != n_features)
        return err->error(da_status_invalid_array_dimension,
                          "n_features = " + std::to_string(d) +
                              " doesn't match the expected value " +
                              std::to_string(n_features) + ".");
    return check_2d(*err, order(), nq, d, Xt, ldt, "n_queries", "n_features", "X_test",
                    "ldx_test", 1, 1, opts.key("check data") == 1);
}

// Run the fused distance + top-k kernels; ind/dist are q-major (q*k + r), or
// the results go to the caller's arrays in the storage order `ord` (to).
template <typename T>
da_status NN<T>::kneighbors_compute(da_int nq, da_int d, const T *Xt, da_int ldt, da_order ord,
                                    da_int k, std::vector<da_int> &ind, std::vector<T> *dist,
                                    const KnnOut *to) {
    da_status s = ensure_device_data();
    if (s != da_status_success) return s;
    cudaStream_t st = cuda->stream;
    // metric -> accumulation family, selection key and output transform
    int acc = ACC_SQEUC, post = POST_NONE, tf = 0, norm_kind = -1;
    switch (metric) {
    case M_EUC: acc = ACC_SQEUC; post = POST_NONE; tf = 1; break;
    case M_SQEUC: acc = ACC_SQEUC; post = POST_NONE; break;
    case M_EUC_GEMM: acc = ACC_DOT; post = POST_GEMM_SQ_CLAMP; tf = 1; norm_kind = 0; break;
    case M_SQEUC_GEMM: acc = ACC_DOT; post = POST_GEMM_SQ_CLAMP; norm_kind = 0; break;
    case M_MANH: acc = ACC_MANHATTAN; break;
    case M_COS: acc = ACC_DOT; post = POST_COSINE; norm_kind = 1; break;
    case M_IP: acc = ACC_DOT; post = POST_NEG; tf = 2; break;
    case M_MINK:
        if (p == T(2)) { acc = ACC_SQEUC; tf = 1; }
        else if (p == T(1)) { acc = ACC_MANHATTAN; }
        else { acc = ACC_MINKOWSKI; post = POST_POW; }
        break;
    }
    const bool fp64 = sizeof(T) == 8;
    const int kc = opts.key("reference isa") == 1 ? (fp64 ? 32 : 64) : (fp64 ? 512 : 256);
    // queries -> device
    if (!dQ.ensure((size_t)nq * ld * sizeof(T)))
        return err->error(da_status_memory_error, "Device memory allocation failed.");
    B200_TRY(upload_matrix<T>(ord, nq, d, Xt, ldt, dQ.as<T>(), ld, dStage, st), "upload of X_test");
    cuda->stats["tensor_core"] = 0.0;
    cuda->stats["knn_select_fallback"] = 0.0;
    cuda->stats["knn_select_again"] = 0.0;
    cuda->stats["knn_tc_again_queries"] = 0.0;
    cuda->stats["knn_tc_fallback_queries"] = 0.0;
    cuda->stats["knn_tc_fallback_list_overflow"] = 0.0;
    cuda->stats["knn_tc_fallback_few_survivors"] = 0.0;
    KnnWay way{acc, post, tf, kc, nullptr, nullptr};
    bool tc_done = false;
    size_t n_extra = 0; // ints after the indices: tc_finish's, or the flags below
    const bool tc_metric = metric == M_EUC || metric == M_SQEUC || metric == M_COS ||
                           (metric == M_MINK && p == T(2));
    // The tensor-core pass from about 5e8 multiply-adds on (a batch counts at
    // least 64 queries, one tile of either path): there it takes 100 us where
    // the plain path takes 155 (65,536 x 32, 256 queries, k = 10; 75 against
    // 194 at 200,000 x 64, one query; 215 against 294 at 16,384 x 32, 2,048
    // queries).  Below, its five launches are no shorter and its bf16 copies
    // and lists are more to set up.
    if (!fp64 && tc_metric && opts.key("precision mode") != 0 &&
        knn_tc_supported((int)n_samples, (int)d, (int)k) && n_samples >= 16384 &&
        (double)n_samples * (double)std::max<da_int>(nq, 64) * (double)d >= 5.0e8) {
        s = kneighbors_tc(nq, d, k, way, n_extra, tc_done);
        if (s != da_status_success) return s;
        if (!tc_done) n_extra = 0;
        if (tc_done && metric == M_COS) {
            way.qn = dQn.as<T>();
            way.xn = dXn.as<T>();
        }
    }
    // the plain path: bounds first (launch_knn_select) in query batches of at
    // most 256 MB of lists, each with its own flag after the indices, then a flag
    // per query; running lists (knn_lists) where that does not apply.  Queries whose
    // flag comes back set are searched again (the others' results stay)
    KnnSelPlan sel{};
    da_int sel_qb = 0;
    if (!tc_done) {
        if (knn_sel_plan((int)n_samples, (int)std::min<da_int>(nq, 65536), (int)k, fp64, sel)) {
            sel_qb = std::min(nq, (da_int)sel_batch(sel));
            // a handle's first search: lists within 1 MB, in a few batches, come out
            // of a block that the driver has, where more cost 0.35 ms to allocate
            const size_t per = knn_sel_bytes(sel, 1, fp64);
            const da_int few = (da_int)((1u << 20) / per / 64 * 64);
            if (!dPartK.p && few > 0 && few < nq && (nq + few - 1) / few <= 4) sel_qb = few;
            n_extra = (size_t)((nq + sel_qb - 1) / sel_qb);
        }
        if (norm_kind >= 0) {
            if (!dQn.ensure((size_t)nq * sizeof(T)) || !dXn.ensure((size_t)n_samples * sizeof(T)))
                return err->error(da_status_memory_error, "Device memory allocation failed.");
            if (norm_kind == 0) {
                B200_TRY(launch_row_sqnorms<T>(dQ.as<T>(), ld, nq, d, dQn.as<T>(), st), "norms");
                if (xn_kind != 0)
                    B200_TRY(launch_row_sqnorms<T>(dX.as<T>(), ld, n_samples, d, dXn.as<T>(), st), "norms");
            } else {
                B200_TRY(launch_row_norms_eps1<T>(dQ.as<T>(), ld, nq, d, dQn.as<T>(), st), "norms");
                if (xn_kind != 1)
                    B200_TRY(launch_row_norms_eps1<T>(dX.as<T>(), ld, n_samples, d, dXn.as<T>(), st), "norms");
            }
            xn_kind = norm_kind;
            way.qn = dQn.as<T>();
            way.xn = dXn.as<T>();
        }
        if (k > knn_max_k(fp64))
            return err->error(da_status_not_implemented,
                              "k = " + std::to_string(k) + " exceeds the largest supported number "
                              "of neighbours per query (" + std::to_string(knn_max_k(fp64)) + ").");
        // (no room for its lists: the running lists, which take less)
        if (n_extra > 0 && !dPartK.ensure(knn_sel_bytes(sel, (int)sel_qb, fp64))) n_extra = 0;
        if (!dOutK.ensure(out_bytes((size_t)nq * k, n_extra > 0 ? n_extra + nq : 0)))
            return err->error(da_status_memory_error, "Device memory allocation failed.");
        if (n_extra > 0) {
            const KnnArgs a{acc, post, kc, (double)p, (int)k, 0, 0};
            int *flags = out_idx((size_t)nq * k) + (size_t)nq * k, *redo = flags + n_extra;
            for (da_int q0 = 0; q0 < nq; q0 += sel_qb, ++flags) {
                const da_int nb = std::min(sel_qb, nq - q0);
                B200_TRY(cuda->timed("knn_select", [&] {
                    return launch_knn_select<T>(
                        dQ.as<T>() + (size_t)q0 * ld, (int)nb, dX.as<T>(), (int)n_samples, ld, (int)d,
                        way.qn ? way.qn + q0 : nullptr, way.xn, a, sel, dPartK.p, tf,
                        dOutK.as<T>() + (size_t)q0 * k, out_idx((size_t)nq * k) + (size_t)q0 * k,
                        flags, redo + q0, nullptr, st);
                }), "kNN selection kernels");
            }
        } else {
            s = knn_lists(nq, d, k, way, nullptr);
            if (s != da_status_success) return s;
        }
    }
    // the indices follow the distances, the state words the indices.  A few
    // results come back in one copy; many go to the caller's arrays directly,
    // column-major ones transposed on the device first (the upload's stage is
    // free by now)
    const size_t nk = (size_t)nq * k;
    const bool want = to ? to->dist != nullptr : dist != nullptr;
    const bool cm = to && ord == column_major && nq > 1 && k > 1;
    bool small = out_bytes(nk, n_extra) <= 256 * 1024;
    std::vector<int> extra, tmp;
    if (!to) {
        ind.resize(nk);
        if (dist) dist->resize(nk);
    }
    T *const hd = to ? to->dist : dist ? dist->data() : nullptr;
    da_int *const hi = to ? to->ind : ind.data();
    for (;;) {
        const T *od = dOutK.as<T>();
        const int *oi = out_idx(nk);
        extra.resize(n_extra);
        if (!small && cm) small = !dStage.ensure(nk * (sizeof(T) + sizeof(int))); // no room there
        if (small) {
            // in words of four bytes: the distances if wanted, indices, state
            const size_t dw = want ? nk * sizeof(T) / 4 : 0, words = dw + nk + n_extra;
            tmp.resize(words);
            B200_TRY(copy_down({tmp.data(), words * 4, want ? (void *)od : (void *)oi, words * 4,
                                words * 4, 1}, st), "kNN");
            const int *ti = tmp.data() + dw;
            const T *td = reinterpret_cast<const T *>(tmp.data());
            for (size_t q = 0, e = 0; q < (size_t)nq; ++q)
                for (size_t r = 0; r < (size_t)k; ++r, ++e) {
                    const size_t at = cm ? r * nq + q : e;
                    hi[at] = (da_int)ti[e];
                    if (want) std::memcpy(&hd[at], &td[e], sizeof(T));
                }
            std::copy(ti + nk, ti + nk + n_extra, extra.begin());
        } else {
            if (cm) {
                T *td = dStage.as<T>();
                float *ti = reinterpret_cast<float *>(td + nk); // four-byte words
                B200_TRY(launch_rowmajor_to_colmajor<float>(reinterpret_cast<const float *>(oi),
                                                            (int)nq, (int)k, (int)k, ti, (long)nq,
                                                            st), "transpose");
                if (want)
                    B200_TRY(launch_rowmajor_to_colmajor<T>(od, (int)nq, (int)k, (int)k, td,
                                                            (long)nq, st), "transpose");
                oi = reinterpret_cast<const int *>(ti);
                od = td;
            }
            if (n_extra)
                B200_TRY(cudaMemcpyAsync(extra.data(), out_idx(nk) + nk, n_extra * sizeof(int),
                                         cudaMemcpyDeviceToHost, st), "download");
            if (want)
                B200_TRY(copy_down({hd, nk * sizeof(T), const_cast<T *>(od), nk * sizeof(T),
                                    nk * sizeof(T), 1}, st), "download");
            B200_TRY(download_ints(oi, nk, hi, st), "kNN");
        }
        if (n_extra == 0) break;
        if (tc_done) {
            bool redone = false;
            s = tc_finish(nq, d, k, way, extra.data(), redone);
            if (s != da_status_success) return s;
            if (!redone) break;
        } else {
            if (std::all_of(extra.begin(), extra.end(), [](int f) { return f == 0; })) break;
            Redo r; // the queries whose list overflowed
            std::vector<int> fresh;
            s = flagged_queries(out_idx(nk) + nk + n_extra, (size_t)nq, nullptr, r);
            if (s != da_status_success) return s;
            cuda->stats["knn_select_again"] = (double)r.again.size();
            s = knn_redo(nq, d, k, way, fresh, r);
            if (s != da_status_success) return s;
        }
        n_extra = 0;
    }
    return da_status_success;
}

// The queries Q (nq rows on the device) on the tensor cores: the rows that may
// be within thr, then their exact distances (knn_tc.cu).  Not taken where a
// buffer is not to be had, where a query has no finite threshold, and from one
// pair in eight on, where re-scoring them one by one costs what the plain
// path's block does.
template <typename T>
da_status NN<T>::radius_tc(da_int nq, da_int d, const T *Q, T thr, int kc, bool want_val,
                           da_int *cnt_out, long long *start_out, std::vector<da_int> &idx_out,
                           std::vector<T> &val_out, bool &done) {
    done = false;
    if constexpr (std::is_same_v<T, float>) {
        cudaStream_t st = cuda->stream;
        const cudaError_t te = tc_train_copies(d);
        if (te == cudaErrorMemoryAllocation) {
            drop_tc();
            return da_status_success;
        }
        B200_TRY(te, "tensor-core training copies");
        const int n = (int)n_samples, words = radius_tc_words(n);
        // state words, their number of candidates; offsets; per query counts
        // of candidates and hits
        struct Head {
            int state[KNN_TC_STATE];
            long long total;
        } head;
        const size_t off_at = 64, hit_at = off_at + (size_t)nq * 8, cnt_at = hit_at + (size_t)nq * 4;
        if (!dTkQ.ensure(radius_tc_query_bytes((int)nq, tc_ldbf)) ||
            !dD.ensure((size_t)nq * words * 4) || !dRs.ensure(cnt_at + (size_t)nq * 4)) {
            drop_tc();
            return da_status_success;
        }
        char *w = dRs.as<char>();
        int *state = reinterpret_cast<int *>(w), *hits = reinterpret_cast<int *>(w + hit_at),
            *cnt = reinterpret_cast<int *>(w + cnt_at);
        long long *off = reinterpret_cast<long long *>(w + off_at);
        B200_TRY(cuda->timed("radius_distances", [&] {
            return launch_radius_tc(dXh.p, dXl.p, dXsq.as<float>(), dTkScal.as<float>(), n, ld,
                                    tc_ldbf, (int)d, Q, (int)nq, thr, dTkQ.p, dD.as<unsigned>(),
                                    cnt, state, st);
        }), "radius search's tensor-core pass");
        B200_TRY(cuda->timed("radius_count", [&] {
            return launch_radius_cand_scan(cnt, (int)nq, off,
                                           reinterpret_cast<long long *>(w + sizeof(head.state)), st);
        }), "count");
        B200_TRY(cudaMemcpyAsync(&head, w, sizeof(head), cudaMemcpyDeviceToHost, st), "copy");
        B200_TRY(cudaStreamSynchronize(st), "radius search");
        if (head.state[1] != 0)
            return err->error(da_status_internal_error,
                              "The radius search's tensor-core kernel timed out waiting on a "
                              "pipeline barrier (code " + std::to_string(head.state[1]) + ").");
        const size_t tot = (size_t)head.total;
        if (tot > (size_t)nq * n / 8) return da_status_success;
        if (!dRi.ensure(std::max<size_t>(tot, 1) * sizeof(int)) ||
            !dRv.ensure(std::max<size_t>(tot, 1) * sizeof(T)))
            return da_status_success;
        B200_TRY(cuda->timed("radius_emit", [&] {
            return launch_radius_exact(dX.as<float>(), n, ld, (int)d, Q, (int)nq, kc, thr,
                                       dD.as<unsigned>(), cnt, off, hits, dRi.as<int>(),
                                       dRv.as<float>(), st);
        }), "compaction");
        std::vector<char> meta(cnt_at - off_at);
        B200_TRY(cudaMemcpyAsync(meta.data(), off, meta.size(), cudaMemcpyDeviceToHost, st), "copy");
        size_t at = idx_out.size();
        const size_t from = at;
        idx_out.resize(at + tot);
        if (want_val) val_out.resize(at + tot);
        if (tot > 0) {
            B200_TRY(download_ints(dRi.as<int>(), tot, idx_out.data() + at, st), "copy");
            if (want_val)
                B200_TRY(copy_down({val_out.data() + at, tot * sizeof(T), dRv.p, tot * sizeof(T),
                                    tot * sizeof(T), 1}, st), "copy");
        }
        B200_TRY(cudaStreamSynchronize(st), "radius search");
        // a query's hits are its first candidates: move them together
        const long long *ho = reinterpret_cast<const long long *>(meta.data());
        const int *hh = reinterpret_cast<const int *>(meta.data() + (hit_at - off_at));
        for (da_int i = 0; i < nq; ++i) {
            start_out[i] = (long long)at;
            cnt_out[i] = (da_int)hh[i];
            const size_t o = from + (size_t)ho[i];
            if (o != at) {
                std::copy(idx_out.begin() + o, idx_out.begin() + o + hh[i], idx_out.begin() + at);
                if (want_val)
                    std::copy(val_out.begin() + o, val_out.begin() + o + hh[i],
                              val_out.begin() + at);
            }
            at += (size_t)hh[i];
        }
        idx_out.resize(at);
        if (want_val) val_out.resize(at);
        done = true;
    } else {
        (void)nq, (void)d, (void)Q, (void)thr, (void)kc, (void)want_val, (void)cnt_out;
        (void)start_out, (void)idx_out, (void)val_out;
    }
    return da_status_success;
}

// Core of the radius search (radius_neighbors_compute, nearest_neighbors.cpp:
// 1983-2068): per query its count and start in the flat index / value arrays,
// rows in index order; values (only when want_val) as computed, squared for
// euclidean (`squares`).  Options and queries are validated by the caller.
template <typename T>
da_status NN<T>::radius_compute(da_int nq, da_int d, const T *Xt, da_int ldt, T r, bool want_val,
                                std::vector<da_int> &cnt_out, std::vector<long long> &start_out,
                                std::vector<da_int> &idx_out, std::vector<T> &val_out,
                                bool &squares) {
    da_status s;
    cnt_out.assign((size_t)nq, 0);
    start_out.assign((size_t)nq, 0);
    idx_out.clear();
    val_out.clear();
    s = ensure_device_data();
    if (s != da_status_success) return s;
    cudaStream_t st = cuda->stream;
    int acc = ACC_SQEUC, post = POST_NONE, tf = 0, norm_kind = -1;
    switch (metric) {
    case M_EUC: acc = ACC_SQEUC; tf = 1; break;
    case M_SQEUC: acc = ACC_SQEUC; break;
    case M_EUC_GEMM: acc = ACC_DOT; post = POST_GEMM_SQ_CLAMP; tf = 1; norm_kind = 0; break;
    case M_SQEUC_GEMM: acc = ACC_DOT; post = POST_GEMM_SQ_CLAMP; norm_kind = 0; break;
    case M_MANH: acc = ACC_MANHATTAN; break;
    case M_COS: acc = ACC_DOT; post = POST_COSINE; norm_kind = 1; break;
    case M_IP: acc = ACC_DOT; break; // radius predict only: rows with dot <= r
    case M_MINK:
        if (p == T(2)) { acc = ACC_SQEUC; tf = 1; }
        else if (p == T(1)) { acc = ACC_MANHATTAN; }
        else { acc = ACC_MINKOWSKI; post = POST_POW; }
        break;
    }
    squares = tf == 1;
    const T thr = squares ? r * r : r;
    const bool fp64 = sizeof(T) == 8;
    const int kc = opts.key("reference isa") == 1 ? (fp64 ? 32 : 64) : (fp64 ? 512 : 256);
    if (!dQ.ensure((size_t)nq * ld * sizeof(T)))
        return err->error(da_status_memory_error, "Device memory allocation failed.");
    B200_TRY(upload_matrix<T>(order(), nq, d, Xt, ldt, dQ.as<T>(), ld, dStage, st), "upload of X_test");
    const T *qn = nullptr, *xn = nullptr;
    if (norm_kind >= 0) {
        if (!dQn.ensure((size_t)nq * sizeof(T)) || !dXn.ensure((size_t)n_samples * sizeof(T)))
            return err->error(da_status_memory_error, "Device memory allocation failed.");
        if (norm_kind == 0) {
            B200_TRY(launch_row_sqnorms<T>(dQ.as<T>(), ld, nq, d, dQn.as<T>(), st), "norms");
            if (xn_kind != 0)
                B200_TRY(launch_row_sqnorms<T>(dX.as<T>(), ld, n_samples, d, dXn.as<T>(), st), "norms");
        } else {
            B200_TRY(launch_row_norms_eps1<T>(dQ.as<T>(), ld, nq, d, dQn.as<T>(), st), "norms");
            if (xn_kind != 1)
                B200_TRY(launch_row_norms_eps1<T>(dX.as<T>(), ld, n_samples, d, dXn.as<T>(), st), "norms");
        }
        xn_kind = norm_kind;
        qn = dQn.as<T>();
        xn = dXn.as<T>();
    }
    cuda->stats["tensor_core"] = 0.0;
    const size_t n = (size_t)n_samples;
    // testing hook: the offsets' waits run out (AOCLDA_B200_TEST_RADIUS_WAIT=1)
    const char *tw = std::getenv("AOCLDA_B200_TEST_RADIUS_WAIT");
    const int test_wait = (tw && tw[0] == '1') ? 1 : 0;
    // the tensor-core path, block by block until one is not taken; in blocks
    // whose masks fit in 256 MB.  The rule is that of kneighbors (200,000 x 64,
    // one query: 117 us, the plain path 189; 16,384 x 64, 512 queries: 125
    // against 180), once the copies of the training rows exist or the handle's
    // radius searches come to 4e9 multiply-adds: the copies and buffers cost
    // 0.6 ms to set up, what a search of that size saves (3.1 -> 0.9 ms at
    // 1.3e10, 200,000 x 32, 2,000 queries).  A refused search has paid for the
    // mask (a tenth of the plain path): those of no smaller radius after it skip
    // this path 1, 2, 4 .. 16 times before it is tried again.
    da_int first = 0;
    const double work = (double)n * (double)std::max<da_int>(nq, 64) * (double)d;
    if (!fp64 && acc == ACC_SQEUC && std::isfinite((double)thr) && test_wait == 0 &&
        opts.key("precision mode") != 0 && knn_tc_supported((int)n, (int)d, 1) && n >= 16384 &&
        work >= 5.0e8 && (tc_train_ready || (radius_work += work) >= 4.0e9) &&
        !(thr >= radius_refused && --radius_skip >= 0)) {
        da_int Bt = (da_int)std::max<size_t>(
            1, std::min<size_t>({(size_t)nq, (256u << 20) / ((size_t)radius_tc_words((int)n) * 4),
                                 (size_t)65535}));
        if (Bt < nq && Bt > 128) Bt -= Bt % 128;
        bool done = true;
        while (done && first < nq) {
            const da_int b = std::min<da_int>(Bt, nq - first);
            s = radius_tc(b, d, dQ.as<T>() + (size_t)first * ld, thr, kc, want_val,
                          cnt_out.data() + first, start_out.data() + first, idx_out, val_out, done);
            if (s != da_status_success) return s;
            if (done) first += b;
        }
        if (first == nq) {
            cuda->stats["tensor_core"] = 1.0;
            if (thr >= radius_refused) radius_accepted();
            return da_status_success;
        }
        radius_refused = thr;
        radius_skip = radius_wait = std::min(16, std::max(1, 2 * radius_wait));
    }
    // query blocks whose distance rows fit in 256 MB
    // (at most 65,535 rows: the count / compaction grids put the rows on y)
    // (and a whole number of the distance kernel's 64-row tiles when there
    // are more queries: a partial last tile row costs a full one)
    da_int B = (da_int)std::max<size_t>(
        1, std::min<size_t>({(size_t)nq, (256u << 20) / (n * sizeof(T)), (size_t)65535}));
    if (B < nq && B > 64) B -= B % 64;
    const int nch = radius_chunks((int)n);
    if (!dD.ensure((size_t)B * n * sizeof(T)) ||
        !dRc.ensure(radius_scan_work_bytes((int)B, (int)n) + 64) ||
        !dRs.ensure((size_t)B * nch * sizeof(long long)) ||
        !dRh.ensure((size_t)B * nch * sizeof(int)))
        return err->error(da_status_memory_error, "Device memory allocation failed.");
    std::vector<long long> start((size_t)B * nch + 2);
    // the distance kernel also counts each (row, chunk) piece's hits
    PairwiseArgs pa{acc, post, kc, (double)p, false, true};
    pa.thr = (double)thr;
    pa.hits = dRh.as<int>();
    long long *d_total = reinterpret_cast<long long *>(dRc.as<char>() +
                                                       radius_scan_work_bytes((int)B, (int)n));
    int *d_err = reinterpret_cast<int *>(d_total + 1);
    for (da_int q0 = first; q0 < nq; q0 += B) {
        const int b = (int)std::min<da_int>(B, nq - q0);
        B200_TRY(cudaMemsetAsync(dRh.p, 0, (size_t)b * nch * sizeof(int), st), "memset");
        B200_TRY(cuda->timed("radius_distances", [&] {
            return launch_pairwise<T>(dQ.as<T>() + (size_t)q0 * ld, ld, b, dX.as<T>(), ld, (int)n,
                                      (int)d, qn ? qn + q0 : nullptr, xn, pa, dD.as<T>(), st);
        }), "distance kernel");
        // counts and offsets in (row, chunk) order on the device: every row's
        // hits stay in index order
        B200_TRY(cuda->timed("radius_count", [&] {
            return launch_radius_count_scan<T>(dD.as<T>(), b, (int)n, n, thr, dRc.p,
                                               dRs.as<long long>(), d_total, d_err, test_wait, st,
                                               dRh.as<int>());
        }), "count");
        B200_TRY(cudaMemcpyAsync(start.data(), dRs.p, (size_t)b * nch * sizeof(long long),
                                 cudaMemcpyDeviceToHost, st), "copy");
        B200_TRY(cudaMemcpyAsync(start.data() + (size_t)b * nch, d_total, 2 * sizeof(long long),
                                 cudaMemcpyDeviceToHost, st), "copy");
        B200_TRY(cudaStreamSynchronize(st), "radius search");
        int scan_err = 0;
        std::memcpy(&scan_err, start.data() + (size_t)b * nch + 1, sizeof(int));
        if (scan_err != 0)
            return err->error(da_status_internal_error,
                              "The radius search's offset scan timed out waiting for another "
                              "block of the GPU.");
        const long long tot = start[(size_t)b * nch];
        const size_t base = idx_out.size();
        for (int i = 0; i < b; ++i) {
            const long long s0 = start[(size_t)i * nch];
            const long long s1 = i + 1 < b ? start[(size_t)(i + 1) * nch] : tot;
            start_out[(size_t)q0 + i] = (long long)base + s0;
            cnt_out[(size_t)q0 + i] = (da_int)(s1 - s0);
        }
        if (tot == 0) continue;
        if (!dRi.ensure((size_t)tot * sizeof(int)) || !dRv.ensure((size_t)tot * sizeof(T)))
            return err->error(da_status_memory_error, "Device memory allocation failed.");
        B200_TRY(cuda->timed("radius_emit", [&] {
            return launch_radius_emit<T>(dD.as<T>(), b, (int)n, n, thr, dRs.as<long long>(),
                                         dRi.as<int>(), dRv.as<T>(), st);
        }), "compaction");
        idx_out.resize(base + (size_t)tot);
        if (want_val) val_out.resize(base + (size_t)tot);
        std::vector<int> ii((size_t)tot);
        B200_TRY(cudaMemcpyAsync(ii.data(), dRi.p, (size_t)tot * sizeof(int),
                                 cudaMemcpyDeviceToHost, st), "copy");
        if (want_val)
            B200_TRY(cudaMemcpyAsync(val_out.data() + base, dRv.p, (size_t)tot * sizeof(T),
                                     cudaMemcpyDeviceToHost, st), "copy");
        B200_TRY(cudaStreamSynchronize(st), "radius search");
        for (size_t i = 0; i < (size_t)tot; ++i) idx_out[base + i] = (da_int)ii[i];
    }
    return da_status_success;
}

// nearest_neighbors.cpp:940-1015
// Radius neighbours, brute force (nearest_neighbors.cpp:1915-2068 and the
// brute-force search :2070-2247): the distance block of the kNN path's
// metric plan (squared for euclidean, compared with radius^2), the rows
// within the radius in index order per query, then (sort_results) a stable
// sort by distance as sorted_n_dist_n_ind (nearest_neighbors_utils.hpp:73-101).
template <typename T>
da_status NN<T>::radius_neighbors(da_int nq, da_int d, const T *Xt, da_int ldt, T r,
                                  da_int return_distance, da_int sort_results) {
    if (!return_distance && sort_results)
        return err->error(da_status_invalid_input,
                          "Cannot sort results if distances are not returned.");
    if (!have_X)
        return err->error(da_status_no_data,
                          "No training data have been set. Please call da_nn_set_data_s or "
                          "da_nn_set_data_d.");
    da_status s = check_options_update();
    if (s != da_status_success) return s;
    if (metric == M_IP)
        return err->error(da_status_incompatible_options,
                          "The inner product metric is not compatible with radius neighbors. "
                          "Use da_nn_kneighbors to find the k most similar training vectors by "
                          "inner product.");
    s = validate_queries(nq, d, Xt, ldt);
    if (s != da_status_success) return s;
    if (r < T(0)) r = (T)opts.r("radius");
    model_trained = false;
    s = radius_compute(nq, d, Xt, ldt, r, return_distance || sort_results, rnn_count, rnn_start,
                       rnn_idx, rnn_val, rnn_squares);
    if (s != da_status_success) return s;
    rnn_dist = return_distance != 0;
    if (sort_results) {
        std::vector<da_int> perm, ti;
        std::vector<T> tv;
        for (da_int q = 0; q < nq; ++q) {
            const size_t o = (size_t)rnn_start[q], m = (size_t)rnn_count[q];
            perm.resize(m);
            for (size_t i = 0; i < m; ++i) perm[i] = (da_int)i;
            std::stable_sort(perm.begin(), perm.end(), [&](da_int a, da_int b) {
                return rnn_val[o + a] < rnn_val[o + b];
            });
            ti.assign(rnn_idx.begin() + o, rnn_idx.begin() + o + m);
            tv.assign(rnn_val.begin() + o, rnn_val.begin() + o + m);
            for (size_t i = 0; i < m; ++i) {
                rnn_idx[o + i] = ti[perm[i]];
                rnn_val[o + i] = tv[perm[i]];
            }
        }
    }
    model_trained = true;
    return da_status_success;
}

// Result queries of the radius search (nearest_neighbors.cpp:118-260).
template <typename T> da_status NN<T>::radius_values(da_result q, da_int *dim, T *out) {
    if (!model_trained)
        return err->warn(da_status_no_data,
                         "Radius neighbors have not been computed. Please call "
                         "da_nn_radius_neighbors_s or da_nn_radius_neighbors_d first.");
    if (q != da_nn_radius_neighbors_distances && q != da_nn_radius_neighbors_distances_index)
        return err->warn(da_status_unknown_query, "The requested result could not be found.");
    if (!rnn_dist)
        return err->warn(da_status_no_data,
                         "Distances were not requested during radius neighbors computation. "
                         "Please set return_distance to true in da_nn_radius_neighbors_s or "
                         "da_nn_radius_neighbors_d call.");
    const da_int nq = (da_int)rnn_count.size();
    auto put = [&](da_int qi, T *dst) {
        const size_t o = (size_t)rnn_start[qi];
        for (da_int i = 0; i < rnn_count[qi]; ++i)
            dst[i] = rnn_squares ? std::sqrt(rnn_val[o + i]) : rnn_val[o + i];
    };
    if (q == da_nn_radius_neighbors_distances_index) {
        const da_int qi = (da_int)out[0];
        if (qi < 0 || qi >= nq)
            return err->warn(da_status_invalid_input,
                             "The provided index is out of bounds. It should be in the range [0, " +
                                 std::to_string(nq - 1) + "].");
        if (rnn_count[qi] > *dim) {
            *dim = rnn_count[qi];
            return err->warn(da_status_invalid_array_dimension,
                             "The array is too small. Please provide an array of at least size: " +
                                 std::to_string(rnn_count[qi]) + ".");
        }
        put(qi, out);
        return da_status_success;
    }
    const da_int total = (da_int)rnn_val.size();
    if (total > *dim) {
        *dim = total;
        return err->warn(da_status_invalid_array_dimension,
                         "The array is too small. Please provide an array of at least size: " +
                             std::to_string(total) + ".");
    }
    da_int a = 0;
    for (da_int qi = 0; qi < nq; ++qi) {
        put(qi, out + a);
        a += rnn_count[qi];
    }
    return da_status_success;
}
template <typename T> da_status NN<T>::get_result(da_result q, da_int *dim, double *out) {
    if constexpr (std::is_same_v<T, double>) return radius_values(q, dim, out);
    (void)q, (void)dim, (void)out;
    return err->error(da_status_wrong_type, "Wrong precision type.");
}
template <typename T> da_status NN<T>::get_result(da_result q, da_int *dim, float *out) {
    if constexpr (std::is_same_v<T, float>) return radius_values(q, dim, out);
    (void)q, (void)dim, (void)out;
    return err->error(da_status_wrong_type, "Wrong precision type.");
}
template <typename T> da_status NN<T>::get_result_int(da_result q, da_int *dim, da_int *out) {
    if (q == da_trained) return AlgBase::get_result_int(q, dim, out);
    if (!model_trained)
        return err->warn(da_status_no_data,
                         "Radius neighbors have not been computed. Please call "
                         "da_nn_radius_neighbors first.");
    const da_int nq = (da_int)rnn_count.size();
    const da_int total = (da_int)rnn_idx.size();
    switch (q) {
    case da_nn_radius_neighbors_count:
    case da_nn_radius_neighbors_offsets: {
        if (nq + 1 > *dim) {
            *dim = nq + 1;
            return err->warn(da_status_invalid_array_dimension,
                             "The array is too small. Please provide an array of at least size: " +
                                 std::to_string(nq + 1) + ".");
        }
        da_int off = 0;
        for (da_int i = 0; i < nq; ++i) {
            if (q == da_nn_radius_neighbors_count) out[i] = rnn_count[i];
            else out[i] = rnn_count[i] > 0 ? off : -1;
            off += rnn_count[i];
        }
        out[nq] = off;
        return da_status_success;
    }
    case da_nn_radius_neighbors_indices_index: {
        const da_int qi = out[0];
        if (qi < 0 || qi >= nq)
            return err->warn(da_status_invalid_input,
                             "The provided index is out of bounds. It should be in the range [0, " +
                                 std::to_string(nq - 1) + "].");
        if (rnn_count[qi] > *dim) {
            *dim = rnn_count[qi];
            return err->warn(da_status_invalid_array_dimension,
                             "The array is too small. Please provide an array of at least size: " +
                                 std::to_string(rnn_count[qi]) + ".");
        }
        for (da_int i = 0; i < rnn_count[qi]; ++i) out[i] = rnn_idx[(size_t)rnn_start[qi] + i];
        return da_status_success;
    }
    case da_nn_radius_neighbors_indices: {
        if (total > *dim) {
            *dim = total;
            return err->warn(da_status_invalid_array_dimension,
                             "The array is too small. Please provide an array of at least size: " +
                                 std::to_string(total) + ".");
        }
        da_int a = 0;
        for (da_int qi = 0; qi < nq; ++qi)
            for (da_int i = 0; i < rnn_count[qi]; ++i) out[a++] = rnn_idx[(size_t)rnn_start[qi] + i];
        return da_status_success;
    }
    default:
        return err->warn(da_status_unknown_query, "The requested result could not be found.");
    }
}

template <typename T>
da_status NN<T>::kneighbors(da_int nq, da_int d, const T *Xt, da_int ldt, da_int *n_ind,
                            T *n_dist, da_int k, da_int return_distance) {
    if (!have_X)
        return err->error(da_status_no_data,
                          "No training data have been set. Please call da_nn_set_data_s or "
                          "da_nn_set_data_d.");
    da_status s = check_options_update();
    if (s != da_status_success) return s;
    if (n_ind == nullptr) return err->error(da_status_invalid_pointer, "n_ind is not a valid pointer.");
    s = validate_queries(nq, d, Xt, ldt);
    if (s != da_status_success) return s;
    if (k <= 0 && n_neighbors <= 0)
        return err->error(da_status_invalid_input, "Number of requested neighbors must be positive.");
    if (k <= 0) k = n_neighbors;
    if (k > n_samples)
        return err->error(da_status_invalid_input,
                          "Number of requested neighbors must be at least as big as the number "
                          "of samples.");
    if (return_distance && n_dist == nullptr)
        return err->error(da_status_invalid_pointer, "n_dist is not a valid pointer.");
    std::vector<da_int> ind;
    const KnnOut to{n_ind, return_distance ? n_dist : nullptr};
    // outputs: q-major for row-major storage, n_queries x k column-major otherwise
    return kneighbors_compute(nq, d, Xt, ldt, order(), k, ind, nullptr, &to);
}

template <typename T> da_status NN<T>::available_classes() {
    if (!have_X)
        return err->error(da_status_no_data,
                          "No training data have been set. Please call da_nn_set_data_s or "
                          "da_nn_set_data_d.");
    if (!have_labels)
        return err->error(da_status_no_data,
                          "No classification labels have been set. Please call "
                          "da_nn_set_labels_s or da_nn_set_labels_d.");
    std::set<da_int> s(y_class, y_class + n_samples);
    classes.assign(s.begin(), s.end());
    classes_done = true;
    return da_status_success;
}

template <typename T> da_status NN<T>::classes_api(da_int *n_classes, da_int *cls) {
    if (n_classes == nullptr)
        return err->error(da_status_invalid_pointer, "n_classes is not a valid pointer.");
    if (!classes_done) {
        da_status s = available_classes();
        if (s != da_status_success) return s;
    }
    const da_int nc = (da_int)classes.size();
    if (*n_classes <= 0 || cls == nullptr) {
        *n_classes = nc;
        return da_status_success;
    }
    if (*n_classes < nc) {
        *n_classes = nc;
        return err->error(da_status_invalid_array_dimension,
                          "The classes array is too small, it must be at least " +
                              std::to_string(nc) + ".");
    }
    for (da_int i = 0; i < nc; ++i) cls[i] = classes[i];
    *n_classes = nc;
    return da_status_success;
}

// Vote of predict_proba_compute_knn (nearest_neighbors.cpp:1166-1272):
// proba is q-major (q * n_classes + c).
template <typename T>
da_status NN<T>::compute_proba(da_int nq, da_int d, const T *Xt, da_int ldt,
                               std::vector<T> &proba) {
    if (metric == M_IP && weights == 1)
        return err->error(da_status_incompatible_options,
                          "The inner product metric is not compatible with "
                          "weights=\"distance\". Use weights=\"uniform\" instead.");
    if (!classes_done) {
        da_status s = available_classes();
        if (s != da_status_success) return s;
    }
    const da_int k = n_neighbors;
    if (k > n_samples)
        return err->error(da_status_invalid_input,
                          "Number of requested neighbors must be at least as big as the number "
                          "of samples.");
    std::vector<da_int> ind;
    std::vector<T> dist;
    da_status s = kneighbors_compute(nq, d, Xt, ldt, order(), k, ind, weights == 1 ? &dist : nullptr);
    if (s != da_status_success) return s;
    const da_int nc = (da_int)classes.size();
    proba.assign((size_t)nq * nc, T(0));
    for (da_int q = 0; q < nq; ++q) {
        T *pq = proba.data() + (size_t)q * nc;
        // per class, the neighbours' weights in neighbour order
        for (da_int r = 0; r < k; ++r) {
            const da_int at = ind[(size_t)q * k + r];
            if (at < 0) continue; // fewer than k rows at a distance that is a number
            const da_int lbl = y_class[at];
            const da_int c = (da_int)(std::lower_bound(classes.begin(), classes.end(), lbl) -
                                      classes.begin());
            if (c == nc || classes[c] != lbl) continue;
            T v = T(1);
            if (weights != 0) {
                const T w = dist[(size_t)q * k + r];
                v = (w <= std::numeric_limits<T>::epsilon()) ? T(1) : T(1) / w;
            }
            pq[c] += v;
        }
        T den = T(0);
        for (da_int c = 0; c < nc; ++c) den += pq[c];
        for (da_int c = 0; c < nc; ++c) pq[c] /= den;
    }
    return da_status_success;
}

// Radius-mode vote (predict_proba_compute_rnn, nearest_neighbors.cpp:1280-1479):
// the rows within the "radius" option of each query vote for their labels,
// with weight 1 (uniform) or 1 / distance (distance; 1 at distance <= eps).
// A query with no row within the radius is an error under outlier handling
// "none"; "manual" gives it probability 1 for the "outlier label" (all zero
// and a warning when that label is not a training label), "most frequent"
// probability 1 for the most frequent training label.  proba is q-major.
template <typename T>
da_status NN<T>::compute_proba_rnn(da_int nq, da_int d, const T *Xt, da_int ldt,
                                   std::vector<T> &proba) {
    if (metric == M_IP && weights == 1)
        return err->error(da_status_incompatible_options,
                          "The inner product metric is not compatible with "
                          "weights=\"distance\". Use weights=\"uniform\" instead.");
    if (!classes_done) {
        da_status s = available_classes();
        if (s != da_status_success) return s;
    }
    const da_int oh = opts.key("outlier handling");
    const da_int nc = (da_int)classes.size();
    const da_int mf = oh == OH_MOST_FREQUENT ? most_frequent_label() : 0;
    da_int manual_idx = -1;
    if (oh == OH_MANUAL) {
        auto it = std::lower_bound(classes.begin(), classes.end(), (da_int)opts.i("outlier label"));
        if (it != classes.end() && *it == (da_int)opts.i("outlier label"))
            manual_idx = (da_int)(it - classes.begin());
    }
    std::vector<da_int> cnt, idx;
    std::vector<long long> start;
    std::vector<T> val;
    bool squares = false;
    da_status s = radius_compute(nq, d, Xt, ldt, (T)opts.r("radius"), weights == 1, cnt, start,
                                 idx, val, squares);
    if (s != da_status_success) return s;
    proba.assign((size_t)nq * nc, T(0));
    bool outliers = false;
    for (da_int q = 0; q < nq; ++q) {
        T *pq = proba.data() + (size_t)q * nc;
        const size_t o = (size_t)start[q], m = (size_t)cnt[q];
        if (m == 0) {
            if (oh == OH_NONE)
                return err->error(da_status_operation_failed,
                                  "Failed to compute probabilities for query " + std::to_string(q) +
                                      " since it does not have any neighbors within the "
                                      "specified radius.");
            if (oh == OH_MANUAL) {
                outliers = true;
                if (manual_idx != -1) pq[manual_idx] = T(1);
            } else {
                for (da_int c = 0; c < nc; ++c) pq[c] = classes[c] == mf ? T(1) : T(0);
            }
            continue;
        }
        // per class, the neighbours' weights in neighbour order
        for (size_t i = 0; i < m; ++i) {
            const da_int c = (da_int)(std::lower_bound(classes.begin(), classes.end(),
                                                       y_class[idx[o + i]]) - classes.begin());
            pq[c] += weights == 0 ? T(1) : radius_weight(val[o + i], squares);
        }
        T den = T(0);
        for (da_int c = 0; c < nc; ++c) den += pq[c];
        for (da_int c = 0; c < nc; ++c) pq[c] /= den;
    }
    if (oh == OH_MANUAL && outliers && manual_idx == -1)
        return err->warn(da_status_outlier_warning,
                         "The manually set outlier label is not present in the training labels. "
                         "Setting probabilities to 0.0.");
    return da_status_success;
}

// most_frequent_element (nearest_neighbors.cpp:1037-1058): the most frequent
// training label, the smallest of equally frequent ones.
template <typename T> da_int NN<T>::most_frequent_label() {
    std::map<da_int, da_int> freq;
    for (da_int i = 0; i < n_samples; ++i) freq[y_class[i]]++;
    da_int best = y_class[0], top = 0;
    for (const auto &f : freq)
        if (f.second > top) {
            top = f.second;
            best = f.first;
        }
    return best;
}

// get_weights (nearest_neighbors.cpp:1021-1033) of one radius neighbour; the
// stored value is squared for euclidean.
template <typename T> T NN<T>::radius_weight(T v, bool squares) {
    const T w = squares ? std::sqrt(v) : v;
    return w <= std::numeric_limits<T>::epsilon() ? T(1) : T(1) / w;
}

template <typename T>
da_status NN<T>::predict_proba(da_int nq, da_int d, const T *Xt, da_int ldt, T *proba,
                               da_nn_search_mode mode) {
    if (!have_X)
        return err->error(da_status_no_data,
                          "No training data have been set. Please call da_nn_set_data_s or "
                          "da_nn_set_data_d.");
    if (!have_labels)
        return err->error(da_status_no_data,
                          "No classification labels have been set. Please call "
                          "da_nn_set_labels_s or da_nn_set_labels_d.");
    da_status s = check_options_update();
    if (s != da_status_success) return s;
    if (proba == nullptr) return err->error(da_status_invalid_pointer, "proba is not a valid pointer.");
    if (nq < 1)
        return err->error(da_status_invalid_array_dimension,
                          "Number of queries must be greater than zero.");
    if (d < 1)
        return err->error(da_status_invalid_array_dimension,
                          "Number of features must be greater than zero.");
    s = validate_queries(nq, d, Xt, ldt);
    if (s != da_status_success) return s;
    if (mode != knn_search_mode && mode != radius_search_mode)
        return err->error(da_status_invalid_input,
                          "Unknown search mode: " + std::to_string((int)mode) + ".");
    std::vector<T> pr;
    s = mode == knn_search_mode ? compute_proba(nq, d, Xt, ldt, pr)
                                : compute_proba_rnn(nq, d, Xt, ldt, pr);
    if (s != da_status_success && s != da_status_outlier_warning) return s;
    const da_int nc = (da_int)classes.size();
    const bool cm = order() == column_major;
    for (da_int q = 0; q < nq; ++q)
        for (da_int c = 0; c < nc; ++c)
            proba[cm ? (size_t)c * nq + q : (size_t)q * nc + c] = pr[(size_t)q * nc + c];
    return s;
}

template <typename T>
da_status NN<T>::predict(da_int nq, da_int d, const T *Xt, da_int ldt, da_int *y,
                         da_nn_search_mode mode) {
    da_status s = check_options_update();
    if (s != da_status_success) return s;
    if (!have_X)
        return err->error(da_status_no_data,
                          "No training data have been set. Please call da_nn_set_data_s or "
                          "da_nn_set_data_d.");
    if (!have_labels)
        return err->error(da_status_no_data,
                          "No classification labels have been set. Please call "
                          "da_nn_set_labels_s or da_nn_set_labels_d.");
    if (y == nullptr) return err->error(da_status_invalid_pointer, "y_test is not a valid pointer.");
    if (nq < 1)
        return err->error(da_status_invalid_array_dimension, "n_queries must be greater than 0.");
    s = validate_queries(nq, d, Xt, ldt);
    if (s != da_status_success) return s;
    if (mode != knn_search_mode && mode != radius_search_mode)
        return err->error(da_status_invalid_input,
                          "Unknown search mode: " + std::to_string((int)mode) + ".");
    std::vector<T> pr;
    s = mode == knn_search_mode ? compute_proba(nq, d, Xt, ldt, pr)
                                : compute_proba_rnn(nq, d, Xt, ldt, pr);
    if (s != da_status_success && s != da_status_outlier_warning) return s;
    const da_int nc = (da_int)classes.size();
    // radius mode with outlier handling: an all-zero row (a query without
    // neighbours) takes the outlier label or the most frequent label
    // (nearest_neighbors.cpp:1566-1599)
    const da_int oh = mode == knn_search_mode ? OH_NONE : opts.key("outlier handling");
    const da_int fill = oh == OH_MANUAL ? (da_int)opts.i("outlier label")
                        : oh == OH_MOST_FREQUENT ? most_frequent_label() : 0;
    for (da_int q = 0; q < nq; ++q) {
        // first maximum (cblas_iamax semantics, nearest_neighbors.cpp:1566-1573)
        da_int best = 0;
        T bv = std::fabs(pr[(size_t)q * nc]);
        for (da_int c = 1; c < nc; ++c) {
            const T v = std::fabs(pr[(size_t)q * nc + c]);
            if (v > bv) {
                bv = v;
                best = c;
            }
        }
        y[q] = (oh != OH_NONE && pr[(size_t)q * nc + best] == T(0)) ? fill : classes[best];
    }
    return s;
}

template <typename T>
da_status NN<T>::predict_reg(da_int nq, da_int d, const T *Xt, da_int ldt, T *y,
                             da_nn_search_mode mode) {
    if (!have_X)
        return err->error(da_status_no_data,
                          "No training data have been set. Please call da_nn_set_data_s or "
                          "da_nn_set_data_d.");
    if (!have_targets)
        return err->error(da_status_no_data,
                          "No regression targets have been set. Please call "
                          "da_nn_set_targets_s or da_nn_set_targets_d.");
    da_status s = check_options_update();
    if (s != da_status_success) return s;
    if (y == nullptr) return err->error(da_status_invalid_pointer, "y_test is not a valid pointer.");
    if (nq < 1)
        return err->error(da_status_invalid_array_dimension, "n_queries must be greater than 0.");
    s = validate_queries(nq, d, Xt, ldt);
    if (s != da_status_success) return s;
    if (mode != knn_search_mode && mode != radius_search_mode)
        return err->error(da_status_invalid_input,
                          "Unknown search mode: " + std::to_string((int)mode) + ".");
    if (metric == M_IP && weights == 1)
        return err->error(da_status_incompatible_options,
                          "The inner product metric is not compatible with "
                          "weights=\"distance\". Use weights=\"uniform\" instead.");
    if (mode == radius_search_mode) return predict_reg_rnn(nq, d, Xt, ldt, y);
    const da_int k = n_neighbors;
    if (k > n_samples)
        return err->error(da_status_invalid_input,
                          "Number of requested neighbors must be at least as big as the number "
                          "of samples.");
    std::vector<da_int> ind;
    std::vector<T> dist;
    s = kneighbors_compute(nq, d, Xt, ldt, order(), k, ind, weights == 1 ? &dist : nullptr);
    if (s != da_status_success) return s;
    // nearest_neighbors.cpp:1707-1747
    // (a query with fewer than k rows at a distance that is a number has no value)
    const auto target = [&](size_t e) {
        return ind[e] < 0 ? std::numeric_limits<T>::quiet_NaN() : y_reg[ind[e]];
    };
    for (da_int q = 0; q < nq; ++q) {
        if (weights == 0) {
            T sum = T(0);
            for (da_int r = 0; r < k; ++r) sum += target((size_t)q * k + r);
            y[q] = sum / T(k);
        } else {
            T num = T(0), den = T(0);
            for (da_int r = 0; r < k; ++r) {
                const T dv = dist[(size_t)q * k + r];
                const T w = (dv <= std::numeric_limits<T>::epsilon()) ? T(1) : T(1) / dv;
                num += target((size_t)q * k + r) * w;
                den += w;
            }
            y[q] = num / den;
        }
    }
    return da_status_success;
}

// Radius-mode regression (predict_targets_rnn, nearest_neighbors.cpp:1763-1909):
// the mean target of the rows within the radius (uniform) or their
// 1 / distance weighted mean (distance).  A query without neighbours is an
// error under outlier handling "none"; it takes the mean training target
// under "most frequent" and the "outlier target" (with a warning) under
// "manual".
template <typename T>
da_status NN<T>::predict_reg_rnn(da_int nq, da_int d, const T *Xt, da_int ldt, T *y) {
    const da_int oh = opts.key("outlier handling");
    T mean_target = T(0);
    if (oh == OH_MOST_FREQUENT) {
        for (da_int i = 0; i < n_samples; ++i) mean_target += y_reg[i];
        mean_target /= T(n_samples);
    }
    const T manual_target = (T)opts.r("outlier target");
    std::vector<da_int> cnt, idx;
    std::vector<long long> start;
    std::vector<T> val;
    bool squares = false;
    da_status s = radius_compute(nq, d, Xt, ldt, (T)opts.r("radius"), weights == 1, cnt, start,
                                 idx, val, squares);
    if (s != da_status_success) return s;
    bool outliers = false;
    for (da_int q = 0; q < nq; ++q) {
        const size_t o = (size_t)start[q], m = (size_t)cnt[q];
        if (m == 0) {
            if (oh == OH_NONE)
                return err->error(da_status_operation_failed,
                                  std::string(weights == 0 ? "Failed to compute targets for query "
                                                           : "Failed to predict targets for query ") +
                                      std::to_string(q) +
                                      " since it does not have any neighbors within the "
                                      "specified radius.");
            if (oh == OH_MOST_FREQUENT) {
                y[q] = mean_target;
            } else {
                outliers = true;
                y[q] = manual_target;
            }
            continue;
        }
        if (weights == 0) {
            T sum = T(0);
            for (size_t i = 0; i < m; ++i) sum += y_reg[idx[o + i]];
            y[q] = sum / T(m);
        } else {
            T num = T(0), den = T(0);
            for (size_t i = 0; i < m; ++i) {
                const T w = radius_weight(val[o + i], squares);
                num += y_reg[idx[o + i]] * w;
                den += w;
            }
            y[q] = num / den;
        }
    }
    if (oh == OH_MANUAL && outliers)
        return err->warn(da_status_outlier_warning,
                         "One or more samples have no neighbors within the specified radius. "
                         "Setting the corresponding targets to " + std::to_string(manual_target) +
                             ".");
    return da_status_success;
}

template struct NN<float>;
template struct NN<double>;

} // namespace b200
