/* C ABI of the surrogate library's whole-network passes
 * (dense_b200/_lib/libdense_b200_surrogate.so): training, prediction and
 * ranking with a launch or a few each, beside the single kernels of
 * dense_b200_surrogate.h and under its rules (device pointers unless stated;
 * 0 launched, 1 refused before any CUDA call, 2 launch error). */
#ifndef DENSE_B200_NETWORK_H
#define DENSE_B200_NETWORK_H

#include <stdint.h>

#ifdef __cplusplus
extern "C" {
#endif

/* Whole passes of the surrogate's network: n_in <= 64 inputs, three hidden
 * layers of 256 with GELU, n_out <= 128 outputs.  FP32 weights W[4] are
 * [256][64], [256][256], [256][256], [128][256] (row-major, rows past n_out
 * and columns past n_in zero), biases b[4] of 256, 256, 256 and 128; W, bias,
 * dW, db and the moments are HOST arrays of device pointers (16-byte
 * aligned).  `packed` is dense_mlp_packed_bytes() of device memory that
 * dense_mlp_pack fills with the BF16 weights in the order the passes read
 * them; `backward` != 0 adds the part that training needs. */
int64_t dense_mlp_packed_bytes(void);
int dense_mlp_pack(const float* const* W, void* packed, int backward, void* stream);

/* out[rows][n_out] = network(X[rows][n_in]) (leading dimension ldx). */
int dense_mlp_predict(const float* X, int ldx, int rows, int n_in, const void* packed, const float* const* bias,
                      int n_out, float* out, int* err, void* stream);

/* Ranking scores of candidates P[rows][ldp] (FP64): the encoding of
 * dense_features_encode, every network of the ensemble (packed[nets],
 * bias[nets][4]; at most 64) and dense_features_score in one launch. */
int dense_mlp_rank(const double* P, int ldp, int rows, const int* cols, const double* tmpl, int n_in,
                   double log_spread, int nets, const void* const* packed, const float* const* bias, int n_out,
                   const float* mu, const float* sd, double weight, double period, double tol, double amp_min,
                   double ramp, double* out, int* err, void* stream);

/* One batch forward and back: rows idx[0..rows) of X, T and mask (idx NULL:
 * the first `rows` rows; indices outside [0, x_rows) give zero rows).
 * loss += sum mask (Y - T)^2 * inv_count (read from the device when
 * inv_count is not NULL, else inv_value); the gradients' parts stay in
 * `work` (dense_mlp_train_bytes(rows, n_out) bytes, 256-byte aligned, one
 * stream) for dense_mlp_train_finish, which sums them into dW and db (when
 * given) and, when `hyper` ({lr, b1, b2, eps, 1 - b1^t, 1 - b2^t} on the
 * device) is given, applies Adam and packs the new weights. */
int64_t dense_mlp_train_bytes(int rows, int n_out);
int dense_mlp_train_pass(const float* X, int ldx, int x_rows, int n_in, const float* T, const float* mask, int n_out,
                         const int* idx, int rows, const void* packed, const float* const* bias,
                         const float* inv_count, float inv_value, float* loss, void* work, int64_t work_bytes,
                         int* err, void* stream);
int dense_mlp_train_finish(const void* work, int64_t work_bytes, int rows, int n_out, float* const* dW,
                           float* const* db, const float* hyper, float* const* W, float* const* b, float* const* mW,
                           float* const* vW, float* const* mb, float* const* vb, void* packed, void* stream);

/* `steps` steps of such a pass and finish one after the other: step j takes
 * the `rows` rows idx[j * rows ..] and the scalars hyper[8 * j ..] ({lr, b1,
 * b2, eps, 1 - b1^t, 1 - b2^t, inv_count}), both on the device.  `packed`
 * holds the weights' packing on entry, and that of the new weights after. */
int dense_mlp_train_epoch(const float* X, int ldx, int x_rows, int n_in, const float* T, const float* mask, int n_out,
                          const int* idx, int rows, int steps, const float* hyper, float* loss, void* work,
                          int64_t work_bytes, float* const* W, float* const* b, float* const* mW, float* const* vW,
                          float* const* mb, float* const* vb, void* packed, int* err, void* stream);

#ifdef __cplusplus
}
#endif

#endif /* DENSE_B200_NETWORK_H */
