// Candidate-kNN classifier pieces on device buffers (column-major FP64).
#pragma once

#include <vector>

#include "common.cuh"

namespace fpls {

// Rows grouped by class code: class c (0-based) holds rows offs[c] .. offs[c + 1] - 1.
struct ClassRows {
  double* Ts = nullptr;         // rows in class order, row-major (offs[C] x k)
  const int* d_offs = nullptr;  // C + 1, device
  std::vector<int> offs;        // C + 1, host
};

// Class-contiguous slots of the codes (1..C, others dropped) given the class
// offsets: dest[i] = slot of code i (-1 when dropped), perm[slot] = i,
// sorted[slot] = its 0-based class; each may be null.
void class_slots(const int* codes, int n, int C, const int* d_offs, int* dest, int* perm, int* sorted);

// Class-contiguous, row-major copy of the rows of dT (n x k, column-major).
ClassRows group_rows_by_class(const double* dT, int n, int k, const int* dcodes, int C);

// dTn (n x k) = row_l2(dT dCk), or row_l2(dT) when dCk is null.
void candidate_scores_device(const double* dT, int n, int k, const double* dCk, double* dTn);

// The rows of row_l2(dT dCk), row-major: row i to dTs row dest[i] (dropped when negative).
void candidate_score_rows_device(const double* dT, int n, int k, const double* dCk, const int* dest, double* dTs);

// dCent (C x k) = row_l2 of the per-class means of the rows.
void candidate_centroids_device(const ClassRows& cr, int k, int C, double* dCent);

// Candidate selection, smoothed class-kNN scoring and rerank against the
// training rows cr; d_ti / d_ts are ntest x max(1, min(top_k, C)).  dbias may
// be null (zeros).
void candidate_knn_predict_device(const double* dTt, int ntest, const ClassRows& cr, int kdim, const double* dC,
                                  int C, const double* dbias, int top_k, int top_m, int knn_k, double tau,
                                  double alpha, int* d_ti, double* d_ts);

}  // namespace fpls
