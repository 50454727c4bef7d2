// The object behind an opaque bse_handle of the C ABI.
#pragma once

#include <memory>

#include "bse_ops.cuh"
#include "uks_ops.cuh"

struct bse_handle {
  int kind = 0;  // 0: BSE operator, 1: dense operator, 2: unrestricted (UKS) BSE operator
  std::unique_ptr<vgb::BseOperator> bse;
  std::unique_ptr<vgb::DenseOperator> dense;
  std::unique_ptr<vgb::UksOperator> uks;
  cudaStream_t stream = nullptr;
  vgb::DeviceBuffer<double> dX, dY, dD;
  int64_t size() const { return kind == 0 ? bse->dim : kind == 2 ? uks->dim : dense->n; }
  void matmul(const vgb::Coef &c, const double *X, int64_t ldx, int64_t k, double *Y, int64_t ldy,
              cudaStream_t s) {
    if (kind == 0) bse->matmul(c, X, ldx, k, Y, ldy, s);
    else if (kind == 2) uks->matmul(c, X, ldx, k, Y, ldy, s);
    else dense->matmul(X, ldx, k, Y, ldy, s);
  }
  void diagonal(const vgb::Coef &c, double *D, cudaStream_t s) {
    if (kind == 0) bse->diagonal(c, D, s);
    else if (kind == 2) uks->diagonal(c, D, s);
    else dense->diagonal(D, s);
  }
  void check_errors(cudaStream_t s) {
    if (kind == 0) bse->check_errors(s);
    else if (kind == 2) uks->check_errors(s);
    else dense->ws.check();
  }
};
