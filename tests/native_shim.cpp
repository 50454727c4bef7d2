// C entries into the C++ core for tests that the C ABI does not reach: error codes planted on the host
// in place of a device wait that gave up.
#include <string>

#include "../votca_gb300/csrc/handle.cuh"
#include "../votca_gb300/csrc/tc_engine.cuh"

namespace {

thread_local std::string g_error;

template <class F>
int guarded(F &&f) {
  try {
    f();
    return BSE_OK;
  } catch (const vgb::Error &e) {
    g_error = e.what();
    return e.code;
  }
}

// f(stream) with device buffers on that stream.
template <class F>
int on_stream(F &&f) {
  return guarded([&] {
    cudaStream_t s;
    VGB_CUDA(cudaStreamCreate(&s));
    {
      vgb::AllocStreamScope scope(s);
      try {
        f(s);
      } catch (...) {
        cudaStreamSynchronize(s);
        throw;
      }
    }
    VGB_CUDA(cudaStreamSynchronize(s));
    cudaStreamDestroy(s);
  });
}

}  // namespace

extern "C" {

const char *shim_last_error() { return g_error.c_str(); }

// The code a kernel of the handle's FP64 products would leave when a bounded wait gives up.
void shim_plant_error(bse_handle *h, int code) {
  vgb::GemmWorkspace &ws = h->kind == 0 ? h->bse->ws : h->kind == 1 ? h->dense->ws : h->uks->alpha.ws;
  *ws.error_slot() = code;
}

// The same for the handle's split-precision engine.
int shim_plant_engine_error(bse_handle *h, int code) {
  return guarded([&] {
    VGB_CUDA(cudaMemcpy(h->bse->mixed->error_flag(), &code, sizeof(int), cudaMemcpyHostToDevice));
  });
}

// Staging with a dense screening after such a code.
int shim_stage_dense_screening(const bse_mmn_desc *d, const double *const *slices, const double *w,
                               const double *hqp, int64_t nh, const bse_options *opt, int code) {
  return on_stream([&](cudaStream_t s) {
    vgb::BseOperator op;
    *op.ws.error_slot() = code;
    op.stage(*d, slices, w, true, hqp, nh, nh, *opt, BSE_PRECISION_FP64, s);
  });
}

// The same for an unrestricted operator with this Mmn in both spins, the code in its cross-spin products.
int shim_stage_dense_screening_uks(const bse_mmn_desc *d, const double *const *slices, const double *w,
                                   const double *hqp, int64_t nh, const bse_options *opt, int code) {
  return on_stream([&](cudaStream_t s) {
    vgb::UksOperator op;
    *op.workspace().error_slot() = code;
    const bse_uks_options o = {opt->homo, opt->homo, opt->rpamin, opt->qpmin, opt->vmin, opt->cmax};
    op.stage(*d, slices, *d, slices, w, true, hqp, nh, nh, hqp, nh, nh, o, BSE_PRECISION_FP64, s);
  });
}

}  // extern "C"
