// C entries into the C++ core for tests that the C ABI does not reach: error codes planted on the host
// in place of a device wait that gave up, single FP64 products, the memory pools, and the small dense
// solvers in both of their forms, and single slice products.
#include <string>

#include "../votca_gb300/csrc/davidson.cuh"
#include "../votca_gb300/csrc/handle.cuh"
#include "../votca_gb300/csrc/oz_gemm.cuh"
#include "../votca_gb300/csrc/slice_gemm.cuh"
#include "../votca_gb300/csrc/small_eig.cuh"
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

template <class T>
struct Dev : vgb::DeviceBuffer<T> {
  cudaStream_t s;
  Dev(const T *h, int64_t n, cudaStream_t s_) : vgb::DeviceBuffer<T>((size_t)n), s(s_) {
    if (h) VGB_CUDA(cudaMemcpyAsync(this->get(), h, n * sizeof(T), cudaMemcpyHostToDevice, s));
    else VGB_CUDA(cudaMemsetAsync(this->get(), 0, n * sizeof(T), s));
  }
  void read(T *h, int64_t n) {
    VGB_CUDA(cudaMemcpyAsync(h, this->get(), n * sizeof(T), cudaMemcpyDeviceToHost, s));
    VGB_CUDA(cudaStreamSynchronize(s));
  }
};

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

// A strided batched product on the tensor-core path; d: M, N, K, nb1, nb2, a_rs, a_cs, a_b1, a_b2,
// b_rs, b_cs, b_b1, b_b2, c_rs, c_cs, c_b1, c_b2; wait_us: the limit of its waits; *taken: whether that
// path took it; *keep: bytes the workspace holds afterwards.
int shim_oz_dgemm(const int64_t *v, const double *A, int64_t na, const double *B, int64_t nb, double *C, int64_t nc,
                  double alpha, double beta, int64_t budget, int wait_us, int *taken, int64_t *keep) {
  return on_stream([&](cudaStream_t s) {
    Dev<double> a(A, na, s), b(B, nb, s), c(C, nc, s);
    vgb::GemmWorkspace ws;
    ws.plane_budget = budget;
    ws.wait_us = wait_us;
    vgb::GemmDesc d;
    d.M = v[0]; d.N = v[1]; d.K = v[2]; d.nb1 = v[3]; d.nb2 = v[4];
    d.A = a.get(); d.a_rs = v[5]; d.a_cs = v[6]; d.a_b1 = v[7]; d.a_b2 = v[8];
    d.B = b.get(); d.b_rs = v[9]; d.b_cs = v[10]; d.b_b1 = v[11]; d.b_b2 = v[12];
    d.C = c.get(); d.c_rs = v[13]; d.c_cs = v[14]; d.c_b1 = v[15]; d.c_b2 = v[16];
    d.alpha = alpha; d.beta = beta;
    *taken = vgb::oz_dgemm(d, s, &ws) ? 1 : 0;
    c.read(C, nc);
    ws.check();
    *keep = (int64_t)(ws.oz_a.bytes() + ws.oz_b.bytes() + ws.oz_int.bytes());
  });
}

// A product whose digit planes no GPU can hold: nothing is launched, *keep: bytes left in the workspace.
int shim_oz_no_room(int *taken, int64_t *keep) {
  return on_stream([&](cudaStream_t s) {
    vgb::GemmWorkspace ws;
    ws.plane_budget = 1LL << 50;
    vgb::GemmDesc d;  // planes of A: 2^26 x 512 x 14 bytes
    d.M = 1LL << 26; d.N = 64; d.K = 512;
    d.a_colmajor(nullptr, d.M, false).b_colmajor(nullptr, d.K, false).c_colmajor(nullptr, d.M);
    *taken = vgb::oz_dgemm(d, s, &ws) ? 1 : 0;
    *keep = (int64_t)(ws.oz_a.bytes() + ws.oz_b.bytes() + ws.oz_int.bytes() + ws.partial.bytes());
  });
}

// The default memory pool: reserved bytes, and its release threshold.
int shim_pool_state(uint64_t *reserved, uint64_t *threshold) {
  return guarded([&] {
    int dev = 0;
    cudaMemPool_t p;
    VGB_CUDA(cudaGetDevice(&dev));
    VGB_CUDA(cudaDeviceGetDefaultMemPool(&p, dev));
    VGB_CUDA(cudaMemPoolGetAttribute(p, cudaMemPoolAttrReservedMemCurrent, reserved));
    VGB_CUDA(cudaMemPoolGetAttribute(p, cudaMemPoolAttrReleaseThreshold, threshold));
  });
}

// What a handle keeps (used) and has given back to the pool (unused).
static vgb::DeviceBuffer<char> *g_used = nullptr;
int shim_pool_hold(int64_t used, int64_t unused) {
  return on_stream([&](cudaStream_t) {
    g_used = new vgb::DeviceBuffer<char>((size_t)used);
    vgb::DeviceBuffer<char> tmp((size_t)unused);
  });
}
int shim_pool_release() {
  return on_stream([&](cudaStream_t) {
    delete g_used;
    g_used = nullptr;
  });
}

// Cholesky QR of a Gram matrix.
int shim_cholqr(const double *G, int nb, const double *norms0, int check, int fast, double *Rinv, int *ok, int *flag) {
  return on_stream([&](cudaStream_t s) {
    Dev<double> g(G, nb * nb, s), n0(norms0, nb, s), r(nullptr, nb * nb, s);
    Dev<int> o(nullptr, 2, s);
    vgb::cholqr(g.get(), nb, r.get(), n0.get(), check != 0, o.get(), o.get() + 1, fast != 0, s);
    int h[2];
    o.read(h, 2);
    r.read(Rinv, nb * nb);
    *ok = h[0];
    *flag = h[1];
  });
}

// One symmetric eigenproblem (m x m, nw lowest pairs).
int shim_sym_eig(const double *T, int64_t m, int64_t nw, int fast, double *lam, double *U) {
  return on_stream([&](cudaStream_t s) {
    Dev<double> t(T, m * m, s), l(nullptr, nw, s), u(nullptr, m * nw, s), w(nullptr, vgb::sym_eig_work_doubles(m, nw), s);
    Dev<int> info(nullptr, 1, s);
    vgb::SymEigJob j;
    j.T = t.get(); j.ldt = m; j.m = m; j.nw = nw; j.U = u.get(); j.ldu = m; j.lam = l.get();
    j.work = w.get(); j.info = info.get(); j.fast = fast != 0;
    vgb::sym_eig_device(&j, 1, s);
    int st = 0;
    info.read(&st, 1);
    if (st) vgb::fail(BSE_ERR_NUMERICAL, "sym_eig");
    l.read(lam, nw);
    u.read(U, m * nw);
  });
}

// One harmonic-Ritz problem.
int shim_gen_eig(const double *T, const double *B, int64_t m, int64_t nw, int fast, double *lam, double *U,
                 int *selected) {
  return on_stream([&](cudaStream_t s) {
    Dev<double> t(T, m * m, s), b(B, m * m, s), l(nullptr, nw, s), u(nullptr, m * nw, s),
        w(nullptr, vgb::gen_eig_work_doubles(m, nw), s);
    Dev<int> info(nullptr, 2, s);
    vgb::GenEigJob j;
    j.T = t.get(); j.B = b.get(); j.ldt = m; j.m = m; j.nw = nw; j.U = u.get(); j.ldu = m; j.lam = l.get();
    j.work = w.get(); j.info = info.get(); j.fast = fast != 0;
    vgb::gen_eig_device(&j, 1, s);
    int st[2];
    info.read(st, 2);
    if (st[0]) vgb::fail(BSE_ERR_NUMERICAL, "gen_eig " + std::to_string(st[0]));
    *selected = st[1];
    l.read(lam, nw);
    u.read(U, m * nw);
  });
}

// C (M x N, column-major) = A B^T for A (M x K) and B (N x K), rows contiguous, as one slice product.
int shim_slice_gemm(const double *A, const double *B, int64_t M, int64_t N, int64_t K, int64_t chain, double *C) {
  return on_stream([&](cudaStream_t s) {
    constexpr int S = 5;
    Dev<double> a(A, M * K, s), b(B, N * K, s), c(nullptr, M * N, s);
    Dev<uint16_t> pa(nullptr, S * M * K, s), pb(nullptr, S * N * K, s);
    Dev<int> err(nullptr, 1, s);
    vgb::SplitMap m;
    m.rdiv = 1; m.rs1 = K; m.rs2 = 0; m.cs = 1; m.rlim = 1;
    vgb::slice_f64(a.get(), M, K, m, S, chain, pa.get(), K, M * K, s);
    vgb::slice_f64(b.get(), N, K, m, S, chain, pb.get(), K, N * K, s);
    vgb::TcEpilogue e;
    e.kind = vgb::TcEpilogue::AXPBY_F64;
    e.rd = M; e.ro2 = 1; e.rlim = M;
    e.cd = N; e.co2 = M; e.clim = N;
    e.out_f64 = c.get(); e.alpha = 1.0; e.beta = 0.0;
    vgb::DeviceBuffer<double> gpart;
    vgb::slice_gemm(vgb::SliceMat{pa.get(), K, M, 0}, vgb::SliceMat{pb.get(), K, N, 0}, M, N, K, chain, S, e, gpart,
                    err.get(), s);
    c.read(C, M * N);
  });
}

// A^-1 of a positive definite matrix with the factor in place of A's lower triangle.
int shim_cholesky_inverse_in_place(int64_t n, const double *A, double *inv) {
  return on_stream([&](cudaStream_t s) { vgb::cholesky_inverse(n, A, n, inv, n, s, true); });
}

}  // extern "C"
