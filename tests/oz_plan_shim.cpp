// C entry of the digit-product plan for tests/test_oz_plan.py: runs a strided batched GEMM through
// the plan's maps, K splits and chunks on the CPU, and by the plain loops.
#include <cstdlib>

#include "../votca_gb300/csrc/oz_plan.hpp"

using vgb::GemmDesc;
using vgb::OzPlan;

static void loops(const GemmDesc &d) {
  for (int64_t b1 = 0; b1 < d.nb1; ++b1)
    for (int64_t b2 = 0; b2 < d.nb2; ++b2)
      for (int64_t i = 0; i < d.M; ++i)
        for (int64_t n = 0; n < d.N; ++n) {
          double s = 0.0;
          for (int64_t k = 0; k < d.K; ++k)
            s += d.A[b1 * d.a_b1 + b2 * d.a_b2 + i * d.a_rs + k * d.a_cs] *
                 d.B[b1 * d.b_b1 + b2 * d.b_b2 + k * d.b_rs + n * d.b_cs];
          double *c = d.C + b1 * d.c_b1 + b2 * d.c_b2 + i * d.c_rs + n * d.c_cs;
          *c = d.alpha * s + d.beta * *c;
        }
}

// the chunk, batch, split and tile walk of oz_dgemm; counts[offset] += 1 per output written
static void planned(const GemmDesc &d, const OzPlan &q, int32_t *counts) {
  for (int64_t t0 = 0; t0 < q.nbatch; t0 += q.tb_chunk)
    for (int64_t m0 = 0; m0 < q.M; m0 += q.m_chunk) {
      const int64_t tn = std::min(q.tb_chunk, q.nbatch - t0), mn = std::min(q.m_chunk, q.M - m0);
      for (int64_t b = 0; b < tn; ++b)
        for (int64_t i = 0; i < (q.nbatch > 1 ? q.M : mn); ++i)
          for (int64_t n = 0; n < q.N; ++n) {
            double s = 0.0;
            for (int sp = 0; sp < q.splits; ++sp) {
              const int64_t k0 = (int64_t)sp * q.kb_per * vgb::kOzStageK;
              const int64_t k1 = std::min(d.K, k0 + (int64_t)q.kb_per * vgb::kOzStageK);
              for (int64_t k = k0; k < k1; ++k)
                s += q.A[q.amap.at(t0 * q.M + m0 + b * q.M + i) + k * q.ka] *
                     q.B[q.bmap.at(t0 * q.N + b * q.N + n) + k * q.kb];
            }
            const int64_t off = q.cbatch.at(t0 + b) + q.crow.at(m0 + i) + q.ccol.at(n);
            d.C[off] = d.alpha * s + d.beta * d.C[off];
            counts[off] += 1;
          }
    }
}

extern "C" int oz_plan_run(const int64_t *v, const double *A, const double *B, double *C, double *C2, double alpha,
                           double beta, int64_t sms, int64_t budget, int32_t *counts, int64_t *out) {
  GemmDesc d;
  d.M = v[0]; d.N = v[1]; d.K = v[2]; d.nb1 = v[3]; d.nb2 = v[4];
  d.a_rs = v[5]; d.a_cs = v[6]; d.a_b1 = v[7]; d.a_b2 = v[8];
  d.b_rs = v[9]; d.b_cs = v[10]; d.b_b1 = v[11]; d.b_b2 = v[12];
  d.c_rs = v[13]; d.c_cs = v[14]; d.c_b1 = v[15]; d.c_b2 = v[16];
  d.A = A; d.B = B; d.C = C; d.alpha = alpha; d.beta = beta;
  OzPlan q;
  if (!vgb::oz_plan(d, (int)sms, budget, q)) return 0;
  planned(d, q, counts);
  d.C = C2;
  loops(d);
  out[0] = q.splits; out[1] = q.m_chunk; out[2] = q.tb_chunk; out[3] = q.M; out[4] = q.N; out[5] = q.nbatch;
  out[6] = q.kb_per; out[7] = q.nkb; out[8] = q.faster;
  return 1;
}

// the FMA plan: tile, splits, K elements per split, and the fixed split rule
extern "C" void fma_plan_of(const int64_t *v, int64_t sms, int32_t splitk, int64_t *out) {
  GemmDesc d;
  d.M = v[0]; d.N = v[1]; d.K = v[2]; d.nb1 = v[3];
  const vgb::FmaPlan f = vgb::fma_plan(d, (int)sms, splitk);
  out[0] = f.tm; out[1] = f.tn; out[2] = f.splits; out[3] = f.kchunk; out[4] = vgb::fma_chain_splits(d, (int)sms);
}
