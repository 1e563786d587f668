// Legendre stage of a batch as FP32 products (kernels/leg_gemm.cuh): the
// tables and the launchers.
#include "kernels/leg_gemm.cuh"
#include "runtime.h"

namespace {

int lg_k16(int lmax, int m, int par) { return (((lmax - m + 2 - par) >> 1) + 15) & ~15; }
int lg_nhp(ts_plan p) { return (p->nh + TS_LG_ROWS - 1) / TS_LG_ROWS * TS_LG_ROWS; }

// floats of one direction's table, and its bytes with the onsets
size_t lg_floats(ts_plan p) { return (size_t)ts_lg_off(p->lmax, p->mmax + 1) * lg_nhp(p); }
size_t lg_bytes(ts_plan p) {
  return sizeof(float) * lg_floats(p) + sizeof(int) * (size_t)(p->mmax + 1) * lg_nhp(p);
}
bool lg_fits(ts_plan p) {
  if (p->precision == TS_PREC_FP32) return p->lmax <= 2047 && lg_bytes(p) <= (size_t)512 << 20;
  return p->lmax <= 1535 && lg_bytes(p) <= (size_t)2 << 30;
}

// the plan's table, made by the first call that wants it on a tensor-core plan
// (whose large batches never do): false when there is none and it cannot be
// made now, because the stream is being captured or memory is short
bool lg_ready(ts_plan p, cudaStream_t s) {
  if (p->lg_tab) return true;
  if (p->precision == TS_PREC_FP32) return false;
  if (ts_capturing(s)) return false;
  ts_lg_init(p, s);
  if (p->lg_tab) TS_CUDA(cudaStreamSynchronize(s));  // later calls may come on other streams
  return p->lg_tab != nullptr;
}

// columns of a tile (2 per field) with the least work for nf fields in whole
// instances of na: a tile of fewer columns re-reads more table values per
// multiply-add
int lg_ncol(int nf, int na) {
  static const struct {
    int ncol;
    double cost;
  } shapes[] = {{64, 64.}, {32, 40.}, {16, 26.}};
  int best = 64;
  double least = 1e30;
  for (auto &s : shapes) {
    const int per_cta = na * (s.ncol / 2 / na);
    if (!per_cta) continue;
    const double c = (double)((nf + per_cta - 1) / per_cta) * s.cost;
    if (c < least) {
      least = c;
      best = s.ncol;
    }
  }
  return best;
}

template <int NCOL>
void synth_t(ts_plan p, const TsLegGemmTab &g, const TsFields &q, float2 *fm, long fs, int nf,
             cudaStream_t s) {
  using S = TsLg<NCOL>;
  ts_allow_smem((const void *)ts_leg_synth_gemm<NCOL>, p->ctx->device, S::SYN_SMEM);
  dim3 grid(g.nhp / TS_LG_ROWS, (nf + S::NF - 1) / S::NF, p->mmax + 1);
  ts_launch(ts_early(p, nf), ts_leg_synth_gemm<NCOL>, grid, TS_LG_THREADS, S::SYN_SMEM, s, p->leg, g, q, fm, fs, nf);
}

template <int NCOL>
void analys_t(ts_plan p, const TsLegGemmTab &g, const float2 *gm, long gs, const TsLgStore &out,
              int nf, cudaStream_t s) {
  using S = TsLg<NCOL>;
  const auto kernel = ts_leg_analys_gemm<NCOL, TsLgStore>;
  ts_allow_smem((const void *)kernel, p->ctx->device, S::ANA_SMEM);
  dim3 grid((p->lmax + 2 * TS_LG_ROWS) / (2 * TS_LG_ROWS), (nf + S::NF - 1) / S::NF, p->mmax + 1);
  ts_launch(ts_early(p, nf), kernel, grid, TS_LG_THREADS, S::ANA_SMEM, s, p->leg, g, gm, gs, out, nf, (int)S::NF);
}

template <int F>
void synth_few(ts_plan p, const TsLegGemmTab &g, const TsFields &q, float2 *fm, long fs, int nf,
               cudaStream_t s) {
  const size_t smem = sizeof(float2) * (size_t)(p->lmax + 1) * F;
  ts_allow_smem((const void *)ts_leg_synth_few<F>, p->ctx->device, smem);
  ts_launch(ts_early(p, nf), ts_leg_synth_few<F>, dim3(g.nhp / TS_LG_ROWS, p->mmax + 1), 256, smem, s, p->leg, g, q, fm, fs, nf);
}

size_t few_smem(ts_plan p, int F) { return sizeof(float2) * F * (2 * (size_t)p->nh + 16 * TS_LG_ROWS); }

template <int F>
void analys_few(ts_plan p, const TsLegGemmTab &g, const float2 *gm, long gs, const TsLgStore &out,
                int nf, cudaStream_t s) {
  const auto kernel = ts_leg_analys_few<F, TsLgStore>;
  ts_allow_smem((const void *)kernel, p->ctx->device, few_smem(p, F));
  dim3 grid((p->lmax + 2 * TS_LG_ROWS) / (2 * TS_LG_ROWS), p->mmax + 1);
  ts_launch(ts_early(p, nf), kernel, grid, 512, few_smem(p, F), s, p->leg, g, gm, gs, out, nf);
}

// One or two fields take the kernels without staging (us, tiled | these, lmax
// 255: synthesis 1 field 12.5 | 9.2, 2: 12.6 | 10.5, 4: 12.5 | 12.7; analysis 1:
// 16.8 | 10.4, 2: 16.8 | 10.5, 4: 17.4 | 14.7; lmax 1023, whole transforms:
// synthesis 1: 343 | 222, 4: 389 | 426; analysis 1: 382 | 252, 4: 425 | 486).
// Their analysis holds the columns of every latitude in shared memory: up to
// some 13500 latitudes for two fields and 28000 for one.
bool lg_few(int nf) { return nf <= 2; }
bool lg_few_analys(ts_plan p, int nf) {
  return lg_few(nf) && few_smem(p, nf) + 64 <= p->ctx->smem_optin;  // (64: the static part)
}

}  // namespace

// Which calls take the products.  On B200 (us, recurrence kernel | product):
//   synthesis  lmax 31: 1 field 6.9 | 7.1, 8: 8.5 | 6.9;  lmax 63: 1: 8.1 | 4.7;  lmax 255: 1: 20.6 | 12.6,
//              8: 33 | 12.5, 256: 365 | 154;  lmax 511: 1: 41 | 54, 2: 45 | 54, 3: 73 | 54, 8: 113 | 57
//   analysis   lmax 31: 1: 6.6 | 7.2, 8: 9.0 | 7.4;  lmax 63: 1: 8.6 | 6.5;  lmax 255: 1: 47 | 16.7,
//              256: 742 | 181;  lmax 511: 1: 107 | 65, 8: 162 | 72
// so all but a few fields on the smallest grids (a table under 384 KB), and
// one or two fields' synthesis where the table comes from HBM (over 64 MB).
// Above 512 MB a direction the tables are not made, nor above lmax 2047 (the
// recurrence coefficients of an order are held in shared memory).
//
// On tensor-core plans the contraction works in blocks of 64 fields, so a small
// batch is mostly padding there; the products read half the table bytes and
// round the table once (error against 64 bits at lmax 511: 4.4e-7, contraction
// 4.9e-6).  Whole transforms (us, contraction | products; 3/2 grids):
//   synthesis  lmax 63: 1 field 19.3 | 12.2, 64: 21.6 | 13.6;  lmax 127: 1: 24.8 | 12.4, 64: 32 | 27.5;
//              lmax 255: 1: 42 | 18.7, 16: 51 | 28, 48: 67 | 61, 64: 76 | 76;  lmax 511: 1: 148 | 63,
//              32: 241 | 225, 48: 287 | 343;  lmax 1023: 1: 759 | 343, 16: 961 | 660, 24: 1064 | 1132
//   analysis   lmax 63: 1: 13.2 | 12.4, 48: 16.5 | 12.8;  lmax 127: 1: 18.7 | 12.9, 16: 18.7 | 17.1,
//              24: 19.7 | 22.8;  lmax 255: 1: 35 | 24, 16: 43 | 35, 24: 48 | 55;  lmax 1023: 16: 869 | 677,
//              24: 966 | 1195
// so the line lies at 16 fields, or for the synthesis at 48 where the table
// stays in the L2 and 32 up to 256 MB, and for the smallest analyses at 48.
// No tables above 2 GB a direction or lmax 1535.  The two directions' are made
// together by the first call that wants either (3.3 GB at lmax 1023 x 1536),
// and a plan that has no memory for them then stays with the contraction.
//
// Not in a model's forward_backward: a parameter's gradient can be a difference
// of large terms (the derivative to dt sums the rate of change, A - (B + 1) u +
// u u v at a Brusselator's steady state), so the contraction's 1e-6 is up to
// 4e-4 of it (lmax 235), and the gradient of an instance would change by as much
// with the number of instances beside it.  Even the rounding of a step's
// statements, compiled otherwise, is 6e-5 (lmax 127): its forward steps are the
// same kernels whatever the batch.
int ts_lg_most_analys(ts_plan p) { return lg_bytes(p) < (size_t)2 << 20 ? 48 : 16; }

bool ts_lg_use(ts_plan p, int nf, bool analysis) {
  const size_t bytes = lg_bytes(p);
  if (p->lg_none || !lg_fits(p)) return false;
  if (p->precision != TS_PREC_FP32) {
    // the adjoint of a model takes the contraction whatever the batch; the test
    // hook is about the tensor-core kernels
    if (p->in_adjoint || ts_tc_stalled(p)) return false;
    if (analysis) return nf <= ts_lg_most_analys(p);
    return nf <= (bytes <= (size_t)64 << 20 ? 48 : bytes <= (size_t)256 << 20 ? 32 : 16);
  }
  if (bytes < (size_t)384 << 10) return nf >= 8;
  return analysis || nf >= 3 || bytes <= (size_t)64 << 20;
}

void ts_lg_init(ts_plan p, cudaStream_t s) {
  if (!lg_fits(p)) return;
  const size_t n = lg_floats(p), no = (size_t)(p->mmax + 1) * lg_nhp(p);
  float *tab = nullptr;
  const cudaError_t e = cudaMalloc(&tab, 2 * sizeof(float) * n + sizeof(int) * no);
  if (e != cudaSuccess) {
    (void)cudaGetLastError();
    p->lg_none = e == cudaErrorMemoryAllocation;
    return;
  }
  int *onset = (int *)(tab + 2 * n);
  const int nhp = lg_nhp(p), pairs = 2 * lg_k16(p->lmax, 0, 0) + 4;
  const dim3 grid(nhp / 64, p->mmax + 1);
  try {
    if (p->precision == TS_PREC_FP32) {
      const size_t smem = sizeof(float2) * pairs;
      ts_leg_ptab_f32<false><<<grid, 64, smem, s>>>(p->leg, nhp, tab, onset);
      TS_CUDA(cudaGetLastError());
      ts_leg_ptab_f32<true><<<grid, 64, smem, s>>>(p->leg, nhp, tab + n, onset);
    } else {
      const size_t smem = sizeof(double2) * pairs;
      ts_leg_ptab_f64<false><<<grid, 64, smem, s>>>(p->d_x64, p->d_ab64, p->d_amm64, p->lmax, p->nh, nhp,
                                                    tab, onset);
      TS_CUDA(cudaGetLastError());
      ts_leg_ptab_f64<true><<<grid, 64, smem, s>>>(p->d_x64, p->d_ab64, p->d_amm64, p->lmax, p->nh, nhp,
                                                   tab + n, onset);
    }
    TS_CUDA(cudaGetLastError());
  } catch (...) {  // a table that is not written is no table
    cudaFree(tab);
    throw;
  }
  p->lg_tab = tab;
  p->lg_syn = TsLegGemmTab{tab, onset, nhp};
  p->lg_ana = TsLegGemmTab{tab + n, onset, nhp};
}

bool ts_launch_leg_synth_gemm(ts_plan p, const TsFields &q, float2 *fm, long fs, int nf,
                              cudaStream_t s) {
  if (!ts_lg_use(p, nf, false) || !lg_ready(p, s)) return false;
  const TsLegGemmTab &g = p->lg_syn;
  if (lg_few(nf))
    nf == 1 ? synth_few<1>(p, g, q, fm, fs, nf, s) : synth_few<2>(p, g, q, fm, fs, nf, s);
  else switch (lg_ncol(nf, 1)) {
    case 64: synth_t<64>(p, g, q, fm, fs, nf, s); break;
    case 32: synth_t<32>(p, g, q, fm, fs, nf, s); break;
    default: synth_t<16>(p, g, q, fm, fs, nf, s); break;
  }
  TS_CUDA(cudaGetLastError());
  return true;
}

bool ts_launch_leg_analys_gemm(ts_plan p, const float2 *gm, long gs, float2 *out, long os, int nf,
                               cudaStream_t s) {
  if (!ts_lg_use(p, nf, true) || !lg_ready(p, s)) return false;
  const TsLegGemmTab &g = p->lg_ana;
  TsLgStore st{};
  st.base[0] = out;
  st.inst_stride[0] = os;
  st.nper = 1;
  if (lg_few_analys(p, nf))
    nf == 1 ? analys_few<1>(p, g, gm, gs, st, nf, s) : analys_few<2>(p, g, gm, gs, st, nf, s);
  else switch (lg_ncol(nf, 1)) {
    case 64: analys_t<64>(p, g, gm, gs, st, nf, s); break;
    case 32: analys_t<32>(p, g, gm, gs, st, nf, s); break;
    default: analys_t<16>(p, g, gm, gs, st, nf, s); break;
  }
  TS_CUDA(cudaGetLastError());
  return true;
}

bool ts_lg_prepare(ts_plan p, cudaStream_t s) { return lg_ready(p, s); }

void ts_lg_analys_shape(ts_plan p, int nf, int na, TsLgShape *sh) {
  const unsigned chunks = (p->lmax + 2 * TS_LG_ROWS) / (2 * TS_LG_ROWS), M = p->mmax + 1;
  if (lg_few_analys(p, nf)) {
    sh->few = nf;
    sh->per_cta = nf;
    sh->threads = 512;
    sh->smem = few_smem(p, nf);
    sh->grid[0] = chunks;
    sh->grid[1] = M;
    sh->grid[2] = 1;
    return;
  }
  sh->ncol = lg_ncol(nf, na);
  sh->per_cta = na * (sh->ncol / 2 / na);
  sh->threads = TS_LG_THREADS;
  sh->smem = sh->ncol == 64 ? TsLg<64>::ANA_SMEM : sh->ncol == 32 ? TsLg<32>::ANA_SMEM : TsLg<16>::ANA_SMEM;
  sh->grid[0] = chunks;
  sh->grid[1] = (nf + sh->per_cta - 1) / sh->per_cta;
  sh->grid[2] = M;
}
