// Legendre stage of a batch as FP32 register-blocked products with a table of
// Legendre values in memory:
//   synthesis  F_par[lat, c] = sum_j P_par[j, lat] Q_par[j, c],   north = F_0 + F_1, south = F_0 - F_1
//   analysis   Q_par[j, c]   = sum_lat P_par[lat, j] W_par[lat, c], W_0, W_1 = (G_north +- G_south) w
// for one order m, degrees l = m + 2j + par, real columns c = 2 field + re|im.
// The table, written once per plan, holds what the on-the-fly recurrence of
// leg_f32.cuh gives or, for the small batches of a tensor-core plan, the FP64
// functions rounded to FP32.  The recurrence kernels spend most of their
// time on 8-byte shared loads per two multiply-adds (synthesis) and on a
// shuffle reduction per pair of degrees (analysis); these are bound by the
// FP32 pipe.  At lmax 255 (384 latitudes), 256 fields: synthesis 364 -> 154
// us, analysis 744 -> 181 us, of 94 at the FP32 pipe's measured 120
// multiply-adds per clock and SM; the rest is the padding to 16 degrees, the
// coefficients' and latitudes' way through shared memory, and the ends of
// short orders.
//
// A CTA of 4 warps owns up to 64 rows of each parity (latitudes or degrees)
// and NCOL columns; a warp holds up to 32 rows of one parity, a lane 2 NP rows
// by CT = NCOL / 8 columns.  Rows are packed in pairs (fma.rn.f32x2): one
// instruction for two multiply-adds leaves issue slots to the loads (a k-step
// of 8 x 8 values alone: 110 of 120 multiply-adds per clock and SM, 100 with
// scalar instructions).  Four CTAs an SM, so that one's loads and stores
// overlap the products of the others.
#pragma once
#include "ts_common.cuh"

#define TS_LG_ROWS 64     // rows (latitudes or degrees) of a parity per CTA
#define TS_LG_KT 16       // k-steps per shared-memory stage
#define TS_LG_THREADS 128
// k-steps unrolled in the full-size loop: the whole stage, half of it where the
// kernel is compiled with a model (2 % slower, half the compile time)
#ifdef __CUDACC_RTC__
#define TS_LG_UNROLL 8
#else
#define TS_LG_UNROLL TS_LG_KT
#endif

// Geometry of a table (TsLegGemmTab): of order m, parity 0 has ts_lg_k16(m, 0) rows of
// degrees (a multiple of 16; zeros from the parity's count on), then parity 1;
// ts_lg_off(lmax, m) degree rows lie before it; nhp latitudes (a multiple of
// 64, zeros from nh on).  Synthesis layout [degree row][latitude], analysis
// layout [m][parity][latitude][degree].

TS_DEV int ts_lg_kpar(int lmax, int m, int par) { return (lmax - m + 2 - par) >> 1; }
TS_DEV int ts_lg_k16(int lmax, int m, int par) { return (ts_lg_kpar(lmax, m, par) + 15) & ~15; }
// degree rows (both parities) of all orders with up to n = 32 q + r degrees: an
// order of 32 q' + r' degrees (0 < r' <= 32) has 32 q' + 16, and 16 more from r' = 2 on
__host__ __device__ inline long ts_lg_rows(int n) {
  const long q = n >> 5, r = n & 31;
  return 512 * q * (q - 1) + 1008 * q + 32 * q * r + (r ? 32 * r - 16 : 0);
}
__host__ __device__ inline long ts_lg_off(int lmax, int m) {
  return ts_lg_rows(lmax + 1) - ts_lg_rows(lmax + 1 - m);
}

// one packed multiply-add: (a.x b.x + c.x, a.y b.y + c.y), each rounded once
TS_DEV void ts_fma2(float2 &c, float2 a, float2 b) {
  asm("fma.rn.f32x2 %0, %1, %2, %0;"
      : "+l"(reinterpret_cast<unsigned long long &>(c))
      : "l"(reinterpret_cast<unsigned long long &>(a)), "l"(reinterpret_cast<unsigned long long &>(b)));
}

TS_DEV void ts_lg_cp16(void *dst, const void *src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(
                   (unsigned)__cvta_generic_to_shared(dst)),
               "l"(src)
               : "memory");
}
// 8 bytes, or zeros when !live
TS_DEV void ts_lg_cp8(void *dst, const void *src, bool live) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;" ::"r"(
                   (unsigned)__cvta_generic_to_shared(dst)),
               "l"(src), "r"(live ? 8 : 0)
               : "memory");
}
TS_DEV void ts_lg_cp_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
// all but the latest N groups of copies of this thread have landed
template <int N>
TS_DEV void ts_lg_cp_wait() {
  asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}

// ------------------------------------------------------------------ tables
//
// One thread per order and latitude walks a recurrence over the degrees, 8
// pairs (l - m = 2j, 2j + 1) at a time; zeros in the padding.  onset is the
// first l - m with a value that is not zero (lmax + 1: none), so that the
// products can leave out what is zero near the poles.  The synthesis layout is
// written as it comes (16 degrees at a time, lanes on consecutive latitudes),
// the analysis layout by way of shared memory, 32 degrees of a parity as one
// 128-byte line of a latitude.
// grid = (nhp / 64, mmax + 1), 64 threads, 2 ts_lg_k16(lmax, 0, 0) + 4
// coefficient pairs of the recurrence's type in shared memory.

// The recurrence of ts_leg_synth_f32, its products and sums rounded as they are
// there (a synthesis by way of the table gives the same bits).  A value counts
// only once the running exponent is zero.  Coefficients past lmax are read as
// zeros, which ends the recurrence without a test; the rescaling tests run only
// while some latitude of the warp still carries an exponent.
struct TsLgRec32 {
  using Pair = float2;
  TsLegTab t;
  float ct, y0, y1;
  int ny, first;
  TS_DEV explicit TsLgRec32(const TsLegTab &t_) : t(t_) {}
  TS_DEV Pair coeff(long lm) const { return t.ab[lm]; }
  TS_DEV void init(int m, int lat, const Pair *sab) {
    const bool live = lat < t.nh;
    ct = live ? t.ct[lat] : 0.f;
    y0 = y1 = 0.f;
    ny = 0;
    first = live ? -1 : t.lmax + 1;
    if (live) {
      ts_sinpow(t.st[lat], m, y0, ny);
      y0 *= t.amm[m];
      y1 = sab[1].x * ct * y0;
    }
  }
  TS_DEV void advance(const Pair *sab, int i) {
    const float4 a = *reinterpret_cast<const float4 *>(sab + i + 2);
    const float t0 = fmaf(__fmul_rn(a.x, ct), y1, __fmul_rn(a.y, y0));
    y1 = fmaf(a.w, y1, __fmul_rn(__fmul_rn(a.z, ct), t0));
    y0 = t0;
  }
  TS_DEV void next8(const Pair *sab, int j0, float (&v)[2][8]) {
    if (__any_sync(0xffffffffu, first < 0)) {
#pragma unroll
      for (int u = 0; u < 8; u++) {
        const int i = 2 * (j0 + u);
        const bool on = ny == 0;
        if (on && first < 0) first = i;
        v[0][u] = on ? y0 : 0.f;
        v[1][u] = on ? y1 : 0.f;
        const bool up = !on && fabsf(y0) > TS_RESCALE_THR;
        const float f = up ? TS_INV_SCALE : 1.0f;
        ny += up ? 1 : 0;
        y0 *= f;
        y1 *= f;
        advance(sab, i);
      }
    } else {
#pragma unroll
      for (int u = 0; u < 8; u++) {
        v[0][u] = y0;
        v[1][u] = y1;
        advance(sab, 2 * (j0 + u));
      }
    }
  }
};

// The recurrence of the tensor-core tables in FP64 (a running pair scaled by
// powers of 2^500), each value rounded once to FP32; values below 1e-15 before
// the first larger one count as zero, as in the FP32 recurrence.
struct TsLgRec64 {
  using Pair = double2;
  const double *x, *ab, *amm;
  int lmax, nh;
  double ct, y0, y1;
  int e, first;
  TS_DEV TsLgRec64(const double *x_, const double *ab_, const double *amm_, int lmax_, int nh_)
      : x(x_), ab(ab_), amm(amm_), lmax(lmax_), nh(nh_) {}
  TS_DEV Pair coeff(long lm) const { return make_double2(ab[2 * lm], ab[2 * lm + 1]); }
  TS_DEV void init(int m, int lat, const Pair *sab) {
    const bool live = lat < nh;
    ct = live ? x[lat] : 0.0;
    first = live ? -1 : lmax + 1;
    e = 0;
    y0 = y1 = 0.0;
    if (!live) return;
    const double st = sqrt(1.0 - ct * ct);
    double y = 1.0;
    for (int i = 0; i < m; i++) {
      y *= st;
      if (y < 0x1p-500) {
        y *= 0x1p500;
        e -= 500;
      }
    }
    y0 = y * amm[m];
    y1 = sab[1].x * ct * y0;
  }
  TS_DEV float value(double y, int i) {
    const double p = e < -1100 ? 0.0 : e == 0 ? y : ldexp(y, e);
    if (first < 0 && fabs(p) >= 1e-15) first = i;
    return first < 0 ? 0.f : (float)p;
  }
  TS_DEV void next8(const Pair *sab, int j0, float (&v)[2][8]) {
#pragma unroll
    for (int u = 0; u < 8; u++) {
      const int i = 2 * (j0 + u);
      v[0][u] = value(y0, i);
      v[1][u] = value(y1, i + 1);
      const double2 a0 = sab[i + 2], a1 = sab[i + 3];
      y0 = a0.x * ct * y1 + a0.y * y0;
      y1 = a1.x * ct * y0 + a1.y * y1;
      if (fabs(y1) > 0x1p500) {
        y0 *= 0x1p-500;
        y1 *= 0x1p-500;
        e += 500;
      }
    }
  }
};

template <bool ANALYSIS, class Rec>
TS_DEV void ts_lg_table(Rec rec, int lmax, int nhp, float *__restrict__ tab, int *__restrict__ onset) {
  extern __shared__ __align__(16) char ts_smem_pt[];
  using Pair = typename Rec::Pair;
  constexpr int VP = 36;  // pitch: 16-byte rows, 8 lanes in distinct banks
  __shared__ __align__(16) float sv[ANALYSIS ? 2 * 64 * VP : 4];
  const int m = blockIdx.y, lat0 = blockIdx.x * 64, lat = lat0 + threadIdx.x;
  const int K = lmax - m + 1, k0 = ts_lg_k16(lmax, m, 0), k1 = ts_lg_k16(lmax, m, 1);
  const long base = ts_lm_base(lmax, m);
  Pair *sab = reinterpret_cast<Pair *>(ts_smem_pt);
  for (int i = threadIdx.x; i < 2 * k0 + 4; i += blockDim.x) sab[i] = i < K ? rec.coeff(base + i) : Pair{};
  __syncthreads();
  rec.init(m, lat, sab);
  float *mt = tab + ts_lg_off(lmax, m) * nhp;
  for (int j0 = 0; j0 < k0; j0 += 8) {
    float v[2][8];
    rec.next8(sab, j0, v);
    if constexpr (ANALYSIS) {
#pragma unroll
      for (int par = 0; par < 2; par++) {
        float4 *dst = reinterpret_cast<float4 *>(sv + (par * 64 + threadIdx.x) * VP + (j0 & 31));
        dst[0] = make_float4(v[par][0], v[par][1], v[par][2], v[par][3]);
        dst[1] = make_float4(v[par][4], v[par][5], v[par][6], v[par][7]);
      }
      if ((j0 & 31) == 24 || j0 + 8 >= k0) {
        __syncthreads();
        const int jj = (j0 & ~31) + 4 * (threadIdx.x & 7), r0 = threadIdx.x >> 3;
#pragma unroll
        for (int par = 0; par < 2; par++) {
          const int kp = par ? k1 : k0;
          float *dst = mt + (par ? (long)k0 * nhp : 0) + jj;
          if (jj < kp)
#pragma unroll
            for (int u = 0; u < 8; u++)
              *reinterpret_cast<float4 *>(dst + (long)(lat0 + r0 + 8 * u) * kp) =
                  *reinterpret_cast<const float4 *>(sv + (par * 64 + r0 + 8 * u) * VP + (jj & 31));
        }
        __syncthreads();
      }
    } else {
#pragma unroll
      for (int par = 0; par < 2; par++) {
        if (j0 >= (par ? k1 : k0)) continue;
        float *dst = mt + (long)((par ? k0 : 0) + j0) * nhp + lat;
#pragma unroll
        for (int u = 0; u < 8; u++) dst[(long)u * nhp] = v[par][u];
      }
    }
  }
  onset[(long)m * nhp + lat] = rec.first < 0 ? lmax + 1 : rec.first;
}

template <bool ANALYSIS>
__global__ void __launch_bounds__(64)
ts_leg_ptab_f32(TsLegTab t, int nhp, float *__restrict__ tab, int *__restrict__ onset) {
  ts_lg_table<ANALYSIS>(TsLgRec32(t), t.lmax, nhp, tab, onset);
}

template <bool ANALYSIS>
__global__ void __launch_bounds__(64)
ts_leg_ptab_f64(const double *x, const double *ab, const double *amm, int lmax, int nh, int nhp,
                float *__restrict__ tab, int *__restrict__ onset) {
  ts_lg_table<ANALYSIS>(TsLgRec64(x, ab, amm, lmax, nh), lmax, nhp, tab, onset);
}

// ------------------------------------------------------------ shared parts

template <int V>
struct TsLgInt {
  static constexpr int value = V;
};

template <int NCOL>
struct TsLg {
  static constexpr int CT = NCOL / 8;        // columns per lane: 8 lanes along columns, 4 along rows
  static constexpr int NF = NCOL / 2;        // fields
  static constexpr int A = 2 * TS_LG_KT * TS_LG_ROWS;  // floats of a stage's table values
  // synthesis: a stage's coefficients [field][2 KT degrees] (an odd pitch in
  // complex values: the lanes' fields fall in distinct banks)
  static constexpr int QP = 2 * TS_LG_KT + 1;
  static constexpr int SB = 2 * QP * NF;
  static constexpr int SP = 2 * TS_LG_ROWS + 4;  // staging: floats per (parity, field)
  static constexpr int SYN = 2 * (A + SB), SSTG = 2 * NF * SP;
  static constexpr int SYN_SMEM = sizeof(float) * (SYN > SSTG ? SYN : SSTG);
  // analysis: the grid values of a stage, NR pairs per thread, and the columns
  // [parity][latitude][field re, im] folded from them, 2 stages
  static constexpr int BP = NCOL + 4;
  static constexpr int AB = 2 * TS_LG_KT * BP;
  static constexpr int NR = NF / 8;
  static constexpr int RAW = NR * 4 * TS_LG_THREADS;
  static constexpr int AP = 4 * TS_LG_ROWS + 2;  // staging: floats per field
  static constexpr int ANA = 2 * (A + AB) + RAW, ASTG = NF * AP;
  static constexpr int ANA_SMEM = sizeof(float) * (ANA > ASTG ? ANA : ASTG);
};

// one k-step of a lane: its 2 NP table values (row pairs) times CT columns
template <int NP, int CT>
TS_DEV void ts_lg_step(const float *sa, const float (&b)[CT], float2 (&acc)[4][CT]) {
  float2 a[NP];
  if constexpr (NP % 2 == 0) {
#pragma unroll
    for (int p = 0; p < NP; p += 2) {
      const float4 x = *reinterpret_cast<const float4 *>(sa + 2 * p);
      a[p] = make_float2(x.x, x.y);
      a[p + 1] = make_float2(x.z, x.w);
    }
  } else {
#pragma unroll
    for (int p = 0; p < NP; p++) a[p] = *reinterpret_cast<const float2 *>(sa + 2 * p);
  }
#pragma unroll
  for (int c = 0; c < CT; c++) {
    const float2 bb = make_float2(b[c], b[c]);
#pragma unroll
    for (int p = 0; p < NP; p++) ts_fma2(acc[p][c], a[p], bb);
  }
}

// Where the analysis puts its values: a functor with NA fields per instance
// that takes an instance's NA values of one coefficient.  This one stores them,
// field f to instance f / nper of base[f % nper].
struct TsLgStore {
  static constexpr int NA = 1;
  float2 *base[TS_MAXIO];
  long inst_stride[TS_MAXIO];
  int nper;
  TS_DEV void operator()(long f, long lm, const float2 (&v)[NA]) const {
    const int s = (int)(f % nper);
    base[s][f / nper * inst_stride[s] + lm] = v[0];
  }
};

// --------------------------------------------------------------- synthesis
//
// grid = (nhp / 64, ceil(nfields / NF), mmax + 1).  k-tiles (16 degrees of
// each parity) before the first value of the CTA's latitudes, and of a warp's,
// are left out; the last tile ends, in steps of 4, with the order's degrees.
template <int NCOL>
__global__ void __launch_bounds__(TS_LG_THREADS, 4)
ts_leg_synth_gemm(TsLegTab t, TsLegGemmTab g, TsFields q, float2 *__restrict__ fm, long fm_stride,
                  int nfields) {
  using S = TsLg<NCOL>;
  extern __shared__ __align__(16) float ts_smem_lg[];
  __shared__ const float2 *src[S::NF];
  __shared__ int first[2];
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int lat0 = blockIdx.x * TS_LG_ROWS, f0 = blockIdx.y * S::NF, m = blockIdx.z;
  const int k0 = ts_lg_k16(t.lmax, m, 0), k1 = ts_lg_k16(t.lmax, m, 1), K = t.lmax - m + 1;
  const int par = warp >> 1, cg = lane & 7, rl = (warp & 1) * 32 + (lane >> 3) * 8;
  const float *mt = g.tab + ts_lg_off(t.lmax, m) * g.nhp + lat0;
  const long base = ts_lm_base(t.lmax, m);
  ts_grid_go();
  ts_grid_wait();
  for (int f = tid; f < S::NF; f += TS_LG_THREADS)
    src[f] = f0 + f < nfields ? ts_field(q, f0 + f) + base : nullptr;
  if (tid < TS_LG_ROWS) {
    const int o = __reduce_min_sync(0xffffffffu, g.onset[(long)m * g.nhp + lat0 + tid]);
    if (lane == 0) first[tid >> 5] = o;
  }
  __syncthreads();
  const int nkt = k0 / TS_LG_KT;
  const int kta = min(first[0], first[1]) / (2 * TS_LG_KT);
  const int ka = first[warp & 1] / (2 * TS_LG_KT);  // this warp's first k-tile
  const int kp = ts_lg_kpar(t.lmax, m, par);

  // stage k-tile kt by asynchronous copies: 2 x 16 table rows of 64 latitudes,
  // and the tile's 32 degrees of every field (lane = degree: whole lines)
  auto load = [&](int kt) {
    float *dst = ts_smem_lg + ((kt - kta) & 1) * (S::A + S::SB);
    const float *a = mt + (long)(kt * TS_LG_KT + (tid >> 4)) * g.nhp + (tid & 15) * 4;
#pragma unroll
    for (int u = 0; u < 4; u++) {
      const int row = (tid >> 4) + 8 * u;
      if (u < 2 || kt * TS_LG_KT < k1)
        ts_lg_cp16(dst + row * TS_LG_ROWS + (tid & 15) * 4,
                   a + (long)(u < 2 ? 8 * u : k0 + 8 * (u - 2)) * g.nhp);
    }
    const int i = 2 * kt * TS_LG_KT + lane;
    float2 *b = reinterpret_cast<float2 *>(dst + S::A) + lane;
#pragma unroll
    for (int u = 0; u < S::NF / 4; u++) {
      const int f = warp + 4 * u;
      const float2 *s = *const_cast<const float2 *volatile *>(&src[f]);
      ts_lg_cp8(b + f * S::QP, s ? s + min(i, K - 1) : t.ab, s && i < K);
    }
    ts_lg_cp_commit();
  };

  float2 acc[4][S::CT];
#pragma unroll
  for (int p = 0; p < 4; p++)
#pragma unroll
    for (int c = 0; c < S::CT; c++) acc[p][c] = make_float2(0.f, 0.f);
  if (kta < nkt) load(kta);
  for (int kt = kta; kt < nkt; kt++) {
    ts_lg_cp_wait<0>();
    __syncthreads();  // tile kt is here; every warp is done with tile kt - 1
    if (kt + 1 < nkt) load(kt + 1);
    const float *cur = ts_smem_lg + ((kt - kta) & 1) * (S::A + S::SB);
    const float *sa = cur + par * TS_LG_KT * TS_LG_ROWS + rl;
    const float2 *sb = reinterpret_cast<const float2 *>(cur + S::A) + cg * S::QP + par;
    auto step = [&](int k) {
      float b[S::CT];
#pragma unroll
      for (int u = 0; u < S::CT / 2; u++) {
        const float2 x = sb[2 * k + 8 * u * S::QP];
        b[2 * u] = x.x;
        b[2 * u + 1] = x.y;
      }
      ts_lg_step<4, S::CT>(sa + k * TS_LG_ROWS, b, acc);
    };
    const int n = kt < ka ? 0 : min(TS_LG_KT, kp - kt * TS_LG_KT);
    if (n == TS_LG_KT) {
#pragma unroll
      for (int k = 0; k < TS_LG_KT; k++) step(k);
    } else {
      for (int k = 0; k < n; k += 4)
#pragma unroll
        for (int u = 0; u < 4; u++) step(k + u);
    }
  }
  __syncthreads();

  // [parity][field][latitude re, im] in shared memory, then whole rows out
#pragma unroll
  for (int u = 0; u < S::CT / 2; u++) {
    float *row = ts_smem_lg + (par * S::NF + cg + 8 * u) * S::SP + 2 * rl;
#pragma unroll
    for (int p = 0; p < 4; p++)
      *reinterpret_cast<float4 *>(row + 4 * p) =
          make_float4(acc[p][2 * u].x, acc[p][2 * u + 1].x, acc[p][2 * u].y, acc[p][2 * u + 1].y);
  }
  __syncthreads();
  for (int f = warp; f < S::NF; f += 4) {
    if (f0 + f >= nfields) break;
    float2 *dst = fm + (long)(f0 + f) * fm_stride + (long)m * t.nlat;
    const float2 *e = reinterpret_cast<const float2 *>(ts_smem_lg + f * S::SP);
    const float2 *o = reinterpret_cast<const float2 *>(ts_smem_lg + (S::NF + f) * S::SP);
#pragma unroll
    for (int u = 0; u < 2; u++) {
      const int r = lane + 32 * u, lat = lat0 + r, south = t.nlat - 1 - lat;
      if (lat >= t.nh) continue;
      dst[lat] = c_add(e[r], o[r]);
      if (south != lat) dst[south] = c_sub(e[r], o[r]);
    }
  }
}

// ---------------------------------------------------------------- analysis
//
// grid = (ceil((lmax + 1) / 128), ceil(nfields / per_cta), mmax + 1), per_cta
// <= NF whole instances of Epi::NA fields: the degrees of an order are split
// evenly over its ceil(K / 128) CTAs; the others leave at once.  A CTA's degrees
// of a parity (a multiple of 8 up to 32, of 16 up to 64) are one or two equal
// blocks of 8 NP; with two blocks of each parity a warp takes one, with one
// block two warps share it: each takes half of every stage's k-steps, and the
// halves are added up at the end.  Latitudes before the first value of a warp's
// degrees are left out.
template <int NCOL, class Epi>
__global__ void __launch_bounds__(TS_LG_THREADS, 4)
ts_leg_analys_gemm(TsLegTab t, TsLegGemmTab g, const float2 *gm, long g_stride, Epi epi,
                   int nfields, int per_cta) {
  using S = TsLg<NCOL>;
  extern __shared__ __align__(16) float ts_smem_lg[];
  __shared__ int first[2];
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int f0 = blockIdx.y * per_cta, nf = min(per_cta, nfields - f0), m = blockIdx.z;
  const int K = t.lmax - m + 1, kp0 = ts_lg_k16(t.lmax, m, 0), kp1 = ts_lg_k16(t.lmax, m, 1);
  const int nch = (K + 2 * TS_LG_ROWS - 1) / (2 * TS_LG_ROWS);
  if ((int)blockIdx.x >= nch) return;
  ts_grid_go();
  ts_grid_wait();
  int per = (((K + 1) >> 1) + nch - 1) / nch;  // degrees of a parity per CTA
  per = per > 32 ? (per + 15) & ~15 : (per + 7) & ~7;
  const int j0 = blockIdx.x * per;
  const int rows = per > 32 ? per / 2 : per, np = rows / 8;  // a block, and its row pairs per lane
  const int par = warp >> 1, half = warp & 1;
  const int jb = per > 32 ? half * rows : 0;  // the warp's degrees j0 + jb ..
  const int cg = lane & 7, rl = (lane >> 3) * 2 * np;
  const bool active = j0 + jb < ts_lg_kpar(t.lmax, m, par);
  const float *mt = g.tab + ts_lg_off(t.lmax, m) * g.nhp;
  const int nkt = (t.nh + TS_LG_KT - 1) / TS_LG_KT;

  // first latitude with a value among the first / all of the CTA's degrees
  if (tid < 2) first[tid] = t.nh;
  __syncthreads();
  {
    int lo[2] = {t.nh, t.nh};
    for (int lat = t.nh - 1 - tid; lat >= 0; lat -= TS_LG_THREADS) {
      const int o = g.onset[(long)m * g.nhp + lat];
      if (o < 2 * (j0 + rows)) lo[0] = lat;
      if (o < 2 * (j0 + per)) lo[1] = lat;
    }
#pragma unroll
    for (int b = 0; b < 2; b++) {
      const int x = __reduce_min_sync(0xffffffffu, lo[b]);
      if (lane == 0) atomicMin(&first[b], x);
    }
  }
  __syncthreads();
  const int kta = first[1] / TS_LG_KT;
  const int ka = first[per > 32 ? half : 1] / TS_LG_KT;

  // stage latitudes 16 kt .. by asynchronous copies: per parity 16 table rows
  // of `per` degrees, and the north and south values of every field, which the
  // thread that copied them folds and weights into the stage's columns (lanes
  // 8 latitudes x 4 fields: a half-warp's stores fall in distinct banks)
  const int bl = (lane & 7) + 8 * (warp & 1), bf = 4 * (warp >> 1) + (lane >> 3);
  float *const sA = ts_smem_lg, *const sB = sA + 2 * S::A;
  float2 *const raw = reinterpret_cast<float2 *>(sB + 2 * S::AB) + tid;
  auto load_raw = [&](int kt) {
    const int lat = kt * TS_LG_KT + bl, south = t.nlat - 1 - lat;
    const bool live = lat < t.nh;
#pragma unroll
    for (int u = 0; u < S::NR; u++) {
      const int f = bf + 8 * u;
      const bool on = live && f < nf;
      const float2 *s = gm + (on ? (long)(f0 + f) * g_stride + (long)m * t.nlat : 0);
      ts_lg_cp8(raw + 2 * u * TS_LG_THREADS, s + (on ? lat : 0), on);
      ts_lg_cp8(raw + (2 * u + 1) * TS_LG_THREADS, s + (on ? south : 0), on && south != lat);
    }
    ts_lg_cp_commit();
  };
  auto load_a = [&](int kt) {
    float *dst = sA + (kt & 1) * S::A + (tid >> 4) * TS_LG_ROWS + (tid & 15) * 4;
    const int j = j0 + (tid & 15) * 4, lat = kt * TS_LG_KT + (tid >> 4);
    if ((tid & 15) * 4 < per) {
#pragma unroll
      for (int u = 0; u < 2; u++) {
        if (j < kp0)
          ts_lg_cp16(dst + 8 * u * TS_LG_ROWS, mt + (long)(lat + 8 * u) * kp0 + j);
        if (j < kp1)
          ts_lg_cp16(dst + (TS_LG_KT + 8 * u) * TS_LG_ROWS,
                     mt + (long)kp0 * g.nhp + (long)(lat + 8 * u) * kp1 + j);
      }
    }
    ts_lg_cp_commit();
  };
  auto fold = [&](int kt) {
    const int lat = kt * TS_LG_KT + bl;
    const float w = lat < t.nh ? __ldg(t.wq + lat) : 0.f;
    float *dst = sB + (kt & 1) * S::AB + bl * S::BP + 2 * bf;
#pragma unroll
    for (int u = 0; u < S::NR; u++) {
      const float2 n = raw[2 * u * TS_LG_THREADS], s = raw[(2 * u + 1) * TS_LG_THREADS];
      *reinterpret_cast<float2 *>(dst + 16 * u) = c_scale(c_add(n, s), w);
      *reinterpret_cast<float2 *>(dst + TS_LG_KT * S::BP + 16 * u) = c_scale(c_sub(n, s), w);
    }
  };

  float2 acc[4][S::CT];
#pragma unroll
  for (int p = 0; p < 4; p++)
#pragma unroll
    for (int c = 0; c < S::CT; c++) acc[p][c] = make_float2(0.f, 0.f);
  // k-steps [k, kend) of a stage with blocks of 8 NP rows, U at a time
  auto steps = [&](int kt, int k, int kend, auto npc, auto uc) {
    constexpr int NP = decltype(npc)::value, U = decltype(uc)::value;
    const float *sa = sA + (kt & 1) * S::A + par * TS_LG_KT * TS_LG_ROWS + jb + rl;
    const float *sb = sB + (kt & 1) * S::AB + par * TS_LG_KT * S::BP + (S::CT == 8 ? 4 : S::CT) * cg;
#pragma unroll 1
    for (; k < kend; k += U) {
#pragma unroll
      for (int i = 0; i < U; i++) {
        float b[S::CT];
        const float *r = sb + (k + i) * S::BP;
        if constexpr (S::CT == 8) {  // columns 4 cg .. and 32 + 4 cg ..
          const float4 x = *reinterpret_cast<const float4 *>(r), y = *reinterpret_cast<const float4 *>(r + 32);
          b[0] = x.x, b[1] = x.y, b[2] = x.z, b[3] = x.w;
          b[4] = y.x, b[5] = y.y, b[6] = y.z, b[7] = y.w;
        } else if constexpr (S::CT == 4) {
          const float4 x = *reinterpret_cast<const float4 *>(r);
          b[0] = x.x, b[1] = x.y, b[2] = x.z, b[3] = x.w;
        } else {
          const float2 x = *reinterpret_cast<const float2 *>(r);
          b[0] = x.x, b[1] = x.y;
        }
        ts_lg_step<NP, S::CT>(sa + (k + i) * TS_LG_ROWS, b, acc);
      }
    }
  };
  if (kta < nkt) {
    load_raw(kta);
    load_a(kta);
    ts_lg_cp_wait<1>();
    fold(kta);
    if (kta + 1 < nkt) load_raw(kta + 1);
  }
  for (int kt = kta; kt < nkt; kt++) {
    ts_lg_cp_wait<0>();  // this thread's raw values of tile kt + 1, table rows of tile kt
    __syncthreads();     // everyone's rows and columns of tile kt; all are done with tile kt - 1
    if (kt + 1 < nkt) {
      fold(kt + 1);
      load_a(kt + 1);
      if (kt + 2 < nkt) load_raw(kt + 2);
    }
    if (active && kt >= ka) {  // two warps to a block: half of the k-steps each
      const int k = per > 32 ? 0 : half * (TS_LG_KT / 2), kend = per > 32 ? TS_LG_KT : k + TS_LG_KT / 2;
      if (np == 4)
        per > 32 ? steps(kt, k, kend, TsLgInt<4>(), TsLgInt<TS_LG_UNROLL>())
                 : steps(kt, k, kend, TsLgInt<4>(), TsLgInt<8>());
      else if (np == 3)
        steps(kt, k, kend, TsLgInt<3>(), TsLgInt<8>());
      else if (np == 2)
        steps(kt, k, kend, TsLgInt<2>(), TsLgInt<4>());
      else
        steps(kt, k, kend, TsLgInt<1>(), TsLgInt<4>());
    }
  }
  __syncthreads();

  // [field][warp][32 degrees re, im] in shared memory, then (a shared block's
  // halves added) whole runs of degrees out
#pragma unroll
  for (int u = 0; u < S::CT / 2; u++) {
    const int f = S::CT == 8 ? 2 * cg + (u & 1) + 16 * (u >> 1) : S::CT / 2 * cg + u;
    float *row = ts_smem_lg + f * S::AP + 64 * warp + 2 * rl;
#pragma unroll
    for (int p = 0; p < 4; p++) {
      if (p >= np) break;
      *reinterpret_cast<float2 *>(row + 4 * p) = make_float2(acc[p][2 * u].x, acc[p][2 * u + 1].x);
      *reinterpret_cast<float2 *>(row + 4 * p + 2) = make_float2(acc[p][2 * u].y, acc[p][2 * u + 1].y);
    }
  }
  __syncthreads();
  const long lm0 = ts_lm_base(t.lmax, m) + 2 * j0;
  const int n = min(2 * per, K - 2 * j0);
  for (int q = warp; q < nf / Epi::NA; q += 4) {
    for (int i = lane; i < n; i += 32) {
      const int j = i >> 1, second = per > 32 && j >= rows;
      const float *x = ts_smem_lg + q * Epi::NA * S::AP + 64 * (2 * (i & 1) + second) + 2 * (j - (second ? rows : 0));
      float2 v[Epi::NA];
#pragma unroll
      for (int a = 0; a < Epi::NA; a++) {
        v[a] = *reinterpret_cast<const float2 *>(x + a * S::AP);
        if (per <= 32) v[a] = c_add(v[a], *reinterpret_cast<const float2 *>(x + a * S::AP + 64));
      }
      epi(f0 / Epi::NA + q, lm0 + i, v);
    }
  }
}

// ------------------------------------------------------------- few fields
//
// One or two fields: every table value meets two or four numbers, so the
// products are bound by reading the table (25 MB a direction at lmax 255, from
// the L2) and by the latency of a CTA's few stages.  No staging then: a warp's
// lanes read whole rows of the table straight into registers, pairs of
// neighbours each, with eight rows in flight, and the columns come as broadcasts
// from shared memory.  The rows of a CTA are dealt out to its warps, whose sums
// are added up at the end.

// a load of what the kernel before this one wrote: not through the read-only
// path, and not moved ahead of ts_grid_wait()
TS_DEV float2 ts_lg_ld(const float2 *p) {
  float2 v;
  asm volatile("ld.global.v2.f32 {%0, %1}, [%2];" : "=f"(v.x), "=f"(v.y) : "l"(p) : "memory");
  return v;
}

template <int F>
TS_DEV void ts_lg_columns(float2 (&c)[F], const float2 *s) {
  if constexpr (F == 1) {
    c[0] = s[0];
  } else {
#pragma unroll
    for (int f = 0; f < F; f += 2) {
      const float4 x = *reinterpret_cast<const float4 *>(s + f);
      c[f] = make_float2(x.x, x.y);
      c[f + 1] = make_float2(x.z, x.w);
    }
  }
}

// grid = (nhp / 64, mmax + 1), 256 threads: warp = (parity, one of 4 parts of
// its degrees), lane = 2 of 64 latitudes.  Shared memory: (lmax + 1) F float2.
template <int F>
__global__ void __launch_bounds__(256)
ts_leg_synth_few(TsLegTab t, TsLegGemmTab g, TsFields q, float2 *__restrict__ fm, long fm_stride,
                 int nfields) {
  extern __shared__ __align__(16) float2 ts_smem_fs[];
  __shared__ float2 red[8][F][TS_LG_ROWS];
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, par = warp & 1, part = warp >> 1;
  const int lat0 = blockIdx.x * TS_LG_ROWS, m = blockIdx.y, K = t.lmax - m + 1;
  const long base = ts_lm_base(t.lmax, m);
  const int *on = g.onset + (long)m * g.nhp + lat0 + 2 * lane;
  ts_grid_go();
  ts_grid_wait();
  const int o0 = __ldg(on), o1 = __ldg(on + 1);
  const float2 *src[F];
#pragma unroll
  for (int f = 0; f < F; f++) src[f] = ts_field(q, min(f, nfields - 1)) + base;
  for (int i0 = tid; i0 < K; i0 += 1024) {  // every load of a thread before its stores
    float2 v[4][F];
#pragma unroll
    for (int u = 0; u < 4; u++)
#pragma unroll
      for (int f = 0; f < F; f++) v[u][f] = ts_lg_ld(src[f] + min(i0 + 256 * u, K - 1));
#pragma unroll
    for (int u = 0; u < 4; u++)
#pragma unroll
      for (int f = 0; f < F; f++)
        if (i0 + 256 * u < K) ts_smem_fs[(i0 + 256 * u) * F + f] = v[u][f];
  }
  const int first = __reduce_min_sync(0xffffffffu, min(o0, o1));
  const int kp = ts_lg_kpar(t.lmax, m, par);
  const float *row = g.tab + (ts_lg_off(t.lmax, m) + (par ? ts_lg_k16(t.lmax, m, 0) : 0)) * g.nhp + lat0 + 2 * lane;
  float2 acc[F][2];
#pragma unroll
  for (int f = 0; f < F; f++) acc[f][0] = acc[f][1] = make_float2(0.f, 0.f);
  __syncthreads();
  for (int j = (first >> 1) + part; j < kp; j += 32) {
    float2 p[8];
#pragma unroll
    for (int u = 0; u < 8; u++)
      p[u] = j + 4 * u < kp ? __ldg(reinterpret_cast<const float2 *>(row + (long)(j + 4 * u) * g.nhp))
                            : make_float2(0.f, 0.f);
#pragma unroll
    for (int u = 0; u < 8; u++) {
      float2 c[F];
      ts_lg_columns<F>(c, ts_smem_fs + (2 * min(j + 4 * u, kp - 1) + par) * F);
#pragma unroll
      for (int f = 0; f < F; f++) {
        ts_fma2(acc[f][0], make_float2(p[u].x, p[u].x), c[f]);
        ts_fma2(acc[f][1], make_float2(p[u].y, p[u].y), c[f]);
      }
    }
  }
#pragma unroll
  for (int f = 0; f < F; f++) {
    red[warp][f][2 * lane] = acc[f][0];
    red[warp][f][2 * lane + 1] = acc[f][1];
  }
  __syncthreads();
  for (int i = tid; i < TS_LG_ROWS * F; i += 256) {
    const int f = i / TS_LG_ROWS, r = i % TS_LG_ROWS, lat = lat0 + r, south = t.nlat - 1 - lat;
    if (f >= nfields || lat >= t.nh) continue;
    float2 e = red[0][f][r], o = red[1][f][r];
#pragma unroll
    for (int k = 2; k < 8; k += 2) {
      e = c_add(e, red[k][f][r]);
      o = c_add(o, red[k + 1][f][r]);
    }
    float2 *dst = fm + (long)f * fm_stride + (long)m * t.nlat;
    dst[lat] = c_add(e, o);
    if (south != lat) dst[south] = c_sub(e, o);
  }
}

// grid = (ceil((lmax + 1) / 128), mmax + 1), 512 threads: 64 degrees of each
// parity per CTA; warp = (parity, one of 8 parts of the latitudes), lane = 2
// degrees (rows of up to 16 or 32 degrees: 4 or 2 latitudes a load).  Shared
// memory: 2 nh F + 16 F 64 float2.
template <int F, class Epi>
__global__ void __launch_bounds__(512)
ts_leg_analys_few(TsLegTab t, TsLegGemmTab g, const float2 *gm, long g_stride, Epi epi,
                  int nfields) {
  extern __shared__ __align__(16) float2 ts_smem_fa[];  // [parity][latitude][F], then [warp][F][64]
  __shared__ int first;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, par = warp & 1, part = warp >> 1;
  const int m = blockIdx.y, j0 = blockIdx.x * TS_LG_ROWS, K = t.lmax - m + 1;
  if (2 * j0 >= K) return;
  ts_grid_go();
  ts_grid_wait();
  const int kp0 = ts_lg_k16(t.lmax, m, 0), kp = par ? ts_lg_k16(t.lmax, m, 1) : kp0;
  if (tid == 0) first = t.nh;
  __syncthreads();
  for (int lat = tid; lat < t.nh; lat += 512) {
    if (__ldg(g.onset + (long)m * g.nhp + lat) < 2 * (j0 + TS_LG_ROWS)) atomicMin(&first, lat);
    const int south = t.nlat - 1 - lat;
    const float w = __ldg(t.wq + lat);
#pragma unroll
    for (int f = 0; f < F; f++) {
      float2 n = make_float2(0.f, 0.f), s = n;
      if (f < nfields) {
        const float2 *src = gm + (long)f * g_stride + (long)m * t.nlat;
        n = ts_lg_ld(src + lat);
        if (south != lat) s = ts_lg_ld(src + south);
      }
      ts_smem_fa[lat * F + f] = c_scale(c_add(n, s), w);
      ts_smem_fa[(t.nh + lat) * F + f] = c_scale(c_sub(n, s), w);
    }
  }
  __syncthreads();
  const int jn = min(TS_LG_ROWS, kp - j0);  // (a multiple of 16, or none)
  const int lpr = jn <= 16 ? 8 : jn <= 32 ? 16 : 32, rpw = 32 / lpr;  // lanes of a row, rows of a load
  const int sub = lane / lpr, jl = 2 * (lane & (lpr - 1));
  const bool on = jl < jn;
  const float *row = g.tab + ts_lg_off(t.lmax, m) * g.nhp + (par ? (long)kp0 * g.nhp : 0) + j0 + (on ? jl : 0);
  const float2 *col = ts_smem_fa + par * t.nh * F;
  float2 acc[F][2];
#pragma unroll
  for (int f = 0; f < F; f++) acc[f][0] = acc[f][1] = make_float2(0.f, 0.f);
  const int step = 8 * rpw;
  if (on)
    for (int lat = first + part * rpw + sub; lat < t.nh; lat += 8 * step) {
      float2 p[8];
#pragma unroll
      for (int u = 0; u < 8; u++)
        p[u] = lat + u * step < t.nh ? __ldg(reinterpret_cast<const float2 *>(row + (long)(lat + u * step) * kp))
                                     : make_float2(0.f, 0.f);
#pragma unroll
      for (int u = 0; u < 8; u++) {
        float2 c[F];
        ts_lg_columns<F>(c, col + min(lat + u * step, t.nh - 1) * F);
#pragma unroll
        for (int f = 0; f < F; f++) {
          ts_fma2(acc[f][0], make_float2(p[u].x, p[u].x), c[f]);
          ts_fma2(acc[f][1], make_float2(p[u].y, p[u].y), c[f]);
        }
      }
    }
  float2 *red = ts_smem_fa + 2 * t.nh * F;
#pragma unroll
  for (int f = 0; f < F; f++)
#pragma unroll
    for (int e = 0; e < 2; e++) {
      float2 v = acc[f][e];
      for (int d = lpr; d < 32; d <<= 1) {
        v.x += __shfl_xor_sync(0xffffffffu, v.x, d);
        v.y += __shfl_xor_sync(0xffffffffu, v.y, d);
      }
      if (on && sub == 0) red[(warp * F + f) * TS_LG_ROWS + jl + e] = v;
    }
  __syncthreads();
  const long lm0 = ts_lm_base(t.lmax, m) + 2 * j0;
  const int n = min(2 * TS_LG_ROWS, K - 2 * j0), ni = nfields / Epi::NA;
  for (int i = tid; i < n * ni; i += 512) {
    const int inst = i / n, d = i % n;
    float2 v[Epi::NA];
#pragma unroll
    for (int a = 0; a < Epi::NA; a++) {
      const float2 *r = red + ((d & 1) * F + inst * Epi::NA + a) * TS_LG_ROWS + (d >> 1);
      v[a] = r[0];
#pragma unroll
      for (int k = 1; k < 8; k++) v[a] = c_add(v[a], r[2 * k * F * TS_LG_ROWS]);
    }
    epi(inst, lm0 + d, v);
  }
}
