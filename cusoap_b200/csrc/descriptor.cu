// Fused per-centre SOAP descriptor: radial table x real solid harmonics ->
// c_nlm accumulated in registers -> power spectrum / cc / raw epilogue.
//
// Reference: _coefficients_gto (soap_generator.py:1294-1391), the self term
// (:765-850, here the kept r=0 edge of the centre's own atom, whose value is
// exactly B_n0(0) Y00), _power_spectrum (:1634-1689) with the DScribe
// feature order of _build_feature_slices (:1215-1245), and _projection_cc /
// _to_dscribe_cc (:1603-1632).  average 'inner' and 'outer' are centre-wise
// in the reference (coeffs_use = coeffs, :1651-1657), i.e. identical to 'off'.
//
// Mapping: one warp per centre, centres taken from an atomic work queue.
// Lanes are grouped by l: floor(32 / (L+1)) lanes per l, each owning GN radial
// functions (n, l) of the same l, so one shared-memory read of R_lm feeds GN
// accumulators and the m loop is the same for all of them.  The centre's
// pairs arrive sorted by (species, radial segment): the species switch
// flushes the accumulators into the warp's coefficient buffer, the segment
// switch (warp-uniform) reloads the lane's table coefficients, so the
// per-pair work is 7 FMAs of Horner per function plus one FMA per (n, l, m).
// For l_max <= 4, where one stream leaves lanes idle, each half-warp walks its
// own stream of the pairs (k_descriptor_2s).  Solid harmonics are computed 16
// pairs at a time (32 with two pair streams), one pair per lane, into shared
// memory.  The power-spectrum epilogue walks the DScribe blocks (species pair,
// l) in one non-unrolled l loop; each lane writes consecutive features, so
// the row is stored coalesced.
#include "common.cuh"

namespace soapb {

struct DescArgs {
  const int64_t* pair_off;
  const float4* pairs;
  int64_t n_centres;
  const float* tab_b;
  const float* tab_p;  // pair-interleaved table (radial-index lanes)
  const float* selfv;  // w0 B_nl(0): value of r = 0 edges (the centre's own Gaussian)
  float* out;
  float* coeff_out;  // optional raw c[s][n][lm] rows (S N K floats per centre)
  int* counter;        // work queue; nullptr: at least as many warps as centres, one each
  int N, S, nseg, F, mode, crossover;
  float inv_h;
  float self_ratio;  // w0 / w(0): an r = 0 edge's table value times this is its self value
};

// Position of harmonic block l in a pair's Y row: l^2 plus a padding that
// starts every block on a different shared-memory bank (the lane groups of the
// l blocks read the same slot m of their blocks at once: no conflicts).  Plain
// l^2 puts l = 6 on the bank of l = 2 (36 = 4 mod 32), l = 8 on that of l = 0
// and l = 12 on that of l = 4; one float of padding from l = 6, another from
// l = 8 and two more from l = 12 separate them (checked below).
__host__ __device__ constexpr int ybase(int l) { return l * l + (l >= 6) + (l >= 8) + 2 * (l >= 12); }
// Y row position of harmonic index idx = l^2 + l + m (idx >= 36: l >= 6, >= 64: l >= 8, >= 144: l >= 12).
__host__ __device__ constexpr int ypos(int idx) { return idx + (idx >= 36) + (idx >= 64) + 2 * (idx >= 144); }

constexpr bool ybase_banks_distinct() {
  for (int l = 0; l <= kMaxL; ++l) {
    if (l > 0 && ybase(l) < ybase(l - 1) + 2 * l - 1) return false;  // blocks overlap
    for (int k = 0; k < l; ++k)
      if (ybase(k) % 32 == ybase(l) % 32) return false;
    for (int m = 0; m <= 2 * l; ++m)
      if (ypos(l * l + m) != ybase(l) + m) return false;
  }
  return true;
}
static_assert(ybase_banks_distinct(), "Y row blocks must start on distinct banks");

// Extra offset of the Y rows of pairs 16..31 (two pair streams per warp): the
// smallest shift that keeps the l blocks of row q and row q + 16 -- read by
// the two half-warps at once -- on distinct banks.
__host__ __device__ constexpr int half_offset(int L, int YS) {
  for (int h = 0; h < 32; ++h) {
    bool ok = true;
    for (int l = 0; l <= L; ++l)
      for (int k = 0; k <= L; ++k)
        if ((16 * YS + h + ybase(l)) % 32 == ybase(k) % 32) ok = false;
    if (ok) return h;
  }
  return 0;
}

template <int L>
struct DescShape {
  static constexpr int K = (L + 1) * (L + 1);
  static constexpr int YS = (ybase(L) + 2 * L + 1) | 1;  // odd strides: conflict-free row writes
  static constexpr int HOFF = half_offset(L, YS);
  static constexpr int KC = K | 1;
  __host__ __device__ static int warp_floats(int S, int N) { return 32 * YS + HOFF + 96 + S * N * KC; }
  // one pair stream: 16 staged pairs per batch
  __host__ __device__ static int warp_floats16(int S, int N) { return 16 * YS + 48 + S * N * KC; }
};

// Functions per lane for (N, L): floor(32 / (L+1)) lanes share each l.
inline int desc_group(int N, int L) {
  const int lpl = 32 / (L + 1);
  int gn = (N + lpl - 1) / lpl;
  if (gn == 5) gn = 6;
  return gn;
}

// Two pair streams per warp (each half-warp walks 16 of every 32 pairs, lanes
// grouped by l inside the half, at most 3 functions per lane), for l_max <= 4
// when one stream leaves more than a quarter of the lanes without a function
// (n_max 8, l_max 4: 20 of 32 lanes busy with one stream, 30 with two).
inline bool desc_two_streams(int N, int L) {
  if (L > 4) return false;
  const int lpl = 16 / (L + 1);
  if ((N + lpl - 1) / lpl > 3) return false;
  const int gn = desc_group(N, L);
  return (L + 1) * ((N + gn - 1) / gn) <= 24;
}

constexpr int kMaxBlocks = kMaxS * (kMaxS + 1) / 2;
constexpr int kMaxTri = kMaxN * (kMaxN + 1) / 2;

// Per-block tables of the power-spectrum epilogue: the prefactor
// sqrt(8 pi^2 / (2l+1)) per l, the DScribe species blocks (j | jd << 8, first
// feature) and the (n, n') pairs of the upper-triangle index.
template <int L>
__device__ __forceinline__ void desc_tables(const DescArgs& a, float* s_pref, int* s_blk, unsigned char* s_tri) {
  const int N = a.N, S = a.S;
  if (threadIdx.x <= L) s_pref[threadIdx.x] = sqrtf(8.0f * (float)(kPi * kPi) / (2.0f * threadIdx.x + 1.0f));
  if (threadIdx.x == 0) {
    int nb = 0, f = 0;
    for (int j = 0; j < S; ++j)
      for (int jd = j; jd < (a.crossover ? S : j + 1); ++jd) {
        s_blk[2 * nb] = j | (jd << 8);
        s_blk[2 * nb + 1] = f;
        f += (j == jd ? N * (N + 1) / 2 : N * N) * (L + 1);
        ++nb;
      }
    int p = 0;
    for (int n = 0; n < N; ++n)
      for (int nd = n; nd < N; ++nd, ++p) {
        s_tri[2 * p] = (unsigned char)n;
        s_tri[2 * p + 1] = (unsigned char)nd;
      }
  }
}

// One centre's outputs from its coefficients cbuf[(s N + n) KC + lm]
// (KC = K | 1), written by the whole warp: the raw coefficient row when
// requested, then the power spectrum in DScribe order (each lane writes
// consecutive features of a block, so rows are stored coalesced), or the
// cc / raw projection.
template <int L>
__device__ __forceinline__ void desc_epilogue(const DescArgs& a, int64_t c, const float* cbuf, int lane,
                                              const float* s_pref, const int* s_blk, const unsigned char* s_tri) {
  constexpr int K = (L + 1) * (L + 1), KC = K | 1;
  const int N = a.N, S = a.S;
  if (a.coeff_out) {
    float* crow = a.coeff_out + (size_t)c * S * N * K;
    for (int f = lane; f < S * N * K; f += 32) {
      const int sn = f / K;
      crow[f] = cbuf[sn * KC + (f - sn * K)];
    }
  }
  float* orow = a.out + (size_t)c * a.F;
  if (a.mode == SOAPB_OUT_PS) {
    const int nblk = a.crossover ? S * (S + 1) / 2 : S;
    const int q32 = 32 / N, r32 = 32 % N;  // p -> p + 32 in the off-diagonal (n, n') order
    for (int b = 0; b < nblk; ++b) {
      const int jj = s_blk[2 * b], fb0 = s_blk[2 * b + 1];
      const int j = jj & 255, jd = jj >> 8;
      const bool diag = j == jd;
      const int np = diag ? N * (N + 1) / 2 : N * N;
#pragma unroll 1  // one copy of the l loop: smaller code, fewer instruction-fetch stalls
      for (int l = 0; l <= L; ++l) {
        float* o = orow + fb0 + l * np;
        int n = lane / N, nd = lane - (lane / N) * N;  // off-diagonal (n, n') of p, advanced by 32 per step
        for (int p = lane; p < np; p += 32) {
          if (diag) {
            n = s_tri[2 * p];
            nd = s_tri[2 * p + 1];
          }
          const float* x = cbuf + (j * N + n) * KC + l * l;
          const float* y = cbuf + (jd * N + nd) * KC + l * l;
          float s = 0.0f;
#pragma unroll
          for (int m = 0; m < 2 * l + 1; ++m) s = fmaf(x[m], y[m], s);
          o[p] = s * s_pref[l];
          if (!diag) {
            n += q32;
            nd += r32;
            if (nd >= N) { nd -= N; ++n; }
          }
        }
      }
    }
  } else {
    const bool cc = a.mode == SOAPB_OUT_CC;
    const float pi_m15 = (float)(1.0 / (kPi * 1.7724538509055160273));  // pi^-3/2
    for (int f = lane; f < a.F; f += 32) {
      const int sn = f / K, lm = f - sn * K;
      int src = lm;
      float scale = 1.0f;
      if (cc) {
        // l = 1 stored (z, x, y) = source lm (2, 3, 1); lm >= 4 scaled by pi^-3/2
        if (lm >= 1 && lm <= 3) src = (lm == 3) ? 1 : lm + 1;
        if (lm >= 4) scale = pi_m15;
      }
      orow[f] = cbuf[sn * KC + src] * scale;
    }
  }
}

// H pair streams per warp (1, or 2 for small l_max): half-warp h takes pairs
// 16 h .. 16 h + 15 of every staged batch of 32.  Each stream keeps its own
// species and segment; the streams flush their species partials into the
// centre's coefficient buffer one after the other, so sums are deterministic.
template <int L, int GN, int H>
__device__ __forceinline__ void descriptor_body(const DescArgs& a) {
  using Sh = DescShape<L>;
  constexpr int YS = Sh::YS, KC = Sh::KC, M = 2 * L + 1;
  constexpr int HL = 32 / H;           // lanes per stream
  constexpr int LPL = HL / (L + 1);    // lanes per l
  constexpr int HOFF = (H == 2) ? Sh::HOFF : 0;
  extern __shared__ float sm[];
  __shared__ float s_pref[kMaxL + 1];
  __shared__ int s_blk[2 * kMaxBlocks];              // (j | jd << 8, first feature) per species block
  __shared__ unsigned char s_tri[2 * kMaxTri];       // (n, n') of the upper-triangle index
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  const int N = a.N, S = a.S, NF = N * (L + 1);
  const int cbn = S * N * KC;
  // pairs staged per batch: 16 with one stream (half the harmonic rows in shared
  // memory, so more warps fit an SM), 32 with two (16 per stream)
  constexpr int BQ = (H == 2) ? 32 : 16;
  float* Y = sm + (size_t)wid * ((H == 2) ? Sh::warp_floats(S, N) : Sh::warp_floats16(S, N));
  float* tt = Y + BQ * YS + ((H == 2) ? Sh::HOFF : 0);
  int* sg = (int*)(tt + BQ);
  int* spp = sg + BQ;
  float* cbuf = (float*)(spp + BQ);
  desc_tables<L>(a, s_pref, s_blk, s_tri);
  __syncthreads();

  // lane -> stream, l and its functions n = k GN + g
  const int h = (H == 2) ? (lane >> 4) : 0, hl = lane & (HL - 1);
  const int l_me = hl / LPL, k_me = hl % LPL;
  const bool active = l_me <= L && k_me * GN < N;
  const int lme = active ? l_me : 0;
  const int mme = 2 * lme + 1;
  const int ybm = ybase(lme) + h * (16 * YS + HOFF);  // this stream's row block
  float selfb[GN];
#pragma unroll
  for (int g = 0; g < GN; ++g) {
    const int n = k_me * GN + g;
    selfb[g] = (active && n < N) ? __ldg(a.selfv + fn_index(n, lme, N)) : 0.0f;
  }

  for (;;) {
    int c32 = 0;
    if (lane == 0) c32 = atomicAdd(a.counter, 1);
    const int64_t c = __shfl_sync(0xffffffffu, c32, 0);
    if (c >= a.n_centres) break;
    for (int i = lane; i < cbn; i += 32) cbuf[i] = 0.0f;
    float acc[GN][M];
#pragma unroll
    for (int g = 0; g < GN; ++g)
#pragma unroll
      for (int m = 0; m < M; ++m) acc[g][m] = 0.0f;
    float cf[GN][kNCoef];
#pragma unroll
    for (int g = 0; g < GN; ++g)
#pragma unroll
      for (int k = 0; k < kNCoef; ++k) cf[g][k] = 0.0f;
    int cur_sp = -1, cur_seg = -1;
    const int64_t p0 = a.pair_off[c], p1 = a.pair_off[c + 1];
    __syncwarp();

    auto flush = [&](int sp) {
      if (active) {
#pragma unroll
        for (int g = 0; g < GN; ++g) {
          const int n = k_me * GN + g;
          if (n < N) {
            float* dst = cbuf + (sp * N + n) * KC + lme * lme;
#pragma unroll
            for (int m = 0; m < M; ++m)
              if (m < mme) dst[m] += acc[g][m];
          }
        }
      }
#pragma unroll
      for (int g = 0; g < GN; ++g)
#pragma unroll
        for (int m = 0; m < M; ++m) acc[g][m] = 0.0f;
    };

    for (int64_t base = p0; base < p1; base += BQ) {
      const int nt = (int)min((int64_t)BQ, p1 - base);
      if (lane < nt) {
        const float4 pr = __ldg(a.pairs + base + lane);
        const int w = __float_as_int(pr.w);
        const float r = sqrtf(pr.x * pr.x + pr.y * pr.y + pr.z * pr.z);
        int seg;
        float t;
        seg_coord(r, a.inv_h, a.nseg, seg, t);
        tt[lane] = (r > 0.0f) ? t : 3.0f;  // 3: r = 0 edge, takes the self value
        sg[lane] = seg;
        spp[lane] = (int)((unsigned)w >> kAtomBits);
        float* yrow = Y + lane * YS + ((H == 2 && lane >= 16) ? HOFF : 0);
        SolidHarmonics<L>::values(pr.x, pr.y, pr.z, [&](int idx, float v) { yrow[ypos(idx)] = v; });
      }
      __syncwarp();
      const int nq = (H == 2) ? min(nt, 16) : nt;
      for (int j = 0; j < nq; ++j) {
        const int q = h * 16 + j;
        const bool valid = (H == 1) || q < nt;  // the second stream of a short batch idles
        const int sp = valid ? spp[q] : cur_sp;
        if (H == 1) {
          if (sp != cur_sp) {
            if (cur_sp >= 0) flush(cur_sp);
            cur_sp = sp;
          }
        } else if (__any_sync(0xffffffffu, sp != cur_sp)) {
#pragma unroll
          for (int hh = 0; hh < H; ++hh) {  // stream 0 first, then stream 1
            if (h == hh && sp != cur_sp && cur_sp >= 0) flush(cur_sp);
            __syncwarp();
          }
          cur_sp = sp;
        }
        const int seg = valid ? sg[q] : cur_seg;
        if (seg != cur_seg) {
          if (active) {
#pragma unroll
            for (int g = 0; g < GN; ++g) {
              const int n = k_me * GN + g;
              if (n < N) load_coef(a.tab_b, seg, fn_index(n, lme, N), NF, cf[g]);
            }
          }
          cur_seg = seg;
        }
        if (valid) {
          const float t = tt[q];
          float B[GN];
#pragma unroll
          for (int g = 0; g < GN; ++g) B[g] = (t > 2.0f) ? selfb[g] : horner7(cf[g], t);
          // all M slots, without a per-lane test: slots m >= 2l+1 read on along
          // the row (position <= ybase(l) + 2L < YS, in bounds) and collect
          // values that flush() never stores, so no branch is needed per slot
          const float* yr = Y + j * YS + ybm;
#pragma unroll
          for (int m = 0; m < M; ++m) {
            const float yv = yr[m];
#pragma unroll
            for (int g = 0; g < GN; ++g) acc[g][m] = fmaf(B[g], yv, acc[g][m]);
          }
        }
      }
      __syncwarp();
    }
#pragma unroll
    for (int hh = 0; hh < H; ++hh) {
      if (h == hh && cur_sp >= 0) flush(cur_sp);
      __syncwarp();
    }
    desc_epilogue<L>(a, c, cbuf, lane, s_pref, s_blk, s_tri);
    __syncwarp();
  }
}

template <int L, int GN>
__global__ void __launch_bounds__(128) k_descriptor(DescArgs a) {
  descriptor_body<L, GN, 1>(a);
}

// Two pair streams (l_max <= 4): up to 128 registers, 4 blocks of 4 warps per
// SM (1M-atom cluster: 28.7 ms, against 33.6 ms capped at 96 registers for 5 blocks).
template <int L, int GN>
__global__ void __launch_bounds__(128, 4) k_descriptor_2s(DescArgs a) {
  descriptor_body<L, GN, 2>(a);
}

// Order of the (l, m) slots in the rows of the radial-index-lane kernel:
// slots are the operands of packed FMAs, so the row is made of pairs (lm, lm')
// whose radial functions sit in one register pair.  The l pairs (L, L - 1),
// (L - 2, L - 3), ... of the interleaved table give 2 lo + 1 slot pairs each
// and leave two slots of their larger l; the leftovers of two l pairs are
// paired with each other, those of a last one among themselves, and l = 0 is
// the single last slot when L is even.  With plain order, half of the pairs
// would mix neighbouring l and need two moves each to assemble an operand.
template <int L>
struct YOrder {
  static constexpr int K = (L + 1) * (L + 1), NS = K / 2;  // NS packed slots, K odd: one scalar (lm = 0)
  static constexpr int NLP = (L + 1) / 2;                  // l pairs
  int lm[K];   // lm at each position
  int pos[K];  // position of each lm
  constexpr YOrder() : lm(), pos() {
    int i = 0;
    for (int p = 0; p < NLP; ++p) {
      const int hi = L - 2 * p, lo = hi - 1;
      for (int m = 0; m < 2 * lo + 1; ++m) {
        lm[i++] = hi * hi + m;
        lm[i++] = lo * lo + m;
      }
    }
    for (int p = 0; p + 1 < NLP; p += 2)
      for (int k = 0; k < 2; ++k) {
        const int h0 = L - 2 * p, h1 = L - 2 * p - 2;
        lm[i++] = h0 * h0 + 2 * h0 - 1 + k;
        lm[i++] = h1 * h1 + 2 * h1 - 1 + k;
      }
    if (NLP % 2 == 1) {
      const int h = L - 2 * (NLP - 1);
      lm[i++] = h * h + 2 * h - 1;
      lm[i++] = h * h + 2 * h;
    }
    if (K % 2 == 1) lm[i++] = 0;
    for (int k = 0; k < K; ++k) pos[lm[k]] = k;
  }
  static constexpr int l_of(int lm_) {
    int l = 0;
    while ((l + 1) * (l + 1) <= lm_) ++l;
    return l;
  }
};
template <int L>
__device__ constexpr YOrder<L> kYOrder{};

// Epilogue of the radial-index-lane kernel: coefficient rows KR = K4 floats
// apart (16-byte aligned), slots in YOrder.  For the power spectrum each lane
// takes one (n, n') pair of a species block and contracts the two rows with
// packed FMAs, reading them as float4; for each l the lanes write consecutive
// features (coalesced).  Same outputs and DScribe order as desc_epilogue.
template <int L, int KR>
__device__ __forceinline__ void desc_epilogue_n(const DescArgs& a, int64_t c, const float* cbuf, int lane,
                                                const float* s_pref, const int* s_blk, const unsigned char* s_tri,
                                                const unsigned char* s_pos) {
  constexpr int K = (L + 1) * (L + 1);
  using YO = YOrder<L>;
  const int N = a.N, S = a.S;
  if (a.coeff_out) {
    float* crow = a.coeff_out + (size_t)c * S * N * K;
    for (int f = lane; f < S * N * K; f += 32) {
      const int sn = f / K;
      crow[f] = cbuf[sn * KR + s_pos[f - sn * K]];
    }
  }
  float* orow = a.out + (size_t)c * a.F;
  if (a.mode != SOAPB_OUT_PS) {
    const bool cc = a.mode == SOAPB_OUT_CC;
    const float pi_m15 = (float)(1.0 / (kPi * 1.7724538509055160273));  // pi^-3/2
    for (int f = lane; f < a.F; f += 32) {
      const int sn = f / K, lm = f - sn * K;
      int src = lm;
      float scale = 1.0f;
      if (cc) {
        // l = 1 stored (z, x, y) = source lm (2, 3, 1); lm >= 4 scaled by pi^-3/2
        if (lm >= 1 && lm <= 3) src = (lm == 3) ? 1 : lm + 1;
        if (lm >= 4) scale = pi_m15;
      }
      orow[f] = cbuf[sn * KR + s_pos[src]] * scale;
    }
    return;
  }
  const int nblk = a.crossover ? S * (S + 1) / 2 : S;
  for (int b = 0; b < nblk; ++b) {
    const int jj = s_blk[2 * b], fb0 = s_blk[2 * b + 1];
    const int j = jj & 255, jd = jj >> 8;
    const bool diag = j == jd;
    const int np = diag ? N * (N + 1) / 2 : N * N;
    for (int p = lane; p < np; p += 32) {
      int n, nd;
      if (diag) {
        n = s_tri[2 * p];
        nd = s_tri[2 * p + 1];
      } else {
        n = p / N;
        nd = p - n * N;
      }
      const ulonglong2* x2 = reinterpret_cast<const ulonglong2*>(cbuf + (j * N + n) * KR);
      const ulonglong2* y2 = reinterpret_cast<const ulonglong2*>(cbuf + (jd * N + nd) * KR);
      // sums of slot pairs with the same two l, one per l pair of the table; the last two products
      // of the larger l follow, packed with those of the next l pair: every sum runs over m in order
      constexpr int NLP = YO::NLP;
      f32x2 sum[NLP > 0 ? NLP : 1], tail = 0ull;
#pragma unroll
      for (int k = 0; k < NLP; ++k) sum[k] = 0ull;
      float sl[L + 1];
#pragma unroll
      for (int q = 0; q < (K + 3) / 4; ++q) {
        const ulonglong2 u = x2[q], v = y2[q];
#pragma unroll
        for (int hh = 0; hh < 2; ++hh) {
          const int i = 2 * q + hh;  // slot pair
          const f32x2 x = hh ? u.y : u.x, y = hh ? v.y : v.x;
          if (i < YO::NS) {
            const int ma = kYOrder<L>.lm[2 * i], la = YO::l_of(ma), lb = YO::l_of(kYOrder<L>.lm[2 * i + 1]);
            const int k = (L - la) / 2;
            if (lb == la - 1) {
              sum[k] = fma2(x, y, sum[k]);
            } else {
              float s0, s1, t_;
              if (ma == la * la + 2 * la - 1) {  // the first of the last two
                unpack2(sum[k], s0, sl[la - 1]);
                if (lb == la) {
                  float xa, xb, ya, yb;
                  unpack2(x, xa, xb);
                  unpack2(y, ya, yb);
                  sl[la] = fmaf(xb, yb, fmaf(xa, ya, s0));
                } else {
                  unpack2(sum[k + 1 < NLP ? k + 1 : k], s1, t_);
                  sl[lb - 1] = t_;
                  tail = fma2(x, y, pack2(s0, s1));
                }
              } else {
                tail = fma2(x, y, tail);
                unpack2(tail, sl[la], sl[lb]);
              }
            }
          } else if (K % 2 == 1 && i == YO::NS) {
            float xa, xb, ya, yb;
            unpack2(x, xa, xb);
            unpack2(y, ya, yb);
            sl[0] = xa * ya;
          }
        }
      }
      float* o = orow + fb0 + p;
#pragma unroll
      for (int l = 0; l <= L; ++l) o[l * np] = sl[l] * s_pref[l];
    }
  }
}

// ---------------------------------------------------------------------------
// Radial-index lanes (n_max <= 8, l_max <= 6): lane n of a stream owns the
// radial index n and ALL K = (l_max+1)^2 accumulators c[n][lm] of it, so
// every lane does the same work per pair -- l_max+1 Horner evaluations
// (its functions (n, 0..l_max)) and K FMAs -- with no idle m slots.  NP
// lanes form a stream (NP = 8, or 4 for n_max <= 4); the 32 / NP streams of
// a warp walk contiguous, equal parts of the centre's pair list, so each
// stream sees only its part's species and segment runs and reloads its
// coefficients rarely.  32 pairs (NP per stream) are staged per batch, one
// per lane, as rows of solid harmonics in shared memory; the rows of different
// streams are 4 floats off each other, so the streams' reads of the same slots
// hit different groups of four banks.
//
// Instruction issue is the bound (1M atoms: 35 warp instructions per pair, of
// which 15 are the algorithmic FMAs), so two values go into each FMA: the
// table interleaves pairs of l, whose Horner passes run packed, and the row's
// slots are ordered so that most slot pairs take such a register pair as it
// is (YOrder).  Each half of a packed FMA is the scalar one, every sum keeps its
// order over the neighbours, and the harmonics are staged with their norms: the
// coefficients are those of scalar FMAs bit by bit, as float64 position gradients
// need (norms applied to the sums instead: 13.95 against 14.05 ms for 1M atoms, and
// a larger error).  The pair loop branches around the coefficient reloads and is
// unrolled over the batch or not (DescDispatch).  1M atoms (l_max 4): 14.65 -> 14.05 ms;
// 48 cells (l_max 6): 266 -> 255 us; 3000 atoms (l_max 3): 73 -> 67 us.  The gain is less than the
// instructions saved because packed and scalar FMAs with three distinct
// operands share the register ports (2.3 - 2.7 and 1.6 - 1.9 cycles each,
// measured) and 4 warps per scheduler leave 45 % of the issue slots to the
// latency of the reloads and row reads.  Measured slower: the polynomials as
// trees over t^2, t^4 (14.36 ms), two pairs per step (16.0 ms), 3 blocks per SM
// (14.8 ms; l_max 6, where they spill: 288 against 268 us for the 48 cells), the
// loop unrolled by 2 (14.7 ms); a block per centre (its sums would depend on
// the number of centres, or cost 24 % where there are many).
//
// The r = 0 edge of the centre's own atom needs no test in the pair loop:
// its solid harmonics are (Y00, 0, ..., 0) and its table value is
// w(0) B_n0(0), so staging scales its R_00 by self_ratio = w0 / w(0) and the
// edge adds exactly w0 B_n0(0) Y00.  A stream whose species changes flushes
// its accumulators into the centre's coefficient buffer; streams flush one
// after the other, and in a fixed order at the end, so sums are
// deterministic.
template <int L, int NP>
struct NShape {
  static constexpr int K = (L + 1) * (L + 1);
  static constexpr int K4 = (K + 3) & ~3;  // row length in floats: float4 reads and writes
  static constexpr int H = 32 / NP;
  // coefficient rows c[s][n][0..K) also K4 floats apart: 16-byte aligned for the epilogue's
  // float4 reads, and the 8 rows n of a species (K4 = 4, 12, 16, 28, 36 or 52) start on 8
  // different groups of four banks
  static constexpr int KC = K4;
  // row q = h NP + j starts at q K4 + 4 h: the H streams' float4 reads of the
  // same slot fall on different groups of four banks whatever K4 is
  static constexpr int YF = 32 * K4 + 4 * H;
  // a multiple of 4 floats, so every warp's rows stay 16-byte aligned for the float4 accesses
  __host__ __device__ static int warp_floats(int S, int N) { return (YF + 4 * 32 + S * N * KC + 3) & ~3; }
};

// A radial-index lane's coefficients of one segment: interleaved l pairs and,
// for even L, l = 0.
template <int L, int NP>
struct LaneCoefs {
  static constexpr int NLP = (L + 1) / 2;
  f32x2 p[NLP > 0 ? NLP : 1][kNCoef];
  float s[kNCoef];
  // blk: the segment's first chunk of the lane's n; chunks NP float4 apart
  __device__ __forceinline__ void load(const float* __restrict__ blk) {
    const ulonglong2* q = reinterpret_cast<const ulonglong2*>(blk);
#pragma unroll
    for (int i = 0; i < NLP; ++i)
#pragma unroll
      for (int k = 0; k < kNCoef; k += 2) {
        const ulonglong2 v = __ldg(q + (i * (kNCoef / 2) + k / 2) * NP);
        p[i][k] = v.x;
        p[i][k + 1] = v.y;
      }
    if (L % 2 == 0) {
      const float4* f = reinterpret_cast<const float4*>(blk) + NLP * (kNCoef / 2) * NP;
      const float4 u = __ldg(f), v = __ldg(f + NP);
      s[0] = u.x; s[1] = u.y; s[2] = u.z; s[3] = u.w;
      s[4] = v.x; s[5] = v.y; s[6] = v.z; s[7] = v.w;
    }
  }
};

// A lane's accumulators, packed as its row's slots.
template <int L>
struct LaneSums {
  static constexpr int K = (L + 1) * (L + 1), NS = K / 2;
  f32x2 p[NS > 0 ? NS : 1];
  float s;
  __device__ __forceinline__ void clear() {
#pragma unroll
    for (int i = 0; i < NS; ++i) p[i] = 0ull;
    s = 0.0f;
  }
};

// One pair's contribution to a radial-index lane: the lane's l_max + 1 radial
// functions at t (Horner, two l per FMA), then acc[lm] += B_l R_lm over the
// pair's harmonic row, two slots per FMA.
template <int L, int NP, int K4>
__device__ __forceinline__ void accumulate_pair(LaneSums<L>& acc, const LaneCoefs<L, NP>& cf, f32x2 t2,
                                                const float* yrow) {
  using YO = YOrder<L>;
  constexpr int K = YO::K, NLP = YO::NLP;
  f32x2 B[NLP > 0 ? NLP : 1];
  float hi[NLP > 0 ? NLP : 1], lo[NLP > 0 ? NLP : 1], b0 = 0.0f;
#pragma unroll
  for (int i = 0; i < NLP; ++i) {
    f32x2 b = cf.p[i][kDeg];
#pragma unroll
    for (int k = kDeg - 1; k >= 0; --k) b = fma2(b, t2, cf.p[i][k]);
    B[i] = b;
    unpack2(b, hi[i], lo[i]);
  }
  if (L % 2 == 0) {
    float t, t_;
    unpack2(t2, t, t_);
    b0 = horner7(cf.s, t);
  }
  const ulonglong2* yr = reinterpret_cast<const ulonglong2*>(yrow);
#pragma unroll
  for (int q = 0; q < K4 / 4; ++q) {
    const ulonglong2 v = yr[q];
#pragma unroll
    for (int hh = 0; hh < 2; ++hh) {
      const int i = 2 * q + hh;  // slot pair: compile time
      const f32x2 y = hh ? v.y : v.x;
      if (i < YO::NS) {
        const int la = YO::l_of(kYOrder<L>.lm[2 * i]), lb = YO::l_of(kYOrder<L>.lm[2 * i + 1]);
        if (lb == la - 1) {
          acc.p[i] = fma2(B[(L - la) / 2], y, acc.p[i]);
        } else {  // two slots of larger l left over: scalar FMAs on the halves (a packed operand would take two moves)
          float ya, yb, sa, sb;
          unpack2(y, ya, yb);
          unpack2(acc.p[i], sa, sb);
          sa = fmaf(hi[(L - la) / 2], ya, sa);
          sb = fmaf(hi[(L - lb) / 2], yb, sb);
          acc.p[i] = pack2(sa, sb);
        }
      } else if (K % 2 == 1 && i == YO::NS) {
        float ya, yb;
        unpack2(y, ya, yb);
        acc.s = fmaf(b0, ya, acc.s);
      }
    }
  }
}

// Adds a lane's K accumulators to its 16-byte-aligned coefficient row (float4
// read-modify-write; the row's K4 - K padding slots stay zero).
template <int L, int K4>
__device__ __forceinline__ void flush_row(float* row, const LaneSums<L>& acc) {
  constexpr int K = (L + 1) * (L + 1);
  float4* r4 = reinterpret_cast<float4*>(row);
#pragma unroll
  for (int q = 0; q < K4 / 4; ++q) {
    const float4 v = r4[q];
    float w[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
    for (int hh = 0; hh < 2; ++hh) {
      const int i = 2 * q + hh;
      float x = 0.0f, y = 0.0f;
      if (i < K / 2) unpack2(acc.p[i], x, y);
      else if (K % 2 == 1 && i == K / 2) x = acc.s;
      if (2 * i < K) w[2 * hh] += x;
      if (2 * i + 1 < K) w[2 * hh + 1] += y;
    }
    r4[q] = make_float4(w[0], w[1], w[2], w[3]);
  }
}

// U: pairs of a batch without a species change that the loop is unrolled over.
template <int L, int NP, int U>
__device__ __forceinline__ void descriptor_n_body(const DescArgs& a) {
  using Sh = NShape<L, NP>;
  constexpr int K = Sh::K, K4 = Sh::K4, KC = Sh::KC, H = Sh::H;
  extern __shared__ __align__(16) float sm[];
  __shared__ float s_pref[kMaxL + 1];
  __shared__ int s_blk[2 * kMaxBlocks];
  __shared__ unsigned char s_tri[2 * kMaxTri];
  __shared__ unsigned char s_pos[K];  // row position of each lm
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  const int N = a.N, S = a.S;
  float* Y = sm + (size_t)wid * Sh::warp_floats(S, N);
  // per staged pair: segment coordinate (t, t), segment, species
  f32x2* tt = reinterpret_cast<f32x2*>(Y + Sh::YF);
  int* sg = reinterpret_cast<int*>(tt + 32);
  int* spp = sg + 32;
  float* cbuf = Y + Sh::YF + 4 * 32;
  desc_tables<L>(a, s_pref, s_blk, s_tri);
  for (int k = threadIdx.x; k < K; k += blockDim.x) s_pos[kYOrder<L>.lm[k]] = (unsigned char)k;
  __syncthreads();
  const int h = lane / NP, n = lane - h * NP;
  const float* tab = a.tab_p + 4 * n;  // this lane's first chunk of segment 0
  constexpr int seg_floats = NP * (L + 1) * kNCoef;
  bool first = true;
  const unsigned row_mask = NP == 8 ? 0x01010101u : 0x11111111u;  // row j of every stream's block, shifted by j
  const bool active = n < N;
  const int cbn = S * N * KC;
  float4* myrow = reinterpret_cast<float4*>(Y + lane * K4 + 4 * h);  // the row this lane stages

  for (;;) {
    int64_t c;
    if (a.counter) {
      int c32 = 0;
      if (lane == 0) c32 = atomicAdd(a.counter, 1);
      c = __shfl_sync(0xffffffffu, c32, 0);
    } else {
      c = first ? (int64_t)blockIdx.x * (blockDim.x >> 5) + wid : a.n_centres;
      first = false;
    }
    if (c >= a.n_centres) break;
    for (int i = lane; i < cbn / 4; i += 32) reinterpret_cast<float4*>(cbuf)[i] = make_float4(0.f, 0.f, 0.f, 0.f);
    // offsets inside the centre's list are 32-bit: 2^31 pairs of one centre would be 34 GB of list
    const int64_t p0 = a.pair_off[c];
    const int P = (int)(a.pair_off[c + 1] - p0);
    const float4* pc = a.pairs + p0;
    const int s0 = (int)(((int64_t)P * h) / H), s1 = (int)(((int64_t)P * (h + 1)) / H);  // this stream's pairs
    const int rounds = (P + H - 1) / H;                                                  // longest stream
    LaneSums<L> acc;
    acc.clear();
    LaneCoefs<L, NP> cf = {};
    // each stream starts on the species of its first pair, so the centre's first batch takes the
    // fast path unless a species changes inside it
    int cur_sp = (s0 < s1) ? (int)((unsigned)__float_as_int(__ldg(&pc[s0].w)) >> kAtomBits) : -1;
    int cur_seg = -1;
    __syncwarp();

    for (int base = 0; base < rounds; base += NP) {
      // stage: lane (h, n) takes pair s0 + base + n of its stream into row `lane`
      const int e = s0 + base + n;
      const bool valid = e < s1;
      const int nvalid = max(0, min(NP, s1 - (s0 + base)));  // this stream's block
      int seg = -1, sp = -1;
      float t = 0.0f;
      {
        // a row past the end of this stream is the harmonics of the origin, (Y00, 0, ..., 0),
        // with R_00 scaled to 0: a zero row that adds nothing
        float yv[K4];
#pragma unroll
        for (int k = K; k < K4; ++k) yv[k] = 0.0f;
        const float4 pr = valid ? __ldg(pc + e) : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        // the stream's pair of the next batch: into L1 while this batch runs
        if (e + NP < s1) asm volatile("prefetch.global.L1 [%0];" ::"l"(pc + e + NP));
        const float r = sqrtf(pr.x * pr.x + pr.y * pr.y + pr.z * pr.z);
        seg_coord(r, a.inv_h, a.nseg, seg, t);
        sp = (int)((unsigned)__float_as_int(pr.w) >> kAtomBits);
        SolidHarmonics<L>::values(pr.x, pr.y, pr.z, [&](int idx, float v) { yv[kYOrder<L>.pos[idx]] = v; });
        // the centre's own Gaussian (r = 0): w0 B_n0(0) Y00
        yv[kYOrder<L>.pos[0]] *= valid ? ((r > 0.0f) ? 1.0f : a.self_ratio) : 0.0f;
        if (!valid) {
          seg = -1;
          sp = -1;
          t = 0.0f;
        }
#pragma unroll
        for (int k4 = 0; k4 < K4 / 4; ++k4)
          myrow[k4] = make_float4(yv[4 * k4], yv[4 * k4 + 1], yv[4 * k4 + 2], yv[4 * k4 + 3]);
      }
      // rows past the end repeat the segment and species of the block's last pair (or the
      // stream's current ones), so they change nothing; then one bit per row marks where
      // the segment or the species differs from the stream's previous row
      const int last = h * NP + (nvalid > 0 ? nvalid - 1 : 0);
      const int seg_last = __shfl_sync(0xffffffffu, seg, last), sp_last = __shfl_sync(0xffffffffu, sp, last);
      if (!valid) {
        seg = nvalid > 0 ? seg_last : cur_seg;
        sp = nvalid > 0 ? sp_last : cur_sp;
      }
      int seg_prev = __shfl_up_sync(0xffffffffu, seg, 1), sp_prev = __shfl_up_sync(0xffffffffu, sp, 1);
      if (n == 0) {
        seg_prev = cur_seg;
        sp_prev = cur_sp;
      }
      const unsigned seg_chg = __ballot_sync(0xffffffffu, seg != seg_prev);
      const unsigned sp_chg = __ballot_sync(0xffffffffu, sp != sp_prev);
      tt[lane] = pack2(t, t);
      sg[lane] = seg;
      spp[lane] = sp;
      __syncwarp();
      if (sp_chg == 0) {
        // no species change in any stream: t, a coefficient reload where the segment changes,
        // Horner and the K FMAs per pair
#pragma unroll (U)
        for (int j = 0; j < NP; ++j) {
          const int q = h * NP + j;
          // one warp-uniform branch for the streams' reloads, kept a branch by the barrier: the ten
          // loads of a reload are otherwise issued, predicated off, for every pair
          if (seg_chg & (row_mask << j)) {
            __syncwarp();
            if (((seg_chg >> q) & 1u) && active) cf.load(tab + (size_t)sg[q] * seg_floats);
          }
          accumulate_pair<L, NP, K4>(acc, cf, tt[q], Y + q * K4 + 4 * h);
        }
      } else {
#pragma unroll 1
        for (int j = 0; j < NP; ++j) {
          const int q = h * NP + j;
          const int spq = spp[q];
          if (__any_sync(0xffffffffu, spq != cur_sp)) {
#pragma unroll
            for (int hh = 0; hh < H; ++hh) {  // streams flush one after the other
              if (h == hh && spq != cur_sp) {
                if (cur_sp >= 0 && active) {
                  flush_row<L, K4>(cbuf + (cur_sp * N + n) * KC, acc);
                }
                acc.clear();
                cur_sp = spq;
              }
              __syncwarp();
            }
          }
          if (seg_chg & (row_mask << j)) {
            __syncwarp();
            if (((seg_chg >> q) & 1u) && active) cf.load(tab + (size_t)sg[q] * seg_floats);
          }
          accumulate_pair<L, NP, K4>(acc, cf, tt[q], Y + q * K4 + 4 * h);
        }
      }
      cur_seg = sg[h * NP + NP - 1];
      cur_sp = spp[h * NP + NP - 1];
      __syncwarp();
    }
#pragma unroll
    for (int hh = 0; hh < H; ++hh) {
      if (h == hh && cur_sp >= 0 && active) {
        flush_row<L, K4>(cbuf + (cur_sp * N + n) * KC, acc);
      }
      __syncwarp();
    }
    desc_epilogue_n<L, KC>(a, c, cbuf, lane, s_pref, s_blk, s_tri, s_pos);
    __syncwarp();
  }
}

// l_max <= 4: 4 blocks of 4 warps per SM at 128 registers; l_max 5: 3 blocks; l_max 6: 2 blocks,
// so its 49 accumulators and 7 x 8 coefficients per lane stay in registers (at 3 blocks they spill).
// With few accumulators the unrolled loop's loads would take the registers of further blocks: 8 at
// l_max 0 and 6 at l_max 2 (96 cells of 4 species, n_max 8: 107 -> 88 and 180 -> 155 us).
constexpr int lane_blocks(int L) { return L == 0 ? 8 : L == 2 ? 6 : L <= 4 ? 4 : L == 5 ? 3 : 2; }
template <int L, int NP, int U>
__global__ void __launch_bounds__(128, lane_blocks(L)) k_descriptor_n(DescArgs a) {
  descriptor_n_body<L, NP, U>(a);
}

template <int L, int NP, int U = NP>
static int launch_descriptor_n(const DescArgs& a, int wpb_tuned, cudaStream_t st) {
  const int per_warp = 4 * NShape<L, NP>::warp_floats(a.S, a.N);
  if (per_warp % 16 != 0) return set_error(SOAPB_ERR_ARG, "descriptor: warp slice of %d B not 16-byte aligned", per_warp);
  int wpb = (200 * 1024) / per_warp;
  wpb = wpb > 4 ? 4 : wpb;
  if ((wpb_tuned == 1 || wpb_tuned == 2 || wpb_tuned == 4) && wpb_tuned <= wpb) wpb = wpb_tuned;
  if (wpb < 1) return set_error(SOAPB_ERR_UNSUPPORTED, "descriptor shared memory %d B per warp too large", per_warp);
  const int smem = wpb * per_warp;
  auto kern = k_descriptor_n<L, NP, U>;
  int rc = check_cuda(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, smem),
                      "descriptor smem attribute");
  if (rc) return rc;
  int dev = 0, nsm = 148, occ = 1;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev);
  cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, kern, 32 * wpb, smem);
  if (occ < 1) occ = 1;
  int64_t blocks = (int64_t)nsm * occ;
  const int64_t need = (a.n_centres + wpb - 1) / wpb;
  DescArgs b = a;
  if (blocks >= need) {  // one centre per warp: no work queue to reset
    blocks = need;
    b.counter = nullptr;
  } else if ((rc = check_cuda(cudaMemsetAsync(a.counter, 0, sizeof(int32_t), st), "reset work counter"))) {
    return rc;
  }
  kern<<<(unsigned)blocks, 32 * wpb, smem, st>>>(b);
  return check_launch("k_descriptor_n");
}

template <int L, int GN, int H>
static int launch_descriptor(const DescArgs& a, int wpb_tuned, cudaStream_t st) {
  const int per_warp =
      4 * ((H == 2) ? DescShape<L>::warp_floats(a.S, a.N) : DescShape<L>::warp_floats16(a.S, a.N));
  int wpb = (200 * 1024) / per_warp;
  wpb = wpb > 4 ? 4 : wpb;
  if ((wpb_tuned == 1 || wpb_tuned == 2 || wpb_tuned == 4) && wpb_tuned <= wpb) wpb = wpb_tuned;
  if (wpb < 1) return set_error(SOAPB_ERR_UNSUPPORTED, "descriptor shared memory %d B per warp too large", per_warp);
  const int smem = wpb * per_warp;
  auto kern = [] {
    if constexpr (H == 2) return k_descriptor_2s<L, GN>;
    else return k_descriptor<L, GN>;
  }();
  int rc = check_cuda(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, smem),
                      "descriptor smem attribute");
  if (rc) return rc;
  int dev = 0, nsm = 148, occ = 1;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev);
  cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, kern, 32 * wpb, smem);
  if (occ < 1) occ = 1;
  int64_t blocks = (int64_t)nsm * occ;
  const int64_t need = (a.n_centres + wpb - 1) / wpb;
  if (blocks > need) blocks = need;
  if ((rc = check_cuda(cudaMemsetAsync(a.counter, 0, sizeof(int32_t), st), "reset work counter"))) return rc;
  kern<<<(unsigned)blocks, 32 * wpb, smem, st>>>(a);
  return check_launch("k_descriptor");
}

template <int L>
struct DescDispatch {
  static int run(const DescArgs& a, int gn, int wpb, bool lgroup_only, cudaStream_t st) {
    if constexpr (L <= kMaxLNLanes) {
      if (!lgroup_only && radial_lanes(a.N, L) && isfinite(a.self_ratio)) {
        // At l_max 6 a pair's 49 FMAs and 7 Horner passes are long enough that the unrolled loop, and
        // the one for batches with a species change, exceed what the instruction caches hold: rolled
        // with 4 lanes (512 cells, 4 species: 2718 -> 2196 us; 20000 atoms of one species: 391 -> 399),
        // and with 8 from 3 species on (2634 -> 2495 us; 2001 atoms of 2 species: 75 -> 79).  At
        // l_max 4 with 8 lanes unrolled: 14.05 ms for 1M atoms, 14.7 unrolled by 2; with 4 lanes, whose
        // streams are shorter, rolled from l_max 4 on (96 cells of 4 species: 227 -> 212 us, l_max 5 296 -> 269).
        if (a.N <= 4) return launch_descriptor_n<L, 4, (L >= 4 ? 1 : 4)>(a, wpb, st);
        if constexpr (L == 6)
          if (a.S >= 3) return launch_descriptor_n<L, 8, 1>(a, wpb, st);
        return launch_descriptor_n<L, 8>(a, wpb, st);
      }
    }
    if constexpr (L <= 4) {
      if (desc_two_streams(a.N, L)) {  // functions per lane fixed by (N, L): ceil(N / floor(16 / (L+1)))
        const int lpl = 16 / (L + 1), g2 = (a.N + lpl - 1) / lpl;
        switch (g2) {
          case 1: return launch_descriptor<L, 1, 2>(a, wpb, st);
          case 2: return launch_descriptor<L, 2, 2>(a, wpb, st);
          default: return launch_descriptor<L, 3, 2>(a, wpb, st);
        }
      }
    }
    if constexpr (L >= 10) {  // two lanes per l: 4 radial functions per lane cover n_max <= 8
      if (a.N > 8) return set_error(SOAPB_ERR_UNSUPPORTED, "descriptor: l_max %d is built for n_max <= 8", L);
      return launch_descriptor<L, 4, 1>(a, wpb, st);
    } else {
      switch (gn) {
        case 1: return launch_descriptor<L, 1, 1>(a, wpb, st);
        case 2: return launch_descriptor<L, 2, 1>(a, wpb, st);
        case 3: return launch_descriptor<L, 3, 1>(a, wpb, st);
        case 4: return launch_descriptor<L, 4, 1>(a, wpb, st);
        case 6: return launch_descriptor<L, 6, 1>(a, wpb, st);
        default: return set_error(SOAPB_ERR_UNSUPPORTED, "descriptor: %d radial functions per lane not built", gn);
      }
    }
  }
};

}  // namespace soapb

using namespace soapb;

extern "C" int soapb_descriptor(const soapb_basis* b, int64_t n_centres, const int64_t* d_pair_off,
                                const void* d_pairs, int32_t out_mode, float* d_out, float* d_coeff,
                                int32_t* d_counter, void* stream) {
  if (!b || !b->dev) return set_error(SOAPB_ERR_ARG, "basis not built");
  if (n_centres < 0 || n_centres >= (int64_t)1 << 31) return set_error(SOAPB_ERR_ARG, "bad n_centres");
  if (out_mode != SOAPB_OUT_PS && out_mode != SOAPB_OUT_CC && out_mode != SOAPB_OUT_RAW)
    return set_error(SOAPB_ERR_ARG, "bad out_mode");
  if (n_centres == 0) return SOAPB_OK;
  if (!d_pair_off || !d_out || !d_counter) return set_error(SOAPB_ERR_ARG, "null argument");
  const int N = b->n_max, L = b->l_max;
  cudaStream_t st = (cudaStream_t)stream;
  DescArgs a;
  a.pair_off = d_pair_off;
  a.pairs = (const float4*)d_pairs;
  a.n_centres = n_centres;
  a.tab_b = (const float*)((const char*)b->dev + b->off_tab_b);
  a.tab_p = (const float*)((const char*)b->dev + off_tab_pairs(b));
  a.selfv = (const float*)((const char*)b->dev + b->off_self);
  a.out = d_out;
  a.coeff_out = d_coeff;
  a.counter = d_counter;
  a.N = N;
  a.S = b->n_species;
  a.nseg = b->n_seg;
  a.F = out_mode == SOAPB_OUT_PS ? b->n_feat_ps : b->n_feat_cc;
  a.mode = out_mode;
  a.crossover = b->crossover ? 1 : 0;
  a.inv_h = (float)(1.0 / b->seg_width);
  {
    // self_ratio = w0 / w(0) of the weighting (the r = 0 table value is w(0) B_n0(0)); not finite
    // (a weighting singular at r = 0) sends the call to the kernels that use the self table
    const double w0 = b->weighting == SOAPB_W_NONE ? 1.0 : b->w_w0;
    double w_at0 = 1.0;
    if (b->weighting == SOAPB_W_POLY) w_at0 = b->w_c;
    else if (b->weighting == SOAPB_W_POW) w_at0 = b->w_c / (b->w_d + pow(0.0, b->w_m));
    else if (b->weighting == SOAPB_W_EXP) w_at0 = b->w_c / (b->w_d + 1.0);
    a.self_ratio = (float)(w0 / w_at0);
  }
  int gn = desc_group(N, L);
  const int tg = b->tune[1];
  if (tg > gn && (tg == 2 || tg == 3 || tg == 4 || tg == 6)) gn = tg;
  return dispatch_l<DescDispatch>(L, a, gn, b->tune[0], b->tune[3] == 1, st);
}
