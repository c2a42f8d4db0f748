// Cell-list radius neighbour search into a per-centre CSR pair list.
//
// Reference: SOAP._build_neighbor_list (soap_generator.py:1128-1181),
// _radius_edges (:1042-1125), _extend_periodic (:1015-1021), _pbc_offsets
// (:382-396) and _perpendicular_lengths (:369-379).  The reference
// replicates every atom over all (2 n_rep + 1)^3 image offsets and runs an
// all-pairs GEMM distance test; here atoms are binned once per structure
// (counting sort into bins in the cell's fractional frame, a quarter or half of
// the cutoff wide, periodic axes wrapped) and each centre scans only the runs of
// bins that its cutoff sphere reaches, generating images on the fly.  The image
// set is the reference's: image offset n = T - w_atom + w_centre (T the
// cell-window shift, w the wrap shifts) must satisfy |n_i| <= n_rep_i on
// periodic axes.
//
// Pairs of a centre are written sorted by (neighbour species, radial table
// segment) -- the order the descriptor kernels consume them in -- and, inside
// a key, by bin (z, y, x, counted on through the images) and atom index.  That
// order fixes the FP32 sums over a centre's neighbours, so the bins (grid_setup,
// locate) are part of the results: they are computed in FP64, and another width
// or another order of the images moves every gradient in its last digits.
// Whether a candidate is within the cutoff is decided in FP64: FP32 copies of
// the positions decide all candidates but those within their rounding of the
// cutoff.  Differences are taken in FP64; rvec is stored FP32.
#include <math.h>

#include <mutex>

#include "common.cuh"

namespace soapb {

struct GridDesc {
  double H[9];     // rows: lattice a, b, c (identity for non-periodic structures)
  double Hinv[9];  // f_j = sum_i x_i Hinv[i*3+j]
  double fmin[3];  // bin origin in fractional coordinates (non-periodic axes)
  double binw[3];  // fractional bin width (locate)
  double ibinw[3]; // bins per fractional unit (the window)
  int nrep[3];
  int wrapped;     // an atom has a wrap shift: pairs need the image test
  short nb[3];
  signed char per[3];
  signed char orth;  // 1: diagonal frame (every non-periodic structure, rectangular cells), 0: another,
                     // -1: no frame (a periodic cell without a volume, or so thin that its images
                     // could not be counted, or not of numbers): no pairs
  signed char wide;  // an axis has more images than pack3 holds: image shifts in pack_wide
  // FP32 geometry of the window (Angstrom): perpendicular bin widths; for other than diagonal
  // frames the direction of lattice row a, the reciprocal of a bin's length along it, the edges
  // of a bin along b and c, and the largest distance of a bin's point from the bin row's axis
  float wp[3], dir[3], ialong, eb[3], ec[3], rho;
  // squared FP32 distances up to c2lo are within the cutoff, above c2hi beyond it
  float c2lo, c2hi;
  __device__ __forceinline__ bool any_per() const { return (per[0] | per[1] | per[2]) != 0; }
};
// the workspace per structure must not grow: soapb_neighbors_noalloc has a fixed one
static_assert(sizeof(GridDesc) <= 312, "GridDesc");

struct NLWork {
  GridDesc* grids;
  unsigned long long* fbox;  // (n_struct, 6) ordered-int encodings of fractional min/max
  int* bins_per_struct;      // (n_struct)
  int64_t* bin_off;          // (n_struct + 1)
  int* bin_count;            // (max_bins)
  int* bin_start;            // (max_bins + 1)
  int* arrival;              // (n_atoms) order in which the atoms reached their bins (in sorted_f's memory)
  int* atom_bin;             // (n_atoms)
  int* sorted_atom;          // (n_atoms) atoms by bin, in arrival order inside a bin
  double4* sorted_pos;       // (n_atoms) {wrapped x, y, z, packed info} (see pack_info)
  float4* sorted_f;          // (n_atoms) {x, y, z} of sorted_pos from the origin of coord_origin
  double4* cpos;             // (n_centres) wrapped centre positions
  int4* cinfo;               // (n_centres) {bin xyz, struct, wrap, atom}
  int* counts;               // (n_centres)
  int64_t* partials;         // scan partials
  int* status;               // {error flags, finished blocks of k_count, largest pair count of a centre, 0}
  int64_t max_bins;
};

// ---------------------------------------------------------------------------
// helpers
// ---------------------------------------------------------------------------

__device__ __forceinline__ unsigned long long ord_encode(double v) {
  unsigned long long b = (unsigned long long)__double_as_longlong(v);
  return (b >> 63) ? ~b : (b | 0x8000000000000000ull);
}
__host__ __device__ inline double ord_decode(unsigned long long e) {
  unsigned long long b = (e >> 63) ? (e & 0x7fffffffffffffffull) : ~e;
#ifdef __CUDA_ARCH__
  return __longlong_as_double((long long)b);
#else
  double d;
  memcpy(&d, &b, 8);
  return d;
#endif
}

__device__ __forceinline__ int pack3(int a, int b, int c) { return (a + 512) | ((b + 512) << 10) | ((c + 512) << 20); }
__device__ __forceinline__ void unpack3(int p, int (&v)[3]) {
  v[0] = (p & 1023) - 512;
  v[1] = ((p >> 10) & 1023) - 512;
  v[2] = ((p >> 20) & 1023) - 512;
}
// Cell-window shifts of a frame with more images than 10 bits hold (a cell thinner
// than about cutoff / 500): fields as wide as the axes need.
constexpr int kPackedReps = 508;  // largest n_rep of pack3 (the window reaches one cell further)
__device__ __forceinline__ int shift_bits(int nrep) { return 32 - __clz(2 * (nrep + 2)); }
__device__ __forceinline__ int pack_wide(const int* nrep, int a, int b, int c) {
  const int s1 = shift_bits(nrep[0]), s2 = s1 + shift_bits(nrep[1]);
  return (int)((unsigned)(a + nrep[0] + 2) | (unsigned)(b + nrep[1] + 2) << s1 | (unsigned)(c + nrep[2] + 2) << s2);
}
__device__ __forceinline__ void unpack_wide(const int* nrep, int p, int (&v)[3]) {
  const int s1 = shift_bits(nrep[0]), s2 = s1 + shift_bits(nrep[1]);
  const unsigned u = (unsigned)p;
  v[0] = (int)(u & ((1u << s1) - 1u)) - nrep[0] - 2;
  v[1] = (int)((u >> s1) & ((1u << (s2 - s1)) - 1u)) - nrep[1] - 2;
  v[2] = (int)(u >> s2) - nrep[2] - 2;
}
// atom (27 bits) | species (5 bits) | packed wrap shifts (30 bits), carried in
// the fourth double of a sorted-atom record so a candidate is one 32-byte load
// (the bits are only moved, never used as a floating-point value).
__device__ __forceinline__ double pack_info(int atom, int sp, int wrap) {
  const unsigned long long bits = (unsigned long long)(unsigned)atom | ((unsigned long long)(unsigned)sp << kAtomBits) |
                                  ((unsigned long long)(unsigned)wrap << 32);
  return __longlong_as_double((long long)bits);
}
__device__ __forceinline__ void unpack_info(double w, int& atom, int& sp, int& wrap) {
  const unsigned long long bits = (unsigned long long)__double_as_longlong(w);
  atom = (int)(bits & kAtomMask);
  sp = (int)((bits >> kAtomBits) & 31u);
  wrap = (int)(bits >> 32);
}
__device__ __forceinline__ int floordiv(int a, int b) { return (a >= 0) ? a / b : -((-a + b - 1) / b); }

__device__ __forceinline__ int struct_of_atom(const int64_t* atom_off, int n_struct, int64_t a) {
  int lo = 0, hi = n_struct - 1;
  while (lo < hi) {
    const int mid = (lo + hi + 1) >> 1;
    if (atom_off[mid] <= a) lo = mid; else hi = mid - 1;
  }
  return lo;
}

// Arithmetic that decides a bin or a pair has its roundings written out: it is done in several
// kernels (bins and records, count and fill), which have to agree to the last bit where an atom
// lies on the edge of a bin or a pair at the cutoff.
__device__ __forceinline__ void to_frac(const GridDesc& g, double x, double y, double z, double (&f)[3]) {
#pragma unroll
  for (int j = 0; j < 3; ++j) f[j] = fma(z, g.Hinv[6 + j], fma(x, g.Hinv[j], __dmul_rn(y, g.Hinv[3 + j])));
}

// Component k of t[0] a + t[1] b + t[2] c.
__device__ __forceinline__ double lattice_sum(const double* H, const int (&t)[3], int k) {
  return fma((double)t[2], H[6 + k], fma((double)t[0], H[k], __dmul_rn((double)t[1], H[3 + k])));
}

// Bin, wrap shift and wrapped position of a point of structure g.
__device__ __forceinline__ bool locate(const GridDesc& g, double x, double y, double z, int (&b)[3], int (&w)[3],
                                       double (&wp)[3]) {
  double f[3];
  to_frac(g, x, y, z, f);
  bool ok = true;
#pragma unroll
  for (int i = 0; i < 3; ++i) {
    if (g.per[i]) {
      const double fl = floor(f[i]);
      w[i] = (int)fl;
      double fr = f[i] - fl;
      int bi = (int)(fr * g.nb[i]);
      b[i] = min(max(bi, 0), g.nb[i] - 1);
      ok &= (w[i] > -512 && w[i] < 511);
    } else {
      w[i] = 0;
      const int bi = (int)floor((f[i] - g.fmin[i]) / g.binw[i]);
      b[i] = min(max(bi, 0), g.nb[i] - 1);
    }
  }
  wp[0] = __dsub_rn(x, lattice_sum(g.H, w, 0));
  wp[1] = __dsub_rn(y, lattice_sum(g.H, w, 1));
  wp[2] = __dsub_rn(z, lattice_sum(g.H, w, 2));
  return ok;
}

// ---------------------------------------------------------------------------
// exclusive scan int32 -> int64 (n + 1 outputs)
// ---------------------------------------------------------------------------

__device__ __forceinline__ int64_t block_incl_scan(int64_t v, int64_t* s_warp) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int64_t t = __shfl_up_sync(0xffffffffu, v, o);
    if (lane >= o) v += t;
  }
  if (lane == 31) s_warp[warp] = v;
  __syncthreads();
  if (warp == 0) {
    int64_t w = (lane < (int)(blockDim.x >> 5)) ? s_warp[lane] : 0;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int64_t t = __shfl_up_sync(0xffffffffu, w, o);
      if (lane >= o) w += t;
    }
    s_warp[lane] = w;
  }
  __syncthreads();
  if (warp > 0) v += s_warp[warp - 1];
  return v;
}

template <class Out>
__global__ void __launch_bounds__(1024) k_scan_blocks(const int* in, int64_t n, Out* out, int64_t* partials) {
  __shared__ int64_t s_warp[32];
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  const int64_t v = (i < n) ? in[i] : 0;
  const int64_t inc = block_incl_scan(v, s_warp);
  if (i < n) out[i] = (Out)(inc - v);
  if (threadIdx.x == blockDim.x - 1) partials[blockIdx.x] = inc;
}

template <class Out>
__global__ void __launch_bounds__(1024) k_scan_partials(int64_t* partials, int64_t nblk, Out* total_out) {
  __shared__ int64_t s_warp[32];
  __shared__ int64_t s_carry;
  if (threadIdx.x == 0) s_carry = 0;
  __syncthreads();
  for (int64_t base = 0; base < nblk; base += blockDim.x) {
    const int64_t i = base + threadIdx.x;
    const int64_t v = (i < nblk) ? partials[i] : 0;
    const int64_t inc = block_incl_scan(v, s_warp);
    const int64_t carry = s_carry;
    if (i < nblk) partials[i] = carry + inc - v;
    __syncthreads();
    if (threadIdx.x == blockDim.x - 1) s_carry = carry + inc;
    __syncthreads();
  }
  if (threadIdx.x == 0) *total_out = (Out)s_carry;
}

template <class Out>
__global__ void k_scan_add(Out* out, int64_t n, const int64_t* partials) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) out[i] += (Out)partials[i / 1024];
}

template <class Out>
static int exclusive_scan(const int* in, int64_t n, Out* out, int64_t* partials, cudaStream_t st) {
  const int64_t nblk = (n + 1023) / 1024;
  if (n > 0) {
    k_scan_blocks<<<(unsigned)nblk, 1024, 0, st>>>(in, n, out, partials);
  }
  k_scan_partials<<<1, 1024, 0, st>>>(partials, nblk, out + n);
  if (n > 0) k_scan_add<<<(unsigned)((n + 255) / 256), 256, 0, st>>>(out, n, partials);
  return check_launch("exclusive_scan", n > 0 ? 3 : 1);
}

// Exclusive scan of n ints by one block: every thread sums a contiguous chunk,
// one block scan of the sums, then the chunk's offsets.  The inputs were
// written by other blocks of the same launch: they are read from L2.  Returns
// the total (every thread) and, in *largest, the largest input.
template <class Out>
__device__ __forceinline__ int64_t block_scan_chunks(const int* in, int64_t n, Out* out, int64_t* s_warp,
                                                     int* s_max, int* largest) {
  const int nth = blockDim.x;
  // chunks of a multiple of 4, loaded as int4 (in is 16-byte aligned)
  const int64_t per = ((n + nth - 1) / nth + 3) & ~(int64_t)3;
  const int64_t i0 = min((int64_t)threadIdx.x * per, n), i1 = min(i0 + per, n);
  auto load4 = [&](int64_t i, int (&v)[4]) {
    if (i + 4 <= i1) {
      const int4 q = __ldcg(reinterpret_cast<const int4*>(in + i));
      v[0] = q.x; v[1] = q.y; v[2] = q.z; v[3] = q.w;
    } else {
#pragma unroll
      for (int k = 0; k < 4; ++k) v[k] = i + k < i1 ? __ldcg(in + i + k) : 0;
    }
  };
  int64_t sum = 0;
  int mx = 0;
#pragma unroll 4
  for (int64_t i = i0; i < i1; i += 4) {
    int v[4];
    load4(i, v);
    sum += (int64_t)v[0] + v[1] + v[2] + v[3];
    mx = max(max(mx, max(v[0], v[1])), max(v[2], v[3]));
  }
  mx = __reduce_max_sync(0xffffffffu, mx);
  if ((threadIdx.x & 31) == 0) s_max[threadIdx.x >> 5] = mx;
  const int64_t inc = block_incl_scan(sum, s_warp);
  int64_t run = inc - sum;
  int next[4];
  load4(i0, next);
  for (int64_t i = i0; i < i1; i += 4) {  // the next four are loaded before these are stored
    const int v[4] = {next[0], next[1], next[2], next[3]};
    load4(i + 4, next);
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      if (i + k < i1) out[i + k] = (Out)run;
      run += v[k];
    }
  }
  __syncthreads();
  if (largest) {
    int m = 0;
    for (int k = 0; k < (nth >> 5); ++k) m = max(m, s_max[k]);
    *largest = m;
  }
  const int64_t total = s_warp[(nth >> 5) - 1];  // inclusive sum up to the last warp
  if (threadIdx.x == 0) out[n] = (Out)total;
  return total;
}

// ---------------------------------------------------------------------------
// cell lists
// ---------------------------------------------------------------------------

// Each stage below is a device function over (index, stride), so the separate
// kernels of large inputs and the fused kernel of small ones (k_cells) share it.
__device__ __forceinline__ void grid_init(const soapb_structs& s, const NLWork& w, double cutoff, int i) {
  GridDesc g;
  int anyp = 0;
  for (int k = 0; k < 3; ++k) anyp |= s.d_pbc[i * 3 + k] ? 1 : 0;
  for (int k = 0; k < 9; ++k) g.H[k] = anyp ? s.d_cells[i * 9 + k] : ((k % 4 == 0) ? 1.0 : 0.0);
  const double* H = g.H;
  // inverse of the row-vector matrix: x = f H  =>  f = x H^-1.  The roundings are written out: the
  // bin of an atom on a bin's edge (a lattice site of a skewed cell) depends on the last one.
  auto minor = [&](int a, int b, int c, int d) { return fma(H[a], H[b], -__dmul_rn(H[c], H[d])); };
  const double m0 = minor(4, 8, 5, 7), m6 = minor(3, 7, 4, 6);
  const double m3 = __dsub_rn(__dmul_rn(H[3], H[8]), __dmul_rn(H[5], H[6]));
  const double det = fma(H[2], m6, fma(H[0], m0, -__dmul_rn(H[1], m3)));
  const double id = !anyp ? 1.0 : fabs(det) < 1e-300 ? 0.0 : 1.0 / det;
  g.Hinv[0] = m0 * id;
  g.Hinv[1] = minor(2, 7, 1, 8) * id;
  g.Hinv[2] = minor(1, 5, 2, 4) * id;
  g.Hinv[3] = minor(5, 6, 3, 8) * id;
  g.Hinv[4] = minor(0, 8, 2, 6) * id;
  g.Hinv[5] = minor(2, 3, 0, 5) * id;
  g.Hinv[6] = m6 * id;
  g.Hinv[7] = minor(1, 6, 0, 7) * id;
  g.Hinv[8] = minor(0, 4, 1, 3) * id;
  for (int k = 0; k < 3; ++k) {
    g.per[k] = anyp ? (s.d_pbc[i * 3 + k] ? 1 : 0) : 0;
    g.fmin[k] = 0.0;
    g.binw[k] = g.ibinw[k] = 1.0;
    g.nb[k] = 1;
    g.nrep[k] = 0;
  }
  g.wrapped = 0;
  g.orth = 1;
  for (int k = 0; k < 9; ++k)
    if (k % 4 == 0 ? !(H[k] > 0.0) : H[k] != 0.0) g.orth = 0;
  if (anyp && !(fabs(det) >= 1e-300 && fabs(det) < INFINITY)) g.orth = -1;
  // perpendicular widths |det| / |cross of the other two rows| (SG:369-379)
  if (anyp)
    for (int k = 0; k < 3; ++k) {
      const double* u = H + 3 * ((k + 1) % 3);
      const double* v = H + 3 * ((k + 2) % 3);
      const double cx = u[1] * v[2] - u[2] * v[1], cy = u[2] * v[0] - u[0] * v[2], cz = u[0] * v[1] - u[1] * v[0];
      const double perp = fabs(det) / (sqrt(cx * cx + cy * cy + cz * cz) + 1e-12);
      if (g.per[k]) g.nrep[k] = (int)ceil(cutoff / (perp + 1e-12));  // SG:389
    }
  g.wide = max(g.nrep[0], max(g.nrep[1], g.nrep[2])) > kPackedReps;
  // thinner than a millionth of the cutoff (vectors in a plane, up to rounding): millions of images
  for (int k = 0; k < 3; ++k)
    if (g.nrep[k] > 1 << 20) g.orth = -1;
  if (g.orth >= 0 && shift_bits(g.nrep[0]) + shift_bits(g.nrep[1]) + shift_bits(g.nrep[2]) > 32) g.orth = -1;
  w.grids[i] = g;
  for (int k = 0; k < 3; ++k) {
    w.fbox[i * 6 + k] = ord_encode(INFINITY);
    w.fbox[i * 6 + 3 + k] = ord_encode(-INFINITY);
  }
}

// Smallest (largest) key of a warp: the high words, then the low words of those that have it.
__device__ __forceinline__ unsigned long long warp_min(unsigned long long v) {
  const unsigned hi = (unsigned)(v >> 32), h = __reduce_min_sync(0xffffffffu, hi);
  const unsigned l = __reduce_min_sync(0xffffffffu, hi == h ? (unsigned)v : 0xffffffffu);
  return (unsigned long long)h << 32 | l;
}
__device__ __forceinline__ unsigned long long warp_max(unsigned long long v) { return ~warp_min(~v); }

// Fractional bounding box of the open axes of every structure (warp-strided
// over atoms base = first, first + stride, ...), without atoms whose
// coordinate is NaN.  Atoms of a structure are contiguous, so a warp keeps a
// running minimum and maximum while its atoms belong to one structure and
// issues atomics only when the structure changes or its atoms end.
__device__ __forceinline__ void frac_bbox(const soapb_structs& s, const NLWork& w, int64_t first, int64_t stride) {
  const int lane = threadIdx.x & 31;
  int cur = -1;  // structure of the running bounds (warp-uniform)
  unsigned long long lo[3], hi[3];
  auto flush = [&]() {
    if (cur < 0) return;
#pragma unroll
    for (int k = 0; k < 3; ++k) {
      const unsigned long long l = warp_min(lo[k]), h = warp_max(hi[k]);
      if (lane == 0 && !w.grids[cur].per[k]) {
        atomicMin(&w.fbox[cur * 6 + k], l);
        atomicMax(&w.fbox[cur * 6 + 3 + k], h);
      }
    }
  };
  for (int64_t base = first; base < s.n_atoms; base += stride) {
    const int64_t a = base + lane;
    const bool valid = a < s.n_atoms;
    int si = 0;
    unsigned long long key[3];
    bool num[3] = {false, false, false};
    if (valid) {
      si = struct_of_atom(s.d_atom_off, s.n_struct, a);
      double f[3];
      to_frac(w.grids[si], s.d_positions[3 * a], s.d_positions[3 * a + 1], s.d_positions[3 * a + 2], f);
#pragma unroll
      for (int k = 0; k < 3; ++k) {
        key[k] = ord_encode(f[k]);
        num[k] = f[k] == f[k];
      }
    }
    const int si0 = __shfl_sync(0xffffffffu, si, 0);  // lane 0 is always valid here
    if (__all_sync(0xffffffffu, !valid || si == si0)) {
      if (si0 != cur) {
        flush();
        cur = si0;
#pragma unroll
        for (int k = 0; k < 3; ++k) { lo[k] = ~0ull; hi[k] = 0ull; }
      }
#pragma unroll
      for (int k = 0; k < 3; ++k)
        if (num[k]) { lo[k] = min(lo[k], key[k]); hi[k] = max(hi[k], key[k]); }
    } else {
      for (int k = 0; k < 3; ++k) {
        if (!num[k] || w.grids[si].per[k]) continue;
        atomicMin(&w.fbox[si * 6 + k], key[k]);
        atomicMax(&w.fbox[si * 6 + 3 + k], key[k]);
      }
    }
  }
  flush();
}

__device__ __forceinline__ void grid_setup(const soapb_structs& s, const NLWork& w, double cutoff, int i) {
  GridDesc g = w.grids[i];
  const double* H = g.H;
  // (roundings written out: a width of a whole number of bins, up to the last bit, sets that number)
  auto minor = [](double a, double b, double c, double d) { return fma(a, b, -__dmul_rn(c, d)); };
  const double det = fabs(fma(H[2], minor(H[3], H[7], H[4], H[6]),
                              fma(H[0], minor(H[4], H[8], H[5], H[7]),
                                  -__dmul_rn(H[1], minor(H[3], H[8], H[5], H[6])))));
  if (g.orth < 0) {  // one bin of which nothing is visited (its window would have no end)
    // (flagged here, behind a barrier from the clear of the flags)
    if (det < INFINITY) atomicOr(w.status, 1);
    w.bins_per_struct[i] = 1;
    if (s.n_struct == 1) {
      w.bin_off[0] = 0;
      w.bin_off[1] = 1;
    }
    return;
  }
  double perp[3] = {1.0, 1.0, 1.0}, binw[3];
  if (g.any_per())
    for (int k = 0; k < 3; ++k) {
      const double* u = H + 3 * ((k + 1) % 3);
      const double* v = H + 3 * ((k + 2) % 3);
      const double cx = minor(u[1], v[2], u[2], v[1]), cy = minor(u[2], v[0], u[0], v[2]),
                   cz = minor(u[0], v[1], u[1], v[0]);
      perp[k] = det / (sqrt(fma(cz, cz, fma(cx, cx, __dmul_rn(cy, cy)))) + 1e-300);
    }
  const int64_t A = s.d_atom_off[i + 1] - s.d_atom_off[i];
  // Bins of perpendicular width >= cutoff / 4 in diagonal frames, unless a
  // periodic x axis would get fewer than 3 of them, and >= cutoff / 2 in the
  // others; every bin row of the window is trimmed to the cutoff sphere (visit).
  // The line is where it always was: the bins set the order of the pairs.
  // Quarter bins everywhere would gain little (501 atoms, triclinic: count 18
  // instead of 19 us, fill 22 instead of 23).
  const double bin_min = (g.orth && !(g.per[0] && perp[0] < 0.75 * cutoff) ? 0.25 : 0.5) * cutoff;
  double far[3];  // largest |fractional coordinate| of a wrapped atom, from the origin of the FP32 copies
  for (int k = 0; k < 3; ++k) {
    if (g.per[k]) {
      const int nb = (int)floor(perp[k] / bin_min);
      g.nb[k] = min(max(nb, 1), 1023);
      g.fmin[k] = 0.0;
      binw[k] = 1.0 / g.nb[k];
      far[k] = 1.0;
    } else {
      double lo = ord_decode(__ldcg(&w.fbox[i * 6 + k])), hi = ord_decode(__ldcg(&w.fbox[i * 6 + 3 + k]));
      if (!(hi >= lo)) { lo = 0.0; hi = 0.0; }  // no atoms
      const double span = hi - lo;
      far[k] = g.any_per() ? fmax(fabs(lo), fabs(hi)) : span;
      const int nb = (int)floor(span * perp[k] / bin_min);
      g.nb[k] = min(max(nb, 1), 1023);
      g.fmin[k] = lo;
      binw[k] = span > 0.0 ? span / g.nb[k] : 1.0;
    }
  }
  // cap the bin count of the structure at 2 A + 8
  const int64_t cap = 2 * A + 8;
  while ((int64_t)g.nb[0] * g.nb[1] * g.nb[2] > cap) {
    int k = 0;
    if (g.nb[1] > g.nb[k]) k = 1;
    if (g.nb[2] > g.nb[k]) k = 2;
    const double span = binw[k] * g.nb[k];
    g.nb[k] = max(1, g.nb[k] / 2);
    binw[k] = span / g.nb[k];
  }
  for (int k = 0; k < 3; ++k) {
    g.binw[k] = binw[k];
    // a single bin of an open axis may be as thin as its atoms; the window takes it at least 1e-3 A wide
    if (!g.per[k] && g.nb[k] == 1) binw[k] = fmax(binw[k], 1e-3 / perp[k]);
    g.ibinw[k] = 1.0 / binw[k];
    g.wp[k] = (float)(binw[k] * perp[k]);
  }
  if (!g.orth) {
    const double la = sqrt(H[0] * H[0] + H[1] * H[1] + H[2] * H[2]);
    double p2 = 0.0, m2 = 0.0;
    for (int k = 0; k < 3; ++k) {
      const double eb = binw[1] * H[3 + k], ec = binw[2] * H[6 + k];
      g.dir[k] = (float)(la > 0.0 ? H[k] / la : 0.0);
      g.eb[k] = (float)eb;
      g.ec[k] = (float)ec;
      p2 += (eb + ec) * (eb + ec);
      m2 += (eb - ec) * (eb - ec);
    }
    g.ialong = (float)(1.0 / (binw[0] * la));
    g.rho = (float)(0.5 * sqrt(fmax(p2, m2)) + 1e-4);
  }
  // FP32 test: copies of coordinates up to m, shifts up to m + cutoff and differences up to the
  // cutoff are each rounded by 2^-24 of their size, so a component is off by at most 1.2e-7 (m +
  // cutoff); twice that is allowed for, and the rounding of the squares
  double m = 0.0;
  for (int k = 0; k < 3; ++k)
    m = fmax(m, far[0] * fabs(H[k]) + far[1] * fabs(H[3 + k]) + far[2] * fabs(H[6 + k]));
  const double band = 3.5 * cutoff * 2.4e-7 * (m + 2.0 * cutoff) + 1e-6 * cutoff * cutoff;
  const bool fits = band < 0.5 * cutoff * cutoff;  // false for NaN as well
  g.c2lo = fits ? (float)(cutoff * cutoff - band) : -1.0f;
  g.c2hi = fits ? (float)(cutoff * cutoff + band) : INFINITY;
  w.grids[i] = g;
  const int bins = g.nb[0] * g.nb[1] * g.nb[2];
  w.bins_per_struct[i] = bins;
  if (s.n_struct == 1) {  // no scan needed
    w.bin_off[0] = 0;
    w.bin_off[1] = bins;
  }
}

// Origin of the FP32 coordinates: the corner of an open structure's box, else
// the cell's (positions are wrapped into it).
__device__ __forceinline__ void coord_origin(const GridDesc& g, double (&o)[3]) {
#pragma unroll
  for (int k = 0; k < 3; ++k) o[k] = g.any_per() ? 0.0 : g.fmin[k];
}

// An atom's place: bin, order of arrival in it, wrapped position and wrap shift.
struct AtomPlace {
  int bin, arrival, wrap, si;
  double wp[3];
};

__device__ __forceinline__ AtomPlace bin_atom(const soapb_structs& s, const NLWork& w, int64_t a) {
  AtomPlace p;
  p.si = struct_of_atom(s.d_atom_off, s.n_struct, a);
  const GridDesc& g = w.grids[p.si];
  int b[3], wr[3];
  if (!locate(g, s.d_positions[3 * a], s.d_positions[3 * a + 1], s.d_positions[3 * a + 2], b, wr, p.wp))
    atomicOr(w.status, 2);
  if ((wr[0] | wr[1] | wr[2]) != 0 && !g.wrapped) atomicOr(&w.grids[p.si].wrapped, 1);
  p.bin = (int)(w.bin_off[p.si] + ((int64_t)b[2] * g.nb[1] + b[1]) * g.nb[0] + b[0]);
  p.arrival = atomicAdd(&w.bin_count[p.bin], 1);
  p.wrap = pack3(wr[0], wr[1], wr[2]);
  return p;
}

// The records of atom a in its final slot.
__device__ __forceinline__ void write_records(const NLWork& w, const GridDesc& g, int a, int species, const double* wp,
                                              int wrap, int slot) {
  w.sorted_pos[slot] = make_double4(wp[0], wp[1], wp[2], pack_info(a, species, wrap));
  double o[3];
  coord_origin(g, o);
  w.sorted_f[slot] = make_float4((float)(wp[0] - o[0]), (float)(wp[1] - o[1]), (float)(wp[2] - o[2]), 0.0f);
}

__device__ __forceinline__ void place_centre(const soapb_centres& c, const NLWork& w, int64_t i) {
  const int si = c.d_struct[i];
  const GridDesc& g = w.grids[si];
  int b[3], wr[3];
  double wp[3];
  if (!locate(g, c.d_xyz[3 * i], c.d_xyz[3 * i + 1], c.d_xyz[3 * i + 2], b, wr, wp)) atomicOr(w.status, 2);
  w.cpos[i] = make_double4(wp[0], wp[1], wp[2], 0.0);
  w.cinfo[i] = make_int4(b[0] | (b[1] << 10) | (b[2] << 20), si, pack3(wr[0], wr[1], wr[2]), c.d_atom[i]);
}

// The atom of a slot goes to its final place in the bin, its rank by atom index
// (the number of smaller indices in the bin), so the candidate order -- and the
// FP32 accumulation order -- is deterministic.  Bins hold a few atoms: the
// quadratic count is a few loads from L1, where sorting each bin by a warp took
// a pass over all bins (1M atoms: 143 us for the sort kernel alone).
__device__ __forceinline__ void gather_atom(const soapb_structs& s, const NLWork& w, int64_t slot) {
  const int a = w.sorted_atom[slot];
  const int gb = w.atom_bin[a];
  const int s0 = w.bin_start[gb], s1 = w.bin_start[gb + 1];
  int rank = 0;
  for (int i = s0; i < s1; ++i) rank += w.sorted_atom[i] < a;
  const int si = struct_of_atom(s.d_atom_off, s.n_struct, a);
  const GridDesc& g = w.grids[si];
  int b[3], wr[3];
  double wp[3];
  locate(g, s.d_positions[3 * (int64_t)a], s.d_positions[3 * (int64_t)a + 1], s.d_positions[3 * (int64_t)a + 2],
         b, wr, wp);
  write_records(w, g, a, s.d_species[a], wp, pack3(wr[0], wr[1], wr[2]), s0 + rank);
}

// ---- large inputs: one kernel per stage ----

__global__ void k_grid_init(soapb_structs s, NLWork w, double cutoff) {
  const int64_t nth = (int64_t)gridDim.x * blockDim.x, t0 = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  for (int64_t i = t0; i < s.n_struct; i += nth) grid_init(s, w, cutoff, (int)i);
  for (int64_t i = t0; i < w.max_bins; i += nth) w.bin_count[i] = 0;
}

__global__ void k_frac_bbox(soapb_structs s, NLWork w) {
  frac_bbox(s, w, (int64_t)blockIdx.x * blockDim.x + (threadIdx.x & ~31), (int64_t)gridDim.x * blockDim.x);
}

__global__ void k_grid_setup(soapb_structs s, NLWork w, double cutoff) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < s.n_struct) grid_setup(s, w, cutoff, i);
}

__global__ void k_bin_atoms(soapb_structs s, soapb_centres c, NLWork w) {
  const int64_t nth = (int64_t)gridDim.x * blockDim.x, t0 = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  for (int64_t a = t0; a < s.n_atoms; a += nth) {
    const AtomPlace p = bin_atom(s, w, a);
    w.atom_bin[a] = p.bin;
    w.arrival[a] = p.arrival;
  }
  for (int64_t i = t0; i < c.n_centres; i += nth) place_centre(c, w, i);
}

__global__ void k_scatter_atoms(int64_t n_atoms, NLWork w) {
  for (int64_t a = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; a < n_atoms;
       a += (int64_t)gridDim.x * blockDim.x)
    w.sorted_atom[w.bin_start[w.atom_bin[a]] + w.arrival[a]] = (int)a;
}

__global__ void k_gather_atoms(soapb_structs s, NLWork w) {
  for (int64_t slot = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; slot < s.n_atoms;
       slot += (int64_t)gridDim.x * blockDim.x)
    gather_atom(s, w, slot);
}

// ---- small inputs: every stage in one launch ----
//
// The stages are a chain of short dependent passes over few atoms, so separate
// kernels cost their launches (16 launches and 3 memsets, 2-5 us each, for
// 24 to 3000 atoms).  One cluster of up to 8 CTAs runs them all, with a cluster
// barrier between stages (one CTA: a block barrier); intermediate arrays stay
// in the workspace, in L2.  24 atoms: 15 us, 3000: 21 us, 48 cells
// of 200 atoms: 53 us.
constexpr int kCellsThreads = 512;
constexpr int kCellsMaxCtas = 8;

__global__ void __launch_bounds__(kCellsThreads) k_cells(soapb_structs s, soapb_centres c, NLWork w, double cutoff) {
  __shared__ int64_t s_warp[32];
  __shared__ int s_max[32];
  // the grid is one cluster: blockIdx.x is the rank in it
  const int nth = gridDim.x * kCellsThreads, t0 = blockIdx.x * kCellsThreads + threadIdx.x;
  auto sync = [&]() {
    if (gridDim.x == 1) {
      __syncthreads();
    } else {
      asm volatile("barrier.cluster.arrive.release.aligned;\n" ::: "memory");
      asm volatile("barrier.cluster.wait.acquire.aligned;\n" ::: "memory");
    }
  };
  if (t0 < 4) w.status[t0] = 0;
  for (int i = t0; i < s.n_struct; i += nth) grid_init(s, w, cutoff, i);
  for (int64_t i = t0; i < w.max_bins; i += nth) w.bin_count[i] = 0;
  sync();
  frac_bbox(s, w, t0 & ~31, nth);
  sync();
  for (int i = t0; i < s.n_struct; i += nth) grid_setup(s, w, cutoff, i);
  sync();
  if (s.n_struct > 1) {
    if (blockIdx.x == 0) block_scan_chunks(w.bins_per_struct, s.n_struct, w.bin_off, s_warp, s_max, nullptr);
    sync();
  }
  // an atom per thread stays in registers through the sort; centres are taken from the last
  // thread on, so with threads for both neither waits for the other
  const bool one = s.n_atoms <= nth;
  AtomPlace p = {};
  for (int64_t a = t0; a < s.n_atoms; a += nth) {
    p = bin_atom(s, w, a);
    if (!one) {
      w.atom_bin[a] = p.bin;
      w.arrival[a] = p.arrival;
    }
  }
  for (int64_t i = nth - 1 - t0; i < c.n_centres; i += nth) place_centre(c, w, i);
  sync();
  if (blockIdx.x == 0)
    block_scan_chunks(w.bin_count, __ldcg(w.bin_off + s.n_struct), w.bin_start, s_warp, s_max, nullptr);
  sync();
  if (one) {
    const bool mine = t0 < s.n_atoms;
    int s0 = 0, n = 0;
    if (mine) {
      s0 = __ldcg(w.bin_start + p.bin);
      n = __ldcg(w.bin_start + p.bin + 1) - s0;
      w.sorted_atom[s0 + p.arrival] = t0;
    }
    sync();
    if (mine) {
      int rank = 0;
#pragma unroll 4
      for (int i = 0; i < n; ++i) rank += __ldcg(w.sorted_atom + s0 + i) < t0;
      write_records(w, w.grids[p.si], t0, s.d_species[t0], p.wp, p.wrap, s0 + rank);
    }
  } else {
    for (int64_t a = t0; a < s.n_atoms; a += nth) w.sorted_atom[w.bin_start[w.atom_bin[a]] + w.arrival[a]] = (int)a;
    sync();
    for (int64_t slot = t0; slot < s.n_atoms; slot += nth) gather_atom(s, w, slot);
  }
}

// ---------------------------------------------------------------------------
// candidate enumeration (warp-synchronous; one warp per centre)
// ---------------------------------------------------------------------------

struct VisitArgs {
  const GridDesc* grids;
  const int64_t* bin_off;
  const int* bin_start;
  const double4* sorted_pos;
  const float4* sorted_f;
  const double4* cpos;
  const int4* cinfo;
  int* status;
  double cutoff, cutoff2;
  int mode;
};

// Shared memory of a warp's enumeration: per nonempty run, the slot of its
// first atom minus its place in the candidate stream, and for periodic
// structures that place and the image shift minus the centre (FP32), packed T in w.
struct VisitMem {
  float4 shift[64];
  int start[64], adj[64];
};

// The centre of a warp.
struct VisitCentre {
  double4 cp;
  int atom;  // centre atom or -1
  int cw[3];
  const GridDesc* g;
  bool per;
  __device__ __forceinline__ int pack(int a, int b, int c) const {
    return g->wide ? pack_wide(g->nrep, a, b, c) : pack3(a, b, c);
  }
  __device__ __forceinline__ void unpack(int p, int (&v)[3]) const {
    if (g->wide) unpack_wide(g->nrep, p, v);
    else unpack3(p, v);
  }
};

// One sorted-atom record through the read-only path (the lists are built by earlier kernels).
__device__ __forceinline__ double4 load_record(const double4* p) {
  const double2 a = __ldg(reinterpret_cast<const double2*>(p)), b = __ldg(reinterpret_cast<const double2*>(p) + 1);
  return make_double4(a.x, a.y, b.x, b.y);
}

// rvec of the candidate in a slot with cell-window shift T (of a periodic frame), in FP64.
__device__ __forceinline__ void exact_rvec(const VisitCentre& C, const double4& p, const int (&T)[3], double& rx,
                                           double& ry, double& rz) {
  const double* H = C.g->H;
  if (!C.per) {
    rx = p.x - C.cp.x;
    ry = p.y - C.cp.y;
    rz = p.z - C.cp.z;
  } else {
    rx = __dadd_rn(p.x, __dsub_rn(lattice_sum(H, T, 0), C.cp.x));
    ry = __dadd_rn(p.y, __dsub_rn(lattice_sum(H, T, 1), C.cp.y));
    rz = __dadd_rn(p.z, __dsub_rn(lattice_sum(H, T, 2), C.cp.z));
  }
}

// Whether a candidate is a pair, in FP64: the cutoff, the image set, and for
// create() the r <= 1e-12 edges other than the centre's own (SG:1171-1179).
__device__ __forceinline__ bool exact_test(const VisitArgs& A, const VisitCentre& C, int slot, int Tpacked) {
  const double4 p = load_record(A.sorted_pos + slot);
  int T[3] = {0, 0, 0};
  if (C.per) C.unpack(Tpacked, T);
  double rx, ry, rz;
  exact_rvec(C, p, T, rx, ry, rz);
  const double r2 = fma(rz, rz, fma(rx, rx, __dmul_rn(ry, ry)));
  if (!(r2 <= A.cutoff2)) return false;
  int atom, sp, wrap;
  unpack_info(p.w, atom, sp, wrap);
  if (C.per) {
    int aw[3];
    unpack3(wrap, aw);
#pragma unroll
    for (int k = 0; k < 3; ++k)
      if (C.g->per[k] && abs(T[k] - aw[k] + C.cw[k]) > C.g->nrep[k]) return false;
  }
  return !(A.mode == SOAPB_NL_CREATE && r2 <= 1e-24 && atom != C.atom);
}

__device__ __forceinline__ float sqrt_approx(float x) {
  float r;
  asm("sqrt.approx.f32 %0, %1;" : "=f"(r) : "f"(x));
  return r;
}

// Candidate enumeration of one centre by a warp.  The rows (by, bz) of unwrapped
// bins within the cutoff are taken 32 at a time, one per lane, each trimmed to
// the bins x that the cutoff sphere reaches (in FP32, against the cutoff plus
// 1e-3 A, which covers its rounding).  A row is one run of bin-sorted atoms, or
// in a cell periodic along x one per image Tx, two of them to a lane.  The runs
// form one candidate stream that all lanes walk 32 at a time: the runs that
// start inside a tile give one bit each (an OR-reduction), and a lane's run is
// the number of bits up to its own.  An FP32 copy of the position settles almost every
// candidate; those within rounding of the cutoff (or near r = 0 in create(), or
// all of them when wrap shifts make the image set matter) take the FP64 test.
// Order: z, y and x bins (through the images), then atom index.
// fn(ok, slot, T) is called with all lanes.
//
// The enumeration is bound by instruction issue and the latency of the loads: 5
// warp instructions per pair in the count, against 8 with FP64 row geometry
// (six divisions and a square root a centre, one a row) and tests (1M atoms:
// count 3.31 -> 2.32 ms; 48 periodic cells 85 -> 43 us).  Other than diagonal
// frames scanned the full window of half-cutoff bins before
// (501 atoms, triclinic: count and scan 46 -> 21 us, fill 45 -> 22 us).
// Writing the candidate slots of all runs into a list first, instead of finding
// each lane's run, took as many instructions as it saved.
template <bool PER, int UNROLL, class Fn>
__device__ __forceinline__ void visit_runs(const VisitArgs& A, VisitMem& M, const VisitCentre& C, const int4& ci,
                                           Fn&& fn) {
  const int lane = threadIdx.x & 31;
  const GridDesc& g = *C.g;
  const int cb[3] = {ci.x & 1023, (ci.x >> 10) & 1023, (ci.x >> 20) & 1023};
  const float R = (float)A.cutoff + 1e-3f;
  // the centre inside its bin (beyond [0, 1] for centres outside an open structure's box), and
  // the bins, from its own, that the cutoff reaches on each axis
  float f[3], iw[3];
  int lo[3], hi[3];
  {
    double fr[3];
    if (PER) {
      to_frac(g, C.cp.x, C.cp.y, C.cp.z, fr);
    } else {  // the identity frame
      fr[0] = C.cp.x;
      fr[1] = C.cp.y;
      fr[2] = C.cp.z;
    }
#pragma unroll
    for (int k = 0; k < 3; ++k) {
      f[k] = (float)fma(fr[k] - g.fmin[k], g.ibinw[k], -(double)cb[k]);
      f[k] = fminf(fmaxf(f[k], -1e6f), 1e6f);
      iw[k] = 1.0f / g.wp[k];
      const float reach = fmaf(R, iw[k], 1e-3f);
      lo[k] = (int)floorf(fmaxf(f[k] - reach, -1e9f));
      hi[k] = (int)floorf(fminf(f[k] + reach, 1e9f));
      if (!PER || !g.per[k]) {
        lo[k] = max(lo[k], -cb[k]);
        hi[k] = min(hi[k], g.nb[k] - 1 - cb[k]);
      } else {  // (R is 1e-3 A longer than the cutoff: many cells, if they are thin)
        lo[k] = max(lo[k], -(g.nrep[k] + 1) * g.nb[k] - cb[k]);
        hi[k] = min(hi[k], (g.nrep[k] + 2) * g.nb[k] - 1 - cb[k]);
      }
    }
  }
  const int ny = hi[1] - lo[1] + 1, nz = hi[2] - lo[2] + 1;
  int T0 = 0, nT = 1;
  if (PER && g.per[0]) {
    T0 = floordiv(cb[0] + lo[0], g.nb[0]);
    nT = floordiv(cb[0] + hi[0], g.nb[0]) - T0 + 1;
  }
  int nrows = (ny > 0 && nz > 0 && lo[0] <= hi[0]) ? ny * nz : 0;
  // row / ny is exact with the half added for rows below 2^20 (open axes have at most 1023 bins) and
  // off by one at most for more of them
  const float inv_ny = 1.0f / (float)ny;
  const int boff = (int)A.bin_off[ci.y];
  double o[3];
  coord_origin(g, o);
  const float sx0 = (float)(o[0] - C.cp.x), sy0 = (float)(o[1] - C.cp.y), sz0 = (float)(o[2] - C.cp.z);
  const bool image_test = PER && (g.wrapped || (C.cw[0] | C.cw[1] | C.cw[2]) != 0);
  const float c2lo = image_test ? -1.0f : g.c2lo, c2hi = g.c2hi;
  const float near2 = A.mode == SOAPB_NL_CREATE ? 1e-4f : -1.0f;
  const unsigned upto = 0xffffffffu >> (31 - lane);
  const bool orth = !PER || g.orth;
  const int groups = PER ? (nT + 1) >> 1 : 1;  // pairs of images of a row
  // (thin cells have more rows than an int holds)
  if (PER && (float)ny * (float)nz * (float)groups > 2e9f) nrows = nrows != 0 ? 2000000000 / groups : 0;
  const int nlanes = nrows * groups;
  for (int p0 = 0; p0 < nlanes; p0 += 32) {
    int row = p0 + lane, tg = 0;
    if (PER && groups > 1) {
      const int i = row;
      row = i / groups;
      tg = i - row * groups;
    }
    constexpr int Q = PER ? 2 : 1;  // runs of a row
    int len[Q], s0[Q];
    float4 sh[Q];
#pragma unroll
    for (int q = 0; q < Q; ++q) {
      len[q] = s0[q] = 0;
      sh[q] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    }
    if (row < nrows) {
      int iz = (int)(((float)row + 0.5f) * inv_ny), iy = row - iz * ny;
      if (PER) {
        if (iy < 0) { --iz; iy += ny; }
        if (iy >= ny) { ++iz; iy -= ny; }
      }
      const int dz = lo[2] + iz, dy = lo[1] + iy;
      float mid, ext2, slack = 1e-3f, iwx;  // x range in bins from the centre's: mid +- (sqrt(ext2) iwx + slack)
      if (orth) {
        const float ay = fmaxf(0.0f, fmaxf((float)dy - f[1], f[1] - (float)(dy + 1)) * g.wp[1]);
        const float az = fmaxf(0.0f, fmaxf((float)dz - f[2], f[2] - (float)(dz + 1)) * g.wp[2]);
        ext2 = R * R - ay * ay - az * az;
        mid = f[0];
        iwx = iw[0];
      } else {
        const float qy = (float)dy + 0.5f - f[1], qz = (float)dz + 0.5f - f[2];
        const float vx = qy * g.eb[0] + qz * g.ec[0], vy = qy * g.eb[1] + qz * g.ec[1],
                    vz = qy * g.eb[2] + qz * g.ec[2];
        const float par = vx * g.dir[0] + vy * g.dir[1] + vz * g.dir[2];
        const float px = vx - par * g.dir[0], py = vy - par * g.dir[1], pz = vz - par * g.dir[2];
        const float perp = fmaxf(0.0f, sqrt_approx(px * px + py * py + pz * pz) - g.rho - 1e-4f);
        ext2 = R * R - perp * perp;
        iwx = g.ialong;
        mid = f[0] - par * iwx;
        slack += g.rho * iwx;
      }
      if (ext2 >= 0.0f) {
        const float e = fmaf(sqrt_approx(ext2), iwx, slack);
        const int x0 = max((int)floorf(fmaxf(mid - e, -1e9f)), lo[0]),
                  x1 = min((int)floorf(fminf(mid + e, 1e9f)), hi[0]);
        int byw = cb[1] + dy, bzw = cb[2] + dz, Ty = 0, Tz = 0;
        if (PER) {
          if (g.per[1]) { Ty = floordiv(byw, g.nb[1]); byw -= Ty * g.nb[1]; }
          if (g.per[2]) { Tz = floordiv(bzw, g.nb[2]); bzw -= Tz * g.nb[2]; }
        }
        const int gb = boff + (bzw * g.nb[1] + byw) * g.nb[0];
#pragma unroll
        for (int q = 0; q < Q; ++q) {
          const int Tx = T0 + 2 * tg + q;
          int bx = cb[0], xa = x0, xb = x1;
          if (PER && g.per[0]) {  // the part of the row in this image
            bx -= Tx * g.nb[0];
            xa = max(xa, -bx);
            xb = min(xb, g.nb[0] - 1 - bx);
          }
          if (xa <= xb && (q == 0 || 2 * tg + q < nT)) {
            s0[q] = __ldg(A.bin_start + gb + bx + xa);
            len[q] = __ldg(A.bin_start + gb + bx + xb + 1) - s0[q];
            if (PER) {
              const double* H = g.H;
              sh[q] = make_float4((float)(Tx * H[0] + Ty * H[3] + Tz * H[6] - C.cp.x),
                                  (float)(Tx * H[1] + Ty * H[4] + Tz * H[7] - C.cp.y),
                                  (float)(Tx * H[2] + Ty * H[5] + Tz * H[8] - C.cp.z),
                                  __int_as_float(C.pack(Tx, Ty, Tz)));
            }
          }
        }
      }
    }
    const int mine = PER ? len[0] + len[Q - 1] : len[0];
    int end = mine;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
      const int v = __shfl_up_sync(0xffffffffu, end, d);
      if (lane >= d) end += v;
    }
    const int total = __shfl_sync(0xffffffffu, end, 31);
    int nruns = 0;
    {
      const unsigned b0 = __ballot_sync(0xffffffffu, len[0] > 0), before = upto >> 1;
      int ord = __popc(b0 & before), start = end - mine;
      nruns = __popc(b0);
      if (PER) {
        const unsigned b1 = __ballot_sync(0xffffffffu, len[Q - 1] > 0);
        ord += __popc(b1 & before);
        nruns += __popc(b1);
      }
#pragma unroll
      for (int q = 0; q < Q; ++q)
        if (len[q] > 0) {
          M.adj[ord] = s0[q] - start;
          if (PER) {
            M.start[ord] = start;
            M.shift[ord] = sh[q];
          }
          start += len[q];
          ++ord;
        }
    }
    __syncwarp();
    int before = -1;  // runs started before the tile, minus one
    // the run of this lane's candidate in the tile at k0
    auto run_of = [&](int k0) {
      unsigned d = 32u;
      if (PER) {
        const int idx = before + 1 + lane;
        if (idx < nruns) d = (unsigned)(M.start[idx] - k0);
      } else if (len[0] > 0) {  // this lane's own run
        d = (unsigned)(end - len[0] - k0);
      }
      const unsigned mask = __reduce_or_sync(0xffffffffu, d < 32u ? 1u << d : 0u);
      const int run = before + __popc(mask & upto);
      before += __popc(mask);
      return run;
    };
    // the next tile's position is loaded while this one is tested
    int run_n = run_of(0), slot_n = lane < total ? M.adj[run_n] + lane : 0;
    float4 pos_n = __ldg(A.sorted_f + slot_n);
#pragma unroll (UNROLL)
    for (int k0 = 0; k0 < total; k0 += 32) {
      const bool valid = k0 + lane < total;
      const int slot = slot_n, run = run_n;
      const float4 p = pos_n;
      if (k0 + 32 < total) {
        run_n = run_of(k0 + 32);
        slot_n = k0 + 32 + lane < total ? M.adj[run_n] + k0 + 32 + lane : 0;
        pos_n = __ldg(A.sorted_f + slot_n);
      }
      float sx = sx0, sy = sy0, sz = sz0;
      int T = 0;
      if (PER) {
        const float4 v = M.shift[valid ? run : 0];
        sx = v.x;
        sy = v.y;
        sz = v.z;
        T = __float_as_int(v.w);
      }
      const float rx = p.x + sx, ry = p.y + sy, rz = p.z + sz;
      const float r2 = fmaf(rx, rx, fmaf(ry, ry, rz * rz));
      bool ok = valid && r2 <= c2lo && r2 > near2;
      const bool unsure = valid && !ok && !(r2 > c2hi);
      if (__any_sync(0xffffffffu, unsure)) {
        if (unsure) ok = exact_test(A, C, slot, T);
        __syncwarp();
      }
      fn(ok, slot, T);
    }
    __syncwarp();  // the run table is rewritten
  }
}

template <int UNROLL, class Fn>
__device__ __forceinline__ void visit(const VisitArgs& A, int64_t c, VisitMem& M, VisitCentre& C, Fn&& fn) {
  const int4 ci = A.cinfo[c];
  C.g = A.grids + ci.y;
  C.cp = A.cpos[c];
  C.atom = ci.w;
  C.per = C.g->any_per();
  if (C.g->orth < 0) return;
  unpack3(ci.z, C.cw);
  if (C.per) visit_runs<true, UNROLL>(A, M, C, ci, fn);
  else visit_runs<false, UNROLL>(A, M, C, ci, fn);
}

// The i-th centre of a warp, or n_centres.  A block takes consecutive centres,
// its warps in turn: neighbouring centres share most of their candidates, so
// the warps find each other's records in L1.
__device__ __forceinline__ int64_t nth_centre(int i, int64_t n_centres) {
  const int64_t W = blockDim.x >> 5, per = (n_centres + gridDim.x * W - 1) / (gridDim.x * W);
  return i < per ? min((blockIdx.x * per + i) * W + (threadIdx.x >> 5), n_centres) : n_centres;
}

// Pairs of every centre, one warp per centre, 8 blocks of 4 warps per SM (64
// registers, 130 B of spills): the count is latency-bound with little work per
// candidate, so more resident warps pay (1M atoms with the set-up: 2.48 ms, 6
// blocks 2.66).  The largest count goes to
// status[2].  With pair_off, the last block to finish scans the counts into it
// and, with stats, writes {total, largest, flags} -- the caller gets offsets and
// summary from this launch (kLastBlockScan centres: the scan by 128 threads
// costs less than the three launches of the general one).
constexpr int64_t kLastBlockScan = 8192;

__global__ void __launch_bounds__(128, 8) k_count(VisitArgs A, int64_t n_centres, int* counts, int64_t* pair_off,
                                                  int64_t* stats) {
  __shared__ VisitMem s_mem[4];
  __shared__ int s_cnt[4];
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  int most = 0;
  for (int i = 0;; ++i) {
    const int64_t c = nth_centre(i, n_centres);
    if (c >= n_centres) break;
    int cnt = 0;
    VisitCentre C;
    visit<2>(A, c, s_mem[wid], C, [&](bool ok, int, int) { cnt += ok; });
    cnt = __reduce_add_sync(0xffffffffu, cnt);
    if (lane == 0) counts[c] = cnt;
    most = max(most, cnt);
  }
  if (lane == 0) s_cnt[wid] = most;
  __syncthreads();
  if (!pair_off) {
    if (threadIdx.x == 0) atomicMax(A.status + 2, max(max(s_cnt[0], s_cnt[1]), max(s_cnt[2], s_cnt[3])));
    return;
  }
  __shared__ int s_last;
  if (threadIdx.x == 0) {
    __threadfence();  // this block's counts before its ticket (ordered after them by the barrier above)
    s_last = atomicAdd(A.status + 1, 1) == (int)gridDim.x - 1;
    __threadfence();
  }
  __syncthreads();
  if (!s_last) return;
  __shared__ int64_t s_warp[32];
  int largest;
  const int64_t total = block_scan_chunks(counts, n_centres, pair_off, s_warp, s_cnt, &largest);
  if (threadIdx.x == 0) {
    A.status[2] = largest;
    if (stats) {
      stats[0] = total;
      stats[1] = largest;
      stats[2] = __ldcg(A.status);
    }
  }
}

// Fill: one warp per centre.  The slots and image shifts of the centre's pairs are
// collected in shared memory in candidate order (one enumeration, 8 bytes a
// pair), then ranked within their key (species, radial segment) by a stable
// counting sort and written to the centre's CSR slice from the FP64 records.  A
// centre with more than `stage` pairs, or in a cell so small that shifts need
// more than 4 bits an axis, enumerates twice instead (histogram, then scatter).
// Either way the order is: by key, and by candidate order within a key.  The key
// is computed from the FP32 pair record (the radius and segment the descriptor
// kernels compute).
//
// The latency of the record loads and of the ranking bounds this kernel, so it
// keeps little per pair: 20 bytes (the FP32 record, key and rank, a tile's
// records loaded while the next is tested) leave fewer warps and less L1 and
// measured slower (1M atoms: 7.0 ms).  1M atoms: 7.25 -> 6.01 ms; 3000 atoms at
// 700 pairs a centre: 63 -> 43 us (768 staged pairs, no second enumeration); 48
// cells: 124 -> 74 us.  7 blocks per SM, at 72 registers with 200 B of spills
// around the enumerations: 6 take 6.5 ms; 8 the same, but 3000 atoms 51 us with
// the launch instead of 48.
__host__ __device__ inline int fill_warp_bytes(int nkeys, int stage) {
  return (int)sizeof(VisitMem) + 8 * stage + ((4 * nkeys + 15) & ~15);
}

__global__ void __launch_bounds__(128, 7) k_fill(VisitArgs A, int64_t n_centres, const int64_t* pair_off, float4* pairs,
                                              int64_t capacity, int nseg, float inv_h, int nkeys, int stage,
                                              int* status) {
  extern __shared__ __align__(16) unsigned char s_raw[];
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  unsigned char* mine = s_raw + (size_t)wid * fill_warp_bytes(nkeys, stage);
  VisitMem& M = *reinterpret_cast<VisitMem*>(mine);
  int* st_slot = reinterpret_cast<int*>(mine + sizeof(VisitMem));
  unsigned* st_meta = reinterpret_cast<unsigned*>(st_slot + stage);  // T + 8 per axis (4 bits) | key << 12 | rank << 22
  int* hist = reinterpret_cast<int*>(st_meta + stage);
  if (pair_off[n_centres] > capacity) {
    if (threadIdx.x == 0 && blockIdx.x == 0) atomicOr(status, 4);
    return;
  }
  // species * nseg + segment of the FP32 record.  The roundings are written out: they place a pair
  // within one of them of a segment's edge, and so the order of the centre's sums.
  auto keyof = [&](const float4& p) {
    const float r = sqrtf(fmaf(p.z, p.z, fmaf(p.x, p.x, __fmul_rn(p.y, p.y))));
    return (int)((unsigned)__float_as_int(p.w) >> kAtomBits) * nseg + min((int)(r * inv_h), nseg - 1);
  };
  auto scan_hist = [&]() {  // exclusive scan of hist (each lane a contiguous chunk)
    const int per = (nkeys + 31) / 32;
    const int k0 = min(lane * per, nkeys), k1 = min(k0 + per, nkeys);
    int sum = 0;
    for (int k = k0; k < k1; ++k) sum += hist[k];
    int inc = sum;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int t = __shfl_up_sync(0xffffffffu, inc, o);
      if (lane >= o) inc += t;
    }
    int run = inc - sum;
    for (int k = k0; k < k1; ++k) {
      const int v = hist[k];
      hist[k] = run;
      run += v;
    }
    __syncwarp();
  };
  for (int ic = 0;; ++ic) {
    const int64_t c = nth_centre(ic, n_centres);
    if (c >= n_centres) break;
    for (int k = lane; k < nkeys; k += 32) hist[k] = 0;
    const int64_t base = pair_off[c];
    const int64_t P = pair_off[c + 1] - base;
    __syncwarp();
    VisitCentre C;
    auto record = [&](int slot, const int (&T)[3]) {
      const double4 p = load_record(A.sorted_pos + slot);
      double rx, ry, rz;
      exact_rvec(C, p, T, rx, ry, rz);
      // the record's low word is atom | species << kAtomBits already
      return make_float4((float)rx, (float)ry, (float)rz, __int_as_float((int)__double_as_longlong(p.w)));
    };
    auto staged = [&](int i) {
      const unsigned t = st_meta[i];
      const int T[3] = {(int)(t & 15u) - 8, (int)((t >> 4) & 15u) - 8, (int)((t >> 8) & 15u) - 8};
      return record(st_slot[i], T);
    };
    auto unstaged = [&](int slot, int Tpacked) {
      int T[3] = {0, 0, 0};
      if (C.per) C.unpack(Tpacked, T);
      return record(slot, T);
    };
    // slots of one key in a warp's 32 pairs, ranked in lane order behind those counted before
    auto rank_in_key = [&](bool ok, int key) {
      const unsigned peers = __match_any_sync(0xffffffffu, ok ? key : -1 - lane);
      const int before = ok ? hist[key] : 0;
      __syncwarp();
      if (ok && lane == __ffs(peers) - 1) hist[key] = before + __popc(peers);
      __syncwarp();
      return before + __popc(peers & ((1u << lane) - 1u));
    };
    const GridDesc& g = A.grids[A.cinfo[c].y];
    // positions are wrapped: a pair's |T| is at most ceil(cutoff / width) = n_rep on each axis
    if (P <= stage && max(g.nrep[0], max(g.nrep[1], g.nrep[2])) <= 7) {
      int n = 0;
      visit<1>(A, c, M, C, [&](bool ok, int slot, int T) {
        const unsigned bal = __ballot_sync(0xffffffffu, ok);
        const int pos = n + __popc(bal & ((1u << lane) - 1u));
        if (ok && pos < stage) {
          st_slot[pos] = slot;
          int v[3];
          unpack3(T, v);
          st_meta[pos] = C.per ? (unsigned)(v[0] + 8) | (unsigned)(v[1] + 8) << 4 | (unsigned)(v[2] + 8) << 8 : 0u;
        }
        n += __popc(bal);
      });
      __syncwarp();
      const int m = min(n, stage);
      for (int i0 = 0; i0 < m; i0 += 64) {  // two tiles' records in flight
        int key[2];
#pragma unroll
        for (int u = 0; u < 2; ++u) key[u] = keyof(staged(min(i0 + 32 * u + lane, m - 1)));
#pragma unroll
        for (int u = 0; u < 2; ++u) {
          const int i = i0 + 32 * u + lane;
          const int rank = rank_in_key(i < m, key[u]);
          if (i < m) st_meta[i] |= (unsigned)key[u] << 12 | (unsigned)rank << 22;
        }
      }
      scan_hist();
#pragma unroll 4
      for (int i = lane; i < m; i += 32) {
        const unsigned t = st_meta[i];
        pairs[base + hist[(t >> 12) & 1023u] + (t >> 22)] = staged(i);
      }
    } else {
      visit<1>(A, c, M, C, [&](bool ok, int slot, int T) {
        if (ok) atomicAdd(&hist[keyof(unstaged(slot, T))], 1);
      });
      __syncwarp();
      scan_hist();
      visit<1>(A, c, M, C, [&](bool ok, int slot, int T) {
        float4 rec = make_float4(0.f, 0.f, 0.f, 0.f);
        if (ok) rec = unstaged(slot, T);
        const int pos = rank_in_key(ok, ok ? keyof(rec) : 0);
        if (ok) pairs[base + pos] = rec;
      });
    }
    __syncwarp();
  }
}

// Total pairs, the largest per-centre count (from the count) and the status
// flags, so the host learns all three from one read.
__global__ void k_stats(const int64_t* pair_off, int64_t n_centres, const int* status, int64_t* out) {
  out[0] = pair_off[n_centres];
  out[1] = status[2];
  out[2] = status[0];
}

// One block: out[0] = the list's total; when it exceeds capacity, every
// offset is set to 0 (all lists empty), so kernels launched after it read
// nothing beyond the pair buffer.  One block: the total is read once before
// any offset is rewritten.
__global__ void __launch_bounds__(1024) k_clamp(int64_t* pair_off, int64_t n_centres, int64_t capacity, int64_t* out) {
  __shared__ int64_t s_total;
  if (threadIdx.x == 0) s_total = pair_off[n_centres];
  __syncthreads();
  const int64_t total = s_total;
  if (threadIdx.x == 0) out[0] = total;
  if (total <= capacity) return;
  for (int64_t i = threadIdx.x; i <= n_centres; i += blockDim.x) pair_off[i] = 0;
}

// ---------------------------------------------------------------------------
// host side
// ---------------------------------------------------------------------------

struct NLLayout {
  int64_t grids, fbox, bps, bin_off, bin_count, bin_start, atom_bin, sorted_atom, sorted_pos, sorted_f, cpos,
      cinfo, counts, partials, status, total;
  int64_t max_bins;
};

static NLLayout nl_layout(const soapb_structs* s, const soapb_centres* c) {
  NLLayout L{};
  const int64_t ns = s->n_struct, na = s->n_atoms, nc = c->n_centres;
  L.max_bins = 2 * na + 8 * ns + 64;
  int64_t maxn = L.max_bins > nc ? L.max_bins : nc;  // longest scan
  if (maxn < ns) maxn = ns;
  int64_t off = 0;
  auto take = [&](int64_t bytes) { const int64_t o = off; off = align_up(off + bytes, 256); return o; };
  L.grids = take(sizeof(GridDesc) * ns);
  L.fbox = take(8 * 6 * ns);
  L.bps = take(4 * ns);
  L.bin_off = take(8 * (ns + 1));
  L.bin_count = take(4 * L.max_bins);
  L.bin_start = take(4 * (L.max_bins + 1));
  L.atom_bin = take(4 * na);
  L.sorted_atom = take(4 * na);
  L.sorted_pos = take(32 * na);
  L.sorted_f = take(16 * na);
  L.cpos = take(32 * nc);
  L.cinfo = take(16 * nc);
  L.counts = take(4 * nc);
  L.partials = take(8 * ((maxn + 1023) / 1024 + 2));
  L.status = take(16);
  L.total = off;
  return L;
}

static NLWork nl_work(const NLLayout& L, void* base_) {
  char* base = (char*)base_;
  NLWork w;
  w.grids = (GridDesc*)(base + L.grids);
  w.fbox = (unsigned long long*)(base + L.fbox);
  w.bins_per_struct = (int*)(base + L.bps);
  w.bin_off = (int64_t*)(base + L.bin_off);
  w.bin_count = (int*)(base + L.bin_count);
  w.bin_start = (int*)(base + L.bin_start);
  w.sorted_f = (float4*)(base + L.sorted_f);
  w.arrival = (int*)(base + L.sorted_f);  // read by the scatter, before the gather writes sorted_f
  w.atom_bin = (int*)(base + L.atom_bin);
  w.sorted_atom = (int*)(base + L.sorted_atom);
  w.sorted_pos = (double4*)(base + L.sorted_pos);
  w.cpos = (double4*)(base + L.cpos);
  w.cinfo = (int4*)(base + L.cinfo);
  w.counts = (int*)(base + L.counts);
  w.partials = (int64_t*)(base + L.partials);
  w.status = (int*)(base + L.status);
  w.max_bins = L.max_bins;
  return w;
}

static int check_inputs(const soapb_basis* b, const soapb_structs* s, const soapb_centres* c) {
  if (!b || !b->dev) return set_error(SOAPB_ERR_ARG, "basis not built");
  if (!s || !c) return set_error(SOAPB_ERR_ARG, "null structures or centres");
  if (s->n_struct < 1) return set_error(SOAPB_ERR_ARG, "need at least one structure");
  if (s->n_atoms < 0 || c->n_centres < 0) return set_error(SOAPB_ERR_ARG, "negative sizes");
  if (s->n_atoms >= (int64_t)kAtomMask) return set_error(SOAPB_ERR_ARG, "too many atoms (max %d)", kAtomMask);
  if (s->n_atoms > 0 && (!s->d_positions || !s->d_species)) return set_error(SOAPB_ERR_ARG, "null atom arrays");
  if (!s->d_atom_off || !s->d_cells || !s->d_pbc) return set_error(SOAPB_ERR_ARG, "null structure arrays");
  if (c->n_centres > 0 && (!c->d_xyz || !c->d_struct || !c->d_atom)) return set_error(SOAPB_ERR_ARG, "null centre arrays");
  return SOAPB_OK;
}

static VisitArgs visit_args(const soapb_basis* b, const NLWork& w, int mode) {
  VisitArgs A;
  A.grids = w.grids;
  A.bin_off = w.bin_off;
  A.bin_start = w.bin_start;
  A.sorted_pos = w.sorted_pos;
  A.sorted_f = w.sorted_f;
  A.cpos = w.cpos;
  A.cinfo = w.cinfo;
  A.status = w.status;
  A.cutoff = b->cutoff;
  A.cutoff2 = b->cutoff * b->cutoff;
  A.mode = mode;
  return A;
}

static int grid_blocks(int64_t n, int threads) {
  int64_t g = (n + threads - 1) / threads;
  if (g < 1) g = 1;
  if (g > 148 * 64) g = 148 * 64;
  return (int)g;
}

}  // namespace soapb

using namespace soapb;

extern "C" int soapb_neighbors_workspace(const soapb_basis* b, const soapb_structs* s, const soapb_centres* c,
                                         int64_t* bytes) {
  int rc = check_inputs(b, s, c);
  if (rc) return rc;
  if (!bytes) return set_error(SOAPB_ERR_ARG, "null bytes");
  *bytes = nl_layout(s, c).total;
  return SOAPB_OK;
}

// Inputs up to this many atoms and centres build their cell lists in one
// launch (k_cells).
constexpr int64_t kCellsFused = 16384;

static int launch_cells(const soapb_structs& s, const soapb_centres& c, const NLWork& w, double cutoff,
                        cudaStream_t st) {
  // a thread for every atom and centre, as far as one cluster goes
  int ctas = 1;
  while (ctas < kCellsMaxCtas && ctas * kCellsThreads < s.n_atoms + c.n_centres) ctas *= 2;
  cudaLaunchAttribute at;
  at.id = cudaLaunchAttributeClusterDimension;
  at.val.clusterDim.x = (unsigned)ctas;
  at.val.clusterDim.y = at.val.clusterDim.z = 1;
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3((unsigned)ctas);
  cfg.blockDim = dim3(kCellsThreads);
  cfg.stream = st;
  cfg.attrs = &at;
  cfg.numAttrs = 1;
  const int rc = check_cuda(cudaLaunchKernelEx(&cfg, k_cells, s, c, w, cutoff), "k_cells");
  return rc ? rc : check_launch("k_cells");
}

static int neighbors_count(const soapb_basis* b, const soapb_structs* s, const soapb_centres* c, int32_t mode,
                           void* d_work, int64_t work_bytes, int64_t* d_pair_off, int64_t* d_stats, void* stream) {
  int rc = check_inputs(b, s, c);
  if (rc) return rc;
  if (mode != SOAPB_NL_CREATE && mode != SOAPB_NL_ALL) return set_error(SOAPB_ERR_ARG, "bad neighbour mode");
  const NLLayout L = nl_layout(s, c);
  if (!d_work || work_bytes < L.total) return set_error(SOAPB_ERR_ARG, "workspace too small (%lld < %lld)",
                                                        (long long)work_bytes, (long long)L.total);
  if (!d_pair_off) return set_error(SOAPB_ERR_ARG, "null pair_off");
  cudaStream_t st = (cudaStream_t)stream;
  NLWork w = nl_work(L, d_work);
  const int ns = s->n_struct;
  const double cutoff = b->cutoff;
  if (s->n_atoms <= kCellsFused && c->n_centres <= kCellsFused && ns <= kCellsFused) {
    if ((rc = launch_cells(*s, *c, w, cutoff, st))) return rc;
  } else {
    if ((rc = check_cuda(cudaMemsetAsync(w.status, 0, 16, st), "memset status"))) return rc;
    k_grid_init<<<grid_blocks(L.max_bins, 256), 256, 0, st>>>(*s, w, cutoff);
    // at least 8 atoms a lane: a warp reduces its bounds once
    k_frac_bbox<<<grid_blocks((s->n_atoms + 7) / 8, 256), 256, 0, st>>>(*s, w);
    k_grid_setup<<<(ns + 127) / 128, 128, 0, st>>>(*s, w, cutoff);
    if ((rc = check_launch("grid setup", 3))) return rc;
    if ((rc = exclusive_scan(w.bins_per_struct, ns, w.bin_off, w.partials, st))) return rc;
    k_bin_atoms<<<grid_blocks(s->n_atoms > c->n_centres ? s->n_atoms : c->n_centres, 256), 256, 0, st>>>(*s, *c, w);
    if ((rc = check_launch("k_bin_atoms"))) return rc;
    if ((rc = exclusive_scan(w.bin_count, L.max_bins, w.bin_start, w.partials, st))) return rc;
    k_scatter_atoms<<<grid_blocks(s->n_atoms, 256), 256, 0, st>>>(s->n_atoms, w);
    k_gather_atoms<<<grid_blocks(s->n_atoms, 256), 256, 0, st>>>(*s, w);
    if ((rc = check_launch("cell lists", 2))) return rc;
  }
  const VisitArgs A = visit_args(b, w, mode);
  const bool tail = c->n_centres > 0 && c->n_centres <= kLastBlockScan;
  if (c->n_centres > 0)
    k_count<<<grid_blocks(c->n_centres, 4), 128, 0, st>>>(A, c->n_centres, w.counts, tail ? d_pair_off : nullptr,
                                                          tail ? d_stats : nullptr);
  if ((rc = check_launch("k_count", c->n_centres > 0 ? 1 : 0))) return rc;
  if (tail) return SOAPB_OK;
  if ((rc = exclusive_scan(w.counts, c->n_centres, d_pair_off, w.partials, st))) return rc;
  if (!d_stats) return SOAPB_OK;
  k_stats<<<1, 1, 0, st>>>(d_pair_off, c->n_centres, w.status, d_stats);
  return check_launch("k_stats");
}

extern "C" int soapb_neighbors_count(const soapb_basis* b, const soapb_structs* s, const soapb_centres* c,
                                     int32_t mode, void* d_work, int64_t work_bytes, int64_t* d_pair_off,
                                     void* stream) {
  return neighbors_count(b, s, c, mode, d_work, work_bytes, d_pair_off, nullptr, stream);
}

extern "C" int soapb_neighbors_count_stats(const soapb_basis* b, const soapb_structs* s, const soapb_centres* c,
                                           int32_t mode, void* d_work, int64_t work_bytes, int64_t* d_pair_off,
                                           int64_t* d_stats, void* stream) {
  if (!d_stats) return set_error(SOAPB_ERR_ARG, "null stats");
  return neighbors_count(b, s, c, mode, d_work, work_bytes, d_pair_off, d_stats, stream);
}

extern "C" int soapb_neighbors_fill(const soapb_basis* b, const soapb_structs* s, const soapb_centres* c,
                                    int32_t mode, void* d_work, int64_t work_bytes, const int64_t* d_pair_off,
                                    void* d_pairs, int64_t capacity, void* stream) {
  int rc = check_inputs(b, s, c);
  if (rc) return rc;
  const NLLayout L = nl_layout(s, c);
  if (!d_work || work_bytes < L.total) return set_error(SOAPB_ERR_ARG, "workspace too small");
  if (!d_pair_off || (!d_pairs && capacity > 0)) return set_error(SOAPB_ERR_ARG, "null pair arrays");
  if (((uintptr_t)d_pairs) % 16) return set_error(SOAPB_ERR_ARG, "pairs must be 16-byte aligned");
  cudaStream_t st = (cudaStream_t)stream;
  NLWork w = nl_work(L, d_work);
  const VisitArgs A = visit_args(b, w, mode);
  if (c->n_centres > 0) {
    // staged pairs per centre: 512, or 768 when the cutoff sphere holds more at condensed-matter
    // density (0.12 atoms / A^3); more would cost resident warps
    const int stage = 4.19 * b->cutoff * b->cutoff * b->cutoff * 0.12 > 512.0 ? 768 : 512;
    const int smem = 4 * fill_warp_bytes(b->n_keys, stage);
    int rc2 = check_cuda(cudaFuncSetAttribute(k_fill, cudaFuncAttributeMaxDynamicSharedMemorySize, smem),
                         "fill smem attribute");
    if (rc2) return rc2;
    k_fill<<<grid_blocks(c->n_centres, 4), 128, smem, st>>>(A, c->n_centres, d_pair_off, (float4*)d_pairs,
                                                            capacity, b->n_seg, (float)(1.0 / b->seg_width),
                                                            b->n_keys, stage, w.status);
  }
  return check_launch("k_fill", c->n_centres > 0 ? 1 : 0);
}

extern "C" int soapb_neighbors_status(const soapb_basis* b, const soapb_structs* s, const soapb_centres* c,
                                      void* d_work, int32_t* h_status, void* stream) {
  int rc = check_inputs(b, s, c);
  if (rc) return rc;
  const NLLayout L = nl_layout(s, c);
  NLWork w = nl_work(L, d_work);
  cudaStream_t st = (cudaStream_t)stream;
  if ((rc = check_cuda(cudaMemcpyAsync(h_status, w.status, 4, cudaMemcpyDeviceToHost, st), "status download")))
    return rc;
  return check_cuda(cudaStreamSynchronize(st), "status sync");
}

extern "C" int soapb_neighbors_stats(const soapb_basis* b, const soapb_structs* s, const soapb_centres* c,
                                     const void* d_work, const int64_t* d_pair_off, int64_t* d_stats, void* stream) {
  int rc = check_inputs(b, s, c);
  if (rc) return rc;
  if (!d_work || !d_pair_off || !d_stats) return set_error(SOAPB_ERR_ARG, "null workspace, pair_off or stats");
  const NLLayout L = nl_layout(s, c);
  const NLWork w = nl_work(L, const_cast<void*>(d_work));
  k_stats<<<1, 1, 0, (cudaStream_t)stream>>>(d_pair_off, c->n_centres, w.status, d_stats);
  return check_launch("k_stats");
}

extern "C" int soapb_neighbors_clamp(int64_t* d_pair_off, int64_t n_centres, int64_t capacity, int64_t* d_total,
                                     void* stream) {
  if (!d_pair_off || !d_total || n_centres < 0 || capacity < 0) return set_error(SOAPB_ERR_ARG, "bad clamp arguments");
  k_clamp<<<1, 1024, 0, (cudaStream_t)stream>>>(d_pair_off, n_centres, capacity, d_total);
  return check_launch("k_clamp");
}

// ---------------------------------------------------------------------------
// Neighbour list without any device allocation
// ---------------------------------------------------------------------------
// The regular entry points take a caller-sized workspace.  Some callers have
// no way to provide one at the moment they need a neighbour list: a plain C or
// Fortran molecular-dynamics driver that owns a fixed device-memory budget
// and forbids libraries from allocating after set-up, or a time-step loop
// where cudaMalloc / cudaFree would synchronise the device and stall it.
// soapb_neighbors_noalloc serves them: its scratch is one fixed device array
// that exists from module load to process exit on every GPU that loads the
// library, so the call itself allocates nothing.
namespace soapb {

constexpr int64_t kNoAllocScratchBytes = 8ll << 20;  // 8 MiB per device
static __device__ __align__(256) unsigned char g_nl_scratch[kNoAllocScratchBytes];

static std::mutex g_scratch_mu;
struct ScratchSlot {
  unsigned long long ctx_id;  // id of the CUDA context the address belongs to (0 = unknown)
  void* ptr;
};
static ScratchSlot g_scratch_slot[64] = {};

// Process-unique id of the calling thread's current CUDA context, or 0 when
// the driver cannot report one.  A device reset destroys the context (and
// the module with g_nl_scratch); the next context gets a new id, so a cached
// address is used only inside the context it was looked up in.  The driver
// functions come through the runtime's entry-point query: no link to libcuda.
static unsigned long long current_context_id() {
  typedef int (*GetCurrentFn)(void**);
  typedef int (*GetIdFn)(void*, unsigned long long*);
  static GetCurrentFn get_current = nullptr;
  static GetIdFn get_id = nullptr;
  static std::once_flag once;
  std::call_once(once, [] {
    void* f = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPointByVersion("cuCtxGetCurrent", &f, 4000, cudaEnableDefault, &q) == cudaSuccess &&
        q == cudaDriverEntryPointSuccess)
      get_current = (GetCurrentFn)f;
    f = nullptr;
    if (cudaGetDriverEntryPointByVersion("cuCtxGetId", &f, 12000, cudaEnableDefault, &q) == cudaSuccess &&
        q == cudaDriverEntryPointSuccess)
      get_id = (GetIdFn)f;
  });
  if (!get_current || !get_id) return 0;
  void* ctx = nullptr;
  unsigned long long id = 0;
  if (get_current(&ctx) != 0 || !ctx) return 0;
  if (get_id(ctx, &id) != 0) return 0;
  return id;
}

// Device address of g_nl_scratch in the current device's context (the
// host-side symbol is not a device address).  Looked up once per context and
// cached: again after a cudaDeviceReset, and on every call when the context
// id is unavailable.
static int scratch_address(void** out) {
  int dev = 0;
  int rc = check_cuda(cudaGetDevice(&dev), "cudaGetDevice");
  if (rc) return rc;
  if (dev < 0 || dev >= 64) return set_error(SOAPB_ERR_ARG, "device index %d out of range", dev);
  std::lock_guard<std::mutex> lock(g_scratch_mu);
  ScratchSlot& slot = g_scratch_slot[dev];
  const unsigned long long id = current_context_id();
  if (!slot.ptr || id == 0 || slot.ctx_id != id) {
    void* p = nullptr;
    // also creates the device's primary context if this thread has none yet
    rc = check_cuda(cudaGetSymbolAddress(&p, g_nl_scratch), "cudaGetSymbolAddress(g_nl_scratch)");
    if (rc) return rc;
    slot.ptr = p;
    slot.ctx_id = current_context_id();
  }
  *out = slot.ptr;
  return SOAPB_OK;
}

}  // namespace soapb

extern "C" int soapb_neighbors_noalloc(const soapb_basis* b, const soapb_structs* s, const soapb_centres* c,
                                       int32_t mode, int64_t* d_pair_off, void* d_pairs, int64_t capacity,
                                       int32_t* d_status, void* stream) {
  int rc = check_inputs(b, s, c);
  if (rc) return rc;
  if (!d_pair_off || !d_status) return set_error(SOAPB_ERR_ARG, "null pair_off or status");
  const NLLayout L = nl_layout(s, c);
  if (L.total > kNoAllocScratchBytes)
    return set_error(SOAPB_ERR_ARG,
                     "soapb_neighbors_noalloc: this input needs %lld bytes of scratch but the fixed scratch array "
                     "holds %lld bytes (about 67,000 atoms with every atom a centre); use soapb_neighbors_count/_fill with a workspace",
                     (long long)L.total, (long long)kNoAllocScratchBytes);
  void* scratch = nullptr;
  if ((rc = scratch_address(&scratch))) return rc;
  // count clears the scratch words that must start at zero (status, bin counts, bin cursors)
  if ((rc = soapb_neighbors_count(b, s, c, mode, scratch, kNoAllocScratchBytes, d_pair_off, stream))) return rc;
  if ((rc = soapb_neighbors_fill(b, s, c, mode, scratch, kNoAllocScratchBytes, d_pair_off, d_pairs, capacity,
                                 stream)))
    return rc;
  const NLWork w = nl_work(L, scratch);
  return check_cuda(cudaMemcpyAsync(d_status, w.status, sizeof(int32_t), cudaMemcpyDeviceToDevice,
                                    (cudaStream_t)stream),
                    "status copy");
}
