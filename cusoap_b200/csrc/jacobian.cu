// Dense descriptor Jacobian d desc[c, f] / d x[a, d], written once per
// element (zeros included) in the DScribe layout (C, n_inc, 3, F).
//
// Reference: derivatives_analytical_ps (soap_generator.py:2270-2626) and its
// Triton kernels _ps_uv_kernel / _ps_jacobian_dense_kernel /
// _cc_jacobian_dense_kernel (:50-220).  Per edge e (centre c -> atom a,
// rvec = x_a - x_c, species s):
//   g[d, n, lm] = r_d Bhat_nl R_lm + B_nl dR_lm/dx_d
//   cc:  d c[s, n, lm] / d x_a,d         = sum_e g
//   ps:  d p[(j n), (j' n'), l] / dx_a,d = pref_l sum_e [ d_{j s} (r_d Bhat_nl U[j'n'l] + B_nl V_d[j'n'l])
//                                                        + d_{j' s} (r_d Bhat_n'l U[jnl] + B_n'l V_d[jnl]) ]
//   with U[k q l] = sum_m R_lm c[k q lm], V_d[k q l] = sum_m dR_lm/dx_d c[k q lm].
// Unlike the reference kernels this accumulates every edge of an atom, so
// periodic images are handled; attach=1 adds the centre-motion term
// (-sum over the centre's edges on the centre atom's row).
//
// The output is ~99% of the traffic (45 GB for 3000 atoms at F=420) and
// mostly zeros, so the kernel is an HBM write stream: one CTA per centre
// writes its contiguous (n_inc, 3, F) block front to back, computing the few
// nonzero rows in between.  Each staged edge is pre-contracted into
//   X0[a] = {U, Q, P_x, V_x},  X1[a] = {P_y, V_y, P_z, V_z},  a = (j, n, l),
//   Q = d_{j s} B_nl, P_d = d_{j s} r_d Bhat_nl (times the entry's sign),
// so a nonzero element is pref_l (P_d[a] U[b] + Q[a] V_d[b] + P_d[b] U[a] + Q[b] V_d[a]):
// four FMAs on two pairs of 16-byte shared-memory loads (X is stored l-major,
// a = (l S + j) N + n, so consecutive features read consecutive float4s).
//
// Two launches, sharing a workspace:
//   k_jac_entries  per centre: the (row, edge) entries of its included atoms,
//                  sorted by row, a bitmap of its nonzero rows, and its
//                  compute tasks: runs of whole rows of about eb entries;
//   k_jacobian     warp roles inside every block: warp 0 streams the block's
//                  share of the zero rows (64-row chunks in global row order)
//                  with TMA bulk copies of a zero tile in shared memory --
//                  one issuing lane, no load/store-unit traffic -- while warps
//                  1..7 take compute tasks (entries staged in shared memory,
//                  each thread four consecutive features of a row in the three
//                  directions, stored as 16-byte vectors).
// A task is one staged batch, not one centre: staging a batch is a chain of
// barriers and shared-memory latencies, so with centres as tasks a centre's
// batches ran one after the other in one block while most blocks had no centre
// (50 centres of a 3000-atom cluster, F = 420: 452 us a launch, 148 us as it is
// now, 115 us of it to write the output; 1536 atoms, 12 GB: 2.35 and 1.76 ms).
// Zero and nonzero rows are disjoint, so every element is written once and the
// two roles never synchronise.
#include "common.cuh"

namespace soapb {

struct JacArgs {
  const int64_t* pair_off;
  const float4* pairs;
  const float* coeff;
  const int* inc_row;
  const int* centre_atom;
  const float* tab_b;
  const float* tab_bh;   // D = d(w B)/dr; Bhat = D / r
  const float* selfv;    // w0 B_nl(0) for r = 0 edges
  const int* ftab;
  float* out;
  int* counter;                  // {next task, next zero chunk, tasks, 0}
  int2* tasks;                   // {centre, entries (negative: the centre's own row)}, {first entry in ent: low, high
                                 // word}; 8-byte loads, the alignment that a workspace always needed
  unsigned long long* ent;       // sorted entries, centre c at ent_mult * pair_off[c]
  unsigned long long* ent_tmp;   // merge buffer of a centre with more than cap entries, same offsets
  unsigned int* bitmap;          // (n_centres * n_inc) nonzero-row bits
  int64_t n_centres, n_inc;
  int N, S, nseg, F, mode, attach, cap, eb, ent_mult;
  int centre_eb;  // entries per batch of a moving centre's own row (centre_row), 0: as any other row
  float inv_h;
};

template <int L>
struct JacShape {
  static constexpr int K = (L + 1) * (L + 1);
  static constexpr int KC = K | 1;
  static constexpr int LP = L + 1;
  // staged entry: header(8: rx ry rz species sign) | B, Bhat (NF each) | R (K) | dR (3K) |
  // X0, X1 (4 SNL floats each, ps only, 16-byte aligned); total rounded to 16 bytes
  __host__ __device__ static int xoff(int N) { return (8 + 2 * N * LP + 4 * K + 3) & ~3; }
  __host__ __device__ static int entry_floats(int N, int S, int mode) {
    const int f = xoff(N) + (mode == SOAPB_OUT_PS ? 8 * S * N * LP : 0);
    return (f + 3) & ~3;
  }
  __host__ __device__ static int cs_floats(int N, int S) { return (S * N * KC + 3) & ~3; }
};

// The (row, edge) entries of the centre's included atoms, in any order: each is
// handed to put(k, key) with k = 0, 1, ... from a block counter.  Returns the
// count (all threads of the CTA; ends with a barrier).
template <class Put>
__device__ int gather_entries(const JacArgs& a, int64_t p0, int P, int catom, int crow, int* s_nent, Put put) {
  const int tid = threadIdx.x, nth = blockDim.x;
  if (tid == 0) *s_nent = 0;
  __syncthreads();
  for (int e = tid; e < P; e += nth) {
    const int atom = __float_as_int(a.pairs[p0 + e].w) & kAtomMask;
    if (a.attach && atom == catom) continue;  // centre and neighbour terms cancel
    const int row = a.inc_row[atom];
    if (row >= 0) put(atomicAdd(s_nent, 1), ((unsigned long long)row << 32) | (unsigned)e);
    if (crow >= 0) put(atomicAdd(s_nent, 1), ((unsigned long long)crow << 32) | (unsigned)e);
  }
  __syncthreads();
  return *s_nent;
}

// Ascending bitonic sort of n2 (a power of two) keys in shared memory (all threads of the CTA).
__device__ void block_bitonic(unsigned long long* keys, int n2) {
  const int tid = threadIdx.x, nth = blockDim.x;
  for (int k = 2; k <= n2; k <<= 1)
    for (int j = k >> 1; j > 0; j >>= 1) {
      for (int i = tid; i < n2; i += nth) {
        const int ixj = i ^ j;
        if (ixj > i) {
          const unsigned long long x = keys[i], y = keys[ixj];
          const bool asc = (i & k) == 0;
          if (asc ? (x > y) : (x < y)) { keys[i] = y; keys[ixj] = x; }
        }
      }
      __syncthreads();
    }
}

constexpr int kEntThreads = 256;

// Ascending bitonic sort of n <= R kEntThreads keys, R per thread in registers
// (key i of thread i mod kEntThreads): exchanges inside a warp are shuffles and
// those of a multiple of the block stay in the thread, so 12 of the 55 steps of
// 1024 keys go through shared memory and its barriers instead of all of them.
// 1536 atoms at 384 entries a centre: k_jac_entries 67 -> 36 us; 50 centres at 700:
// 17 -> 11 us.
template <int R>
__device__ void register_bitonic(unsigned long long* keys, int n) {
  const int tid = threadIdx.x;
  unsigned long long v[R];
#pragma unroll
  for (int r = 0; r < R; ++r) v[r] = tid + kEntThreads * r < n ? keys[tid + kEntThreads * r] : ~0ull;
  int n2 = 1;
  while (n2 < n) n2 <<= 1;
  auto keep = [&](int r, unsigned long long other, int k, int j) {  // this key's or its partner's, by direction
    const bool low = (tid & j) == 0, asc = ((tid + kEntThreads * r) & k) == 0;
    v[r] = (low == asc) == (other < v[r]) ? other : v[r];
  };
  for (int k = 2; k <= n2; k <<= 1)
    for (int j = k >> 1; j > 0; j >>= 1) {
      if (j >= kEntThreads) {
#pragma unroll
        for (int d = 1; d < R; d <<= 1)
          if (j == d * kEntThreads)
#pragma unroll
            for (int r = 0; r < R; ++r)
              if ((r & d) == 0) {
                const unsigned long long x = v[r], y = v[r | d];
                if ((x > y) == (((tid + kEntThreads * r) & k) == 0)) {
                  v[r] = y;
                  v[r | d] = x;
                }
              }
      } else if (j >= 32) {
        __syncthreads();
#pragma unroll
        for (int r = 0; r < R; ++r) keys[tid + kEntThreads * r] = v[r];
        __syncthreads();
#pragma unroll
        for (int r = 0; r < R; ++r) keep(r, keys[(tid ^ j) + kEntThreads * r], k, j);
      } else {
#pragma unroll
        for (int r = 0; r < R; ++r) keep(r, __shfl_xor_sync(0xffffffffu, v[r], j), k, j);
      }
    }
  __syncthreads();
#pragma unroll
  for (int r = 0; r < R; ++r)
    if (tid + kEntThreads * r < n) keys[tid + kEntThreads * r] = v[r];
  __syncthreads();
}

// Sorts n keys (n <= cap) in shared memory (room for a power of two, and for
// kEntThreads keys).
__device__ void sort_tile(unsigned long long* keys, int n) {
  __syncthreads();
  if (n <= kEntThreads) return register_bitonic<1>(keys, n);
  if (n <= 2 * kEntThreads) return register_bitonic<2>(keys, n);
  if (n <= 4 * kEntThreads) return register_bitonic<4>(keys, n);
  int n2 = 1;
  while (n2 < n) n2 <<= 1;
  for (int i = n + threadIdx.x; i < n2; i += blockDim.x) keys[i] = ~0ull;
  __syncthreads();
  block_bitonic(keys, n2);
}

// Merges the sorted runs A[0, na) and B[0, nb) (distinct keys) into O: thread t
// writes a contiguous share of the outputs, starting where a binary search of
// the merge path puts its first output (all threads of the CTA).
__device__ void merge_runs(const unsigned long long* A, int na, const unsigned long long* B, int nb,
                           unsigned long long* O) {
  const int total = na + nb, nth = blockDim.x;
  const int per = (total + nth - 1) / nth;
  const int o0 = threadIdx.x * per, o1 = min(o0 + per, total);
  if (o0 >= total) return;
  int lo = max(0, o0 - nb), hi = min(o0, na);
  while (lo < hi) {  // fewest outputs from A such that the next A key follows the last B key taken
    const int i = (lo + hi) >> 1;
    if (A[i] < B[o0 - i - 1]) lo = i + 1;
    else hi = i;
  }
  int i = lo, j = o0 - lo;
  for (int o = o0; o < o1; ++o) O[o] = (j >= nb || (i < na && A[i] < B[j])) ? A[i++] : B[j++];
}

// Per-centre entries sorted by row into dst (global memory).  Centres whose
// entries fit the shared-memory buffer (cap keys) are gathered and sorted
// there.  Larger centres are gathered straight into dst, sorted in tiles of
// cap keys in shared memory, and the sorted runs merged pairwise through tmp
// (the same slot in a second buffer) until one run is left.  Keys are
// distinct, so the order is the same however the gather was interleaved.
__device__ int centre_entries(const JacArgs& a, int64_t p0, int P, int catom, int crow, unsigned long long* skeys,
                              unsigned long long* dst, unsigned long long* tmp, int* s_nent) {
  const int tid = threadIdx.x, nth = blockDim.x;
  if (a.ent_mult * P <= a.cap) {
    const int nent = gather_entries(a, p0, P, catom, crow, s_nent,
                                    [&](int k, unsigned long long key) { skeys[k] = key; });
    sort_tile(skeys, nent);
    for (int i = tid; i < nent; i += nth) dst[i] = skeys[i];
    __syncthreads();
    return nent;
  }
  const int nent = gather_entries(a, p0, P, catom, crow, s_nent,
                                  [&](int k, unsigned long long key) { dst[k] = key; });
  for (int t0 = 0; t0 < nent; t0 += a.cap) {
    const int n = min(a.cap, nent - t0);
    for (int i = tid; i < n; i += nth) skeys[i] = dst[t0 + i];
    sort_tile(skeys, n);
    for (int i = tid; i < n; i += nth) dst[t0 + i] = skeys[i];
    __syncthreads();
  }
  unsigned long long *src = dst, *out = tmp;
  for (int w = a.cap; w < nent; w *= 2) {
    for (int lo = 0; lo < nent; lo += 2 * w) {
      const int mid = min(lo + w, nent), hi = min(lo + 2 * w, nent);
      merge_runs(src + lo, mid - lo, src + mid, hi - mid, out + lo);
    }
    __syncthreads();
    unsigned long long* s = src;
    src = out;
    out = s;
  }
  if (src != dst) {
    for (int i = tid; i < nent; i += nth) dst[i] = src[i];
    __syncthreads();
  }
  return nent;
}

__global__ void __launch_bounds__(kEntThreads) k_jac_entries(JacArgs a) {
  extern __shared__ __align__(16) unsigned long long skeys[];
  __shared__ int s_nent, s_task0;
  for (int64_t c = blockIdx.x; c < a.n_centres; c += gridDim.x) {
    const int64_t p0 = a.pair_off[c];
    const int P = (int)(a.pair_off[c + 1] - p0);
    const int catom = a.attach ? a.centre_atom[c] : -1;
    const int crow = (catom >= 0) ? a.inc_row[catom] : -1;
    unsigned long long* dst = a.ent + (size_t)a.ent_mult * p0;
    unsigned long long* tmp = a.ent_tmp + (size_t)a.ent_mult * p0;
    const int nent = centre_entries(a, p0, P, catom, crow, skeys, dst, tmp, &s_nent);
    for (int i = threadIdx.x; i < nent; i += blockDim.x) {
      const int64_t r = (int64_t)c * a.n_inc + (int64_t)(dst[i] >> 32);
      atomicOr(a.bitmap + (r >> 5), 1u << (r & 31));
    }
    // compute tasks: runs of about eb entries, both ends moved up to the next row boundary.  A
    // moving centre's own row holds an entry of every edge: a task of its own (centre_row) splits
    // the others into those before it, [0, g0), and after it, [g1, nent).
    auto lower = [&](unsigned long long key) {  // first entry not below key
      int lo = 0, hi = nent;
      while (lo < hi) {
        const int mid = (lo + hi) >> 1;
        if (dst[mid] < key) lo = mid + 1;
        else hi = mid;
      }
      return lo;
    };
    auto row_boundary = [&](int i) {  // first entry >= i that starts a row
      if (i == 0 || i >= nent) return min(i, nent);
      const unsigned long long next = ((dst[i - 1] >> 32) + 1) << 32;  // first key of the following rows
      return dst[i] >= next ? i : lower(next);
    };
    int g0 = nent, g1 = nent;
    if (crow >= 0 && a.centre_eb > 0) {
      g0 = lower((unsigned long long)crow << 32);
      g1 = lower(((unsigned long long)crow + 1) << 32);
      if (g1 - g0 <= a.eb) g0 = g1 = nent;
    }
    const int n0 = (g0 + a.eb - 1) / a.eb, n1 = (nent - g1 + a.eb - 1) / a.eb, own = g1 > g0 ? 1 : 0;
    const int nt = n0 + n1 + own;
    if (threadIdx.x == 0) s_task0 = nt > 0 ? atomicAdd(a.counter + 2, nt) : 0;
    __syncthreads();
    for (int k = threadIdx.x; k < nt; k += blockDim.x) {
      int b, e;
      if (k < own) {  // the long task first
        b = g0;
        e = g1;
      } else if (k < own + n0) {
        b = min(row_boundary((k - own) * a.eb), g0);
        e = min(row_boundary((k - own + 1) * a.eb), g0);
      } else {
        b = row_boundary(g1 + (k - own - n0) * a.eb);
        e = row_boundary(g1 + (k - own - n0 + 1) * a.eb);
      }
      const unsigned long long first = (unsigned long long)((size_t)a.ent_mult * p0 + b);
      int2* t = a.tasks + 2 * (int64_t)(s_task0 + k);
      t[0] = make_int2((int)c, k < own ? b - e : e - b);
      t[1] = make_int2((int)(unsigned)first, (int)(unsigned)(first >> 32));
    }
    __syncthreads();
  }
}

constexpr int kZeroTile = 16384;  // bytes of the shared-memory zero tile
constexpr int kZeroChunkRows = 64;

__device__ __forceinline__ void bulk_s2g(void* g, const void* s, uint32_t bytes) {
  asm volatile("cp.async.bulk.global.shared::cta.bulk_group [%0], [%1], %2;\n" ::"l"(g),
               "r"((uint32_t)__cvta_generic_to_shared(s)), "r"(bytes)
               : "memory");
}

// Zero rows of 64-row chunks (global row order) claimed from a work queue
// (zq), by TMA bulk copies of the zero tile; lane 0 issues, the copies run
// asynchronously and the lane waits for all of them before returning (the
// tile must outlive them).  Every block's zero warp runs this from the start
// and its compute warps join once the task queue is empty, so the zero
// stream ends together with the compute work.  Rows are 12 F bytes: a run of
// rows that does not start or end on 16 bytes (F not a multiple of 4) gets its
// first and last words by plain stores.  (4-byte stores of such runs by the
// zero warps alone, of two blocks per SM, made them the longer part: 501 atoms,
// F = 63: 196 us, 118 us with these copies.)
__device__ void jac_zero_rows(const JacArgs& a, const void* ztile, int* zq) {
  if ((threadIdx.x & 31) != 0) return;
  const int64_t nrows = a.n_centres * a.n_inc;
  const int64_t row_words = 3 * (int64_t)a.F;
  const int64_t nchunks = (nrows + kZeroChunkRows - 1) / kZeroChunkRows;
  for (;;) {
    const int64_t k = (int64_t)(unsigned)atomicAdd(zq, 1);
    if (k >= nchunks) break;
    const int64_t r0 = k * kZeroChunkRows, r1 = min(r0 + (int64_t)kZeroChunkRows, nrows);
    int64_t run = -1;
    for (int64_t r = r0; r <= r1; ++r) {
      const bool zero = (r < r1) && !((a.bitmap[r >> 5] >> (r & 31)) & 1u);
      if (zero && run < 0) run = r;
      if (!zero && run >= 0) {  // zero rows [run, r)
        const int64_t i0 = run * row_words, i1 = r * row_words;
        const int64_t b0 = min((i0 + 3) & ~(int64_t)3, i1), b1 = max(i1 & ~(int64_t)3, b0);  // multiples of 16 bytes
        for (int64_t i = i0; i < b0; ++i) __stcs(a.out + i, 0.0f);
        for (int64_t i = b0; i < b1; i += kZeroTile / 4) {
          const int64_t bytes = 4 * (b1 - i);
          bulk_s2g(a.out + i, ztile, (uint32_t)(bytes < kZeroTile ? bytes : kZeroTile));
        }
        for (int64_t i = b1; i < i1; ++i) __stcs(a.out + i, 0.0f);
        run = -1;
      }
    }
    asm volatile("cp.async.bulk.commit_group;\n" ::: "memory");
  }
  asm volatile("cp.async.bulk.wait_group 0;\n" ::: "memory");
}

// Named barrier over the compute warps only (id 1; id 0 is __syncthreads).
__device__ __forceinline__ void compute_bar(int nthreads) {
  asm volatile("bar.sync 1, %0;\n" ::"r"(nthreads) : "memory");
}

// Asynchronous copy of one T (4, 8 or 16 bytes) global -> shared.
template <class T>
__device__ __forceinline__ void copy_async(T* s, const T* g) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], %2;\n" ::"r"((uint32_t)__cvta_generic_to_shared(s)), "l"(g),
               "n"(sizeof(T))
               : "memory");
}
__device__ __forceinline__ void copy_async_wait() { asm volatile("cp.async.wait_all;\n" ::: "memory"); }

// Entry of thread tid (< nb): header, harmonics and their gradients.
template <int L>
__device__ __forceinline__ void stage_harmonics(const JacArgs& a, const float4& pr, bool centre_row, float* h) {
  constexpr int K = JacShape<L>::K;
  const int NF = a.N * (L + 1);
  const float r = sqrtf(fmaf(pr.z, pr.z, fmaf(pr.x, pr.x, __fmul_rn(pr.y, pr.y))));
  int seg;
  float t;
  seg_coord(r, a.inv_h, a.nseg, seg, t);
  h[0] = pr.x; h[1] = pr.y; h[2] = pr.z;
  h[3] = (float)((unsigned)__float_as_int(pr.w) >> kAtomBits);
  h[4] = centre_row ? -1.0f : 1.0f;
  h[5] = r; h[6] = t; h[7] = __int_as_float(seg);
  float* R = h + 8 + 2 * NF;
  float* dR = R + K;
  SolidHarmonics<L>::with_gradients(pr.x, pr.y, pr.z, [&](int idx, float v, float dx, float dy, float dz) {
    R[idx] = v; dR[idx] = dx; dR[K + idx] = dy; dR[2 * K + idx] = dz;
  });
}

// Radial functions of the nb staged entries (all compute threads).
__device__ __forceinline__ void stage_radial(const JacArgs& a, int nb, float* ed, int EF, int NF, int tid, int nth) {
  auto one = [&](float* h, int fn) {
    const float r = h[5], t = h[6];
    const int seg = __float_as_int(h[7]);
    float cb[kNCoef], cd[kNCoef];
    load_coef(a.tab_b, seg, fn, NF, cb);
    load_coef(a.tab_bh, seg, fn, NF, cd);
    h[8 + fn] = (r > 0.0f) ? horner7(cb, t) : __ldg(a.selfv + fn);
    h[8 + NF + fn] = (r > 0.0f) ? horner7(cd, t) / r : 0.0f;
  };
  if (NF <= nth) {  // thread owns radial function fn, entries stepped (division-free loop)
    const int fn = tid % NF, istep = nth / NF;
    if (tid < istep * NF)
      for (int i = tid / NF; i < nb; i += istep) one(ed + (size_t)i * EF, fn);
  } else {  // more radial functions than threads
    for (int t = tid; t < nb * NF; t += nth) one(ed + (size_t)(t / NF) * EF, t % NF);
  }
}

// ps: the pre-contracted vectors X0, X1 of the nb staged entries (all compute threads).
template <int L>
__device__ __forceinline__ void stage_vectors(const JacArgs& a, int nb, const float* cs, float* ed, int EF,
                                              const float* sqrt_pref, int tid, int nth) {
  using Sh = JacShape<L>;
  constexpr int K = Sh::K, KC = Sh::KC, LP = Sh::LP;
  const int N = a.N, S = a.S, NF = N * LP, SNL = S * N * LP, XO = Sh::xoff(N);
  {
    // thread -> coefficient index ai = (l S + j) N + n (decoded once) and first entry;
    // entries stepped by istep (division-free loop)
    const bool small = SNL <= nth;
    const int istep = small ? nth / SNL : 1;
    const int ai0 = small ? tid % SNL : tid;
    const int i0 = small ? (tid < istep * SNL ? tid / SNL : nb) : 0;
    for (int ai = ai0; ai < SNL; ai += (small ? SNL : nth)) {
      const int l = ai / (S * N), jn = ai % (S * N);
      const int j = jn / N, n = jn % N;
      const float* cr = cs + jn * KC + l * l;
      for (int i = i0; i < nb; i += istep) {
        const float* h = ed + (size_t)i * EF;
        const float* R = h + 8 + 2 * NF;
        const float* dR = R + K;
        float u = 0.f, v0 = 0.f, v1 = 0.f, v2 = 0.f;
        for (int m = 0; m < 2 * l + 1; ++m) {
          const float cv = cr[m];
          u = fmaf(R[l * l + m], cv, u);
          v0 = fmaf(dR[l * l + m], cv, v0);
          v1 = fmaf(dR[K + l * l + m], cv, v1);
          v2 = fmaf(dR[2 * K + l * l + m], cv, v2);
        }
        // both factors carry sqrt(pref_l): the value is bilinear in X[a], X[b] of the same l
        const float sp = sqrt_pref[l];
        const bool own = ((int)h[3] == j);
        const float q = own ? sp * h[4] * h[8 + l * N + n] : 0.0f;
        const float bh = own ? sp * h[4] * h[8 + NF + l * N + n] : 0.0f;
        u *= sp; v0 *= sp; v1 *= sp; v2 *= sp;
        float4* X = reinterpret_cast<float4*>(ed + (size_t)i * EF + XO);
        X[ai] = make_float4(u, q, h[0] * bh, v0);
        X[SNL + ai] = make_float4(h[1] * bh, v1, h[2] * bh, v2);
      }
    }
  }
}

// The four features 4q .. 4q + 3 of a thread, decoded once per task.  ps: the
// coefficient-pair code ia | ib << 12 | l << 24.  cc: species, radial function
// index, source harmonic and output scale.
struct QuadCode {
  int code[4], sp[4], src[4];
  float scale[4];
};

template <int L>
__device__ __forceinline__ void quad_decode(const JacArgs& a, int q, QuadCode& qc) {
  constexpr int K = JacShape<L>::K;
  const int N = a.N, F = a.F;
  if (a.mode == SOAPB_OUT_PS) {
    if ((F & 3) == 0) {
      const int4 c4 = __ldg(reinterpret_cast<const int4*>(a.ftab) + q);
      qc.code[0] = c4.x; qc.code[1] = c4.y; qc.code[2] = c4.z; qc.code[3] = c4.w;
    } else {
#pragma unroll
      for (int k = 0; k < 4; ++k) qc.code[k] = (4 * q + k < F) ? __ldg(a.ftab + 4 * q + k) : 0;
    }
  } else {
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const int f = min(4 * q + k, F - 1);
      const int sf = f / (N * K), rem = f - sf * N * K, n = rem / K, lo = rem - n * K;
      int src = lo;
      // DScribe cc layout: l = 1 stored (z, x, y) = source lm (2, 3, 1); lm >= 4 scaled by pi^-3/2
      if (lo >= 1 && lo <= 3) src = (lo == 3) ? 1 : lo + 1;
      int l = 0;
      while ((l + 1) * (l + 1) <= src) ++l;
      qc.code[k] = l * N + n;
      qc.sp[k] = (4 * q + k < F) ? sf : -1;
      qc.src[k] = src;
      qc.scale[k] = lo >= 4 ? (float)(1.0 / (kPi * 1.7724538509055160273)) : 1.0f;
    }
  }
}

// Values of a thread's four features in the three directions, summed over
// staged entries [g0, g1).  ps: X already carries sqrt(pref_l) on both sides.
template <int L>
__device__ __forceinline__ void quad_values(const JacArgs& a, const float* ed, int EF, int g0, int g1,
                                            const QuadCode& qc, float (&v)[3][4]) {
  using Sh = JacShape<L>;
  constexpr int K = Sh::K, LP = Sh::LP;
  const int N = a.N, S = a.S, NF = N * LP, SNL = S * N * LP, XO = Sh::xoff(N);
#pragma unroll
  for (int k = 0; k < 4; ++k) v[0][k] = v[1][k] = v[2][k] = 0.f;
  if (a.mode == SOAPB_OUT_PS) {
    for (int i = g0; i < g1; ++i) {
      const float4* X = reinterpret_cast<const float4*>(ed + (size_t)i * EF + XO);
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        const int ia = qc.code[k] & 4095, ib = (qc.code[k] >> 12) & 4095;
        const float4 pa = X[ia], qa = X[SNL + ia], pb = X[ib], qb = X[SNL + ib];
        v[0][k] += fmaf(pb.y, pa.w, fmaf(pb.z, pa.x, fmaf(pa.z, pb.x, __fmul_rn(pa.y, pb.w))));
        v[1][k] += fmaf(pb.y, qa.y, fmaf(qb.x, pa.x, fmaf(qa.x, pb.x, __fmul_rn(pa.y, qb.y))));
        v[2][k] += fmaf(pb.y, qa.w, fmaf(qb.z, pa.x, fmaf(qa.z, pb.x, __fmul_rn(pa.y, qb.w))));
      }
    }
  } else {
    for (int i = g0; i < g1; ++i) {
      const float* h = ed + (size_t)i * EF;
      const float* R = h + 8 + 2 * NF;
      const float* dR = R + K;
      const int sp = (int)h[3];
      const float sign = h[4], x = h[0], y = h[1], z = h[2];
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        if (qc.sp[k] != sp) continue;
        const int fn = qc.code[k], src = qc.src[k];
        const float bh = sign * h[8 + NF + fn] * R[src], b = sign * h[8 + fn];
        v[0][k] += qc.scale[k] * (x * bh + b * dR[src]);
        v[1][k] += qc.scale[k] * (y * bh + b * dR[K + src]);
        v[2][k] += qc.scale[k] * (z * bh + b * dR[2 * K + src]);
      }
    }
  }
}

// A moving centre's own row: minus the sum over all its n edges.  The sum of
// dc / dx_d over the edges is formed first, D[d][s][n][lm] in shared memory
// (3 N K FMAs an edge), and contracted with the coefficients once, instead of
// 12 FMAs an edge for every feature in batches of eb that follow one another
// (192 atoms, 130 edges a centre, cc: 193 us against 89 us, entries
// included).  The edges are sorted by species, so a thread keeps its
// (n, lm) in registers and adds it to D when the species changes.  An edge's
// two terms, which often cancel, are added first, then eight edges, then those
// of a batch: 1.74e-7 from float64 for these 192 atoms.  One FMA after the other
// is 1.92e-7 away, batches of edges for every feature 1.81e-7; the time is the same.
// pref is the factor sqrt(8 pi^2 / (2 l + 1)) itself: the square of its root that
// the staged vectors carry is off by up to 1.25e-7, for every feature of an l.
template <int L>
__device__ void centre_row(const JacArgs& a, int64_t p0, const unsigned long long* keys, int n, const float* cs,
                           float* smem, float* orow, const float* pref, int tid, int nth) {
  using Sh = JacShape<L>;
  constexpr int K = Sh::K, KC = Sh::KC;
  const int N = a.N, SNK = a.S * N * K, NK = N * K, NF = N * (L + 1), EF = Sh::xoff(N), F = a.F;
  float* D = smem;
  float* ed = smem + ((3 * SNK + 3) & ~3);
  for (int i = tid; i < 3 * SNK; i += nth) D[i] = 0.0f;
  for (int b0 = 0; b0 < n; b0 += a.centre_eb) {
    const int nb = min(a.centre_eb, n - b0);
    if (tid < nb)
      stage_harmonics<L>(a, a.pairs[p0 + (int)(keys[b0 + tid] & 0xffffffffu)], true, ed + (size_t)tid * EF);
    compute_bar(nth);
    stage_radial(a, nb, ed, EF, NF, tid, nth);
    compute_bar(nth);
    for (int it = tid; it < NK; it += nth) {
      const int nn = it / K, lm = it - nn * K;
      int l = 0;
      while ((l + 1) * (l + 1) <= lm) ++l;
      const int fn = 8 + l * N + nn, iR = 8 + 2 * NF + lm;
      float v0 = 0.0f, v1 = 0.0f, v2 = 0.0f, w0 = 0.0f, w1 = 0.0f, w2 = 0.0f;
      int cur = (int)ed[3];
      auto flush = [&]() {
        float* d = D + cur * NK + it;
        d[0] -= w0 + v0;
        d[SNK] -= w1 + v1;
        d[2 * SNK] -= w2 + v2;
        v0 = v1 = v2 = w0 = w1 = w2 = 0.0f;
      };
      for (int i = 0; i < nb; ++i) {
        const float* h = ed + (size_t)i * EF;
        if ((int)h[3] != cur) {
          flush();
          cur = (int)h[3];
        }
        if ((i & 7) == 0) {
          w0 += v0; w1 += v1; w2 += v2;
          v0 = v1 = v2 = 0.0f;
        }
        const float bR = h[fn + NF] * h[iR], b = h[fn];
        v0 += fmaf(h[0], bR, b * h[iR + K]);
        v1 += fmaf(h[1], bR, b * h[iR + 2 * K]);
        v2 += fmaf(h[2], bR, b * h[iR + 3 * K]);
      }
      flush();
    }
    compute_bar(nth);
  }
  if (a.mode == SOAPB_OUT_PS) {
    for (int f = tid; f < F; f += nth) {
      const int code = __ldg(a.ftab + f), l = code >> 24, base = l * a.S * N;
      const int ja = (code & 4095) - base, jb = ((code >> 12) & 4095) - base;
      const float *ca = cs + ja * KC + l * l, *cb = cs + jb * KC + l * l;
      const float *da = D + ja * K + l * l, *db = D + jb * K + l * l;
      float v0 = 0.0f, v1 = 0.0f, v2 = 0.0f;
      for (int m = 0; m < 2 * l + 1; ++m) {
        const float x = ca[m], y = cb[m];
        v0 += da[m] * y + x * db[m];
        v1 += da[SNK + m] * y + x * db[SNK + m];
        v2 += da[2 * SNK + m] * y + x * db[2 * SNK + m];
      }
      __stcs(orow + f, pref[l] * v0);
      __stcs(orow + F + f, pref[l] * v1);
      __stcs(orow + 2 * F + f, pref[l] * v2);
    }
  } else {
    for (int f = tid; f < F; f += nth) {
      const int sn = f / K, lo = f - sn * K;
      const int src = (lo >= 1 && lo <= 3) ? ((lo == 3) ? 1 : lo + 1) : lo;  // as in quad_decode
      const float scale = lo >= 4 ? (float)(1.0 / (kPi * 1.7724538509055160273)) : 1.0f;
      for (int d = 0; d < 3; ++d) __stcs(orow + d * F + f, scale * D[d * SNK + sn * K + src]);
    }
  }
  compute_bar(nth);  // D, the entries and cs are rewritten by the next task
}

// Nonzero rows: tasks from a work queue, a task's entries staged in batches of
// eb (one batch, unless a row has many entries), each thread (row group, four
// consecutive features), stored as 16-byte vectors.  A task is a chain of short
// stages, so its global loads run ahead: the next task is claimed while the
// harmonics are computed, its keys are loaded during the radial stage and its
// pairs during the contraction, and the centre's coefficient row comes in by
// asynchronous copies.  1536 atoms, entries (then 67 us) included: 2.08 ms
// without this, 1.83 ms with it (12 GB take 1.81 ms at the measured copy rate).
//
// Two blocks per SM, whose registers hold the four features of a thread; three
// (80 registers, small spills) for rows of few features, where the stages'
// latencies are the time (see JacDispatch).
template <int L, int B>
__global__ void __launch_bounds__(256, B) k_jacobian(JacArgs a) {
  using Sh = JacShape<L>;
  constexpr int K = Sh::K, KC = Sh::KC;
  constexpr int kCT = 224;  // compute threads (warps 1..7)
  const int N = a.N, S = a.S, F = a.F;
  const int Q = (F + 3) >> 2;
  const bool vec = (F & 3) == 0;
  extern __shared__ __align__(128) float smf[];
  float* ztile = smf;                            // kZeroTile bytes of zeros
  float* cs = ztile + kZeroTile / 4;
  float* ed = cs + Sh::cs_floats(N, S);
  const int EF = Sh::entry_floats(N, S, a.mode);
  __shared__ float s_sqrt_pref[kMaxL + 1], s_pref[kMaxL + 1];
  __shared__ int s_gstart[33], s_grow[32];  // first entry and output row of each row group of the batch
  __shared__ int s_ng;
  __shared__ int4 s_task[2];
  // the next task's offset, keys and pairs (an entry's key and pair are written and read by its own thread)
  __shared__ int64_t s_p0;
  __shared__ unsigned long long s_key[32];
  __shared__ __align__(16) float4 s_pair[32];
  if (threadIdx.x <= L) {
    s_pref[threadIdx.x] = sqrtf(8.0f * (float)(kPi * kPi) / (2.0f * threadIdx.x + 1.0f));
    s_sqrt_pref[threadIdx.x] = sqrtf(s_pref[threadIdx.x]);
  }
  for (int i = threadIdx.x; i < kZeroTile / 4; i += blockDim.x) ztile[i] = 0.0f;
  asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");  // tile visible to the bulk-copy engine
  __syncthreads();
  if (threadIdx.x < 32) {  // zero role
    jac_zero_rows(a, ztile, a.counter + 1);
    return;
  }
  // compute role: warps 1..7, named barrier 1
  const int tid = threadIdx.x - 32;
  // thread -> (quad q0, first group g0t): quads stepped by qstep, groups by gstep (division-free loop)
  const int qstep = Q >= kCT ? kCT : Q, gstep = Q >= kCT ? 1 : kCT / Q;
  const int q0 = Q >= kCT ? tid : tid % Q;
  const int g0t = Q >= kCT ? 0 : (tid < gstep * Q ? tid / Q : 1 << 30);
  const int ntasks = a.counter[2];
  const int NF = N * (L + 1), SNK = S * N * K;
  auto claim = [&]() {
    const int t = atomicAdd(a.counter, 1);
    if (t >= ntasks) return make_int4(-1, 0, 0, 0);
    const int2 u = a.tasks[2 * (int64_t)t], v = a.tasks[2 * (int64_t)t + 1];
    return make_int4(u.x, u.y, v.x, v.y);
  };
  auto keys_of = [&](const int4& t) {
    return a.ent + (((unsigned long long)(unsigned)t.w << 32) | (unsigned)t.z);
  };
  if (tid == 0) s_task[0] = claim();
  compute_bar(kCT);
  int4 task = s_task[0];
  if (task.x >= 0 && tid < min(task.y, a.eb)) {
    s_key[tid] = keys_of(task)[tid];
    s_pair[tid] = a.pairs[a.pair_off[task.x] + (int)(s_key[tid] & 0xffffffffu)];
  }
  for (int it = 1; task.x >= 0; it ^= 1) {
    const int64_t c = task.x;
    const int nent = task.y;
    const unsigned long long* keys = keys_of(task);
    int4 next = make_int4(-1, 0, 0, 0);
    if (tid == 0) next = claim();
    for (int i = tid; i < SNK; i += kCT) copy_async(cs + (i / K) * KC + (i % K), a.coeff + (size_t)c * SNK + i);
    const int catom = a.attach ? a.centre_atom[c] : -1;
    const int crow = (catom >= 0) ? a.inc_row[catom] : -1;
    float* obase = a.out + (size_t)c * a.n_inc * 3 * F;
    if (nent < 0) {
      copy_async_wait();  // cs: visible to all after centre_row's first barrier
      centre_row<L>(a, a.pair_off[c], keys, -nent, cs, ed, obase + (size_t)crow * 3 * F, s_pref, tid, kCT);
      if (tid == 0) s_task[it] = next;
      compute_bar(kCT);
      task = s_task[it];
      if (task.x >= 0 && tid < min(task.y, a.eb)) {
        s_key[tid] = keys_of(task)[tid];
        s_pair[tid] = a.pairs[a.pair_off[task.x] + (int)(s_key[tid] & 0xffffffffu)];
      }
      continue;
    }
    int last_row = -1;
    for (int b0 = 0; b0 == 0 || b0 < nent; b0 += a.eb) {
      const int nb = min(a.eb, nent - b0);
      const bool in = tid < nb;
      int row = -1;
      float4 pr = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
      if (in) {
        unsigned long long key;
        if (b0 == 0) {
          key = s_key[tid];
          pr = s_pair[tid];
        } else {  // a row with more entries than one batch holds
          key = keys[b0 + tid];
          pr = a.pairs[a.pair_off[c] + (int)(key & 0xffffffffu)];
        }
        row = (int)(key >> 32);
      }
      if (tid < 32) {  // row groups of this batch (eb <= 32: one lane per entry)
        const int prev = __shfl_up_sync(0xffffffffu, row, 1);
        const unsigned starts = __ballot_sync(0xffffffffu, in && (tid == 0 || row != prev));
        if ((starts >> tid) & 1u) {
          const int g = __popc(starts & ((1u << tid) - 1u));
          s_gstart[g] = tid;
          s_grow[g] = row;
        }
        if (tid == 0) {
          s_ng = __popc(starts);
          s_gstart[__popc(starts)] = nb;
        }
      }
      if (in) stage_harmonics<L>(a, pr, a.attach && row == crow, ed + (size_t)tid * EF);
      if (b0 == 0 && tid == 0) s_task[it] = next;
      compute_bar(kCT);
      if (b0 == 0 && tid < 32 && s_task[it].x >= 0) {
        const int4 tn = s_task[it];
        if (tid < min(tn.y, a.eb)) copy_async(&s_key[tid], keys_of(tn) + tid);
        if (tid == 0) copy_async(&s_p0, a.pair_off + tn.x);
      }
      stage_radial(a, nb, ed, EF, NF, tid, kCT);
      copy_async_wait();
      compute_bar(kCT);
      if (b0 == 0 && s_task[it].x >= 0 && tid < min(s_task[it].y, a.eb))
        copy_async(&s_pair[tid], a.pairs + s_p0 + (int)(s_key[tid] & 0xffffffffu));
      if (a.mode == SOAPB_OUT_PS) {
        stage_vectors<L>(a, nb, cs, ed, EF, s_sqrt_pref, tid, kCT);
        compute_bar(kCT);
      }
      const int ng = s_ng;
      for (int q = q0; q < Q; q += qstep) {
        QuadCode qc;
        quad_decode<L>(a, q, qc);
        for (int g = g0t; g < ng; g += gstep) {
          const int grow = s_grow[g];
          const bool cont = (g == 0 && grow == last_row);  // continues from the previous batch
          float v[3][4];
          quad_values<L>(a, ed, EF, s_gstart[g], s_gstart[g + 1], qc, v);
          float* orow = obase + (size_t)grow * 3 * F;
#pragma unroll
          for (int d = 0; d < 3; ++d) {
            float* p = orow + d * F + 4 * q;
            if (vec) {
              float4 w = make_float4(v[d][0], v[d][1], v[d][2], v[d][3]);
              if (cont) {
                const float4 o = __ldcg(reinterpret_cast<const float4*>(p));  // written by this CTA last batch
                w.x += o.x; w.y += o.y; w.z += o.z; w.w += o.w;
              }
              __stcs(reinterpret_cast<float4*>(p), w);
            } else {
              for (int k = 0; k < 4 && 4 * q + k < F; ++k) p[k] = cont ? __ldcg(p + k) + v[d][k] : v[d][k];
            }
          }
        }
      }
      last_row = ng > 0 ? s_grow[ng - 1] : -1;
      copy_async_wait();
      compute_bar(kCT);  // staged entries, groups and cs are rewritten by the next batch
    }
    task = s_task[it];
  }
  // task queue empty: this warp joins the zero-row stream
  jac_zero_rows(a, ztile, a.counter + 1);
}

// ---------------------------------------------------------------------------
// host side
// ---------------------------------------------------------------------------

struct JacLayout {
  int64_t counter, tasks, ent, ent_tmp, bitmap, total;
};

constexpr int kMinBatch = 4;  // smallest eb (staged entries per task)

static JacLayout jac_layout(int64_t n_centres, int64_t n_pairs, int64_t n_inc, int attach) {
  JacLayout L{};
  int64_t off = 0;
  auto take = [&](int64_t bytes) { const int64_t o = off; off = align_up(off + bytes, 256); return o; };
  L.counter = take(16);  // and the bitmap behind it: cleared together
  L.bitmap = take(4 * ((n_centres * n_inc + 31) / 32));
  // a centre has at most entries / eb + 2 tasks (the parts before and after its own row)
  L.tasks = take(16 * ((attach ? 2 : 1) * n_pairs / kMinBatch + 2 * n_centres + 1));
  L.ent = take(8 * (attach ? 2 : 1) * (n_pairs > 0 ? n_pairs : 1));
  L.ent_tmp = take(8 * (attach ? 2 : 1) * (n_pairs > 0 ? n_pairs : 1));
  L.total = off;
  return L;
}

static int sm_count() {
  int dev = 0, nsm = 148;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev);
  return nsm;
}

template <int L>
struct JacDispatch {
  static int run(JacArgs a, cudaStream_t st) {
    using Sh = JacShape<L>;
    const int nsm = sm_count();
    int rc;
    const int EF = Sh::entry_floats(a.N, a.S, a.mode);
    const size_t base = kZeroTile + 4 * (size_t)Sh::cs_floats(a.N, a.S);
    const size_t budget = 56 * 1024;  // registers allow two CTAs per SM; 80 and 100 KB (32 staged entries) measured equal
    int eb = base < budget ? (int)((budget - base) / (4 * (size_t)EF)) : 0;
    eb = eb > 32 ? 32 : eb;
    if (eb < kMinBatch) eb = kMinBatch;
    a.eb = eb;
    a.centre_eb = 0;
    if (a.attach) {  // what the batch buffer leaves beside D, if it is worth having
      const int left = eb * EF - ((3 * a.S * a.N * Sh::K + 3) & ~3), ceb = left > 0 ? left / Sh::xoff(a.N) : 0;
      if (ceb >= kMinBatch) a.centre_eb = ceb > 224 ? 224 : ceb;
    }
    // 1. entries, bitmap and tasks
    {
      const size_t smem = 8 * (size_t)(a.cap > kEntThreads ? a.cap : kEntThreads);
      auto kern = k_jac_entries;
      rc = check_cuda(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem),
                      "entries smem attribute");
      if (rc) return rc;
      int occ = 1;
      cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, kern, kEntThreads, smem);
      int64_t blocks = (int64_t)nsm * (occ < 1 ? 1 : occ);
      if (blocks > a.n_centres) blocks = a.n_centres;
      kern<<<(unsigned)blocks, kEntThreads, smem, st>>>(a);
      if ((rc = check_launch("k_jac_entries"))) return rc;
    }
    // 2. one launch: in every block warp 0 streams zero rows, warps 1..7 compute
    const size_t smem = base + 4 * (size_t)eb * EF;
    if (smem > 220 * 1024) return set_error(SOAPB_ERR_UNSUPPORTED, "jacobian shared memory %zu B too large", smem);
    // Three blocks per SM for l_max <= 4 with at most 192 features and a centre for each block.
    // 900 atoms: F = 8 97 -> 85 us, F = 144 284 -> 263, F = 180 359 -> 327; 1536 atoms, F = 72:
    // 607 -> 540.  More features or fewer centres are slower with three (900 atoms, F = 272: 407
    // and 415 us; 192 atoms, F = 144: 46 and 53).
    auto kern = k_jacobian<L, 2>;
    if constexpr (L <= 4)
      if (a.F <= 192 && a.n_centres >= 3 * (int64_t)nsm) kern = k_jacobian<L, 3>;
    rc = check_cuda(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem),
                    "jacobian smem attribute");
    if (rc) return rc;
    int occ = 1;
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, kern, 256, smem);
    const int64_t blocks = (int64_t)nsm * (occ < 1 ? 1 : occ);
    kern<<<(unsigned)blocks, 256, smem, st>>>(a);
    return check_launch("k_jacobian");
  }
};

}  // namespace soapb

using namespace soapb;

extern "C" int soapb_jacobian_workspace(const soapb_basis* b, int64_t n_centres, int64_t n_pairs, int64_t n_inc,
                                        int32_t attach, int64_t* bytes) {
  if (!b || !bytes) return set_error(SOAPB_ERR_ARG, "null argument");
  if (n_centres < 0 || n_pairs < 0 || n_inc < 0) return set_error(SOAPB_ERR_ARG, "negative sizes");
  *bytes = jac_layout(n_centres, n_pairs, n_inc, attach).total;
  return SOAPB_OK;
}

extern "C" int soapb_jacobian(const soapb_basis* b, int64_t n_centres, const int64_t* d_pair_off, const void* d_pairs,
                              int64_t n_pairs, const float* d_coeff, const int32_t* d_inc_row, int64_t n_inc,
                              const int32_t* d_centre_atom, int32_t attach, int32_t max_pairs, int32_t out_mode,
                              float* d_out, void* d_work, int64_t work_bytes, int32_t* d_status, void* stream) {
  if (!b || !b->dev) return set_error(SOAPB_ERR_ARG, "basis not built");
  if (out_mode != SOAPB_OUT_PS && out_mode != SOAPB_OUT_CC) return set_error(SOAPB_ERR_ARG, "bad out_mode");
  if (n_centres <= 0 || n_inc <= 0) return SOAPB_OK;
  if (!d_pair_off || !d_coeff || !d_inc_row || !d_out || !d_status || !d_work)
    return set_error(SOAPB_ERR_ARG, "null argument");
  if (attach && !d_centre_atom) return set_error(SOAPB_ERR_ARG, "attach needs centre atoms");
  if (max_pairs < 0 || n_pairs < 0) return set_error(SOAPB_ERR_ARG, "bad pair counts");
  if (((uintptr_t)d_out) % 16) return set_error(SOAPB_ERR_ARG, "output must be 16-byte aligned");
  const JacLayout Lw = jac_layout(n_centres, n_pairs, n_inc, attach);
  if (work_bytes < Lw.total) return set_error(SOAPB_ERR_ARG, "jacobian workspace too small (%lld < %lld)",
                                              (long long)work_bytes, (long long)Lw.total);
  // shared-memory sort buffer of the entries kernel: the largest centre's entries, at most 8192
  // keys (64 KB); each centre with more entries takes the tiled merge in the workspace
  const int64_t need = (int64_t)(attach ? 2 : 1) * (max_pairs > 0 ? max_pairs : 1);
  int cap = 64;
  while (cap < need && cap < 8192) cap <<= 1;
  cudaStream_t st = (cudaStream_t)stream;
  char* w = (char*)d_work;
  JacArgs a;
  a.pair_off = d_pair_off;
  a.pairs = (const float4*)d_pairs;
  a.coeff = d_coeff;
  a.inc_row = d_inc_row;
  a.centre_atom = d_centre_atom;
  a.tab_b = (const float*)((const char*)b->dev + b->off_tab_b);
  a.tab_bh = (const float*)((const char*)b->dev + b->off_tab_bh);
  a.selfv = (const float*)((const char*)b->dev + b->off_self);
  a.ftab = (const int*)((const char*)b->dev + b->off_ftab);
  a.out = d_out;
  a.counter = (int*)(w + Lw.counter);
  a.tasks = (int2*)(w + Lw.tasks);
  a.ent = (unsigned long long*)(w + Lw.ent);
  a.ent_tmp = (unsigned long long*)(w + Lw.ent_tmp);
  a.bitmap = (unsigned int*)(w + Lw.bitmap);
  a.n_centres = n_centres;
  a.n_inc = n_inc;
  a.N = b->n_max;
  a.S = b->n_species;
  a.nseg = b->n_seg;
  a.F = out_mode == SOAPB_OUT_PS ? b->n_feat_ps : b->n_feat_cc;
  a.mode = out_mode;
  a.attach = attach ? 1 : 0;
  a.cap = cap;
  a.eb = 1;
  a.ent_mult = attach ? 2 : 1;
  a.inv_h = (float)(1.0 / b->seg_width);
  int rc = check_cuda(cudaMemsetAsync(a.counter, 0, Lw.bitmap - Lw.counter + 4 * ((n_centres * n_inc + 31) / 32), st),
                      "clear work counters and row bitmap");
  if (rc) return rc;
  return dispatch_l<JacDispatch>(b->l_max, a, st);
}
