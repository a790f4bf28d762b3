// Jacobi-PCG on a CSR matrix as one cooperative launch, sm_100a.
//
// The systems of the general-mesh RVE and of small macro meshes have 10^2 to 3 10^4 rows: an
// iteration reads a few MB that stay on the chip, and three launches per iteration with a host
// read every 16 cost about 17 us of which the arithmetic is under one.  Here every SM keeps
// its rows' values and 16-bit column numbers, and its part of r, x and q, in shared memory for
// the whole solve.  The column numbers point into the CTA's own list of the columns that its
// rows touch, for which it also keeps the direction p: each CTA reads the listed z, forms
// p = z + beta p for them in the same way as their owner does, and multiplies out of shared
// memory.  So only z and the dot products cross between SMs.
//
// An iteration has one all-reduce.  Beside p.q it sums z.q and q.(dinv q), from which the next
// r.z follows as r.z - 2 alpha z.q + alpha^2 q.(dinv q) before the update is made (the
// rearrangement of D'Azevedo, Eijkhout and Romine, LAPACK Working Note 56, 1993); it serves
// beta only, alpha and the stopping test take the r.z and r.r that the same all-reduce sums from
// the current r.  A solve therefore stops one matrix product later than it could, with the
// iteration count and residual of the usual arrangement.
//
// What crosses carries its own readiness: each half of a double stands in a 64-bit word beside
// the number of its exchange, and a reader reads until that number is there.  No fence, no
// separate flag: an exchange costs a store and a load through L2.  One CTA per dot product adds
// its partial sums in a fixed order and publishes the sum (a solve repeats bitwise); with every
// CTA reading every partial sum the readers filled the L2's bandwidth (7,000 cycles per
// all-reduce of 148 CTAs, now 4,000).  A word is overwritten only after an all-reduce in which
// every reader of its former value took part after reading it.  The launch is cooperative (all
// CTAs resident), and a wait that lasts longer than two seconds gives the solve back to the caller.
//
// Six right-hand sides (the sensitivities of an effective tangent) go through one solve: the
// matrix is read once for all and the exchanges are shared; each has its own scalars and stops
// by itself.
//
// Bound by the latency of the exchanges.  Per iteration, one right-hand side / six together:
// O-grid of 7,677 rows (621,171 entries) 4.6 / 8.4 us, 957 rows 5.1 / 6.4 us, 117 rows
// 3.7 / 4.7 us; a launch per phase took 18.6, 14.9 and 17.7 us for one.  Starting and ending a
// solve costs about 70 us.
#include <cuda_runtime.h>
#include <math.h>
#include <stdint.h>

#include "cib_common.cuh"
#include "csr_pcg_grid.cuh"

namespace cib {
namespace {

constexpr unsigned FULL = 0xffffffffu;
// Rows per CTA: more rows of 81 entries would not fit, and n <= 28,416 on 148 SMs (28,416 rows of
// 81 entries, 13 iterations: 165 us here, 406 us with a launch per phase).
constexpr int MAX_ROWS = 192;
constexpr int MIN_ROWS = 18;   // an n-vector holds the ten words of a CTA's partial sums
constexpr int MIN_N = 64;      // the ten words do not fit below (64 rows: 126 us here, 63 rows 495 us by phases)
constexpr unsigned long long WAIT_NS = 2000000000ull;

enum { PQ, ZQ, QQ, RZ, RR, DOTS = PCG_GRID_DOTS };  // dot products: p.q, z.q, q.(dinv q), r.z, r.r

template <int NV>
struct Shape {
  static constexpr int PAD = NV == 1 ? 1 : 8;   // right-hand sides, padded for row_sums
  static constexpr int WPV = NV == 1 ? 16 : 3;  // warps that own a right-hand side
  static constexpr int WARPS = NV * WPV;
  static constexpr int THREADS = 32 * WARPS;
};

__device__ __forceinline__ double warp_sum(double v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(FULL, v, o);
  return v;
}

// Sums over eight neighbouring lanes: of s[0] in all of them (N = 1), of s[l] in lane l (N = 8:
// a lane passes on the half that the other one keeps).  The sum is in s[0].
template <int N>
__device__ __forceinline__ void row_sums(double (&s)[N], int lane) {
#pragma unroll
  for (int o = 4; o > 0; o >>= 1) {
    if constexpr (N == 1) {
      s[0] += __shfl_xor_sync(FULL, s[0], o);
    } else {
      const bool high = (lane & o) != 0;
#pragma unroll
      for (int k = 0; k < o; ++k) {
        const double other = __shfl_xor_sync(FULL, high ? s[k] : s[k + o], o);
        s[k] = (high ? s[k + o] : s[k]) + other;
      }
    }
  }
}

__device__ __forceinline__ unsigned long long now_ns() {
  unsigned long long t;
  asm volatile("mov.u64 %0, %globaltimer;" : "=l"(t));
  return t;
}

using Word = unsigned long long;

__device__ __forceinline__ void put(Word* lo, Word* hi, double v, unsigned epoch) {
  const Word bits = __double_as_longlong(v), tag = (Word)epoch << 32;
  asm volatile("st.relaxed.gpu.global.u64 [%0], %1;" ::"l"(lo), "l"(tag | (bits & 0xffffffffull)) : "memory");
  asm volatile("st.relaxed.gpu.global.u64 [%0], %1;" ::"l"(hi), "l"(tag | (bits >> 32)) : "memory");
}

// Waits for K doubles (those of `waiting`) whose words stand at lo[at[k]] and hi[at[k]]: all
// loads of a try are in flight together.  False when the wait ran out.
template <int K>
__device__ __forceinline__ bool get(const Word* lo, const Word* hi, const int64_t (&at)[K], unsigned waiting,
                                    unsigned epoch, double (&v)[K]) {
  unsigned tries = 0;
  unsigned long long since = 0;
  while (waiting) {
    Word l[K], h[K];
#pragma unroll
    for (int k = 0; k < K; ++k) {
      l[k] = h[k] = 0;
      if (waiting >> k & 1) {
        asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];" : "=l"(l[k]) : "l"(lo + at[k]));
        asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];" : "=l"(h[k]) : "l"(hi + at[k]));
      }
    }
#pragma unroll
    for (int k = 0; k < K; ++k)
      if ((waiting >> k & 1) && (unsigned)(l[k] >> 32) == epoch && (unsigned)(h[k] >> 32) == epoch) {
        v[k] = __longlong_as_double((long long)((h[k] << 32) | (l[k] & 0xffffffffull)));
        waiting &= ~(1u << k);
      }
    if (waiting && (++tries & 1023) == 0) {
      const unsigned long long now = now_ns();
      if (since == 0) since = now;
      if (now - since > WAIT_NS) return false;
    }
  }
  return true;
}

// sums[v] = sum over the grid of the partial sums red[v][.]; called between barriers.  `part`
// holds [DOTS NV][grid] and then [DOTS NV] (the sums) pairs of words.  False when a wait ran out.
template <int NV>
__device__ __forceinline__ bool all_reduce(Word* part, const double* red, double* sums, unsigned epoch) {
  using S = Shape<NV>;
  constexpr int N = DOTS * NV, K = PCG_GRID_MAX / 32;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, grid = gridDim.x;
  Word* total = part + 2 * (int64_t)N * grid;
  bool ok = true;
#pragma unroll 1
  for (int v = warp; v < N && warp < S::WARPS - 1; v += S::WARPS - 1) {  // the last warp waits for the sums
    const double mine = warp_sum(lane < S::WARPS ? red[v * S::WARPS + lane] : 0.0);
    Word* of = part + 2 * (int64_t)v * grid;
    if (lane == 0) put(of + 2 * blockIdx.x, of + 2 * blockIdx.x + 1, mine, epoch);
  }
#pragma unroll 1
  for (int v = warp; v < N && warp < S::WARPS - 1; v += S::WARPS - 1)
    if (v % grid == blockIdx.x) {
      Word* of = part + 2 * (int64_t)v * grid;
      int64_t at[K];
      double got[K];
      unsigned waiting = 0;
#pragma unroll
      for (int k = 0; k < K; ++k) {
        got[k] = 0.0;
        at[k] = 2 * (lane + 32 * k);
        if (lane + 32 * k < grid) waiting |= 1u << k;
      }
      ok &= get<K>(of, of + 1, at, waiting, epoch, got);
      __syncwarp();
      static_assert(K == 5, "the sum below");
      const double s = warp_sum(((got[0] + got[1]) + (got[2] + got[3])) + got[4]);
      if (lane == 0) put(total + 2 * v, total + 2 * v + 1, s, epoch);
    }
  if (warp == S::WARPS - 1) {
    static_assert(N <= 32, "a lane per sum");
    const int64_t at[1] = {2 * lane};
    double got[1] = {0.0};
    ok &= get<1>(total, total + 1, at, lane < N, epoch, got);
    if (lane < N) sums[lane] = got[0];
  }
  return ok;
}

struct GridArgs {
  CsrSystem a;
  int rows_per, smem;
  const double* b;
  double* x;
  Word *zlo, *zhi;  // halves of z [NV][n]
  Word* part;       // see all_reduce
  double* out;      // [NV][3] status (1 converged, 0 limit, 2 breakdown), iterations, rel; then: not solved
  double rtol;
  int maxit;
};

template <int NV>
__global__ void __launch_bounds__(Shape<NV>::THREADS, 1) csr_pcg_grid_kernel(const GridArgs g) {
  using S = Shape<NV>;
  extern __shared__ __align__(16) double sm[];
  const int t = threadIdx.x, warp = t >> 5, lane = t & 31;
  const CsrSystem& a = g.a;
  const int64_t n = a.n, r0 = (int64_t)blockIdx.x * g.rows_per;
  const int nr = (int)min((int64_t)g.rows_per, n - r0), words = (int)((n + 31) / 32);
  const int64_t e0 = a.indptr[r0];
  const int64_t entries = a.indptr[r0 + nr] - e0;
  double* red = sm;                                // [DOTS NV][WARPS] sums of the warps
  double* sums = red + DOTS * NV * S::WARPS;       // [DOTS NV] of the grid
  double* r = sums + DOTS * NV;                    // [NV][rows_per]
  double* x = r + NV * g.rows_per;
  double* q = x + NV * g.rows_per;
  double* dinv = q + NV * g.rows_per;              // [rows_per]
  int* row = reinterpret_cast<int*>(dinv + g.rows_per);  // [rows_per + 1] first entry of a row
  unsigned* bits = reinterpret_cast<unsigned*>(row + g.rows_per + 1);  // [words] columns in use
  unsigned* rank = bits + words;                   // [words] of them before a word
  unsigned* fixed = rank + words;                  // [MAX_ROWS / 32] fixed rows
  int* group = reinterpret_cast<int*>(fixed + MAX_ROWS / 32);  // [MAX_ROWS / 4 + 1] first step of four rows
  int* misc = group + MAX_ROWS / 4 + 1;            // columns in use, lost
  volatile int* lost = misc + 1;
  const int fixed_bytes = (int)(reinterpret_cast<char*>(misc + 2) - reinterpret_cast<char*>(sm) + 7) & ~7;

  // 1. the columns that these rows touch, in ascending order
#pragma unroll 1
  for (int i = t; i < words; i += S::THREADS) bits[i] = 0;
  if (t < MAX_ROWS / 32) fixed[t] = 0;
  if (t == 0) *lost = 0;
  __syncthreads();
#pragma unroll 1
  for (int64_t e = t; e < entries; e += S::THREADS) {
    const int64_t c = a.indices[e0 + e];
    atomicOr(&bits[c >> 5], 1u << (c & 31));
  }
#pragma unroll 1
  for (int i = t; i < nr; i += S::THREADS) {
    const int64_t c = r0 + i;
    atomicOr(&bits[c >> 5], 1u << (c & 31));
    dinv[i] = a.dinv[c];
    if (!a.free_mask[c]) atomicOr(&fixed[i >> 5], 1u << (i & 31));
  }
#pragma unroll 1
  for (int i = t; i <= nr; i += S::THREADS) row[i] = (int)(a.indptr[r0 + i] - e0);
  __syncthreads();
  if (warp == 0) {
    int before = 0;
#pragma unroll 1
    for (int base = 0; base < words; base += 32) {
      const int own = base + lane < words ? __popc(bits[base + lane]) : 0;
      int upto = own;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const int other = __shfl_up_sync(FULL, upto, o);
        if (lane >= o) upto += other;
      }
      if (base + lane < words) rank[base + lane] = before + upto - own;
      before += __shfl_sync(FULL, upto, 31);
    }
    if (lane == 0) misc[0] = before;
  } else if (warp == 1) {
    int before = 0;
#pragma unroll 1
    for (int base = 0; 4 * base < nr; base += 32) {
      int steps = 0;
      for (int i = 4 * (base + lane); i < min(4 * (base + lane) + 4, nr); ++i) steps = max(steps, (row[i + 1] - row[i] + 7) / 8);
      int upto = steps;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const int other = __shfl_up_sync(FULL, upto, o);
        if (lane >= o) upto += other;
      }
      if (4 * (base + lane) < nr) group[base + lane] = before + upto - steps;
      before += __shfl_sync(FULL, upto, 31);
    }
    if (lane == 0) group[(nr + 3) / 4] = before;
  }
  __syncthreads();
  const int used = misc[0];
  // Entries of four rows step by step, eight of a row at a time: a warp's 32 stand together.
  const int64_t slots = 32 * (int64_t)group[(nr + 3) / 4];
  const bool fits = used <= 65535 && entries < (1 << 24) && fixed_bytes + (int64_t)used * (8 * NV + 4) + slots * 10 <= g.smem;
  double* p = reinterpret_cast<double*>(reinterpret_cast<char*>(sm) + fixed_bytes);  // [NV][used]
  double* val = p + (int64_t)NV * used;                                              // [slots]
  int* col = reinterpret_cast<int*>(val + slots);                                  // [used]
  uint16_t* idx = reinterpret_cast<uint16_t*>(col + used);                           // [slots]
  const int own = (int)(rank[r0 >> 5] + __popc(bits[r0 >> 5] & ((1u << (r0 & 31)) - 1u)));  // of row r0; the rest follow
  if (fits) {
#pragma unroll 1
    for (int i = t; i < words; i += S::THREADS) {
      int k = (int)rank[i];
      for (unsigned b = bits[i]; b; b &= b - 1) col[k++] = 32 * i + __ffs(b) - 1;
    }
#pragma unroll 1
    for (int i = warp; 4 * i < nr; i += S::WARPS) {
      const int k = 4 * i + (lane >> 3), end = k < nr ? row[k + 1] : 0;
      int e = (k < nr ? row[k] : 0) + (lane & 7);
#pragma unroll 4
      for (int at = 32 * group[i] + lane; at < 32 * group[i + 1]; at += 32, e += 8) {
        const int64_t c = e < end ? a.indices[e0 + e] : r0;
        idx[at] = (uint16_t)(rank[c >> 5] + __popc(bits[c >> 5] & ((1u << (c & 31)) - 1u)));
        val[at] = e < end ? a.values[e0 + e] : 0.0;
      }
    }
#pragma unroll 1
    for (int i = t; i < NV * used; i += S::THREADS) p[i] = 0.0;
  }

  // 2. x = 0, r = b on free rows, z = dinv r.  A warp owns one right-hand side's vectors.
  const int v = warp / S::WPV, mine = 32 * (warp % S::WPV) + lane;
  constexpr int STEP = 32 * S::WPV;
  Word *zlo = g.zlo + v * n, *zhi = g.zhi + v * n;
#pragma unroll 1
  for (int i = mine; i < nr; i += STEP) {
    const double ri = fixed[i >> 5] >> (i & 31) & 1 ? 0.0 : g.b[v * n + r0 + i];
    x[v * g.rows_per + i] = 0.0;
    r[v * g.rows_per + i] = ri;
    put(zlo + r0 + i, zhi + r0 + i, dinv[i] * ri, 1);
  }
  __syncthreads();

  // State of this thread's right-hand side: the same in all its warps and all CTAs.
  int status = 0, iters = 0;  // 0 running, 1 converged, 2 breakdown, 3 limit
  double beta = 0.0, rr0 = 0.0, rr = 0.0, near_stop = 0.0;
  for (int it = 0;; ++it) {
    // p = z + beta p on the listed columns
    if (status == 0 && fits) {
      constexpr int K = 2;
#pragma unroll 1
      for (int base = mine; base < used; base += K * STEP) {
        int64_t at[K];
        double z[K];
        unsigned waiting = 0;
#pragma unroll
        for (int k = 0; k < K; ++k) {
          at[k] = 0;
          if (base + k * STEP < used) {
            waiting |= 1u << k;
            at[k] = col[base + k * STEP];
          }
        }
        if (!get<K>(zlo, zhi, at, waiting, it + 1, z)) *lost = 1;
#pragma unroll
        for (int k = 0; k < K; ++k)
          if (base + k * STEP < used) {
            double* pk = p + v * used + base + k * STEP;
            *pk = fma(beta, *pk, z[k]);
          }
      }
    }
    if (!__syncthreads_or(status == 0) || *lost) break;
    // q = A p on free rows, and the dot products.  Eight lanes to a row, four rows to a warp.
    // (A CTA whose rows do not fit stops them all here: its dot products are not finite.)
    // Lane l of a row's eight holds right-hand side l of the row after the sums.
    constexpr int CHAINS = NV == 1 ? 4 : 2;
    double dots[DOTS] = {0.0, 0.0, 0.0, 0.0, 0.0};
#pragma unroll 1
    for (int base = 4 * warp; base < nr; base += 4 * S::WARPS) {
      const int i = base + (lane >> 3), j = lane & 7;
      double s[S::PAD], part[CHAINS][NV];  // several chains: the latency of an FP64 add is the longer time
#pragma unroll
      for (int c = 0; c < CHAINS; ++c)
#pragma unroll
        for (int k = 0; k < NV; ++k) part[c][k] = 0.0;
      if (fits) {
        const int last = 32 * group[base / 4 + 1] - 32 + lane;
#pragma unroll 1
        for (int at = 32 * group[base / 4] + lane; at <= last; at += 32 * 4) {  // loads of four steps together
          double w[4];
          int c[4];
#pragma unroll
          for (int u = 0; u < 4; ++u) {
            const int k = min(at + 32 * u, last);
            w[u] = val[k];
            c[u] = idx[k];
          }
#pragma unroll
          for (int u = 0; u < 4; ++u) {
            if (at + 32 * u > last) w[u] = 0.0;
#pragma unroll
            for (int k = 0; k < NV; ++k) part[u % CHAINS][k] = fma(w[u], p[k * used + c[u]], part[u % CHAINS][k]);
          }
        }
      }
#pragma unroll
      for (int k = 0; k < S::PAD; ++k) {
        s[k] = 0.0;
        if (k < NV) s[k] = part[0][k] + part[1][k];
        if (k < NV && CHAINS == 4) s[k] += part[CHAINS - 2][k] + part[CHAINS - 1][k];
      }
      row_sums<S::PAD>(s, lane);
      if (i < nr && j < NV) {
        const int k = j * g.rows_per + i;
        const double qv = fixed[i >> 5] >> (i & 31) & 1 ? 0.0 : s[0], rv = r[k], zv = dinv[i] * rv;
        q[k] = qv;
        dots[PQ] = fma(fits ? p[j * used + own + i] : 0.0, qv, dots[PQ]);
        dots[ZQ] = fma(zv, qv, dots[ZQ]);
        dots[QQ] = fma(dinv[i] * qv, qv, dots[QQ]);
        dots[RZ] = fma(rv, zv, dots[RZ]);
        dots[RR] = fma(rv, rv, dots[RR]);
      }
    }
#pragma unroll
    for (int d = 0; d < DOTS; ++d) {  // over the four rows
      double s = dots[d];
      s += __shfl_xor_sync(FULL, s, 8);
      s += __shfl_xor_sync(FULL, s, 16);
      if (lane < NV) red[(d * NV + lane) * S::WARPS + warp] = fits ? s : __longlong_as_double(0x7ff8000000000000ll);
    }
    __syncthreads();
    if (!all_reduce<NV>(g.part, red, sums, it + 1)) *lost = 1;
    __syncthreads();
    if (*lost) break;
    if (status == 0) {
      const double pq = sums[PQ * NV + v], rz = sums[RZ * NV + v];
      rr = sums[RR * NV + v];
      if (it == 0) {
        rr0 = rr;
        near_stop = 1.0001 * g.rtol * g.rtol * rr0;  // the quotient decides only below this
      }
      iters = it;
      if (!(isfinite(rz) && isfinite(rr)))
        status = 2;
      else if (rr == 0.0 && it == 0)
        status = 1;
      else if (it > 0 && rr <= near_stop && sqrt(rr) / sqrt(rr0) <= g.rtol)
        status = 1;
      else if (it >= g.maxit)
        status = 3;
      else if (!(pq > 0.0) || !isfinite(pq))
        status = 2;
      if (status == 0) {
        const double inverse = 1.0 / pq;
        const bool tiny = !isfinite(inverse);  // a right-hand side near the end of the range
        const double alpha = tiny ? rz / pq : rz * inverse;
#pragma unroll 1
        for (int i = mine; i < nr; i += STEP) {
          const int k = v * g.rows_per + i;
          const double ri = fma(-alpha, q[k], r[k]);
          put(zlo + r0 + i, zhi + r0 + i, dinv[i] * ri, it + 2);
          r[k] = ri;
          x[k] = fma(alpha, p[v * used + own + i], x[k]);
        }
        // the next r.z over this one; rounding can leave nothing of it
        const double change = fma(alpha, sums[QQ * NV + v], -2.0 * sums[ZQ * NV + v]);
        beta = fmax(tiny ? 1.0 + change / pq : fma(change, inverse, 1.0), 0.0);
      }
    }
    __syncthreads();  // p of the own rows has been read
  }
  if (*lost || !fits) {
    if (t == 0) g.out[3 * NV] = 1.0;
    return;
  }
#pragma unroll 1
  for (int i = mine; i < nr; i += STEP) g.x[v * n + r0 + i] = x[v * g.rows_per + i];
  if (blockIdx.x == 0 && mine == 0) {
    g.out[3 * v] = status == 3 ? 0.0 : (double)status;
    g.out[3 * v + 1] = (double)iters;
    g.out[3 * v + 2] = rr0 > 0.0 ? sqrt(rr) / sqrt(rr0) : 0.0;
  }
}

template <int NV>
int solve(const CsrSystem& a, const double* b, double* x, const PcgGridWork& w, double rtol, int32_t maxit,
          int32_t* status, int32_t* iterations, double* relative_residual, cudaStream_t st) {
  const int sms = sm_count() < PCG_GRID_MAX ? sm_count() : PCG_GRID_MAX;
  int64_t rows = (a.n + sms - 1) / sms;
  if (rows > MAX_ROWS || a.n < MIN_N) return CIB_ERANGE;
  if (rows < MIN_ROWS) rows = MIN_ROWS;
  const int64_t grid = (a.n + rows - 1) / rows;
  constexpr int SMEM = 224 * 1024;
  const void* kernel = reinterpret_cast<const void*>(csr_pcg_grid_kernel<NV>);
  const int rc = allow_dynamic_smem(kernel, SMEM);
  if (rc != CIB_OK) return rc;
  const size_t part = sizeof(double) * 2 * DOTS * NV * (size_t)(grid + 1), z = sizeof(double) * NV * (size_t)a.n;
  GridArgs g{a, (int)rows, SMEM, b, x, reinterpret_cast<Word*>(w.zlo), reinterpret_cast<Word*>(w.zhi),
             reinterpret_cast<Word*>(w.part), w.out, rtol, maxit};
  double host[3 * NV + 1];
  void* args[] = {&g};
  cudaError_t e = cudaMemsetAsync(w.zlo, 0, z, st);
  if (e == cudaSuccess) e = cudaMemsetAsync(w.zhi, 0, z, st);
  if (e == cudaSuccess) e = cudaMemsetAsync(w.part, 0, part, st);
  if (e == cudaSuccess) e = cudaMemsetAsync(w.out, 0, sizeof(host), st);
  if (e == cudaSuccess) {
    e = cudaLaunchCooperativeKernel(kernel, dim3((unsigned)grid), dim3(Shape<NV>::THREADS), args, SMEM, st);
    if (e == cudaErrorCooperativeLaunchTooLarge) {  // a partition of the device: a launch per phase
      cudaGetLastError();
      return CIB_ERANGE;
    }
  }
  if (e == cudaSuccess) e = cudaMemcpyAsync(host, w.out, sizeof(host), cudaMemcpyDeviceToHost, st);
  if (e == cudaSuccess) e = cudaStreamSynchronize(st);
  if (e != cudaSuccess) {
    cudaGetLastError();
    last_cuda_error_slot() = (int)e;
    return CIB_ECUDA;
  }
  if (host[3 * NV] != 0.0) return CIB_ERANGE;  // a CTA's rows do not fit, or a wait ran out
  for (int j = 0; j < NV; ++j) {
    status[j] = host[3 * j] == 1.0 ? 0 : (host[3 * j] == 2.0 ? 2 : 1);
    iterations[j] = (int32_t)host[3 * j + 1];
    relative_residual[j] = host[3 * j + 2];
  }
  return CIB_OK;
}

}  // namespace

int csr_pcg_grid(const CsrSystem& a, int rhs, const double* b, double* x, const PcgGridWork& w, double rtol,
                 int32_t maxit, int32_t* status, int32_t* iterations, double* relative_residual, cudaStream_t st) {
  if (rhs == 1) return solve<1>(a, b, x, w, rtol, maxit, status, iterations, relative_residual, st);
  if (rhs == PCG_BLOCK_RHS)
    return solve<PCG_BLOCK_RHS>(a, b, x, w, rtol, maxit, status, iterations, relative_residual, st);
  return CIB_ERANGE;
}

}  // namespace cib
