// Energy-based RVE-RNO update on the GPU (FP32), sm_100a.
//
// Restates the reference's EnergyDissipationRVERNO._constitutive_tensors
// (src/concrete_impact/nn/models/rve_rno.py:334-418; direct_rate evolution, both
// integrators), ScalarMLP.value_and_input_gradient (:110-129), the SiLU MultilayerPerceptron
// (:63-93) and prepare_energy_anchors (:227-247).  Per point and step: the equilibrium
// potential and its strain gradient, the non-equilibrium potential and its gradient at the
// previous state, the state-evolution network there, the forward-Euler latent candidate,
// and the non-equilibrium potential and gradient at the candidate -- four network passes and
// three hand-written input-gradient passes of 6/12 -> hidden^layers -> 1 (or 6) networks.
//
// One CTA of 128 threads per tile of 32 points.  Forward layers: thread j owns hidden unit j
// and keeps the 32 points' accumulators in registers; the layer's input sits in shared
// memory feature-major (the 32 points of a feature read as eight float4 broadcasts) and the
// transposed weights are read along j (coalesced).  Input-gradient layers: thread k owns
// input k and reads the weights along k (coalesced).  Pre-activations of every layer stay in
// shared memory for the backward pass.
// Everything is FP32 like the reference model (its dtype float32); no waits besides
// __syncthreads.
#include <cuda_runtime.h>
#include <math.h>
#include <stdint.h>

#include "cib_common.cuh"
#include "f32x2.cuh"

namespace cib {
namespace {

constexpr int ER_TILE = 32;
constexpr int ER_THREADS = 128;
constexpr int ER_XLD = 16;  // input rows: 6 + latent <= 14, padded

// Parameter layout of one network (floats), for each hidden layer l: W [hidden][in_l],
// Wt [in_l][hidden], b [hidden]; then Wo [out][hidden], bo [out].
__host__ __device__ inline int64_t net_size(int in, int out, int hidden, int layers) {
  int64_t s = 0;
  for (int l = 0; l < layers; ++l) {
    const int in_l = l == 0 ? in : hidden;
    s += 2LL * hidden * in_l + hidden;
  }
  return s + (int64_t)out * hidden + out;
}

struct NetView {
  const float* base;
  int in, out;
};

__device__ __forceinline__ void layer_ptrs(const NetView& n, int hidden, int l, const float** W, const float** Wt,
                                           const float** b) {
  const float* p = n.base;
  for (int i = 0; i < l; ++i) {
    const int in_i = i == 0 ? n.in : hidden;
    p += 2LL * hidden * in_i + hidden;
  }
  const int in_l = l == 0 ? n.in : hidden;
  *W = p;
  *Wt = p + (int64_t)hidden * in_l;
  *b = p + 2LL * hidden * in_l;
}

__device__ __forceinline__ const float* output_ptr(const NetView& n, int hidden, int layers) {
  const float* p = n.base;
  for (int i = 0; i < layers; ++i) {
    const int in_i = i == 0 ? n.in : hidden;
    p += 2LL * hidden * in_i + hidden;
  }
  return p;  // Wo [out][hidden], then bo [out]
}

__device__ __forceinline__ float silu(float z) { return z / (1.0f + expf(-z)); }

__device__ __forceinline__ float silu_prime(float z) {
  const float s = 1.0f / (1.0f + expf(-z));
  return s * (1.0f + z * (1.0f - s));
}

// Shared buffers are feature-major, one row of ER_TILE floats per feature (input, hidden
// unit), so a layer reads the 32 points of one feature as eight float4 broadcasts.  The
// float4 groups of row r are XOR-swizzled by r & 7: a thread writing its own row and a
// thread reading one point across rows both hit 32 distinct banks.
__device__ __forceinline__ int sw(int row, int p) { return row * ER_TILE + ((((p >> 2) ^ (row & 7)) << 2) | (p & 3)); }

__device__ __forceinline__ float4* grp(float* buf, int row, int g) {
  return reinterpret_cast<float4*>(buf + row * ER_TILE + ((g ^ (row & 7)) << 2));
}

__device__ __forceinline__ const float4* grp(const float* buf, int row, int g) {
  return reinterpret_cast<const float4*>(buf + row * ER_TILE + ((g ^ (row & 7)) << 2));
}

struct Smem {
  float* x;    // [XLD rows][TILE] network input
  float* gin;  // [XLD rows][TILE] input gradient
  float* h0;   // [hidden rows][TILE]
  float* h1;   // [hidden rows][TILE]
  float* z;    // [layers][hidden rows][TILE] pre-activations
};

// Forward pass of the hidden layers; returns the buffer holding the last activation.
__device__ float* forward_hidden(const NetView& n, int hidden, int layers, const Smem& s) {
  const int j = threadIdx.x;
  const float* hin = s.x;
  float* hout = s.h0;
  for (int l = 0; l < layers; ++l) {
    const float *W, *Wt, *b;
    layer_ptrs(n, hidden, l, &W, &Wt, &b);
    const int in_l = l == 0 ? n.in : hidden;
    float* zl = s.z + (int64_t)l * hidden * ER_TILE;
    if (j < hidden) {
      float acc[ER_TILE];
      const float bj = b[j];
#pragma unroll
      for (int p = 0; p < ER_TILE; ++p) acc[p] = bj;
      int k = 0;
      for (; k + 4 <= in_l; k += 4) {  // four weights in flight per thread
        const float w0 = Wt[(int64_t)k * hidden + j], w1 = Wt[(int64_t)(k + 1) * hidden + j];
        const float w2 = Wt[(int64_t)(k + 2) * hidden + j], w3 = Wt[(int64_t)(k + 3) * hidden + j];
#pragma unroll
        for (int g = 0; g < ER_TILE / 4; ++g) {
          const float4 v0 = *grp(hin, k, g), v1 = *grp(hin, k + 1, g), v2 = *grp(hin, k + 2, g),
                       v3 = *grp(hin, k + 3, g);
          acc[4 * g] = fmaf(w3, v3.x, fmaf(w2, v2.x, fmaf(w1, v1.x, fmaf(w0, v0.x, acc[4 * g]))));
          acc[4 * g + 1] = fmaf(w3, v3.y, fmaf(w2, v2.y, fmaf(w1, v1.y, fmaf(w0, v0.y, acc[4 * g + 1]))));
          acc[4 * g + 2] = fmaf(w3, v3.z, fmaf(w2, v2.z, fmaf(w1, v1.z, fmaf(w0, v0.z, acc[4 * g + 2]))));
          acc[4 * g + 3] = fmaf(w3, v3.w, fmaf(w2, v2.w, fmaf(w1, v1.w, fmaf(w0, v0.w, acc[4 * g + 3]))));
        }
      }
      for (; k < in_l; ++k) {
        const float w = Wt[(int64_t)k * hidden + j];
#pragma unroll
        for (int g = 0; g < ER_TILE / 4; ++g) {
          const float4 v = *grp(hin, k, g);
          acc[4 * g] = fmaf(w, v.x, acc[4 * g]);
          acc[4 * g + 1] = fmaf(w, v.y, acc[4 * g + 1]);
          acc[4 * g + 2] = fmaf(w, v.z, acc[4 * g + 2]);
          acc[4 * g + 3] = fmaf(w, v.w, acc[4 * g + 3]);
        }
      }
#pragma unroll
      for (int g = 0; g < ER_TILE / 4; ++g) {
        *grp(zl, j, g) = make_float4(acc[4 * g], acc[4 * g + 1], acc[4 * g + 2], acc[4 * g + 3]);
        *grp(hout, j, g) = make_float4(silu(acc[4 * g]), silu(acc[4 * g + 1]), silu(acc[4 * g + 2]),
                                       silu(acc[4 * g + 3]));
      }
    }
    __syncthreads();
    hin = hout;
    hout = (hout == s.h0) ? s.h1 : s.h0;
  }
  return const_cast<float*>(hin);
}

// Scalar potential value per point (threads p < TILE) into value[p].
__device__ void scalar_output(const NetView& n, int hidden, int layers, const float* h, float* value) {
  const float* wo = output_ptr(n, hidden, layers);
  const int p = threadIdx.x;
  if (p < ER_TILE) {
    float v = 0.0f;
    for (int j = 0; j < hidden; ++j) v = fmaf(wo[j], h[sw(j, p)], v);
    value[p] = v;
  }
  __syncthreads();
}

// Input gradient of a scalar network into rows 0..in of s.gin (pre-activations in s.z).
__device__ void input_gradient(const NetView& n, int hidden, int layers, const Smem& s) {
  const float* wo = output_ptr(n, hidden, layers);
  const int t = threadIdx.x;
  float* g = s.h0;  // gradient wrt the activation of layer l
  float* d = s.h1;  // gradient wrt the pre-activation of layer l
  for (int l = layers - 1; l >= 0; --l) {
    const float* zl = s.z + (int64_t)l * hidden * ER_TILE;
    if (t < hidden) {
      const float wt = wo[t];
#pragma unroll
      for (int q = 0; q < ER_TILE / 4; ++q) {
        const float4 zz = *grp(zl, t, q);
        const float4 gv = (l == layers - 1) ? make_float4(wt, wt, wt, wt) : *grp(g, t, q);
        *grp(d, t, q) = make_float4(gv.x * silu_prime(zz.x), gv.y * silu_prime(zz.y), gv.z * silu_prime(zz.z),
                                    gv.w * silu_prime(zz.w));
      }
    }
    __syncthreads();
    const float *W, *Wt, *b;
    layer_ptrs(n, hidden, l, &W, &Wt, &b);
    const int in_l = l == 0 ? n.in : hidden;
    float* dst = l == 0 ? s.gin : g;
    if (t < in_l) {
      float acc[ER_TILE];
#pragma unroll
      for (int p = 0; p < ER_TILE; ++p) acc[p] = 0.0f;
      int jj = 0;
      for (; jj + 4 <= hidden; jj += 4) {
        const float w0 = W[(int64_t)jj * in_l + t], w1 = W[(int64_t)(jj + 1) * in_l + t];
        const float w2 = W[(int64_t)(jj + 2) * in_l + t], w3 = W[(int64_t)(jj + 3) * in_l + t];
#pragma unroll
        for (int q = 0; q < ER_TILE / 4; ++q) {
          const float4 v0 = *grp(d, jj, q), v1 = *grp(d, jj + 1, q), v2 = *grp(d, jj + 2, q), v3 = *grp(d, jj + 3, q);
          acc[4 * q] = fmaf(v3.x, w3, fmaf(v2.x, w2, fmaf(v1.x, w1, fmaf(v0.x, w0, acc[4 * q]))));
          acc[4 * q + 1] = fmaf(v3.y, w3, fmaf(v2.y, w2, fmaf(v1.y, w1, fmaf(v0.y, w0, acc[4 * q + 1]))));
          acc[4 * q + 2] = fmaf(v3.z, w3, fmaf(v2.z, w2, fmaf(v1.z, w1, fmaf(v0.z, w0, acc[4 * q + 2]))));
          acc[4 * q + 3] = fmaf(v3.w, w3, fmaf(v2.w, w2, fmaf(v1.w, w1, fmaf(v0.w, w0, acc[4 * q + 3]))));
        }
      }
      for (; jj < hidden; ++jj) {
        const float w = W[(int64_t)jj * in_l + t];
#pragma unroll
        for (int q = 0; q < ER_TILE / 4; ++q) {
          const float4 v = *grp(d, jj, q);
          acc[4 * q] = fmaf(v.x, w, acc[4 * q]);
          acc[4 * q + 1] = fmaf(v.y, w, acc[4 * q + 1]);
          acc[4 * q + 2] = fmaf(v.z, w, acc[4 * q + 2]);
          acc[4 * q + 3] = fmaf(v.w, w, acc[4 * q + 3]);
        }
      }
#pragma unroll
      for (int q = 0; q < ER_TILE / 4; ++q)
        *grp(dst, t, q) = make_float4(acc[4 * q], acc[4 * q + 1], acc[4 * q + 2], acc[4 * q + 3]);
    }
    __syncthreads();
  }
}

struct EnergyArgs {
  int hidden, layers, latent, integrator;
  float tau;
  const float* params;
  const float* scale;  // 6
  int64_t n;
  const float* strain;      // n x 6
  const float* latent_in;   // n x L
  const float* time_step;   // n
  const float* anchors;     // 14: eq value, eq grad (6), neq value, neq strain grad (6); NULL = zeros
  float* stress;            // n x 6
  float* latent_out;        // n x L
  float* rate;              // n x L
  float* rate_dimless;      // n x L
  float* scalars;           // 4 x n: dissipation, free energy, violation, energy increment
  float* anchors_out;       // anchor mode: 14 outputs (point 0 of a zero input)
  float* tangent;           // tangent kernel: n x 6 x 6
};

// Anchors, or the anchored energies, stress, rates and dissipation of a tile of P points
// (thread p owns point p).
__device__ void finish_update(const EnergyArgs& a, int64_t p0, int P, const float* eps, const float* zdl,
                              const float* zc, const float* geq, const float* gpr, const float* gca,
                              const float* val) {
  const int L = a.latent, t = threadIdx.x;
  if (a.anchors_out) {
    if (t == 0) {
      a.anchors_out[0] = val[0];
      for (int c = 0; c < 6; ++c) a.anchors_out[1 + c] = geq[c];
      a.anchors_out[7] = val[P];
      for (int c = 0; c < 6; ++c) a.anchors_out[8 + c] = gpr[c];
    }
    return;
  }
  if (t < P && p0 + t < a.n) {
    const int p = t;
    const int64_t q = p0 + p;
    float av_eq = 0.0f, av_neq = 0.0f, ag_eq[6], ag_neq[6];
    for (int c = 0; c < 6; ++c) {
      ag_eq[c] = a.anchors ? a.anchors[1 + c] : 0.0f;
      ag_neq[c] = a.anchors ? a.anchors[8 + c] : 0.0f;
    }
    if (a.anchors) {
      av_eq = a.anchors[0];
      av_neq = a.anchors[7];
    }
    float xe = 0.0f, xn = 0.0f;
    for (int c = 0; c < 6; ++c) {
      xe += eps[p * 6 + c] * ag_eq[c];
      xn += eps[p * 6 + c] * ag_neq[c];
    }
    const float equilibrium = val[p] - av_eq - xe;
    const float prev_neq = val[P + p] - av_neq - xn;
    const float cand_neq = val[2 * P + p] - av_neq - xn;
    float diss = 0.0f;
    for (int o = 0; o < L; ++o) {
      const float r = zdl[p * 8 + o] / a.tau;
      a.rate[q * L + o] = r;
      a.rate_dimless[q * L + o] = zdl[p * 8 + o];
      a.latent_out[q * L + o] = zc[p * 8 + o];
      diss += gpr[p * 16 + 6 + o] * r;
    }
    diss = -diss;
    const float* gresp = a.integrator == 1 ? gca + p * 16 : gpr + p * 16;
    for (int c = 0; c < 6; ++c)
      a.stress[q * 6 + c] = (geq[p * 6 + c] - ag_eq[c]) / a.scale[c] + (gresp[c] - ag_neq[c]) / a.scale[c];
    a.scalars[q] = diss;
    a.scalars[a.n + q] = equilibrium + (a.integrator == 1 ? cand_neq : prev_neq);
    a.scalars[2 * a.n + q] = fmaxf(-diss, 0.0f);
    a.scalars[3 * a.n + q] = cand_neq - prev_neq;
  }
}

__global__ void __launch_bounds__(ER_THREADS) energy_rno_kernel(const EnergyArgs a) {
  extern __shared__ float sm[];
  const int hidden = a.hidden, layers = a.layers, L = a.latent;
  Smem s;
  s.x = sm;
  s.gin = s.x + ER_TILE * ER_XLD;
  s.h0 = s.gin + ER_TILE * ER_XLD;
  s.h1 = s.h0 + ER_TILE * hidden;
  s.z = s.h1 + ER_TILE * hidden;
  float* eps = s.z + (int64_t)layers * ER_TILE * hidden;  // [TILE][6] network strain
  float* zin = eps + ER_TILE * 6;                      // [TILE][8] previous latent
  float* zdl = zin + ER_TILE * 8;                      // [TILE][8] dimensionless rate
  float* zc = zdl + ER_TILE * 8;                       // [TILE][8] candidate latent
  float* geq = zc + ER_TILE * 8;                       // [TILE][6]
  float* gpr = geq + ER_TILE * 6;                      // [TILE][16]
  float* gca = gpr + ER_TILE * 16;                     // [TILE][16]
  float* val = gca + ER_TILE * 16;                     // [3][TILE]: eq, previous, candidate values
  const int t = threadIdx.x;
  const int64_t p0 = (int64_t)blockIdx.x * ER_TILE;
  const bool anchor_mode = a.anchors_out != nullptr;
  const NetView eq{a.params, 6, 1};
  const NetView neq{a.params + net_size(6, 1, hidden, layers), 6 + L, 1};
  const NetView evo{neq.base + net_size(6 + L, 1, hidden, layers), 6 + L, L};
  // per-point inputs (zeros beyond n and in anchor mode)
  for (int i = t; i < ER_TILE * 8; i += ER_THREADS) {
    const int p = i >> 3, c = i & 7;
    const bool live = !anchor_mode && p0 + p < a.n;
    if (c < 6) eps[p * 6 + c] = live ? a.strain[(p0 + p) * 6 + c] / a.scale[c] : 0.0f;
    zin[i] = (live && c < L) ? a.latent_in[(p0 + p) * L + c] : 0.0f;
  }
  __syncthreads();
  // 1. equilibrium potential and gradient at the network strain
  for (int i = t; i < ER_TILE * ER_XLD; i += ER_THREADS) {
    const int p = i / ER_XLD, c = i % ER_XLD;
    s.x[sw(c, p)] = c < 6 ? eps[p * 6 + c] : 0.0f;
  }
  __syncthreads();
  scalar_output(eq, hidden, layers, forward_hidden(eq, hidden, layers, s), val);
  input_gradient(eq, hidden, layers, s);
  for (int i = t; i < ER_TILE * 6; i += ER_THREADS) geq[i] = s.gin[sw(i % 6, i / 6)];
  // 2. previous state [eps, z_n]: non-equilibrium potential and gradient, then the evolution net
  for (int i = t; i < ER_TILE * ER_XLD; i += ER_THREADS) {
    const int p = i / ER_XLD, c = i % ER_XLD;
    s.x[sw(c, p)] = c < 6 ? eps[p * 6 + c] : (c < 6 + L ? zin[p * 8 + c - 6] : 0.0f);
  }
  __syncthreads();
  scalar_output(neq, hidden, layers, forward_hidden(neq, hidden, layers, s), val + ER_TILE);
  input_gradient(neq, hidden, layers, s);
  for (int i = t; i < ER_TILE * 16; i += ER_THREADS) gpr[i] = s.gin[sw(i % 16, i / 16)];
  __syncthreads();
  {
    const float* h = forward_hidden(evo, hidden, layers, s);  // s.x still holds the previous state
    const float* wo = output_ptr(evo, hidden, layers);
    const float* bo = wo + (int64_t)L * hidden;
    for (int i = t; i < ER_TILE * L; i += ER_THREADS) {
      const int p = i / L, o = i % L;
      float v = bo[o];
      for (int j = 0; j < hidden; ++j) v = fmaf(wo[(int64_t)o * hidden + j], h[sw(j, p)], v);
      zdl[p * 8 + o] = v;
    }
    __syncthreads();
  }
  // 3. forward-Euler candidate and the non-equilibrium potential there
  for (int i = t; i < ER_TILE * 8; i += ER_THREADS) {
    const int p = i >> 3, c = i & 7;
    const bool live = !anchor_mode && p0 + p < a.n;
    const float dt = live ? a.time_step[p0 + p] : 0.0f;
    zc[i] = c < L ? zin[i] + (dt / a.tau) * zdl[i] : 0.0f;
  }
  __syncthreads();
  for (int i = t; i < ER_TILE * ER_XLD; i += ER_THREADS) {
    const int p = i / ER_XLD, c = i % ER_XLD;
    s.x[sw(c, p)] = c < 6 ? eps[p * 6 + c] : (c < 6 + L ? zc[p * 8 + c - 6] : 0.0f);
  }
  __syncthreads();
  scalar_output(neq, hidden, layers, forward_hidden(neq, hidden, layers, s), val + 2 * ER_TILE);
  input_gradient(neq, hidden, layers, s);
  for (int i = t; i < ER_TILE * 16; i += ER_THREADS) gca[i] = s.gin[sw(i % 16, i / 16)];
  __syncthreads();
  finish_update(a, p0, ER_TILE, eps, zdl, zc, geq, gpr, gca, val);
}

// ---------------------------------------------------------------------------------------
// The update for hidden width 128 (the reference's models): a CTA of 128 threads per tile of
// P points (32 or 16), two per SM so that one multiplies while the other is between products.
// A layer is a 128 x P product with 8 x P/8 accumulators per thread in registers: per k a
// thread reads two 16-byte rows of weights (four distinct ones per warp) and its points'
// activations (one row per warp) from shared memory for P multiply-adds, two to an
// instruction, where one hidden unit per thread read eight 16-byte broadcasts for 32.  The
// weights stream through two 16-row slices across layer and network boundaries (the slice list
// is laid out once per CTA); activations, and the gradients of the backward pass, are updated in
// place, and what the forward pass keeps for the backward one is silu' (formed beside silu from
// the same exponential).  Every sum runs over k in ascending order from its bias or zero, as in
// the kernel above: the same results.
//
// Bound by issue slots and the latency between slices: two warps per scheduler, FMA pipe about
// half busy.  131,072 points, 4 x 128 (93 GFLOP): 2.61 ms, 36 TFLOP/s of FP32
// (the kernel above: 5.55 ms).
constexpr int ET_THREADS = 128;
constexpr int ET_HID = 128;
constexpr int ET_ROWS = 16;   // weight rows per slice
constexpr int ET_SLICES = 2;  // slices in shared memory

struct Slice {
  int off;   // floats from the parameters' start
  int rows;
};

__host__ __device__ constexpr int in_slices(int in) { return (in + ET_ROWS - 1) / ET_ROWS; }
__host__ __device__ constexpr int hidden_slices(int layers) { return (layers - 1) * (ET_HID / ET_ROWS); }

// One pass over a network's weights: its input layer (rows of W^T) when `input`, then the
// hidden products forwards (W^T) or backwards (W).
struct Pass {
  const NetView* net;
  bool input, hidden, back;
};

template <int THREADS, int N>
__device__ __forceinline__ int slice_list(const float* params, int layers, const Pass (&passes)[N], Slice* list) {
  int base = 0;
#pragma unroll
  for (int part = 0; part < N; ++part) {
    const Pass& q = passes[part];
    const int in = q.input ? in_slices(q.net->in) : 0, len = in + (q.hidden ? hidden_slices(layers) : 0);
    for (int i = threadIdx.x; i < len; i += THREADS) {
      const float *W, *Wt, *b;
      Slice c;
      if (i < in) {
        layer_ptrs(*q.net, ET_HID, 0, &W, &Wt, &b);
        c.rows = min(ET_ROWS, q.net->in - i * ET_ROWS);
        c.off = (int)(Wt - params) + i * ET_ROWS * ET_HID;
      } else {
        const int h = (i - in) / (ET_HID / ET_ROWS), r = (i - in) % (ET_HID / ET_ROWS);
        layer_ptrs(*q.net, ET_HID, q.back ? layers - 1 - h : 1 + h, &W, &Wt, &b);
        c.rows = ET_ROWS;
        c.off = (int)((q.back ? W : Wt) - params) + r * ET_ROWS * ET_HID;
      }
      list[base + i] = c;
    }
    base += len;
  }
  return base;
}

template <int P>
__host__ __device__ inline size_t tile_smem(int layers) {
  return sizeof(float) * ((size_t)ET_HID * P * (1 + layers) + (size_t)ET_SLICES * ET_ROWS * ET_HID +
                          (size_t)P * (2 * ER_XLD + 6 + 8 + 8 + 8 + 6 + 16 + 16 + 3)) +
         sizeof(Slice) * (size_t)(7 * hidden_slices(layers) + 4 * in_slices(ER_XLD));
}

// silu(z) = z / d and silu'(z) = q (1 + z (1 - q)), q = 1 / d, d = 1 + e^-z, with the
// quotients correctly rounded by Markstein's sequences (IBM J. Res. Dev. 34, 1990): a
// reciprocal estimate, one Newton step, and one correction of the quotient by its exact
// remainder.  They are straight-line code, so the units of a thread overlap where a division's
// own branch serialises them.  For |z| <= 69, where d stays below 2^100 and its reciprocal a
// normal number (the caller divides elsewhere); a zero h may differ from the division's in its
// sign.  tests/test_energy_quotients_gpu.py compares silu and silu' with the divisions over every
// 499th float from 1e-30 to 120 of both signs: the same bits.
__device__ __noinline__ float2 silu_general(float z) { return make_float2(silu(z), silu_prime(z)); }

__device__ __forceinline__ float silu_fast(float z, float d, float& q) {
  float r;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(d));
  q = fmaf(r, fmaf(-d, r, 1.0f), r);
  const float h = z * q;
  return fmaf(fmaf(-h, d, z), q, h);
}

// C consecutive floats of a row of shared memory, at a multiple of C from an aligned start.
template <int C>
__device__ __forceinline__ void load_row(const float* src, float (&v)[C]) {
  constexpr int V = C % 4 == 0 ? 4 : C % 2 == 0 ? 2 : 1;
#pragma unroll
  for (int c = 0; c < C; c += V) {
    if constexpr (V == 4) {
      const float4 t = *reinterpret_cast<const float4*>(src + c);
      v[c] = t.x, v[c + 1] = t.y, v[c + 2] = t.z, v[c + 3] = t.w;
    } else if constexpr (V == 2) {
      const float2 t = *reinterpret_cast<const float2*>(src + c);
      v[c] = t.x, v[c + 1] = t.y;
    } else {
      v[c] = src[c];
    }
  }
}
template <int C>
__device__ __forceinline__ void store_row(float* dst, const float (&v)[C]) {
  constexpr int V = C % 4 == 0 ? 4 : C % 2 == 0 ? 2 : 1;
#pragma unroll
  for (int c = 0; c < C; c += V) {
    if constexpr (V == 4)
      *reinterpret_cast<float4*>(dst + c) = make_float4(v[c], v[c + 1], v[c + 2], v[c + 3]);
    else if constexpr (V == 2)
      *reinterpret_cast<float2*>(dst + c) = make_float2(v[c], v[c + 1]);
    else
      dst[c] = v[c];
  }
}
template <int J, int C>
__device__ __forceinline__ float unit(const f32x2 (&acc)[J][C], int j, int c) {  // row j of the thread's 2 J
  const float2 v = unpack2(acc[j / 2][c]);
  return j & 1 ? v.y : v.x;
}
template <int J, int C>
__device__ __forceinline__ void fill_rows(const float* v, f32x2 (&acc)[J][C]) {  // acc = v[row], global
#pragma unroll
  for (int j = 0; j < J; ++j) {
    const f32x2 t = v ? pack2(__ldg(v + 2 * j), __ldg(v + 2 * j + 1)) : 0;
#pragma unroll
    for (int c = 0; c < C; ++c) acc[j][c] = t;
  }
}

// The weight slices of a CTA's products, in the order of its list: the next slice travels in
// registers (4-byte loads: the networks follow each other without padding) while the current
// one is multiplied, and shared memory holds two.
template <int THREADS>
struct WeightStream {
  static constexpr int STAGE = ET_ROWS * ET_HID / THREADS;  // weights of a slice per thread
  const float* params;
  const Slice* list;
  float* w;    // [ET_SLICES][ET_ROWS][128]; free for other use between products
  int count;   // slices of the list
  int next;    // slice the next product starts with
  Slice ahead; // the one after the slice in flight
  float stage[STAGE];

  __device__ __forceinline__ WeightStream(const float* prm, const Slice* slices, int n, float* smem)
      : params(prm), list(slices), w(smem), count(n), next(0), ahead(slices[0]) {
    fetch(0);
  }
  __device__ __forceinline__ void fetch(int i) {
    if (i < count) {
      const Slice c = ahead;
      if (i + 1 < count) ahead = list[i + 1];
      const float* src = params + c.off + threadIdx.x;
      if (c.rows == ET_ROWS) {
#pragma unroll
        for (int e = 0; e < STAGE; ++e) stage[e] = __ldg(src + e * THREADS);
      } else {
#pragma unroll
        for (int e = 0; e < STAGE; ++e)
          stage[e] = threadIdx.x + e * THREADS < c.rows * ET_HID ? __ldg(src + e * THREADS) : 0.0f;
      }
    }
  }
  // acc[j][c] (rows row + 2 j and + 1) += sum_k W[k][.] in[k][col + c] over the next `slices`
  // slices, k ascending; `in` has rows of ld floats.
  template <int J, int C>
  __device__ __forceinline__ void product(const float* in, int ld, int row, int col, int slices, f32x2 (&acc)[J][C]) {
    for (int i = next; i < next + slices; ++i) {
      float* dst = w + (i % ET_SLICES) * ET_ROWS * ET_HID;
      const int rows = list[i].rows;
#pragma unroll
      for (int e = 0; e < STAGE; ++e) dst[threadIdx.x + e * THREADS] = stage[e];
      __syncthreads();  // also: the slice that the next store overwrites has been consumed
      fetch(i + 1);
      const float* wr = dst + row;
      const float* v = in + (i - next) * ET_ROWS * ld + col;
      if (rows == ET_ROWS) {
#pragma unroll
        for (int k = 0; k < ET_ROWS; ++k) step<J, C>(wr + k * ET_HID, v + k * ld, acc);
      } else {
        for (int k = 0; k < rows; ++k) step<J, C>(wr + k * ET_HID, v + k * ld, acc);
      }
    }
    next += slices;
  }
  template <int J, int C>
  __device__ __forceinline__ void step(const float* wr, const float* v, f32x2 (&acc)[J][C]) const {
    f32x2 wj[J];
#pragma unroll
    for (int j = 0; j < J; j += 2) {
      const ulonglong2 t = *reinterpret_cast<const ulonglong2*>(wr + 2 * j);
      wj[j] = t.x, wj[j + 1] = t.y;
    }
    float a[C];
    load_row<C>(v, a);
#pragma unroll
    for (int c = 0; c < C; ++c) {
      const f32x2 aa = pack2(a[c], a[c]);
#pragma unroll
      for (int j = 0; j < J; ++j) acc[j][c] = fma2(wj[j], aa, acc[j][c]);
    }
  }
};

template <int P>
struct TileSmem {
  float* act;   // [128][P] activations / gradients, in place
  float* dact;  // [layers][128][P] silu' of the forward pass
  float* x;     // [ER_XLD][P] network input
  float* gin;   // [ER_XLD][P] input gradient
};

template <int P>
struct Tile {
  static constexpr int THREADS = ET_THREADS;
  static constexpr int PT = P / 8;  // points per thread
  const TileSmem<P>& s;
  WeightStream<THREADS>& ws;
  int row, col;  // the thread's first hidden unit (of eight) and point

  __device__ Tile(const TileSmem<P>& smem, WeightStream<THREADS>& stream) : s(smem), ws(stream) {
    col = PT * (threadIdx.x & 7);
    row = 8 * (threadIdx.x >> 3);
  }

  // Hidden layers of a network; silu' is kept when a backward pass follows.
  __device__ __forceinline__ void forward(const NetView& n, int layers, bool keep) {
    for (int l = 0; l < layers; ++l) {
      const float *W, *Wt, *b;
      layer_ptrs(n, ET_HID, l, &W, &Wt, &b);
      f32x2 acc[4][PT];
      fill_rows(b + row, acc);
      ws.product(l == 0 ? s.x : s.act, P, row, col, l == 0 ? in_slices(n.in) : ET_HID / ET_ROWS, acc);
      __syncthreads();  // every thread has read the layer's input
      float* dl = s.dact + (int64_t)l * ET_HID * P;
      bool large = false;
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        float h[PT], dh[PT];
#pragma unroll
        for (int p = 0; p < PT; ++p) {
          const float z = unit(acc, j, p), d = 1.0f + expf(-z);
          large |= !(fabsf(z) <= 69.0f);
          float q;
          h[p] = silu_fast(z, d, q);
          dh[p] = q * (1.0f + z * (1.0f - q));
        }
        store_row<PT>(s.act + (row + j) * P + col, h);
        if (keep) store_row<PT>(dl + (row + j) * P + col, dh);
      }
      if (large) {
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          float h[PT], dh[PT];
#pragma unroll
          for (int p = 0; p < PT; ++p) {
            const float2 both = silu_general(unit(acc, j, p));
            h[p] = both.x;
            dh[p] = both.y;
          }
          store_row<PT>(s.act + (row + j) * P + col, h);
          if (keep) store_row<PT>(dl + (row + j) * P + col, dh);
        }
      }
    }
    __syncthreads();
  }

  // Output rows of the network from the last activation into out[point * ld + row].  The
  // potentials have no output bias.
  __device__ __forceinline__ void outputs(const NetView& n, int layers, int rows, bool bias, float* out, int ld) {
    const float* wo = output_ptr(n, ET_HID, layers);
    for (int i = threadIdx.x; i < rows * ET_HID; i += THREADS) ws.w[i] = __ldg(wo + i);  // between products
    __syncthreads();
    for (int i = threadIdx.x; i < rows * P; i += THREADS) {
      const int p = i % P, o = i / P;
      float v = bias ? __ldg(wo + rows * ET_HID + o) : 0.0f;
#pragma unroll 16
      for (int j = 0; j < ET_HID; ++j) v = fmaf(ws.w[o * ET_HID + j], s.act[j * P + p], v);
      out[p * ld + o] = v;
    }
    __syncthreads();
  }

  // Input gradient of a scalar network after forward(keep), into rows 0..in-1 of s.gin.
  __device__ __forceinline__ void backward(const NetView& n, int layers) {
    const float* wo = output_ptr(n, ET_HID, layers);
    f32x2 acc[4][PT];
    fill_rows(wo + row, acc);
    for (int l = layers - 1;; --l) {
      const float* dl = s.dact + (int64_t)l * ET_HID * P;
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        float v[PT];
        load_row<PT>(dl + (row + j) * P + col, v);
#pragma unroll
        for (int p = 0; p < PT; ++p) v[p] = unit(acc, j, p) * v[p];
        store_row<PT>(s.act + (row + j) * P + col, v);
      }
      if (l == 0) break;
      fill_rows(nullptr, acc);
      ws.product(s.act, P, row, col, ET_HID / ET_ROWS, acc);
      __syncthreads();  // every thread has read the gradient
    }
    const float *W, *Wt, *b;
    layer_ptrs(n, ET_HID, 0, &W, &Wt, &b);
    for (int i = threadIdx.x; i < ET_HID * n.in; i += THREADS) ws.w[i] = __ldg(W + i);  // between products
    __syncthreads();
    constexpr int G = THREADS / P;  // rows in flight
    constexpr int GR = (14 + G - 1) / G;
    const int p = threadIdx.x % P;
    float g[GR];
#pragma unroll
    for (int i = 0; i < GR; ++i) g[i] = 0.0f;
#pragma unroll 8
    for (int j = 0; j < ET_HID; ++j) {
      const float v = s.act[j * P + p];
#pragma unroll
      for (int i = 0; i < GR; ++i) {
        const int t = threadIdx.x / P + i * G;
        if (t < n.in) g[i] = fmaf(v, ws.w[j * n.in + t], g[i]);
      }
    }
#pragma unroll
    for (int i = 0; i < GR; ++i) {
      const int t = threadIdx.x / P + i * G;
      if (t < n.in) s.gin[t * P + p] = g[i];
    }
    __syncthreads();
  }
};

template <int P>
__global__ void __launch_bounds__(ET_THREADS, 2) energy_rno_tile_kernel(const EnergyArgs a) {
  extern __shared__ __align__(16) float sm[];
  const int layers = a.layers, L = a.latent, t = threadIdx.x;
  TileSmem<P> s;
  s.act = sm;
  s.dact = s.act + ET_HID * P;
  float* w = s.dact + (int64_t)layers * ET_HID * P;
  s.x = w + ET_SLICES * ET_ROWS * ET_HID;
  s.gin = s.x + ER_XLD * P;
  float* eps = s.gin + ER_XLD * P;  // [P][6] network strain
  float* zin = eps + P * 6;         // [P][8] previous latent
  float* zdl = zin + P * 8;         // [P][8] dimensionless rate
  float* zc = zdl + P * 8;          // [P][8] candidate latent
  float* geq = zc + P * 8;          // [P][6]
  float* gpr = geq + P * 6;         // [P][16]
  float* gca = gpr + P * 16;        // [P][16]
  float* val = gca + P * 16;        // [3][P]: eq, previous, candidate values
  Slice* list = reinterpret_cast<Slice*>(val + 3 * P);
  const int64_t p0 = (int64_t)blockIdx.x * P;
  const bool anchor_mode = a.anchors_out != nullptr;
  const NetView eq{a.params, 6, 1};
  const NetView neq{a.params + net_size(6, 1, ET_HID, layers), 6 + L, 1};
  const NetView evo{neq.base + net_size(6 + L, 1, ET_HID, layers), 6 + L, L};
  // eq forward and backward, neq both, evolution forward, neq both at the candidate
  const Pass passes[7] = {{&eq, true, true, false},  {&eq, false, true, true},
                          {&neq, true, true, false}, {&neq, false, true, true},
                          {&evo, true, true, false}, {&neq, true, true, false},
                          {&neq, false, true, true}};
  const int total = slice_list<ET_THREADS>(a.params, layers, passes, list);
  for (int i = t; i < P * 8; i += ET_THREADS) {
    const int p = i >> 3, c = i & 7;
    const bool live = !anchor_mode && p0 + p < a.n;
    if (c < 6) eps[p * 6 + c] = live ? a.strain[(p0 + p) * 6 + c] / a.scale[c] : 0.0f;
    zin[i] = (live && c < L) ? a.latent_in[(p0 + p) * L + c] : 0.0f;
  }
  __syncthreads();
  WeightStream<ET_THREADS> ws(a.params, list, total, w);
  Tile<P> tile(s, ws);
  auto set_input = [&](const float* latent) {  // [eps, latent] (latent may be null: zeros)
    for (int i = t; i < P * ER_XLD; i += ET_THREADS) {
      const int p = i % P, c = i / P;
      s.x[c * P + p] = c < 6 ? eps[p * 6 + c] : (latent && c < 6 + L ? latent[p * 8 + c - 6] : 0.0f);
    }
    __syncthreads();
  };
  auto keep_gradient = [&](float* dst, int width) {
    for (int i = t; i < P * width; i += ET_THREADS) dst[i] = s.gin[(i % width) * P + i / width];
    __syncthreads();
  };
  // the equilibrium potential and its gradient at the network strain; the non-equilibrium ones
  // at the previous state [eps, z_n]; the evolution network there and the forward-Euler
  // candidate; the non-equilibrium potential and gradient at the candidate
#pragma unroll 1
  for (int part = 0; part < 4; ++part) {
    const bool evolution = part == 2;
    const NetView n = part == 0 ? eq : evolution ? evo : neq;
    if (!evolution) set_input(part == 0 ? nullptr : part == 1 ? zin : zc);
    tile.forward(n, layers, !evolution);
    tile.outputs(n, layers, n.out, evolution, evolution ? zdl : val + (part == 3 ? 2 : part) * P, evolution ? 8 : 1);
    if (!evolution) {
      tile.backward(n, layers);
      keep_gradient(part == 0 ? geq : part == 1 ? gpr : gca, part == 0 ? 6 : 16);
    } else {
      for (int i = t; i < P * 8; i += ET_THREADS) {
        const int p = i >> 3, c = i & 7;
        const bool live = !anchor_mode && p0 + p < a.n;
        const float dt = live ? a.time_step[p0 + p] : 0.0f;
        zc[i] = c < L ? zin[i] + (dt / a.tau) * zdl[i] : 0.0f;
      }
      __syncthreads();
    }
  }
  finish_update(a, p0, P, eps, zdl, zc, geq, gpr, gca, val);
}

// ---------------------------------------------------------------------------------------
// Algorithmic tangent d stress / d strain (the reference differentiates the stress with
// autograd, rve_rno.py:283-297).  With network strain e^ = strain / scale,
//   stress_i = (dW_eq/de^_i (e^) + dW_neq/de^_i (e^, z*)) / s_i  (+ constants)
// where z* is the candidate latent z + (dt / tau) f(e^, z) of the current-state integrator
// (the previous latent for the other integrator, which does not depend on the strain), so
//   C_ij = (H_eq(e^)_ij + [H_neq(e^, z*) v_j]_i) / (s_i s_j),  v_j = (e_j, (dt / tau) J_f e_j)
// with J_f the strain Jacobian of the evolution network.  Every Hessian-vector product is
// a forward-over-reverse pass of a SiLU MLP y = w_o . h_{L-1}, h_l = silu(a_l),
// a_l = W_l h_{l-1} + b_l:
//   primal:   a_l (kept), g_{L-1} = w_o, g_{l-1} = W_l^T (g_l * silu'(a_l)) (kept)
//   forward:  adot_0 = W_0 v, adot_l = W_l (silu'(a_{l-1}) * adot_{l-1}) (kept)
//   backward: ddot_{L-1} = w_o * silu''(a_{L-1}) adot_{L-1},
//             ddot_l = (W_{l+1}^T ddot_{l+1}) * silu'(a_l) + g_l * silu''(a_l) adot_l,
//             H v = W_0^T ddot_0.
// One CTA of 128 threads per tile of 32 points, the same feature-major shared layout as
// the update kernel; the tangent directions are looped (6 per network).

__device__ __forceinline__ float silu_second(float z) {
  const float s = 1.0f / (1.0f + expf(-z));
  return s * (1.0f - s) * (2.0f + z * (1.0f - 2.0f * s));
}

struct TanSmem {
  float* x;    // [XLD][TILE] primal input, then the tangent direction
  float* gin;  // [XLD][TILE] input gradient / Hessian-vector product
  float* h0;   // [hidden][TILE] work
  float* h1;   // [hidden][TILE] work
  float* z;    // [layers][hidden][TILE] pre-activations a_l
  float* ad;   // [layers][hidden][TILE] tangent pre-activations adot_l
  float* g;    // [layers - 1][hidden][TILE] activation gradients g_l, l < L - 1
};

// out[j][p] = sum_k W_l[j][k] in[k][p] (+ b_j), thread j < hidden (weights read transposed).
__device__ void tan_mat_forward(const float* Wt, const float* b, int in_l, int hidden, const float* in, float* out) {
  const int j = threadIdx.x;
  if (j < hidden) {
    float acc[ER_TILE];
    const float bj = b ? b[j] : 0.0f;
#pragma unroll
    for (int p = 0; p < ER_TILE; ++p) acc[p] = bj;
    for (int k = 0; k < in_l; ++k) {
      const float w = Wt[(int64_t)k * hidden + j];
#pragma unroll
      for (int q = 0; q < ER_TILE / 4; ++q) {
        const float4 v = *grp(in, k, q);
        acc[4 * q] = fmaf(w, v.x, acc[4 * q]);
        acc[4 * q + 1] = fmaf(w, v.y, acc[4 * q + 1]);
        acc[4 * q + 2] = fmaf(w, v.z, acc[4 * q + 2]);
        acc[4 * q + 3] = fmaf(w, v.w, acc[4 * q + 3]);
      }
    }
#pragma unroll
    for (int q = 0; q < ER_TILE / 4; ++q)
      *grp(out, j, q) = make_float4(acc[4 * q], acc[4 * q + 1], acc[4 * q + 2], acc[4 * q + 3]);
  }
  __syncthreads();
}

// out[t][p] = sum_j W_l[j][t] d[j][p], thread t < in_l.
__device__ void tan_mat_backward(const float* W, int in_l, int hidden, const float* d, float* out) {
  const int t = threadIdx.x;
  if (t < in_l) {
    float acc[ER_TILE];
#pragma unroll
    for (int p = 0; p < ER_TILE; ++p) acc[p] = 0.0f;
    for (int j = 0; j < hidden; ++j) {
      const float w = W[(int64_t)j * in_l + t];
#pragma unroll
      for (int q = 0; q < ER_TILE / 4; ++q) {
        const float4 v = *grp(d, j, q);
        acc[4 * q] = fmaf(v.x, w, acc[4 * q]);
        acc[4 * q + 1] = fmaf(v.y, w, acc[4 * q + 1]);
        acc[4 * q + 2] = fmaf(v.z, w, acc[4 * q + 2]);
        acc[4 * q + 3] = fmaf(v.w, w, acc[4 * q + 3]);
      }
    }
#pragma unroll
    for (int q = 0; q < ER_TILE / 4; ++q)
      *grp(out, t, q) = make_float4(acc[4 * q], acc[4 * q + 1], acc[4 * q + 2], acc[4 * q + 3]);
  }
  __syncthreads();
}

// Elementwise over a [hidden][TILE] buffer (thread j owns row j).
template <typename F>
__device__ __forceinline__ void tan_rows(int hidden, F f) {
  const int j = threadIdx.x;
  if (j < hidden)
#pragma unroll
    for (int p = 0; p < ER_TILE; ++p) f(j, p);
  __syncthreads();
}

// Primal forward (a_l kept) and backward (g_l kept) of a network at the input in s.x;
// returns the buffer of the last activation h_{L-1} (for the output layer).
__device__ const float* tan_primal(const NetView& n, int hidden, int layers, const TanSmem& s, bool backward) {
  const float* hin = s.x;
  float* hout = s.h0;
  for (int l = 0; l < layers; ++l) {
    const float *W, *Wt, *b;
    layer_ptrs(n, hidden, l, &W, &Wt, &b);
    float* zl = s.z + (int64_t)l * hidden * ER_TILE;
    tan_mat_forward(Wt, b, l == 0 ? n.in : hidden, hidden, hin, zl);
    tan_rows(hidden, [&](int j, int p) { hout[sw(j, p)] = silu(zl[sw(j, p)]); });
    hin = hout;
    hout = (hout == s.h0) ? s.h1 : s.h0;
  }
  const float* last = hin;
  if (!backward) return last;
  const float* wo = output_ptr(n, hidden, layers);
  // g_{L-1} = w_o; d = g * silu'(a); g_{l-1} = W_l^T d
  float* d = (last == s.h0) ? s.h1 : s.h0;  // keep h_{L-1} intact
  for (int l = layers - 1; l >= 1; --l) {
    const float* zl = s.z + (int64_t)l * hidden * ER_TILE;
    const float* gl = l == layers - 1 ? nullptr : s.g + (int64_t)l * hidden * ER_TILE;
    tan_rows(hidden, [&](int j, int p) {
      const float gv = gl ? gl[sw(j, p)] : wo[j];
      d[sw(j, p)] = gv * silu_prime(zl[sw(j, p)]);
    });
    const float *W, *Wt, *b;
    layer_ptrs(n, hidden, l, &W, &Wt, &b);
    tan_mat_backward(W, hidden, hidden, d, s.g + (int64_t)(l - 1) * hidden * ER_TILE);
  }
  return last;
}

// Forward tangent from the direction in s.x: adot_l kept in s.ad; returns the buffer of
// hdot_{L-1} = silu'(a_{L-1}) adot_{L-1}.
__device__ const float* tan_forward(const NetView& n, int hidden, int layers, const TanSmem& s) {
  const float* in = s.x;
  float* hd = s.h0;
  for (int l = 0; l < layers; ++l) {
    const float *W, *Wt, *b;
    layer_ptrs(n, hidden, l, &W, &Wt, &b);
    float* adl = s.ad + (int64_t)l * hidden * ER_TILE;
    tan_mat_forward(Wt, nullptr, l == 0 ? n.in : hidden, hidden, in, adl);
    const float* zl = s.z + (int64_t)l * hidden * ER_TILE;
    tan_rows(hidden, [&](int j, int p) { hd[sw(j, p)] = silu_prime(zl[sw(j, p)]) * adl[sw(j, p)]; });
    in = hd;
    hd = (hd == s.h0) ? s.h1 : s.h0;
  }
  return in;
}

// Backward tangent after tan_forward: H v into rows 0..in of s.gin.
__device__ void tan_backward(const NetView& n, int hidden, int layers, const TanSmem& s) {
  const float* wo = output_ptr(n, hidden, layers);
  float* gd = s.h0;  // W_{l+1}^T ddot_{l+1}
  float* dd = s.h1;  // ddot_l
  for (int l = layers - 1; l >= 0; --l) {
    const float* zl = s.z + (int64_t)l * hidden * ER_TILE;
    const float* adl = s.ad + (int64_t)l * hidden * ER_TILE;
    const float* gl = l == layers - 1 ? nullptr : s.g + (int64_t)l * hidden * ER_TILE;
    tan_rows(hidden, [&](int j, int p) {
      const float z = zl[sw(j, p)];
      const float second = (gl ? gl[sw(j, p)] : wo[j]) * silu_second(z) * adl[sw(j, p)];
      dd[sw(j, p)] = (gl ? gd[sw(j, p)] * silu_prime(z) : 0.0f) + second;
    });
    const float *W, *Wt, *b;
    layer_ptrs(n, hidden, l, &W, &Wt, &b);
    tan_mat_backward(W, l == 0 ? n.in : hidden, hidden, dd, l == 0 ? s.gin : gd);
  }
}

__global__ void __launch_bounds__(ER_THREADS) energy_rno_tangent_kernel(const EnergyArgs a) {
  extern __shared__ float sm[];
  const int hidden = a.hidden, layers = a.layers, L = a.latent;
  TanSmem s;
  s.x = sm;
  s.gin = s.x + ER_TILE * ER_XLD;
  s.h0 = s.gin + ER_TILE * ER_XLD;
  s.h1 = s.h0 + ER_TILE * hidden;
  s.z = s.h1 + ER_TILE * hidden;
  s.ad = s.z + (int64_t)layers * ER_TILE * hidden;
  s.g = s.ad + (int64_t)layers * ER_TILE * hidden;
  float* eps = s.g + (int64_t)(layers - 1) * ER_TILE * hidden;  // [TILE][6] network strain
  float* zin = eps + ER_TILE * 6;                                // [TILE][8] previous latent
  float* zc = zin + ER_TILE * 8;                                 // [TILE][8] candidate latent
  float* jf = zc + ER_TILE * 8;                                  // [TILE][8][6] (dt / tau) J_f
  float* cdt = jf + ER_TILE * 48;                                // [TILE] dt / tau
  const int t = threadIdx.x;
  const int64_t p0 = (int64_t)blockIdx.x * ER_TILE;
  const NetView eq{a.params, 6, 1};
  const NetView neq{a.params + net_size(6, 1, hidden, layers), 6 + L, 1};
  const NetView evo{neq.base + net_size(6 + L, 1, hidden, layers), 6 + L, L};
  for (int i = t; i < ER_TILE * 8; i += ER_THREADS) {
    const int p = i >> 3, c = i & 7;
    const bool live = p0 + p < a.n;
    if (c < 6) eps[p * 6 + c] = live ? a.strain[(p0 + p) * 6 + c] / a.scale[c] : 0.0f;
    zin[i] = (live && c < L) ? a.latent_in[(p0 + p) * L + c] : 0.0f;
    if (c == 0) cdt[p] = live ? a.time_step[p0 + p] / a.tau : 0.0f;
  }
  __syncthreads();
  auto set_input = [&](const float* latent) {  // s.x = [e^, latent]
    for (int i = t; i < ER_TILE * ER_XLD; i += ER_THREADS) {
      const int p = i / ER_XLD, c = i % ER_XLD;
      s.x[sw(c, p)] = c < 6 ? eps[p * 6 + c] : (latent && c < 6 + L ? latent[p * 8 + c - 6] : 0.0f);
    }
    __syncthreads();
  };
  // s.x = (e_j, latent part per point (or 0))
  auto set_direction = [&](int j, const float* latent_dir) {
    for (int i = t; i < ER_TILE * ER_XLD; i += ER_THREADS) {
      const int p = i / ER_XLD, c = i % ER_XLD;
      s.x[sw(c, p)] = c < 6 ? (c == j ? 1.0f : 0.0f) : (latent_dir && c < 6 + L ? latent_dir[p * 48 + (c - 6) * 6 + j] : 0.0f);
    }
    __syncthreads();
  };
  // accumulate rows 0..5 of s.gin as column j of the tangent (thread p < TILE owns point p)
  auto store_column = [&](int j, bool add) {
    if (t < ER_TILE && p0 + t < a.n) {
      float* out = a.tangent + (p0 + t) * 36;
      for (int i = 0; i < 6; ++i) {
        const float v = s.gin[sw(i, t)] / (a.scale[i] * a.scale[j]);
        out[6 * i + j] = add ? out[6 * i + j] + v : v;
      }
    }
    __syncthreads();
  };
  // 1. equilibrium potential: its Hessian in the strain block
  set_input(nullptr);
  tan_primal(eq, hidden, layers, s, true);
  for (int j = 0; j < 6; ++j) {
    set_direction(j, nullptr);
    tan_forward(eq, hidden, layers, s);
    tan_backward(eq, hidden, layers, s);
    store_column(j, false);
  }
  // 2. non-equilibrium potential at the stress state, in the total strain direction
  const float* latent_dir = nullptr;
  const float* state = zin;
  if (a.integrator == 1) {
    set_input(zin);
    const float* h = tan_primal(evo, hidden, layers, s, false);
    const float* wo = output_ptr(evo, hidden, layers);
    const float* bo = wo + (int64_t)L * hidden;
    for (int i = t; i < ER_TILE * 8; i += ER_THREADS) {
      const int p = i >> 3, o = i & 7;
      float v = 0.0f;
      if (o < L) {
        v = bo[o];
        for (int j = 0; j < hidden; ++j) v = fmaf(wo[(int64_t)o * hidden + j], h[sw(j, p)], v);
      }
      zc[i] = o < L ? zin[i] + cdt[p] * v : 0.0f;
    }
    __syncthreads();
    for (int j = 0; j < 6; ++j) {
      set_direction(j, nullptr);
      const float* hd = tan_forward(evo, hidden, layers, s);
      for (int i = t; i < ER_TILE * 8; i += ER_THREADS) {
        const int p = i >> 3, o = i & 7;
        float v = 0.0f;
        if (o < L)
          for (int k = 0; k < hidden; ++k) v = fmaf(wo[(int64_t)o * hidden + k], hd[sw(k, p)], v);
        jf[p * 48 + o * 6 + j] = cdt[p] * v;
      }
      __syncthreads();
    }
    latent_dir = jf;
    state = zc;
  }
  set_input(state);
  tan_primal(neq, hidden, layers, s, true);
  for (int j = 0; j < 6; ++j) {
    set_direction(j, latent_dir);
    tan_forward(neq, hidden, layers, s);
    tan_backward(neq, hidden, layers, s);
    store_column(j, true);
  }
}

// ---------------------------------------------------------------------------------------
// The tangent for hidden width 128: a CTA of 256 threads takes NP points and carries their six
// directions through a network together, as 6 NP columns of one product per layer (eight rows
// and 3 NP / 8 columns of it per thread), where a direction at a time streamed every layer's
// weights through 21 passes of 32 columns.  The derivatives of silu do not depend on the
// direction: the primal pass leaves silu'(a_l) and g_l silu''(a_l) in shared memory, the last
// layer's go into its epilogue.  adot_l is kept for the inner layers only: the first layer's is
// formed again (its product has at most 14 terms), the last one's is consumed at once.  The
// weights stream through the same slices as in the update.
//
// Bound like the update; the 16-column primal passes by the latency between slices.  2,048
// points, 4 x 128, with the update before it: 371 us (a direction at a time: 3.91 ms).
constexpr int TT_THREADS = 256;

struct Silu {
  float h, first, second;  // silu, silu', silu''
};

__device__ __noinline__ Silu silu_three_general(float z) { return {silu(z), silu_prime(z), silu_second(z)}; }

template <int NP>
inline size_t tangent_tile_smem(int layers) {
  const size_t floats = (size_t)ET_HID * 6 * NP * (1 + (layers > 2 ? layers - 2 : 0)) +
                        (size_t)ET_HID * NP * (2 * layers - 1) + (size_t)ET_SLICES * ET_ROWS * ET_HID +
                        (size_t)NP * (6 * ER_XLD + ER_XLD + 6 + 8 + 1);
  return floats * sizeof(float) + sizeof(Slice) * (size_t)(10 * hidden_slices(layers) + 8 * in_slices(ER_XLD));
}

template <int NP>
__global__ void __launch_bounds__(TT_THREADS, 1) energy_rno_tangent_tile_kernel(const EnergyArgs a) {
  constexpr int COLS = 6 * NP;
  constexpr int C = COLS / (TT_THREADS / 16);  // columns per thread of a direction product
  constexpr int CP = NP / 8;                   // columns per thread of a primal product
  extern __shared__ __align__(16) float sm[];
  const int layers = a.layers, L = a.latent, t = threadIdx.x, last = layers - 1;
  const int inner = layers > 2 ? layers - 2 : 0;
  float* act = sm;                          // [128][COLS] (primal passes: [128][NP])
  float* ad = act + ET_HID * COLS;          // [inner][128][COLS] adot_1 .. adot_{last-1}
  float* sp = ad + inner * ET_HID * COLS;   // [last][128][NP] silu'(a_l)
  float* gs = sp + last * ET_HID * NP;      // [layers][128][NP] g_l silu''(a_l); silu' of evolution's last layer
  float* w = gs + layers * ET_HID * NP;
  float* xdir = w + ET_SLICES * ET_ROWS * ET_HID;  // [XLD][COLS] directions
  float* x = xdir + ER_XLD * COLS;                 // [XLD][NP] state
  float* eps = x + ER_XLD * NP;                    // [NP][6]
  float* zin = eps + NP * 6;                       // [NP][8]
  float* cdt = zin + NP * 8;                       // [NP] dt / tau
  Slice* list = reinterpret_cast<Slice*>(cdt + NP);
  const int64_t p0 = (int64_t)blockIdx.x * NP;
  const NetView eq{a.params, 6, 1};
  const NetView neq{a.params + net_size(6, 1, ET_HID, layers), 6 + L, 1};
  const NetView evo{neq.base + net_size(6 + L, 1, ET_HID, layers), 6 + L, L};
  const bool moving = a.integrator == 1;  // the stress state depends on the strain
  const Pass passes[12] = {{&eq, true, true, false},      {&eq, false, true, true},      {&eq, true, true, false},
                           {&eq, false, true, true},      {&eq, true, false, false},     {&evo, moving, moving, false},
                           {&evo, moving, moving, false}, {&neq, true, true, false},     {&neq, false, true, true},
                           {&neq, true, true, false},     {&neq, false, true, true},     {&neq, true, false, false}};
  const int total = slice_list<TT_THREADS>(a.params, layers, passes, list);
  for (int i = t; i < NP * 8; i += TT_THREADS) {
    const int p = i >> 3, c = i & 7;
    const bool live = p0 + p < a.n;
    if (c < 6) eps[p * 6 + c] = live ? a.strain[(p0 + p) * 6 + c] / a.scale[c] : 0.0f;
    zin[i] = (live && c < L) ? a.latent_in[(p0 + p) * L + c] : 0.0f;
    if (c == 0) cdt[p] = live ? a.time_step[p0 + p] / a.tau : 0.0f;
  }
  for (int i = t; i < ER_XLD * COLS; i += TT_THREADS) xdir[i] = i / COLS == i % 6 ? 1.0f : 0.0f;
  __syncthreads();
  for (int i = t; i < ER_XLD * NP; i += TT_THREADS) x[i] = i / NP < 6 ? eps[(i % NP) * 6 + i / NP] : 0.0f;
  WeightStream<TT_THREADS> ws(a.params, list, total, w);
  const int warp = t >> 5, lane = t & 31;
  const int group = (warp & 1) * 8 + (lane & 7), col = C * group, pt = col / 6;
  const int row = 8 * ((warp >> 1) * 4 + (lane >> 3));
  const int pcol = CP * (lane & 7), prow = 4 * (warp * 4 + (lane >> 3));

  // a_l of the state in x: silu' and silu'' (of a potential times g_l, by its backward pass);
  // act = h_{L-1} of the evolution network.
  auto primal = [&](const NetView& n, bool potential) {
    const float* wo = output_ptr(n, ET_HID, layers);
#pragma unroll 1
    for (int l = 0; l < layers; ++l) {
      const float *W, *Wt, *b;
      layer_ptrs(n, ET_HID, l, &W, &Wt, &b);
      f32x2 acc[2][CP];
      fill_rows(b + prow, acc);
      ws.product(l == 0 ? x : act, NP, prow, pcol, l == 0 ? in_slices(n.in) : ET_HID / ET_ROWS, acc);
      __syncthreads();  // every thread has read the layer's input
      Silu v[4][CP];
      bool large = false;
#pragma unroll
      for (int j = 0; j < 4; ++j)
#pragma unroll
        for (int c = 0; c < CP; ++c) {
          const float z = unit(acc, j, c);
          large |= !(fabsf(z) <= 69.0f);
          float q;
          v[j][c].h = silu_fast(z, 1.0f + expf(-z), q);
          v[j][c].first = q * (1.0f + z * (1.0f - q));
          v[j][c].second = q * (1.0f - q) * (2.0f + z * (1.0f - 2.0f * q));
        }
      if (large) {
#pragma unroll
        for (int j = 0; j < 4; ++j)
#pragma unroll
          for (int c = 0; c < CP; ++c) v[j][c] = silu_three_general(unit(acc, j, c));
      }
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const int at = (prow + j) * NP + pcol;
        const float wj = __ldg(wo + prow + j);
        float h[CP], f[CP], g[CP];
#pragma unroll
        for (int c = 0; c < CP; ++c) {
          const bool top = potential && l == last;  // g_{L-1} = w_o
          h[c] = top ? wj * v[j][c].first : v[j][c].h;
          f[c] = v[j][c].first;
          g[c] = top ? wj * v[j][c].second : potential ? v[j][c].second : v[j][c].first;
        }
        store_row<CP>(act + at, h);
        if (l < last) store_row<CP>(sp + l * ET_HID * NP + at, f);
        store_row<CP>(gs + l * ET_HID * NP + at, g);
      }
    }
    if (potential) {
#pragma unroll 1
      for (int l = last; l >= 1; --l) {
        f32x2 acc[2][CP];
        fill_rows(nullptr, acc);
        ws.product(act, NP, prow, pcol, ET_HID / ET_ROWS, acc);
        __syncthreads();  // every thread has read the gradient
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const int at = (l - 1) * ET_HID * NP + (prow + j) * NP + pcol;
          float f[CP], g[CP];
          load_row<CP>(sp + at, f);
          load_row<CP>(gs + at, g);
#pragma unroll
          for (int c = 0; c < CP; ++c) {
            const float gl = unit(acc, j, c);
            g[c] = gl * g[c];
            f[c] = gl * f[c];
          }
          store_row<CP>(gs + at, g);
          store_row<CP>(act + (prow + j) * NP + pcol, f);
        }
      }
    }
    __syncthreads();
  };
  // Directions in xdir: act = ddot_{L-1} of a potential, hdot_{L-1} of the evolution network.
  auto forward = [&](const NetView& n, bool potential) {
#pragma unroll 1
    for (int l = 0; l < layers; ++l) {
      f32x2 acc[4][C];
      fill_rows(nullptr, acc);
      ws.product(l == 0 ? xdir : act, COLS, row, col, l == 0 ? in_slices(n.in) : ET_HID / ET_ROWS, acc);
      __syncthreads();
      const float* factor = l < last ? sp + l * ET_HID * NP : gs + last * ET_HID * NP;
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        const float f = factor[(row + j) * NP + pt];
        float v[C];
#pragma unroll
        for (int c = 0; c < C; ++c) v[c] = unit(acc, j, c);
        if (potential && l >= 1 && l < last) store_row<C>(ad + ((l - 1) * ET_HID + row + j) * COLS + col, v);
#pragma unroll
        for (int c = 0; c < C; ++c) v[c] = f * v[c];
        store_row<C>(act + (row + j) * COLS + col, v);
      }
    }
    __syncthreads();
  };
  // H v of a potential after forward(): its six strain rows are a contribution to the tangent.
  auto backward = [&](const NetView& n, bool add) {
#pragma unroll 1
    for (int l = last - 1; l >= 0; --l) {
      f32x2 acc[4][C];
      fill_rows(nullptr, acc);
      ws.product(act, COLS, row, col, ET_HID / ET_ROWS, acc);
      f32x2 first[4][C];
      fill_rows(nullptr, first);
      if (l == 0) ws.product(xdir, COLS, row, col, in_slices(n.in), first);
      __syncthreads();
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        const int at = l * ET_HID * NP + (row + j) * NP + pt;
        const float f = sp[at], g = gs[at];
        float d[C];
        if (l == 0) {
#pragma unroll
          for (int c = 0; c < C; ++c) d[c] = unit(first, j, c);
        } else {
          load_row<C>(ad + ((l - 1) * ET_HID + row + j) * COLS + col, d);
        }
#pragma unroll
        for (int c = 0; c < C; ++c) d[c] = unit(acc, j, c) * f + g * d[c];
        store_row<C>(act + (row + j) * COLS + col, d);
      }
    }
    const float *W, *Wt, *b;
    layer_ptrs(n, ET_HID, 0, &W, &Wt, &b);
    for (int i = t; i < ET_HID * n.in; i += TT_THREADS) w[i] = __ldg(W + i);  // between products
    __syncthreads();
    for (int e = t; e < 6 * COLS; e += TT_THREADS) {
      const int i = e / COLS, q = e % COLS, p = q / 6, j = q % 6;
      float v = 0.0f;
#pragma unroll 16
      for (int k = 0; k < ET_HID; ++k) v = fmaf(act[k * COLS + q], w[k * n.in + i], v);
      if (p0 + p < a.n) {
        float* out = a.tangent + (p0 + p) * 36 + 6 * i + j;
        v = v / (a.scale[i] * a.scale[j]);
        *out = add ? *out + v : v;  // the same thread wrote it
      }
    }
    __syncthreads();
  };
  // 1. equilibrium potential: its Hessian in the strain block
  primal(eq, true);
  forward(eq, true);
  backward(eq, false);
  // 2. non-equilibrium potential at the stress state, in the total strain direction
  for (int i = t; i < L * NP; i += TT_THREADS) x[6 * NP + i] = zin[(i % NP) * 8 + i / NP];
  __syncthreads();
  if (moving) {
    const float* wo = output_ptr(evo, ET_HID, layers);
    primal(evo, false);
    for (int i = t; i < L * ET_HID; i += TT_THREADS) w[i] = __ldg(wo + i);  // between products
    __syncthreads();
    for (int i = t; i < L * NP; i += TT_THREADS) {
      const int o = i / NP, p = i % NP;
      float v = __ldg(wo + L * ET_HID + o);
#pragma unroll 16
      for (int k = 0; k < ET_HID; ++k) v = fmaf(w[o * ET_HID + k], act[k * NP + p], v);
      x[6 * NP + i] = zin[p * 8 + o] + cdt[p] * v;
    }
    __syncthreads();
    forward(evo, false);
    for (int i = t; i < L * ET_HID; i += TT_THREADS) w[i] = __ldg(wo + i);
    __syncthreads();
    for (int i = t; i < L * COLS; i += TT_THREADS) {
      const int o = i / COLS, q = i % COLS;
      float v = 0.0f;
#pragma unroll 16
      for (int k = 0; k < ET_HID; ++k) v = fmaf(w[o * ET_HID + k], act[k * COLS + q], v);
      xdir[6 * COLS + i] = cdt[q / 6] * v;
    }
    __syncthreads();
  }
  primal(neq, true);
  forward(neq, true);
  backward(neq, true);
}

inline size_t tangent_smem(int hidden, int layers) {
  const size_t floats = (size_t)ER_TILE * ER_XLD * 2 + (size_t)ER_TILE * hidden * (2 + 3 * layers - 1) +
                        (size_t)ER_TILE * (6 + 8 + 8 + 48 + 1);
  return floats * sizeof(float);
}

inline size_t energy_smem(int hidden, int layers) {
  const size_t floats = (size_t)ER_TILE * ER_XLD * 2 + (size_t)ER_TILE * hidden * (2 + layers) +
                        (size_t)ER_TILE * (6 + 8 + 8 + 8 + 6 + 16 + 16) + 3 * ER_TILE;
  return floats * sizeof(float);
}

template <int P>
int launch_energy_tile(const EnergyArgs& a, cudaStream_t st) {
  const int64_t blocks = a.anchors_out ? 1 : (a.n + P - 1) / P;
  const size_t smem = tile_smem<P>(a.layers);
  const int rc = allow_dynamic_smem(reinterpret_cast<const void*>(energy_rno_tile_kernel<P>), (int)smem);
  if (rc != CIB_OK) return rc;
  energy_rno_tile_kernel<P><<<(unsigned)blocks, ET_THREADS, smem, st>>>(a);
  return check_launch();
}

// Width 128 with at most four layers (what a tile's shared memory holds) takes the register
// tiles, two CTAs per SM: 16 points each while that leaves no CTA waiting (2,368 points: 167 us,
// with 32-point tiles 189 us), else 32, which read each weight for twice the points (9,400
// points: 230 us against 327 us).  Other widths keep one hidden unit per thread.
int launch_energy(const cib_energy_rno* m, const EnergyArgs& a, int64_t blocks, cudaStream_t st) {
  if (m->hidden == ET_HID && m->layers <= 4)
    return a.n <= 32 * (int64_t)sm_count() ? launch_energy_tile<16>(a, st) : launch_energy_tile<32>(a, st);
  const size_t smem = energy_smem(m->hidden, m->layers);
  if (smem > 200 * 1024) return CIB_ERANGE;
  const int rc = allow_dynamic_smem(reinterpret_cast<const void*>(energy_rno_kernel), 200 * 1024);
  if (rc != CIB_OK) return rc;
  energy_rno_kernel<<<(unsigned)blocks, ER_THREADS, smem, st>>>(a);
  return check_launch();
}

template <int NP>
int launch_tangent_tile(const EnergyArgs& a, cudaStream_t st) {
  const size_t smem = tangent_tile_smem<NP>(a.layers);
  const int rc = allow_dynamic_smem(reinterpret_cast<const void*>(energy_rno_tangent_tile_kernel<NP>), (int)smem);
  if (rc != CIB_OK) return rc;
  energy_rno_tangent_tile_kernel<NP><<<(unsigned)((a.n + NP - 1) / NP), TT_THREADS, smem, st>>>(a);
  return check_launch();
}

bool valid_model(const cib_energy_rno* m) {
  return m && m->params && m->strain_scale && m->hidden >= 1 && m->hidden <= ER_THREADS && m->layers >= 1 &&
         m->layers <= 8 && m->latent >= 1 && m->latent <= 8 && (m->integrator == 0 || m->integrator == 1) &&
         m->reference_time_scale > 0.0;
}

EnergyArgs base_args(const cib_energy_rno* m) {
  EnergyArgs a{};
  a.hidden = m->hidden;
  a.layers = m->layers;
  a.latent = m->latent;
  a.integrator = m->integrator;
  a.tau = (float)m->reference_time_scale;
  a.params = m->params;
  a.scale = m->strain_scale;
  return a;
}

}  // namespace
}  // namespace cib

using namespace cib;

extern "C" int64_t cib_energy_rno_param_count(int32_t hidden, int32_t layers, int32_t latent) {
  if (hidden < 1 || layers < 1 || latent < 1) return -1;
  return net_size(6, 1, hidden, layers) + net_size(6 + latent, 1, hidden, layers) +
         net_size(6 + latent, latent, hidden, layers);
}

extern "C" int cib_energy_rno_anchors(const cib_energy_rno* model, float* anchors, void* stream) {
  if (!valid_model(model) || !anchors) return CIB_EINVAL;
  EnergyArgs a = base_args(model);
  a.n = 1;
  a.anchors_out = anchors;
  return launch_energy(model, a, 1, reinterpret_cast<cudaStream_t>(stream));
}

extern "C" int cib_energy_rno_update(const cib_energy_rno* model, int64_t n, const float* strain, const float* latent,
                                     const float* time_step, const float* anchors, float* stress, float* latent_out,
                                     float* state_rate, float* dimensionless_rate, float* scalars, void* stream) {
  if (!valid_model(model) || n < 0 || !strain || !latent || !time_step || !stress || !latent_out || !state_rate ||
      !dimensionless_rate || !scalars)
    return CIB_EINVAL;
  if (n == 0) return CIB_OK;
  EnergyArgs a = base_args(model);
  a.n = n;
  a.strain = strain;
  a.latent_in = latent;
  a.time_step = time_step;
  a.anchors = anchors;
  a.stress = stress;
  a.latent_out = latent_out;
  a.rate = state_rate;
  a.rate_dimless = dimensionless_rate;
  a.scalars = scalars;
  return launch_energy(model, a, (n + ER_TILE - 1) / ER_TILE, reinterpret_cast<cudaStream_t>(stream));
}

extern "C" int cib_energy_rno_tangent(const cib_energy_rno* model, int64_t n, const float* strain, const float* latent,
                                      const float* time_step, float* tangent, void* stream) {
  if (!valid_model(model) || n < 0 || !strain || !latent || !time_step || !tangent) return CIB_EINVAL;
  if (model->layers < 2) return CIB_EINVAL;
  if (n == 0) return CIB_OK;
  EnergyArgs a = base_args(model);
  a.n = n;
  a.strain = strain;
  a.latent_in = latent;
  a.time_step = time_step;
  a.tangent = tangent;
  // 8 points a tile while one wave of them holds all points (1,184 points: 240 us, 16 a tile
  // 310 us), else 16 (2,048: 310 us against 430 us).
  if (model->hidden == ET_HID && model->layers <= 4)
    return n <= 8 * (int64_t)sm_count() ? launch_tangent_tile<8>(a, reinterpret_cast<cudaStream_t>(stream))
                                        : launch_tangent_tile<16>(a, reinterpret_cast<cudaStream_t>(stream));
  const size_t smem = tangent_smem(model->hidden, model->layers);
  if (smem > 227 * 1024) return CIB_ERANGE;  // e.g. more than 4 hidden layers of 128
  const int rc = allow_dynamic_smem(reinterpret_cast<const void*>(energy_rno_tangent_kernel), 227 * 1024);
  if (rc != CIB_OK) return rc;
  energy_rno_tangent_kernel<<<(unsigned)((n + ER_TILE - 1) / ER_TILE), ER_THREADS, smem,
                              reinterpret_cast<cudaStream_t>(stream)>>>(a);
  return check_launch();
}
