// Matrix-free Jacobi-PCG of the reduced periodic tangent systems (sm_100a).
//
// Replaces the reference's K_red dw = -r direct solve (src/fem/rve/solver.py:143-144) for
// structured periodic boxes.  A cluster of C CTAs (C = 1, 2, 4, 8) solves one system; rank q
// owns the element and node layers of its z slab.
//
// One thread applies one whole element; it reads the search direction of its 8 nodes from
// shared memory, the tangent parameters of its points as 16- or 8-byte vectors (a warp's
// elements are neighbours, so these are contiguous), and writes its 24 nodal contributions
// component-major to shared memory, from where every node gathers its 8 contributions in a
// fixed order.  FP64 sum-factorises the element (hex8_box.cuh: ~690 operations against ~2,600
// for a thread per Gauss point with its shuffles); FP32 keeps the strain-displacement
// products and their rounding.  As many z layers as fit share one such step (all of an 8^3
// RVE in FP64), and where the vectors of a slab fit they stay in shared memory, so an
// iteration of a small system is a handful of barriers and no global traffic but the
// tangent parameters.
//
// FP64 dot products are formed the same way for every C and block size: the z layers are cut
// into 8 fixed groups ("octants"; a rank owns 8 / C of them) and a layer's nodes into chunks
// of 32, summed per octant and chunk column by one warp, and the 8 x min(chunks, 16) partial
// sums are added in one order on every warp of every rank.  Results are therefore bitwise the
// same whatever the launch shape, and the launcher is free to give a system more CTAs than
// asked for when the grid would leave SMs idle.  FP32 dot products are summed per thread,
// block and rank in the order of a plain strided loop, which fixes the result for a given C
// and block size.
//
// What bounds it: latency.  An 8^3 FP64 iteration over 8 CTAs is 14,000 cycles (7.5 us; one
// thread per Gauss point: 36.5 us on one CTA, 9.1 on eight): 4,500 element apply, 1,900 gather,
// 3,200 barriers, 2,300 partial sums, 3,100 vector updates.  Full grids overlap two or four
// CTAs per SM: 1,152 8^3 systems 9.9 ms (24.0), 512 in FP32 2.8 ms (6.0), 96 uneven FP32
// systems over 8 CTAs 7.8 ms (14.7); in brackets a thread per Gauss point with the vectors in
// L2.  Below some 64 elements a thread per element leaves too few threads: 8 x 8 x 1 takes
// 5.9 us an iteration (5.2), 2 x 2 x 2 in FP32 5.6 (4.9).
#include <cooperative_groups.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include <atomic>
#include <type_traits>

#include "cib_common.cuh"
#include "hex8_box.cuh"
#include "rve.cuh"

namespace cg = cooperative_groups;

namespace cib {
namespace {

constexpr int OCTANTS = 8;
constexpr int MAX_COLUMNS = 16;  // chunk columns a layer's partial sums are kept in
// partial sums: p.Ap of each octant's first layer and of its other layers, r.r, r.z, x.x, 0
enum { PART_FIRST = 0, PART_REST, PART_RR, PART_RZ, PART_XX, PART_ZERO, PART_COUNT };

// 4 consecutive tangent values (the points of one x half), as 16-byte loads when VEC.
template <bool VEC>
__device__ __forceinline__ void load4(const double* p, double (&v)[4]) {
  if (VEC) {
    const double2 s = __ldg(reinterpret_cast<const double2*>(p)), t = __ldg(reinterpret_cast<const double2*>(p) + 1);
    v[0] = s.x, v[1] = s.y, v[2] = t.x, v[3] = t.y;
  } else {
#pragma unroll
    for (int k = 0; k < 4; ++k) v[k] = __ldg(p + k);
  }
}

// tau = C eps at the points of one element: C = K 1(x)1 + f P + c n(x)n at a viscoplastic
// point (its flag set), f = 2G, c = 0 at an elastic one.
template <bool VEC>
struct TangentPoint {
  const double* __restrict__ tparam;  // component 0 of the element's first point
  int64_t stride;   // between components
  uint32_t flags;   // bit q: point q is viscoplastic
  double K, two_g;
  double n[6][4], f[4], c[4];

  __device__ __forceinline__ void half(int h) {
    const uint32_t four = (flags >> (4 * h)) & 15u;
#pragma unroll
    for (int t = 0; t < 4; ++t) {
#pragma unroll
      for (int k = 0; k < 6; ++k) n[k][t] = 0.0;
      f[t] = two_g;
      c[t] = 0.0;
    }
    if (four) {
      const double* p = tparam + 4 * h;
#pragma unroll
      for (int k = 0; k < 6; ++k) load4<VEC>(p + k * stride, n[k]);
      load4<VEC>(p + 6 * stride, f);
      load4<VEC>(p + 7 * stride, c);
      if (four != 15u)
#pragma unroll
        for (int t = 0; t < 4; ++t)
          if (!((four >> t) & 1u)) {
#pragma unroll
            for (int k = 0; k < 6; ++k) n[k][t] = 0.0;
            f[t] = two_g;
            c[t] = 0.0;
          }
    }
  }

  __device__ __forceinline__ void operator()(int t, const double (&e)[6], double (&s)[6]) const {
    const double tr = e[0] + e[1] + e[2];
    const double ne = n[0][t] * e[0] + n[1][t] * e[1] + n[2][t] * e[2] + n[3][t] * e[3] + n[4][t] * e[4] + n[5][t] * e[5];
    const double cne = c[t] * ne;
    const double vol = K * tr - f[t] * tr * (1.0 / 3.0);
    const double hf = 0.5 * f[t];
#pragma unroll
    for (int k = 0; k < 3; ++k) s[k] = vol + f[t] * e[k] + cne * n[k][t];
#pragma unroll
    for (int k = 3; k < 6; ++k) s[k] = hf * e[k] + cne * n[k][t];
  }
};

// The same for box_element_points, two points at a time (a thread holds all 8 stresses there).
template <bool VEC>
struct TangentPair {
  const float* __restrict__ tparam;
  int64_t stride;
  uint32_t flags;
  float K, two_g;
  float n[6][2], f[2], c[2];

  __device__ __forceinline__ void pair(int j) {
    const uint32_t two = (flags >> (2 * j)) & 3u;
    const float* p = tparam + 2 * j;
    float v[8][2];
#pragma unroll
    for (int k = 0; k < 8; ++k) {
      v[k][0] = v[k][1] = 0.0f;
      if (two) {
        if (VEC) {
          const float2 t = __ldg(reinterpret_cast<const float2*>(p + k * stride));
          v[k][0] = t.x, v[k][1] = t.y;
        } else {
          v[k][0] = __ldg(p + k * stride), v[k][1] = __ldg(p + k * stride + 1);
        }
      }
    }
#pragma unroll
    for (int t = 0; t < 2; ++t) {
      const bool on = (two >> t) & 1u;
#pragma unroll
      for (int k = 0; k < 6; ++k) n[k][t] = on ? v[k][t] : 0.0f;
      f[t] = on ? v[6][t] : two_g;
      c[t] = on ? v[7][t] : 0.0f;
    }
  }

  __device__ __forceinline__ void operator()(int t, const float (&e)[6], float (&s)[6]) const {
    const float tr = e[0] + e[1] + e[2];
    const float ne = n[0][t] * e[0] + n[1][t] * e[1] + n[2][t] * e[2] + n[3][t] * e[3] + n[4][t] * e[4] + n[5][t] * e[5];
    const float cne = c[t] * ne;
    const float vol = K * tr - f[t] * tr * (float)(1.0 / 3.0);
    const float hf = 0.5f * f[t];
#pragma unroll
    for (int k = 0; k < 3; ++k) s[k] = vol + f[t] * e[k] + cne * n[k][t];
#pragma unroll
    for (int k = 3; k < 6; ++k) s[k] = hf * e[k] + cne * n[k][t];
  }
};

// Flags of the element's 8 points (bytes 8 e ..) as a bit mask.
__device__ __forceinline__ uint32_t point_flags(const uint8_t* f) {
  uint32_t m = 0;
#pragma unroll 1
  for (int k = 0; k < 8; ++k) m |= (f[k] ? 1u : 0u) << k;
  return m;
}

// Sums of N values (a power of two) over the 32 lanes: lane l returns the sum of value
// l / (32 / N).  A lane keeps half of its values per step, so the N sums cost about N + 3
// exchanges instead of 5 N; every value is added in the order of the plain butterfly (16, 8,
// 4, 2, 1), whichever slot it is in.
template <int N>
__device__ __forceinline__ double warp_sums(double (&v)[N], int lane) {
  int o = 16;
#pragma unroll
  for (int n = N / 2; n >= 1; n /= 2, o /= 2) {
    const bool up = (lane & o) != 0;
#pragma unroll
    for (int t = 0; t < n; ++t) {
      const double send = up ? v[t] : v[t + n], keep = up ? v[t + n] : v[t];
      v[t] = keep + __shfl_xor_sync(0xffffffffu, send, o);
    }
  }
  double x = v[0];
#pragma unroll
  for (; o > 0; o /= 2) x += __shfl_xor_sync(0xffffffffu, x, o);
  return x;
}

// A uniform flag the compiler may not specialise loops on: the kernel's body has to stay small
// enough for the instruction cache (unswitched copies of its loops made it 130 KB, and every
// phase of a short iteration then waited for instructions).
__device__ __forceinline__ bool opaque(bool v) {
  int x = v;
  asm volatile("mov.b32 %0, %0;" : "+r"(x));
  return x != 0;
}

// The solve of one system by one cluster.
//
// Vectors are addressed by 3 * (node of the RVE) + d.  Three plans, by the room in shared
// memory (the rule is in plan()):
//  * lean: several ranks, every vector of the slab on chip.  The rank also applies the element
//    layer below its slab and keeps the direction of the node layers on both sides, which it
//    updates itself, as their owners do, from the z = dinv r (FP32: the r) that its neighbours
//    send with their r update: an iteration then needs only the two cluster barriers of its dot
//    products.
//  * on chip: the same vectors in shared memory on a single rank, in one or two steps.
//  * otherwise the vectors stay in global memory (L2); ranks exchange the contributions to
//    their first node layer and the direction above their last through shared memory.
template <typename T, int THREADS, bool VEC>
struct Solver {
  static constexpr int WARPS = THREADS / 32;
  static constexpr bool MIXED = sizeof(T) == 4;  // the direction is kept in double beside sp
  const RvePcgArgs<T>& a;
  const RveDesc d;
  cg::cluster_group cl;
  const int C, rank;  // ranks that share the system: of two or more, no one owns every layer
  int tid, warp, lane;
  int nxy, nchunk, columns, octs;  // octants of this rank
  int k0, k1;
  int prev_rank, prev_layers, next_rank;  // owners of the layers below k0 and from k1 on
  bool wraps;     // one rank owns every layer (the same on every rank: it decides barriers)
  bool lean, onchip, resident;  // resident: sp holds the slab's direction during the solve
  bool wide;      // MIXED, lean: dinv of the layers beside the slab is on chip as well (during the solve
                  // in a partial sum that MIXED does not use: FP32 has no register left, 24^3 over 8
                  // CTAs 8.31 ms, 8.48 with the flag in one)
  bool sends;     // the first node layer's direction goes to the rank below (resident, not lean)
  int kb;         // element layers per step
  int below;      // 1 when sp, ye and info begin at layer k0 - 1 (lean), else 0
  int sp_layers, es;
  float inv_nx, inv_nxy, inv_columns;
  // shared memory
  double* parts;   // [PART_COUNT][octs * columns]
  double* carry;   // [1 or 2][3 nxy]: contributions of a step's last element layer to the next node layer
  double* halo;    // lean: z of node layers k0 - 1 and k1, [2][3 nxy], written by the neighbours (MIXED: r
                   // has these layers, and dinv where `wide`)
  T* sp;           // [sp_layers][3 nxy] search direction
  T* ye;           // [24][es] element contributions
  uint16_t* info;  // flags of the 8 points | phase << 8 per element of the slab (not resident: of the step)
  const double* b;
  const double* dinv;
  double *x, *r, *p, *Ap;
  double* x_out;
  const double* dinv_in;

  __device__ Solver(const RvePcgArgs<T>& args, const RveDesc& desc, cg::cluster_group cluster, int ranks)
      : a(args), d(desc), cl(cluster), C(ranks), rank((int)cluster.block_rank()) {}

  __device__ __forceinline__ int octant_layer(int o) const { return (int)(((int64_t)o * d.nz) / OCTANTS); }
  __device__ __forceinline__ int slab_start(int q) const { return octant_layer(q * (OCTANTS / C)); }
  __device__ __forceinline__ void barrier() {
    if (C > 1)
      cl.sync();
    else
      __syncthreads();
  }
  __device__ __forceinline__ bool p_kept() const { return MIXED || !opaque(resident); }
  __device__ __forceinline__ int wrap_layer(int k) const { return k < 0 ? k + d.nz : k >= d.nz ? k - d.nz : k; }

  // Shared-memory plan, the same on every rank (remote buffers are addressed by offset).
  __device__ void plan(unsigned char* smem, int bytes) {
    tid = threadIdx.x;
    warp = tid >> 5;
    lane = tid & 31;
    nxy = d.nx * d.ny;
    nchunk = (nxy + 31) / 32;
    columns = nchunk < MAX_COLUMNS ? nchunk : MAX_COLUMNS;
    octs = OCTANTS / C;
    inv_nx = 1.0f / (float)d.nx;
    inv_nxy = 1.0f / (float)nxy;
    inv_columns = 1.0f / (float)columns;
    k0 = slab_start(rank);
    k1 = slab_start(rank + 1);
    wraps = C == 1;
    int most = 0;
    for (int q = 0; q < C; ++q) most = max(most, slab_start(q + 1) - slab_start(q));
    prev_rank = next_rank = rank;
    prev_layers = k1 - k0;
    if (!wraps) {  // ranks may be empty
      for (int q = 1; q < C; ++q) {
        prev_rank = (rank + C - q) % C;
        prev_layers = slab_start(prev_rank + 1) - slab_start(prev_rank);
        if (prev_layers > 0) break;
      }
      for (int q = 1; q < C; ++q) {
        next_rank = (rank + q) % C;
        if (slab_start(next_rank + 1) > slab_start(next_rank)) break;
      }
    }
    const int layer_d = 3 * nxy * (int)sizeof(double), layer_t = 3 * nxy * (int)sizeof(T);
    const int part_count = PART_COUNT * (MIXED ? WARPS : octs * columns);
    const int left = bytes - part_count * (int)sizeof(double);
    const int vec_bytes = 4 * most * layer_d;  // r, Ap, x, dinv
    auto info_bytes = [&](int layers) { return (layers * nxy * 2 + 15) & ~15; };
    lean = onchip = false;
    resident = true;
    below = 0;
    int carries = 0;
    const int lean_bytes = info_bytes(most + 1) + 2 * layer_d + (most + 2) * (layer_t + (MIXED ? layer_d : 0)) +
                           (most + 1) * 8 * layer_t + vec_bytes;
    wide = false;
    if (!wraps && lean_bytes <= left) {
      wide = MIXED && lean_bytes + 2 * layer_d <= left;
      lean = onchip = true;
      below = 1;
      kb = most + 1;
      sp_layers = most + 2;
    } else {
      const int sp_res = most + (C > 1 ? 1 : 0);
      const int base = info_bytes(most) + sp_res * layer_t;
      const int chip = base + vec_bytes + (MIXED ? most * layer_d : 0);
      const int half = (most + 1) / 2;
      sp_layers = sp_res;
      if (wraps && chip + layer_d + most * 8 * layer_t <= left) {
        onchip = true;
        carries = 1;
        kb = most;
      } else if (wraps && chip + 2 * layer_d + half * 8 * layer_t <= left && half * nxy >= THREADS) {
        onchip = true;
        carries = 2;
        kb = half;
      } else if (base + layer_d + most * 8 * layer_t <= left) {
        carries = 1;
        kb = most;
      } else {
        // the direction stays resident unless that leaves a step without enough elements and
        // staging it per step would at least double them
        carries = 2;
        kb = (left - base - 2 * layer_d) / (8 * layer_t);
        if (kb < 1 || kb * nxy < THREADS) {
          const int staged = (left - 2 * layer_d - layer_t - 16) / (9 * layer_t + 2 * nxy);
          if (kb < 1 || staged > 2 * kb) {
            resident = false;
            kb = staged > 1 ? staged : 1;  // the launcher guarantees the room for one
            sp_layers = kb + 1;
          }
        }
      }
    }
    sends = resident && !lean && !wraps;
    es = kb * nxy;
    double* at = reinterpret_cast<double*>(smem);
    auto take = [&](int64_t n) {
      double* q = at;
      at += n;
      return q;
    };
    const int64_t row = 3 * (int64_t)nxy, own = row * k0;
    parts = take(part_count);
    carry = take(carries * row);
    if (!MIXED) halo = lean ? take(2 * row) : nullptr;
    if (onchip) {
      r = take((most + (MIXED ? 2 * below : 0)) * row) + (MIXED ? below : 0) * row - own;
      Ap = take(most * row) - own;
      x = take(most * row) - own;
      dinv = take((most + 2 * wide) * row) + wide * row - own;
      if (MIXED) p = take((most + 2 * below) * row) + below * row - own;
    }
    sp = reinterpret_cast<T*>(at);
    ye = sp + sp_layers * row;
    info = reinterpret_cast<uint16_t*>(ye + (int64_t)24 * es);
  }

  __device__ __forceinline__ int steps(int layers) const { return (layers + kb - 1) / kb; }

  // A unit is one (octant, chunk column); each belongs to one warp.
  struct Unit {
    int lo, hi, column;  // layers [lo, hi)
  };
  __device__ __forceinline__ Unit unit(int u) const {
    const int o = (int)(((float)u + 0.5f) * inv_columns);
    return {octant_layer(rank * octs + o), octant_layer(rank * octs + o + 1), u - o * columns};
  }

  // Sums of all ranks' partial sums: p.Ap (kind FIRST, both of its parts) or the pair r.r,
  // r.z (kind RR), the same bits on every warp of every rank.
  __device__ __forceinline__ void total(int kind, double& v0, double& v1) {
    const int per = octs * columns;
    double s0 = 0.0, s1 = 0.0;
    int q = 0, slot = lane;
#pragma unroll 1
    for (int i = lane; i < OCTANTS * columns; i += 32) {
      while (slot >= per) {
        slot -= per;
        ++q;
      }
      const double* src = parts + kind * per + slot;
      if (C > 1) src = cl.map_shared_rank(src, q);
      s0 += src[0];
      s1 += src[per];
      slot += 32;
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      s0 += __shfl_xor_sync(0xffffffffu, s0, o);
      s1 += __shfl_xor_sync(0xffffffffu, s1, o);
    }
    v0 = s0;
    v1 = s1;
  }

  // A unit's pair of sums into kinds `kind` and `kind` + 1.
  __device__ __forceinline__ void store_parts(int kind, int u, double v0, double v1) {
    double v[2] = {v0, v1};
    const double x = warp_sums(v, lane);
    if ((lane & 15) == 0) parts[(kind + (lane >> 4)) * octs * columns + u] = x;
  }

  // MIXED: sums of N values over the cluster, the same on every thread: warp butterflies, the
  // block's warps by a butterfly, the ranks in order.  Holds the barrier of the dot product.
  template <int N>
  __device__ __forceinline__ void sums(int kind, double (&v)[N]) {
    double* mine = parts + kind * WARPS;
#pragma unroll
    for (int t = 0; t < N; ++t) {
      double one[1] = {v[t]};
      const double x = warp_sums(one, lane);
      if (lane == 0) mine[t * WARPS + warp] = x;
    }
    barrier();
#pragma unroll
    for (int t = 0; t < N; ++t) v[t] = 0.0;
#pragma unroll 1
    for (int q0 = 0; q0 < C; q0 += 32 / WARPS) {  // 32 / WARPS ranks at a time, a lane group each
      const int q = q0 + lane / WARPS;
      double x[N];
#pragma unroll
      for (int t = 0; t < N; ++t) {
        const double* src = mine + t * WARPS + (lane & (WARPS - 1));
        x[t] = q >= C ? 0.0 : C > 1 ? *cl.map_shared_rank(src, q) : *src;
      }
#pragma unroll
      for (int t = 0; t < N; ++t) {
#pragma unroll
        for (int o = WARPS / 2; o > 0; o >>= 1) x[t] += __shfl_xor_sync(0xffffffffu, x[t], o);
#pragma unroll
        for (int g = 0; g < 32 / WARPS; ++g) {
          const double y = __shfl_sync(0xffffffffu, x[t], g * WARPS);
          if (q0 + g < C) v[t] += y;
        }
      }
    }
  }

  // Publish a direction value: own layer k, and (not lean) the layer above the rank below.
  __device__ __forceinline__ void put_direction(int k, int f, int64_t i, double v) {
    if (p_kept()) p[i] = v;
    if (!opaque(resident)) return;
    const int row = 3 * nxy;
    sp[(k - k0 + below) * row + f] = (T)v;
    if (opaque(sends) && k == k0) cl.map_shared_rank(sp, prev_rank)[prev_layers * row + f] = (T)v;
  }
  __device__ __forceinline__ double direction(int k, int f, int64_t i) const {
    return p_kept() ? p[i] : (double)sp[(k - k0 + below) * 3 * nxy + f];
  }

  __device__ __forceinline__ uint32_t element_info(int64_t ge) const {
    return point_flags(a.tflag + 8 * ge) | (uint32_t)a.phase[ge] << 8;
  }

  // Elements of layers [ka, kz): contributions into ye.
  __device__ __forceinline__ void elements(int ka, int kz, const BoxCoef<T>& coef, const BoxGrad<T>& grad) {
    const int count = (kz - ka) * nxy, row = 3 * nxy;
    const int first = resident ? ka - k0 + below : 0;         // layer of sp and info
    const int close = resident && wraps ? d.nz : d.nz + 1;    // the layer above it is the first one
#pragma unroll 1
    for (int e = tid; e < count; e += THREADS) {
      const int l = (int)(((float)e + 0.5f) * inv_nxy), n = e - l * nxy;
      const int j = (int)(((float)n + 0.5f) * inv_nx), i = n - j * d.nx;
      const int i1 = i + 1 == d.nx ? 0 : i + 1, j1 = j + 1 == d.ny ? 0 : j + 1;
      const int lb = first + l, lt = lb + 1 == close ? 0 : lb + 1;
      const T* bot = sp + lb * row;
      const T* top = sp + lt * row;
      const int n00 = 3 * (j * d.nx + i), n10 = 3 * (j * d.nx + i1), n01 = 3 * (j1 * d.nx + i), n11 = 3 * (j1 * d.nx + i1);
      auto node = [&](int aa, int dd) -> T {
        const int in = (aa & 1) ? ((aa & 2) ? n11 : n10) : ((aa & 2) ? n01 : n00);
        return ((aa & 4) ? top : bot)[in + dd];
      };
      std::conditional_t<MIXED, TangentPair<VEC>, TangentPoint<VEC>> pt;
      const uint32_t w = info[first * nxy + e];
      pt.flags = w & 255u;
      pt.stride = a.ngp;
      pt.tparam = a.tparam + 8 * (d.eoff + n + (int64_t)nxy * wrap_layer(ka + l));
      const PhaseMat<T>& m = a.mats.m[w >> 8];
      pt.K = m.K;
      pt.two_g = (T)2 * m.G;
      T* y = ye + e;
      auto out = [&](int aa, int dd, T v) { y[(3 * aa + dd) * es] = v; };
      if constexpr (MIXED)
        box_element_points(grad, (T)(d.hx * d.hy * d.hz / 8.0), node, pt, out);
      else
        box_element<T>(coef, node, pt, out);
    }
  }

  // In-plane elements around node n whose local node s is n (s = 0..3).
  __device__ __forceinline__ void around(int n, int (&el)[4]) const {
    const int j = (int)(((float)n + 0.5f) * inv_nx), i = n - j * d.nx;
    const int im = i == 0 ? d.nx - 1 : i - 1, jm = j == 0 ? d.ny - 1 : j - 1;
    el[0] = j * d.nx + i;
    el[1] = j * d.nx + im;
    el[2] = jm * d.nx + i;
    el[3] = jm * d.nx + im;
  }
  // Sum of their contributions to it; y: the layer's contributions to local nodes 0 (4: top).
  __device__ __forceinline__ void gather4(const T* y, const int (&el)[4], double (&v)[3]) const {
    T t[4][3];
#pragma unroll
    for (int s = 0; s < 4; ++s)
#pragma unroll
      for (int dd = 0; dd < 3; ++dd) t[s][dd] = y[(3 * s + dd) * es + el[s]];
#pragma unroll
    for (int dd = 0; dd < 3; ++dd)
      v[dd] = (((double)t[0][dd] + (double)t[1][dd]) + (double)t[2][dd]) + (double)t[3][dd];
  }

  // Ap on the slab and the p.Ap partial sums.
  __device__ __forceinline__ void apply(const BoxCoef<T>& coef, const BoxGrad<T>& grad, double (&pap_mine)[1]) {
    const int layers = k1 - k0, nsteps = lean ? (layers > 0 ? 1 : 0) : steps(layers);
    const bool direct = lean || (wraps && nsteps == 1);  // every contribution to the slab is in ye
    const int per = octs * columns;
    double* p_first = parts + PART_FIRST * per;
    double* p_rest = parts + PART_REST * per;
#pragma unroll 1
    for (int st = 0; st < nsteps; ++st) {
      const int ka = lean ? k0 - 1 : k0 + st * kb, kz = min(k1, ka + kb);
      if (!resident) {  // stage node layers ka .. kz of the direction
        const int row = 3 * nxy;
#pragma unroll 1
        for (int l = 0; l <= kz - ka; ++l) {
          const double* src = p + (int64_t)row * wrap_layer(ka + l);
          for (int f = tid; f < row; f += THREADS) sp[l * row + f] = (T)__ldcg(src + f);
        }
#pragma unroll 1
        for (int e = tid; e < (kz - ka) * nxy; e += THREADS)
          info[e] = (uint16_t)element_info(d.eoff + (int64_t)nxy * ka + e);
        __syncthreads();
      }
      elements(ka, kz, coef, grad);
      __syncthreads();
      const double* carry_in = carry + (size_t)((st + 1) & 1) * 3 * nxy;
      double* carry_out = carry + (size_t)(st & 1) * 3 * nxy;
      // node n of layer k: Ap and the returned part of p.Ap (0 while the layer is open)
      auto gather = [&](int k, int n, double pap) {
        const bool all = opaque(direct);
        const bool open = k == k0 && !all;      // completed after the exchange
        const bool last = k == kz - 1 && !all;  // its top contributions are carried on
        const T* here = ye + (k - ka) * nxy;
        const T* down = ye + 12 * es + (k > ka ? k - ka - 1 : layers - 1) * nxy;
        const int64_t i = 3 * ((int64_t)nxy * k + n);
        int el[4];
        around(n, el);
        double v[3], top[3];
        gather4(here, el, v);
        if (k > ka || all) {
          gather4(down, el, top);
        } else {
#pragma unroll
          for (int dd = 0; dd < 3; ++dd) top[dd] = open ? 0.0 : carry_in[3 * n + dd];
        }
#pragma unroll
        for (int dd = 0; dd < 3; ++dd) {
          v[dd] = (k == 0 && n == 0 && !open) ? 0.0 : top[dd] + v[dd];
          if (!open) pap += direction(k, 3 * n + dd, i + dd) * v[dd];
        }
#pragma unroll
        for (int dd = 0; dd < 3; ++dd) Ap[i + dd] = v[dd];
        if (last) {
          gather4(here + 12 * es, el, v);
#pragma unroll
          for (int dd = 0; dd < 3; ++dd) carry_out[3 * n + dd] = v[dd];
        }
        return pap;
      };
      if constexpr (MIXED) {  // a rank's first layer comes last, whether or not it is complete here
        const int from = max(ka, k0), count = kz - from;
#pragma unroll 1
        for (int l = 0; l < count; ++l) {
          const int k = direct ? (l + 1 < count ? from + l + 1 : from) : from + l;
#pragma unroll 1
          for (int n = tid; n < nxy; n += THREADS) pap_mine[0] = gather(k, n, pap_mine[0]);
        }
      } else {
#pragma unroll 1
        for (int u = warp; u < per; u += WARPS) {
          const Unit m = unit(u);
          const int hi = min(m.hi, kz);
#pragma unroll 1
          for (int k = max(m.lo, max(ka, k0)); k < hi; ++k) {
            double pap[1] = {0.0};
#pragma unroll 1
            for (int n = 32 * m.column + lane; n < nxy; n += 32 * columns) pap[0] = gather(k, n, pap[0]);
            if (k == k0 && !opaque(direct)) continue;
            const double sum = warp_sums(pap, lane);
            if (lane == 0) {
              if (k == m.lo)
                p_first[u] = sum;
              else
                p_rest[u] = k == m.lo + 1 ? sum : p_rest[u] + sum;
            }
          }
        }
      }
      if (st + 1 < nsteps) __syncthreads();
    }
    if (direct || lean) return;
    barrier();  // every rank's last carry is complete
    if (layers == 0) return;
    const double* from = carry + (size_t)((steps(prev_layers) - 1) & 1) * 3 * nxy;
    if (!wraps) from = cl.map_shared_rank(from, prev_rank);
    auto close = [&](int n, double pap) {
      const int64_t i = 3 * ((int64_t)nxy * k0 + n);
      double v[3];
#pragma unroll
      for (int dd = 0; dd < 3; ++dd) {
        v[dd] = (k0 == 0 && n == 0) ? 0.0 : from[3 * n + dd] + Ap[i + dd];
        pap += direction(k0, 3 * n + dd, i + dd) * v[dd];
      }
#pragma unroll
      for (int dd = 0; dd < 3; ++dd) Ap[i + dd] = v[dd];
      return pap;
    };
    if constexpr (MIXED) {
#pragma unroll 1
      for (int n = tid; n < nxy; n += THREADS) pap_mine[0] = close(n, pap_mine[0]);
    } else {
#pragma unroll 1
      for (int u = warp; u < per; u += WARPS) {
        const Unit m = unit(u);
        if (m.lo != k0 || m.hi == k0) continue;
        double pap[1] = {0.0};
#pragma unroll 1
        for (int n = 32 * m.column + lane; n < nxy; n += 32 * columns) pap[0] = close(n, pap[0]);
        const double sum = warp_sums(pap, lane);
        if (lane == 0) p_first[u] = sum;
      }
    }
  }

  // The next direction, dinv r + beta p.  Its owner and, beside a slab, a neighbour form it, and
  // the launch decides where that is: the operations are named, so that every launch rounds
  // alike.  FP32 Newton steps stop on thresholds and keep the form that rounds the owner's
  // product last (4e-6 of a batch's results hang on it); FP64 needs z only.
  __device__ __forceinline__ static double next_direction(double di, double r, double beta, double p) {
    return MIXED ? fma(di, r, __dmul_rn(beta, p)) : fma(beta, p, __dmul_rn(di, r));
  }

  // Lean: the direction of the node layers beside the slab, half of the threads each.
  __device__ __forceinline__ void halo_direction(double beta) {
    const int row = 3 * nxy, side = tid >= THREADS / 2;
    const int k = side ? k1 : k0 - 1;
    T* to = sp + (side ? k1 - k0 + 1 : 0) * row;
    if constexpr (MIXED) {
      const int64_t i = (int64_t)row * k;
      const double* di = parts[PART_ZERO * WARPS] != 0.0 ? dinv + i : dinv_in + (int64_t)row * wrap_layer(k);
      const double* ri = r + i;
      double* pi = p + i;
#pragma unroll 1
      for (int f = tid - side * (THREADS / 2); f < row; f += THREADS / 2) {
        const double v = next_direction(di[f], ri[f], beta, pi[f]);
        pi[f] = v;
        to[f] = (T)v;
      }
    } else {
      const double* z = halo + side * row;
#pragma unroll 1
      for (int f = tid - side * (THREADS / 2); f < row; f += THREADS / 2) to[f] = fma(beta, to[f], z[f]);
    }
  }

  __device__ __forceinline__ void prologue() {
    const int layers = k1 - k0;
#pragma unroll 1
    for (int t = tid; t < PART_COUNT * (MIXED ? WARPS : octs * columns); t += THREADS)
      parts[t] = MIXED && wide && t == PART_ZERO * WARPS ? 1.0 : 0.0;
    if (layers == 0) return;
#pragma unroll 1
    for (int e = tid; e < (layers + below) * nxy; e += THREADS) {
      const int l = (int)(((float)e + 0.5f) * inv_nxy);
      const int64_t ge = d.eoff + (e - l * nxy) + (int64_t)nxy * wrap_layer(k0 - below + l);
      if (resident) info[e] = (uint16_t)element_info(ge);
    }
    if (!lean) return;
    const int row = 3 * nxy;
#pragma unroll 1
    for (int t = tid; t < 2 * row; t += THREADS) {  // the first direction beside the slab
      const int side = t >= row, f = t - side * row;
      const int k = side ? k1 : k0 - 1;
      const int64_t i = (int64_t)row * k + f, g = (int64_t)row * wrap_layer(k) + f;
      const double di = dinv_in[g], v = di * b[g];
      if (wide) const_cast<double*>(dinv)[i] = di;
      if (MIXED) p[i] = v;
      sp[(side ? k1 - k0 + 1 : 0) * row + f] = (T)v;
    }
  }

  __device__ __forceinline__ void solve(int s) {
    const BoxCoef<T> coef = box_coef<T>(d.hx, d.hy, d.hz);
    const BoxGrad<T> grad = box_grad<T>(d.hx, d.hy, d.hz);
    const int row = 3 * nxy;
    prologue();
    barrier();  // parts cleared; every CTA of the cluster runs before its shared memory is written
    const int per = octs * columns;
    double rz = 0.0, rr = 0.0;
    auto start = [&](int k, int f, double& sr, double& sz) {
      const int64_t i = (int64_t)row * k + f;
      const double bi = b[i], di = dinv_in[i], z = di * bi;
      x[i] = 0.0;
      r[i] = bi;
      if (opaque(onchip)) const_cast<double*>(dinv)[i] = di;
      put_direction(k, f, i, z);
      sr += bi * bi;
      sz += bi * z;
    };
    const int entries = (k1 - k0) * row;
    const float inv_row = inv_nxy * (1.0f / 3.0f);
    if constexpr (MIXED) {
      double v[2] = {0.0, 0.0};
#pragma unroll 1
      for (int t = tid; t < entries; t += THREADS) {
        const int l = (int)(((float)t + 0.5f) * inv_row);
        start(k0 + l, t - l * row, v[0], v[1]);
      }
      sums(PART_RR, v);
      rr = v[0];
      rz = v[1];
    } else {
#pragma unroll 1
      for (int u = warp; u < per; u += WARPS) {
        const Unit m = unit(u);
        double bb = 0.0, bz = 0.0;
#pragma unroll 1
        for (int k = m.lo; k < m.hi; ++k)
#pragma unroll 1
          for (int f0 = 96 * m.column + lane; f0 < row; f0 += 96 * columns)
#pragma unroll
            for (int j = 0; j < 3; ++j)
              if (f0 + 32 * j < row) start(k, f0 + 32 * j, bb, bz);
        store_parts(PART_RR, u, bb, bz);
      }
      barrier();
      total(PART_RR, rr, rz);
    }
    const double bnorm = sqrt(rr);
    const double tol = (a.rtol_dev ? *a.rtol_dev : a.rtol) * bnorm;
    int status = 1, iters = 0;
    if (bnorm == 0.0 || !(bnorm == bnorm)) {
      status = (bnorm == 0.0) ? 0 : 2;
    } else {
      for (iters = 0; iters < a.maxit;) {
        double mine[1] = {0.0};  // MIXED: this thread's part of p.Ap
        apply(coef, grad, mine);
        double pap;
        if constexpr (MIXED) {
          sums(PART_FIRST, mine);
          pap = mine[0];
        } else {
          double rest;
          barrier();
          total(PART_FIRST, pap, rest);
          pap += rest;
        }
        if (!(pap > 0.0) || !isfinite(pap)) {
          status = 2;
          break;
        }
        const double alpha = rz / pap;
        // r -= alpha Ap at up to three entries f0, f0 + step, .. of layer k (or of the slab, MIXED)
        double next;
        // the neighbours' copies of the slab's first and last layer
        auto to_prev = [&]() {
          return MIXED ? cl.map_shared_rank(r + (int64_t)row * k0, prev_rank) + prev_layers * row
                       : cl.map_shared_rank(halo, prev_rank) + row;
        };
        auto to_next = [&]() {
          return MIXED ? cl.map_shared_rank(r + (int64_t)row * k0, next_rank) - row : cl.map_shared_rank(halo, next_rank);
        };
        if constexpr (MIXED) {
          double v[2] = {0.0, 0.0};
          const int64_t own = (int64_t)row * k0;
#pragma unroll 1
          for (int t0 = tid; t0 < entries; t0 += 3 * THREADS) {
            double rv[3], av[3], di[3];  // every load before the stores
#pragma unroll
            for (int j = 0; j < 3; ++j) {
              const int t = t0 + j * THREADS;
              const bool in = t < entries;
              rv[j] = in ? r[own + t] : 0.0;
              av[j] = in ? Ap[own + t] : 0.0;
              di[j] = in ? dinv[own + t] : 0.0;
            }
#pragma unroll
            for (int j = 0; j < 3; ++j) {
              const int t = t0 + j * THREADS;
              if (t >= entries) continue;
              const double rn = rv[j] - alpha * av[j], z = rn * di[j];
              r[own + t] = rn;
              v[0] += rn * rn;
              v[1] += z * rn;
            }
          }
          if (opaque(lean) && entries > 0) {  // every thread sends what it wrote
            double* to = to_prev();
#pragma unroll 1
            for (int t = tid; t < row; t += THREADS) to[t] = r[own + t];
            to = to_next();
            const int from = entries - row;
#pragma unroll 1
            for (int t = from + (tid + THREADS - from % THREADS) % THREADS; t < entries; t += THREADS) to[t - from] = r[own + t];
          }
          sums(PART_RR, v);
          rr = v[0];
          next = v[1];
        } else {
#pragma unroll 1
          for (int u = warp; u < per; u += WARPS) {
            const Unit m = unit(u);
            double rs = 0.0, rzs = 0.0;
#pragma unroll 1
            for (int k = m.lo; k < m.hi; ++k)
#pragma unroll 1
              for (int f0 = 96 * m.column + lane; f0 < row; f0 += 96 * columns) {
                const int64_t i = (int64_t)row * k + f0;
                double rv[3], av[3], di[3];  // every load before the stores
#pragma unroll
                for (int j = 0; j < 3; ++j) {
                  const bool in = f0 + 32 * j < row;
                  rv[j] = in ? r[i + 32 * j] : 0.0;
                  av[j] = in ? Ap[i + 32 * j] : 0.0;
                  di[j] = in ? dinv[i + 32 * j] : 0.0;
                }
#pragma unroll
                for (int j = 0; j < 3; ++j) {
                  const double rn = rv[j] - alpha * av[j], z = __dmul_rn(di[j], rn);
                  rs += rn * rn;
                  rzs += rn * z;
                  if (f0 + 32 * j >= row) continue;
                  r[i + 32 * j] = rn;
                  if (opaque(lean)) {
                    if (k == k0) to_prev()[f0 + 32 * j] = z;
                    if (k == k1 - 1) to_next()[f0 + 32 * j] = z;
                  }
                }
              }
            store_parts(PART_RR, u, rs, rzs);
          }
          barrier();
          total(PART_RR, rr, next);
        }
        ++iters;
        // x += alpha p of every iteration, the last one included; the next direction beside it
        const bool stop = !isfinite(rr) || sqrt(rr) <= tol;
        const double beta = stop ? 0.0 : next / rz;
        rz = next;
        if constexpr (MIXED) {
          const int64_t own = (int64_t)row * k0;
#pragma unroll 1
          for (int t0 = tid; t0 < entries; t0 += 2 * THREADS) {
            double rv[2], di[2], pv[2], xv[2];
#pragma unroll
            for (int j = 0; j < 2; ++j) {
              const int t = t0 + j * THREADS;
              const bool in = t < entries;
              rv[j] = in ? r[own + t] : 0.0;
              di[j] = in ? dinv[own + t] : 0.0;
              pv[j] = in ? p[own + t] : 0.0;
              xv[j] = in ? x[own + t] : 0.0;
            }
#pragma unroll
            for (int j = 0; j < 2; ++j) {
              const int t = t0 + j * THREADS;
              if (t >= entries) continue;
              const double v = next_direction(di[j], rv[j], beta, pv[j]);
              x[own + t] = xv[j] + alpha * pv[j];
              p[own + t] = v;
              if (!opaque(resident)) continue;
              sp[below * row + t] = (T)v;
              if (opaque(sends) && t < row) cl.map_shared_rank(sp, prev_rank)[prev_layers * row + t] = (T)v;
            }
          }
        } else {
#pragma unroll 1
          for (int u = warp; u < per; u += WARPS) {
            const Unit m = unit(u);
#pragma unroll 1
            for (int k = m.lo; k < m.hi; ++k)
#pragma unroll 1
              for (int f0 = 96 * m.column + lane; f0 < row; f0 += 96 * columns) {
                const int64_t i = (int64_t)row * k + f0;
                double rv[3], di[3], pv[3], xv[3];
#pragma unroll
                for (int j = 0; j < 3; ++j) {
                  const bool in = f0 + 32 * j < row;
                  rv[j] = in ? r[i + 32 * j] : 0.0;
                  di[j] = in ? dinv[i + 32 * j] : 0.0;
                  pv[j] = in ? direction(k, f0 + 32 * j, i + 32 * j) : 0.0;
                  xv[j] = in ? x[i + 32 * j] : 0.0;
                }
#pragma unroll
                for (int j = 0; j < 3; ++j) {
                  if (f0 + 32 * j >= row) continue;
                  x[i + 32 * j] = xv[j] + alpha * pv[j];
                  put_direction(k, f0 + 32 * j, i + 32 * j, next_direction(di[j], rv[j], beta, pv[j]));
                }
              }
          }
        }
        if (stop) {
          status = isfinite(rr) ? 0 : 2;
          break;
        }
        if (lean) {
          if (k1 > k0) halo_direction(beta);
          __syncthreads();
        } else {
          barrier();  // the direction of every rank is visible before the next apply
        }
      }
    }
    const double rnorm = sqrt(rr);
    double xx = 0.0;
    if constexpr (MIXED) {
      double v[1] = {0.0};
      const int64_t own = (int64_t)row * k0;
#pragma unroll 1
      for (int t = tid; t < entries; t += THREADS) {
        const double xv = x[own + t];
        if (opaque(onchip)) x_out[own + t] = xv;
        v[0] += xv * xv;
      }
      sums(PART_XX, v);
      xx = v[0];
    } else {
#pragma unroll 1
      for (int u = warp; u < per; u += WARPS) {
        const Unit m = unit(u);
        double part = 0.0;
#pragma unroll 1
        for (int k = m.lo; k < m.hi; ++k)
#pragma unroll 1
          for (int f0 = 96 * m.column + lane; f0 < row; f0 += 96 * columns)
#pragma unroll
            for (int j = 0; j < 3; ++j) {
              if (f0 + 32 * j >= row) continue;
              const int64_t i = (int64_t)row * k + f0 + 32 * j;
              const double xv = x[i];
              if (opaque(onchip)) x_out[i] = xv;
              part += xv * xv;
            }
        store_parts(PART_XX, u, part, 0.0);
      }
      barrier();
      double zero;
      total(PART_XX, xx, zero);
    }
    if (rank == 0 && tid == 0) {
      a.status[s] = status;
      a.iterations[s] = iters;
      a.rel_residual[s] = bnorm > 0.0 ? rnorm / bnorm : 0.0;
      a.xnorm[s] = sqrt(xx);
    }
    barrier();  // no rank leaves while another may still read its shared memory
  }
};

template <typename T, int THREADS, int MIN_BLOCKS, bool VEC>
__global__ void __launch_bounds__(THREADS, MIN_BLOCKS)
    rve_pcg_kernel(const RvePcgArgs<T> a, const int requested, const int smem_bytes) {
  extern __shared__ __align__(16) unsigned char smem[];
  cg::cluster_group cl = cg::this_cluster();
  const int C = (int)cl.num_blocks();
  const int s = blockIdx.x / C;
  const int r = a.sys_rve[s];
  if (a.active && !a.active[r]) return;  // the whole cluster leaves together
  const RveDesc d = a.desc[r];
  const int64_t E = (int64_t)d.nx * d.ny * d.nz;
  const int64_t off = a.sys_off[s];  // vector offset of this system (3 * node base)
  // a caller that asks for C CTAs needs a layer for each; a library-owned work vector must hold the system
  const bool outside = a.vec_len >= 0 && (off < 0 || E < 0 || off + 3 * E > a.vec_len);
  if (d.nz < requested || outside) {
    if (cl.block_rank() == 0 && threadIdx.x == 0) {
      a.status[s] = 3;
      a.iterations[s] = 0;
      a.rel_residual[s] = 0.0;
      a.xnorm[s] = 0.0;
    }
    return;
  }
  // A single layer has one owner: it solves alone, without a cluster barrier, and the ranks that
  // the launcher added leave (it does not know the layers).  From two layers on two ranks or more
  // own some, whatever C.
  const int ranks = d.nz > 1 ? C : 1;
  if ((int)cl.block_rank() >= ranks) return;
  Solver<T, THREADS, VEC> S(a, d, cl, ranks);
  S.b = a.b + off;
  S.dinv = S.dinv_in = a.dinv + 3 * d.eoff;
  S.x = S.x_out = a.x + off;
  S.r = a.r + off;
  S.p = a.p + off;
  S.Ap = a.Ap + off;
  S.plan(smem, smem_bytes);
  S.solve(s);
}

template <typename T, int THREADS, int MIN_BLOCKS, bool VEC>
int launch_shape(const RvePcgArgs<T>& a, int nsys, int max_nxy, int requested, int cluster, cudaStream_t st) {
  const void* fn = reinterpret_cast<const void*>(rve_pcg_kernel<T, THREADS, MIN_BLOCKS, VEC>);
  constexpr int SM_BYTES = 228 * 1024, RESERVED = 1024, MOST = 227 * 1024;
  // CTAs an SM has to hold at once: a small grid gives each of them more shared memory
  const int64_t waves = ((int64_t)nsys * cluster + sm_count() - 1) / sm_count();
  const int per_sm = waves < MIN_BLOCKS ? (int)waves : MIN_BLOCKS;
  int smem = SM_BYTES / per_sm - RESERVED - 128;
  // one element layer, its staged direction and both carries always fit (with the partial sums of
  // a system that one CTA solves, where the caller asked for one)
  const int columns = max_nxy >= 32 * MAX_COLUMNS ? MAX_COLUMNS : (max_nxy + 31) / 32;
  const int64_t least = (int64_t)PART_COUNT * (OCTANTS / requested) * columns * 8 + (int64_t)max_nxy * (50 + 30 * sizeof(T)) + 32;
  if (least > smem) smem = (int)((least + 15) & ~15LL);
  if (smem > MOST) return CIB_ERANGE;
  const int rc = allow_dynamic_smem(fn, smem > MOST ? MOST : smem);
  if (rc != CIB_OK) return rc;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)nsys * (unsigned)cluster, 1, 1);
  cfg.blockDim = dim3(THREADS, 1, 1);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = (unsigned)cluster;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  cudaLaunchKernelEx(&cfg, rve_pcg_kernel<T, THREADS, MIN_BLOCKS, VEC>, a, requested, smem);
  return check_launch();
}

// Clusters of C CTAs, an SM's whole shared memory each, that run at the same time: fewer than
// sm_count() / C, as a cluster stays within a GPC (15 of 8 and 33 of 4 on the B200s measured).
// Beyond them a launch takes a second turn: 18 systems of 8^3 in clusters of 8 1.54 ms, of 4
// 0.98; 36 in clusters of 4 1.83 ms, of 2 1.33.  Kept per device; 0 where none runs.
int resident_clusters(int C) {
  static std::atomic<int> kept[64][9];  // 1 + the number
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return 0;
  if (const int k = kept[dev][C].load()) return k - 1;
  const auto fn = rve_pcg_kernel<double, 128, 2, true>;
  constexpr int SMEM = 227 * 1024;
  if (allow_dynamic_smem(reinterpret_cast<const void*>(fn), SMEM) != CIB_OK) return 0;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)C, 1, 1);
  cfg.blockDim = dim3(128, 1, 1);
  cfg.dynamicSmemBytes = SMEM;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = (unsigned)C;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  int n = 0;
  if (cudaOccupancyMaxActiveClusters(&n, fn, &cfg) != cudaSuccess) {
    cudaGetLastError();
    return 0;
  }
  kept[dev][C].store(1 + n);
  return n;
}

}  // namespace

// cluster: the CTAs per system (1, 2, 4 or 8) in bits 0-3 and the launch shape in bits 4-7
// (block size: 0 the default, 1 128 threads, 2 FP32 512 / FP64 256, 3 FP32 256 / FP64 64).
//
// FP64: neither the shape nor the number of CTAs changes a result, so a launch that would
// leave SMs idle gets up to 8 CTAs per system while all clusters run at once (one 8^3 system: 4.2 ms with one CTA before,
// 0.8 ms with 8; 1 to 16 elements per CTA still gain, 4^3 0.31 ms against 0.40 with one; of a
// system of one layer only the first CTA stays), and
// the default block is 256 threads where an SM holds one CTA of wide layers (one 24^3 system:
// 19.3 ms at 128 threads, 16.4 at 256) and 128 otherwise (1,152 8^3 systems: 10.0 ms against
// 10.4; 22.8 ms with a thread per Gauss point).
// FP32: dot products are summed per block and rank, so both are taken as given; the shape applies
// to two CTAs or more (one CTA is the solve of cib_rve_pcg).
template <typename T>
int launch_rve_pcg_cluster(const RvePcgArgs<T>& a, int nsys, int max_nxy, int cluster, cudaStream_t st) {
  const int c = cluster & 15, shape = (cluster >> 4) & 15;
  if ((cluster >> 8) != 0 || shape > 3) return CIB_EINVAL;
  if (c != 1 && c != 2 && c != 4 && c != 8) return CIB_EINVAL;
  // largest layer: the accepted range of the entry points
  const size_t layer = c == 1 ? (24 + 9) * sizeof(double) : 24 * sizeof(T) + 12 * sizeof(double);
  if ((size_t)max_nxy * layer > 200 * 1024) return CIB_ERANGE;
  const bool vec = aligned16(a.tparam) && (a.ngp % (16 / (int)sizeof(T))) == 0;  // rows of 16-byte loads
  if constexpr (sizeof(T) == 4) {
    switch (c == 1 ? 0 : shape) {
      case 1:
        return vec ? launch_shape<T, 128, 4, true>(a, nsys, max_nxy, c, c, st)
                   : launch_shape<T, 128, 4, false>(a, nsys, max_nxy, c, c, st);
      case 2:
        return vec ? launch_shape<T, 512, 1, true>(a, nsys, max_nxy, c, c, st)
                   : launch_shape<T, 512, 1, false>(a, nsys, max_nxy, c, c, st);
      default:
        return vec ? launch_shape<T, 256, 2, true>(a, nsys, max_nxy, c, c, st)
                   : launch_shape<T, 256, 2, false>(a, nsys, max_nxy, c, c, st);
    }
  } else {
    int C = c;
    while (C < 8 && (int64_t)nsys * (2 * C) <= sm_count() && nsys <= resident_clusters(2 * C)) C *= 2;
    if (!vec) return launch_shape<T, 128, 2, false>(a, nsys, max_nxy, c, C, st);
    const bool wide = (int64_t)nsys * C <= sm_count() && max_nxy >= 256;
    if (shape == 3) return launch_shape<T, 64, 4, true>(a, nsys, max_nxy, c, C, st);
    if (shape == 2 || (shape == 0 && wide)) return launch_shape<T, 256, 1, true>(a, nsys, max_nxy, c, C, st);
    return launch_shape<T, 128, 2, true>(a, nsys, max_nxy, c, C, st);
  }
}

template <typename T>
int launch_rve_pcg(const RvePcgArgs<T>& a, int nsys, int max_nxy, cudaStream_t st) {
  return launch_rve_pcg_cluster<T>(a, nsys, max_nxy, 1, st);
}

template int launch_rve_pcg<float>(const RvePcgArgs<float>&, int, int, cudaStream_t);
template int launch_rve_pcg<double>(const RvePcgArgs<double>&, int, int, cudaStream_t);
template int launch_rve_pcg_cluster<float>(const RvePcgArgs<float>&, int, int, int, cudaStream_t);
template int launch_rve_pcg_cluster<double>(const RvePcgArgs<double>&, int, int, int, cudaStream_t);

}  // namespace cib
