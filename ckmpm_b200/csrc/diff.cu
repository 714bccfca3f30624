// Differentiable form: a rollout of the fixed-corotated CK-MPM substep with
// per-particle Young's modulus, its hand-written adjoint (diff_math.cuh), and
// substep checkpointing with recomputation.  No counterpart in the reference.
//
// Device layout (cells per axis n_c, nodes nn = 2 n_c^3 over both staggered grids):
//  * particles sorted once per rollout (perm), so that a CTA's lie in a small box
//    of nodes: it makes that box's velocities, or their adjoints, itself from the sums and
//    collects its deposits in a shared tile;
//  * gsum[3]: int64 fixed-point node sums [node][m, mvx, mvy, mvz] per unit
//    particle mass (2^36 scale, as the substep's P2G tile), one read, one written
//    and one cleared in a substep; exact, so a recomputed segment reproduces the
//    forward bit for bit;
//  * bbox[s]: node-coordinate box of what substep s reads (min x,y,z, max x,y,z);
//    clearing runs over that box only;
//  * particles SoA (x[3][n], F[9][n]); checkpoints every K substeps hold x, F
//    and the node velocities of that substep (the forward writes those states
//    straight into their checkpoint slots); the backward recomputes one segment
//    at a time into a tape of the segment's other K - 1 substeps, then runs the
//    adjoint.  With K = 1 every substep is a checkpoint and the backward is the
//    adjoint alone (about 2.2 GB for 50k particles, 200 substeps and a 64^3
//    grid: HBM, not recomputation, holds the rollout);
//  * vbar[3]: the node-velocity adjoint the particle adjoints scatter, as exact
//    int64 fixed-point sums like the forward's, so gradients are bitwise
//    reproducible too.  Its unit is set on the device at the start of each
//    backward from the largest incoming adjoint (the backward is linear in its
//    seed): 2^-40 of that largest component.
#include <climits>

#include "diff_math.cuh"

namespace ckmpm {
namespace diffk {

using diff::DenseGrid;
using diff::Fwd;
using diff::Particle;

constexpr int kThreads = 128;
constexpr float kScale = 68719476736.0f;  // 2^36
constexpr float kMaxValue = 131072.0f;    // 2^17
constexpr uint32_t kErrOutside = 1u, kErrRange = 2u;
// CTAs of a particle kernel at least: those past the particles help to zero a box that is
// large for the few particles in it (500 particles spread over a 64^3-cell domain: 93 us a forward
// substep zeroed by their 4 CTAs, 25 by 296, 26 by 592).
constexpr uint32_t kZeroCtas = 296;
constexpr float kAdjUnits = 1099511627776.0f;  // 2^40 fixed-point units per largest seed component
constexpr float kAdjMaxUnits = 4.6e18f;        // |contribution| bound in units (< 2^62)

struct Box {
  int lo[3], hi[3];
};

struct Dev {
  DenseGrid G;
  uint32_t n;
  float dx, inv_dx, mass, vol_over_mass, unit;  // unit = mass * 2^-36
  uint32_t* status;
  float* adj_scale;  // [0]: fixed-point units per adjoint unit, [1]: its inverse; [2]: max |seed| (bits)
};

__device__ __forceinline__ uint32_t particle_ctas(const Dev& d) { return (d.n + kThreads - 1) / kThreads; }

__device__ __forceinline__ void box_reset(int* b) {
  b[0] = b[1] = b[2] = INT_MAX;
  b[3] = b[4] = b[5] = INT_MIN;
}

// ---- Particle order
//
// The rollout keeps its particles in an order of its own, made from x0 by every
// forward: pencils of 2 x 2 cells in x and y, run through in z, neighbouring
// pencils in opposite directions, so that the kThreads particles of a CTA lie in
// a few cells of one pencil.  Their stencils then read the same nodes (L1 hits
// instead of L2 gathers) and their deposits fit a small shared tile.  Nothing
// depends on the order: every particle computes by itself and the node sums are
// exact.  Within a chunk of kThreads, particle j of the sorted order takes place
// (j % 4) * 32 + j / 4: a warp's lanes then spread over the whole chunk's cells,
// so fewer of them add to the same words at once.
__host__ __device__ __forceinline__ uint32_t order_bins(const DenseGrid& G) {
  return static_cast<uint32_t>(G.n[0] / 2) * static_cast<uint32_t>(G.n[1] / 2) * static_cast<uint32_t>(G.n[2]);
}

__device__ __forceinline__ uint32_t order_bin(const Dev& d, const float* x) {
  int c[3];
#pragma unroll
  for (int a = 0; a < 3; ++a) c[a] = min(max(static_cast<int>(x[a] * d.inv_dx), 0), d.G.n[a] - 1);
  const int px = c[0] >> 1, py = c[1] >> 1, ny = d.G.n[1] >> 1;
  const int y = (px & 1) ? ny - 1 - py : py;
  const int z = ((px * ny + y) & 1) ? d.G.n[2] - 1 - c[2] : c[2];
  return static_cast<uint32_t>((px * ny + y) * d.G.n[2] + z);
}

__global__ void order_count_kernel(Dev d, const float* __restrict__ x0, uint32_t* __restrict__ bins,
                                   uint32_t* __restrict__ bin, uint32_t* __restrict__ rank) {
  const uint32_t p = blockIdx.x * blockDim.x + threadIdx.x;
  if (p >= d.n) return;
  const uint32_t b = order_bin(d, x0 + 3 * static_cast<size_t>(p));
  bin[p] = b;
  rank[p] = atomicAdd(bins + b, 1u);
}

__global__ void order_place_kernel(uint32_t n, const uint32_t* __restrict__ first, const uint32_t* __restrict__ bin,
                                   const uint32_t* __restrict__ rank, uint32_t* __restrict__ perm) {
  const uint32_t p = blockIdx.x * blockDim.x + threadIdx.x;
  if (p >= n) return;
  uint32_t j = first[bin[p]] + rank[p];
  const uint32_t chunk = j / kThreads * kThreads;
  if (chunk + kThreads <= n) j = chunk + ((j - chunk) % 4) * (kThreads / 4) + (j - chunk) / 4;
  perm[j] = p;
}

// ---- CTA tile
//
// Box of base cells (both grids) of the CTA's particles and the nodes they reach.
// Deposits go to a shared tile of exact 64-bit sums over that box, two native
// 32-bit atomics per value with the carry from the low word (as the substep's
// P2G tile), and from there to the grid, one reduction per touched node and
// channel; a box of more than kTileCap nodes deposits into the grid directly.
// The sums are exact either way.  Bound before: 64 global 64-bit reductions per
// particle, 3.2 M a launch on the 50k-particle cube.
constexpr int kTileCap = 1024;  // nodes of both grids

struct CtaBox {
  int lo[3], e[3];  // first node, nodes per axis (one grid)
  int nodes;        // of both grids; 0: no tile
};

__device__ __forceinline__ void cta_box_merge(int* s_box, bool use, const int* lo, const int* hi) {
#pragma unroll
  for (int a = 0; a < 3; ++a) {
    const int l = __reduce_min_sync(0xffffffffu, use ? lo[a] : INT_MAX);
    const int h = __reduce_max_sync(0xffffffffu, use ? hi[a] : INT_MIN);
    if ((threadIdx.x & 31) == 0) {
      atomicMin(s_box + a, l);
      atomicMax(s_box + 3 + a, h);
    }
  }
}

__device__ __forceinline__ CtaBox cta_box(const int* s_box) {
  CtaBox b;
  int64_t v = 2;
#pragma unroll
  for (int a = 0; a < 3; ++a) {
    b.lo[a] = s_box[a];
    b.e[a] = s_box[3 + a] >= s_box[a] ? s_box[3 + a] - s_box[a] + 1 : 0;
    v *= b.e[a];
  }
  b.nodes = v <= kTileCap ? static_cast<int>(v) : 0;
  return b;
}

__device__ __forceinline__ void tile_zero(unsigned* tile, int words) {
  for (int i = threadIdx.x; i < words / 4; i += kThreads) reinterpret_cast<uint4*>(tile)[i] = make_uint4(0u, 0u, 0u, 0u);
}

// Exact add to word pair `lo_word`, its high word `plane` words later.
__device__ __forceinline__ void tile_add(unsigned* lo_word, int plane, long long v) {
  const unsigned lo = static_cast<unsigned>(v);
  const unsigned old = atomicAdd(lo_word, lo);
  atomicAdd(lo_word + plane, static_cast<unsigned>(v >> 32) + (old + lo < lo ? 1u : 0u));
}

// First and last node of a particle's stencils over both grids.  A position far
// outside (or infinite) saturates the base cells, so `hi` may wrap: box_in_grid
// bounds both ends.
__device__ __forceinline__ void stencil_box(const diff::Stencil<float>& st, int* lo, int* hi) {
#pragma unroll
  for (int a = 0; a < 3; ++a) {
    lo[a] = min(st.a[0][a].base, st.a[1][a].base);
    hi[a] = max(st.a[0][a].base, st.a[1][a].base) + 1;
  }
}

__device__ __forceinline__ bool box_in_grid(const DenseGrid& G, const int* lo, const int* hi) {
  bool in = true;
#pragma unroll
  for (int a = 0; a < 3; ++a) in &= lo[a] >= 0 && lo[a] < G.n[a] && hi[a] >= lo[a] && hi[a] < G.n[a];
  return in;
}

// Node (g, x, y, z) of entry i of a CTA box.
__device__ __forceinline__ int box_node(const Dev& d, const CtaBox& b, int i, int& cx, int& cy, int& cz) {
  const int per = b.nodes >> 1, g = i >= per ? 1 : 0, j = i - g * per;
  const int z = j % b.e[2], xy = j / b.e[2], y = xy % b.e[1], x = xy / b.e[1];
  cx = b.lo[0] + x;
  cy = b.lo[1] + y;
  cz = b.lo[2] + z;
  return diff::node_index(d.G, g, cx, cy, cz);
}

// Entry of a node in a CTA box's tile.
__device__ __forceinline__ int box_entry(const CtaBox& b, int g, int cx, int cy, int cz) {
  return g * (b.nodes >> 1) + ((cx - b.lo[0]) * b.e[1] + cy - b.lo[1]) * b.e[2] + cz - b.lo[2];
}

// Adds the tile's touched words to the grid arrays (kCh channels per node).
template <int kCh>
__device__ __forceinline__ void tile_flush(const Dev& d, const CtaBox& b, const unsigned* tile,
                                           unsigned long long* __restrict__ out) {
  const int plane = kCh * kTileCap;
  for (int i = threadIdx.x; i < b.nodes; i += kThreads) {
    int cx, cy, cz;
    unsigned long long* q = out + kCh * static_cast<size_t>(box_node(d, b, i, cx, cy, cz));
#pragma unroll
    for (int c = 0; c < kCh; ++c) {
      const unsigned long long v = static_cast<unsigned long long>(tile[c * kTileCap + i]) |
                                   (static_cast<unsigned long long>(tile[c * kTileCap + i + plane]) << 32);
      if (v) atomicAdd(q + c, v);
    }
  }
}

// Grid update of one node from its sums: velocity and mass.
struct NodeSums {
  ulonglong2 s01, s23;
};

__device__ __forceinline__ NodeSums load_sums(const unsigned long long* __restrict__ gsum, int id) {
  const ulonglong2* q = reinterpret_cast<const ulonglong2*>(gsum + 4 * static_cast<size_t>(id));
  return {q[0], q[1]};
}

__device__ __forceinline__ float4 node_from_sums(const Dev& d, const NodeSums& s, int cx, int cy, int cz, float dt) {
  const ulonglong2 s01 = s.s01, s23 = s.s23;
  const float m = __ll2float_rn(static_cast<long long>(s01.x)) * d.unit;
  const float mv[3] = {__ll2float_rn(static_cast<long long>(s01.y)) * d.unit,
                       __ll2float_rn(static_cast<long long>(s23.x)) * d.unit,
                       __ll2float_rn(static_cast<long long>(s23.y)) * d.unit};
  float v[3];
  diff::node_update(d.G, cx, cy, cz, m, mv, dt, v);
  return make_float4(v[0], v[1], v[2], m);
}

// Grid-update adjoint of one node: its velocity adjoint -> (mbar, mvbar).
__device__ __forceinline__ float4 node_adjoint(const Dev& d, const unsigned long long* __restrict__ vbar, const float4& v4,
                                               int id, int cx, int cy, int cz, float dt) {
  const unsigned long long* vb = vbar + 3 * static_cast<size_t>(id);
  const float inv_units = d.adj_scale[1];
  const float vbv[3] = {__ll2float_rn(static_cast<long long>(vb[0])) * inv_units,
                        __ll2float_rn(static_cast<long long>(vb[1])) * inv_units,
                        __ll2float_rn(static_cast<long long>(vb[2])) * inv_units};
  const float v[3] = {v4.x, v4.y, v4.z};
  float out[4];
  diff::node_update_adjoint(d.G, cx, cy, cz, v4.w, v, dt, vbv, out);
  return make_float4(out[0], out[1], out[2], out[3]);
}

// Zeroes kCh sums per node over a substep's node box, shared out over the grid's first
// `ctas` CTAs, or over all of them if the box has more nodes than those have threads.
template <int kCh>
__device__ __forceinline__ void zero_box(const Dev& d, const int* __restrict__ b, unsigned long long* __restrict__ sums,
                                         uint32_t ctas) {
  if (!sums || b[0] > b[3]) return;
  const int ex = b[3] - b[0] + 1, ey = b[4] - b[1] + 1, ez = b[5] - b[2] + 1;
  const int total = 2 * ex * ey * ez;
  if (static_cast<uint32_t>(total) > ctas * blockDim.x) ctas = gridDim.x;
  if (blockIdx.x >= ctas) return;
  for (int t = blockIdx.x * blockDim.x + threadIdx.x; t < total; t += ctas * blockDim.x) {
    const int z = t % ez, xy = t / ez, y = xy % ey, gx = xy / ey, x = gx % ex, g = gx / ex;
    unsigned long long* q =
        sums + kCh * static_cast<size_t>(diff::node_index(d.G, g, b[0] + x, b[1] + y, b[2] + z));
#pragma unroll
    for (int c = 0; c < kCh; ++c) q[c] = 0ull;
  }
}

template <int kCh>
__global__ void zero_box_kernel(Dev d, const int* __restrict__ b, unsigned long long* __restrict__ sums) {
  zero_box<kCh>(d, b, sums, gridDim.x);
}

// Deposits of the CTA's particles (per unit mass) into gsum and the merge of their
// node box into `box`.  Collective; s_box holds an empty box on entry and the tile
// zeros (both before the caller's last barrier).  A particle whose stencil leaves
// the grid is reported and deposits the nodes it has inside.
__device__ __forceinline__ void cta_deposit(const Dev& d, bool active, const Fwd<float>& f, unsigned* tile, int* s_box,
                                            unsigned long long* __restrict__ gsum, int* box) {
  int lo[3] = {0, 0, 0}, hi[3] = {0, 0, 0};
  bool inside = false;
  if (active) {
    stencil_box(f.stn, lo, hi);
    inside = box_in_grid(d.G, lo, hi);
    if (!inside) {
      atomicOr(d.status, kErrOutside);
#pragma unroll
      for (int a = 0; a < 3; ++a) {  // the part of the stencil that is in the grid
        lo[a] = min(max(lo[a], 0), d.G.n[a] - 1);
        hi[a] = min(max(hi[a], 0), d.G.n[a] - 1);
      }
    }
  }
  cta_box_merge(s_box, active, lo, hi);
  __syncthreads();
  const CtaBox b = cta_box(s_box);
  if (threadIdx.x < 3 && b.e[0] > 0 && b.e[1] > 0 && b.e[2] > 0) {
    atomicMin(box + threadIdx.x, s_box[threadIdx.x]);
    atomicMax(box + 3 + threadIdx.x, s_box[3 + threadIdx.x]);
  }
  if (active) {
    diff::particle_deposit(f, d.dx, d.inv_dx, [&](int g, int cx, int cy, int cz, float w, const float* wv) {
      if (!inside && !diff::node_in_grid(d.G, cx, cy, cz)) return;
      if (!(fabsf(wv[0]) < kMaxValue && fabsf(wv[1]) < kMaxValue && fabsf(wv[2]) < kMaxValue)) {
        atomicOr(d.status, kErrRange);
        return;
      }
      const long long v[4] = {__float2ll_rn(w * kScale), __float2ll_rn(wv[0] * kScale), __float2ll_rn(wv[1] * kScale),
                              __float2ll_rn(wv[2] * kScale)};
      if (b.nodes) {
        unsigned* q = tile + box_entry(b, g, cx, cy, cz);
#pragma unroll
        for (int c = 0; c < 4; ++c) tile_add(q + c * kTileCap, 4 * kTileCap, v[c]);
      } else {
        unsigned long long* q = gsum + 4 * diff::node_index(d.G, g, cx, cy, cz);
#pragma unroll
        for (int c = 0; c < 4; ++c) atomicAdd(q + c, static_cast<unsigned long long>(v[c]));
      }
    });
  }
  __syncthreads();
  tile_flush<4>(d, b, tile, gsum);
}

constexpr size_t kNodeTile = sizeof(float4) * kTileCap;                // 16 KB
constexpr size_t kDepositTile = sizeof(unsigned) * 2 * 4 * kTileCap;   // 32 KB
constexpr size_t kAdjointTile = sizeof(unsigned) * 2 * 3 * kTileCap;   // 24 KB
constexpr size_t kForwardSmem = kDepositTile + kNodeTile;
constexpr size_t kAdjointSmem = kAdjointTile + kNodeTile;

// AoS inputs -> SoA state; lambda / mu from log E; F = I.
__global__ void init_kernel(Dev d, const float* __restrict__ x0, const float* __restrict__ logE, float nu,
                            const uint32_t* __restrict__ perm, float* __restrict__ x, float* __restrict__ F,
                            float* __restrict__ lam, float* __restrict__ mu) {
  const uint32_t p = blockIdx.x * blockDim.x + threadIdx.x;
  if (p >= d.n) return;
  const uint32_t u = perm[p];
  for (int a = 0; a < 3; ++a) x[a * d.n + p] = x0[3 * u + a];
  for (int k = 0; k < 9; ++k) F[k * d.n + p] = (k & 3) ? 0.f : 1.f;
  const float E = expf(logE[u]);
  mu[p] = E / (2.f * (1.f + nu));
  lam[p] = E * nu / ((1.f + nu) * (1.f - 2.f * nu));
}

__global__ void __launch_bounds__(kThreads) raster_kernel(Dev d, const float* __restrict__ x, const float* __restrict__ v0,
                                                          const uint32_t* __restrict__ perm,
                                                          unsigned long long* __restrict__ gsum, int* box) {
  extern __shared__ __align__(16) unsigned tile[];
  __shared__ int s_box[6];
  const uint32_t p = blockIdx.x * blockDim.x + threadIdx.x;
  tile_zero(tile, 8 * kTileCap);
  if (threadIdx.x == 0) box_reset(s_box);
  Fwd<float> f;
  if (p < d.n) {
    const uint32_t u = perm[p];
    const float xp[3] = {x[p], x[d.n + p], x[2 * d.n + p]};
    for (int a = 0; a < 3; ++a) {
      f.xn[a] = xp[a];
      f.v[a] = v0[3 * u + a];
    }
    for (int k = 0; k < 9; ++k) f.A[k] = 0.f;
    diff::make_stencil(xp, d.inv_dx, f.stn);
  }
  __syncthreads();
  cta_deposit(d, p < d.n, f, tile, s_box, gsum, box);
}

// Every substep's box starts empty; deposits widen it.  A recomputed segment
// deposits exactly what the forward did, so its boxes are unchanged.
__global__ void box_init_kernel(int* boxes, uint32_t count) {
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < count) box_reset(boxes + 6 * i);
}

// Grid update over box b: int64 sums -> float4 (v, m); zero the sums read.  For the
// last state of a recomputed segment, which no forward substep reads.
__global__ void grid_kernel(Dev d, unsigned long long* __restrict__ gsum, const int* __restrict__ b, float dt,
                            float4* __restrict__ vel) {
  if (b[0] > b[3]) return;
  const int ex = b[3] - b[0] + 1, ey = b[4] - b[1] + 1, ez = b[5] - b[2] + 1;
  const int64_t total = 2ll * ex * ey * ez;
  for (int64_t t = blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x; t < total;
       t += static_cast<int64_t>(gridDim.x) * blockDim.x) {
    const int z = static_cast<int>(t % ez), y = static_cast<int>((t / ez) % ey);
    const int x = static_cast<int>((t / (static_cast<int64_t>(ez) * ey)) % ex);
    const int g = static_cast<int>(t / (static_cast<int64_t>(ez) * ey * ex));
    const int cx = b[0] + x, cy = b[1] + y, cz = b[2] + z;
    const int id = diff::node_index(d.G, g, cx, cy, cz);
    vel[id] = node_from_sums(d, load_sums(gsum, id), cx, cy, cz, dt);
    ulonglong2* q = reinterpret_cast<ulonglong2*>(gsum + 4 * static_cast<size_t>(id));
    q[0] = make_ulonglong2(0ull, 0ull);
    q[1] = make_ulonglong2(0ull, 0ull);
  }
}

// Node velocities of G2P: from the CTA's tile; where there is none, from the
// velocities of the substep or (sums given) from the node sums themselves, and then
// written to the tape as well.
struct VelReader {
  const Dev* d;
  const CtaBox* b;
  const float4* tile;
  float4* vel;
  const unsigned long long* sums;
  float dt;
  bool tiled, inside;  // the particle's stencil lies in the tile / in the grid
  // The nodes (g, cx, cy + i, cz + j), v[2 i + j].  All four are loaded before the first is
  // used: one after another, each behind the branches of the last one's grid update, the 16
  // loads of a particle took 4 us of a 20 us substep of a sparse cloud.
  __device__ void quad(int g, int cx, int cy, int cz, float (*v)[3]) const {
    float4 q[4];
    if (tiled) {
#pragma unroll
      for (int k = 0; k < 4; ++k) q[k] = tile[box_entry(*b, g, cx, cy + (k >> 1), cz + (k & 1))];
    } else {
      int id[4];
      bool in[4];
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        in[k] = inside || diff::node_in_grid(d->G, cx, cy + (k >> 1), cz + (k & 1));
        id[k] = in[k] ? diff::node_index(d->G, g, cx, cy + (k >> 1), cz + (k & 1)) : 0;
      }
      if (sums) {
        NodeSums s[4];
#pragma unroll
        for (int k = 0; k < 4; ++k) s[k] = load_sums(sums, id[k]);
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          q[k] = node_from_sums(*d, s[k], cx, cy + (k >> 1), cz + (k & 1), dt);
          if (in[k]) vel[id[k]] = q[k];
        }
      } else {
#pragma unroll
        for (int k = 0; k < 4; ++k) q[k] = vel[id[k]];
      }
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        if (in[k]) continue;
        atomicOr(d->status, kErrOutside);
        q[k] = make_float4(0.f, 0.f, 0.f, 0.f);
      }
    }
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      v[k][0] = q[k].x;
      v[k][1] = q[k].y;
      v[k][2] = q[k].z;
    }
  }
  __device__ void operator()(int g, int cx, int cy, int cz, float* v) const {
    float4 q;
    if (tiled) {
      q = tile[box_entry(*b, g, cx, cy, cz)];
    } else if (!inside && !diff::node_in_grid(d->G, cx, cy, cz)) {
      atomicOr(d->status, kErrOutside);
      q = make_float4(0.f, 0.f, 0.f, 0.f);
    } else {
      q = vel[diff::node_index(d->G, g, cx, cy, cz)];
    }
    v[0] = q.x;
    v[1] = q.y;
    v[2] = q.z;
  }
};

struct Svd {
  __device__ void operator()(const float* F, float* U, float* S, float* V) const { svd3(F, U, S, V); }
};

__device__ __forceinline__ void load_particle(const Dev& d, const float* x, const float* F, uint32_t p,
                                              Particle<float>& pp) {
  for (int a = 0; a < 3; ++a) pp.x[a] = x[a * d.n + p];
  for (int k = 0; k < 9; ++k) pp.F[k] = F[k * d.n + p];
}

// Forward substep of every particle: grid update and G2P at x, x and F update,
// stress, deposit at x' into gsum_out; new state to (xo, Fo).  The grid update runs
// as the CTA's node tile is filled, from gsum_in (the velocities then go to the
// tape `vel` too), or, gsum_in null, the velocities are read from `vel`.  The sums are
// triple-buffered: gsum_zero, which the previous substep read (box bzero), is zeroed
// here for the next substep's deposits.
__global__ void __launch_bounds__(kThreads) particle_kernel(
    Dev d, const float* __restrict__ x, const float* __restrict__ F, const float* __restrict__ lam,
    const float* __restrict__ mu, float4* __restrict__ vel, const unsigned long long* __restrict__ gsum_in, float dt,
    float ndt, unsigned long long* __restrict__ gsum_out, int* bnext, unsigned long long* __restrict__ gsum_zero,
    const int* __restrict__ bzero, float* __restrict__ xo, float* __restrict__ Fo) {
  extern __shared__ __align__(16) unsigned tile[];
  float4* vtile = reinterpret_cast<float4*>(tile + 8 * kTileCap);
  __shared__ int s_box[2][6];
  const uint32_t p = blockIdx.x * blockDim.x + threadIdx.x;
  if (blockIdx.x * kThreads >= d.n) {  // no particles: a CTA that only zeroes
    zero_box<4>(d, bzero, gsum_zero, particle_ctas(d));
    return;
  }
  const bool active = p < d.n;
  if (threadIdx.x < 2) box_reset(s_box[threadIdx.x]);
  __syncthreads();
  Particle<float> pp;
  int lo[3] = {0, 0, 0}, hi[3] = {0, 0, 0};
  bool inside = false;
  if (active) {
    load_particle(d, x, F, p, pp);
    diff::Stencil<float> st;
    diff::make_stencil(pp.x, d.inv_dx, st);
    stencil_box(st, lo, hi);
    inside = box_in_grid(d.G, lo, hi);
  }
  cta_box_merge(s_box[0], inside, lo, hi);
  zero_box<4>(d, bzero, gsum_zero, particle_ctas(d));
  tile_zero(tile, 8 * kTileCap);
  __syncthreads();
  const CtaBox b = cta_box(s_box[0]);
  for (int i = threadIdx.x; i < b.nodes; i += kThreads) {
    int cx, cy, cz;
    const int id = box_node(d, b, i, cx, cy, cz);
    if (gsum_in) {
      const float4 q = node_from_sums(d, load_sums(gsum_in, id), cx, cy, cz, dt);
      vtile[i] = q;
      vel[id] = q;  // every CTA that reads the node writes the same value
    } else {
      vtile[i] = vel[id];
    }
  }
  __syncthreads();
  Fwd<float> f;
  if (active) {
    float U[9], S[3], V[9];
    const VelReader vr{&d, &b, vtile, vel, gsum_in, dt, inside && b.nodes, inside};
    diff::particle_forward(pp, lam[p], mu[p], d.vol_over_mass, dt, ndt, d.dx, d.inv_dx, vr, Svd{}, f, U, S, V);
    for (int a = 0; a < 3; ++a) xo[a * d.n + p] = f.xn[a];
    for (int k = 0; k < 9; ++k) Fo[k * d.n + p] = f.Fn[k];
  }
  cta_deposit(d, active, f, tile, s_box[1], gsum_out, bnext);
}

// Adjoint of one substep for every particle.  xb / Fb hold the adjoints of the
// substep's outputs on entry and of its inputs on exit.
// The fixed-point unit of the velocity adjoint: the largest |component| of the
// incoming adjoints (x and F at the end of the rollout), then 2^40 units per it.
__global__ void adj_seed_max_kernel(uint32_t n, const float* __restrict__ xb, const float* __restrict__ Fb,
                                    float* adj_scale) {
  float m = 0.f;
  for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < 12 * n; i += gridDim.x * blockDim.x)
    m = fmaxf(m, fabsf(i < 3 * n ? xb[i] : Fb[i - 3 * n]));
  for (int o = 16; o > 0; o >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, o));
  // non-negative floats order like their bit patterns
  if ((threadIdx.x & 31) == 0 && m > 0.f) atomicMax(reinterpret_cast<unsigned*>(adj_scale + 2), __float_as_uint(m));
}

__global__ void adj_scale_kernel(float* adj_scale) {
  if (threadIdx.x == 0 && blockIdx.x == 0) {
    const float m = adj_scale[2];
    adj_scale[0] = m > 0.f ? __fdiv_rn(kAdjUnits, m) : 1.f;
    adj_scale[1] = m > 0.f ? __fdiv_rn(m, kAdjUnits) : 1.f;
  }
}

// The adjoint of the deposit at x' (xn, the state after the substep; bit for bit what
// the forward deposited at) is gathered from a CTA tile that applies the grid-update
// adjoint of the next substep as it is filled, from vbar_in and that substep's
// velocities vel_next; both null for the last substep, whose deposit nothing reads.
// The velocity adjoints go to vbar_out through a tile of exact sums.  vbar is
// triple-buffered like the forward's sums.
__global__ void __launch_bounds__(kThreads, 3) particle_adjoint_kernel(
    Dev d, const float* __restrict__ x, const float* __restrict__ F, const float* __restrict__ xn,
    const float* __restrict__ lam, const float* __restrict__ mu, float4* __restrict__ vel,
    const float4* __restrict__ vel_next, float dt, float ndt, const unsigned long long* __restrict__ vbar_in,
    float* __restrict__ xb, float* __restrict__ Fb, float* __restrict__ mub, float* __restrict__ lamb,
    unsigned long long* __restrict__ vbar_out, unsigned long long* __restrict__ vbar_zero, const int* __restrict__ bzero) {
  extern __shared__ __align__(16) unsigned tile[];
  float4* gtile = reinterpret_cast<float4*>(tile + 6 * kTileCap);
  __shared__ int s_box[2][6];
  const uint32_t p = blockIdx.x * blockDim.x + threadIdx.x;
  if (blockIdx.x * kThreads >= d.n) {  // no particles: a CTA that only zeroes
    zero_box<3>(d, bzero, vbar_zero, particle_ctas(d));
    return;
  }
  const bool active = p < d.n;
  if (threadIdx.x < 2) box_reset(s_box[threadIdx.x]);
  __syncthreads();
  // The boxes of the nodes that G2P reads at x, where the velocity adjoints go, and of
  // the deposit's at x'.
  Particle<float> pp;
  float xd[3] = {0.f, 0.f, 0.f};
  int lo[3] = {0, 0, 0}, hi[3] = {0, 0, 0}, lo2[3] = {0, 0, 0}, hi2[3] = {0, 0, 0};
  bool inside = false, inside2 = false;
  if (active) {
    load_particle(d, x, F, p, pp);
    for (int a = 0; a < 3; ++a) xd[a] = xn[a * d.n + p];
    diff::Stencil<float> st;
    diff::make_stencil(pp.x, d.inv_dx, st);
    stencil_box(st, lo, hi);
    inside = box_in_grid(d.G, lo, hi);
    diff::make_stencil(xd, d.inv_dx, st);
    stencil_box(st, lo2, hi2);
    inside2 = box_in_grid(d.G, lo2, hi2);
  }
  cta_box_merge(s_box[0], inside, lo, hi);
  cta_box_merge(s_box[1], inside2, lo2, hi2);
  zero_box<3>(d, bzero, vbar_zero, particle_ctas(d));
  tile_zero(tile, 6 * kTileCap);
  __syncthreads();
  const CtaBox b = cta_box(s_box[0]), b2 = cta_box(s_box[1]);
  if (vbar_in) {
    for (int i = threadIdx.x; i < b2.nodes; i += kThreads) {
      int cx, cy, cz;
      const int id = box_node(d, b2, i, cx, cy, cz);
      gtile[i] = node_adjoint(d, vbar_in, vel_next[id], id, cx, cy, cz, ndt);
    }
  }
  __syncthreads();
  if (active) {
    Fwd<float> f;
    float U[9], S[3], V[9];
    const VelReader vr{&d, &b, nullptr, vel, nullptr, dt, false, inside};
    diff::particle_forward(pp, lam[p], mu[p], d.vol_over_mass, dt, ndt, d.dx, d.inv_dx, vr, Svd{}, f, U, S, V, xd);
    const bool tiled2 = inside2 && b2.nodes;
    auto ga = [&](int g, int cx, int cy, int cz, float* out) {
      float4 q = make_float4(0.f, 0.f, 0.f, 0.f);
      if (vbar_in) {
        if (tiled2) {
          q = gtile[box_entry(b2, g, cx, cy, cz)];
        } else if (inside2 || diff::node_in_grid(d.G, cx, cy, cz)) {
          const int id = diff::node_index(d.G, g, cx, cy, cz);
          q = node_adjoint(d, vbar_in, vel_next[id], id, cx, cy, cz, ndt);
        }
      }
      out[0] = q.x;
      out[1] = q.y;
      out[2] = q.z;
      out[3] = q.w;
    };
    const float units = d.adj_scale[0];
    auto vs = [&](int g, int cx, int cy, int cz, const float* vb) {
      if (!inside && !diff::node_in_grid(d.G, cx, cy, cz)) return;
      long long u[3];
      bool ok = true;
#pragma unroll
      for (int c = 0; c < 3; ++c) {
        const float t = vb[c] * units;
        ok &= fabsf(t) < kAdjMaxUnits;
        u[c] = fabsf(t) < kAdjMaxUnits ? __float2ll_rn(t) : 0ll;
      }
      if (!ok) atomicOr(d.status, kErrRange);
      if (inside && b.nodes) {
        unsigned* q = tile + box_entry(b, g, cx, cy, cz);
#pragma unroll
        for (int c = 0; c < 3; ++c) tile_add(q + c * kTileCap, 3 * kTileCap, u[c]);
      } else {
        unsigned long long* q = vbar_out + 3 * static_cast<size_t>(diff::node_index(d.G, g, cx, cy, cz));
#pragma unroll
        for (int c = 0; c < 3; ++c) atomicAdd(q + c, static_cast<unsigned long long>(u[c]));
      }
    };
    float xnb[3], Fnb[9], xo[3], Fo[9];
    for (int a = 0; a < 3; ++a) xnb[a] = xb[a * d.n + p];
    for (int k = 0; k < 9; ++k) Fnb[k] = Fb[k * d.n + p];
    float mb = mub[p], lb = lamb[p];
    diff::particle_adjoint(pp, f, U, S, V, d.mass, lam[p], mu[p], d.vol_over_mass, dt, ndt, d.dx, d.inv_dx, vr, ga, vs,
                           xnb, Fnb, xo, Fo, mb, lb);
    for (int a = 0; a < 3; ++a) xb[a * d.n + p] = xo[a];
    for (int k = 0; k < 9; ++k) Fb[k * d.n + p] = Fo[k];
    mub[p] = mb;
    lamb[p] = lb;
  }
  __syncthreads();
  tile_flush<3>(d, b, tile, vbar_out);
}

// Rasterisation adjoint and the outputs: gx0 (AoS), gv0 (AoS), glogE.
__global__ void finish_kernel(Dev d, const float* __restrict__ x, const float* __restrict__ v0,
                              const unsigned long long* __restrict__ vbar, const float4* __restrict__ vel,
                              const float* __restrict__ xb,
                              const float* __restrict__ lam, const float* __restrict__ mu,
                              const float* __restrict__ mub, const float* __restrict__ lamb,
                              const uint32_t* __restrict__ perm, float* __restrict__ gx0,
                              float* __restrict__ gv0, float* __restrict__ glogE) {
  const uint32_t p = blockIdx.x * blockDim.x + threadIdx.x;
  if (p >= d.n) return;
  const float xp[3] = {x[p], x[d.n + p], x[2 * d.n + p]};
  const uint32_t u = perm[p];
  const float vp[3] = {v0[3 * u], v0[3 * u + 1], v0[3 * u + 2]};
  float xo[3] = {xb[p], xb[d.n + p], xb[2 * d.n + p]}, vo[3] = {0.f, 0.f, 0.f};
  diff::raster_adjoint(xp, vp, d.mass, d.inv_dx,
                       [&](int g, int cx, int cy, int cz, float* out) {
                         float4 q = make_float4(0.f, 0.f, 0.f, 0.f);
                         if (diff::node_in_grid(d.G, cx, cy, cz)) {
                           const int id = diff::node_index(d.G, g, cx, cy, cz);
                           q = node_adjoint(d, vbar, vel[id], id, cx, cy, cz, 0.f);
                         }
                         out[0] = q.x;
                         out[1] = q.y;
                         out[2] = q.z;
                         out[3] = q.w;
                       },
                       xo, vo);
  for (int a = 0; a < 3; ++a) {
    gx0[3 * u + a] = xo[a];
    gv0[3 * u + a] = vo[a];
  }
  glogE[u] = mub[p] * mu[p] + lamb[p] * lam[p];
}

// SoA (rollout order) <-> AoS (the caller's order) for the outputs and the incoming adjoints.
__global__ void soa_to_aos_kernel(uint32_t n, int w, const uint32_t* __restrict__ perm, const float* __restrict__ soa,
                                  float* __restrict__ aos) {
  const uint32_t p = blockIdx.x * blockDim.x + threadIdx.x;
  if (p >= n) return;
  const size_t u = perm[p];
  for (int k = 0; k < w; ++k) aos[static_cast<size_t>(w) * u + k] = soa[static_cast<size_t>(k) * n + p];
}

__global__ void aos_to_soa_kernel(uint32_t n, int w, const uint32_t* __restrict__ perm, const float* __restrict__ aos,
                                  float* __restrict__ soa) {
  const uint32_t p = blockIdx.x * blockDim.x + threadIdx.x;
  if (p >= n) return;
  const size_t u = perm[p];
  for (int k = 0; k < w; ++k) soa[static_cast<size_t>(k) * n + p] = aos[static_cast<size_t>(w) * u + k];
}

}  // namespace diffk
}  // namespace ckmpm

// ------------------------------------------------------------------ host side
struct ckmpm_diff {
  ckmpm::diffk::Dev d{};
  int device = 0;
  uint32_t nsteps = 0, every = 20, nseg = 0;
  float dt = 0.f, nu = 0.3f;
  size_t nn = 0;
  cudaStream_t stream = nullptr;
  cudaEvent_t ev_in = nullptr, ev_out = nullptr, t0 = nullptr, t1 = nullptr;
  std::vector<std::pair<void*, size_t>> allocs;
  // inputs / outputs (internal, fixed addresses for the graphs)
  float *x0 = nullptr, *v0 = nullptr, *logE = nullptr, *xT = nullptr, *FT = nullptr;
  float *gxT = nullptr, *gFT = nullptr, *gx0 = nullptr, *gv0 = nullptr, *glogE = nullptr;
  float *lam = nullptr, *mu = nullptr;
  float* xs[2] = {nullptr, nullptr};  // forward ping-pong (SoA x: 3n, F: 9n in one array of 12n)
  float* ck = nullptr;                // checkpoints: nseg x 12n
  float4* ckvel = nullptr;            // nseg x nn
  float* tape = nullptr;              // max(every - 1, 1) x 12n: substeps s0 + 1 .. s1 - 1 of a segment
  float4* tapevel = nullptr;          // every x nn; a segment's first substep has its checkpoint's, so slot 0 is free:
  float4* vel = nullptr;              // scratch node velocities (forward pass), in that slot
  unsigned long long* gsum[3] = {nullptr, nullptr, nullptr};  // substep s reads [s % 3], deposits into [(s + 1) % 3]
  int* box = nullptr;                 // (nsteps + 1) x 6
  float *xb = nullptr, *Fb = nullptr, *mub = nullptr, *lamb = nullptr;
  // Substep s's velocity adjoints: [s % 3].  In gsum's memory when every substep is a checkpoint.
  unsigned long long* vbar[3] = {nullptr, nullptr, nullptr};
  // Particle order: perm[slot] = input particle; bins and their scan, each particle's bin and place in it.
  uint32_t *perm = nullptr, *bins = nullptr, *first = nullptr, *scan = nullptr, *bin = nullptr, *rank = nullptr;
  cudaGraphExec_t gfwd = nullptr, gbwd = nullptr;
  uint64_t generation = 0;
  bool have_forward = false;
  float ms_fwd = 0.f, ms_bwd = 0.f;
  std::string err;
};

namespace {

thread_local std::string g_diff_error;

ckmpm_status dfail(ckmpm_diff* h, ckmpm_status code, const std::string& msg) {
  if (h) h->err = msg;
  else g_diff_error = msg;
  return code;
}

#define DK_CUDA(h, call)                                                                        \
  do {                                                                                          \
    cudaError_t e_ = (call);                                                                    \
    if (e_ != cudaSuccess)                                                                      \
      return dfail((h), CKMPM_ERR_CUDA, std::string(#call) + ": " + cudaGetErrorString(e_));    \
  } while (0)

template <typename T>
cudaError_t dk_alloc(ckmpm_diff* h, T** p, size_t count) {
  void* q = nullptr;
  const size_t bytes = std::max<size_t>(count, 1) * sizeof(T);
  cudaError_t e = cudaMalloc(&q, bytes);
  if (e == cudaSuccess) h->allocs.emplace_back(q, bytes);
  *p = static_cast<T*>(q);
  return e;
}

using namespace ckmpm::diffk;

unsigned blocks_for(uint32_t n) { return (n + kThreads - 1) / kThreads; }

unsigned zeroing_blocks(uint32_t n) { return std::max<unsigned>(blocks_for(n), kZeroCtas); }

int grid_ctas(const ckmpm_diff* h) {
  int sms = 148;
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, h->device);
  return sms * 8;
}

}  // namespace

extern "C" {

ckmpm_status ckmpm_diff_create(const ckmpm_scene_desc* desc, uint32_t n, float mass, float volume, float nu,
                               uint32_t nsteps, float dt, uint32_t checkpoint_every, ckmpm_diff** out) {
  if (!desc || !out) return dfail(nullptr, CKMPM_ERR_INVALID, "null argument");
  *out = nullptr;
  if (n == 0 || nsteps == 0 || checkpoint_every == 0) return dfail(nullptr, CKMPM_ERR_INVALID, "empty rollout");
  if (!(mass > 0.f) || !(volume > 0.f) || !(dt >= 0.f) || !(nu > -1.f && nu < 0.5f))
    return dfail(nullptr, CKMPM_ERR_INVALID, "bad mass, volume, dt or nu");
  if (!(desc->dx > 0.f)) return dfail(nullptr, CKMPM_ERR_INVALID, "dx must be positive");
  for (int a = 0; a < 3; ++a)
    if (desc->domain_blocks[a] < 5 || desc->domain_blocks[a] > 64)
      return dfail(nullptr, CKMPM_ERR_INVALID, "domain_blocks must be 5..64 for the dense differentiable grid");
  if (desc->boundary != CKMPM_BOUNDARY_STICKY_BLOCKS && desc->boundary != CKMPM_BOUNDARY_SLIP_FLOOR)
    return dfail(nullptr, CKMPM_ERR_INVALID, "unknown boundary kind");
  if (cudaSetDevice(desc->device) != cudaSuccess) return dfail(nullptr, CKMPM_ERR_CUDA, "cudaSetDevice failed");
  ckmpm_diff* h = new ckmpm_diff();
  auto bail = [&](ckmpm_status st) {
    g_diff_error = h->err;
    ckmpm_diff_destroy(h);
    return st;
  };
  h->device = desc->device;
  h->nsteps = nsteps;
  h->every = std::min(checkpoint_every, nsteps);
  h->nseg = (nsteps + h->every - 1) / h->every;
  h->dt = dt;
  h->nu = nu;
  Dev& d = h->d;
  for (int a = 0; a < 3; ++a) {
    d.G.nb[a] = desc->domain_blocks[a];
    d.G.n[a] = 4 * desc->domain_blocks[a];
  }
  d.G.gravity = desc->gravity;
  d.G.mass_clamp = desc->mass_clamp;
  d.G.floor_cells = desc->floor_cells;
  d.G.boundary = desc->boundary;
  d.n = n;
  d.dx = desc->dx;
  d.inv_dx = static_cast<float>(1.0 / static_cast<double>(desc->dx));
  d.mass = mass;
  d.vol_over_mass = volume / mass;
  d.unit = mass * 1.4551915228366852e-11f;  // 2^-36
  h->nn = static_cast<size_t>(2) * d.G.n[0] * d.G.n[1] * d.G.n[2];
  const size_t nn = h->nn;
  if (cudaStreamCreateWithFlags(&h->stream, cudaStreamNonBlocking) != cudaSuccess ||
      cudaEventCreateWithFlags(&h->ev_in, cudaEventDisableTiming) != cudaSuccess ||
      cudaEventCreateWithFlags(&h->ev_out, cudaEventDisableTiming) != cudaSuccess ||
      cudaEventCreate(&h->t0) != cudaSuccess || cudaEventCreate(&h->t1) != cudaSuccess)
    return bail(dfail(h, CKMPM_ERR_CUDA, "stream / event creation failed"));
  bool ok = dk_alloc(h, &d.status, 1) == cudaSuccess && dk_alloc(h, &h->x0, 3 * n) == cudaSuccess &&
            dk_alloc(h, &h->v0, 3 * n) == cudaSuccess && dk_alloc(h, &h->logE, n) == cudaSuccess &&
            dk_alloc(h, &h->xT, 3 * n) == cudaSuccess && dk_alloc(h, &h->FT, 9 * n) == cudaSuccess &&
            dk_alloc(h, &h->gxT, 3 * n) == cudaSuccess && dk_alloc(h, &h->gFT, 9 * n) == cudaSuccess &&
            dk_alloc(h, &h->gx0, 3 * n) == cudaSuccess && dk_alloc(h, &h->gv0, 3 * n) == cudaSuccess &&
            dk_alloc(h, &h->glogE, n) == cudaSuccess && dk_alloc(h, &h->lam, n) == cudaSuccess &&
            dk_alloc(h, &h->mu, n) == cudaSuccess && dk_alloc(h, &h->xs[0], 12 * n) == cudaSuccess &&
            dk_alloc(h, &h->xs[1], 12 * n) == cudaSuccess &&
            dk_alloc(h, &h->ck, static_cast<size_t>(h->nseg) * 12 * n) == cudaSuccess &&
            dk_alloc(h, &h->ckvel, static_cast<size_t>(h->nseg) * nn) == cudaSuccess &&
            dk_alloc(h, &h->tape, static_cast<size_t>(std::max<uint32_t>(h->every, 2) - 1) * 12 * n) == cudaSuccess &&
            dk_alloc(h, &h->tapevel, static_cast<size_t>(h->every) * nn) == cudaSuccess &&
            dk_alloc(h, &h->gsum[0], 4 * nn) == cudaSuccess &&
            dk_alloc(h, &h->gsum[1], 4 * nn) == cudaSuccess && dk_alloc(h, &h->gsum[2], 4 * nn) == cudaSuccess &&
            dk_alloc(h, &h->box, 6 * static_cast<size_t>(nsteps + 1)) == cudaSuccess &&
            dk_alloc(h, &h->xb, 3 * n) == cudaSuccess && dk_alloc(h, &h->Fb, 9 * n) == cudaSuccess &&
            dk_alloc(h, &h->mub, n) == cudaSuccess && dk_alloc(h, &h->lamb, n) == cudaSuccess &&
            dk_alloc(h, &h->d.adj_scale, 4) == cudaSuccess && dk_alloc(h, &h->perm, n) == cudaSuccess &&
            dk_alloc(h, &h->bin, n) == cudaSuccess && dk_alloc(h, &h->rank, n) == cudaSuccess &&
            dk_alloc(h, &h->bins, order_bins(d.G)) == cudaSuccess &&
            dk_alloc(h, &h->first, order_bins(d.G)) == cudaSuccess &&
            dk_alloc(h, &h->scan, scan_tiles(order_bins(d.G))) == cudaSuccess;
  // A backward that recomputes nothing touches no node sums, and every pass leaves them and
  // the velocity adjoints at zero: they share their memory then.
  for (int k = 0; k < 3; ++k) {
    if (h->every == 1) h->vbar[k] = h->gsum[k];
    else ok = ok && dk_alloc(h, &h->vbar[k], 3 * nn) == cudaSuccess;
  }
  h->vel = h->tapevel;
  if (!ok) return bail(dfail(h, CKMPM_ERR_CUDA, "device allocation failed"));
  // Sums and velocity adjoints start (and are always left) at zero inside every box.
  if (cudaFuncSetAttribute(reinterpret_cast<const void*>(particle_kernel), cudaFuncAttributeMaxDynamicSharedMemorySize,
                           static_cast<int>(kForwardSmem)) != cudaSuccess ||
      cudaFuncSetAttribute(reinterpret_cast<const void*>(particle_adjoint_kernel),
                           cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(kAdjointSmem)) != cudaSuccess)
    return bail(dfail(h, CKMPM_ERR_CUDA, "cudaFuncSetAttribute failed"));
  for (int k = 0; k < 3; ++k)
    if (cudaMemsetAsync(h->gsum[k], 0, 32 * nn, h->stream) != cudaSuccess ||
        (h->vbar[k] != h->gsum[k] && cudaMemsetAsync(h->vbar[k], 0, 24 * nn, h->stream) != cudaSuccess))
      return bail(dfail(h, CKMPM_ERR_CUDA, "initialisation failed"));
  if (cudaMemsetAsync(h->d.adj_scale, 0, 4 * sizeof(float), h->stream) != cudaSuccess ||
      cudaMemsetAsync(h->vel, 0, 16 * nn, h->stream) != cudaSuccess ||
      cudaStreamSynchronize(h->stream) != cudaSuccess)
    return bail(dfail(h, CKMPM_ERR_CUDA, "initialisation failed"));
  *out = h;
  return CKMPM_OK;
}

const char* ckmpm_diff_last_error(const ckmpm_diff* h) { return h ? h->err.c_str() : g_diff_error.c_str(); }

ckmpm_status ckmpm_diff_destroy(ckmpm_diff* h) {
  if (!h) return CKMPM_OK;
  cudaSetDevice(h->device);
  if (h->stream) cudaStreamSynchronize(h->stream);
  if (h->gfwd) cudaGraphExecDestroy(h->gfwd);
  if (h->gbwd) cudaGraphExecDestroy(h->gbwd);
  for (auto& p : h->allocs) cudaFree(p.first);
  if (h->ev_in) cudaEventDestroy(h->ev_in);
  if (h->ev_out) cudaEventDestroy(h->ev_out);
  if (h->t0) cudaEventDestroy(h->t0);
  if (h->t1) cudaEventDestroy(h->t1);
  if (h->stream) cudaStreamDestroy(h->stream);
  delete h;
  return CKMPM_OK;
}

}  // extern "C"

namespace {

// One forward substep s.  `sums` null: its node velocities are in vel already.
// zero_prev: the sums that substep s - 1 read are still to be zeroed.
void forward_substep(ckmpm_diff* h, uint32_t s, const float* in, float* outp, float4* vel, const unsigned long long* sums,
                     float cdt, float ndt, bool zero_prev) {
  const uint32_t n = h->d.n;
  particle_kernel<<<zeroing_blocks(n), kThreads, kForwardSmem, h->stream>>>(
      h->d, in, in + 3 * n, h->lam, h->mu, vel, sums, cdt, ndt, h->gsum[(s + 1) % 3], h->box + 6 * (s + 1),
      zero_prev ? h->gsum[(s + 2) % 3] : nullptr, h->box + 6 * (s > 0 ? s - 1 : 0), outp, outp + 3 * n);
}

// The whole forward rollout: init, rasterise, nsteps substeps; checkpoint k
// (x, F and node velocities of substep k * every) on the way; outputs xT, FT.
cudaError_t enqueue_rollout(ckmpm_diff* h) {
  const Dev& d = h->d;
  const uint32_t n = d.n;
  const size_t nn = h->nn;
  const int ctas = grid_ctas(h);
  cudaStream_t st = h->stream;
  cudaError_t e = cudaMemsetAsync(d.status, 0, sizeof(uint32_t), st);
  if (e != cudaSuccess) return e;
  // State of substep s: its checkpoint slot when it has one, else a ping-pong buffer.
  auto state = [&](uint32_t s) -> float* {
    return (s < h->nsteps && s % h->every == 0) ? h->ck + static_cast<size_t>(s / h->every) * 12 * n
                                                 : h->xs[s & 1];
  };
  // The rollout's particle order.
  const uint32_t nbins = order_bins(d.G), ntiles = scan_tiles(nbins);
  e = cudaMemsetAsync(h->bins, 0, sizeof(uint32_t) * nbins, st);
  if (e != cudaSuccess) return e;
  order_count_kernel<<<blocks_for(n), kThreads, 0, st>>>(d, h->x0, h->bins, h->bin, h->rank);
  ckmpm::scan_reduce_kernel<<<ntiles, ckmpm::kScanThreads, 0, st>>>(h->bins, nbins, h->scan);
  ckmpm::scan_sums_kernel<<<1, ckmpm::kScanThreads, 0, st>>>(h->scan, ntiles);
  ckmpm::scan_apply_kernel<<<ntiles, ckmpm::kScanThreads, 0, st>>>(h->bins, nbins, h->scan, h->first);
  order_place_kernel<<<blocks_for(n), kThreads, 0, st>>>(n, h->first, h->bin, h->rank, h->perm);
  init_kernel<<<blocks_for(n), kThreads, 0, st>>>(d, h->x0, h->logE, h->nu, h->perm, state(0), state(0) + 3 * n,
                                                  h->lam, h->mu);
  box_init_kernel<<<(h->nsteps + 1 + 127) / 128, 128, 0, st>>>(h->box, h->nsteps + 1);
  raster_kernel<<<blocks_for(n), kThreads, kDepositTile, st>>>(d, state(0), h->v0, h->perm, h->gsum[0], h->box);
  for (uint32_t s = 0; s < h->nsteps; ++s) {
    const float cdt = s == 0 ? 0.f : h->dt, ndt = h->dt;
    const bool ck = (s % h->every) == 0;
    const uint32_t k = s / h->every;
    float4* vs = ck ? h->ckvel + static_cast<size_t>(k) * nn : h->vel;
    float* in = state(s);
    float* outp = state(s + 1);
    forward_substep(h, s, in, outp, vs, h->gsum[s % 3], cdt, ndt, s > 0);
  }
  // Leave the last two substeps' sums at zero (nothing reads the last deposit).
  const uint32_t N = h->nsteps;
  zero_box_kernel<4><<<ctas, 256, 0, st>>>(d, h->box + 6 * (N - 1), h->gsum[(N - 1) % 3]);
  zero_box_kernel<4><<<ctas, 256, 0, st>>>(d, h->box + 6 * N, h->gsum[N % 3]);
  const float* fin = state(h->nsteps);
  soa_to_aos_kernel<<<blocks_for(n), kThreads, 0, st>>>(n, 3, h->perm, fin, h->xT);
  soa_to_aos_kernel<<<blocks_for(n), kThreads, 0, st>>>(n, 9, h->perm, fin + 3 * n, h->FT);
  return cudaGetLastError();
}

// The whole backward: for each segment from the last, recompute its substeps
// from the checkpoint into the tape, then run the adjoint in reverse.
cudaError_t enqueue_backward(ckmpm_diff* h) {
  const Dev& d = h->d;
  const uint32_t n = d.n;
  const size_t nn = h->nn;
  const int ctas = grid_ctas(h);
  cudaStream_t st = h->stream;
  aos_to_soa_kernel<<<blocks_for(n), kThreads, 0, st>>>(n, 3, h->perm, h->gxT, h->xb);
  aos_to_soa_kernel<<<blocks_for(n), kThreads, 0, st>>>(n, 9, h->perm, h->gFT, h->Fb);
  cudaError_t e = cudaMemsetAsync(h->d.adj_scale + 2, 0, sizeof(float), st);
  if (e != cudaSuccess) return e;
  adj_seed_max_kernel<<<ctas, 256, 0, st>>>(n, h->xb, h->Fb, h->d.adj_scale);
  adj_scale_kernel<<<1, 32, 0, st>>>(h->d.adj_scale);
  e = cudaMemsetAsync(h->mub, 0, sizeof(float) * n, st);
  if (e != cudaSuccess) return e;
  e = cudaMemsetAsync(h->lamb, 0, sizeof(float) * n, st);
  if (e != cudaSuccess) return e;
  const uint32_t N = h->nsteps;
  const float* xnext = h->xs[N & 1];   // x of the state after the substep at hand (the rollout's last state first)
  const float4* vnext = nullptr;       // node velocities of the substep after it (none after the last)
  for (int k = static_cast<int>(h->nseg) - 1; k >= 0; --k) {
    const uint32_t s0 = static_cast<uint32_t>(k) * h->every;
    const uint32_t s1 = std::min(N, s0 + h->every);
    // recompute: the segment's first state is its checkpoint, state s0 + j (j >= 1)
    // tape slot j - 1; tapevel slot j holds the node velocities of substep s0 + j
    auto statep = [&](uint32_t s) -> float* {
      return s == s0 ? h->ck + static_cast<size_t>(k) * 12 * n : h->tape + static_cast<size_t>(s - s0 - 1) * 12 * n;
    };
    auto velp = [&](uint32_t s) -> float4* {
      return s == s0 ? h->ckvel + static_cast<size_t>(k) * nn : h->tapevel + static_cast<size_t>(s - s0) * nn;
    };
    for (uint32_t s = s0; s + 1 < s1; ++s)
      forward_substep(h, s, statep(s), statep(s + 1), velp(s), s == s0 ? nullptr : h->gsum[s % 3],
                      s == 0 ? 0.f : h->dt, h->dt, s > s0 + 1);
    if (s1 - s0 > 1) {
      // The last state's velocities; this zeroes its sums, and those read before it.
      grid_kernel<<<ctas, 256, 0, st>>>(d, h->gsum[(s1 - 1) % 3], h->box + 6 * (s1 - 1), h->dt, velp(s1 - 1));
      if (s1 - s0 > 2) zero_box_kernel<4><<<ctas, 256, 0, st>>>(d, h->box + 6 * (s1 - 2), h->gsum[(s1 - 2) % 3]);
    }
    // reverse through the segment
    for (int i = static_cast<int>(s1) - 1; i >= static_cast<int>(s0); --i) {
      const uint32_t s = static_cast<uint32_t>(i);
      const float cdt = s == 0 ? 0.f : h->dt, ndt = h->dt;
      const float* in = statep(s);
      // vbar of substep s + 2, which substep s + 1 read, is zeroed here.
      particle_adjoint_kernel<<<zeroing_blocks(n), kThreads, kAdjointSmem, st>>>(
          d, in, in + 3 * n, xnext, h->lam, h->mu, velp(s), vnext, cdt, ndt, vnext ? h->vbar[(s + 1) % 3] : nullptr, h->xb,
          h->Fb, h->mub, h->lamb, h->vbar[s % 3], s + 2 < N ? h->vbar[(s + 2) % 3] : nullptr,
          h->box + 6 * std::min(s + 2, N));
      xnext = in;
      vnext = velp(s);
    }
  }
  finish_kernel<<<blocks_for(n), kThreads, 0, st>>>(d, h->ck, h->v0, h->vbar[0], h->ckvel, h->xb, h->lam, h->mu, h->mub,
                                                    h->lamb, h->perm, h->gx0, h->gv0, h->glogE);
  zero_box_kernel<3><<<ctas, 256, 0, st>>>(d, h->box, h->vbar[0]);
  if (N > 1) zero_box_kernel<3><<<ctas, 256, 0, st>>>(d, h->box + 6, h->vbar[1]);
  return cudaGetLastError();
}

cudaError_t capture(ckmpm_diff* h, bool fwd, cudaGraphExec_t* exec) {
  cudaGraph_t g = nullptr;
  cudaError_t e = cudaStreamBeginCapture(h->stream, cudaStreamCaptureModeThreadLocal);
  if (e != cudaSuccess) return e;
  e = fwd ? enqueue_rollout(h) : enqueue_backward(h);
  cudaError_t e2 = cudaStreamEndCapture(h->stream, &g);
  if (e != cudaSuccess) {
    if (g) cudaGraphDestroy(g);
    return e;
  }
  if (e2 != cudaSuccess) return e2;
  e = cudaGraphInstantiate(exec, g, 0);
  cudaGraphDestroy(g);
  return e;
}

ckmpm_status check_status(ckmpm_diff* h) {
  uint32_t s = 0;
  DK_CUDA(h, cudaMemcpyAsync(&s, h->d.status, sizeof(uint32_t), cudaMemcpyDeviceToHost, h->stream));
  DK_CUDA(h, cudaStreamSynchronize(h->stream));
  if (s & kErrOutside) return dfail(h, CKMPM_ERR_CAPACITY, "a particle's stencil left the dense grid");
  if (s & kErrRange) return dfail(h, CKMPM_ERR_NUMERIC, "out-of-range P2G contribution");
  return CKMPM_OK;
}

}  // namespace

extern "C" {

ckmpm_status ckmpm_diff_forward(ckmpm_diff* h, const float* x0, const float* v0, const float* logE, float* xT,
                                float* FT, void* cuda_stream) {
  if (!h || !x0 || !v0 || !logE) return dfail(h, CKMPM_ERR_INVALID, "null argument");
  DK_CUDA(h, cudaSetDevice(h->device));
  cudaStream_t user = static_cast<cudaStream_t>(cuda_stream);
  const uint32_t n = h->d.n;
  DK_CUDA(h, cudaEventRecord(h->ev_in, user));
  DK_CUDA(h, cudaStreamWaitEvent(h->stream, h->ev_in, 0));
  DK_CUDA(h, cudaMemcpyAsync(h->x0, x0, sizeof(float) * 3 * n, cudaMemcpyDeviceToDevice, h->stream));
  DK_CUDA(h, cudaMemcpyAsync(h->v0, v0, sizeof(float) * 3 * n, cudaMemcpyDeviceToDevice, h->stream));
  DK_CUDA(h, cudaMemcpyAsync(h->logE, logE, sizeof(float) * n, cudaMemcpyDeviceToDevice, h->stream));
  if (!h->gfwd) DK_CUDA(h, capture(h, true, &h->gfwd));
  DK_CUDA(h, cudaEventRecord(h->t0, h->stream));
  DK_CUDA(h, cudaGraphLaunch(h->gfwd, h->stream));
  DK_CUDA(h, cudaEventRecord(h->t1, h->stream));
  if (xT) DK_CUDA(h, cudaMemcpyAsync(xT, h->xT, sizeof(float) * 3 * n, cudaMemcpyDeviceToDevice, h->stream));
  if (FT) DK_CUDA(h, cudaMemcpyAsync(FT, h->FT, sizeof(float) * 9 * n, cudaMemcpyDeviceToDevice, h->stream));
  ckmpm_status st = check_status(h);
  cudaEventElapsedTime(&h->ms_fwd, h->t0, h->t1);
  if (st != CKMPM_OK) return st;
  DK_CUDA(h, cudaEventRecord(h->ev_out, h->stream));
  DK_CUDA(h, cudaStreamWaitEvent(user, h->ev_out, 0));
  h->have_forward = true;
  ++h->generation;
  return CKMPM_OK;
}

ckmpm_status ckmpm_diff_backward(ckmpm_diff* h, const float* gxT, const float* gFT, float* gx0, float* gv0,
                                 float* glogE, void* cuda_stream) {
  if (!h) return dfail(h, CKMPM_ERR_INVALID, "null argument");
  if (!h->have_forward) return dfail(h, CKMPM_ERR_INVALID, "ckmpm_diff_forward has not run");
  DK_CUDA(h, cudaSetDevice(h->device));
  cudaStream_t user = static_cast<cudaStream_t>(cuda_stream);
  const uint32_t n = h->d.n;
  DK_CUDA(h, cudaEventRecord(h->ev_in, user));
  DK_CUDA(h, cudaStreamWaitEvent(h->stream, h->ev_in, 0));
  if (gxT) DK_CUDA(h, cudaMemcpyAsync(h->gxT, gxT, sizeof(float) * 3 * n, cudaMemcpyDeviceToDevice, h->stream));
  else DK_CUDA(h, cudaMemsetAsync(h->gxT, 0, sizeof(float) * 3 * n, h->stream));
  if (gFT) DK_CUDA(h, cudaMemcpyAsync(h->gFT, gFT, sizeof(float) * 9 * n, cudaMemcpyDeviceToDevice, h->stream));
  else DK_CUDA(h, cudaMemsetAsync(h->gFT, 0, sizeof(float) * 9 * n, h->stream));
  if (!h->gbwd) DK_CUDA(h, capture(h, false, &h->gbwd));
  DK_CUDA(h, cudaEventRecord(h->t0, h->stream));
  DK_CUDA(h, cudaGraphLaunch(h->gbwd, h->stream));
  DK_CUDA(h, cudaEventRecord(h->t1, h->stream));
  if (gx0) DK_CUDA(h, cudaMemcpyAsync(gx0, h->gx0, sizeof(float) * 3 * n, cudaMemcpyDeviceToDevice, h->stream));
  if (gv0) DK_CUDA(h, cudaMemcpyAsync(gv0, h->gv0, sizeof(float) * 3 * n, cudaMemcpyDeviceToDevice, h->stream));
  if (glogE) DK_CUDA(h, cudaMemcpyAsync(glogE, h->glogE, sizeof(float) * n, cudaMemcpyDeviceToDevice, h->stream));
  ckmpm_status st = check_status(h);
  cudaEventElapsedTime(&h->ms_bwd, h->t0, h->t1);
  if (st != CKMPM_OK) return st;
  DK_CUDA(h, cudaEventRecord(h->ev_out, h->stream));
  DK_CUDA(h, cudaStreamWaitEvent(user, h->ev_out, 0));
  return CKMPM_OK;
}

ckmpm_status ckmpm_diff_timing(ckmpm_diff* h, float* ms_out2, uint64_t* generation) {
  if (!h || !ms_out2) return dfail(h, CKMPM_ERR_INVALID, "null argument");
  ms_out2[0] = h->ms_fwd;
  ms_out2[1] = h->ms_bwd;
  if (generation) *generation = h->generation;
  return CKMPM_OK;
}

}  // extern "C"
