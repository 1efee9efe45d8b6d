// k_grid.cu -- grid stages of the FLIP step on the sparse 8^3 brick layout.
//
// P2G (FlipSimulation::TransferParticlesToGrid, common/flip_simulation.cc:
// 809-923, with ScatterWeight<D> :927-1009) runs in two passes, each particle
// visited once.  Pass 1 (one CTA per particle leaf) splats the leaf's
// particles into a 10^3 node block (the leaf's nodes and the layer around
// them, the halo the reference buffers per leaf) in shared-memory fixed-point
// accumulators and writes the block out.  Pass 2 (one CTA per grid leaf)
// sums, per node, its own block entry and the neighbour blocks that cover it,
// and writes each node exactly once: no global atomics.  The fused pass 2
// folds the rest of the per-node work of the step into that write:
// normalisation with the 1e-5 cut, ApplyBoundaryConditions,
// SaveGridVelocities, AddGravity and the second ApplyBoundaryConditions.
//
// The remaining kernels restate ComputeDivergence (:716-736),
// UpdateVelocityFromPressure (:739-778) fused with GetVelocityUpdate
// (:781-801) and the CFL max (:460-488), and the per-stage variants.
// All arithmetic that the reference does in float is done with explicit
// round-to-nearest intrinsics so that nvcc cannot contract it into FMAs.
#include <cstring>
#include <type_traits>

#include "fsim_internal.cuh"

namespace fsim {

namespace {

struct GridArgs {
  const float* part;
  int64_t cap;
  const uint32_t* keys;
  const int32_t* leaf_id;
  const int32_t* nbr;
  const uint2* cell_range;
  const uint2* leaf_range;
  int n_pleaf, n_gleaf;
  int check_dead;
  LeafMap lm;
  SolidDesc sd;
  float* vel;
  float* vold;
  float* weight;
  uint32_t* vel_on;
  uint32_t* vold_on;
  int8_t* marker;
  const float* pres;
  float* div;
  float dt, fx, fy, fz;
  int64_t* cnt;
  unsigned long long* p2g_nodes;  // P2G pass 1 output: [particle leaf][6][1000]
  uint32_t* p2g_touch;            // [particle leaf][32] touched bits of the 1000 nodes
  uint32_t* p2g_low;              // [0]: count; then slot * 1536 + D * 512 + voxel of the
                                  // low-weight faces pass 2 leaves to k_p2g_low
  const unsigned* gave_up;        // fused pressure update: not 0 when the solve in flight timed out
};

__device__ __forceinline__ void origin_of(const GridArgs& a, int s, int o[3]) {
  int lx, ly, lz;
  leaf_coords(a.lm, uint32_t(a.leaf_id[s]), lx, ly, lz);
  o[0] = lx * 8; o[1] = ly * 8; o[2] = lz * 8;
}

__device__ __forceinline__ int nb_index(int dx, int dy, int dz) {
  return (dx + 1) * 9 + (dy + 1) * 3 + (dz + 1);
}

// neighbour-leaf direction of local coordinate t in [-1, 8]
__device__ __forceinline__ int side(int t) { return t < 0 ? -1 : (t > 7 ? 1 : 0); }

__device__ __forceinline__ bool in_box(const int n[3], int i, int j, int k) {
  return i >= 0 && j >= 0 && k >= 0 && i < n[0] && j < n[1] && k < n[2];
}

// P2G sums are accumulated in 64-bit fixed point (2^-32 units): integer
// atomics commute, so the sums -- and every step -- are bitwise reproducible
// whatever order the CTA's threads add in.  Each float term w*u (and w) is
// converted exactly up to 2^-33; the result is then the correctly rounded
// float of the exact sum of the terms.  Range: |sum| < 2^31 per face.
constexpr float kFixScale = 4294967296.0f;  // 2^32
__device__ __forceinline__ unsigned long long to_fix(float x) {
  return static_cast<unsigned long long>(__float2ll_rn(__fmul_rn(x, kFixScale)));
}
// The float nearest the fixed-point value (one rounding; the 2^-32 scaling is
// exact for the sums a grid can hold).
__device__ __forceinline__ float from_fix(unsigned long long v) {
  return __fmul_rn(__ll2float_rn(static_cast<long long>(v)), 1.0f / 4294967296.0f);
}

// P2G in two passes, each particle visited once.
//
// Pass 1 (k_p2g_cells, one CTA per particle leaf): each thread takes whole
// cells of the leaf.  Per component D the particles of a cell reach an
// 18-node box (3 node positions on each tangential axis -- the stencil starts
// at the cell or one below it, by the side of the cell centre the particle is
// on -- and 2 on the normal axis); the thread sums the cell's particles into
// that box in registers, in list order, and adds each reached node into the
// CTA's 10^3 node block (the leaf's 8^3 nodes and the one-node layer around
// them) with one fixed-point shared atomic.  The block is written out per
// leaf: nodes[6][1000] (value sums for D = 0..2, then weight sums) and 1000
// touched bits.
//
// Pass 2 (k_p2g_nodes, one CTA per grid leaf): each node adds its own leaf's
// entry and the entries of the neighbour particle leaves whose outer layer
// covers it (a face node 1, an edge node 3, a corner node 7), then
// normalises.  Fixed-point sums are exact, so the result does not depend on
// which pass or CTA added a term: it equals the one-pass sum over all cells.
constexpr int kNodeBlock = 1000;  // 10^3 node positions, local coordinates -1..8

__device__ __forceinline__ int node_index(int li, int lj, int lk) {
  return ((li + 1) * 10 + (lj + 1)) * 10 + (lk + 1);
}

// Bits t = (i * e1 + j) * e2 + k of a component-D box (extent 2 on axis D,
// 3 on the others) whose coordinate on axis ax is in the position set m.
// A particle reaches the box nodes in the AND of its per-axis sets.
__host__ __device__ constexpr unsigned box_axis_mask(int D, int ax, unsigned m) {
  unsigned r = 0u;
  const int e0 = D == 0 ? 2 : 3, e1 = D == 1 ? 2 : 3, e2 = D == 2 ? 2 : 3;
  for (int i = 0; i < e0; ++i)
    for (int j = 0; j < e1; ++j)
      for (int k = 0; k < e2; ++k) {
        const int c = ax == 0 ? i : (ax == 1 ? j : k);
        if ((m >> c) & 1u) r |= 1u << ((i * e1 + j) * e2 + k);
      }
  return r;
}

// A term x of a node sum as two 32-bit integers, hi 2^27 + lo = round(x 2^32)
// (the same integer as to_fix(x), ties included): hi = round(x 2^5) from the
// low mantissa bits of x + 1.5 2^18, the rest of x exactly, lo = round(rest
// 2^32).  |x| < kPieceMax; 18 terms of a node then keep both sums below 2^31.
constexpr float kPieceMax = 65536.0f;
__device__ __forceinline__ void to_pieces(float x, int& hi, int& lo) {
  constexpr float kMagic = 393216.0f;  // 1.5 * 2^18: its last bit is 2^-5
  const float t = __fadd_rn(x, kMagic);
  hi = __float_as_int(t) - __float_as_int(kMagic);
  lo = __float2int_rn(__fmul_rn(__fsub_rn(x, __fsub_rn(t, kMagic)), kFixScale));
}

// Node sums of one component of the CTA's cells, added into shared memory.
// WIDE: 64-bit atomics (any |x| < 2^31); otherwise the two pieces of a term
// are added by one 32-bit atomic each, which shared memory has in hardware
// (its 64-bit addition is not one; with it the 256^3 dam break's pass took
// 1,065 us, 707 with the pieces, 164 and 111 at 128^3, the same bits; what
// bounds it now is issue, the 18 node sums of each particle first of all).
// Returns whether a term was too large for the pieces.
template <int D, bool WIDE>
__device__ __forceinline__ bool splat_cell(const GridArgs& a, const uint2 rg, const int cl[3],
                                           const int g[3], unsigned long long* sv,
                                           unsigned long long* sw, uint8_t* touched) {
  const float* px = a.part;
  const int64_t cap = a.cap;
  // box extents: 3 on the tangential axes, 2 on the normal axis D
  constexpr int e0 = D == 0 ? 2 : 3, e1 = D == 1 ? 2 : 3, e2 = D == 2 ? 2 : 3;
  float am[18], aw[18];
#pragma unroll
  for (int t = 0; t < 18; ++t) { am[t] = 0.f; aw[t] = 0.f; }
  unsigned reach = 0u;  // box nodes some particle's 8-node stencil includes
  for (uint32_t q = rg.x; q < rg.y; ++q) {
    if (a.check_dead && a.keys[q] == kDeadKey) continue;
    const float uD = px[(3 + D) * cap + q];
    float w1[3][3];   // per-axis weights over the box positions
    unsigned m1[3];   // per-axis reached positions
#pragma unroll
    for (int ax = 0; ax < 3; ++ax) {
      const float pa = px[ax * cap + q];
      const float ga = float(g[ax]);
      if (ax == D) {
        const float x = __fsub_rn(pa, ga);
        w1[ax][0] = __fsub_rn(1.0f, x); w1[ax][1] = x; w1[ax][2] = 0.f;
        m1[ax] = 3u;
      } else {
        const float lo = __fadd_rn(ga, 0.5f);
        if (pa < lo) {  // stencil starts one below the cell
          const float f = __fsub_rn(pa, __fsub_rn(lo, 1.0f));
          w1[ax][0] = __fsub_rn(1.0f, f); w1[ax][1] = f; w1[ax][2] = 0.f;
          m1[ax] = 3u;
        } else {
          const float f = __fsub_rn(pa, lo);
          w1[ax][0] = 0.f; w1[ax][1] = __fsub_rn(1.0f, f); w1[ax][2] = f;
          m1[ax] = 6u;
        }
      }
    }
#pragma unroll
    for (int i = 0; i < e0; ++i) {
#pragma unroll
      for (int j = 0; j < e1; ++j) {
        const float wij = __fmul_rn(w1[0][i], w1[1][j]);
#pragma unroll
        for (int k = 0; k < e2; ++k) {
          const int t = (i * e1 + j) * e2 + k;
          const float ww = __fmul_rn(wij, w1[2][k]);
          am[t] = __fadd_rn(am[t], __fmul_rn(ww, uD));
          aw[t] = __fadd_rn(aw[t], ww);
        }
      }
    }
    unsigned rp = box_axis_mask(D, D, 3u);  // every position on the normal axis
#pragma unroll
    for (int ax = 0; ax < 3; ++ax) {
      if (ax == D) continue;
      rp &= m1[ax] == 3u ? box_axis_mask(D, ax, 3u) : box_axis_mask(D, ax, 6u);
    }
    reach |= rp;
  }
  // flush the reached box nodes (local coordinates -1..8)
  const int b0 = cl[0] - (D == 0 ? 0 : 1), b1 = cl[1] - (D == 1 ? 0 : 1),
            b2 = cl[2] - (D == 2 ? 0 : 1);
  bool wide = false;
#pragma unroll
  for (int i = 0; i < e0; ++i) {
#pragma unroll
    for (int j = 0; j < e1; ++j) {
#pragma unroll
      for (int k = 0; k < e2; ++k) {
        const int t = (i * e1 + j) * e2 + k;
        if (!((reach >> t) & 1u)) continue;
        const int o = node_index(b0 + i, b1 + j, b2 + k);
        if (WIDE) {
          atomicAdd(&sv[o], to_fix(am[t]));
          atomicAdd(&sw[o], to_fix(aw[t]));
        } else {
          int hi, lo;
          to_pieces(am[t], hi, lo);
          wide = wide || !(fabsf(am[t]) < kPieceMax) || !(aw[t] < kPieceMax);
          int* v = reinterpret_cast<int*>(sv);
          atomicAdd(&v[o], hi);
          atomicAdd(&v[kNodeBlock + o], lo);
          to_pieces(aw[t], hi, lo);
          int* w = reinterpret_cast<int*>(sw);
          atomicAdd(&w[o], hi);
          atomicAdd(&w[kNodeBlock + o], lo);
        }
        touched[o] = 1;
      }
    }
  }
  return wide;
}

template <int D, bool WIDE, int NT>
__device__ __forceinline__ bool splat_leaf(const GridArgs& a, int s, const int org[3],
                                           unsigned long long* sv, unsigned long long* sw,
                                           uint8_t* touched) {
  bool wide = false;
  for (int c = threadIdx.x; c < 512; c += NT) {
    const int cl[3] = {c >> 6, (c >> 3) & 7, c & 7};
    const uint2 rg = a.cell_range[int64_t(s) * 512 + c];
    if (rg.x >= rg.y) continue;
    const int g[3] = {org[0] + cl[0], org[1] + cl[1], org[2] + cl[2]};
    wide = splat_cell<D, WIDE>(a, rg, cl, g, sv, sw, touched) || wide;
  }
  return wide;
}

// ND = 3: one CTA per particle leaf takes the three components in turn.
// ND = 1: a CTA per leaf and component (512 threads, a cell each; the touched
// bits of the three CTAs are combined by atomics): launches of few leaves,
// where a CTA's serial work is the kernel's time.
template <int ND, int NT>
__global__ void __launch_bounds__(NT) k_p2g_cells(const __grid_constant__ GridArgs a) {
  __shared__ unsigned long long sv[ND][kNodeBlock];
  __shared__ unsigned long long sw[ND][kNodeBlock];
  __shared__ uint8_t touched[1024];
  const int s = ND == 3 ? int(blockIdx.x) : int(blockIdx.x / 3u);  // particle leaf
  const int tid = threadIdx.x;
  const int d0 = ND == 3 ? 0 : int(blockIdx.x % 3u);
  int org[3];
  origin_of(a, s, org);
  auto clear = [&]() {
    for (int v = tid; v < kNodeBlock; v += NT) {
#pragma unroll
      for (int d = 0; d < ND; ++d) sv[d][v] = sw[d][v] = 0ull;
    }
  };
  auto splat = [&](auto wide_tag) {
    constexpr bool kWide = decltype(wide_tag)::value;
    bool wide = false;
    if (ND == 3 || d0 == 0) wide = splat_leaf<0, kWide, NT>(a, s, org, sv[0], sw[0], touched) || wide;
    if (ND == 3 || d0 == 1)
      wide = splat_leaf<1, kWide, NT>(a, s, org, sv[ND == 3 ? 1 : 0], sw[ND == 3 ? 1 : 0], touched) || wide;
    if (ND == 3 || d0 == 2)
      wide = splat_leaf<2, kWide, NT>(a, s, org, sv[ND == 3 ? 2 : 0], sw[ND == 3 ? 2 : 0], touched) || wide;
    return wide;
  };
  clear();
  for (int v = tid; v < 1024; v += NT) touched[v] = 0;
  __syncthreads();
  const bool wide = __syncthreads_or(splat(std::false_type()));
  if (wide) {  // a term of 65,536 or more: the same sums with 64-bit atomics
    clear();
    __syncthreads();
    splat(std::true_type());
    __syncthreads();
  }
  auto node = [&](const unsigned long long* sums, int v) {
    if (wide) return sums[v];
    const int* p = reinterpret_cast<const int*>(sums);
    return static_cast<unsigned long long>(static_cast<long long>(p[v]) * (1ll << 27) +
                                           p[kNodeBlock + v]);
  };
  unsigned long long* out = a.p2g_nodes + int64_t(s) * 6 * kNodeBlock;
  for (int v = tid; v < kNodeBlock; v += NT) {
#pragma unroll
    for (int d = 0; d < ND; ++d) {
      out[(d0 + d) * kNodeBlock + v] = node(sv[d], v);
      out[(3 + d0 + d) * kNodeBlock + v] = node(sw[d], v);
    }
  }
  for (int v = tid; v < 1024; v += NT) {
    const unsigned bits = __ballot_sync(0xffffffffu, touched[v] != 0);
    if ((tid & 31) == 0) {
      uint32_t* t = a.p2g_touch + int64_t(s) * 32 + (v >> 5);
      if (ND == 3)
        *t = bits;
      else
        atomicOr(t, bits);
    }
  }
}

// Faces whose fixed-point weight sum is below kLowWeight are summed again
// exactly as the reference sums them.  Fixed point has absolute resolution
// (2^-33 per cell term), which is a relative error of up to 1e-4 in the
// weight, and more in v = sum(w u) / sum(w), where the total weight is near
// the 1e-5 normalisation cut; the reference's float sums are relative.  Pass
// 2 lists those faces and k_p2g_low re-sums them, one thread per face, so
// pass 2 keeps its registers and occupancy.
constexpr float kLowWeight = 1e-3f;

// The reference's float sums of component D at node g: ScatterWeight's
// weights (common/flip_simulation.cc:976-990, differences of products) and
// its order -- each particle leaf (in OpenVDB leaf order) sums its particles
// in list order into its halo buffer (:853-868), and the buffers are added
// into the grid leaf by leaf (:870-890).  Leaves of slot s's neighbourhood
// only: a node of slot s is reached from cells within one cell of it.
// The whole warp takes one node: a lane per cell first (at most 18, in
// visiting order), then a lane per particle forms the terms, and only the
// float additions run in sequence.
__device__ __forceinline__ void ref_node_sums(const GridArgs& a, const int* nb, int s, int D,
                                              const int g[3], uint4* cells, float& tm, float& tw) {
  const int lane = threadIdx.x & 31;
  int sl[3];
  leaf_coords(a.lm, uint32_t(a.leaf_id[s]), sl[0], sl[1], sl[2]);
  // cells that reach node g: c_D in {g_D - 1, g_D}, the others in g +- 1;
  // lane L < 18 takes one of them
  int c[3], leaf[3];
  {
    int r = lane;
#pragma unroll
    for (int ax = 2; ax >= 0; --ax) {
      const int e = ax == D ? 2 : 3;
      c[ax] = g[ax] - 1 + r % e;
      r /= e;
      leaf[ax] = fdiv(c[ax], 8);
    }
  }
  uint2 rg = make_uint2(0u, 0u);
  uint32_t id = 0xFFFFFFFFu;  // no particles there
  if (lane < 18) {
    const int dx = leaf[0] - sl[0], dy = leaf[1] - sl[1], dz = leaf[2] - sl[2];
    if (dx >= -1 && dx <= 1 && dy >= -1 && dy <= 1 && dz >= -1 && dz <= 1) {
      const int ns = nb[nb_index(dx, dy, dz)];
      if (ns >= 0 && ns < a.n_pleaf) {
        rg = a.cell_range[int64_t(ns) * 512 + (((c[0] & 7) << 6) | ((c[1] & 7) << 3) | (c[2] & 7))];
        if (rg.y > rg.x) id = uint32_t(a.leaf_id[ns]);
      }
    }
  }
  // the cells in visiting order (leaf by leaf in OpenVDB order, within a leaf
  // as the lanes have them), and the particles before each
  int rank = lane < 18 ? 0 : lane;
  for (int l = 0; l < 18; ++l) {
    const uint32_t oid = __shfl_sync(0xffffffffu, id, l);
    if (lane < 18 && (oid < id || (oid == id && l < lane))) ++rank;
  }
  __syncwarp();  // the previous node's reads of the cells
  cells[rank] = make_uint4(rg.x, id == 0xFFFFFFFFu ? 0u : rg.y - rg.x, id,
                           uint32_t((c[0] - g[0] + 1) | ((c[1] - g[1] + 1) << 2) |
                                    ((c[2] - g[2] + 1) << 4)));
  __syncwarp();
  const int np = lane < 18 ? int(cells[lane].y) : 0;
  int upto = np;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int t = __shfl_up_sync(0xffffffffu, upto, o);
    if (lane >= o) upto += t;
  }
  const int total = __shfl_sync(0xffffffffu, upto, 31);
  const int before = upto - np;
  const float* px = a.part;
  const int64_t cap = a.cap;
  float Tm = 0.f, Tw = 0.f, Bm = 0.f, Bw = 0.f;
  uint32_t cur = 0xFFFFFFFFu;  // leaf being summed into Bm, Bw
  bool touched = false;
  for (int p0 = 0; p0 < total; p0 += 32) {
    // the lane's particle, number p0 + lane: in the last cell that starts at or before it
    const int mine = p0 + lane;
    int cell = 0;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      const int b = __shfl_sync(0xffffffffu, before, min(cell + o, 31));
      if (cell + o < 18 && b <= mine) cell += o;
    }
    const int start = __shfl_sync(0xffffffffu, before, cell);
    const uint4 ce = cells[cell];
    const uint32_t q = ce.x + uint32_t(mine - start), pid = ce.z;
    const int pc[3] = {g[0] - 1 + int(ce.w & 3u), g[1] - 1 + int((ce.w >> 2) & 3u),
                       g[2] - 1 + int((ce.w >> 4) & 3u)};
    bool reach = mine < total && !(a.check_dead && a.keys[q] == kDeadKey);
    float wu = 0.f, w = 0.f;
    if (reach) {
      float f[3];
      int corner[3];
#pragma unroll
      for (int ax = 0; ax < 3; ++ax) {
        const float pa = px[ax * cap + q];
        float lo = float(pc[ax]);
        int st = pc[ax];
        if (ax != D) {
          lo = __fadd_rn(lo, 0.5f);
          if (pa < lo) { lo = __fsub_rn(lo, 1.0f); st -= 1; }
        }
        f[ax] = __fsub_rn(pa, lo);
        corner[ax] = g[ax] - st;
        reach = reach && (corner[ax] == 0 || corner[ax] == 1);
      }
      const float x = f[0], y = f[1], z = f[2];
      const float xy = __fmul_rn(x, y), yz = __fmul_rn(y, z), xz = __fmul_rn(z, x);
      const float xyz = __fmul_rn(xy, z);
      const float w110 = __fsub_rn(xy, xyz), w101 = __fsub_rn(xz, xyz);
      const float w001 = __fsub_rn(__fsub_rn(z, yz), w101);
      switch ((corner[0] << 2) | (corner[1] << 1) | corner[2]) {
        case 7: w = xyz; break;
        case 6: w = w110; break;
        case 5: w = w101; break;
        case 4: w = __fsub_rn(__fsub_rn(x, xz), w110); break;
        case 3: w = __fsub_rn(yz, xyz); break;
        case 2: w = __fsub_rn(__fsub_rn(y, yz), w110); break;
        case 1: w = w001; break;
        default: w = __fsub_rn(__fadd_rn(__fsub_rn(__fsub_rn(1.0f, x), y), xy), w001);
      }
      wu = __fmul_rn(w, px[(3 + D) * cap + q]);
    }
    // the additions, in order (every lane alike)
    for (unsigned todo = __ballot_sync(0xffffffffu, reach); todo != 0u; todo &= todo - 1u) {
      const int l = __ffs(int(todo)) - 1;
      const uint32_t lid = __shfl_sync(0xffffffffu, pid, l);
      const float am = __shfl_sync(0xffffffffu, wu, l), aw = __shfl_sync(0xffffffffu, w, l);
      if (lid != cur) {
        if (touched) {
          Tm = __fadd_rn(Tm, Bm);
          Tw = __fadd_rn(Tw, Bw);
        }
        cur = lid;
        touched = true;
        Bm = Bw = 0.f;
      }
      Bm = __fadd_rn(Bm, am);
      Bw = __fadd_rn(Bw, aw);
    }
  }
  if (touched) {
    Tm = __fadd_rn(Tm, Bm);
    Tw = __fadd_rn(Tw, Bw);
  }
  tm = Tm;
  tw = Tw;
}

// Node sums of one neighbour block (zero when the block does not cover it).
struct NodeSums {
  unsigned long long v[3], w[3];
  uint32_t on;
};
__device__ __forceinline__ void node_sums(const GridArgs& a, int ns, int o, bool use, NodeSums& q) {
  const unsigned long long* blk = a.p2g_nodes + int64_t(use ? ns : 0) * 6 * kNodeBlock + o;
#pragma unroll
  for (int D = 0; D < 3; ++D) {
    q.v[D] = use ? blk[D * kNodeBlock] : 0ull;
    q.w[D] = use ? blk[(3 + D) * kNodeBlock] : 0ull;
  }
  q.on = use ? (a.p2g_touch[int64_t(ns) * 32 + (o >> 5)] >> (o & 31)) & 1u : 0u;
}
__device__ __forceinline__ void node_add(NodeSums& t, const NodeSums& q) {
#pragma unroll
  for (int D = 0; D < 3; ++D) {
    t.v[D] += q.v[D];
    t.w[D] += q.w[D];
  }
  t.on |= q.on;
}

// A thread's node takes its own leaf's sums and those of the neighbours whose
// outer layer covers it: in each axis one side at most (e), so eight blocks at
// most, and the x side is the same for a whole warp.  The loads of two blocks
// are issued together (integer sums: their order does not matter).  Bound by
// latency, so by warps in flight and short CTAs: a quarter leaf per CTA of 64
// registers takes 8.2 us at 156 leaves, 33 at 128^3 and 156 / 280 (plain /
// fused) at 256^3; a whole leaf 8.2, -, 201 / 317; all four blocks of an x
// side at once 10, -, 333 / 451; the loop over neighbours before, one load
// after another for two nodes per thread, 13.6, 38.6, 187 / 335.
constexpr int kNodeThreads = 128;
template <bool FUSED>
__global__ void __launch_bounds__(kNodeThreads, 8) k_p2g_nodes(const __grid_constant__ GridArgs a) {
  __shared__ int nb[27];
  const int s = blockIdx.x / (512 / kNodeThreads);  // grid leaf
  const int v = threadIdx.x + int(blockIdx.x % (512 / kNodeThreads)) * kNodeThreads;
  if (threadIdx.x < 27) nb[threadIdx.x] = a.nbr[int64_t(s) * 27 + threadIdx.x];
  __syncthreads();
  int org[3];
  origin_of(a, s, org);
  const int x = v >> 6, y = (v >> 3) & 7, z = v & 7;
  const int g[3] = {org[0] + x, org[1] + y, org[2] + z};
  const int e[3] = {x == 0 ? -1 : (x == 7 ? 1 : 0), y == 0 ? -1 : (y == 7 ? 1 : 0),
                    z == 0 ? -1 : (z == 7 ? 1 : 0)};
  NodeSums sum = {};
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    const int dx = h ? e[0] : 0;
    if (h && dx == 0) break;  // the same for the whole warp
#pragma unroll
    for (int c0 = 0; c0 < 4; c0 += 2) {
      NodeSums q[2];
#pragma unroll
      for (int c = c0; c < c0 + 2; ++c) {
        const int dy = (c & 2) ? e[1] : 0, dz = (c & 1) ? e[2] : 0;
        const int ns = nb[nb_index(dx, dy, dz)];
        const bool use = ns >= 0 && ns < a.n_pleaf && (!(c & 2) || dy != 0) && (!(c & 1) || dz != 0);
        node_sums(a, ns, node_index(x - 8 * dx, y - 8 * dy, z - 8 * dz), use, q[c - c0]);
      }
#pragma unroll
      for (int c = 0; c < 2; ++c) node_add(sum, q[c]);
    }
  }
  const unsigned long long (&sv)[3] = sum.v, (&sw)[3] = sum.w;
  const bool on = sum.on != 0u;
  float* vel = a.vel + int64_t(s) * 1536;
  float val[3];
  float wsum[3];
#pragma unroll
  for (int D = 0; D < 3; ++D) {
    const float ws = from_fix(sw[D]);
    const float ms = from_fix(sv[D]);
    if (on && ws < kLowWeight)  // re-summed by k_p2g_low, which rewrites this face
      a.p2g_low[1 + atomicAdd(a.p2g_low, 1u)] = unsigned(s) * 1536u + unsigned(D * 512 + v);
    wsum[D] = ws;
    // THRESH is a double literal in the reference: float ws < 1e-5 (double)
    // is ws <= 1e-5f
    val[D] = on ? ((ws <= 1e-5f) ? 0.f : __fdiv_rn(ms, ws)) : 0.f;
  }
  // marker: FLUID for in-box cells holding particles
  bool has = false;
  if (s < a.n_pleaf) {
    const uint2 rg = a.cell_range[int64_t(s) * 512 + v];
    has = rg.y > rg.x;
  }
  int m = (has && in_box(a.lm.n, g[0], g[1], g[2])) ? FSIM_FLUID : FSIM_AIR;
  const unsigned ball = __ballot_sync(0xffffffffu, on);
  if (FUSED) {
    const bool sc = is_solid(a.sd, g[0], g[1], g[2]);
    if (sc) m = FSIM_SOLID;
    bool zero[3];
    zero[0] = sc != is_solid(a.sd, g[0] - 1, g[1], g[2]);
    zero[1] = sc != is_solid(a.sd, g[0], g[1] - 1, g[2]);
    zero[2] = sc != is_solid(a.sd, g[0], g[1], g[2] - 1);
    float* vold = a.vold + int64_t(s) * 1536;
    const float gf[3] = {__fmul_rn(a.dt, a.fx), __fmul_rn(a.dt, a.fy), __fmul_rn(a.dt, a.fz)};
#pragma unroll
    for (int D = 0; D < 3; ++D) {
      float vv = val[D];
      if (on && zero[D]) vv = 0.f;                 // ApplyBoundaryConditions
      vold[D * 512 + v] = vv;                      // SaveGridVelocities
      if (on) vv = (D == 1) ? __fsub_rn(vv, gf[1]) : __fadd_rn(vv, gf[D]);  // AddGravity
      if (on && zero[D]) vv = 0.f;                 // ApplyBoundaryConditions
      vel[D * 512 + v] = vv;
    }
    if ((threadIdx.x & 31) == 0) {
      a.vold_on[int64_t(s) * 16 + (v >> 5)] = ball;
    }
  } else {
    float* wt = a.weight + int64_t(s) * 1536;
#pragma unroll
    for (int D = 0; D < 3; ++D) {
      vel[D * 512 + v] = val[D];
      wt[D * 512 + v] = on ? wsum[D] : 0.f;
    }
    // ClearGridData left the saved velocity empty
    if ((threadIdx.x & 31) == 0) a.vold_on[int64_t(s) * 16 + (v >> 5)] = 0u;
  }
  if ((threadIdx.x & 31) == 0) a.vel_on[int64_t(s) * 16 + (v >> 5)] = ball;
  a.marker[int64_t(s) * 512 + v] = int8_t(m);
}

// The low-weight faces pass 2 listed: the reference's float sums
// (ref_node_sums), normalisation with the 1e-5 cut, and for the fused step
// the rest of pass 2's per-face work (BC, SaveGridVelocities, AddGravity,
// BC), one warp per face.  The faces are independent, so the list's order does
// not matter.  A thread per face walked up to 18 cells' particles one after
// the other, a latency chain: 25 us at 32^3, 33 at 64^3, 38 at 128^3 (few
// listed faces) against 10, 14 and 23 with a warp; on the 256^3 dam break,
// whose list fills the GPU, 101 against 137.
template <bool FUSED>
__global__ void __launch_bounds__(128) k_p2g_low(const __grid_constant__ GridArgs a) {
  __shared__ uint4 cells[4][32];  // per warp: a node's cells in visiting order
  const unsigned n = *a.p2g_low;
  const unsigned lane = threadIdx.x & 31u, wpb = blockDim.x / 32u;
  for (unsigned e = blockIdx.x * wpb + (threadIdx.x >> 5); e < n; e += gridDim.x * wpb) {
    const unsigned code = a.p2g_low[1 + e];
    const int s = int(code / 1536u), D = int((code % 1536u) >> 9), v = int(code & 511u);
    int org[3];
    origin_of(a, s, org);
    const int g[3] = {org[0] + (v >> 6), org[1] + ((v >> 3) & 7), org[2] + (v & 7)};
    float ms, ws;
    ref_node_sums(a, a.nbr + int64_t(s) * 27, s, D, g, cells[threadIdx.x >> 5], ms, ws);
    if (lane != 0u) continue;
    const float val = (ws <= 1e-5f) ? 0.f : __fdiv_rn(ms, ws);
    const int64_t o = int64_t(s) * 1536 + D * 512 + v;
    if (FUSED) {
      const bool sc = is_solid(a.sd, g[0], g[1], g[2]);
      const bool zero = sc != is_solid(a.sd, g[0] - (D == 0), g[1] - (D == 1), g[2] - (D == 2));
      const float gf = __fmul_rn(a.dt, D == 0 ? a.fx : (D == 1 ? a.fy : a.fz));
      float vv = zero ? 0.f : val;                              // ApplyBoundaryConditions
      a.vold[o] = vv;                                           // SaveGridVelocities
      vv = (D == 1) ? __fsub_rn(vv, gf) : __fadd_rn(vv, gf);    // AddGravity
      a.vel[o] = zero ? 0.f : vv;                               // ApplyBoundaryConditions
    } else {
      a.vel[o] = val;
      a.weight[o] = ws;
    }
  }
}

__device__ __forceinline__ bool bit_on(const uint32_t* bits, int s, int v) {
  return (bits[int64_t(s) * 16 + (v >> 5)] >> (v & 31)) & 1u;
}

// ApplyBoundaryConditions (per-stage): marker SOLID on solid cells, normal
// component zeroed on active faces with solid on exactly one side.
__global__ void __launch_bounds__(256) k_apply_bc(const __grid_constant__ GridArgs a) {
  const int s = blockIdx.x;
  int org[3];
  origin_of(a, s, org);
  for (int v = threadIdx.x; v < 512; v += 256) {
    const int g[3] = {org[0] + (v >> 6), org[1] + ((v >> 3) & 7), org[2] + (v & 7)};
    const bool sc = is_solid(a.sd, g[0], g[1], g[2]);
    if (sc) a.marker[int64_t(s) * 512 + v] = FSIM_SOLID;
    if (!bit_on(a.vel_on, s, v)) continue;
    float* vel = a.vel + int64_t(s) * 1536;
    if (sc != is_solid(a.sd, g[0] - 1, g[1], g[2])) vel[v] = 0.f;
    if (sc != is_solid(a.sd, g[0], g[1] - 1, g[2])) vel[512 + v] = 0.f;
    if (sc != is_solid(a.sd, g[0], g[1], g[2] - 1)) vel[1024 + v] = 0.f;
  }
}

__global__ void __launch_bounds__(256) k_save(const __grid_constant__ GridArgs a) {
  const int s = blockIdx.x;
  for (int v = threadIdx.x; v < 512; v += 256) {
    const bool on = bit_on(a.vel_on, s, v);
#pragma unroll
    for (int D = 0; D < 3; ++D)
      a.vold[int64_t(s) * 1536 + D * 512 + v] = on ? a.vel[int64_t(s) * 1536 + D * 512 + v] : 0.f;
    if (v < 16) a.vold_on[int64_t(s) * 16 + v] = a.vel_on[int64_t(s) * 16 + v];
  }
}

__global__ void __launch_bounds__(256) k_gravity(const __grid_constant__ GridArgs a) {
  const int s = blockIdx.x;
  const float gf[3] = {__fmul_rn(a.dt, a.fx), __fmul_rn(a.dt, a.fy), __fmul_rn(a.dt, a.fz)};
  for (int v = threadIdx.x; v < 512; v += 256) {
    if (!bit_on(a.vel_on, s, v)) continue;
    float* vel = a.vel + int64_t(s) * 1536;
    vel[v] = __fadd_rn(vel[v], gf[0]);
    vel[512 + v] = __fsub_rn(vel[512 + v], gf[1]);
    vel[1024 + v] = __fadd_rn(vel[1024 + v], gf[2]);
  }
}

// Particles::DeleteOutsideParticles: particles whose cell is outside the box
// get the dead key (they stop contributing and are dropped at the next sort).
__global__ void k_delete_outside(uint32_t* __restrict__ keys, int64_t n, LeafMap lm,
                                 int64_t* __restrict__ ndead) {
  int64_t i = int64_t(blockIdx.x) * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const uint32_t k = keys[i];
  if (k == kDeadKey) return;
  int lx, ly, lz;
  leaf_coords(lm, k >> 9, lx, ly, lz);
  const int v = int(k & 511u);
  const int c0 = lx * 8 + (v >> 6), c1 = ly * 8 + ((v >> 3) & 7), c2 = lz * 8 + (v & 7);
  if (!in_box(lm.n, c0, c1, c2)) {
    keys[i] = kDeadKey;
    atomicAdd(reinterpret_cast<unsigned long long*>(ndead), 1ull);
  }
}

// velocity component D at global node g, from leaf slot s's neighbourhood
__device__ __forceinline__ float vel_at(const GridArgs& a, const float* field, const int* nb,
                                        const int org[3], int D, int gx, int gy, int gz) {
  const int lx = gx - org[0], ly = gy - org[1], lz = gz - org[2];
  const int ns = nb[nb_index(side(lx), side(ly), side(lz))];
  if (ns < 0) return 0.f;
  const int v = ((gx & 7) << 6) | ((gy & 7) << 3) | (gz & 7);
  return field[int64_t(ns) * 1536 + D * 512 + v];
}

__device__ __forceinline__ int marker_at(const GridArgs& a, const int* nb, const int org[3],
                                         int gx, int gy, int gz) {
  const int lx = gx - org[0], ly = gy - org[1], lz = gz - org[2];
  const int ns = nb[nb_index(side(lx), side(ly), side(lz))];
  if (ns < 0) return FSIM_AIR;
  const int v = ((gx & 7) << 6) | ((gy & 7) << 3) | (gz & 7);
  return a.marker[int64_t(ns) * 512 + v];
}

__device__ __forceinline__ float pres_at(const GridArgs& a, const int* nb, const int org[3],
                                         int gx, int gy, int gz) {
  const int lx = gx - org[0], ly = gy - org[1], lz = gz - org[2];
  const int ns = nb[nb_index(side(lx), side(ly), side(lz))];
  if (ns < 0 || ns >= a.n_pleaf) return 0.f;
  const int v = ((gx & 7) << 6) | ((gy & 7) << 3) | (gz & 7);
  return a.pres[int64_t(ns) * 512 + v];
}

// ComputeDivergence over particle leaves (FLUID cells only live there).
__global__ void __launch_bounds__(256) k_divergence(const __grid_constant__ GridArgs a) {
  __shared__ int nb[27];
  const int s = blockIdx.x;
  if (threadIdx.x < 27) nb[threadIdx.x] = a.nbr[int64_t(s) * 27 + threadIdx.x];
  int org[3];
  origin_of(a, s, org);
  __syncthreads();
  for (int v = threadIdx.x; v < 512; v += 256) {
    const int g[3] = {org[0] + (v >> 6), org[1] + ((v >> 3) & 7), org[2] + (v & 7)};
    float d = 0.f;
    if (a.marker[int64_t(s) * 512 + v] == FSIM_FLUID) {
      const float* vel = a.vel + int64_t(s) * 1536;
      d = __fsub_rn(vel_at(a, a.vel, nb, org, 0, g[0] + 1, g[1], g[2]), vel[v]);
      d = __fadd_rn(d, __fsub_rn(vel_at(a, a.vel, nb, org, 1, g[0], g[1] + 1, g[2]), vel[512 + v]));
      d = __fadd_rn(d, __fsub_rn(vel_at(a, a.vel, nb, org, 2, g[0], g[1], g[2] + 1), vel[1024 + v]));
    }
    a.div[int64_t(s) * 512 + v] = d;
  }
}

__device__ __forceinline__ void atomic_max_pos(int64_t* cnt, float v) {
  // non-negative floats order like their bit patterns
  atomicMax(reinterpret_cast<unsigned long long*>(cnt), (unsigned long long)__float_as_uint(v));
}

// UpdateVelocityFromPressure over faces [0,N]^3; FUSED also forms
// GetVelocityUpdate (v_old := v - v_old on active faces) and the CFL max.
template <bool FUSED>
__global__ void __launch_bounds__(256) k_pressure_update(const __grid_constant__ GridArgs a) {
  __shared__ int nb[27];
  __shared__ float red[8];
  const int s = blockIdx.x;
  if (threadIdx.x < 27) nb[threadIdx.x] = a.nbr[int64_t(s) * 27 + threadIdx.x];
  int org[3];
  origin_of(a, s, org);
  // a pressure that is not a solution leaves the faces as they were (the flag
  // is loaded along with the neighbour table)
  const unsigned gave_up = FUSED && a.gave_up ? *a.gave_up : 0u;
  __syncthreads();
  if (gave_up) return;
  const int* n = a.lm.n;
  float vmax = 0.f;
  for (int v = threadIdx.x; v < 512; v += 256) {
    const int g[3] = {org[0] + (v >> 6), org[1] + ((v >> 3) & 7), org[2] + (v & 7)};
    if (g[0] < 0 || g[1] < 0 || g[2] < 0 || g[0] > n[0] || g[1] > n[1] || g[2] > n[2]) continue;
    float* vel = a.vel + int64_t(s) * 1536;
    const int mc = a.marker[int64_t(s) * 512 + v];
    bool on = bit_on(a.vel_on, s, v);
    float val[3] = {vel[v], vel[512 + v], vel[1024 + v]};
    if (mc != FSIM_SOLID) {
      const float pc = (s < a.n_pleaf) ? a.pres[int64_t(s) * 512 + v] : 0.f;
      bool upd = false;
#pragma unroll
      for (int d = 0; d < 3; ++d) {
        const int h0 = g[0] - (d == 0), h1 = g[1] - (d == 1), h2 = g[2] - (d == 2);
        const int mn = marker_at(a, nb, org, h0, h1, h2);
        if ((mn == FSIM_FLUID || mc == FSIM_FLUID) && mn != FSIM_SOLID) {
          val[d] = __fadd_rn(val[d], __fsub_rn(pc, pres_at(a, nb, org, h0, h1, h2)));
          upd = true;
        }
      }
      if (upd) {
        vel[v] = val[0]; vel[512 + v] = val[1]; vel[1024 + v] = val[2];
        if (!on) {
          atomicOr(&a.vel_on[int64_t(s) * 16 + (v >> 5)], 1u << (v & 31));
          on = true;
        }
      }
    }
    if (FUSED && on) {
      float* vold = a.vold + int64_t(s) * 1536;
#pragma unroll
      for (int D = 0; D < 3; ++D) vold[D * 512 + v] = __fsub_rn(val[D], vold[D * 512 + v]);
      if (g[0] < n[0] && g[1] < n[1] && g[2] < n[2]) {
        if (g[1] != n[1] - 1 && g[2] != n[2] - 1) vmax = fmaxf(vmax, fabsf(val[0]));
        if (g[0] != n[0] - 1 && g[2] != n[2] - 1) vmax = fmaxf(vmax, fabsf(val[1]));
        if (g[0] != n[0] - 1 && g[1] != n[1] - 1) vmax = fmaxf(vmax, fabsf(val[2]));
      }
    }
  }
  if (FUSED) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) vmax = fmaxf(vmax, __shfl_xor_sync(0xffffffffu, vmax, o));
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = vmax;
    __syncthreads();
    if (threadIdx.x == 0) {
      float m = 0.f;
      for (int w = 0; w < 8; ++w) m = fmaxf(m, red[w]);
      if (m > 0.f) atomic_max_pos(a.cnt + 4, m);
    }
  }
}

// GetVelocityUpdate (per-stage) over faces [0,N]^3.
__global__ void __launch_bounds__(256) k_velocity_update(const __grid_constant__ GridArgs a) {
  const int s = blockIdx.x;
  int org[3];
  origin_of(a, s, org);
  const int* n = a.lm.n;
  for (int v = threadIdx.x; v < 512; v += 256) {
    const int g[3] = {org[0] + (v >> 6), org[1] + ((v >> 3) & 7), org[2] + (v & 7)};
    if (g[0] < 0 || g[1] < 0 || g[2] < 0 || g[0] > n[0] || g[1] > n[1] || g[2] > n[2]) continue;
    const bool on = bit_on(a.vel_on, s, v), oo = bit_on(a.vold_on, s, v);
    if (on && !oo) atomicAdd(reinterpret_cast<unsigned long long*>(a.cnt + 3), 1ull);
    if (on && oo) {
      float* vel = a.vel + int64_t(s) * 1536;
      float* vold = a.vold + int64_t(s) * 1536;
#pragma unroll
      for (int D = 0; D < 3; ++D) vold[D * 512 + v] = __fsub_rn(vel[D * 512 + v], vold[D * 512 + v]);
    }
  }
}

// CFL max over active in-box faces (FlipSimulation::CFL).
__global__ void __launch_bounds__(256) k_cfl(const __grid_constant__ GridArgs a) {
  __shared__ float red[8];
  const int s = blockIdx.x;
  int org[3];
  origin_of(a, s, org);
  const int* n = a.lm.n;
  float vmax = 0.f;
  for (int v = threadIdx.x; v < 512; v += 256) {
    const int g[3] = {org[0] + (v >> 6), org[1] + ((v >> 3) & 7), org[2] + (v & 7)};
    if (!in_box(n, g[0], g[1], g[2]) || !bit_on(a.vel_on, s, v)) continue;
    const float* vel = a.vel + int64_t(s) * 1536;
    if (g[1] != n[1] - 1 && g[2] != n[2] - 1) vmax = fmaxf(vmax, fabsf(vel[v]));
    if (g[0] != n[0] - 1 && g[2] != n[2] - 1) vmax = fmaxf(vmax, fabsf(vel[512 + v]));
    if (g[0] != n[0] - 1 && g[1] != n[1] - 1) vmax = fmaxf(vmax, fabsf(vel[1024 + v]));
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) vmax = fmaxf(vmax, __shfl_xor_sync(0xffffffffu, vmax, o));
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = vmax;
  __syncthreads();
  if (threadIdx.x == 0) {
    float m = 0.f;
    for (int w = 0; w < 8; ++w) m = fmaxf(m, red[w]);
    if (m > 0.f) atomic_max_pos(a.cnt + 4, m);
  }
}

// ---- dense downloads ------------------------------------------------------
struct DenseArgs {
  LeafMap lm;
  SolidDesc sd;
  const int32_t* slot;  // dense leaf id -> slot
  int n_pleaf;
  const float* vec;     // slot*1536 (Vec3 fields)
  const uint32_t* on;   // slot*16
  const float* sca;     // pleaf*512 (scalar fields)
  const int8_t* marker;
  int field;            // FSIM_FIELD_* or 100 marker
  int valid, extrap, bc;
  float* out;
  int32_t* iout;
  uint8_t* act;
};

__device__ __forceinline__ int slot_of(const DenseArgs& a, int i, int j, int k) {
  const int lx = fdiv(i, 8), ly = fdiv(j, 8), lz = fdiv(k, 8);
  if (!leaf_valid(a.lm, lx, ly, lz)) return -1;
  return a.slot[leaf_id(a.lm, lx, ly, lz)];
}

// A CTA takes 8 kDenseRows rows of 32 cells (z) of one x plane, so that a
// cell's position costs two 32-bit divisions by launch constants.  Slot,
// marker and value are dependent loads, so a thread's rows go through each
// stage together.  Velocity and pressure of a 256^3 domain 310 -> 192 us, the
// pressure of a 512^3 one 792 -> 489 (with one cell per thread 230 and 678,
// three 64-bit divisions per cell before that).
constexpr int kDenseRows = 4;
unsigned dense_blocks(const int n[3]) {
  return unsigned(n[0] + 2) * unsigned((n[1] + 1) / (8 * kDenseRows) + 1) *
         unsigned((n[2] + 1) / 32 + 1);
}
__global__ void __launch_bounds__(256) k_dense(const __grid_constant__ DenseArgs a) {
  const int* n = a.lm.n;
  const unsigned t2 = unsigned(n[2] + 1) / 32u + 1u,
                 t1 = unsigned(n[1] + 1) / (8u * kDenseRows) + 1u;
  const unsigned row = blockIdx.x / t2, plane = row / t1;
  const int i = int(plane) - 1, k = int((blockIdx.x - row * t2) * 32u + (threadIdx.x & 31u)) - 1;
  const int j0 = int((row - plane * t1) * 8u * kDenseRows + (threadIdx.x >> 5)) - 1;
  if (k > n[2]) return;
  int sl[kDenseRows];
#pragma unroll
  for (int r = 0; r < kDenseRows; ++r)
    sl[r] = j0 + 8 * r <= n[1] ? slot_of(a, i, j0 + 8 * r, k) : -1;
  auto at = [&](int j) { return (int64_t(i + 1) * (n[1] + 2) + (j + 1)) * (n[2] + 2) + (k + 1); };
  auto voxel = [](int x, int y, int z) { return ((x & 7) << 6) | ((y & 7) << 3) | (z & 7); };
  if (a.field == 100 || a.field > FSIM_FIELD_WEIGHT) {
    // marker, or a scalar field on FLUID cells (div, pressure, phi)
    int m[kDenseRows];
    float val[kDenseRows];
#pragma unroll
    for (int r = 0; r < kDenseRows; ++r)
      m[r] = a.valid && sl[r] >= 0 ? a.marker[int64_t(sl[r]) * 512 + voxel(i, j0 + 8 * r, k)] : 0;
    const bool phi = a.field == FSIM_FIELD_PHI;
#pragma unroll
    for (int r = 0; r < kDenseRows; ++r) {
      val[r] = phi ? 5.0f : 0.f;
      if (a.field != 100 && a.valid && sl[r] >= 0 && m[r] == FSIM_FLUID) {
        if (phi) val[r] = -0.5f;
        else if (sl[r] < a.n_pleaf) val[r] = a.sca[int64_t(sl[r]) * 512 + voxel(i, j0 + 8 * r, k)];
      }
    }
#pragma unroll
    for (int r = 0; r < kDenseRows; ++r) {
      const int j = j0 + 8 * r;
      if (j > n[1]) break;
      const int64_t o = at(j);
      if (a.field == 100) {
        if (a.bc && is_solid(a.sd, i, j, k)) m[r] = FSIM_SOLID;
        a.iout[o] = m[r];
        if (a.act) a.act[o] = m[r] != 0;
      } else {
        a.out[o] = val[r];
        if (a.act) a.act[o] = a.valid && sl[r] >= 0 && m[r] == FSIM_FLUID;
      }
    }
    return;
  }
#pragma unroll
  for (int r = 0; r < kDenseRows; ++r) {
    const int j = j0 + 8 * r;
    if (j > n[1]) break;
    const int vox = voxel(i, j, k);
    bool on = a.valid && sl[r] >= 0 &&
              ((a.on[int64_t(sl[r]) * 16 + (vox >> 5)] >> (vox & 31)) & 1u);
    const int c[3] = {i, j, k};
    const bool ghost = a.extrap && a.field != FSIM_FIELD_WEIGHT;
    float val[3];
#pragma unroll
    for (int D = 0; D < 3; ++D) {
      int src[3] = {i, j, k};
      if (ghost) ghost_source(n, D, c, src);
      const bool own = src[0] == i && src[1] == j && src[2] == k;
      const int ss = !a.valid ? -1 : (own ? sl[r] : slot_of(a, src[0], src[1], src[2]));
      const int sv = voxel(src[0], src[1], src[2]);
      // the value with its on bit (off: any bits, not used)
      const float v = ss >= 0 ? a.vec[int64_t(ss) * 1536 + D * 512 + sv] : 0.f;
      val[D] = ss >= 0 && ((a.on[int64_t(ss) * 16 + (sv >> 5)] >> (sv & 31)) & 1u) ? v : 0.f;
    }
    if (ghost && extrap_activated(n, i, j, k)) on = true;
    const int64_t o = at(j);
#pragma unroll
    for (int D = 0; D < 3; ++D) a.out[3 * o + D] = on ? val[D] : 0.f;
    if (a.act) a.act[o] = on;
  }
}

inline unsigned nblk(int64_t n, int b) { return unsigned((n + b - 1) / b); }

GridArgs make_args(fsim_sim* s) {
  GridArgs a;
  a.part = s->part[s->cur];
  a.cap = s->cap_p;
  a.keys = s->keys[0];
  a.leaf_id = s->d_leaf_id;
  a.nbr = s->d_nbr;
  a.cell_range = s->d_cell_range;
  a.leaf_range = s->d_leaf_range;
  a.n_pleaf = s->n_pleaf;
  a.n_gleaf = s->n_gleaf;
  a.check_dead = s->deleted_outside ? 1 : 0;
  a.lm = s->lm;
  a.sd = s->solid;
  a.vel = s->vel;
  a.vold = s->vold;
  a.weight = s->weight;
  a.vel_on = s->vel_on;
  a.vold_on = s->vold_on;
  a.marker = s->marker;
  a.pres = s->pres;
  a.div = s->div;
  a.dt = 0.f;
  a.fx = s->cfg.force[0];
  a.fy = s->cfg.force[1];
  a.fz = s->cfg.force[2];
  a.cnt = s->d_cnt;
  a.p2g_nodes = s->p2g_nodes;
  a.p2g_touch = s->p2g_touch;
  a.gave_up = s->pcg_pending ? &s->d_sc->bar_err : nullptr;
  return a;
}

}  // namespace

// P2G pass 1 runs by component below this many particle leaves per SM: 12
// against 29 us at 24 leaves, 28 against 40 at 159, the same at 490, 783
// against 707 at 8,320 (every component reads the positions again).
constexpr int kP2gSplitLeaves = 2;

int launch_p2g(fsim_sim* s, bool fused, float dt) {
  if (s->p2g_cap < s->cap_pleaf) {
    if (s->p2g_nodes) cudaFree(s->p2g_nodes);
    if (s->p2g_touch) cudaFree(s->p2g_touch);
    s->p2g_nodes = nullptr;
    s->p2g_touch = nullptr;
    s->p2g_cap = 0;
    FSIM_CK(s, cudaMalloc(&s->p2g_nodes, size_t(s->cap_pleaf) * 6 * kNodeBlock * 8));
    FSIM_CK(s, cudaMalloc(&s->p2g_touch, size_t(s->cap_pleaf) * 32 * 4));
    s->p2g_cap = s->cap_pleaf;
  }
  // list of low-weight faces: at most every face of every grid leaf, each
  // coded in 32 bits as slot * 1536 + D * 512 + voxel
  if (int64_t(s->n_gleaf) * 1536 >= (int64_t(1) << 32))
    return fail(s, FSIM_ERR_CAPACITY, "too many grid leaves for the P2G low-weight face list");
  const int64_t low_cap = int64_t(s->cap_leaf) * 1536 + 1;
  if (s->p2g_low_cap < low_cap) {
    if (s->p2g_low) cudaFree(s->p2g_low);
    s->p2g_low = nullptr;
    s->p2g_low_cap = 0;
    FSIM_CK(s, cudaMalloc(&s->p2g_low, size_t(low_cap) * sizeof(uint32_t)));
    s->p2g_low_cap = low_cap;
  }
  GridArgs a = make_args(s);
  a.dt = dt;
  a.p2g_low = s->p2g_low;
  FSIM_CK(s, cudaMemsetAsync(s->p2g_low, 0, sizeof(uint32_t), s->stream));
  const char* cells = fused ? "p2g_cells_fused" : "p2g_cells";
  if (s->n_pleaf < kP2gSplitLeaves * s->num_sms) {
    FSIM_CK(s, cudaMemsetAsync(s->p2g_touch, 0, size_t(s->n_pleaf) * 32 * 4, s->stream));
    FSIM_LAUNCH(s, cells, (k_p2g_cells<1, 512>), s->n_pleaf * 3, 512, 0, a);
  } else {
    FSIM_LAUNCH(s, cells, (k_p2g_cells<3, 256>), s->n_pleaf, 256, 0, a);
  }
  const int lgrid = std::max(1, s->num_sms * 12);
  if (fused) {
    FSIM_LAUNCH(s, "p2g_fused", k_p2g_nodes<true>, s->n_gleaf * (512 / kNodeThreads), kNodeThreads, 0, a);
    FSIM_LAUNCH(s, "p2g_low_fused", k_p2g_low<true>, lgrid, 128, 0, a);
  } else {
    FSIM_LAUNCH(s, "p2g", k_p2g_nodes<false>, s->n_gleaf * (512 / kNodeThreads), kNodeThreads, 0, a);
    FSIM_LAUNCH(s, "p2g_low", k_p2g_low<false>, lgrid, 128, 0, a);
  }
  return FSIM_OK;
}

int launch_apply_bc(fsim_sim* s) {
  FSIM_LAUNCH(s, "apply_bc", k_apply_bc, s->n_gleaf, 256, 0, make_args(s));
  return FSIM_OK;
}

int launch_save_velocities(fsim_sim* s) {
  FSIM_LAUNCH(s, "save_velocities", k_save, s->n_gleaf, 256, 0, make_args(s));
  return FSIM_OK;
}

int launch_add_gravity(fsim_sim* s, float dt) {
  GridArgs a = make_args(s);
  a.dt = dt;
  FSIM_LAUNCH(s, "add_gravity", k_gravity, s->n_gleaf, 256, 0, a);
  return FSIM_OK;
}

int launch_delete_outside(fsim_sim* s) {
  FSIM_LAUNCH(s, "delete_outside", k_delete_outside, nblk(s->n_live, 256), 256, 0, s->keys[0],
              s->n_live, s->lm, s->d_cnt + 6);
  return FSIM_OK;
}

int launch_divergence(fsim_sim* s) {
  FSIM_LAUNCH(s, "divergence", k_divergence, s->n_pleaf, 256, 0, make_args(s));
  return FSIM_OK;
}

int launch_pressure_update(fsim_sim* s, bool fused) {
  if (fused) {
    FSIM_CK(s, cudaMemsetAsync(s->d_cnt + 4, 0, sizeof(int64_t), s->stream));
    FSIM_LAUNCH(s, "pressure_update_fused", k_pressure_update<true>, s->n_gleaf, 256, 0,
                make_args(s));
  } else {
    FSIM_LAUNCH(s, "pressure_update", k_pressure_update<false>, s->n_gleaf, 256, 0, make_args(s));
  }
  return FSIM_OK;
}

int launch_velocity_update(fsim_sim* s) {
  FSIM_CK(s, cudaMemsetAsync(s->d_cnt + 3, 0, sizeof(int64_t), s->stream));
  FSIM_LAUNCH(s, "velocity_update", k_velocity_update, s->n_gleaf, 256, 0, make_args(s));
  return FSIM_OK;
}

int launch_cfl(fsim_sim* s) {
  FSIM_CK(s, cudaMemsetAsync(s->d_cnt + 4, 0, sizeof(int64_t), s->stream));
  FSIM_LAUNCH(s, "cfl_max", k_cfl, s->n_gleaf, 256, 0, make_args(s));
  return FSIM_OK;
}

int ensure_dense(fsim_sim* s, size_t bytes) {
  if (s->dense_tmp.bytes >= bytes) return FSIM_OK;
  if (s->dense_tmp.p) cudaFree(s->dense_tmp.p);
  s->dense_tmp.p = nullptr;
  s->dense_tmp.bytes = 0;
  FSIM_CK(s, cudaMalloc(&s->dense_tmp.p, bytes));
  s->dense_tmp.bytes = bytes;
  return FSIM_OK;
}

static DenseArgs dense_args(fsim_sim* s) {
  DenseArgs a;
  memset(&a, 0, sizeof(a));
  a.lm = s->lm;
  a.sd = s->solid;
  a.slot = s->d_slot;
  a.n_pleaf = s->n_pleaf;
  a.marker = s->marker;
  return a;
}

int download_dense(fsim_sim* s, int field, float* out, uint8_t* active) {
  const int* n = s->lm.n;
  const int64_t tot = int64_t(n[0] + 2) * (n[1] + 2) * (n[2] + 2);
  const int comps = (field <= FSIM_FIELD_WEIGHT) ? 3 : 1;
  const size_t fb = size_t(tot) * comps * sizeof(float);
  int rc = ensure_dense(s, fb + size_t(tot));
  if (rc) return rc;
  DenseArgs a = dense_args(s);
  a.field = field;
  a.out = static_cast<float*>(s->dense_tmp.p);
  a.act = static_cast<uint8_t*>(s->dense_tmp.p) + fb;
  bool have = s->have_topology && s->grid_valid;
  switch (field) {
    case FSIM_FIELD_VELOCITY: a.vec = s->vel; a.on = s->vel_on; a.valid = have; a.extrap = s->extrapolated; break;
    case FSIM_FIELD_VELOCITY_UPDATE: a.vec = s->vold; a.on = s->vold_on; a.valid = have && s->saved; a.extrap = s->extrapolated; break;
    case FSIM_FIELD_WEIGHT: a.vec = s->weight; a.on = s->vel_on; a.valid = have && s->weight_valid; break;
    case FSIM_FIELD_DIVERGENCE: a.sca = s->div; a.valid = have && s->div_valid; break;
    case FSIM_FIELD_PRESSURE: a.sca = s->pres; a.valid = have && s->pres_valid; break;
    case FSIM_FIELD_PHI: a.valid = have && s->phi_valid; break;
    default: return fail(s, FSIM_ERR_INVALID, "unknown field");
  }
  FSIM_LAUNCH(s, "dense_download", k_dense, dense_blocks(n), 256, 0, a);
  FSIM_CK(s, cudaMemcpyAsync(out, a.out, fb, cudaMemcpyDeviceToHost, s->stream));
  if (active)
    FSIM_CK(s, cudaMemcpyAsync(active, a.act, size_t(tot), cudaMemcpyDeviceToHost, s->stream));
  FSIM_CK(s, cudaStreamSynchronize(s->stream));
  return FSIM_OK;
}

int download_marker(fsim_sim* s, int32_t* out, uint8_t* active) {
  const int* n = s->lm.n;
  const int64_t tot = int64_t(n[0] + 2) * (n[1] + 2) * (n[2] + 2);
  int rc = ensure_dense(s, size_t(tot) * 5);
  if (rc) return rc;
  DenseArgs a = dense_args(s);
  a.field = 100;
  a.iout = static_cast<int32_t*>(s->dense_tmp.p);
  a.act = static_cast<uint8_t*>(s->dense_tmp.p) + size_t(tot) * 4;
  a.valid = s->have_topology && s->grid_valid;
  a.bc = s->bc_applied;
  FSIM_LAUNCH(s, "dense_download", k_dense, dense_blocks(n), 256, 0, a);
  FSIM_CK(s, cudaMemcpyAsync(out, a.iout, size_t(tot) * 4, cudaMemcpyDeviceToHost, s->stream));
  if (active)
    FSIM_CK(s, cudaMemcpyAsync(active, a.act, size_t(tot), cudaMemcpyDeviceToHost, s->stream));
  FSIM_CK(s, cudaStreamSynchronize(s->stream));
  return FSIM_OK;
}

}  // namespace fsim
