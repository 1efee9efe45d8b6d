// k_topology.cu -- advection + rebinning and the sparse 8^3 brick topology.
//
// Restates Particles::StepInGrid<VectorGrid,true,1,1> (common/particles.cc:
// 479-546) and DeleteParticlesInSolids (:202-219) as: one kernel that
// advects every particle (pos += gvel*dt, IEEE round-to-nearest, no FMA
// contraction), clamps it to [0,N] exactly as the reference does and emits
// its cell key (dead key for particles in solids) and counts the leaves'
// particles; the leaf topology from those counts (particle leaves, one-leaf
// dilation, slots); a stable sort by key (this reproduces the reference's
// rebuilt cell lists, which keep particles in visiting order): rows into
// their leaf's bin, then one CTA per leaf orders its bin; a gather of the 9
// particle arrays; the 27-neighbour table and the per-cell particle ranges.
#include <algorithm>
#include <cmath>
#include <cstring>

#include <cub/device/device_radix_sort.cuh>
#include <cub/device/device_scan.cuh>

#include "fsim_internal.cuh"

namespace fsim {

// ---- Source<T> (common/sources.cc:66-109), evaluated on the host --------
void source_box(const fsim_source& src, float t, float lo[3], float hi[3]) {
  (void)t;  // the oscillating branch of get_box assigns a shadowed local
  for (int d = 0; d < 3; ++d) {
    lo[d] = src.lo[d];
    hi[d] = src.hi[d] - 1.0f;  // box.set_end(box.get_end() - Vec3(1))
  }
}
void source_velocity(const fsim_source& src, float t, float v[3]) {
  if (!src.velocity_oscillating) {
    for (int d = 0; d < 3; ++d) v[d] = src.velocity[d];
    return;
  }
  const float w = float(M_PI * double(t) / double(src.box_period));  // T w = M_PI*t/box_period_
  for (int d = 0; d < 3; ++d)
    v[d] = float(double(src.velocity[d]) +
                 0.5 * double(src.velocity2[d] - src.velocity[d]) * (double(std::cos(w)) + 1.0));
}
bool source_active(const fsim_source& src, float t) {
  return !src.timed || (t >= src.start_time && t <= src.end_time);
}

namespace {

// Boxes of DeleteFluidInSources (get_box(t) of every source), passed by value.
struct SourceRegions {
  int n;
  float lo[FSIM_MAX_SOURCES][3], hi[FSIM_MAX_SOURCES][3];
};
__device__ __forceinline__ bool in_regions(const SourceRegions& r, const float p[3]) {
  for (int q = 0; q < r.n; ++q) {
    bool in = true;
#pragma unroll
    for (int d = 0; d < 3; ++d) in &= (p[d] >= r.lo[q][d]) & (p[d] <= r.hi[q][d]);  // Cube::IsInside
    if (in) return true;
  }
  return false;
}

__device__ __forceinline__ float fadd(float a, float b) { return __fadd_rn(a, b); }
__device__ __forceinline__ float fmul(float a, float b) { return __fmul_rn(a, b); }

// One more particle of each lane's key in its leaf's count, one atomic per
// leaf in the warp.  Called by all 32 lanes.
__device__ __forceinline__ void count_leaf(uint32_t* __restrict__ lcnt, uint32_t key) {
  const unsigned same = __match_any_sync(0xffffffffu, key >> 9);
  if (key != kDeadKey && int(threadIdx.x & 31) == __ffs(int(same)) - 1)
    atomicAdd(lcnt + (key >> 9), unsigned(__popc(same)));
}
__global__ void k_count_leaves(const uint32_t* __restrict__ k, int64_t n,
                               uint32_t* __restrict__ lcnt) {
  const int64_t i = int64_t(blockIdx.x) * blockDim.x + threadIdx.x;
  count_leaf(lcnt, i < n ? k[i] : kDeadKey);
}

// mode 0: key from current position (upload); positions outside [0,N]
//         are counted as invalid.
// mode 1: advect by gvel*dt, clamp, delete in solids (MoveParticles).
// mode 1 extra: particles inside a source region get the dead key
// (DeleteFluidInSources right after MoveParticles).
__global__ void k_keys(float* __restrict__ part, int64_t cap, const uint32_t* __restrict__ kcur,
                       uint32_t* __restrict__ kout, int64_t n, LeafMap lm, SolidDesc sd, int mode,
                       float dt, unsigned long long* __restrict__ invalid,
                       const SourceRegions reg, uint32_t* __restrict__ lcnt) {
  const int64_t i = int64_t(blockIdx.x) * blockDim.x + threadIdx.x;
  uint32_t k = kDeadKey;
  if (i < n && (mode != 1 || kcur[i] != kDeadKey)) {
    float* px = part;
    const float* gx = part + 6 * cap;
    float p[3] = {px[i], px[cap + i], px[2 * cap + i]};
    int id[3];
    if (mode == 1) {
      const float g[3] = {gx[i], gx[cap + i], gx[2 * cap + i]};
#pragma unroll
      for (int d = 0; d < 3; ++d) {
        p[d] = fadd(p[d], fmul(g[d], dt));
        id[d] = int(floorf(p[d]));
      }
#pragma unroll
      for (int d = 0; d < 3; ++d)
        if (id[d] < 0) { id[d] = 0; p[d] = 0.f; }
#pragma unroll
      for (int d = 0; d < 3; ++d)
        if (id[d] >= lm.n[d]) { id[d] = lm.n[d]; p[d] = float(lm.n[d]); }
      px[i] = p[0];
      px[cap + i] = p[1];
      px[2 * cap + i] = p[2];
      if (!is_solid(sd, id[0], id[1], id[2])) k = cell_key(lm, id[0], id[1], id[2]);
      if (reg.n > 0 && in_regions(reg, p)) k = kDeadKey;
    } else {
      bool ok = true;
#pragma unroll
      for (int d = 0; d < 3; ++d) {
        ok &= (p[d] >= 0.f) && (p[d] <= float(lm.n[d]));
        id[d] = int(floorf(p[d]));
      }
      if (ok)
        k = cell_key(lm, id[0], id[1], id[2]);
      else
        atomicAdd(invalid, 1ull);
    }
  }
  count_leaf(lcnt, k);
  if (i < n) kout[i] = k;
}

// The keys of a step on a host-resident state (fsim_step_host), one pass over
// the uploaded rows: validity and cell key of the uploaded position (kold),
// then mode 1's advection, clamping, deletion in solids and key (knew), with
// the advected position stored (and gvel, for a gather that moves it).  Counts
// positions outside [0, N] and neighbouring rows out of cell order.  The rows
// need no rebinning of their own first: by (new key, old key, row) they are in
// the order that rebinning them, moving them and rebinning again gives.
__global__ void __launch_bounds__(256)
    k_host_keys(const float* __restrict__ pos, const float* __restrict__ gvel,
                float* __restrict__ part, int64_t cap, uint32_t* __restrict__ kold,
                uint32_t* __restrict__ knew, int64_t n, LeafMap lm, SolidDesc sd, float dt,
                int keep_gvel, unsigned long long* __restrict__ invalid,
                unsigned long long* __restrict__ unsorted, uint32_t* __restrict__ lcnt) {
  const int64_t i = int64_t(blockIdx.x) * blockDim.x + threadIdx.x;
  auto old_key = [&](int64_t r, float (&p)[3]) {
    bool ok = true;
    int id[3];
#pragma unroll
    for (int d = 0; d < 3; ++d) {
      p[d] = pos[3 * r + d];
      ok &= (p[d] >= 0.f) && (p[d] <= float(lm.n[d]));
      id[d] = int(floorf(p[d]));
    }
    return ok ? cell_key(lm, id[0], id[1], id[2]) : kDeadKey;
  };
  float p[3] = {0.f, 0.f, 0.f}, q[3];
  const uint32_t old = i < n ? old_key(i, p) : kDeadKey;
  uint32_t next = __shfl_down_sync(0xffffffffu, old, 1);
  if ((threadIdx.x & 31) == 31) next = i + 1 < n ? old_key(i + 1, q) : kDeadKey;
  const unsigned desc = __ballot_sync(0xffffffffu, i + 1 < n && old > next);
  const unsigned bad = __ballot_sync(0xffffffffu, i < n && old == kDeadKey);
  if ((threadIdx.x & 31) == 0) {
    if (desc) atomicAdd(unsorted, static_cast<unsigned long long>(__popc(desc)));
    if (bad) atomicAdd(invalid, static_cast<unsigned long long>(__popc(bad)));
  }
  uint32_t k = kDeadKey;
  if (i < n) {
    int id[3];
    float g[3];
#pragma unroll
    for (int d = 0; d < 3; ++d) {
      g[d] = gvel[3 * i + d];
      p[d] = fadd(p[d], fmul(g[d], dt));
      id[d] = int(floorf(p[d]));
    }
#pragma unroll
    for (int d = 0; d < 3; ++d)
      if (id[d] < 0) { id[d] = 0; p[d] = 0.f; }
#pragma unroll
    for (int d = 0; d < 3; ++d)
      if (id[d] >= lm.n[d]) { id[d] = lm.n[d]; p[d] = float(lm.n[d]); }
#pragma unroll
    for (int d = 0; d < 3; ++d) {
      part[d * cap + i] = p[d];
      if (keep_gvel) part[(6 + d) * cap + i] = g[d];
    }
    if (!is_solid(sd, id[0], id[1], id[2])) k = cell_key(lm, id[0], id[1], id[2]);
    kold[i] = old;
    knew[i] = k;
  }
  // (an invalid upload's rows may lie anywhere; nothing is set up from them)
  count_leaf(lcnt, k);
}

// Four sorted keys per thread (one 16-byte load; key arrays start 256-byte
// aligned), so a warp streams 512 contiguous bytes per request.
constexpr int kKeysPerThread = 4;
__device__ __forceinline__ void load_keys4(const uint32_t* __restrict__ k, int64_t i0, int64_t n,
                                           uint32_t (&v)[kKeysPerThread]) {
  if (i0 + kKeysPerThread <= n) {
    const uint4 q = *reinterpret_cast<const uint4*>(k + i0);
    v[0] = q.x;
    v[1] = q.y;
    v[2] = q.z;
    v[3] = q.w;
  } else {
#pragma unroll
    for (int j = 0; j < kKeysPerThread; ++j) v[j] = i0 + j < n ? k[i0 + j] : kDeadKey;
  }
}

// particles of a leaf that k_sort_leaf orders in shared memory, and the bit
// set in cnt[1] when a leaf holds more
constexpr int kLeafSort = 12288;
constexpr int64_t kLeafOverflow = int64_t(1) << 40;

// Permutes the first NF particle arrays (9: pos, vel, gvel; 6: pos, vel).
template <int NF>
__global__ void k_gather(const float* __restrict__ in, float* __restrict__ out, int64_t cap,
                         const uint32_t* __restrict__ perm, const int64_t* __restrict__ cnt) {
  int64_t i = int64_t(blockIdx.x) * blockDim.x + threadIdx.x;
  const int64_t n = cnt[1] & kLeafOverflow ? 0 : cnt[0];
  if (i >= n) return;
  const int64_t src = perm[i];
#pragma unroll
  for (int f = 0; f < NF; ++f) out[f * cap + i] = in[f * cap + src];
}

// The leaf topology from the particles' counts, in two kernels over tiles of
// 1,024 leaf ids: k_leaf_flags marks the leaves with particles (1) and the
// rest of their one-leaf dilation (2) and adds up its tile; k_leaf_slots adds
// up the tiles before its own and numbers the leaves (those with particles
// first) and the start of each leaf's particles.  The counts come with the
// keys, so this needs no sorted keys and runs before the sort.  Both kernels
// are a latency: 15 us at 4,096 leaf ids and 39 at 64,000 (launches timed one
// by one), where finding the live keys, marking, dilation, a library scan and
// the assignment, in seven launches, took 41 and 71.
constexpr int kLeafTile = 1024;
__global__ void __launch_bounds__(kLeafTile)
    k_leaf_flags(const uint32_t* __restrict__ lcnt, uint8_t* __restrict__ flag,
                 uint4* __restrict__ tile, LeafMap lm) {
  __shared__ uint4 sh[kLeafTile / 32];
  const uint32_t d = blockIdx.x * kLeafTile + threadIdx.x;
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  uint32_t c = 0, f = 0;
  if (d < lm.dense) {
    c = lcnt[d];
    f = c ? 1u : 0u;
    int lx, ly, lz;
    leaf_coords(lm, d, lx, ly, lz);
    if (!c && leaf_valid(lm, lx, ly, lz)) {
      uint32_t any = 0;  // independent loads: no early exit
#pragma unroll
      for (int q = 0; q < 27; ++q) {
        const int ax = lx + q / 9 - 1, ay = ly + (q / 3) % 3 - 1, az = lz + q % 3 - 1;
        if (leaf_valid(lm, ax, ay, az)) any |= lcnt[leaf_id(lm, ax, ay, az)];
      }
      f = any ? 2u : 0u;
    }
    flag[d] = uint8_t(f);
  }
  // tile totals: leaves with particles, dilated ones, particles; the fullest leaf
  uint4 t = make_uint4(__popc(__ballot_sync(0xffffffffu, f == 1u)),
                       __popc(__ballot_sync(0xffffffffu, f == 2u)), c, c);
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    t.z += __shfl_xor_sync(0xffffffffu, t.z, o);
    t.w = max(t.w, __shfl_xor_sync(0xffffffffu, t.w, o));
  }
  if (lane == 0) sh[w] = t;
  __syncthreads();
  if (w == 0) {
    t = sh[lane];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      t.x += __shfl_xor_sync(0xffffffffu, t.x, o);
      t.y += __shfl_xor_sync(0xffffffffu, t.y, o);
      t.z += __shfl_xor_sync(0xffffffffu, t.z, o);
      t.w = max(t.w, __shfl_xor_sync(0xffffffffu, t.w, o));
    }
    if (lane == 0) tile[blockIdx.x] = t;
  }
}

// cnt: live particles; particle leaves, with kLeafOverflow when a leaf holds
// more than kLeafSort; all leaves
__global__ void __launch_bounds__(kLeafTile)
    k_leaf_slots(const uint32_t* __restrict__ lcnt, const uint8_t* __restrict__ flag,
                 const uint4* __restrict__ tile, int32_t* __restrict__ slot,
                 int32_t* __restrict__ leaf_of, uint32_t* __restrict__ start, uint32_t n,
                 int64_t* __restrict__ cnt) {
  __shared__ uint4 sh[kLeafTile / 32], all[kLeafTile / 32];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const uint32_t d = blockIdx.x * kLeafTile + threadIdx.x;
  const uint32_t c = d < n ? lcnt[d] : 0u, f = d < n ? flag[d] : 0u;
  uint4 b = make_uint4(0u, 0u, 0u, 0u), a = b;  // tiles before this one; all tiles
  for (uint32_t q = threadIdx.x; q < gridDim.x; q += kLeafTile) {
    const uint4 t = tile[q];
    a.x += t.x;
    a.y += t.y;
    a.z += t.z;
    a.w = max(a.w, t.w);
    if (q < blockIdx.x) {
      b.x += t.x;
      b.y += t.y;
      b.z += t.z;
    }
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    b.x += __shfl_xor_sync(0xffffffffu, b.x, o);
    b.y += __shfl_xor_sync(0xffffffffu, b.y, o);
    b.z += __shfl_xor_sync(0xffffffffu, b.z, o);
    a.x += __shfl_xor_sync(0xffffffffu, a.x, o);
    a.y += __shfl_xor_sync(0xffffffffu, a.y, o);
    a.z += __shfl_xor_sync(0xffffffffu, a.z, o);
    a.w = max(a.w, __shfl_xor_sync(0xffffffffu, a.w, o));
  }
  // within the warp: leaves by ballot, particles by an inclusive scan
  const unsigned m1 = __ballot_sync(0xffffffffu, f == 1u), m2 = __ballot_sync(0xffffffffu, f == 2u);
  uint32_t incl = c;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const uint32_t v = __shfl_up_sync(0xffffffffu, incl, o);
    if (lane >= o) incl += v;
  }
  // a warp's entry: its share of the tiles before, and its own totals
  __shared__ uint4 own[kLeafTile / 32];
  if (lane == 31) own[w] = make_uint4(__popc(m1), __popc(m2), incl, 0u);
  if (lane == 0) {
    sh[w] = b;
    all[w] = a;
  }
  __syncthreads();
  uint32_t np = 0, p1 = 0, p2 = 0, pc = 0;
  a = all[lane];
  b = sh[lane];
  const uint4 o4 = own[lane];
  if (lane < w) {
    b.x += o4.x;
    b.y += o4.y;
    b.z += o4.z;
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    a.x += __shfl_xor_sync(0xffffffffu, a.x, o);
    a.y += __shfl_xor_sync(0xffffffffu, a.y, o);
    a.z += __shfl_xor_sync(0xffffffffu, a.z, o);
    a.w = max(a.w, __shfl_xor_sync(0xffffffffu, a.w, o));
    b.x += __shfl_xor_sync(0xffffffffu, b.x, o);
    b.y += __shfl_xor_sync(0xffffffffu, b.y, o);
    b.z += __shfl_xor_sync(0xffffffffu, b.z, o);
  }
  np = a.x;
  const unsigned below = (1u << lane) - 1u;
  p1 = b.x + __popc(m1 & below);
  p2 = b.y + __popc(m2 & below);
  pc = b.z + incl - c;
  if (d == 0) {
    cnt[0] = int64_t(a.z);
    cnt[1] = int64_t(np) | (a.w > unsigned(kLeafSort) ? kLeafOverflow : 0);
    cnt[2] = int64_t(np + a.y);
  }
  if (d >= n) return;
  const int sl = f == 1u ? int(p1) : (f == 2u ? int(np + p2) : -1);
  slot[d] = sl;
  if (sl >= 0) leaf_of[sl] = int32_t(d);
  start[d] = pc;
}

// ---- the stable sort by cell key ------------------------------------------------
// The keys are a leaf's number and a cell's, and a leaf's particles fit in
// shared memory, so two kernels do what a radix sort over all key bits takes
// three to four passes through memory for; the old keys of a host step's rows
// (those of appended source particles too) break ties there, instead of a
// sort of their own before.  32.2 M rows, out of order: 600 us against 1,977
// (two library sorts and a permutation); 52,894 rows: 20 against 57.  Bound
// by the bins' traffic (18 to 26 B per row) and shared-memory atomics.
//
// k_bin_rows: each row's number, cell in the leaf and (OLD) old key to the
// next place of its leaf's bin, one atomic per leaf in a warp (rows that were
// in cell order before a move have one or two).  The places within a bin come
// in any order; k_sort_leaf's order does not depend on it.
template <bool OLD>
__global__ void __launch_bounds__(256)
    k_bin_rows(const uint32_t* __restrict__ knew, const uint32_t* __restrict__ kold, int64_t n,
               uint32_t* __restrict__ next, uint32_t* __restrict__ row,
               uint32_t* __restrict__ old, uint16_t* __restrict__ cell) {
  constexpr int kPer = 4;
  const int64_t i0 = (int64_t(blockIdx.x) * 256 + (threadIdx.x & ~31u)) * kPer + (threadIdx.x & 31);
  const int lane = threadIdx.x & 31;
  uint32_t k[kPer], q[kPer];
#pragma unroll
  for (int j = 0; j < kPer; ++j) k[j] = i0 + 32 * j < n ? knew[i0 + 32 * j] : kDeadKey;
#pragma unroll
  for (int j = 0; j < kPer; ++j) {
    const unsigned same = __match_any_sync(0xffffffffu, k[j] >> 9);
    const int lead = __ffs(int(same)) - 1;
    uint32_t b = 0;
    if (k[j] != kDeadKey && lane == lead) b = atomicAdd(next + (k[j] >> 9), unsigned(__popc(same)));
    q[j] = __shfl_sync(0xffffffffu, b, lead) + __popc(same & ((1u << lane) - 1u));
  }
#pragma unroll
  for (int j = 0; j < kPer; ++j) {
    if (k[j] == kDeadKey) continue;
    row[q[j]] = uint32_t(i0 + 32 * j);
    cell[q[j]] = uint16_t(k[j] & 511u);
    if (OLD) old[q[j]] = kold[i0 + 32 * j];
  }
}

// k_sort_leaf: a CTA orders a leaf's bin by (cell, old key, row): a counting
// sort by cell into shared memory, then each entry's rank among its cell's
// (about 8, most of them one broadcast for the warp).  A cell of more than
// kCrowded entries, whose ranks would take the square of that, is sorted in
// place instead, by a warp, or past kWideCell by the CTA.  One leaf of about
// 12,000 rows in cells of 24 / 40 / 64 / 128 / 512 / 1,024 / 6,144 (us, rows
// with old keys): ranks 104 / 73 / 387 / 722 / 2,274 / 3,449 / 4,574, sorted 135 / 94 /
// 72 / 65 / 71 / 85 / 133; the library's sort of the same rows takes 58 to 101.
// keys and perm get the leaf's sorted keys and rows.
constexpr int kLeafSortThreads = 1024;
constexpr int kCrowded = 48, kWideCell = 1024;
template <bool OLD>
using SortEntry = typename std::conditional<OLD, unsigned long long, uint32_t>::type;

// Bitonic sort of e[0 .. m) by threads t of n, sync() between passes.  Every
// comparison puts the smaller entry first, so places past m (up to the power
// of two, where larger entries would be) need not exist.
template <typename E, typename S>
__device__ __forceinline__ void bitonic_sort(E* e, int m, int t0, int n, S&& sync) {
  int lg = 0;
  while ((1 << lg) < m) ++lg;
  auto order = [&](int i, int j) {
    if (j >= m) return;
    const E a = e[i], b = e[j];
    if (b < a) {
      e[i] = b;
      e[j] = a;
    }
  };
  for (int k = 1; k <= lg; ++k) {
    for (int q = k; q > 0; --q) {
      const int h = 1 << (q - 1);  // half a block; the first pass of k compares mirrored places
      for (int t = t0; t < (1 << lg) / 2; t += n) {
        const int off = t & (h - 1), base = (t - off) * 2;
        order(base + off, q == k ? base + 2 * h - 1 - off : base + off + h);
      }
      sync();
    }
  }
}

template <bool OLD>
__global__ void __launch_bounds__(kLeafSortThreads)
    k_sort_leaf(const int32_t* __restrict__ leaf_of, const int64_t* __restrict__ cnt,
                const uint32_t* __restrict__ lcnt, const uint32_t* __restrict__ next,
                const uint32_t* __restrict__ row, const uint32_t* __restrict__ old,
                const uint16_t* __restrict__ cell, uint32_t* __restrict__ keys,
                uint32_t* __restrict__ perm) {
  using E = SortEntry<OLD>;
  extern __shared__ __align__(16) unsigned char sort_smem[];
  E* ent = reinterpret_cast<E*>(sort_smem);  // kLeafSort entries
  __shared__ int at[512];                    // a cell's count, then its next place
  __shared__ int wsum[16];
  __shared__ int crowded, crowd[kLeafSort / kCrowded];  // the crowded cells, in any order
  if (cnt[1] & kLeafOverflow) return;  // the host sorts another way
  const int np = int(cnt[1]), tid = threadIdx.x, lane = tid & 31;
  for (int s = blockIdx.x; s < np; s += gridDim.x) {
    const uint32_t d = uint32_t(leaf_of[s]);
    const int m = int(lcnt[d]);
    const uint32_t b = next[d] - uint32_t(m);  // k_bin_rows left it at the bin's end
    if (tid < 512) at[tid] = 0;
    if (tid == 0) crowded = 0;
    __syncthreads();
    for (int j = tid; j < m; j += kLeafSortThreads) atomicAdd(&at[cell[b + j]], 1);
    __syncthreads();
    int c = 0, first = 0;
    if (tid < 512) {
      c = at[tid];
      first = c;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const int v = __shfl_up_sync(0xffffffffu, first, o);
        if (lane >= o) first += v;
      }
      if (lane == 31) wsum[tid >> 5] = first;
    }
    __syncthreads();
    if (tid < 512) {
      int before = lane < (tid >> 5) ? wsum[lane & 15] : 0;  // at most 15 warps before
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) before += __shfl_xor_sync(0xffffffffu, before, o);
      first += before - c;
      at[tid] = first;
      if (c > kCrowded) crowd[atomicAdd(&crowded, 1)] = tid;
    }
    __syncthreads();
    for (int j = tid; j < m; j += kLeafSortThreads) {
      const int v = cell[b + j];
      const int p = atomicAdd(&at[v], 1);
      E e = row[b + j];
      if constexpr (OLD) e |= static_cast<unsigned long long>(old[b + j]) << 32;
      ent[p] = e;
      keys[b + p] = (d << 9) | uint32_t(v);
    }
    __syncthreads();
    for (int q = 0; q < crowded; ++q) {
      const int v = crowd[q], beg = v ? at[v - 1] : 0, n = at[v] - beg;
      if (n > kWideCell) {
        bitonic_sort(ent + beg, n, tid, kLeafSortThreads, [] { __syncthreads(); });
        for (int j = tid; j < n; j += kLeafSortThreads) perm[b + beg + j] = uint32_t(ent[beg + j]);
      }
    }
    for (int q = tid >> 5; q < crowded; q += kLeafSortThreads / 32) {
      const int v = crowd[q], beg = v ? at[v - 1] : 0, n = at[v] - beg;
      if (n <= kWideCell) {
        bitonic_sort(ent + beg, n, lane, 32, [] { __syncwarp(); });
        for (int j = lane; j < n; j += 32) perm[b + beg + j] = uint32_t(ent[beg + j]);
      }
    }
    for (int j = tid; j < m; j += kLeafSortThreads) {
      const int v = cell[b + j], end = at[v], beg = v ? at[v - 1] : 0;
      if (end - beg > kCrowded) continue;
      E e = row[b + j];
      if constexpr (OLD) e |= static_cast<unsigned long long>(old[b + j]) << 32;
      int rank = 0;
      for (int y = beg; y < end; ++y) rank += ent[y] < e;
      perm[b + beg + rank] = uint32_t(e);
    }
    __syncthreads();  // before the next leaf's counts
  }
}

// For the library sort of leaves too full for k_sort_leaf: row numbers, and
// (new key << 32 | old key)
__global__ void k_rows(uint32_t* __restrict__ v, int64_t n) {
  const int64_t i = int64_t(blockIdx.x) * blockDim.x + threadIdx.x;
  if (i < n) v[i] = uint32_t(i);
}
__global__ void k_join_keys(const uint32_t* __restrict__ knew, const uint32_t* __restrict__ kold,
                            unsigned long long* __restrict__ k64, int64_t n) {
  const int64_t i = int64_t(blockIdx.x) * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const uint32_t k = knew[i];
  k64[i] = k == kDeadKey ? ~0ull : (static_cast<unsigned long long>(k) << 32) | kold[i];
}

__global__ void k_nbr(const int32_t* __restrict__ leaf_of, const int32_t* __restrict__ slot,
                      int32_t* __restrict__ nbr, int ng, LeafMap lm) {
  int64_t t = int64_t(blockIdx.x) * blockDim.x + threadIdx.x;
  if (t >= int64_t(ng) * 27) return;
  int s = int(t / 27), q = int(t % 27);
  int lx, ly, lz;
  leaf_coords(lm, uint32_t(leaf_of[s]), lx, ly, lz);
  int ax = lx + q / 9 - 1, ay = ly + (q / 3) % 3 - 1, az = lz + q % 3 - 1;
  int v = -1;
  if (leaf_valid(lm, ax, ay, az)) v = slot[leaf_id(lm, ax, ay, az)];
  nbr[t] = v;
}

__global__ void k_ranges(const uint32_t* __restrict__ k, const int64_t* __restrict__ cnt,
                         const int32_t* __restrict__ slot, uint2* __restrict__ cr,
                         uint2* __restrict__ lr) {
  const int64_t n = cnt[0];
  const int64_t i0 = (int64_t(blockIdx.x) * blockDim.x + threadIdx.x) * kKeysPerThread;
  if (i0 >= n) return;
  uint32_t v[kKeysPerThread + 2];  // the key before, the four keys, the key after
  {
    uint32_t q[kKeysPerThread];
    load_keys4(k, i0, n, q);
#pragma unroll
    for (int j = 0; j < kKeysPerThread; ++j) v[j + 1] = q[j];
  }
  v[0] = i0 == 0 ? kDeadKey : k[i0 - 1];  // kDeadKey: no live key equals it
  v[kKeysPerThread + 1] = i0 + kKeysPerThread < n ? k[i0 + kKeysPerThread] : kDeadKey;
#pragma unroll
  for (int j = 0; j < kKeysPerThread; ++j) {
    const int64_t i = i0 + j;
    if (i >= n) break;
    const uint32_t key = v[j + 1];
    // past the last live key, v holds kDeadKey, which ends every range
    const uint32_t before = v[j], after = v[j + 2];
    const bool cell_start = before != key, cell_end = after != key;
    if (!(cell_start || cell_end)) continue;
    const int s = slot[key >> 9];
    uint2* c = &cr[int64_t(s) * 512 + (key & 511u)];
    if (cell_start) c->x = uint32_t(i);
    if (cell_end) c->y = uint32_t(i + 1);
    if (cell_start && (before >> 9) != (key >> 9)) lr[s].x = uint32_t(i);
    if (cell_end && (after >> 9) != (key >> 9)) lr[s].y = uint32_t(i + 1);
  }
}

// ---- seeding (FlipSimulation::InitializePhiAndParticles restated) -------
struct SeedArgs {
  int npass;
  fsim_seed_pass pass[8];
  uint64_t seed;
  int nppc;
};

__device__ __forceinline__ uint64_t mix64(uint64_t z) {
  z += 0x9E3779B97F4A7C15ull;
  z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
  z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
  return z ^ (z >> 31);
}
__device__ __forceinline__ float uniform01(uint64_t seed, int pass, int64_t cell, int draw,
                                           int d) {
  uint64_t s = mix64(seed ^ mix64((uint64_t(uint32_t(pass)) << 40) ^ uint64_t(cell)));
  uint64_t z = mix64(s + uint64_t(draw * 3 + d));
  return float(z >> 40) * (1.0f / 16777216.0f);
}
__device__ float shape_phi(const fsim_shape& sh, const float p[3]) {
  if (sh.kind == FSIM_SHAPE_CUBOID) {
    bool in = true;
#pragma unroll
    for (int d = 0; d < 3; ++d) in &= (p[d] >= sh.a[d]) & (p[d] <= sh.b[d]);
    return in ? -1.0f : 1.0f;
  } else if (sh.kind == FSIM_SHAPE_SPHERE) {
    float dx = __fsub_rn(p[0], sh.a[0]), dy = __fsub_rn(p[1], sh.a[1]),
          dz = __fsub_rn(p[2], sh.a[2]);
    float l2 = __fadd_rn(__fadd_rn(__fmul_rn(dx, dx), __fmul_rn(dy, dy)), __fmul_rn(dz, dz));
    return __fsub_rn(__fsqrt_rn(l2), sh.r);
  }
  return __fsub_rn(p[1], sh.a[1]);
}
__device__ float pass_phi(const fsim_seed_pass& ps, const float p[3]) {
  float phi = shape_phi(ps.shapes[0], p);
  for (int i = 1; i < ps.nshapes; ++i) phi = fminf(phi, shape_phi(ps.shapes[i], p));
  return phi;
}

// write == 0: count only (warp-aggregated atomic into cnt[5]);
// write == 1: reserve with the same aggregation and emit particles + keys.
__global__ void k_seed(const __grid_constant__ SeedArgs a, LeafMap lm, SolidDesc sd, int write,
                       unsigned long long* __restrict__ counter, float* __restrict__ part,
                       int64_t cap, uint32_t* __restrict__ kout) {
  const int64_t ncell = int64_t(lm.n[0]) * lm.n[1] * lm.n[2];
  int64_t c = int64_t(blockIdx.x) * blockDim.x + threadIdx.x;
  int count = 0;
  int i = 0, j = 0, k = 0;
  const bool active = c < ncell;
  if (active) {
    i = int(c / (int64_t(lm.n[1]) * lm.n[2]));
    j = int((c / lm.n[2]) % lm.n[1]);
    k = int(c % lm.n[2]);
  }
  const bool use = active && !is_solid(sd, i, j, k);
  const float org[3] = {float(i), float(j), float(k)};
  const float ctr[3] = {__fadd_rn(org[0], 0.5f), __fadd_rn(org[1], 0.5f), __fadd_rn(org[2], 0.5f)};
  if (use) {
    for (int ps = 0; ps < a.npass; ++ps) {
      if (!(pass_phi(a.pass[ps], ctr) < 0.f)) continue;
      if (count >= a.nppc) continue;
      int pi = 0, draw = 0;
      for (int att = 0; att < 32 && pi < a.nppc; ++att, ++draw) {
        float pp[3];
#pragma unroll
        for (int d = 0; d < 3; ++d)
          pp[d] = __fadd_rn(org[d], __fmul_rn(uniform01(a.seed, ps, c, draw, d), 1.0f));
        if (pass_phi(a.pass[ps], pp) > 0.f) continue;
        ++pi;
        ++att;
        ++count;
      }
    }
  }
  // warp-aggregated reservation
  const unsigned lane = threadIdx.x & 31;
  int incl = count;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    int v = __shfl_up_sync(0xffffffffu, incl, o);
    if (lane >= unsigned(o)) incl += v;
  }
  const int wtot = __shfl_sync(0xffffffffu, incl, 31);
  unsigned long long base = 0;
  if (lane == 31 && wtot > 0) base = atomicAdd(counter, (unsigned long long)wtot);
  base = __shfl_sync(0xffffffffu, base, 31);
  if (!write || count == 0) return;
  int64_t o = int64_t(base) + incl - count;
  const uint32_t key = cell_key(lm, i, j, k);
  for (int ps = 0; ps < a.npass; ++ps) {
    if (!(pass_phi(a.pass[ps], ctr) < 0.f)) continue;
    // cells already holding nppc particles skip the pass (count is
    // re-derived in the same order as the counting sweep)
    int before = int(o - (int64_t(base) + incl - count));
    if (before >= a.nppc) continue;
    int pi = 0, draw = 0;
    for (int att = 0; att < 32 && pi < a.nppc; ++att, ++draw) {
      float pp[3];
#pragma unroll
      for (int d = 0; d < 3; ++d)
        pp[d] = __fadd_rn(org[d], __fmul_rn(uniform01(a.seed, ps, c, draw, d), 1.0f));
      if (pass_phi(a.pass[ps], pp) > 0.f) continue;
      if (o < cap) {
#pragma unroll
        for (int d = 0; d < 3; ++d) {
          part[d * cap + o] = pp[d];
          part[(3 + d) * cap + o] = a.pass[ps].velocity[d];
          part[(6 + d) * cap + o] = a.pass[ps].velocity[d];
        }
        kout[o] = key;
      }
      ++o;
      ++pi;
      ++att;
    }
  }
}

__global__ void k_perturb(float* __restrict__ part, int64_t cap, int64_t n, float sigma,
                          uint64_t seed) {
  int64_t i = int64_t(blockIdx.x) * blockDim.x + threadIdx.x;
  if (i >= n) return;
#pragma unroll
  for (int d = 0; d < 3; ++d) {
    float u1 = uniform01(seed, 1 << 20, i, 0, d);
    float u2 = uniform01(seed, 1 << 20, i, 1, d);
    float g = sqrtf(-2.0f * logf(1.0f - u1)) * cosf(6.2831853f * u2);
    float v = __fadd_rn(part[(3 + d) * cap + i], __fmul_rn(sigma, g));
    part[(3 + d) * cap + i] = v;
    part[(6 + d) * cap + i] = v;
  }
}

// ---- AddContributionFromSources (common/flip_simulation.cc:1207-1270) ----
// Work items are (source, cell) pairs, sources in order and each source's
// cells x-major, so that particles land in the reference's list order after
// an exclusive scan of the per-item counts.
struct SourceGen {
  int nsrc;
  int lo[FSIM_MAX_SOURCES][3], dim[FSIM_MAX_SOURCES][3];  // cell range of each source
  int64_t begin[FSIM_MAX_SOURCES + 1];                    // first work item of each source
  float blo[FSIM_MAX_SOURCES][3], bhi[FSIM_MAX_SOURCES][3];  // get_box(t)
  float vel[FSIM_MAX_SOURCES][3];
  int pass[FSIM_MAX_SOURCES];
  uint64_t seed;
  int nppc;
};

// count == nullptr: write pass (offsets from the scan)
__global__ void k_source(const __grid_constant__ SourceGen g, LeafMap lm, uint32_t* __restrict__ cnt,
                         const uint32_t* __restrict__ off, float* __restrict__ part, int64_t cap,
                         int64_t base, uint32_t* __restrict__ kout) {
  const int64_t w = int64_t(blockIdx.x) * blockDim.x + threadIdx.x;
  if (w >= g.begin[g.nsrc]) return;
  int q = 0;
  while (w >= g.begin[q + 1]) ++q;
  const int64_t c = w - g.begin[q];
  const int dy = g.dim[q][1], dz = g.dim[q][2];
  const int i = g.lo[q][0] + int(c / (int64_t(dy) * dz));
  const int j = g.lo[q][1] + int((c / dz) % dy);
  const int k = g.lo[q][2] + int(c % dz);
  const int64_t cell = (int64_t(i) * lm.n[1] + j) * lm.n[2] + k;
  const float org[3] = {float(i), float(j), float(k)};
  int pi = 0;
  int64_t o = cnt ? 0 : base + off[w];
  const uint32_t key = cell_key(lm, i, j, k);
  for (int att = 0; att < 32 && pi < g.nppc; ++att) {
    float pp[3];
    bool in = true;
#pragma unroll
    for (int d = 0; d < 3; ++d) {
      pp[d] = __fadd_rn(org[d], __fmul_rn(uniform01(g.seed, g.pass[q], cell, att, d), 1.0f));
      in &= (pp[d] >= g.blo[q][d]) & (pp[d] <= g.bhi[q][d]);
    }
    if (!in) continue;
    if (!cnt) {
#pragma unroll
      for (int d = 0; d < 3; ++d) {
        part[d * cap + o] = pp[d];
        part[(3 + d) * cap + o] = g.vel[q][d];
        part[(6 + d) * cap + o] = g.vel[q][d];
      }
      kout[o] = key;
      ++o;
    }
    ++pi;
  }
  if (cnt) cnt[w] = uint32_t(pi);
}

// DeleteFluidInSources on sorted particles (per-stage entry): dead keys
__global__ void k_delete_in_regions(const float* __restrict__ part, int64_t cap,
                                    uint32_t* __restrict__ keys, int64_t n,
                                    const SourceRegions reg,
                                    unsigned long long* __restrict__ ndead) {
  const int64_t i = int64_t(blockIdx.x) * blockDim.x + threadIdx.x;
  if (i >= n || keys[i] == kDeadKey) return;
  const float p[3] = {part[i], part[cap + i], part[2 * cap + i]};
  if (in_regions(reg, p)) {
    keys[i] = kDeadKey;
    atomicAdd(ndead, 1ull);
  }
}

// adjacent pairs out of order (k[i] > k[i+1])
__global__ void k_count_desc(const uint32_t* __restrict__ k, int64_t n,
                             unsigned long long* __restrict__ cnt) {
  const int64_t i = int64_t(blockIdx.x) * blockDim.x + threadIdx.x;
  if (i + 1 < n && k[i] > k[i + 1]) atomicAdd(cnt, 1ull);
}

__global__ void k_hi_keys(const unsigned long long* __restrict__ k64, uint32_t* __restrict__ k,
                          int64_t n) {
  const int64_t i = int64_t(blockIdx.x) * blockDim.x + threadIdx.x;
  if (i < n) k[i] = uint32_t(k64[i] >> 32);
}

inline unsigned nblk(int64_t n, int b) { return unsigned((n + b - 1) / b); }

SourceRegions regions_at(const fsim_sim* s, float t) {
  SourceRegions r;
  memset(&r, 0, sizeof(r));
  r.n = int(s->sources.size());
  for (int q = 0; q < r.n; ++q) source_box(s->sources[size_t(q)], t, r.lo[q], r.hi[q]);
  return r;
}

}  // namespace

// stable radix sort of (key, value) pairs by cell key
static int sort_pairs(fsim_sim* s, const uint32_t* kin, uint32_t* kout, const uint32_t* vin,
                      uint32_t* vout, int64_t n) {
  const int bits = key_bits(s->lm);
  size_t need = 0;
  FSIM_CK(s, cub::DeviceRadixSort::SortPairs(nullptr, need, kin, kout, vin, vout, n, 0, bits,
                                             s->stream));
  if (need > s->sort_tmp_bytes) {
    if (s->sort_tmp) cudaFree(s->sort_tmp);
    s->sort_tmp = nullptr;
    s->sort_tmp_bytes = 0;
    FSIM_CK(s, cudaMalloc(&s->sort_tmp, need));
    s->sort_tmp_bytes = need;
  }
  if (n > 0) {
    fsim::ProfScope ps(s, "radix_sort(cub)");
    FSIM_CK(s, cub::DeviceRadixSort::SortPairs(s->sort_tmp, need, kin, kout, vin, vout, n, 0, bits,
                                               s->stream));
  }
  return FSIM_OK;
}

static int ensure_keys64(fsim_sim* s, int64_t n) {
  if (n <= s->cap64) return FSIM_OK;
  s->cap64 = 0;
  for (int b = 0; b < 2; ++b) {
    if (s->keys64[b]) cudaFree(s->keys64[b]);
    s->keys64[b] = nullptr;
    FSIM_CK(s, cudaMalloc(&s->keys64[b], size_t(std::max<int64_t>(n, 1)) * 8));
  }
  s->cap64 = n;
  return FSIM_OK;
}

int launch_host_keys(fsim_sim* s, const float* pos, const float* gvel, float dt, bool keep_gvel,
                     int64_t* invalid) {
  const int64_t n = s->n_total;
  unsigned long long* cnt = reinterpret_cast<unsigned long long*>(s->d_cnt);
  FSIM_CK(s, cudaMemsetAsync(s->d_cnt + 3, 0, 5 * sizeof(int64_t), s->stream));
  FSIM_CK(s, cudaMemsetAsync(s->d_lcnt, 0, size_t(s->lm.dense) * 4, s->stream));
  FSIM_LAUNCH(s, "advect_keys", k_host_keys, nblk(n, 256), 256, 0, pos, gvel, s->part[s->cur],
              s->cap_p, s->keys[0], s->keys[1], n, s->lm, s->solid, dt, keep_gvel ? 1 : 0, cnt + 3,
              cnt + 7, s->d_lcnt);
  FSIM_CK(s, cudaMemcpyAsync(s->h_cnt + 3, s->d_cnt + 3, 5 * sizeof(int64_t),
                             cudaMemcpyDeviceToHost, s->stream));
  FSIM_CK(s, cudaStreamSynchronize(s->stream));
  *invalid = s->h_cnt[3];
  // rows out of cell order: their old cells decide the order within a new cell
  s->composite_sort = s->h_cnt[7] != 0;
  return FSIM_OK;
}

int launch_keys_from_positions(fsim_sim* s, int mode, float dt) {
  const int64_t n = s->n_total;
  FSIM_CK(s, cudaMemsetAsync(s->d_cnt + 3, 0, sizeof(int64_t), s->stream));
  FSIM_CK(s, cudaMemsetAsync(s->d_lcnt, 0, size_t(s->lm.dense) * 4, s->stream));
  if (mode == 0) s->composite_sort = false;  // new particles: no old cells
  SourceRegions reg;
  memset(&reg, 0, sizeof(reg));
  if (mode == 1 && s->delete_in_sources) reg = regions_at(s, s->src_time);
  FSIM_LAUNCH(s, "advect_keys", k_keys, nblk(n, 256), 256, 0, s->part[s->cur], s->cap_p,
              s->keys[0], s->keys[1], n, s->lm, s->solid, mode, dt,
              reinterpret_cast<unsigned long long*>(s->d_cnt + 3), reg, s->d_lcnt);
  s->delete_in_sources = false;
  return FSIM_OK;
}

// the bins of k_bin_rows besides the row numbers (those are in vals[1])
static int ensure_bins(fsim_sim* s, bool old) {
  const size_t need = size_t(s->cap_p) * (old ? 6 : 2) + 256;
  if (need <= s->bin_bytes) return FSIM_OK;
  if (s->bins) cudaFree(s->bins);
  s->bins = nullptr;
  s->bin_bytes = 0;
  FSIM_CK(s, cudaMalloc(&s->bins, need));
  s->bin_bytes = need;
  return FSIM_OK;
}

// keys[1] (with keys[0] as the old keys: OLD) into keys[0] and the rows' order
// into vals[0]
template <bool OLD>
static int sort_by_leaf(fsim_sim* s) {
  const int64_t n = s->n_total;
  const int rc = ensure_bins(s, OLD);
  if (rc) return rc;
  uint16_t* cell = static_cast<uint16_t*>(s->bins);
  uint32_t* old = OLD ? reinterpret_cast<uint32_t*>(static_cast<char*>(s->bins) +
                                                    (size_t(s->cap_p) * 2 + 255) / 256 * 256)
                      : nullptr;
  constexpr size_t smem = size_t(kLeafSort) * sizeof(SortEntry<OLD>);
  FSIM_CK(s, cudaFuncSetAttribute(k_sort_leaf<OLD>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                  int(smem)));
  FSIM_LAUNCH(s, "bin_rows", k_bin_rows<OLD>, nblk(n, 1024), 256, 0, s->keys[1], s->keys[0], n,
              s->d_lnext, s->vals[1], old, cell);
  FSIM_LAUNCH(s, "sort_leaves", k_sort_leaf<OLD>, 2 * s->num_sms, kLeafSortThreads, smem,
              s->d_leaf_id, s->d_cnt, s->d_lcnt, s->d_lnext, s->vals[1], old, cell, s->keys[0],
              s->vals[0]);
  return FSIM_OK;
}

// The same order by the library's radix sort, for a state with a leaf of more
// than kLeafSort particles (keys[0] and keys[1] are as they were).
static int sort_by_library(fsim_sim* s, bool old) {
  const int64_t n = s->n_total;
  FSIM_LAUNCH(s, "sort_rows", k_rows, nblk(n, 256), 256, 0, s->vals[1], n);
  if (!old) return sort_pairs(s, s->keys[1], s->keys[0], s->vals[1], s->vals[0], n);
  // stable sort on (new key << 32 | old key), then the new keys back
  const int bits = key_bits(s->lm);
  int rc = ensure_keys64(s, n);
  if (rc) return rc;
  unsigned long long* k64[2] = {reinterpret_cast<unsigned long long*>(s->keys64[0]),
                                reinterpret_cast<unsigned long long*>(s->keys64[1])};
  FSIM_LAUNCH(s, "join_keys", k_join_keys, nblk(n, 256), 256, 0, s->keys[1], s->keys[0], k64[1], n);
  size_t need = 0;
  FSIM_CK(s, cub::DeviceRadixSort::SortPairs(nullptr, need, k64[1], k64[0], s->vals[1], s->vals[0],
                                             n, 0, 32 + bits, s->stream));
  if (need > s->sort_tmp_bytes) {
    if (s->sort_tmp) cudaFree(s->sort_tmp);
    s->sort_tmp = nullptr;
    s->sort_tmp_bytes = 0;
    FSIM_CK(s, cudaMalloc(&s->sort_tmp, need));
    s->sort_tmp_bytes = need;
  }
  {
    fsim::ProfScope ps(s, "radix_sort64(cub)");
    FSIM_CK(s, cub::DeviceRadixSort::SortPairs(s->sort_tmp, need, k64[1], k64[0], s->vals[1],
                                               s->vals[0], n, 0, 32 + bits, s->stream));
  }
  FSIM_LAUNCH(s, "new_keys", k_hi_keys, nblk(n, 256), 256, 0, k64[0], s->keys[0], n);
  return FSIM_OK;
}

// Permutes the particles by vals[0] into the other buffer.
static int gather_particles(fsim_sim* s) {
  const int64_t n = s->n_total;
  // a velocity upload still in flight on the I/O stream (fsim_step_host)
  if (s->io_vel_pending) {
    FSIM_CK(s, cudaStreamWaitEvent(s->stream, s->ev_io, 0));
    s->io_vel_pending = false;
  }
  if (s->gather_skip_gvel) {
    FSIM_LAUNCH(s, "gather_particles", k_gather<6>, nblk(n, 256), 256, 0, s->part[s->cur],
                s->part[s->cur ^ 1], s->cap_p, s->vals[0], s->d_cnt);
  } else {
    FSIM_LAUNCH(s, "gather_particles", k_gather<9>, nblk(n, 256), 256, 0, s->part[s->cur],
                s->part[s->cur ^ 1], s->cap_p, s->vals[0], s->d_cnt);
  }
  return FSIM_OK;
}

// The leaf topology of the n_total particles whose keys are in keys[1] and
// counted in d_lcnt; sort: and their order (keys[0], vals[0]) and the
// particles in it, else keys[0] holds the keys in order already.
static int rebuild(fsim_sim* s, bool sort) {
  const uint32_t D = s->lm.dense;
  const unsigned tiles = nblk(int64_t(D), kLeafTile);
  FSIM_LAUNCH(s, "leaf_flags", k_leaf_flags, tiles, kLeafTile, 0, s->d_lcnt, s->d_flag, s->d_tile,
              s->lm);
  FSIM_LAUNCH(s, "leaf_slots", k_leaf_slots, tiles, kLeafTile, 0, s->d_lcnt, s->d_flag, s->d_tile,
              s->d_slot, s->d_leaf_id, s->d_lnext, D, s->d_cnt);
  // the host reads the counts while the sort runs
  FSIM_CK(s, cudaMemcpyAsync(s->h_cnt, s->d_cnt, 3 * sizeof(int64_t), cudaMemcpyDeviceToHost,
                             s->stream));
  FSIM_CK(s, cudaEventRecord(s->ev_topo, s->stream));
  int rc;
  const bool old = s->composite_sort;
  if (sort && s->n_total > 0) {
    if ((rc = old ? sort_by_leaf<true>(s) : sort_by_leaf<false>(s))) return rc;
    if ((rc = gather_particles(s))) return rc;
  }
  FSIM_CK(s, cudaEventSynchronize(s->ev_topo));
  if (sort) {
    if (s->n_total > 0 && (s->h_cnt[1] & kLeafOverflow)) {
      s->h_cnt[1] &= kLeafOverflow - 1;
      FSIM_CK(s, cudaMemcpyAsync(s->d_cnt + 1, s->h_cnt + 1, sizeof(int64_t),
                                 cudaMemcpyHostToDevice, s->stream));
      if ((rc = sort_by_library(s, old))) return rc;
      if ((rc = gather_particles(s))) return rc;
    }
    s->cur ^= 1;
  }
  s->composite_sort = false;
  s->n_live = s->h_cnt[0];
  s->n_total = s->n_live;
  s->n_pleaf = int(s->h_cnt[1] & (kLeafOverflow - 1));
  s->n_gleaf = int(s->h_cnt[2]);
  rc = ensure_leaf_capacity(s, s->n_gleaf, s->n_pleaf);
  if (rc != FSIM_OK) return rc;
  FSIM_LAUNCH(s, "neighbour_table", k_nbr, nblk(int64_t(s->n_gleaf) * 27, 256), 256, 0,
              s->d_leaf_id, s->d_slot, s->d_nbr, s->n_gleaf, s->lm);
  if (s->n_pleaf > 0) {
    FSIM_CK(s, cudaMemsetAsync(s->d_cell_range, 0, size_t(s->n_pleaf) * 512 * sizeof(uint2),
                               s->stream));
    FSIM_CK(s, cudaMemsetAsync(s->d_leaf_range, 0, size_t(s->n_pleaf) * sizeof(uint2), s->stream));
  }
  FSIM_LAUNCH(s, "cell_ranges", k_ranges, nblk(s->n_live, 256 * kKeysPerThread), 256, 0, s->keys[0], s->d_cnt,
              s->d_slot, s->d_cell_range, s->d_leaf_range);
  s->have_topology = true;
  s->ranges_match = true;
  s->deleted_outside = false;
  return FSIM_OK;
}

int rebuild_topology(fsim_sim* s) { return rebuild(s, true); }

int seed_fluid(fsim_sim* s, const fsim_seed_pass* passes, int npasses, uint64_t seed) {
  if (npasses < 0 || npasses > 8) return fail(s, FSIM_ERR_INVALID, "npasses must be in [0,8]");
  SeedArgs a;
  memset(&a, 0, sizeof(a));
  a.npass = npasses;
  for (int i = 0; i < npasses; ++i) {
    if (passes[i].nshapes < 1 || passes[i].nshapes > FSIM_MAX_SHAPES)
      return fail(s, FSIM_ERR_INVALID, "each seed pass needs 1..8 shapes");
    a.pass[i] = passes[i];
  }
  a.seed = seed;
  a.nppc = s->cfg.nparticles_per_cell;
  const int64_t ncell = int64_t(s->lm.n[0]) * s->lm.n[1] * s->lm.n[2];
  unsigned long long* ctr = reinterpret_cast<unsigned long long*>(s->d_cnt + 5);
  FSIM_CK(s, cudaMemsetAsync(ctr, 0, sizeof(int64_t), s->stream));
  FSIM_LAUNCH(s, "seed_count", k_seed, nblk(ncell, 256), 256, 0, a, s->lm, s->solid, 0, ctr,
              s->part[s->cur], s->cap_p, s->keys[1]);
  FSIM_CK(s, cudaMemcpyAsync(s->h_cnt + 5, s->d_cnt + 5, sizeof(int64_t), cudaMemcpyDeviceToHost,
                             s->stream));
  FSIM_CK(s, cudaStreamSynchronize(s->stream));
  const int64_t total = s->h_cnt[5];
  if (total > s->cap_p)
    return fail(s, FSIM_ERR_CAPACITY, "seeded particle count exceeds max_particles");
  FSIM_CK(s, cudaMemsetAsync(ctr, 0, sizeof(int64_t), s->stream));
  FSIM_LAUNCH(s, "seed_write", k_seed, nblk(ncell, 256), 256, 0, a, s->lm, s->solid, 1, ctr,
              s->part[s->cur], s->cap_p, s->keys[1]);
  s->n_total = total;
  s->composite_sort = false;
  FSIM_CK(s, cudaMemsetAsync(s->d_lcnt, 0, size_t(s->lm.dense) * 4, s->stream));
  FSIM_LAUNCH(s, "seed_leaves", k_count_leaves, nblk(total, 256), 256, 0, s->keys[1], total, s->d_lcnt);
  return rebuild_topology(s);
}

// Upload helper: keys (mode 0) are in keys[1]; when they are already in cell
// order (particles that came from a download) the sort and the gather are
// skipped.  Returns FSIM_OK and sets *invalid to the number of positions
// outside [0, N].
int rebin_uploaded(fsim_sim* s, int64_t* invalid) {
  const int64_t n = s->n_total;
  FSIM_CK(s, cudaMemsetAsync(s->d_cnt + 7, 0, sizeof(int64_t), s->stream));
  FSIM_LAUNCH(s, "count_unsorted", k_count_desc, nblk(n, 256), 256, 0, s->keys[1], n,
              reinterpret_cast<unsigned long long*>(s->d_cnt + 7));
  FSIM_CK(s, cudaMemcpyAsync(s->h_cnt + 3, s->d_cnt + 3, 5 * sizeof(int64_t),
                             cudaMemcpyDeviceToHost, s->stream));
  FSIM_CK(s, cudaStreamSynchronize(s->stream));
  *invalid = s->h_cnt[3];
  if (*invalid) return FSIM_OK;
  if (s->h_cnt[7] == 0) {
    std::swap(s->keys[0], s->keys[1]);  // sorted already: keep the order
    return rebuild(s, false);
  }
  return rebuild_topology(s);
}

int add_source_particles(fsim_sim* s, float t) {
  SourceGen g;
  memset(&g, 0, sizeof(g));
  g.seed = s->seed;
  g.nppc = s->cfg.nparticles_per_cell;
  const int64_t call = s->source_calls++;
  int64_t items = 0;
  for (size_t q = 0; q < s->sources.size(); ++q) {
    const fsim_source& src = s->sources[q];
    g.begin[g.nsrc] = items;
    if (!source_active(src, t)) continue;
    float lo[3], hi[3];
    source_box(src, t, lo, hi);
    int a[3], b[3];
    bool empty = false;
    for (int d = 0; d < 3; ++d) {
      // Coord(float) truncates; the domain box is [0, N-1]
      a[d] = std::max(int(lo[d]), 0);
      b[d] = std::min(int(hi[d]), s->lm.n[d] - 1);
      empty |= b[d] < a[d];
    }
    if (empty) continue;
    const int r = g.nsrc;
    for (int d = 0; d < 3; ++d) {
      g.lo[r][d] = a[d];
      g.dim[r][d] = b[d] - a[d] + 1;
      g.blo[r][d] = lo[d];
      g.bhi[r][d] = hi[d];
    }
    source_velocity(src, t, g.vel[r]);
    g.pass[r] = (1 << 22) + int((call & 0x1FFFF) * 32) + int(q);
    g.begin[r] = items;
    items += int64_t(g.dim[r][0]) * g.dim[r][1] * g.dim[r][2];
    ++g.nsrc;
  }
  g.begin[g.nsrc] = items;
  if (items == 0) return FSIM_OK;
  // counts, exclusive scan, then the particles after the current ones
  size_t sneed = 0;
  uint32_t* cnt = nullptr;
  FSIM_CK(s, cub::DeviceScan::ExclusiveSum(nullptr, sneed, cnt, cnt, int(items + 1), s->stream));
  const size_t cnt_bytes = ((size_t(items + 1) * 4 + 255) / 256) * 256;
  if (cnt_bytes * 2 + sneed > s->src_tmp_bytes) {
    if (s->src_tmp) cudaFree(s->src_tmp);
    s->src_tmp = nullptr;
    FSIM_CK(s, cudaMalloc(&s->src_tmp, cnt_bytes * 2 + sneed));
    s->src_tmp_bytes = cnt_bytes * 2 + sneed;
  }
  cnt = static_cast<uint32_t*>(s->src_tmp);
  uint32_t* off = reinterpret_cast<uint32_t*>(static_cast<char*>(s->src_tmp) + cnt_bytes);
  void* stmp = static_cast<char*>(s->src_tmp) + 2 * cnt_bytes;
  FSIM_CK(s, cudaMemsetAsync(cnt, 0, size_t(items + 1) * 4, s->stream));
  FSIM_LAUNCH(s, "source_count", k_source, nblk(items, 256), 256, 0, g, s->lm, cnt,
              static_cast<const uint32_t*>(nullptr), s->part[s->cur], s->cap_p, int64_t(0),
              s->keys[0]);
  FSIM_CK(s, cub::DeviceScan::ExclusiveSum(stmp, sneed, cnt, off, int(items + 1), s->stream));
  uint32_t added = 0;
  FSIM_CK(s, cudaMemcpyAsync(&added, off + items, 4, cudaMemcpyDeviceToHost, s->stream));
  FSIM_CK(s, cudaStreamSynchronize(s->stream));
  if (added == 0) return FSIM_OK;
  if (s->n_total + int64_t(added) > s->cap_p) {
    // grow by a quarter more than needed (sources keep adding); the current
    // particles and keys move over
    const int rc = grow_particle_capacity(s, (s->n_total + int64_t(added)) * 5 / 4 + 1024);
    if (rc) return rc;
  }
  FSIM_LAUNCH(s, "source_write", k_source, nblk(items, 256), 256, 0, g, s->lm,
              static_cast<uint32_t*>(nullptr), off, s->part[s->cur], s->cap_p, s->n_total,
              s->keys[0]);
  s->n_total += added;
  s->n_live = s->n_total;
  s->composite_sort = true;
  return FSIM_OK;
}

int delete_in_sources(fsim_sim* s, float t) {
  if (s->sources.empty()) return FSIM_OK;
  // dead keys are counted with DeleteOutsideParticles' (d_cnt[6]) until the next sort
  if (!s->deleted_outside) FSIM_CK(s, cudaMemsetAsync(s->d_cnt + 6, 0, 8, s->stream));
  FSIM_LAUNCH(s, "delete_in_sources", k_delete_in_regions, nblk(s->n_total, 256), 256, 0,
              s->part[s->cur], s->cap_p, s->keys[0], s->n_total, regions_at(s, t),
              reinterpret_cast<unsigned long long*>(s->d_cnt + 6));
  return FSIM_OK;
}

int perturb(fsim_sim* s, float sigma, uint64_t seed) {
  FSIM_LAUNCH(s, "perturb_velocity", k_perturb, nblk(s->n_live, 256), 256, 0, s->part[s->cur],
              s->cap_p, s->n_live, sigma, seed);
  return FSIM_OK;
}

}  // namespace fsim
