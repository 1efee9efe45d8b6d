// pcg_cluster.cuh -- the PCG loop of small systems in one thread-block cluster
// (included by k_pcg.cu, inside its namespace).
//
// A small system's iteration is latency: the spmv / update pair spends 6.4 to
// 6.9 us on two launches whatever the size (24 to 160 particle leaves), and
// the resident loop's grid barriers go through L2 as well.  Here one cluster
// of kClCtas CTAs, one per SM, holds the whole system: a warp owns a leaf
// for the whole solve, a lane two of its z-columns (x-neighbours: three
// neighbour columns are read per own column instead of four, and shared
// memory bandwidth is what bounds the larger systems here), with r, z, p
// and x in registers and p in shared memory too.
// Every exchange of an iteration stays inside the cluster:
//   S: p = z + beta p on the own columns and on the columns of other CTAs'
//      leaves that touch them (kept here too, formed with the owner's
//      operations from its z, read through distributed shared memory);
//      CTA barrier; A p from local shared memory; p.Ap -> alpha
//   U: x += alpha p, r -= alpha A p, z = M r (also left in shared memory for
//      the other CTAs); r.r, r.z -> beta and the loop test.
// A dot product goes up by warp shuffles and a CTA barrier; warp 0 then pushes
// the CTA's partial to every CTA as a 64-bit word that carries the round
// number, polls the 16 words that its own CTA receives and adds them in CTA
// order.  So a reduction crosses the cluster once, one way (about 320 cycles;
// a hardware cluster barrier with release and acquire takes 400 to 515, and
// the full fences that a push needs with it 290 each), the words of U publish
// z as well (fences restricted to shared memory, 30 and 23 cycles), and every
// CTA gets the same bits: a solve repeats bit for bit.  (A push by every warp,
// with every warp polling, measured slower: 3.99 against 3.2 us per
// iteration at 64^3.)  Element-wise arithmetic is the pair's; only the order
// of the dot products differs.  Scalars stay off the narrow FP64 pipe: fp32
// for FP32 (as the reference); for MIXED the totals are double-float pairs, as
// the pair's, and alpha and beta the roundings of their fp64 quotients
// (pcg_scalar.cuh).
// Measured us per iteration, against the pair (sphere drop; particle leaves):
//   leaves        24          84          156         189
//   FP32     2.13 / 6.57  2.62 / 6.42  3.13 / 6.51  3.36 / 6.48
//   MIXED    3.46 / 10.1  4.08 / 9.32  4.78 / 9.17  4.94 / 9.51
// (the resident loop: 3.7 to 4.2 for FP32, 5.1 to 5.6 for MIXED).  At 24
// leaves it is latency (two one-way pushes, four CTA barriers, six warp
// reductions); from about 100 on also the bandwidth of shared memory (156
// leaves: its SMs issue in 28% of their cycles, MIXED 37%, and wait for CTA
// barriers first, then for shared memory).
//
// The polls are bounded (kClPolls): a CTA whose wait gives up leaves the loop,
// the other CTAs' waits run out in turn, and all meet at a last cluster
// barrier, so no CTA's shared memory goes while another may still reach it.
constexpr int kClCtas = 16;                       // CTAs of the cluster (one per SM)
constexpr int kClWarps = 12;                      // warps per CTA, at most (168 registers)
// leaves per warp: one, since p, x and the inverse diagonal are kept for one
// (written as loops over them all the same: without, the compiler's schedule
// takes 2.38 us per iteration at 24 leaves instead of 2.13)
constexpr int kClPerWarp = 1;
static_assert(kClPerWarp == 1, "Pc, X and inv hold one leaf's columns");
constexpr int kClLeaves = kClCtas * kClWarps * kClPerWarp;  // 192 particle leaves
constexpr unsigned kClPolls = 1u << 22;

// p of a CTA's leaves in shared memory (here and in the resident loop), in 16-byte chunk planes: float4 element
// ((leaf * 2 + chunk) * 8 + x) * 8 + y holds the cells z = 4 chunk ..
// 4 chunk + 3 of column (x, y), so the lanes of a quarter warp (consecutive
// y) touch consecutive 16-byte words.  ps_col4 is the float4 index of chunk 0
// of a column; chunk 1 is 64 further, and the in-leaf neighbour columns are
// -8 / +8 (x) and -1 / +1 (y) away, constant offsets from the own column.
__device__ __forceinline__ int ps_col4(int leaf, int x, int y) { return (leaf * 16 + x) * 8 + y; }
__device__ __forceinline__ void ps_ld4(const float* ps, int i, Col<float>& c) {
  const float4* q = reinterpret_cast<const float4*>(ps);
  const float4 u = q[i], w = q[i + 64];
  c.v[0] = u.x; c.v[1] = u.y; c.v[2] = u.z; c.v[3] = u.w;
  c.v[4] = w.x; c.v[5] = w.y; c.v[6] = w.z; c.v[7] = w.w;
}
__device__ __forceinline__ void ps_st4(float* ps, int i, const Col<float>& c) {
  float4* q = reinterpret_cast<float4*>(ps);
  q[i] = make_float4(c.v[0], c.v[1], c.v[2], c.v[3]);
  q[i + 64] = make_float4(c.v[4], c.v[5], c.v[6], c.v[7]);
}

__device__ __forceinline__ unsigned cl_rank() {
  unsigned r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;\n" : "=r"(r));
  return r;
}
__device__ __forceinline__ unsigned cl_map(unsigned saddr, unsigned rank) {
  unsigned d;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;\n" : "=r"(d) : "r"(saddr), "r"(rank));
  return d;
}
__device__ __forceinline__ void cl_sync() {
  asm volatile(
      "barrier.cluster.arrive.release.aligned;\n"
      "barrier.cluster.wait.acquire.aligned;\n" ::
          : "memory");
}
// release of this CTA's shared memory to the cluster, and the acquire of the
// other CTAs' (around the relaxed words of cl_sum)
__device__ __forceinline__ void cl_release() {
  asm volatile("fence.release.sync_restrict::shared::cta.cluster;\n" ::: "memory");
}
__device__ __forceinline__ void cl_acquire() {
  asm volatile("fence.acquire.sync_restrict::shared::cluster.cluster;\n" ::: "memory");
}
__device__ __forceinline__ void cl_ldcol(unsigned addr, Col<float>& c) {
  asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];\n"
               : "=f"(c.v[0]), "=f"(c.v[1]), "=f"(c.v[2]), "=f"(c.v[3])
               : "r"(addr)
               : "memory");
  asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4 + 1024];\n"
               : "=f"(c.v[4]), "=f"(c.v[5]), "=f"(c.v[6]), "=f"(c.v[7])
               : "r"(addr)
               : "memory");
}
__device__ __forceinline__ float cl_ldcell(unsigned addr) {
  float v;
  asm volatile("ld.shared::cluster.f32 %0, [%1];\n" : "=f"(v) : "r"(addr) : "memory");
  return v;
}

template <typename P>
__device__ __forceinline__ P pshfl_xor(P v, int o);
template <>
__device__ __forceinline__ double pshfl_xor<double>(double v, int o) {
  return __shfl_xor_sync(0xffffffffu, v, o);
}
template <>
__device__ __forceinline__ float pshfl_xor<float>(float v, int o) {
  return __shfl_xor_sync(0xffffffffu, v, o);
}
template <>
__device__ __forceinline__ float2 pshfl_xor<float2>(float2 v, int o) {
  return make_float2(__shfl_xor_sync(0xffffffffu, v.x, o), __shfl_xor_sync(0xffffffffu, v.y, o));
}

// Words of a partial: its 32-bit parts, each beside the round number.
__device__ __forceinline__ unsigned long long cl_word(float v, unsigned tag) {
  return (static_cast<unsigned long long>(tag) << 32) | __float_as_uint(v);
}
__device__ __forceinline__ float cl_part(const float& v, int) { return v; }
__device__ __forceinline__ float cl_part(const float2& v, int q) { return q ? v.y : v.x; }
__device__ __forceinline__ void cl_set(float& v, int, float f) { v = f; }
__device__ __forceinline__ void cl_set(float2& v, int q, float f) {
  if (q) v.y = f; else v.x = f;
}

struct ClFrame {
  int W, Wp;       // warps per CTA, and the power of two at or above it
  int warp, lane;
  unsigned limit;  // polls before a wait gives up
  bool mute;       // tests: this CTA pushes nothing in the first round
};

// Sums of NV values over the cluster, the same bits in every thread: warps by
// shuffles, the CTA by its warp 0 (wp), which pushes the CTA's partial to
// every CTA (lane c to CTA c, at dst), polls the words its own CTA receives
// (from src, one CTA per lane) and leaves the total in tot.  The words of
// p.Ap and of r.r, r.z are apart, and each is only rewritten after every CTA
// has pushed the other, and so has read it; so are wp and tot.  PUBLISH: what
// the CTA's threads wrote to shared memory before the call is visible to every
// thread of the cluster after it.  True when the wait gave up, in every thread
// of the CTA.
template <typename P, int NV, bool PUBLISH>
__device__ __forceinline__ bool cl_sum(P (&v)[NV], P* wp, P* tot, const ClFrame& c, unsigned dst,
                                       unsigned src, unsigned tag) {
  constexpr int NW = NV * int(sizeof(P) / 4);  // words per partial
#pragma unroll
  for (int o = 16; o > 0; o >>= 1)
#pragma unroll
    for (int k = 0; k < NV; ++k) v[k] = padd(v[k], pshfl_xor(v[k], o));
  if (c.lane == 0) {
#pragma unroll
    for (int k = 0; k < NV; ++k) wp[k * kClWarps + c.warp] = v[k];
  }
  __syncthreads();
  bool bad = false;
  if (c.warp == 0) {
    const int i = c.lane & (c.Wp - 1);
#pragma unroll
    for (int k = 0; k < NV; ++k) v[k] = i < c.W ? wp[k * kClWarps + i] : pzero<P>();
#pragma unroll
    for (int o = 8; o > 0; o >>= 1) {
      if (o >= c.Wp) continue;
#pragma unroll
      for (int k = 0; k < NV; ++k) v[k] = padd(v[k], pshfl_xor(v[k], o));
    }
    if (PUBLISH) cl_release();
    if (c.lane < kClCtas && !(c.mute && tag == 1u)) {
#pragma unroll
      for (int q = 0; q < NW; ++q)
        asm volatile("st.relaxed.cluster.shared::cluster.u64 [%0], %1;\n" ::"r"(dst + 8u * q),
                     "l"(cl_word(cl_part(v[q * NV / NW], q % (NW / NV)), tag))
                     : "memory");
    }
    __syncwarp();
    unsigned polls = 0;
    for (;;) {
      bool ok = true;
#pragma unroll
      for (int q = 0; q < NW; ++q) {
        unsigned long long m;
        asm volatile("ld.relaxed.cluster.shared::cta.u64 %0, [%1];\n"
                     : "=l"(m)
                     : "r"(src + 8u * q)
                     : "memory");
        ok = ok && unsigned(m >> 32) == tag;
        cl_set(v[q * NV / NW], q % (NW / NV), __uint_as_float(unsigned(m)));
      }
      if (__all_sync(0xffffffffu, ok)) break;
      if (++polls > c.limit) {
        bad = true;
        break;
      }
    }
    if (PUBLISH) cl_acquire();
#pragma unroll
    for (int o = kClCtas / 2; o > 0; o >>= 1)
#pragma unroll
      for (int k = 0; k < NV; ++k) v[k] = padd(v[k], pshfl_xor(v[k], o));
    if (c.lane == 0) {
#pragma unroll
      for (int k = 0; k < NV; ++k) tot[k] = v[k];
    }
  }
  bad = __syncthreads_or(bad);
#pragma unroll
  for (int k = 0; k < NV; ++k) v[k] = tot[k];
  return bad;
}

#include "pcg_scalar.cuh"

// T(diag) of a flags byte: the small integer as the low mantissa bits of 2^23,
// less 2^23 (exact)
__device__ __forceinline__ float cl_diag(unsigned g) {
  return __fsub_rn(__uint_as_float(0x4B000000u | ((g >> 1) & 7u)), 8388608.f);
}

// The loop test in the partials' type: r.r <= thr (RELATIVE) or the fp32
// r.r < thr (ABSOLUTE, as the reference).  A float r.r is at most a double
// thr exactly when it is at most thr rounded down.
template <typename P>
struct ClStop {
  P thr;
  bool fixed, strict;
};
template <typename P>
__device__ __forceinline__ ClStop<P> cl_stop_of(const PcgScalars* sc) {
  ClStop<P> q;
  q.fixed = sc->mode == FSIM_PCG_FIXED;
  q.strict = sc->mode == FSIM_PCG_ABSOLUTE;
  if constexpr (std::is_same<P, float>::value)
    q.thr = q.strict ? float(sc->thr) : __double2float_rd(sc->thr);
  else if constexpr (std::is_same<P, float2>::value)
    cl_threshold(sc->thr, q.thr);
  else
    q.thr = sc->thr;
  return q;
}
__device__ __forceinline__ bool cl_stop(const ClStop<double>& q, double rr) {
  return !q.fixed && (q.strict ? rr < q.thr : rr <= q.thr);
}
__device__ __forceinline__ bool cl_stop(const ClStop<float>& q, float rr) {
  return !q.fixed && (q.strict ? rr < q.thr : rr <= q.thr);
}
__device__ __forceinline__ bool cl_stop(const ClStop<float2>& q, float2 rr) {
  return !q.fixed && cl_at_most(rr, q.thr);
}

// Shared memory of a CTA with W warps, a leaf each: p of its leaves and a zero
// leaf for missing neighbours, z of its leaves, the halo columns (32 per leaf:
// -x, +x faces by y; then -y, +y faces, column x at 16 + x / 2 + 8 (x & 1) and
// 4 further for +y, so that a lane's second column is 8 further, as in a
// leaf) in blocks of 64 columns, all in the resident loop's chunk planes; the
// halo's z cells ([-z, +z][64] per leaf, a lane's second 32 further); where
// each lane's halo comes from.
struct ClLayout {
  unsigned ps, zs, halo, zc, src, bytes;
};
__host__ __device__ inline ClLayout cl_layout(int W) {
  ClLayout l;
  const unsigned nl = unsigned(W * kClPerWarp);
  l.ps = 0;
  l.zs = l.ps + (nl + 1) * 2048u;
  l.halo = l.zs + nl * 2048u;
  l.zc = l.halo + (nl + 1) / 2 * 2048u;
  l.src = l.zc + nl * 512u;
  l.bytes = l.src + nl * 512u;
  return l;
}

template <int DM>
__global__ void __launch_bounds__(kClWarps * 32, 1)
    k_pcg_cluster(const __grid_constant__ PcgArgs a, int per) {
  using P = PartT<DM>;
  extern __shared__ __align__(16) unsigned char cl_mem[];
  __shared__ DiagInv<float> tab[16];
  // received partials (p.Ap, then r.r and r.z; a value and its round per
  // word), the warps' partials and the totals
  constexpr int kWords = int(sizeof(P) / 4);
  __shared__ __align__(16) unsigned long long words[kClCtas * 3 * kWords];
  __shared__ P wp[3 * kClWarps], tot[3];
  const int W = int(blockDim.x) >> 5, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const unsigned rank = cl_rank();
  ClFrame c;
  c.W = W;
  c.Wp = W > 8 ? 16 : (W > 4 ? 8 : (W > 2 ? 4 : W));
  c.warp = warp;
  c.lane = lane;
  c.limit = a.res_withhold ? 256u : kClPolls;
  c.mute = a.res_withhold && rank == 0;
  const unsigned from = unsigned(lane & (kClCtas - 1)), wa = 8u * kWords;
  unsigned src_a = static_cast<unsigned>(__cvta_generic_to_shared(words));
  unsigned src_u = src_a + kClCtas * wa;
  const unsigned dst_a = cl_map(src_a + rank * wa, from), dst_u = cl_map(src_u + rank * 2u * wa, from);
  src_a += from * wa;
  src_u += from * 2u * wa;
  const ClLayout l = cl_layout(W);
  const int nl = W * kClPerWarp;  // leaf places of the CTA; the last ones may be empty
  float* const mem = reinterpret_cast<float*>(cl_mem);
  float* const zs = reinterpret_cast<float*>(cl_mem + l.zs);
  PcgScalars* sc = a.sc;
  const int L0 = int(rank) * per;
  const int x0 = 2 * (lane >> 3), y = lane & 7;  // the lane's columns: (x0, y), (x0 + 1, y)
  fill_diag_table<float>(tab);
  for (unsigned i = threadIdx.x; i < l.bytes / 16; i += blockDim.x)
    reinterpret_cast<float4*>(cl_mem)[i] = make_float4(0.f, 0.f, 0.f, 0.f);
  for (int i = threadIdx.x; i < kClCtas * 3 * kWords; i += blockDim.x) words[i] = 0ull;
  __syncthreads();
  const unsigned sm0 = static_cast<unsigned>(__cvta_generic_to_shared(cl_mem));
  const float* pold = static_cast<const float*>((sc->iter & 1) ? a.p0 : a.p1);
  // Per leaf j = warp + k W of the CTA: the neighbours' places in local shared
  // memory (a leaf, halo columns or the zero leaf; float4 indices of chunk 0
  // of the first column, float indices for the z cells).  rem: bits 0 x face,
  // 1 y face, 2 -z, 3 +z come from another CTA.
  bool own[kClPerWarp];
  int xm_i[kClPerWarp], xp_i[kClPerWarp], ym_i[kClPerWarp], yp_i[kClPerWarp], zm_i[kClPerWarp], zp_i[kClPerWarp];
  unsigned rem[kClPerWarp];
  bool read[kClPerWarp];  // another CTA reads the lane's z
  uint2 f[kClPerWarp][2];
  Col<float> R[kClPerWarp][2], Z[kClPerWarp][2], Pc[2], X[2];
#pragma unroll
  for (int k = 0; k < kClPerWarp; ++k) {
    const int j = warp + k * W;
    const int s = L0 + j;
    own[k] = j < per && s < a.n_pleaf;
    const int nbl = own[k] ? face_slot_lane(a.nbr, s, lane) : -1;
    int fs[6];
    face_slots(nbl, fs);
    rem[k] = 0;
    read[k] = false;
#pragma unroll
    for (int q = 0; q < 2; ++q) {
      f[k][q] = make_uint2(0u, 0u);
#pragma unroll
      for (int z = 0; z < 8; ++z) R[k][q].v[z] = Z[k][q].v[z] = 0.f;
    }
    unsigned from[4] = {0u, 0u, 0u, 0u};
    int idx[6];
#pragma unroll
    for (int q = 0; q < 6; ++q) {
      // the neighbour of the pair: x0 - 1, x0 + 2, or both columns' y / z
      const int nx = q == 0 ? x0 - 1 : (q == 1 ? x0 + 2 : x0);
      const int ny = q == 2 ? y - 1 : (q == 3 ? y + 1 : y);
      const bool in_leaf = q < 4 && nx >= 0 && nx < 8 && ny >= 0 && ny < 8;
      const int slot = in_leaf ? s : fs[q];
      int leaf = nl, r = int(rank);  // the zero leaf
      if (own[k] && slot >= 0 && slot < a.n_pleaf) {
        r = slot / per;
        leaf = slot - r * per;
      }
      const int col = ps_col4(leaf, nx & 7, ny & 7);
      if (r == int(rank)) {
        idx[q] = q < 4 ? col : (col + (q == 4 ? 64 : 0)) * 4 + (q == 4 ? 3 : 0);
      } else {
        read[k] = true;  // adjacency is mutual: that CTA reads this lane's z
        // p of the previous iteration there, and where the owner keeps z
        const unsigned og = unsigned(slot) * 512u + unsigned(((nx & 7) << 6) | ((ny & 7) << 3));
        const unsigned zcol = sm0 + l.zs + unsigned(col) * 16u;
        if (q < 4) {
          const int hc = j * 32 + (q < 2 ? 8 * q + y : 16 + 4 * (q - 2) + (x0 >> 1));
          idx[q] = int(l.halo / 16) + (hc >> 6) * 128 + (hc & 63);
          rem[k] |= q < 2 ? 1u : 2u;
          from[q < 2 ? 0 : 1] = cl_map(zcol, unsigned(r));
          Col<float> p0;
          ldcol(pold, og, p0);
          ps_st4(mem, idx[q], p0);
          if (q >= 2) {
            ldcol(pold, og + 64u, p0);
            ps_st4(mem, idx[q] + 8, p0);
          }
        } else {
          idx[q] = int(l.zc / 4) + (j * 2 + (q - 4)) * 64 + lane;
          rem[k] |= q == 4 ? 4u : 8u;
          from[q - 2] = cl_map(zcol + (q == 4 ? 1024u + 12u : 0u), unsigned(r));
          const unsigned oz = og + (q == 4 ? 7u : 0u);
          mem[idx[q]] = __ldg(pold + oz);
          mem[idx[q] + 32] = __ldg(pold + oz + 64u);
        }
      }
    }
    xm_i[k] = idx[0];
    xp_i[k] = idx[1];
    ym_i[k] = idx[2];
    yp_i[k] = idx[3];
    zm_i[k] = idx[4];
    zp_i[k] = idx[5];
    reinterpret_cast<uint4*>(cl_mem + l.src)[j * 32 + lane] =
        make_uint4(from[0], from[1], from[2], from[3]);
#pragma unroll
    for (int q = 0; q < 2; ++q) {
#pragma unroll
      for (int z = 0; z < 8; ++z) Pc[q].v[z] = X[q].v[z] = 0.f;
      if (own[k]) {
        const unsigned og = unsigned(s) * 512u + unsigned(((x0 + q) << 6) | (y << 3));
        f[k][q] = ldflags(a.flags, og);
        ldcol(static_cast<const float*>(a.r), og, R[k][q]);
        Col<float> p0;
        ldcol(pold, og, p0);  // zero before the first iteration
        Pc[q] = p0;
#pragma unroll
        for (int z = 0; z < 8; ++z)
          Z[k][q].v[z] = tmul(tab[fbyte(f[k][q], z) & 15].inv, R[k][q].v[z]);
        if (read[k]) ps_st4(zs, ps_col4(j, x0 + q, y), Z[k][q]);
      }
    }
  }
  // the inverse diagonal unpacked
  float inv[2][8];
#pragma unroll
  for (int q = 0; q < 2; ++q)
#pragma unroll
    for (int z = 0; z < 8; ++z) inv[q][z] = tab[fbyte(f[0][q], z) & 15].inv;
  // the remote z of the halo, loaded as soon as it is published
  Col<float> hx[kClPerWarp], hy[kClPerWarp][2];
  float hz[kClPerWarp][4];
  auto load_halo = [&]() {
#pragma unroll
    for (int k = 0; k < kClPerWarp; ++k) {
      if (rem[k]) {
        const uint4 from =
            reinterpret_cast<const uint4*>(cl_mem + l.src)[(warp + k * W) * 32 + lane];
        if (rem[k] & 1u) cl_ldcol(from.x, hx[k]);
        if (rem[k] & 2u) {
          cl_ldcol(from.y, hy[k][0]);
          cl_ldcol(from.y + 128u, hy[k][1]);
        }
        if (rem[k] & 4u) {
          hz[k][0] = cl_ldcell(from.z);
          hz[k][1] = cl_ldcell(from.z + 128u);
        }
        if (rem[k] & 8u) {
          hz[k][2] = cl_ldcell(from.w);
          hz[k][3] = cl_ldcell(from.w + 128u);
        }
      }
    }
  };
  // p = z + beta p of a halo column or cell in place
  auto halo_col = [&](int i, const Col<float>& z, float beta) {
    Col<float> p;
    ps_ld4(mem, i, p);
#pragma unroll
    for (int t = 0; t < 8; ++t) p.v[t] = tadd(z.v[t], tmul(beta, p.v[t]));
    ps_st4(mem, i, p);
  };
  auto halo_cell = [&](int i, float z, float beta) { mem[i] = tadd(z, tmul(beta, mem[i])); };
  P rr, rz, rz_old, pap = pzero<P>();
  cl_split(sc->rr, rr);
  cl_split(sc->rz, rz);
  cl_split(sc->rz_old, rz_old);
  float alpha = 0.f, beta = float(sc->beta);
  int it = sc->iter, status = sc->status;
  const int max_it = sc->max_iter;
  const ClStop<P> stop = cl_stop_of<P>(sc);
  const int it0 = it;
  unsigned tag = 0;
  bool bad = false;
  cl_sync();  // every CTA's z and zeroed words are in place
  load_halo();
  // PCGDriver::Solve's loop test, then at the end of each iteration
  bool go = !sc->done && it < max_it && !converged(sc, sc->rr);
  while (go) {
    // S: p = z + beta p, on the own and the halo columns
#pragma unroll
    for (int k = 0; k < kClPerWarp; ++k) {
      if (own[k]) {
        const int j = warp + k * W;
#pragma unroll
        for (int q = 0; q < 2; ++q) {
          const int mine = ps_col4(j, x0 + q, y);
          Col<float> p;
          p = Pc[q];
#pragma unroll
          for (int z = 0; z < 8; ++z) p.v[z] = tadd(Z[k][q].v[z], tmul(beta, p.v[z]));
          ps_st4(mem, mine, p);
          Pc[q] = p;
        }
        if (rem[k] & 1u) halo_col(x0 == 0 ? xm_i[k] : xp_i[k], hx[k], beta);
        if (rem[k] & 2u) {
          const int i = y == 0 ? ym_i[k] : yp_i[k];
          halo_col(i, hy[k][0], beta);
          halo_col(i + 8, hy[k][1], beta);
        }
        if (rem[k] & 4u) {
          halo_cell(zm_i[k], hz[k][0], beta);
          halo_cell(zm_i[k] + 32, hz[k][1], beta);
        }
        if (rem[k] & 8u) {
          halo_cell(zp_i[k], hz[k][2], beta);
          halo_cell(zp_i[k] + 32, hz[k][3], beta);
        }
      }
    }
    __syncthreads();  // the CTA's p is in place
    // A p in the reference's column order: -x, -y, -z, diag, +z, +y, +x
    Dot<DM> dp;
#pragma unroll
    for (int k = 0; k < kClPerWarp; ++k) {
      if (own[k]) {
        const int j = warp + k * W;
        Col<float> p[2], xm, xp, ym[2], yp[2];
        ps_ld4(mem, xm_i[k], xm);
        ps_ld4(mem, ym_i[k], ym[0]);
        ps_ld4(mem, ym_i[k] + 8, ym[1]);
        ps_ld4(mem, yp_i[k], yp[0]);
        ps_ld4(mem, yp_i[k] + 8, yp[1]);
        ps_ld4(mem, xp_i[k], xp);
#pragma unroll
        for (int q = 0; q < 2; ++q) {
          p[q] = Pc[q];
        }
#pragma unroll
        for (int q = 0; q < 2; ++q) {
          const float zm = mem[zm_i[k] + 32 * q], zp = mem[zp_i[k] + 32 * q];
#pragma unroll
          for (int z = 0; z < 8; ++z) {
            const unsigned g = fbyte(f[k][q], z);
            const float vzm = z == 0 ? zm : p[q].v[(z + 7) & 7],
                        vzp = z == 7 ? zp : p[q].v[(z + 1) & 7];
            float t = tsub(0.f, q == 0 ? xm.v[z] : p[0].v[z]);
            t = tsub(t, ym[q].v[z]);
            t = tsub(t, vzm);
            t = tadd(t, tmul(cl_diag(g), p[q].v[z]));
            t = tsub(t, vzp);
            t = tsub(t, yp[q].v[z]);
            t = tsub(t, q == 0 ? p[1].v[z] : xp.v[z]);
            Z[k][q].v[z] = (g & 1u) ? t : 0.f;  // z's registers hold A p until U
            dp.add(p[q].v[z], Z[k][q].v[z]);
          }
        }
      }
    }
    {
      P v[1] = {dp.pvalue()};
      if ((bad = cl_sum<P, 1, false>(v, wp, tot, c, dst_a, src_a, ++tag))) break;
      pap = v[0];
    }
    alpha = cl_div(rz, pap, it == it0, sc->rz, true);
    if (!(alpha <= 1e5f)) {  // CHECK_LE(alpha, LARGE_FLOAT)
      status = FSIM_ERR_BREAKDOWN;
      break;
    }
    // U: x += alpha p, r -= alpha A p, z = M r
    Dot<DM> drr, drz;
    const float nalpha = -alpha;
#pragma unroll
    for (int k = 0; k < kClPerWarp; ++k) {
      if (own[k]) {
        const int j = warp + k * W;
#pragma unroll
        for (int q = 0; q < 2; ++q) {
          const int mine = ps_col4(j, x0 + q, y);
#pragma unroll
          for (int z = 0; z < 8; ++z) X[q].v[z] = tadd(tmul(alpha, Pc[q].v[z]), X[q].v[z]);
#pragma unroll
          for (int z = 0; z < 8; ++z) {
            R[k][q].v[z] = tadd(tmul(nalpha, Z[k][q].v[z]), R[k][q].v[z]);
            drr.add(R[k][q].v[z], R[k][q].v[z]);
            Z[k][q].v[z] = tmul(inv[q][z], R[k][q].v[z]);
            drz.add(R[k][q].v[z], Z[k][q].v[z]);
          }
          if (read[k]) ps_st4(zs, mine, Z[k][q]);
        }
      }
    }
    {
      P v[2] = {drr.pvalue(), drz.pvalue()};
      if ((bad = cl_sum<P, 2, true>(v, wp + kClWarps, tot + 1, c, dst_u, src_u, ++tag))) break;
      load_halo();
      rr = v[0];
      rz_old = rz;
      rz = v[1];
    }
    beta = cl_div(rz, rz_old, it == it0, sc->rz, false);
    ++it;
    if (!(beta <= 1e5f)) status = FSIM_ERR_BREAKDOWN;  // CHECK_LE(beta, LARGE_FLOAT)
    go = status == FSIM_OK && it < max_it && !cl_stop(stop, rr);
  }
  cl_sync();  // nobody reaches into this CTA's shared memory any more
  if (bad) {
    status = FSIM_ERR_TIMEOUT;
    sc->bar_err = 1u;
  }
#pragma unroll
  for (int k = 0; k < kClPerWarp; ++k) {
    if (own[k]) {
      const int j = warp + k * W;
#pragma unroll
      for (int q = 0; q < 2; ++q) {
        const unsigned og = unsigned(L0 + j) * 512u + unsigned(((x0 + q) << 6) | (y << 3));
        const int mine = ps_col4(j, x0 + q, y);
        Col<float> v;
        v = X[q];
        stcol(static_cast<float*>(a.x), og, v);
        // MIXED: the next segment continues with this search direction
        if (DM == 1 && it > it0) {
          ps_ld4(mem, mine, v);
          stcol(static_cast<float*>((it & 1) ? a.p0 : a.p1), og, v);
        }
      }
    }
  }
  if (rank == 0 && threadIdx.x == 0) {
    sc->iter = it;
    sc->done = 1;
    sc->status = status;
    sc->rr = ptod(rr);
    sc->rz = ptod(rz);
    sc->rz_old = ptod(rz_old);
    sc->alpha = double(alpha);
    sc->beta = double(beta);
    sc->pAp = ptod(pap);
  }
}

// A solve's iterations (one MIXED segment) by the cluster, or kLoopRefused.
template <int DM>
int run_cluster(fsim_sim* s, PcgArgs& a) {
  const int per = (a.n_pleaf + kClCtas - 1) / kClCtas;
  const int W = (per + kClPerWarp - 1) / kClPerWarp;
  const void* fn = reinterpret_cast<const void*>(k_pcg_cluster<DM>);
  const int most = int(cl_layout(kClWarps).bytes);
  cudaError_t e = cudaFuncSetAttribute(fn, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
  if (e == cudaSuccess)
    e = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, most);
  a.cond = 0;
  LoopTimer lt(s);
  if (e == cudaSuccess) {
    // (profiles find a solve's iterations by their first kernel's name, pcg_spmv*)
    fsim::ProfScope ps(s, DM == 0 ? "pcg_spmv_update_cluster" : "pcg_spmv_update_cluster_mixed");
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(kClCtas);
    cfg.blockDim = dim3(unsigned(W) * 32u);
    cfg.dynamicSmemBytes = cl_layout(W).bytes;
    cfg.stream = s->stream;
    cudaLaunchAttribute at = {};
    at.id = cudaLaunchAttributeClusterDimension;
    at.val.clusterDim.x = kClCtas;
    at.val.clusterDim.y = at.val.clusterDim.z = 1;
    cfg.attrs = &at;
    cfg.numAttrs = 1;
    void* args[] = {&a, const_cast<int*>(&per)};
    e = cudaLaunchKernelExC(&cfg, fn, args);
  }
  if (e != cudaSuccess) {
    cudaGetLastError();
    return kLoopRefused;
  }
  s->launches++;
  return end_one_launch(s, a, lt);
}
