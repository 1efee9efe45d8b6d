// pcg_resident.cuh -- the on-chip resident PCG loop: one persistent CTA per SM
// (included by k_pcg.cu, inside its namespace).
//
// Solves whose particle leaves fit on chip (FSIM_PCG_RES=1 / 0 forces it on /
// off) run in one cooperative launch per solve, or per segment of a MIXED
// solve.  CTA c owns the contiguous slots [c * per, c * per + nl), per =
// ceil(n_pleaf / G), and keeps every vector of the iteration on chip.  With
// fp32 vectors (FP32, MIXED; up to kResLeaves leaves per SM): p and the flags
// in shared memory, r and A p in tensor memory, x in tensor and shared memory
// (each warp owns up to kResHL half leaves, a lane one z-column of each).
// With fp64 vectors (up to kR64Leaves): p, r, x and A p in shared memory.  Per
// iteration, as the reference's ComputeLocal1-3 (common/solver.cc:297-366):
//   S: p = z + beta p on the own columns (into shared memory, and the
//      columns other CTAs read into a global mirror), then A p (kept) and
//      the p.Ap partials;
//   grid barrier with the sum of p.Ap -> alpha;
//   U: x += alpha p, r -= alpha A p, z = M r (of the columns other CTAs read
//      also into a global mirror), the r.r and r.z partials;
//   grid barrier with their sums -> r.r, r.z, beta and the loop test.
// (One more grid barrier before the first iteration publishes the first z.)
// Stencil neighbours in the CTA's own leaves come from shared memory; those
// in other CTAs' leaves are formed as z + beta p from the mirrors of z and
// the previous p, read through L2 (the owner's operations, so the owner's
// bits; p alternates between two mirror buffers by iteration parity).  A p is
// summed in the reference's column order.  The dot products are summed per
// thread and per CTA in fixed orders and over CTAs exactly or in a fixed
// order (below): the solve is deterministic (its order differs from the
// pair's, so the bits do too).  x is written back whole at the end, and p for
// a MIXED solve's next segment.  Barrier waits are bounded (kResPolls); a CTA
// that gives up sets bar_err and every CTA leaves the loop
// (FSIM_ERR_TIMEOUT), freeing its tensor memory.
// Measured us per iteration (particle leaves; 152 SMs), against the pair (the
// first three columns by k_pcg_resident1, below):
//   leaves        24          488        1,148       3,204       8,320
//   FP32     3.69 / 6.56  4.31 / 8.42  4.74 / 12.5  8.91 / 18.6  14.9 / 31.9
//   MIXED    5.06 / 10.0  5.80 / 10.7  6.50 / 13.5  11.8 / 19.7  19.7 / 34.6
// (before the fixed-point barrier FP32 took 5.90, 6.57, 6.96, 9.80 and 15.9).
constexpr int kResWarps = 28;
constexpr int kResThreads = kResWarps * 32;
constexpr int kResHL = 4;                             // half leaves per warp
constexpr int kResLeaves = kResWarps * kResHL / 2;    // leaves per CTA
// dynamic shared memory: p and the flags of the CTA's leaves, and x of every
// warp's half leaves 1 .. kResHL - 1 (half leaf 0's x is in tensor memory)
constexpr size_t kResSmemX = size_t(kResHL - 1) * kResWarps * 256 * sizeof(float);
constexpr size_t kResSmem = size_t(kResLeaves) * 512 * (sizeof(float) + 1) + kResSmemX;
constexpr unsigned kResPolls = 1u << 22;  // about 2-4 s of L2 round trips

__device__ __forceinline__ unsigned ld_acquire_gpu(const unsigned* p) {
  unsigned v;
  asm volatile("ld.acquire.gpu.global.u32 %0, [%1];\n" : "=r"(v) : "l"(p) : "memory");
  return v;
}

// ---- the grid barrier and its sums -------------------------------------------
// A partial goes up as fixed-point words in one 64-bit add each, which count
// the arrivals as well: bits 56.. count, the bits below sum v 2^s + 2^46 per
// CTA.  So one add and the polls of the same 64 bytes make the barrier and
// the sum: 0.76 us with one word where a counter, its polls and a load of
// the 152 partials take 1.59 (bare barriers on 152 SMs; more words cost about
// 0.06 us each, and a release before the adds 0.3, so only the barrier that
// publishes z has one).  The sums are exact in the words' units, whatever the
// order of the adds.  The scale s puts the previous total of the same dot
// product at 2^40: a CTA's partial may be 2^6 times that, and the total 2^7
// times smaller, before the units are too coarse for fp32 (2^33 of them).
// Partials of more than 24 bits (MIXED, FP64) carry their remainder in a
// second word, 2^-40 of the first's units.  A partial out of range (or not
// finite) is flagged in one more word; then, or when the total is too small,
// every CTA takes the same extra barrier, whose sums go through memory in
// CTA order (res_sum_slow).  Words are never reset during a solve: each CTA
// keeps what it read last and takes differences.
template <typename P>
struct ResWords {
  static constexpr int kPer = sizeof(P) == 4 ? 1 : 2;  // words per value
  static constexpr bool kLanes = std::is_same<P, double>::value;  // fixed point from the lanes
};
constexpr int kResSetWords = 8;  // per phase: at most 2 values of 2 words, and the flags

#include "pcg_fixed.cuh"

__device__ __forceinline__ void res_warp_sum(long long& hi, long long& lo) {
  int l[4];
  res_limbs(hi, lo, l);
#pragma unroll
  for (int k = 0; k < 4; ++k) l[k] = __reduce_add_sync(0xffffffffu, l[k]);
  res_unlimb(l, hi, lo);
}

// The words of the grid barriers: the fourth row of the fp64 partials, which
// nothing else uses (zeroed before each launch).
__host__ __device__ inline unsigned long long* res_words(const PcgArgs& a) {
  return reinterpret_cast<unsigned long long*>(a.part + 3 * a.maxb);
}
// Warp 0's state of the barriers, in shared memory (so that it holds no
// registers in the loop).
struct ResBarrier {
  unsigned long long last[2][kResSetWords];  // the words of each phase, as last read
  unsigned round, slow;                      // barriers so far; target of the next slow one
};

// Waits for all CTAs and sums the partials through memory, in CTA order (lane
// adds partials lane, lane + 32, ..., then the warp's tree).  Warp 0 only.
template <typename P, int NV>
__device__ __noinline__ bool res_sum_slow(const PcgArgs& a, P* rows, P (&v)[NV], unsigned target) {
  const int lane = threadIdx.x & 31, G = int(gridDim.x);
  int ok = 1;
  if (lane == 0) {
#pragma unroll
    for (int k = 0; k < NV; ++k) rows[k * a.maxb + blockIdx.x] = v[k];
    asm volatile("red.release.gpu.global.add.u32 [%0], 1;\n" ::"l"(&a.sc->bar_count) : "memory");
    unsigned polls = 0;
    while (int(ld_acquire_gpu(&a.sc->bar_count) - target) < 0) {
      if ((++polls & 255u) == 0u && (polls > kResPolls || ld_acquire_gpu(&a.sc->bar_err) != 0u)) {
        ok = 0;
        break;
      }
    }
  }
  ok = __shfl_sync(0xffffffffu, ok, 0);
  __syncwarp();  // orders lane 0's acquire before the other lanes' loads
  if (!ok) return false;
#pragma unroll
  for (int k = 0; k < NV; ++k) {
    P x = pzero<P>();
    for (int i = lane; i < G; i += 32) x = padd(x, __ldcg(rows + k * a.maxb + i));
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) x = padd(x, pshfl_xor(x, o));
    v[k] = x;
  }
  return true;
}

template <typename P, int W>
struct ResShared {
  P wp[2][W];                // warps' partials
  long long fp[2][2][W];     // FP64: the same in fixed point
  int ok;                    // kRes*: how the last barrier went, for the whole CTA
  ResBarrier bar;
};
constexpr int kResTimeout = 0, kResOk = 1, kResSlow = 2;

// FP64: the sums of a barrier whose words could not hold them, through memory
// (every CTA alike, the whole CTA).
template <typename P, int NV, int W, typename F>
__device__ __forceinline__ bool res_slow(const PcgArgs& a, P (&v)[NV], ResShared<P, W>& sh, P* rows,
                                         F&& fin) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
#pragma unroll
  for (int k = 0; k < NV; ++k) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v[k] = padd(v[k], pshfl_xor(v[k], o));
    if (lane == 0) sh.wp[k][warp] = v[k];
  }
  __syncthreads();  // also: every thread has read sh.ok
  if (warp == 0) {
#pragma unroll
    for (int k = 0; k < NV; ++k) {
      v[k] = lane < W ? sh.wp[k][lane] : pzero<P>();
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) v[k] = padd(v[k], pshfl_xor(v[k], o));
    }
    const unsigned target = sh.bar.slow + gridDim.x;
    __syncwarp();
    if (lane == 0) sh.bar.slow = target;
    const bool ok = res_sum_slow<P, NV>(a, rows, v, target);
    if (lane == 0) {
      if (ok)
        fin(v);
      else
        atomicExch(&a.sc->bar_err, 1u);
      sh.ok = ok ? kResOk : kResTimeout;
    }
  }
  __syncthreads();
  return sh.ok == kResOk;
}

// The barrier of phase ph (0: p.Ap; 1: r.r, r.z) with the sums of the CTA's
// NV values v[] (of every thread), like[] being totals of their size.  Warp 0
// arrives and waits, and its lane 0 then runs fin(totals) before the closing
// CTA barrier.  PUBLISH: global stores made by the CTA's threads before the
// call are visible to every CTA after it.  False when the wait gave up.  With
// PcgArgs::res_withhold (tests) CTA 0 does not arrive at the first barrier and
// the limit is 256 polls.
// The p.Ap barrier (PUBLISH false) is relaxed in memory: what keeps another
// CTA's store of z in U behind this CTA's loads of it in S is that every value
// loaded goes into A p and so into the partial that arrives, and that the
// store needs alpha, which needs all partials.  A load of z or p that is not
// used before the arrival (a prefetch across it) would need the release and
// acquire of the other barrier.
template <typename P, int NV, bool PUBLISH, int W, typename F>
__device__ __forceinline__ bool res_sync(const PcgArgs& a, P (&v)[NV], const P (&like)[NV],
                                         ResShared<P, W>& sh, P* slow_rows, int ph, F&& fin) {
  constexpr int kPer = ResWords<P>::kPer, NW = NV * kPer + 1;
  constexpr bool kLanes = ResWords<P>::kLanes;
  static_assert(NW <= kResSetWords, "words of a barrier");
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  bool in = true;
  if constexpr (!kLanes) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1)
#pragma unroll
      for (int k = 0; k < NV; ++k) v[k] = padd(v[k], pshfl_xor(v[k], o));
    if (lane == 0) {
#pragma unroll
      for (int k = 0; k < NV; ++k) sh.wp[k][warp] = v[k];
    }
    __syncthreads();  // the CTA's stores before it, too
  } else {
#pragma unroll
    for (int k = 0; k < NV; ++k) {
      long long h, l;
      in = res_fix(v[k], res_scale(like[k]), h, l) && in;
      if (!in) h = l = 0;
      res_warp_sum(h, l);
      if (lane == 0) {
        sh.fp[k][0][warp] = h;
        sh.fp[k][1][warp] = l;
      }
    }
    in = !__syncthreads_or(!in);
  }
  if (warp == 0) {
    const unsigned G = gridDim.x;
    int sc[NV];
    long long hi[NV], lo[NV];
#pragma unroll
    for (int k = 0; k < NV; ++k) {
      sc[k] = res_scale(like[k]);
      if constexpr (!kLanes) {
        v[k] = lane < W ? sh.wp[k][lane] : pzero<P>();
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) v[k] = padd(v[k], pshfl_xor(v[k], o));
        in = res_fix(v[k], sc[k], hi[k], lo[k]) && in;
      } else {
        hi[k] = lane < W ? sh.fp[k][0][lane] : 0ll;
        lo[k] = lane < W ? sh.fp[k][1][lane] : 0ll;
        res_warp_sum(hi[k], lo[k]);
        in = in && hi[k] < (1ll << 46) && hi[k] > -(1ll << 46);
      }
    }
    // word 0 .. NW - 2: the values' words; NW - 1: the flags
    constexpr long long kBias = 1ll << 46;
    unsigned long long add = in ? 0ull : 1ull;
#pragma unroll
    for (int k = 0; k < NV; ++k) {
      if (lane == k * kPer) add = static_cast<unsigned long long>((in ? hi[k] : 0ll) + kBias);
      if (kPer == 2 && lane == k * kPer + 1)
        add = static_cast<unsigned long long>((in ? lo[k] : 0ll) + kBias);
    }
    add += 1ull << 56;
    unsigned long long* w = res_words(a) + ph * kResSetWords + lane;
    const bool hold = a.res_withhold && blockIdx.x == 0 && sh.bar.round == 0u;
    if (PUBLISH) asm volatile("fence.acq_rel.gpu;\n" ::: "memory");
    if (lane < NW && !hold)
      asm volatile("red.relaxed.gpu.global.add.u64 [%0], %1;\n" ::"l"(w), "l"(add) : "memory");
    const unsigned limit = a.res_withhold ? 256u : kResPolls;
    const unsigned long long last = lane < NW ? sh.bar.last[ph][lane] : 0ull;
    unsigned long long got = static_cast<unsigned long long>(G) << 56;
    bool done = lane >= NW;
    int code = kResOk;
    unsigned polls = 0;
    for (;;) {
      if (!done) {
        unsigned long long m;
        if (PUBLISH)
          asm volatile("ld.acquire.gpu.global.u64 %0, [%1];\n" : "=l"(m) : "l"(w) : "memory");
        else
          asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];\n" : "=l"(m) : "l"(w) : "memory");
        got = m - last;
        done = unsigned(got >> 56) == G;
      }
      if (__all_sync(0xffffffffu, done)) break;
      if ((++polls & 255u) == 0u &&
          __any_sync(0xffffffffu, polls > limit || ld_acquire_gpu(&a.sc->bar_err) != 0u)) {
        code = kResTimeout;
        break;
      }
    }
    if (lane < NW) sh.bar.last[ph][lane] = last + got;
    if (lane == 0) sh.bar.round = 1u;
    if (code == kResOk) {
      const long long sum = static_cast<long long>(got & ((1ull << 56) - 1ull)) -
                            (lane < NW - 1 ? static_cast<long long>(G) * kBias : 0ll);
      bool slow = __shfl_sync(0xffffffffu, sum, NW - 1) != 0ll;
      P tot[NV];
#pragma unroll
      for (int k = 0; k < NV; ++k) {
        const long long h = __shfl_sync(0xffffffffu, sum, k * kPer);
        const long long l = kPer == 2 ? __shfl_sync(0xffffffffu, sum, k * kPer + 1) : 0ll;
        slow = slow || h < (1ll << 33);
        res_unfix(h, l, sc[k], tot[k]);
      }
      if (slow) {
        if constexpr (kLanes) {
          code = kResSlow;  // the whole CTA: its partials are not formed yet
        } else {
          P t[NV];  // a copy, so that the values above stay in registers
#pragma unroll
          for (int k = 0; k < NV; ++k) t[k] = v[k];
          const unsigned target = sh.bar.slow + G;
          __syncwarp();
          if (lane == 0) sh.bar.slow = target;
          if (!res_sum_slow<P, NV>(a, slow_rows, t, target)) code = kResTimeout;
#pragma unroll
          for (int k = 0; k < NV; ++k) tot[k] = t[k];
        }
      }
      if (code == kResOk && lane == 0) fin(tot);
    }
    if (lane == 0 && code == kResTimeout) atomicExch(&a.sc->bar_err, 1u);
    if (lane == 0) sh.ok = code;
  }
  __syncthreads();
  if constexpr (kLanes) {
    if (sh.ok == kResSlow) {
      return res_slow<P, NV>(a, v, sh, slow_rows, fin);
    }
  }
  return sh.ok == kResOk;
}

__device__ __forceinline__ void res_start(ResBarrier& b, const PcgScalars* sc) {
  for (int i = 0; i < 2 * kResSetWords; ++i) b.last[i / kResSetWords][i % kResSetWords] = 0ull;
  b.round = 0u;
  b.slow = sc->bar_count;
}
// The barrier before the first iteration (of phase 1's words): every CTA's
// partials are 1 and 1.
template <typename P, int W>
__device__ __forceinline__ bool res_first(const PcgArgs& a, ResShared<P, W>& sh, P* rows) {
  P v[2] = {pzero<P>(), pzero<P>()}, like[2];
  if (threadIdx.x == 0) {
    cl_split(1.0, v[0]);
    cl_split(1.0, v[1]);
  }
  cl_split(double(gridDim.x), like[0]);
  like[1] = like[0];
  return res_sync<P, 2, true>(a, v, like, sh, rows, 1, [](const P (&)[2]) {});
}

// The resident loop's scalar state, kept by warp 0's lane 0 in shared memory,
// in the partials' type (FP32: fp32 as the reference; MIXED: double-float).
template <typename P>
struct ResScalars {
  P rr, rz, rz_old, pAp;
  double rz0;         // the first r.z, from the set-up in fp64
  float alpha, beta;  // FP64 keeps its own
  double alpha64, beta64;
  int status, max_iter;
  ClStop<P> stop;
};
template <typename P>
__device__ __forceinline__ void res_scalars(ResScalars<P>& q, const PcgScalars* sc) {
  cl_split(sc->rr, q.rr);
  cl_split(sc->rz, q.rz);
  q.rz0 = sc->rz;
  cl_split(sc->rz_old, q.rz_old);
  q.pAp = pzero<P>();
  q.alpha = 0.f;
  q.beta = float(sc->beta);
  q.alpha64 = 0.0;
  q.beta64 = sc->beta;
  q.status = sc->status;
  q.max_iter = sc->max_iter;
  q.stop = cl_stop_of<P>(sc);
}
// the solve's scalars back, as the pair leaves them
template <typename P>
__device__ __forceinline__ void res_finish(const ResScalars<P>& q, PcgScalars* sc, int it) {
  sc->iter = it;
  sc->done = 1;
  sc->status = q.status;
  sc->rr = ptod(q.rr);
  sc->rz = ptod(q.rz);
  sc->rz_old = ptod(q.rz_old);
  sc->alpha = sizeof(P) == sizeof(double) && !std::is_same<P, float2>::value ? q.alpha64 : double(q.alpha);
  sc->beta = sizeof(P) == sizeof(double) && !std::is_same<P, float2>::value ? q.beta64 : double(q.beta);
  sc->pAp = ptod(q.pAp);
}

// Where a neighbour of the CTA's cells lives.
struct ResFrame {
  const float* ps;  // shared p of the CTA's leaves
  int L0, nl, n_pleaf;
};
__device__ __forceinline__ bool res_local(const ResFrame& fr, int slot) {
  return slot >= fr.L0 && slot < fr.L0 + fr.nl;
}

// p (current iteration) of cell (x, y, z) of leaf `slot`: from shared memory
// for the CTA's leaves, else formed from the mirrors of z and the previous p.
__device__ __forceinline__ float res_pcell(const ResFrame& fr, const PcgArgs& a,
                                           const float* pm_old, float beta, int slot, int x, int y,
                                           int z) {
  if (res_local(fr, slot)) return fr.ps[(ps_col4(slot - fr.L0, x, y) + (z >> 2) * 64) * 4 + (z & 3)];
  const unsigned o = slot_or_null(slot, fr.n_pleaf) * 512u + unsigned(x * 64 + y * 8 + z);
  // the mirror holds z = M r (the owner's product): pnew_of's operations
  return tadd(__ldcg(static_cast<const float*>(a.r) + o), tmul(beta, __ldcg(pm_old + o)));
}

// The half leaf's faces in other CTAs' leaves (its outward x face and both
// y faces: 16 columns of 8 cells), formed by all 32 lanes in step: lane L
// forms cells 4 (L & 1) .. + 3 of face column t = L >> 1 (t < 8: the x face
// at y = t; 8 .. 11: the -y face at x = xb + t - 8; 12 .. 15: the +y face)
// from the mirrors of z and the previous p, with the owner's operations.
// Faces in the CTA's own leaves are left to shared memory (v stays 0).
__device__ __forceinline__ void res_faces(const ResFrame& fr, const PcgArgs& a, const float* pm_old,
                                          float beta, int xb, const int fs[6], int lane,
                                          float (&v)[4]) {
  const int t = lane >> 1;
  int slot, off;
  if (t < 8) {
    slot = xb == 0 ? fs[0] : fs[1];
    off = (xb == 0 ? 7 : 0) * 64 + t * 8;
  } else if (t < 12) {
    slot = fs[2];
    off = (xb + t - 8) * 64 + 56;
  } else {
    slot = fs[3];
    off = (xb + t - 12) * 64;
  }
  off += 4 * (lane & 1);
#pragma unroll
  for (int j = 0; j < 4; ++j) v[j] = 0.f;
  if (!res_local(fr, slot)) {
    const unsigned o = slot_or_null(slot, fr.n_pleaf) * 512u + unsigned(off);
    // the mirror holds z = M r (the owner's product): pnew_of's operations
    const float4 zm = __ldcg(reinterpret_cast<const float4*>(static_cast<const float*>(a.r) + o));
    const float4 po = __ldcg(reinterpret_cast<const float4*>(pm_old + o));
    v[0] = tadd(zm.x, tmul(beta, po.x));
    v[1] = tadd(zm.y, tmul(beta, po.y));
    v[2] = tadd(zm.z, tmul(beta, po.z));
    v[3] = tadd(zm.w, tmul(beta, po.w));
  }
}
// column c of the faces formed by res_faces (lanes 2 c and 2 c + 1)
__device__ __forceinline__ void res_face_col(const float (&v)[4], int c, Col<float>& out) {
#pragma unroll
  for (int z = 0; z < 8; ++z) out.v[z] = __shfl_sync(0xffffffffu, v[z & 3], 2 * c + (z >> 2));
}

// A p on the lane's column (xb + lx, y) of leaf s (own values P), with the
// faces fv of other CTAs' leaves (res_faces) and the -z / +z face cells.  The
// diagonal comes from the flags' bits (TABLE: from the table in shared
// memory, the same values): 28 warps contend for shared memory more than for
// the ALUs (us per iteration at 3,204, 4,444 and 8,320 leaves 9.19 -> 9.09,
// 11.71 -> 11.29, 15.37 -> 15.18; MIXED 11.96 -> 11.84, 15.03 -> 14.71, 19.86
// -> 19.76), while at one half leaf per warp the table is as fast or faster
// (MIXED at 1,148 leaves 7.33 / 7.43).
template <bool TABLE, typename ZL, typename ZH>
__device__ __forceinline__ void res_stencil(const ResFrame& fr, const DiagInv<float>* tab, int s,
                                            int xb, int lx, int y, const int fs[6],
                                            const Col<float>& P, uint2 f, const float (&fv)[4],
                                            ZL&& zlo, ZH&& zhi, Col<float>& ap) {
  const int x = xb + lx;
  const int own = ps_col4(s - fr.L0, x, y);
  // one neighbour column at a time, in the reference's order: -x, -y, -z,
  // diag, +z, +y, +x
  Col<float> nc;
#pragma unroll
  for (int z = 0; z < 8; ++z) ap.v[z] = 0.f;
  if (xb == 0) res_face_col(fv, y, nc);  // warp-uniform: the outward face is -x
  if (x > 0)
    ps_ld4(fr.ps, own - 8, nc);
  else if (res_local(fr, fs[0]))
    ps_ld4(fr.ps, ps_col4(fs[0] - fr.L0, 7, y), nc);
#pragma unroll
  for (int z = 0; z < 8; ++z) ap.v[z] = tsub(ap.v[z], nc.v[z]);
  Col<float> gy;  // the -y face column for lanes at y = 0, the +y one at y = 7
  res_face_col(fv, (y == 0 ? 8 : 12) + lx, gy);
  if (y > 0)
    ps_ld4(fr.ps, own - 1, nc);
  else if (res_local(fr, fs[2]))
    ps_ld4(fr.ps, ps_col4(fs[2] - fr.L0, x, 7), nc);
  else
    nc = gy;
#pragma unroll
  for (int z = 0; z < 8; ++z) ap.v[z] = tsub(ap.v[z], nc.v[z]);
  const float zm = zlo(), zp = zhi();
#pragma unroll
  for (int z = 0; z < 8; ++z) {
    const uint8_t g = fbyte(f, z);
    const float vzm = z == 0 ? zm : P.v[(z + 7) & 7], vzp = z == 7 ? zp : P.v[(z + 1) & 7];
    ap.v[z] = tsub(ap.v[z], vzm);
    ap.v[z] = tadd(ap.v[z], tmul(TABLE ? tab[g & 15].d : cl_diag(g), P.v[z]));
    ap.v[z] = tsub(ap.v[z], vzp);
  }
  if (y < 7)
    ps_ld4(fr.ps, own + 1, nc);
  else if (res_local(fr, fs[3]))
    ps_ld4(fr.ps, ps_col4(fs[3] - fr.L0, x, 0), nc);
  else
    nc = gy;
#pragma unroll
  for (int z = 0; z < 8; ++z) ap.v[z] = tsub(ap.v[z], nc.v[z]);
  if (xb != 0) res_face_col(fv, y, nc);  // the outward face is +x
  if (x < 7)
    ps_ld4(fr.ps, own + 8, nc);
  else if (res_local(fr, fs[1]))
    ps_ld4(fr.ps, ps_col4(fs[1] - fr.L0, 0, y), nc);
#pragma unroll
  for (int z = 0; z < 8; ++z) {
    ap.v[z] = tsub(ap.v[z], nc.v[z]);
    if (!(fbyte(f, z) & 1)) ap.v[z] = 0.f;
  }
}

// A p on the lane's column (xb + lx, y) of leaf s (own values P), in the
// reference's column order; 0 off-fluid.  Called by all 32 lanes of the
// warp together (res_faces, res_face_col).
__device__ __forceinline__ void res_ap(const ResFrame& fr, const PcgArgs& a, const float* pm_old,
                                       const DiagInv<float>* tab, float beta, int s, int xb, int lx,
                                       int y, int lane, const int fs[6], const Col<float>& P,
                                       uint2 f, Col<float>& ap) {
  float fv[4];
  res_faces(fr, a, pm_old, beta, xb, fs, lane, fv);
  res_stencil<false>(fr, tab, s, xb, lx, y, fs, P, f, fv,
              [&] { return res_pcell(fr, a, pm_old, beta, fs[4], xb + lx, y, 7); },
              [&] { return res_pcell(fr, a, pm_old, beta, fs[5], xb + lx, y, 0); }, ap);
}
// The Jacobi inverse by flags & 15 (the table's values).  U of k_pcg_resident
// reads it from constant memory, off the shared-memory path: most warps ask
// for one entry (us per iteration at 3,204 and 8,320 leaves 9.09 -> 8.96 and
// 15.19 -> 14.93; MIXED the same within 0.3%; by warp shuffles 9.04 and 15.32,
// by a chain of selects 9.93 and 17.40).
__constant__ float c_inv16[16] = {0.f, __builtin_inff(), 0.f, 1.0f, 0.f, 0.5f,
                                  0.f, float(1.0 / 3.0), 0.f, 0.25f, 0.f, float(1.0 / 5.0),
                                  0.f, float(1.0 / 6.0), 0.f, float(1.0 / 7.0)};

// r and A p of the CTA's cells live in tensor memory (TMEM): all 512
// columns, allocated by warp 0; warp w uses TMEM lanes 32 (w % 4) .. + 31
// (the quarter it may access), and for its half leaf k columns (w / 4) * 32
// + 8 k .. + 7 for r and the same + kResTmemAp for A p (lane L holds its
// column's 8 cells).  That leaves the registers to 28 warps, and A p, formed
// once per iteration for p.Ap, is kept for the update of r; from then to the
// next S its columns hold z = M r, formed once for r.z and p = z + beta p.  x of half leaf
// 0 takes columns kResTmemX + (w / 4) * 8 .. + 7; x of half leaves 1 .. 3
// is in shared memory.  So every vector of the iteration stays on chip, and
// x is read and written in global memory once per solve.
constexpr unsigned kResTmemCols = 512;
constexpr unsigned kResTmemVec = (kResWarps + 3) / 4 * kResHL * 8;  // columns of r or A p
constexpr unsigned kResTmemAp = kResTmemVec;
constexpr unsigned kResTmemX = 2 * kResTmemVec;
static_assert(kResTmemX + (kResWarps + 3) / 4 * 8 <= kResTmemCols, "TMEM columns");

// x of the warp's half leaf k >= 1 in shared memory: two 16-byte chunks per
// lane (cells z = 0..3 and 4..7), consecutive lanes in consecutive words
__device__ __forceinline__ void xs_ld(const float4* xs, int k, int warp, int lane, float (&v)[8]) {
  const float4 u = xs[(((k - 1) * kResWarps + warp) * 2 + 0) * 32 + lane];
  const float4 w = xs[(((k - 1) * kResWarps + warp) * 2 + 1) * 32 + lane];
  v[0] = u.x; v[1] = u.y; v[2] = u.z; v[3] = u.w;
  v[4] = w.x; v[5] = w.y; v[6] = w.z; v[7] = w.w;
}
__device__ __forceinline__ void xs_st(float4* xs, int k, int warp, int lane, const float (&v)[8]) {
  xs[(((k - 1) * kResWarps + warp) * 2 + 0) * 32 + lane] = make_float4(v[0], v[1], v[2], v[3]);
  xs[(((k - 1) * kResWarps + warp) * 2 + 1) * 32 + lane] = make_float4(v[4], v[5], v[6], v[7]);
}
__device__ __forceinline__ void tmem_ld8(unsigned t, float (&v)[8]) {
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];\n"
               : "=f"(v[0]), "=f"(v[1]), "=f"(v[2]), "=f"(v[3]), "=f"(v[4]), "=f"(v[5]),
                 "=f"(v[6]), "=f"(v[7])
               : "r"(t)
               : "memory");
  asm volatile("tcgen05.wait::ld.sync.aligned;\n" ::: "memory");
}
__device__ __forceinline__ void tmem_st8(unsigned t, const float (&v)[8]) {
  asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};\n" ::"r"(t),
               "f"(v[0]), "f"(v[1]), "f"(v[2]), "f"(v[3]), "f"(v[4]), "f"(v[5]), "f"(v[6]),
               "f"(v[7])
               : "memory");
}
__device__ __forceinline__ void tmem_wait_st() {
  asm volatile("tcgen05.wait::st.sync.aligned;\n" ::: "memory");
}

template <int DM>
__global__ void __launch_bounds__(kResThreads, 1) k_pcg_resident(const __grid_constant__ PcgArgs a) {
  using P = PartT<DM>;
  extern __shared__ __align__(16) unsigned char res_smem[];
  float* ps = reinterpret_cast<float*>(res_smem);
  uint8_t* fsm = res_smem + size_t(kResLeaves) * 512 * sizeof(float);
  float4* xs = reinterpret_cast<float4*>(res_smem + size_t(kResLeaves) * 512 * (sizeof(float) + 1));
  __shared__ DiagInv<float> tab[16];
  __shared__ int s_done;
  __shared__ ResScalars<P> q;
  __shared__ ResShared<P, kResWarps> sh;
  __shared__ unsigned s_taddr;
  PcgScalars* sc = a.sc;
  const int G = int(gridDim.x);
  const int per = (a.n_pleaf + G - 1) / G;  // the host checks per <= kResLeaves
  ResFrame fr;
  fr.ps = ps;
  fr.L0 = int(blockIdx.x) * per;
  fr.nl = max(0, min(per, a.n_pleaf - fr.L0));
  fr.n_pleaf = a.n_pleaf;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  fill_diag_table<float>(tab);
  for (int i = threadIdx.x; i < fr.nl * 512; i += kResThreads) {
    fsm[i] = a.flags[int64_t(fr.L0) * 512 + i];
  }
  if (warp == 0) {
    const unsigned sa = static_cast<unsigned>(__cvta_generic_to_shared(&s_taddr));
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;\n" ::"r"(sa),
                 "r"(kResTmemCols)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;\n" ::: "memory");
  }
  asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
  const unsigned tbase = s_taddr + ((32u * unsigned(warp & 3)) << 16) + unsigned(warp >> 2) * 32u;
  const unsigned txb = s_taddr + ((32u * unsigned(warp & 3)) << 16) + kResTmemX + unsigned(warp >> 2) * 8u;
  // the warp's half leaves: r and x on chip, the face slots, and which of
  // the lane's columns other CTAs read (bit k of mir: the column is on a face
  // whose neighbour leaf is in another CTA, or the leaf's -z or +z neighbour
  // is, which reads a cell of every column); only those go to the mirrors
  int nbl[kResHL];
  unsigned mir = 0;
  int it = sc->iter;
  const int it0 = it;
#pragma unroll
  for (int k = 0; k < kResHL; ++k) {
    const int hl = warp + k * kResWarps;
    nbl[k] = -1;
    if (hl < 2 * fr.nl) {
      const HalfLeaf h = half_pos(2 * fr.L0 + hl, lane);
      const unsigned og = unsigned(h.s) * 512u + unsigned(h.c);
      Col<float> r0;
      ldcol(static_cast<const float*>(a.r), og, r0);
      tmem_st8(tbase + 8u * k, r0.v);
      Col<float> z0;
      {
        const uint2 f = *reinterpret_cast<const uint2*>(fsm + (hl >> 1) * 512 + h.c);
#pragma unroll
        for (int z = 0; z < 8; ++z) z0.v[z] = tmul(tab[fbyte(f, z) & 15].inv, r0.v[z]);
        tmem_st8(tbase + kResTmemAp + 8u * k, z0.v);
      }
      // p of the previous iteration (zero before the first one)
      ldcol(static_cast<const float*>((it & 1) ? a.p0 : a.p1), og, r0);
      ps_st4(ps, ps_col4(hl >> 1, h.xb + h.lx, h.cy), r0);
      ldcol(static_cast<const float*>(a.x), og, r0);
      if (k == 0)
        tmem_st8(txb, r0.v);
      else
        xs_st(xs, k, warp, lane, r0.v);
      nbl[k] = face_slot_lane(a.nbr, h.s, lane);
      int fs[6];
      face_slots(nbl[k], fs);
      const bool xo = h.xb == 0 ? (h.lx == 0 && !res_local(fr, fs[0]))
                                : (h.lx == 3 && !res_local(fr, fs[1]));
      const bool yo = (h.cy == 0 && !res_local(fr, fs[2])) || (h.cy == 7 && !res_local(fr, fs[3]));
      const bool zo = !res_local(fr, fs[4]) || !res_local(fr, fs[5]);
      if (xo || yo || zo) {
        mir |= 1u << k;
        stcol(static_cast<float*>(a.r), og, z0);  // the mirror of z for the first iteration
      }
    }
  }
  tmem_wait_st();
  // Warp 0's lane 0 runs the loop test and the alpha / beta steps (after the
  // barriers' acquire loads every read of the scalar block would be an L2
  // round trip); the other threads take alpha, beta and the stop flag from
  // shared memory.
  if (threadIdx.x == 0) {
    res_scalars(q, sc);
    res_start(sh.bar, sc);
    s_done = sc->done || it >= q.max_iter || converged(sc, sc->rr);  // PCGDriver::Solve's loop test
  }
  P* const rows = part_rows<DM>(a);
  __syncthreads();
  float* x = static_cast<float*>(a.x);
  float* rmir = static_cast<float*>(a.r);  // during the loop: the mirror of z = M r
  // every CTA's z mirror is written before any CTA's first stencil reads it
  bool ok = res_first(a, sh, rows + a.maxb);
  while (ok && !s_done) {
    float* pm_new = static_cast<float*>((it & 1) ? a.p1 : a.p0);
    const float* pm_old = static_cast<const float*>((it & 1) ? a.p0 : a.p1);
    const float fbeta = q.beta;
    // S: p = z + beta p on the own columns
#pragma unroll
    for (int k = 0; k < kResHL; ++k) {
      const int hl = warp + k * kResWarps;
      if (hl < 2 * fr.nl) {
        const HalfLeaf h = half_pos(2 * fr.L0 + hl, lane);
        Col<float> P;
        const int own = ps_col4(hl >> 1, h.xb + h.lx, h.cy);
        ps_ld4(ps, own, P);
        float zk[8];  // z = M r, left in the A p columns by U (or the set-up)
        tmem_ld8(tbase + kResTmemAp + 8u * k, zk);
#pragma unroll
        for (int z = 0; z < 8; ++z) P.v[z] = tadd(zk[z], tmul(fbeta, P.v[z]));  // pnew_of's operations
        ps_st4(ps, own, P);
        if ((mir >> k) & 1u) stcol(pm_new, unsigned(h.s) * 512u + unsigned(h.c), P);
      }
    }
    __syncthreads();
    Dot<DM> dp;
#pragma unroll
    for (int k = 0; k < kResHL; ++k) {
      const int hl = warp + k * kResWarps;
      int fs[6];
      face_slots(nbl[k], fs);
      if (hl < 2 * fr.nl) {
        const HalfLeaf h = half_pos(2 * fr.L0 + hl, lane);
        const int ol = (hl >> 1) * 512 + h.c;
        Col<float> P, ap;
        ps_ld4(ps, ps_col4(hl >> 1, h.xb + h.lx, h.cy), P);
        const uint2 f = *reinterpret_cast<const uint2*>(fsm + ol);
        res_ap(fr, a, pm_old, tab, fbeta, h.s, h.xb, h.lx, h.cy, lane, fs, P, f, ap);
#pragma unroll
        for (int z = 0; z < 8; ++z) dp.add(P.v[z], ap.v[z]);
        tmem_st8(tbase + kResTmemAp + 8u * k, ap.v);
      }
    }
    tmem_wait_st();
    {
      P v[1] = {dp.pvalue()};
      const P like[1] = {it == it0 ? q.rz : q.pAp};
      ok = res_sync<P, 1, false>(a, v, like, sh, rows, 0, [&](const P (&tot)[1]) {
        q.pAp = tot[0];
        q.alpha = cl_div(q.rz, q.pAp, it == it0, q.rz0, true);
        if (!(q.alpha <= 1e5f)) {  // CHECK_LE(alpha, LARGE_FLOAT)
          q.status = FSIM_ERR_BREAKDOWN;
          s_done = 1;
        }
      });
      if (!ok || s_done) break;
    }
    // U: x += alpha p, r -= alpha A p
    const float fa = q.alpha, fna = -fa;
    Dot<DM> drr, drz;
#pragma unroll
    for (int k = 0; k < kResHL; ++k) {
      const int hl = warp + k * kResWarps;
      if (hl < 2 * fr.nl) {
        const HalfLeaf h = half_pos(2 * fr.L0 + hl, lane);
        const int ol = (hl >> 1) * 512 + h.c;
        const unsigned og = unsigned(h.s) * 512u + unsigned(h.c);
        Col<float> P, X, R;
        if (k == 0)
          tmem_ld8(txb, X.v);
        else
          xs_ld(xs, k, warp, lane, X.v);
        ps_ld4(ps, ps_col4(hl >> 1, h.xb + h.lx, h.cy), P);
        const uint2 f = *reinterpret_cast<const uint2*>(fsm + ol);
#pragma unroll
        for (int z = 0; z < 8; ++z) X.v[z] = tadd(tmul(fa, P.v[z]), X.v[z]);
        if (k == 0)
          tmem_st8(txb, X.v);
        else
          xs_st(xs, k, warp, lane, X.v);
        float ap[8];
        tmem_ld8(tbase + 8u * k, R.v);
        tmem_ld8(tbase + kResTmemAp + 8u * k, ap);
#pragma unroll
        for (int z = 0; z < 8; ++z) {
          const uint8_t g = fbyte(f, z);
          R.v[z] = tadd(tmul(fna, ap[z]), R.v[z]);
          drr.add(R.v[z], R.v[z]);
          ap[z] = tmul(c_inv16[g & 15], R.v[z]);  // z = M r, for r.z and the next S
          drz.add(R.v[z], ap[z]);
        }
        tmem_st8(tbase + 8u * k, R.v);
        tmem_st8(tbase + kResTmemAp + 8u * k, ap);
        if ((mir >> k) & 1u) {
          Col<float> Z;
#pragma unroll
          for (int z = 0; z < 8; ++z) Z.v[z] = ap[z];
          stcol(rmir, og, Z);
        }
      }
    }
    tmem_wait_st();
    {
      P v[2] = {drr.pvalue(), drz.pvalue()};
      const P like[2] = {q.rr, q.rz};
      ok = res_sync<P, 2, true>(a, v, like, sh, rows + a.maxb, 1, [&](const P (&tot)[2]) {
        q.rr = tot[0];
        q.rz_old = q.rz;
        q.rz = tot[1];
        q.beta = cl_div(q.rz, q.rz_old, it == it0, q.rz0, false);
        if (!(q.beta <= 1e5f)) {  // CHECK_LE(beta, LARGE_FLOAT)
          q.status = FSIM_ERR_BREAKDOWN;
          s_done = 1;
        } else {
          s_done = (it + 1 >= q.max_iter) || cl_stop(q.stop, q.rr);  // the next loop test
        }
      });
      if (!ok) break;
      ++it;
    }
  }
  if (!ok && threadIdx.x == 0) q.status = FSIM_ERR_TIMEOUT;
  // x back to global memory, and p for a MIXED solve's next segment; every
  // warp is then done with TMEM, and warp 0 frees it
  tmem_wait_st();
#pragma unroll
  for (int k = 0; k < kResHL; ++k) {
    const int hl = warp + k * kResWarps;
    if (hl < 2 * fr.nl) {
      const HalfLeaf h = half_pos(2 * fr.L0 + hl, lane);
      const unsigned og = unsigned(h.s) * 512u + unsigned(h.c);
      Col<float> X;
      if (k == 0)
        tmem_ld8(txb, X.v);
      else
        xs_ld(xs, k, warp, lane, X.v);
      stcol(x, og, X);
      if (DM == 1 && it > it0) {
        ps_ld4(ps, ps_col4(hl >> 1, h.xb + h.lx, h.cy), X);
        stcol(static_cast<float*>((it & 1) ? a.p0 : a.p1), og, X);
      }
    }
  }
  asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
  __syncthreads();
  if (warp == 0) {
    asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;\n" ::"r"(s_taddr),
                 "r"(kResTmemCols)
                 : "memory");
  }
  if (blockIdx.x == 0 && threadIdx.x == 0) res_finish(q, sc, it);
}

// ---- one or two half leaves per warp -------------------------------------------
// Systems of at most KH kRes1Leaves leaves per SM, KH half leaves per warp: the
// same loop with the vectors of a lane's columns in registers (no tensor
// memory; x in shared memory for KH = 2), and the loads of the faces in other
// CTAs' leaves issued before S, whose work and CTA barrier then hide part of
// their latency.  p of those faces stays with its
// reader, formed from the owner's z like the owner's own p, so z is all that
// CTAs exchange.  The operations and their order are k_pcg_resident's, so the
// bits are too.  Bound by the iteration's chain of latencies (two grid
// barriers, one round trip to L2 for the faces, the CTA barriers: at 1,148
// leaves an SM issues in 18% of its cycles, MIXED 25%).  us per iteration
// against k_pcg_resident, FP32 and MIXED (leaves per SM):
//   KH = 1   488 (4): 4.31 / 5.61, 5.80 / 7.60   1,148 (8): 4.74 / 6.07, 6.50 / 8.17
//   KH = 2   1,278 (9): 5.99 / 6.23, 8.62 / 8.42   1,456 (10): 6.01 / 6.40, 8.63 / 8.54
//            1,584 (11): 6.10 / 6.55, 8.80 / 8.89   1,920 (13): 6.24 / 6.92, 9.04 / 9.37
// (with p mirrored as well, KH = 1 took 4.88 and 6.40, 5.60 and 7.32).  MIXED
// spills a little with KH = 2, so it takes it from 11 leaves per SM on.  More
// than 16 warps leave too few registers (28 warps of 72, KH = 1, 1,278 leaves:
// 6.55 and 9.34).
constexpr int kRes1Warps = 16;  // 128 registers a thread
constexpr int kRes1Leaves = kRes1Warps / 2;
constexpr size_t kRes1Leaf = 512 * sizeof(float);  // shared memory per leaf: p

template <int DM, int KH>
__global__ void __launch_bounds__(kRes1Warps * 32, 1) k_pcg_resident1(const __grid_constant__ PcgArgs a) {
  using P = PartT<DM>;
  extern __shared__ __align__(16) unsigned char res_smem[];
  float* ps = reinterpret_cast<float*>(res_smem);
  __shared__ DiagInv<float> tab[16];
  __shared__ int s_done;
  __shared__ ResScalars<P> q;
  __shared__ ResShared<P, kRes1Warps> sh;
  PcgScalars* sc = a.sc;
  const int G = int(gridDim.x);
  const int per = (a.n_pleaf + G - 1) / G;  // the host checks per <= KH * kRes1Leaves
  float4* const xs = reinterpret_cast<float4*>(res_smem + kRes1Leaf * per);  // x, KH > 1
  ResFrame fr;
  fr.ps = ps;
  fr.L0 = int(blockIdx.x) * per;
  fr.nl = max(0, min(per, a.n_pleaf - fr.L0));
  fr.n_pleaf = a.n_pleaf;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  fill_diag_table<float>(tab);
  // partials of the warps that a smaller block does not have
  for (int i = threadIdx.x; i < kRes1Warps; i += int(blockDim.x))
    sh.wp[0][i] = sh.wp[1][i] = pzero<P>();
  // the warp's half leaf k: half leaf warp + k W of the CTA
  const int W = int(blockDim.x) >> 5;
  auto has = [&](int k) { return warp + k * W < 2 * fr.nl; };
  auto half = [&](int k) { return half_pos(2 * fr.L0 + warp + k * W, lane); };
  float* rmir = static_cast<float*>(a.r);  // during the loop: the mirror of z = M r
  uint2 f[KH];
  Col<float> p[KH], x[1], r[KH], z[KH];  // z: A p from the stencil to U
  int fs[KH][6];
  bool mir[KH];
  // the lane's share of the half leaf's faces in other CTAs' leaves (lanes and
  // cells as in res_faces) and its own -z / +z cells there: where the owners
  // mirror z, and p, which stays here
  bool face[KH], zl[KH], zh[KH];
  unsigned fo[KH];
  float gp[KH][4], gz0[KH], gz1[KH];
  auto zo0 = [&](int k, const HalfLeaf& h) { return unsigned(fs[k][4]) * 512u + unsigned(h.c) + 7u; };
  auto zo1 = [&](int k, const HalfLeaf& h) { return unsigned(fs[k][5]) * 512u + unsigned(h.c); };
  int it = sc->iter;
  const int it0 = it;
  __syncthreads();  // the diagonal's table
#pragma unroll
  for (int k = 0; k < KH; ++k) {
    face[k] = zl[k] = zh[k] = mir[k] = false;
    fo[k] = 0;
    gz0[k] = gz1[k] = 0.f;
#pragma unroll
    for (int e = 0; e < 4; ++e) gp[k][e] = 0.f;
    f[k] = make_uint2(0u, 0u);
    if (has(k)) {
      const HalfLeaf h = half(k);
      const unsigned og = unsigned(h.s) * 512u + unsigned(h.c);
      const float* pold = static_cast<const float*>((it & 1) ? a.p0 : a.p1);
      f[k] = ldflags(a.flags, og);
      ldcol(rmir, og, r[k]);
      ldcol(pold, og, p[k]);
      ldcol(static_cast<const float*>(a.x), og, x[0]);
      if (KH > 1) {
        xs[((k * kRes1Warps + warp) * 2 + 0) * 32 + lane] = make_float4(x[0].v[0], x[0].v[1], x[0].v[2], x[0].v[3]);
        xs[((k * kRes1Warps + warp) * 2 + 1) * 32 + lane] = make_float4(x[0].v[4], x[0].v[5], x[0].v[6], x[0].v[7]);
      }
      face_slots(face_slot_lane(a.nbr, h.s, lane), fs[k]);
#pragma unroll
      for (int e = 0; e < 8; ++e) z[k].v[e] = tmul(tab[fbyte(f[k], e) & 15].inv, r[k].v[e]);
      auto far = [&](int slot) { return slot >= 0 && slot < a.n_pleaf && !res_local(fr, slot); };
      const bool xo = h.xb == 0 ? (h.lx == 0 && far(fs[k][0])) : (h.lx == 3 && far(fs[k][1]));
      const bool yo = (h.cy == 0 && far(fs[k][2])) || (h.cy == 7 && far(fs[k][3]));
      zl[k] = far(fs[k][4]);
      zh[k] = far(fs[k][5]);
      mir[k] = xo || yo || zl[k] || zh[k];
      const int t = lane >> 1;
      const int slot = t < 8 ? (h.xb == 0 ? fs[k][0] : fs[k][1]) : (t < 12 ? fs[k][2] : fs[k][3]);
      face[k] = far(slot);
      if (face[k]) {
        fo[k] = unsigned(slot) * 512u + 4u * unsigned(lane & 1) +
                unsigned(t < 8 ? (h.xb == 0 ? 7 : 0) * 64 + t * 8
                               : (t < 12 ? (h.xb + t - 8) * 64 + 56 : (h.xb + t - 12) * 64));
        const float4 v = *reinterpret_cast<const float4*>(pold + fo[k]);
        gp[k][0] = v.x; gp[k][1] = v.y; gp[k][2] = v.z; gp[k][3] = v.w;
      }
      if (zl[k]) gz0[k] = pold[zo0(k, h)];
      if (zh[k]) gz1[k] = pold[zo1(k, h)];
      if (mir[k]) stcol(rmir, og, z[k]);  // the mirror of z for the first iteration
    }
  }
  if (threadIdx.x == 0) {
    res_scalars(q, sc);
    res_start(sh.bar, sc);
    s_done = sc->done || it >= q.max_iter || converged(sc, sc->rr);  // PCGDriver::Solve's loop test
  }
  P* const rows = part_rows<DM>(a);
  __syncthreads();
  bool ok = res_first(a, sh, rows + a.maxb);
  while (ok && !s_done) {
    const float fbeta = q.beta;
    Dot<DM> dp;
    // z of the remote faces: loads in flight over S
    float4 zv[KH];
    float z0[KH], z1[KH];
#pragma unroll
    for (int k = 0; k < KH; ++k) {
      zv[k] = make_float4(0.f, 0.f, 0.f, 0.f);
      z0[k] = z1[k] = 0.f;
      if (has(k)) {
        const HalfLeaf h = half(k);
        if (face[k]) zv[k] = __ldcg(reinterpret_cast<const float4*>(rmir + fo[k]));
        if (zl[k]) z0[k] = __ldcg(rmir + zo0(k, h));
        if (zh[k]) z1[k] = __ldcg(rmir + zo1(k, h));
      }
    }
#pragma unroll
    for (int k = 0; k < KH; ++k) {
      if (has(k)) {
        const HalfLeaf h = half(k);
#pragma unroll
        for (int e = 0; e < 8; ++e) p[k].v[e] = tadd(z[k].v[e], tmul(fbeta, p[k].v[e]));  // pnew_of's operations
        ps_st4(ps, ps_col4(h.s - fr.L0, h.xb + h.lx, h.cy), p[k]);
      }
    }
#pragma unroll
    for (int k = 0; k < KH; ++k) {
      gp[k][0] = tadd(zv[k].x, tmul(fbeta, gp[k][0]));
      gp[k][1] = tadd(zv[k].y, tmul(fbeta, gp[k][1]));
      gp[k][2] = tadd(zv[k].z, tmul(fbeta, gp[k][2]));
      gp[k][3] = tadd(zv[k].w, tmul(fbeta, gp[k][3]));
      gz0[k] = tadd(z0[k], tmul(fbeta, gz0[k]));
      gz1[k] = tadd(z1[k], tmul(fbeta, gz1[k]));
    }
    __syncthreads();
#pragma unroll
    for (int k = 0; k < KH; ++k) {
      if (has(k)) {
        const HalfLeaf h = half(k);
        auto zcell = [&](int slot, float ghost, int chunk, int e) {
          return res_local(fr, slot)
                     ? ps[(ps_col4(slot - fr.L0, h.xb + h.lx, h.cy) + chunk) * 4 + e] : ghost;
        };
        res_stencil<true>(fr, tab, h.s, h.xb, h.lx, h.cy, fs[k], p[k], f[k], gp[k],
                          [&] { return zcell(fs[k][4], gz0[k], 64, 3); },
                          [&] { return zcell(fs[k][5], gz1[k], 0, 0); }, z[k]);
#pragma unroll
        for (int e = 0; e < 8; ++e) dp.add(p[k].v[e], z[k].v[e]);
      }
    }
    {
      P v[1] = {dp.pvalue()};
      const P like[1] = {it == it0 ? q.rz : q.pAp};
      ok = res_sync<P, 1, false>(a, v, like, sh, rows, 0, [&](const P (&tot)[1]) {
        q.pAp = tot[0];
        q.alpha = cl_div(q.rz, q.pAp, it == it0, q.rz0, true);
        if (!(q.alpha <= 1e5f)) {  // CHECK_LE(alpha, LARGE_FLOAT)
          q.status = FSIM_ERR_BREAKDOWN;
          s_done = 1;
        }
      });
      if (!ok || s_done) break;
    }
    const float fa = q.alpha, fna = -fa;
    Dot<DM> drr, drz;
#pragma unroll
    for (int k = 0; k < KH; ++k) {
      if (has(k)) {
        const HalfLeaf h = half(k);
#pragma unroll
        for (int e = 0; e < 8; ++e) {
          r[k].v[e] = tadd(tmul(fna, z[k].v[e]), r[k].v[e]);
          z[k].v[e] = tmul(tab[fbyte(f[k], e) & 15].inv, r[k].v[e]);
        }
        if (mir[k]) stcol(rmir, unsigned(h.s) * 512u + unsigned(h.c), z[k]);
        if (KH > 1) {
          float4* const q0 = xs + ((k * kRes1Warps + warp) * 2 + 0) * 32 + lane;
          const float4 u = q0[0], w = q0[32];
          q0[0] = make_float4(tadd(tmul(fa, p[k].v[0]), u.x), tadd(tmul(fa, p[k].v[1]), u.y),
                              tadd(tmul(fa, p[k].v[2]), u.z), tadd(tmul(fa, p[k].v[3]), u.w));
          q0[32] = make_float4(tadd(tmul(fa, p[k].v[4]), w.x), tadd(tmul(fa, p[k].v[5]), w.y),
                               tadd(tmul(fa, p[k].v[6]), w.z), tadd(tmul(fa, p[k].v[7]), w.w));
        } else {
#pragma unroll
          for (int e = 0; e < 8; ++e) x[0].v[e] = tadd(tmul(fa, p[k].v[e]), x[0].v[e]);
        }
#pragma unroll
        for (int e = 0; e < 8; ++e) {
          drr.add(r[k].v[e], r[k].v[e]);
          drz.add(r[k].v[e], z[k].v[e]);
        }
      }
    }
    {
      P v[2] = {drr.pvalue(), drz.pvalue()};
      const P like[2] = {q.rr, q.rz};
      ok = res_sync<P, 2, true>(a, v, like, sh, rows + a.maxb, 1, [&](const P (&tot)[2]) {
        q.rr = tot[0];
        q.rz_old = q.rz;
        q.rz = tot[1];
        q.beta = cl_div(q.rz, q.rz_old, it == it0, q.rz0, false);
        if (!(q.beta <= 1e5f)) {  // CHECK_LE(beta, LARGE_FLOAT)
          q.status = FSIM_ERR_BREAKDOWN;
          s_done = 1;
        } else {
          s_done = (it + 1 >= q.max_iter) || cl_stop(q.stop, q.rr);  // the next loop test
        }
      });
      if (!ok) break;
      ++it;
    }
  }
  if (!ok && threadIdx.x == 0) q.status = FSIM_ERR_TIMEOUT;
  // x back to global memory, and p for a MIXED solve's next segment
#pragma unroll
  for (int k = 0; k < KH; ++k) {
    if (has(k)) {
      const HalfLeaf h = half(k);
      const unsigned og = unsigned(h.s) * 512u + unsigned(h.c);
      if (KH > 1) {
        const float4 u = xs[((k * kRes1Warps + warp) * 2 + 0) * 32 + lane],
                     w = xs[((k * kRes1Warps + warp) * 2 + 1) * 32 + lane];
        x[0].v[0] = u.x; x[0].v[1] = u.y; x[0].v[2] = u.z; x[0].v[3] = u.w;
        x[0].v[4] = w.x; x[0].v[5] = w.y; x[0].v[6] = w.z; x[0].v[7] = w.w;
      }
      stcol(static_cast<float*>(a.x), og, x[0]);
      if (DM == 1 && it > it0) stcol(static_cast<float*>((it & 1) ? a.p0 : a.p1), og, p[k]);
    }
  }
  if (blockIdx.x == 0 && threadIdx.x == 0) res_finish(q, sc, it);
}

// ---- fp64 vectors -----------------------------------------------------------------
// The FP64 pair spends 19 us per iteration on any system (its kernels wait at
// their first instruction and sum their heads on the FP64 pipe) and forms A p
// twice.  Here a cell takes 13 FP64 instructions per iteration (p 1, A p 6,
// p.Ap 1, x 1, r 1, z 1, r.r 1, r.z 1: products fused with their sums), and
// everything else stays off that pipe, which at 64 cycles per warp instruction
// and scheduler (3,328 cycles a leaf) is what bounds the loop.  A warp takes
// the lower or upper four cells of the columns of half a leaf at a time, so
// that one leaf already keeps all four schedulers busy.  All vectors are in
// shared memory: p in 16-byte chunk planes ((leaf * 4 + chunk) * 8 + x) * 8 +
// y, the others by unit, chunk and lane.  Measured us per iteration, against
// the pair: 7.5 / 19.4 at 24 leaves, 12.7 / 30.4 at 488 (96^3 sphere drop), 20.3
// / 54.2 at 1,148 (128^3), 24.3 at 1,456.
constexpr int kR64Warps = 16;
constexpr int kR64Threads = kR64Warps * 32;
constexpr int kR64Leaves = 13;
constexpr size_t kR64Vec = size_t(kR64Leaves) * 512 * sizeof(double);
constexpr size_t kR64Smem = 4 * kR64Vec + size_t(kR64Leaves) * 512;

struct Quad {
  double v[4];
};
__device__ __forceinline__ void quad_set(Quad& q, double2 a, double2 b) {
  q.v[0] = a.x;
  q.v[1] = a.y;
  q.v[2] = b.x;
  q.v[3] = b.y;
}
// double2 index of cells z = 4 zh .. of column (x, y) in the chunk planes; the
// next two cells are 64 further
__device__ __forceinline__ int r64_col(int leaf, int x, int y, int zh) {
  return (leaf * 32 + x) * 8 + y + 128 * zh;
}
__device__ __forceinline__ void r64_ld(const double2* p, int i, int stride, Quad& q) {
  quad_set(q, p[i], p[i + stride]);
}
__device__ __forceinline__ void r64_st(double2* p, int i, int stride, const Quad& q) {
  p[i] = make_double2(q.v[0], q.v[1]);
  p[i + stride] = make_double2(q.v[2], q.v[3]);
}

// p (current iteration) of four cells of leaf slot: shared memory, or the
// given cells of another CTA's leaf.  Those a unit needs (its outward x face
// and both y faces, 64 cells) are formed by all 32 lanes, two each, and handed
// out by shuffles: formed where they are used they cost 16 instructions of the
// FP64 pipe for the few lanes at the faces (us per iteration at 156, 488 and
// 1,148 leaves 9.60 -> 8.84, 13.98 -> 12.69, 22.83 -> 20.34; with the first
// unit's loads issued before S 8.69, 12.95, 20.73).
struct R64Frame {
  const double2* ps;
  const double *zm, *pm;
  int L0, nl, n_pleaf;
  double beta;
};
__device__ __forceinline__ bool r64_local(const R64Frame& f, int slot) {
  return slot >= f.L0 && slot < f.L0 + f.nl;
}
__device__ __forceinline__ void r64_pquad(const R64Frame& f, int slot, int x, int y, int zh,
                                          const Quad& ghost, Quad& c) {
  if (r64_local(f, slot))
    r64_ld(f.ps, r64_col(slot - f.L0, x, y, zh), 64, c);
  else
    c = ghost;
}
// one cell of another CTA's leaf, from the mirrors; 0 where the CTA has the
// leaf or there is none
__device__ __forceinline__ double r64_far(const R64Frame& f, int slot, unsigned o) {
  if (slot < 0 || slot >= f.n_pleaf || r64_local(f, slot)) return 0.0;
  o += unsigned(slot) * 512u;
  return __fma_rn(f.beta, __ldcg(f.pm + o), __ldcg(f.zm + o));
}
// p of cell z of column (x, y) of leaf slot
__device__ __forceinline__ double r64_pcell(const R64Frame& f, int slot, int x, int y, int z) {
  if (slot >= f.L0 && slot < f.L0 + f.nl) {
    const double2 v = f.ps[r64_col(slot - f.L0, x, y, 0) + (z >> 1) * 64];
    return (z & 1) ? v.y : v.x;
  }
  if (slot < 0 || slot >= f.n_pleaf) return 0.0;
  const unsigned o = unsigned(slot) * 512u + unsigned(x * 64 + y * 8 + z);
  return __fma_rn(f.beta, __ldcg(f.pm + o), __ldcg(f.zm + o));
}

__global__ void __launch_bounds__(kR64Threads, 1) k_pcg_resident64(const __grid_constant__ PcgArgs a) {
  using P = double;
  extern __shared__ __align__(16) unsigned char res_smem[];
  double2* const ps = reinterpret_cast<double2*>(res_smem);
  double2* const rs = reinterpret_cast<double2*>(res_smem + kR64Vec);
  double2* const zs = reinterpret_cast<double2*>(res_smem + 2 * kR64Vec);  // z, or A p until U
  double2* const xs = reinterpret_cast<double2*>(res_smem + 3 * kR64Vec);
  uint8_t* const fsm = res_smem + 4 * kR64Vec;
  __shared__ DiagInv<double> tab[16];
  __shared__ int nbs[kR64Leaves][6];
  __shared__ int s_done;
  __shared__ ResScalars<P> q;
  __shared__ ResShared<P, kR64Warps> sh;
  PcgScalars* sc = a.sc;
  const int G = int(gridDim.x);
  const int per = (a.n_pleaf + G - 1) / G;  // the host checks per <= kR64Leaves
  R64Frame fr;
  fr.ps = ps;
  fr.zm = static_cast<const double*>(a.r);
  fr.L0 = int(blockIdx.x) * per;
  fr.nl = max(0, min(per, a.n_pleaf - fr.L0));
  fr.n_pleaf = a.n_pleaf;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int nu = 4 * fr.nl;  // units: half leaf u / 2, cells z = 4 (u & 1) .. + 3
  int it = sc->iter;
  fill_diag_table<double>(tab);
  for (int i = threadIdx.x; i < fr.nl * 512; i += kR64Threads)
    fsm[i] = a.flags[int64_t(fr.L0) * 512 + i];
  for (int i = threadIdx.x; i < fr.nl * 6; i += kR64Threads) {
    constexpr int kFace[6] = {4, 22, 10, 16, 12, 14};
    nbs[i / 6][i % 6] = a.nbr[int64_t(fr.L0 + i / 6) * 27 + kFace[i % 6]];
  }
  __syncthreads();
  double* const zmir = static_cast<double*>(a.r);
  // a unit's place: local leaf j, the lane's column (x, y), z half, flags, and
  // the cells' offset in the global vectors
  struct Unit {
    int j, x, y, zh;
    unsigned og;
  };
  auto unit = [&](int u) {
    Unit t;
    t.j = u >> 2;
    t.x = 4 * ((u >> 1) & 1) + (lane >> 3);
    t.y = lane & 7;
    t.zh = u & 1;
    t.og = unsigned(fr.L0 + t.j) * 512u + unsigned(t.x * 64 + t.y * 8 + 4 * t.zh);
    return t;
  };
  auto flags4 = [&](const Unit& t) {
    return *reinterpret_cast<const unsigned*>(fsm + t.j * 512 + t.x * 64 + t.y * 8 + 4 * t.zh);
  };
  auto gld = [](const void* p, unsigned o, Quad& c) {
    r64_ld(reinterpret_cast<const double2*>(static_cast<const double*>(p) + o), 0, 1, c);
  };
  auto gst = [](void* p, unsigned o, const Quad& c) {
    r64_st(reinterpret_cast<double2*>(static_cast<double*>(p) + o), 0, 1, c);
  };
  unsigned mir = 0;  // bit per unit of the warp: other CTAs read some of the lane's cells
  for (int u = warp, k = 0; u < nu; u += kR64Warps, ++k) {
    const Unit t = unit(u);
    Quad c;
    gld((it & 1) ? a.p0 : a.p1, t.og, c);  // zero before the first iteration
    r64_st(ps, r64_col(t.j, t.x, t.y, t.zh), 64, c);
    gld(a.x, t.og, c);
    r64_st(xs, u * 64 + lane, 32, c);
    gld(a.r, t.og, c);
    r64_st(rs, u * 64 + lane, 32, c);
    const unsigned f = flags4(t);
#pragma unroll
    for (int z = 0; z < 4; ++z) c.v[z] = __dmul_rn(tab[(f >> (8 * z)) & 15].inv, c.v[z]);
    r64_st(zs, u * 64 + lane, 32, c);
    auto far = [&](int q) { return nbs[t.j][q] < fr.L0 || nbs[t.j][q] >= fr.L0 + fr.nl; };
    if ((t.x == 0 && far(0)) || (t.x == 7 && far(1)) || (t.y == 0 && far(2)) ||
        (t.y == 7 && far(3)) || far(4 + t.zh)) {
      mir |= 1u << k;
      gst(zmir, t.og, c);  // the mirror of z for the first iteration
    }
  }
  if (threadIdx.x == 0) {
    res_scalars(q, sc);
    res_start(sh.bar, sc);
    s_done = sc->done || it >= q.max_iter || converged(sc, sc->rr);  // PCGDriver::Solve's loop test
  }
  const int it0 = it;
  __syncthreads();
  bool ok = res_first(a, sh, a.part + a.maxb);
  while (ok && !s_done) {
    void* const pm_new = (it & 1) ? a.p1 : a.p0;
    fr.pm = static_cast<const double*>((it & 1) ? a.p0 : a.p1);
    fr.beta = q.beta64;
    // S: p = z + beta p on the own cells
    for (int u = warp, k = 0; u < nu; u += kR64Warps, ++k) {
      const Unit t = unit(u);
      const int own = r64_col(t.j, t.x, t.y, t.zh);
      Quad p, z;
      r64_ld(ps, own, 64, p);
      r64_ld(zs, u * 64 + lane, 32, z);
#pragma unroll
      for (int c = 0; c < 4; ++c) p.v[c] = __fma_rn(fr.beta, p.v[c], z.v[c]);
      r64_st(ps, own, 64, p);
      if ((mir >> k) & 1u) gst(pm_new, t.og, p);
    }
    __syncthreads();
    Dot<2> dp;
    for (int u = warp; u < nu; u += kR64Warps) {
      const Unit t = unit(u);
      const int s = fr.L0 + t.j, x = t.x, y = t.y;
      const int* nb = nbs[t.j];
      const unsigned f = flags4(t);
      const int xb = x & 4, cell = 4 * t.zh + (lane & 3);
      const double gx = r64_far(fr, xb ? nb[1] : nb[0],
                                unsigned((xb ? 0 : 448) + (lane >> 2) * 8 + cell));
      const double gy = r64_far(fr, lane < 16 ? nb[2] : nb[3],
                                unsigned((xb + ((lane >> 2) & 3)) * 64 + (lane < 16 ? 56 : 0) + cell));
      Quad p, w, c, fx, fy;
#pragma unroll
      for (int z = 0; z < 4; ++z) {
        fx.v[z] = __shfl_sync(0xffffffffu, gx, 4 * y + z);
        fy.v[z] = __shfl_sync(0xffffffffu, gy, (y == 0 ? 0 : 16) + 4 * (x & 3) + z);
      }
      r64_pquad(fr, x > 0 ? s : nb[0], (x + 7) & 7, y, t.zh, fx, w);
      r64_pquad(fr, y > 0 ? s : nb[2], x, (y + 7) & 7, t.zh, fy, c);
#pragma unroll
      for (int z = 0; z < 4; ++z) w.v[z] = __dsub_rn(-w.v[z], c.v[z]);
      r64_ld(ps, r64_col(t.j, x, y, t.zh), 64, p);
      const double zm = t.zh ? r64_pcell(fr, s, x, y, 3) : r64_pcell(fr, nb[4], x, y, 7);
      const double zp = t.zh ? r64_pcell(fr, nb[5], x, y, 0) : r64_pcell(fr, s, x, y, 4);
#pragma unroll
      for (int z = 0; z < 4; ++z) {
        w.v[z] = __dsub_rn(w.v[z], z == 0 ? zm : p.v[(z + 3) & 3]);
        w.v[z] = __fma_rn(tab[(f >> (8 * z)) & 15].d, p.v[z], w.v[z]);
        w.v[z] = __dsub_rn(w.v[z], z == 3 ? zp : p.v[(z + 1) & 3]);
      }
      r64_pquad(fr, y < 7 ? s : nb[3], x, (y + 1) & 7, t.zh, fy, c);
#pragma unroll
      for (int z = 0; z < 4; ++z) w.v[z] = __dsub_rn(w.v[z], c.v[z]);
      r64_pquad(fr, x < 7 ? s : nb[1], (x + 1) & 7, y, t.zh, fx, c);
#pragma unroll
      for (int z = 0; z < 4; ++z) {
        w.v[z] = ((f >> (8 * z)) & 1u) ? __dsub_rn(w.v[z], c.v[z]) : 0.0;
        dp.add(p.v[z], w.v[z]);
      }
      r64_st(zs, u * 64 + lane, 32, w);
    }
    {
      P v[1] = {dp.pvalue()};
      const P like[1] = {it == it0 ? q.rz : q.pAp};
      ok = res_sync<P, 1, false>(a, v, like, sh, a.part, 0, [&](const P (&tot)[1]) {
        q.pAp = tot[0];
        q.alpha64 = q.rz / q.pAp;
        if (!(q.alpha64 <= 1e5)) {  // CHECK_LE(alpha, LARGE_FLOAT)
          q.status = FSIM_ERR_BREAKDOWN;
          s_done = 1;
        }
      });
      if (!ok || s_done) break;
    }
    // U: x += alpha p, r -= alpha A p, z = M r
    const double al = q.alpha64;
    Dot<2> drr, drz;
    for (int u = warp, k = 0; u < nu; u += kR64Warps, ++k) {
      const Unit t = unit(u);
      const unsigned f = flags4(t);
      Quad p, x, r, z;
      r64_ld(ps, r64_col(t.j, t.x, t.y, t.zh), 64, p);
      r64_ld(xs, u * 64 + lane, 32, x);
#pragma unroll
      for (int c = 0; c < 4; ++c) x.v[c] = __fma_rn(al, p.v[c], x.v[c]);
      r64_st(xs, u * 64 + lane, 32, x);
      r64_ld(rs, u * 64 + lane, 32, r);
      r64_ld(zs, u * 64 + lane, 32, z);
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        r.v[c] = __fma_rn(-al, z.v[c], r.v[c]);
        z.v[c] = __dmul_rn(tab[(f >> (8 * c)) & 15].inv, r.v[c]);
        drr.add(r.v[c], r.v[c]);
        drz.add(r.v[c], z.v[c]);
      }
      r64_st(rs, u * 64 + lane, 32, r);
      r64_st(zs, u * 64 + lane, 32, z);
      if ((mir >> k) & 1u) gst(zmir, t.og, z);
    }
    {
      P v[2] = {drr.pvalue(), drz.pvalue()};
      const P like[2] = {q.rr, q.rz};
      ok = res_sync<P, 2, true>(a, v, like, sh, a.part + a.maxb, 1, [&](const P (&tot)[2]) {
        q.rr = tot[0];
        q.rz_old = q.rz;
        q.rz = tot[1];
        q.beta64 = q.rz / q.rz_old;
        if (!(q.beta64 <= 1e5)) {  // CHECK_LE(beta, LARGE_FLOAT)
          q.status = FSIM_ERR_BREAKDOWN;
          s_done = 1;
        } else {
          s_done = (it + 1 >= q.max_iter) || cl_stop(q.stop, q.rr);  // the next loop test
        }
      });
      if (!ok) break;
      ++it;
    }
  }
  if (!ok && threadIdx.x == 0) q.status = FSIM_ERR_TIMEOUT;
  for (int u = warp; u < nu; u += kR64Warps) {
    Quad x;
    r64_ld(xs, u * 64 + lane, 32, x);
    gst(a.x, unit(u).og, x);
  }
  __syncthreads();
  if (blockIdx.x == 0 && threadIdx.x == 0) res_finish(q, sc, it);
}

// The loop's kernel for a system that fits: one or two half leaves per warp
// (MIXED with two from 11 leaves per SM on), or the general one, FP64's too.
int res_kernel(const fsim_sim* s, int precision) {
  const int per = (s->n_pleaf + s->num_sms - 1) / s->num_sms;
  if (precision == FSIM_PREC_FP64) return kLoopRes;
  if (per <= kRes1Leaves) return kLoopRes1;
  if (per <= 2 * kRes1Leaves && per >= (precision == FSIM_PREC_FP32 ? 0 : 11)) return kLoopRes2;
  return kLoopRes;
}

// The iterations of a solve (of one MIXED segment) by the resident loop: one
// cooperative launch of one CTA per SM, or kLoopRefused.
template <int DM>
int run_resident(fsim_sim* s, PcgArgs& a) {
  void* fn;
  size_t smem = kResSmem, most = kResSmem;  // this launch's shared memory, and the kernel's most
  int threads = kResThreads;
  const char* name;
  if constexpr (DM == 2) {
    fn = reinterpret_cast<void*>(k_pcg_resident64);
    smem = most = kR64Smem;
    threads = kR64Threads;
    name = "pcg_resident_f64";
  } else {
    fn = reinterpret_cast<void*>(k_pcg_resident<DM>);
    name = DM == 0 ? "pcg_resident" : "pcg_resident_mixed";
    const int per = (s->n_pleaf + s->num_sms - 1) / s->num_sms;
    const int form = res_kernel(s, DM == 0 ? FSIM_PREC_FP32 : FSIM_PREC_MIXED);
    if (form == kLoopRes1) {
      fn = reinterpret_cast<void*>(k_pcg_resident1<DM, 1>);
      smem = kRes1Leaf * per;
      most = kRes1Leaf * kRes1Leaves;
      threads = 64 * per;
    } else if (form == kLoopRes2) {
      fn = reinterpret_cast<void*>(k_pcg_resident1<DM, 2>);
      constexpr size_t kX = size_t(2 * kRes1Warps) * 256 * sizeof(float);
      smem = kRes1Leaf * per + kX;
      most = kRes1Leaf * 2 * kRes1Leaves + kX;
      threads = 32 * kRes1Warps;
    }
  }
  // The attribute belongs to the kernel, not to the handle: every handle sets
  // the same, or another thread's smaller system would have this launch refused.
  int occ = 0;
  if (cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, int(most)) !=
          cudaSuccess ||
      cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, fn, threads, smem) != cudaSuccess ||
      occ < 1) {
    cudaGetLastError();
    return kLoopRefused;
  }
  a.cond = 0;
  FSIM_CK(s, cudaMemsetAsync(res_words(a), 0, 2 * kResSetWords * sizeof(unsigned long long),
                             s->stream));
  LoopTimer lt(s);
  {
    fsim::ProfScope ps(s, name);
    void* args[] = {&a};
    const cudaError_t e = cudaLaunchCooperativeKernel(fn, dim3(unsigned(s->num_sms)),
                                                      dim3(unsigned(threads)), args, smem,
                                                      s->stream);
    if (e != cudaSuccess) {
      cudaGetLastError();
      return kLoopRefused;
    }
  }
  s->launches++;
  return end_one_launch(s, a, lt);
}
