// The lower levels of a cycle as ONE kernel: a thread-block cluster per right-hand side keeps every vector
// and every table of those levels in its CTAs' shared memory and runs the whole sub-cycle -- smoothing,
// residuals, transfers, the coarsest solve, the recursion of V-, W- and full-multigrid cycles -- phase
// by phase.
//
// What bounds the lower levels is latency: a level of 12 to 10,242 vertices is one to two microseconds
// of launch, dependent loads through L2 and drain per kernel, whatever its bytes.  Measured on B200:
// a graph's chain of near-empty kernels with programmatic launch 0.9 us each, a cluster barrier 470
// cycles (0.25 us), __syncthreads 42, a load from L2 310-350, from shared memory 28.  So the small
// levels (kTailRep) are kept by every CTA, which all compute them alike with no barrier but their own;
// the larger ones have their rows split over the cluster, their neighbours in other CTAs are read
// through distributed shared memory, and only phases that read what another CTA wrote start with a
// cluster barrier.  The tables arrive once per launch by asynchronous copies that start before the
// kernel waits for its predecessor.
//
// Table entries name a row in 16 bits, (owning CTA xor own CTA) << 12 | row in the owner's run, so one
// below 4096 is local.  The arithmetic is that of the per-level kernels (sweep_rows, k_sweep_ap, k_restrict,
// k_prolong, the k_cg_* kernels with their sums over blocks of rows), rounding for rounding: a Krylov
// smoother on the singular Laplacian's coarse levels magnifies a last bit to 1e-6 of the result.
//
// Threads per CTA: a phase's cost is mostly issuing it once in every warp, so few warps with two rows a
// thread beat one row a thread.  Icosphere L6, one right-hand side in FP64, V(3,3) to 1e-10: 714 us with
// 704 threads, 625 with 512, 615 with 384, 634 with 256 (852 without this kernel).
#pragma once

template <class T>
struct TailPrm {
  const TailOp* ops;
  int nops, K;
  const unsigned char* image;        // the tables, one image of image_bytes per CTA of a cluster
  uint32_t image_bytes;
  const T* rf;                       // the residual of the level above, its transfer to the tail's finest level
  size_t rf_stride;
  const int32_t *g_rself, *g_ridx;
  const T* g_rw;
  int g_Wq;
  const T* gb;                       // panels of the tail's finest level: right-hand side, iterate in, out
  const T* gx_in;
  T* gx;
  double* gu;                        // FP64 iterate (TT_ADDU)
  uint32_t part, part_len;           // byte offset of the CG sums' block partials (two sets), entries per set
  size_t stride;
  const double* ainv;                // the coarsest operator's inverse (internal order)
};

__device__ __forceinline__ uint32_t cluster_rank() {
  uint32_t r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}
__device__ __forceinline__ uint32_t cluster_size() {
  uint32_t r;
  asm volatile("mov.u32 %0, %%cluster_nctarank;" : "=r"(r));
  return r;
}
__device__ __forceinline__ void cluster_barrier() {
  asm volatile("barrier.cluster.arrive.aligned;\n\tbarrier.cluster.wait.aligned;" ::: "memory");
}
__device__ __forceinline__ uint32_t cluster_map(uint32_t a, uint32_t rank) {
  uint32_t d;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(d) : "r"(a), "r"(rank));
  return d;
}

__device__ __forceinline__ void ld_remote(uint32_t a, float& r) {
  asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(r) : "r"(a) : "memory");
}
__device__ __forceinline__ void ld_remote(uint32_t a, double& r) {
  asm volatile("ld.shared::cluster.f64 %0, [%1];" : "=d"(r) : "r"(a) : "memory");
}
__device__ __forceinline__ void st_remote(uint32_t a, float v) {
  asm volatile("st.shared::cluster.f32 [%0], %1;" ::"r"(a), "f"(v) : "memory");
}
__device__ __forceinline__ void st_remote(uint32_t a, double v) {
  asm volatile("st.shared::cluster.f64 [%0], %1;" ::"r"(a), "d"(v) : "memory");
}

// N consecutive table entries from shared memory in 8-byte (32-bit entries) or 16-byte loads.
template <class E, int N>
__device__ __forceinline__ void ld_n(const unsigned char* p, E (&r)[N]) {
  struct alignas(2 * sizeof(E)) V2 { E v[2]; };
  const V2* q = reinterpret_cast<const V2*>(p);
#pragma unroll
  for (int k = 0; k < N / 2; ++k) {
    const V2 v = q[k];
    r[2 * k] = v.v[0];
    r[2 * k + 1] = v.v[1];
  }
}

// CL: the launch has clusters of more than one CTA.  CG: the program holds CG smoothers (FP64).
template <class T, bool CL, bool CG>
__global__ void __launch_bounds__(kTailThreads, 1) k_tail(const __grid_constant__ TailPrm<T> P) {
  constexpr int NW = kTailThreads / 32;
  constexpr uint32_t Z = sizeof(T);
  extern __shared__ __align__(16) unsigned char S[];
  __shared__ uint4 ring[4][kTailOpWords];                      // the phases ahead
  const uint32_t sbase = (uint32_t)__cvta_generic_to_shared(S);
  const uint32_t rank = CL ? cluster_rank() : 0, C = CL ? cluster_size() : 1;
  const int tid = threadIdx.x;
  auto fetch = [&](int o) {  // phase o into the ring (threads 0 .. 4; one group each)
    if (o < P.nops)
      asm volatile("cp.async.ca.shared.global [%0], [%1], 16;" ::"r"((uint32_t)__cvta_generic_to_shared(&ring[o & 3][tid])),
                   "l"(reinterpret_cast<const uint4*>(P.ops + o) + tid)
                   : "memory");
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  // the tables and the first phases do not depend on the kernel before: copied while it drains
  for (uint32_t i = (uint32_t)tid * 16; i < P.image_bytes; i += kTailThreads * 16)
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(sbase + i),
                 "l"(P.image + (size_t)rank * P.image_bytes + i)
                 : "memory");
  if (tid < kTailOpWords) {
    fetch(0);
    fetch(1);
    fetch(2);
  }
  const int col = (int)(blockIdx.x / C), panel = col / P.K, k0 = col % P.K;
  int parity = 0;
  const int rb_log = 31 - __clz(TB / P.K);  // rows per block of the CG sums: a power of two
  asm volatile("cp.async.wait_all;" ::: "memory");
  pdl_enter();
  __syncthreads();

  auto at = [&](uint32_t byte) -> T& { return *reinterpret_cast<T*>(S + byte); };
  auto local = [&](uint32_t b, int row) -> T& { return at(b + (uint32_t)row * Z); };
  auto name = [&](uint32_t t, int i) -> uint32_t { return *reinterpret_cast<const uint16_t*>(S + t + 2u * (uint32_t)i); };
  // the entry e of the vector at byte offset b: this CTA's row, or another's
  auto near = [&](uint32_t b, uint32_t e) -> T { return at(b + e * Z); };
  auto gather = [&](uint32_t b, uint32_t e) -> T {
    if (!CL || e < 4096u) return near(b, e);
    T r;
    ld_remote(cluster_map(sbase + b + (e & 4095u) * Z, (e >> 12) ^ rank), r);
    return r;
  };
  // six names (three words); true: one of them may be another CTA's
  auto names6 = [&](uint32_t t, int i, uint32_t (&e)[6]) -> bool {
    const uint32_t* q = reinterpret_cast<const uint32_t*>(S + t + 12u * (uint32_t)i);
    const uint32_t w0 = q[0], w1 = q[1], w2 = q[2];
    e[0] = w0 & 0xffffu;
    e[1] = w0 >> 16;
    e[2] = w1 & 0xffffu;
    e[3] = w1 >> 16;
    e[4] = w2 & 0xffffu;
    e[5] = w2 >> 16;
    return CL && ((w0 | w1 | w2) & 0xf000f000u) != 0;
  };
  // a_ii xi + Σ over row i's entries of a_ij x_j: near / far fetch an entry's x_j when all / not all of the
  // row's neighbours are in this CTA
  auto row = [&](const TailOp& op, int i, T xi, auto close, auto far, bool krylov = true) -> T {
    const T dg = local(op.t2, i);
    T acc;
    if (op.W == 6) {
      uint32_t cc[6];
      T vv[6], nb[6];
      const bool some = names6(op.t0, i, cc);
      ld_n(S + op.t1 + (uint32_t)i * (6 * Z), vv);
      if (!some) {
#pragma unroll
        for (int s = 0; s < 6; ++s) nb[s] = close(cc[s]);
      } else {  // one branch per row, few rows
#pragma unroll
        for (int s = 0; s < 6; ++s) nb[s] = far(cc[s]);
      }
      // the k_cg_* kernels' unrolled rows round the first off-diagonal product, sweep_rows the diagonal's
      acc = krylov ? fma_rn(dg, xi, mul_rn(vv[0], nb[0])) : fma_rn(vv[0], nb[0], mul_rn(dg, xi));
#pragma unroll
      for (int s = 1; s < 6; ++s) acc = fma_rn(vv[s], nb[s], acc);
    } else {
      acc = mul_rn(dg, xi);
#pragma unroll 4
      for (int s = 0; s < op.W; ++s) acc = fma_rn(local(op.t1, i * op.W + s), far(name(op.t0, i * op.W + s)), acc);
    }
    return acc;
  };
  // Σ f(row) over the level as the k_cg_* kernels add it: blocks of 256 / K rows in a tree of halves, then the
  // blocks' sums strided over 256 and in a tree.  Every thread of every CTA gets the same total.
  auto reduce = [&](const TailOp& op, int nr, bool own, auto f) -> double {
    const int RB = 1 << rb_log, warp = tid >> 5, lane = tid & 31, nb = (op.n + RB - 1) >> rb_log;
    const uint32_t part = P.part + (uint32_t)parity * P.part_len * 8u;
    const int b0 = own ? 0 : ((int)rank * op.chunk) >> rb_log;  // a CTA's run is whole blocks
    parity ^= 1;
    __syncthreads();
    for (int blk = warp; blk * RB < nr; blk += NW) {
      const int base = (blk << rb_log) + lane, left = min(RB, nr - (blk << rb_log)) - lane;  // rows base + 32 k, 32 k < left
      double s = 0.0;
      if (left > 0) s = f(base);
      if (nr - (blk << rb_log) > 32) {
        double v[8];
        v[0] = s;
#pragma unroll
        for (int k = 1; k < 8; ++k) v[k] = 32 * k < left ? f(base + 32 * k) : 0.0;
        if (RB == 256) s = ((v[0] + v[4]) + (v[2] + v[6])) + ((v[1] + v[5]) + (v[3] + v[7]));
        else if (RB == 128) s = (v[0] + v[2]) + (v[1] + v[3]);
        else if (RB == 64) s = v[0] + v[1];
      }
#pragma unroll
      for (int st = 16; st > 0; st >>= 1) s += __shfl_xor_sync(0xffffffffu, s, st);
      if (own) {
        if (lane == 0) *reinterpret_cast<double*>(S + part + 8u * (uint32_t)blk) = s;
      } else if (lane < (int)C) {
        st_remote(cluster_map(sbase + part + 8u * (uint32_t)(b0 + blk), (uint32_t)lane), s);
      }
    }
    if (own) __syncthreads();
    else cluster_barrier();
    const double* p = reinterpret_cast<const double*>(S + part);
    if (nb <= 4) {  // the tree of 256 with zeros from entry nb on
      if (nb == 1) return p[0];
      const double s1 = nb == 4 ? p[1] + p[3] : p[1];
      return (nb >= 3 ? p[0] + p[2] : p[0]) + s1;
    }
    double s = 0.0;
    if (nb <= 32) {
      if (lane < nb) s = p[lane];
    } else {
      double v[8];
#pragma unroll
      for (int k = 0; k < 8; ++k) {
        v[k] = 0.0;
        for (int b = lane + 32 * k; b < nb; b += TB) v[k] += p[b];
      }
      s = ((v[0] + v[4]) + (v[2] + v[6])) + ((v[1] + v[5]) + (v[3] + v[7]));
    }
#pragma unroll
    for (int st = 16; st > 0; st >>= 1) s += __shfl_xor_sync(0xffffffffu, s, st);
    return s;
  };

  for (int o = 0; o < P.nops; ++o) {
    TailOp op;
    const uint4* w = ring[o & 3];
    uint4* d = reinterpret_cast<uint4*>(&op);
    d[0] = w[0];  // kind, barrier, rows: all a warp without rows needs
    if (tid < kTailOpWords) asm volatile("cp.async.wait_group 1;" ::: "memory");  // phase o + 1 has arrived
    // every phase starts here: once, in all CTAs
    if (CL && op.barrier) cluster_barrier();
    else __syncthreads();
    const int r0 = op.rep ? 0 : (int)rank * op.chunk, nr = min(op.n - r0, op.chunk);  // this CTA's rows
    if (tid < 32) {
      if (tid < kTailOpWords) fetch(o + 3);
      __syncwarp();
    }
    if (op.type < TT_COARSE && (tid & ~31) >= nr) continue;  // phases of rows with no barrier inside
#pragma unroll
    for (int k = 1; k < kTailOpWords; ++k) d[k] = w[k];
    switch (op.type) {
      case TT_RESTRICT_G: {  // R r of the level above (global panels) into b
        const T* f = P.rf + (size_t)panel * P.rf_stride + k0;
        for (int i = tid; i < nr; i += kTailThreads) {
          const int g = r0 + i;
          const T w1 = P.g_rw[2 * (size_t)g], wh = P.g_rw[2 * (size_t)g + 1];
          T acc;
          if (P.g_Wq == 6) {
            int m[6];
            T gv[6];
#pragma unroll
            for (int e = 0; e < 6; ++e) m[e] = P.g_ridx[(size_t)g * 6 + e];
            acc = w1 * f[(size_t)P.g_rself[g] * P.K];
#pragma unroll
            for (int e = 0; e < 6; ++e)
              if (m[e] >= 0) gv[e] = f[(size_t)m[e] * P.K];
#pragma unroll
            for (int e = 0; e < 6; ++e)
              if (m[e] >= 0) acc += wh * gv[e];
          } else {
            acc = w1 * f[(size_t)P.g_rself[g] * P.K];
            for (int e = 0; e < P.g_Wq; ++e) {
              const int m = P.g_ridx[(size_t)g * P.g_Wq + e];
              if (m < 0) break;
              acc += wh * f[(size_t)m * P.K];
            }
          }
          local(op.out, i) = acc;
        }
        break;
      }
      case TT_LOAD:
      case TT_LOADX: {
        const T* s = (op.type == TT_LOAD ? P.gb : P.gx_in) + (size_t)panel * P.stride + k0;
        for (int i = tid; i < nr; i += kTailThreads) local(op.out, i) = s[(size_t)(r0 + i) * P.K];
        break;
      }
      case TT_STORE: {  // a level that every CTA keeps is written by the first
        T* s = P.gx + (size_t)panel * P.stride + k0;
        if (!op.rep || rank == 0)
          for (int i = tid; i < nr; i += kTailThreads) s[(size_t)(r0 + i) * P.K] = local(op.x, i);
        break;
      }
      case TT_ADDU: {
        double* u = P.gu + (size_t)panel * P.stride + k0;
        if (!op.rep || rank == 0)
          for (int i = tid; i < nr; i += kTailThreads) u[(size_t)(r0 + i) * P.K] += (double)local(op.x, i);
        break;
      }
      case TT_ZERO: {
        for (int i = tid; i < nr; i += kTailThreads) local(op.out, i) = T(0);
        break;
      }
      case TT_SWEEP: {
        // sweep_rows; the mode is chosen outside the row loop.  The first Chebyshev step is the recurrence
        // with c1 = 0 and x_prev = 0, from x = 0 there is no A x
        const T c1 = (T)op.p0, c2 = (T)op.p1;
        auto sweep = [&](auto tag) {
          constexpr int M = decltype(tag)::value;
          for (int i = tid; i < nr; i += kTailThreads) {
            T r = local(op.b, i), xi = T(0), prev = T(0), old = T(0), dv = T(0);
            if constexpr (!(M & TM_RESID)) dv = local(op.t3, i);
            if constexpr ((M & TM_OLD) != 0) old = local(op.out, i);
            if constexpr ((M & TM_PZ) != 0) {
              prev = add_rn(T(0), prolong_term(gather(op.z, name(op.t4, i)), gather(op.z, name(op.t5, i))));
            }
            if constexpr (!(M & TM_FROM_ZERO)) {
              xi = local(op.x, i);
              r = sub_rn(r, row(op, i, xi, [&](uint32_t e) { return near(op.x, e); },
                                [&](uint32_t e) { return gather(op.x, e); }, false));
            }
            if constexpr ((M & TM_JACOBI) != 0) {
              r = xi + c2 * (dv * r);
            } else if constexpr (!(M & TM_RESID)) {
              if constexpr ((M & TM_PREV) != 0) prev = old;  // the iterate before x is what out holds
              r = add_rn(xi, fma_rn(c1, sub_rn(xi, prev), mul_rn(c2, mul_rn(dv, r))));
              if constexpr ((M & TM_ADD) != 0) r = add_rn(old, r);  // e + δ
            }
            local(op.out, i) = r;
          }
        };
        switch (op.mode) {
#define DEC_TM(m) \
  case m: sweep(std::integral_constant<int, m>()); break;
          DEC_TM(0) DEC_TM(TM_PREV) DEC_TM(TM_RESID) DEC_TM(TM_FROM_ZERO) DEC_TM(TM_PZ) DEC_TM(TM_PZ | TM_ADD)
          DEC_TM(TM_JACOBI) DEC_TM(TM_JACOBI | TM_FROM_ZERO)
#undef DEC_TM
        }
        break;
      }
      case TT_AP: {  // k_sweep_ap from x0 = P z
        const T inv_theta = (T)op.p0;
        for (int i = tid; i < nr; i += kTailThreads) {
          uint32_t cc[8];
          T vv[8], z[8];
          const uint4 w = *reinterpret_cast<const uint4*>(S + op.t0 + (uint32_t)i * 16u);
          const uint32_t ww[4] = {w.x, w.y, w.z, w.w};
#pragma unroll
          for (int s = 0; s < 8; ++s) cc[s] = (ww[s / 2] >> (16 * (s & 1))) & 0xffffu;
          ld_n(S + op.t1 + (uint32_t)i * (8 * Z), vv);
#pragma unroll
          for (int s = 0; s < 8; ++s) {
            z[s] = T(0);
            if (s < 2 || cc[s] != kTailNone) z[s] = gather(op.z, cc[s]);
          }
          const T pzi = prolong_term(z[0], z[1]), x0 = add_rn(T(0), pzi);
          T acc = T(0);
#pragma unroll
          for (int s = 0; s < 8; ++s) acc = fma_rn(vv[s], z[s], acc);
          local(op.out, i) = add_rn(x0, mul_rn(mul_rn(local(op.t3, i), sub_rn(local(op.b, i), acc)), inv_theta));
        }
        break;
      }
      case TT_RESTRICT: {  // rows of level + 1; split: in shares, each row pushed to every CTA
        for (int i = tid; i < nr; i += kTailThreads) {
          const T w1 = local(op.t2, 2 * i), wh = local(op.t2, 2 * i + 1);
          T res = w1 * gather(op.x, name(op.t0, i));
          if (op.W == 6) {
            uint32_t m[6];
            T gv[6];
            names6(op.t1, i, m);
#pragma unroll
            for (int e = 0; e < 6; ++e)
              if (m[e] != kTailNone) gv[e] = gather(op.x, m[e]);
#pragma unroll
            for (int e = 0; e < 6; ++e)
              if (m[e] != kTailNone) res += wh * gv[e];
          } else {
            for (int e = 0; e < op.W; ++e) {
              const uint32_t m = name(op.t1, i * op.W + e);
              if (m == kTailNone) break;
              res += wh * gather(op.x, m);
            }
          }
          if (CL && op.split) {
            for (uint32_t c = 0; c < C; ++c) st_remote(cluster_map(sbase + op.out + (uint32_t)(r0 + i) * Z, c), res);
          } else {
            local(op.out, i) = res;
          }
        }
        break;
      }
      case TT_PROLONG: {
        for (int i = tid; i < nr; i += kTailThreads) {
          const T za = gather(op.z, name(op.t4, i)), zb = gather(op.z, name(op.t5, i));
          local(op.out, i) = add_rn(op.add ? local(op.out, i) : T(0), prolong_term(za, zb));
        }
        break;
      }
      case TT_COARSE: {
        // x = A⁻¹ b on the coarsest level (kept by every CTA), a warp per row; split: the rows are shared
        // out and every result is pushed to all CTAs
        const bool split = CL && op.split;
        for (int i = (split ? (int)rank * NW : 0) + (tid >> 5); i < op.n; i += (split ? (int)C : 1) * NW) {
          const double* a = P.ainv + (size_t)i * op.n;
          double s = 0.0;
#pragma unroll 8
          for (int j = tid & 31; j < op.n; j += 32) s += __ldg(a + j) * (double)local(op.b, j);
#pragma unroll
          for (int st = 16; st > 0; st >>= 1) s += __shfl_xor_sync(0xffffffffu, s, st);
          const uint32_t c = (uint32_t)(tid & 31);  // lane c writes CTA c's copy
          if (c < (split ? C : 1u)) {
            if (split) st_remote(cluster_map(sbase + op.out + (uint32_t)i * Z, c), (T)s);
            else local(op.out, i) = (T)s;
          }
          __syncwarp();
        }
        break;
      }
      case TT_CG: {  // Krylov.jl's cg with itmax = steps (the k_cg_* kernels), x in place
        if constexpr (CG) {
          const bool own = !CL || op.rep;
          const uint32_t bx = op.x, br = op.out, bq = op.t5, be = op.zero ? op.x : op.t6;  // be: Δx
          uint32_t bp = op.z, bn = op.t4;
          for (int i = tid; i < nr; i += kTailThreads) {
            T rv = local(op.b, i);
            if (!op.zero)
              rv = rv - row(op, i, local(bx, i), [&](uint32_t e) { return near(bx, e); },
                            [&](uint32_t e) { return gather(bx, e); });
            local(br, i) = rv;
            local(be, i) = T(0);
          }
          auto rr = [&](int i) -> double { return mul_rn(local(br, i), local(br, i)); };
          const double eps = 2.220446049250313e-16, rt = 1.4901161193847656e-08;
          double gamma = reduce(op, nr, own, rr), beta = 0.0, pn2 = gamma;
          const double r0n = sqrt(gamma), tol = rt + rt * r0n;
          const int steps = op.steps;
          const bool active = gamma != 0.0 && !(r0n <= tol) && steps > 0;
          // every scalar below is the same in all threads of all CTAs (the sums run in one order), so the
          // loop ends at the same step everywhere
          for (int it = 0; active && it < steps; ++it) {
            if (it == 0) {  // p = r
              for (int i = tid; i < nr; i += kTailThreads) {
                const T pi = local(br, i);
                local(bq, i) = row(op, i, pi, [&](uint32_t e) { return near(br, e); },
                                   [&](uint32_t e) { return gather(br, e); });
                local(bn, i) = pi;
              }
            } else {  // p = r + β p, formed for the row and for its neighbours alike
              const T bt = (T)beta;
              for (int i = tid; i < nr; i += kTailThreads) {
                const T pi = fma_rn(bt, local(bp, i), local(br, i));
                local(bq, i) = row(op, i, pi, [&](uint32_t e) { return fma_rn(bt, near(bp, e), near(br, e)); },
                                   [&](uint32_t e) { return fma_rn(bt, gather(bp, e), gather(br, e)); });
                local(bn, i) = pi;
              }
            }
            const double pap = reduce(op, nr, own, [&](int i) -> double { return mul_rn(local(bn, i), local(bq, i)); });
            if (pap <= eps * pn2 && fabs(pap) <= eps * pn2) break;  // zero curvature
            const double alpha = gamma / pap;
            for (int i = tid; i < nr; i += kTailThreads) {
              local(be, i) = fma_rn((T)alpha, local(bn, i), local(be, i));
              local(br, i) = fma_rn((T)-alpha, local(bq, i), local(br, i));
            }
            const double gnext = reduce(op, nr, own, rr), rnorm = sqrt(gnext);
            if (rnorm <= tol || rnorm + 1.0 <= 1.0) break;
            beta = gnext / gamma;
            pn2 = gnext + beta * beta * pn2;
            gamma = gnext;
            const uint32_t t = bp;
            bp = bn;
            bn = t;
          }
          if (!op.zero)
            for (int i = tid; i < nr; i += kTailThreads) local(bx, i) = local(be, i) + local(bx, i);
        }
        break;
      }
    }
  }
  if (CL) cluster_barrier();  // no CTA leaves while another may still read its shared memory
}

// The tables of one level in the CTA images.  Per image (blockIdx.y = CTA) and row; src_* are the level's
// arrays in its internal numbering.
template <class T>
struct TailPack {
  TailLevel L, Lc;
  int C, has_a, has_dinv, has_p, has_ap, has_r;
  const int32_t *col, *pa, *pb, *apc, *rself, *ridx;
  const T *off, *diag, *dinv, *apv, *rw;
  unsigned char* image;
  size_t image_bytes;
};

template <class T>
__global__ void k_tail_pack(TailPack<T> p) {
  const int rank = blockIdx.y;
  unsigned char* im = p.image + (size_t)rank * p.image_bytes;
  auto name = [&](const TailLevel& L, int r) -> uint16_t {
    if (r < 0) return kTailNone;
    if (L.rep) return (uint16_t)r;
    return (uint16_t)(((r / L.chunk) ^ rank) << 12 | (r % L.chunk));
  };
  const TailLevel& L = p.L;
  const int r0 = L.rep ? 0 : rank * L.chunk, nr = max(0, min(L.n - r0, L.chunk));
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < nr; i += gridDim.x * blockDim.x) {
    const size_t g = (size_t)(r0 + i);
    if (p.has_a)
      for (int s = 0; s < L.W; ++s) {
        reinterpret_cast<uint16_t*>(im + L.t_col)[i * L.W + s] = name(L, p.col[g * L.W + s]);
        reinterpret_cast<T*>(im + L.t_off)[i * L.W + s] = p.off[g * L.W + s];
      }
    reinterpret_cast<T*>(im + L.t_diag)[i] = p.diag[g];
    if (p.has_dinv) reinterpret_cast<T*>(im + L.t_dinv)[i] = p.dinv[g];
    if (p.has_p) {
      reinterpret_cast<uint16_t*>(im + L.t_pa)[i] = name(p.Lc, p.pa[g]);
      reinterpret_cast<uint16_t*>(im + L.t_pb)[i] = name(p.Lc, p.pb[g]);
    }
    if (p.has_ap)
      for (int s = 0; s < kApW; ++s) {
        reinterpret_cast<uint16_t*>(im + L.t_apc)[i * kApW + s] = name(p.Lc, p.apc[g * kApW + s]);
        reinterpret_cast<T*>(im + L.t_apv)[i * kApW + s] = p.apv[g * kApW + s];
      }
  }
  if (!p.has_r) return;
  const int c0 = (p.Lc.rep && L.rep) ? 0 : rank * L.rchunk, ncr = max(0, min(p.Lc.n - c0, L.rchunk));
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < ncr; i += gridDim.x * blockDim.x) {
    const size_t g = (size_t)(c0 + i);
    reinterpret_cast<uint16_t*>(im + L.t_rself)[i] = name(L, p.rself[g]);
    for (int s = 0; s < L.Wq; ++s)
      reinterpret_cast<uint16_t*>(im + L.t_ridx)[i * L.Wq + s] = name(L, p.ridx[g * L.Wq + s]);
    reinterpret_cast<T*>(im + L.t_rw)[2 * i] = p.rw[2 * g];
    reinterpret_cast<T*>(im + L.t_rw)[2 * i + 1] = p.rw[2 * g + 1];
  }
}
