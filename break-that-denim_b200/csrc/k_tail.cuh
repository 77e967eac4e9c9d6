// The V-cycle's coarsest levels in one launch: every level whose colours have at most TAIL_CTAS lines is
// swept by one thread-block cluster, a CTA a line.
//
// On these levels (33^2 and 17^2 nodes under a 256^2 lattice) a colour's line solves take less time than the
// launch between two colours, and a V-cycle has 24 such colours and their transfers. Here the levels'
// unknowns stay in shared memory, a copy in every CTA: a CTA solves its line (k_line.cuh), sends the new
// unknowns to all copies over distributed shared memory (st.async), whose arrival - counted in bytes by an
// mbarrier a CTA - is the only synchronisation between two colours (plain stores and a cluster-scope release
// took 0.5 us more a colour for the fence). The lines' coefficients (a line is visited once or twice a
// V-cycle) are loaded from L2 into registers a colour ahead, while the exchange is under way.
//
// Every CTA sends in every exchange (one without a line sends a 16-byte token), so no CTA can be more than
// one exchange ahead of another: two mbarriers in turn suffice, and what a CTA reads of its copy before it
// sends is not overwritten under it. The waits are bounded (mbarWaitBounded). A CTA whose wait runs out in both
// bounds (a bug; its error flag is up) goes on without the turn that the others are at. So that nothing is then
// sent to a CTA that has left, all leave together, after a barrier of the cluster (every CTA's way to it is
// bounded; it costs nothing that can be measured, 101.8 us a V-cycle of 64 x 64 nodes with it and without).
#pragma once

#include "k_line.cuh"

namespace btd {

constexpr int TAIL_CTAS = 16;
constexpr int TAIL_SIDE = 3 * TAIL_CTAS;  // nodes a side: at most TAIL_CTAS lines a colour
constexpr int TAIL_THREADS = 192;         // four a node of a line
constexpr int TAIL_LEVELS = 4, TAIL_VISITS = 64, TAIL_OPS = TAIL_VISITS + 2 * TAIL_LEVELS;
static_assert(cutThreads(TAIL_SIDE) <= TAIL_THREADS, "a line's threads");

enum TailOp : int { TAIL_PASS = 0, TAIL_RESTRICT = 1, TAIL_PROLONG = 2 };

// One CTA's part of a colour: its line (len 0: none) and the bytes that every copy receives in it.
struct TailVisit {
  int len, fac, n0, st, x0, along, across, level;
  int P, base, extra, bytes;
};

struct TailLevel {
  DLevel d;
  int x0;  // node (0, 0) in the copy (float4 index; rows of nx + 4, two zeros around the lattice)
  int W;
  int b0;  // the right-hand side (float4 index), -1: the first level's, in global memory
};

struct TailArgs {
  TailLevel lev[TAIL_LEVELS];
  const float4* fac[TAIL_LEVELS];
  const TailVisit* visits;  // [colour][CTA]
  const int* ops;           // (TailOp, level) pairs
  int levels, op0, op1, visit0, visits1;
  int rAt, tokenAt, scratchAt, f4;  // float4 indices: residuals, the tokens' slot, the solve's scratch; total
  int load;  // resume at the learned correction between the coarsest sweeps
  uint32_t* err;
};

__device__ __forceinline__ unsigned clusterRank() {
  unsigned r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;\n" : "=r"(r));
  return r;
}
__device__ __forceinline__ void clusterArrive() { asm volatile("barrier.cluster.arrive.release.aligned;\n" ::: "memory"); }
__device__ __forceinline__ void clusterArriveRelaxed() { asm volatile("barrier.cluster.arrive.relaxed.aligned;\n" ::: "memory"); }
__device__ __forceinline__ void clusterWait() { asm volatile("barrier.cluster.wait.acquire.aligned;\n" ::: "memory"); }
__device__ __forceinline__ unsigned mapaOf(unsigned addr, unsigned rank) {
  unsigned r;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;\n" : "=r"(r) : "r"(addr), "r"(rank));
  return r;
}
// 16 bytes to a CTA of the cluster, counted by its mbarrier.
__device__ __forceinline__ void sendAsync(unsigned dst, unsigned bar, float x, float y, float z, float w) {
  asm volatile("st.async.shared::cluster.mbarrier::complete_tx::bytes.v4.f32 [%0], {%1, %2, %3, %4}, [%5];\n" ::"r"(dst), "f"(x), "f"(y),
               "f"(z), "f"(w), "r"(bar)
               : "memory");
}
// mbarTryWait for what other CTAs of the cluster sent.
__device__ __forceinline__ bool mbarTryWaitCluster(uint64_t* bar, unsigned parity) {
  unsigned ok;
  asm volatile(
      "{\n .reg .pred p;\n mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}\n"
      : "=r"(ok)
      : "r"(smemAddr(bar)), "r"(parity)
      : "memory");
  return ok != 0;
}

// Bytes that every copy receives when N nodes are sent by `senders` CTAs (the others send a token).
__host__ __device__ constexpr int tailBytes(int N, int senders) { return 16 * (N + TAIL_CTAS - senders); }
// Nodes of a level dealt to the CTAs in runs.
__host__ __device__ constexpr int tailRun(int N) { return (N + TAIL_CTAS - 1) / TAIL_CTAS; }

template <class Rows>
__global__ void __launch_bounds__(TAIL_THREADS, 1) k_tail(TailArgs a) {
  __shared__ uint64_t bars[2];
  __shared__ TailVisit sv[TAIL_VISITS];
  __shared__ int sops[2 * TAIL_OPS];
  extern __shared__ float4 sm4[];
  const int tid = threadIdx.x, nt = blockDim.x, lane = tid & 3;
  const int rank = (int)clusterRank();
  const int visits = a.visits1 - a.visit0;
  for (int q = tid; q < visits * (int)(sizeof(TailVisit) / 4); q += nt) {
    const int v = q / (int)(sizeof(TailVisit) / 4), w = q % (int)(sizeof(TailVisit) / 4);
    reinterpret_cast<int*>(sv)[q] = __ldg(reinterpret_cast<const int*>(a.visits + (size_t)(a.visit0 + v) * TAIL_CTAS + rank) + w);
  }
  for (int q = tid; q < 2 * (a.op1 - a.op0); q += nt) sops[q] = __ldg(a.ops + 2 * a.op0 + q);
  const int firstTries = g_mbarFirstTries;
  for (int q = tid; q < a.f4; q += nt) sm4[q] = make_float4(0, 0, 0, 0);
  if (tid == 0) {
    mbarInit(&bars[0], 1);
    mbarInit(&bars[1], 1);
  }
  __syncthreads();
  // the coefficients of visits v and v + 1: two sets in turn, so that a set is loaded two colours ahead
  CutRegs<Rows> regs0, regs1;
  float b0 = 0.f, b1 = 0.f;
  auto coefs = [&](CutRegs<Rows>& R, int v) {
    if (v >= visits) return;
    const TailVisit& t = sv[v];
    if (t.len > 0) cutLoad<Rows>(R, a.fac[t.level] + t.fac, t.len, Cut(t.P, t.base, t.extra));
  };
  auto rhs = [&](float& b, int v) {  // the first level's right-hand side, the thread's component
    if (v >= visits) return;
    const TailVisit& t = sv[v];
    if (t.len > 0 && t.level == 0 && lane < 3) b = __ldcg(reinterpret_cast<const float*>(a.lev[0].d.B + t.n0 + min(tid >> 2, t.len - 1) * t.st) + lane);
  };
  auto ready = [&](CutRegs<Rows>& R, int v) {
    if (v < visits && sv[v].len > 0) cutReady<Rows>(R, sv[v].len);
  };
  coefs(regs0, 0);
  coefs(regs1, 1);
  clusterArrive();
  clusterWait();  // every copy is zeroed and every mbarrier initialised before anything is sent
  pdlWait();
  pdlLaunchNext();
  rhs(b0, 0);
  rhs(b1, 1);
  ready(regs0, 0);
  auto copyIndex = [](const TailLevel& L, int n) {
    const int j = n / L.d.one.nx;
    return L.x0 + j * L.W + (n - j * L.d.one.nx);
  };
  if (a.load) {
    for (int l = 0; l < a.levels; ++l) {
      const TailLevel& L = a.lev[l];
      for (int n = tid; n < L.d.N; n += nt) {
        sm4[copyIndex(L, n)] = __ldcg(L.d.X + n);
        if (L.b0 >= 0) sm4[L.b0 + n] = __ldcg(L.d.B + n);
      }
    }
    __syncthreads();
    clusterArrive();
    clusterWait();
  }
  // this thread's destinations' copies and mbarriers: of a line's node its quad's lanes share the CTAs
  const unsigned smBase = smemAddr(sm4), barBase = smemAddr(bars);
  unsigned toCopy[TAIL_CTAS / 4], toBar[TAIL_CTAS / 4];
#pragma unroll
  for (int d = 0; d < TAIL_CTAS / 4; ++d) {
    toCopy[d] = mapaOf(smBase, lane * (TAIL_CTAS / 4) + d);
    toBar[d] = mapaOf(barBase, lane * (TAIL_CTAS / 4) + d);
  }
  int exchange = 0;
  // 16 bytes to CTA dst's copy; the exchange's token of a CTA with nothing to send; and, `bytes` being what
  // every CTA receives, `work` and then the wait for them
  auto send = [&](int f4, int dst, float3 v) {
    sendAsync(mapaOf(smBase + 16u * f4, dst), mapaOf(smemAddr(&bars[exchange & 1]), dst), v.x, v.y, v.z, 0.f);
  };
  auto token = [&]() {
    __syncthreads();  // no warp falls a whole turn of the two mbarriers behind
    if (tid < TAIL_CTAS) send(a.tokenAt, tid, make_float3(0, 0, 0));
  };
  auto exchanged = [&](int bytes, auto work) {
    uint64_t* bar = &bars[exchange & 1];
    if (tid == 0) mbarExpectTx(bar, (unsigned)bytes);
    work();
    mbarWaitBounded(
        bar, (unsigned)(exchange >> 1) & 1u, a.err, [](uint64_t* b, unsigned p) { return mbarTryWaitCluster(b, p); }, firstTries);
    ++exchange;
  };
  // one colour: visit v with its coefficients R, which are then loaded for visit v + 2; `other` are v + 1's
  auto pass = [&](const TailLevel& L, int v, CutRegs<Rows>& R, float& b0, CutRegs<Rows>& other) {
    const TailVisit& t = sv[v];
    if (t.len > 0) {
      const CutScratch s = cutScratch(sm4 + a.scratchAt, t.len);
      const int xi = t.x0 + R.k * t.along;
      const float3 acc = cutCouplings(R, sm4 + xi, [&](int q) { return sm4 + xi + q * t.across; }, t.along);
      const float b = L.b0 < 0 ? b0 : lane < 3 ? reinterpret_cast<const float*>(sm4 + L.b0 + t.n0 + R.k * t.st)[lane] : 0.f;
      const float r = b - (lane == 0 ? acc.x : lane == 1 ? acc.y : acc.z);
      const float4 old = sm4[xi];
      if (lane < 3 && tid < 4 * t.len) {
        if (R.interior)
          s.rI[R.t * CUT_Q + 3 * R.p + lane] = r;
        else
          s.rS[3 * R.t + lane] = r;
      }
      const float x = cutSolve(R, s, t.P);
      const int quad = tid & 28;
      float3 o = make_float3(__shfl_sync(0xffffffffu, x, quad), __shfl_sync(0xffffffffu, x, quad + 1), __shfl_sync(0xffffffffu, x, quad + 2));
      if (R.fixedNode) o = f3(old);
      if (tid < 4 * t.len) {
        const unsigned bar = 8u * (exchange & 1);
#pragma unroll
        for (int d = 0; d < TAIL_CTAS / 4; ++d) sendAsync(toCopy[d] + 16u * xi, toBar[d] + bar, o.x, o.y, o.z, 0.f);
      }
    } else {
      token();
    }
    exchanged(t.bytes, [&] {
      coefs(R, v + 2);
      rhs(b0, v + 2);
      ready(other, v + 1);
    });
  };
  int v = 0;
  for (int op = 0; op < a.op1 - a.op0; ++op) {
    const int kind = sops[2 * op], l = sops[2 * op + 1];
    const TailLevel& L = a.lev[l];
    if (kind == TAIL_PASS) {
      if (v & 1)
        pass(L, v, regs1, b1, regs0);
      else
        pass(L, v, regs0, b0, regs1);
      ++v;
    } else if (kind == TAIL_RESTRICT) {
      // r = b - A x of this CTA's run of nodes, eight lanes a node (see coarseResidualLane), to every copy
      const TailLevel& C = a.lev[l + 1];
      const int run = tailRun(L.d.N), first = rank * run, count = max(0, min(run, L.d.N - first));
      const int lane8 = tid & 7;
      if constexpr (CutOf<Rows>::RHS == 9) {
        for (int q = tid >> 3; q < (count + nt / 8 - 1) / (nt / 8) * (nt / 8); q += nt / 8) {
          const bool valid = q < count;
          const int n = first + (valid ? q : 0), j = n / L.d.one.nx, i = n - j * L.d.one.nx;
          float3 s = make_float3(0, 0, 0);
          if (valid && lane8 < 5) {
            const int f0 = 30 * lane8, p0 = f0 >> 2;
            float4 pl[9];
#pragma unroll
            for (int p = 0; p < 9; ++p) pl[p] = p0 + p < COARSE_PLANES ? __ldg(L.d.op + (size_t)(p0 + p) * L.d.N + n) : make_float4(0, 0, 0, 0);
            const float* w = reinterpret_cast<const float*>(pl);
            const float4* x = sm4 + L.x0 + (j + lane8 - 2) * L.W + i;
            const bool half = (f0 & 3) != 0;  // the row starts two floats into its first plane
#pragma unroll
            for (int d = 0; d < 5; ++d) {
              float c[6];
#pragma unroll
              for (int e = 0; e < 6; ++e) c[e] = half ? w[6 * d + e + 2] : w[6 * d + e];
              s += Sym{c[0], c[1], c[2], c[3], c[4], c[5]} * f3(x[d - 2]);
            }
          }
#pragma unroll
          for (int m = 4; m >= 1; m >>= 1) {
            s.x += __shfl_xor_sync(0xffffffffu, s.x, m);
            s.y += __shfl_xor_sync(0xffffffffu, s.y, m);
            s.z += __shfl_xor_sync(0xffffffffu, s.z, m);
          }
          if (valid) {
            const float4 b = L.b0 < 0 ? __ldcg(L.d.B + n) : sm4[L.b0 + n];
            const float3 r = L.d.fixed[n] ? make_float3(0, 0, 0) : f3(b) - s;
            if (lane8 == 0) L.d.R[n] = make_float4(r.x, r.y, r.z, 0.f);
#pragma unroll
            for (int d = 0; d < TAIL_CTAS / 8; ++d) send(a.rAt + n, lane8 * (TAIL_CTAS / 8) + d, r);
          }
        }
      }
      if (count == 0) token();
      exchanged(tailBytes(L.d.N, (L.d.N + run - 1) / run), [] {});
      // b of the next level, in every copy (restrictAt)
      const DLevelLayer Lf = L.d.one, Lc = C.d.one;
      for (int I = tid; I < C.d.N; I += nt) {
        const int cj = I / Lc.nx, ci = I - cj * Lc.nx;
        const int fi0 = coarseToFine(ci, Lf.nx), fj0 = coarseToFine(cj, Lf.ny);
        float3 s = make_float3(0, 0, 0);
        const uint32_t fixedRow = C.d.fixed[I];
#pragma unroll
        for (int q = 0; q < 9; ++q) {
          const int ai = fi0 - 1 + q % 3, aj = fj0 - 1 + q / 3;
          const bool use = ai >= 0 && ai < Lf.nx && aj >= 0 && aj < Lf.ny && weightOf(ai, ci, Lf.nx) != 0.f && weightOf(aj, cj, Lf.ny) != 0.f;
          const int n = use ? aj * Lf.nx + ai : fj0 * Lf.nx + fi0;
          const float4 w = __ldg(L.d.pw + n);
          const Bracket bai = bracketOf(ai, Lf.nx), baj = bracketOf(aj, Lf.ny);
          if (use) s += pwSlot(w, (bai.lo == ci ? 0 : 1) + 2 * (baj.lo == cj ? 0 : 1)) * f3(sm4[a.rAt + n]);
        }
        sm4[C.b0 + I] = fixedRow ? make_float4(0, 0, 0, 0) : make_float4(s.x, s.y, s.z, 0.f);
      }
      __syncthreads();
    } else {
      // x += P x_c in every copy (prolongAt), before any CTA sends its next line
      const TailLevel& C = a.lev[l + 1];
      const DLevelLayer Lf = L.d.one;
      for (int n = tid; n < L.d.N; n += nt) {
        const int j = n / Lf.nx, i = n - j * Lf.nx;
        const Bracket bi = bracketOf(i, Lf.nx), bj = bracketOf(j, Lf.ny);
        const float4 w = __ldg(L.d.pw + n);
        float3 s = make_float3(0, 0, 0);
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          const float wk = pwSlot(w, q);
          if (wk != 0.f) s += wk * f3(sm4[C.x0 + ((q & 2) ? bj.hi : bj.lo) * C.W + ((q & 1) ? bi.hi : bi.lo)]);
        }
        if (!L.d.fixed[n]) {
          float4& x = sm4[L.x0 + j * L.W + i];
          x = make_float4(x.x + s.x, x.y + s.y, x.z + s.z, 0.f);
        }
      }
      clusterArrive();
      clusterWait();
    }
  }
  __syncthreads();
  clusterArriveRelaxed();
  // the levels' vectors, as the launches of every step would leave them: for the learned correction, the
  // resumed call and readers
  for (int l = 0; l < a.levels; ++l) {
    const TailLevel& L = a.lev[l];
    const int run = tailRun(L.d.N), first = rank * run, end = min(first + run, L.d.N);
    for (int n = first + tid; n < end; n += nt) {
      L.d.X[n] = sm4[copyIndex(L, n)];
      if (L.b0 >= 0) L.d.B[n] = sm4[L.b0 + n];
    }
  }
  clusterWait();
}

}  // namespace btd
