// The compact yarn-line sweep: the same exact line solves as k_smooth, in a form
// whose every step is a short dot product of coefficients already in registers.
//
// A line of len nodes is cut by single separator nodes into P chunks of at most CUT_M nodes. With the
// separators' unknowns given, every chunk's interior is its own small system, so the line solve is
//   rr  = r_S - E r_I          at the separators (E: the couplings into the two chunks beside it times
//                              those chunks' inverses, 3 rows of 2 Q floats)
//   x_S = D rr                 D the inverse of the separators' Schur complement, dense
//   x_I = C r_I + V x_l + W x_r  C the chunk's inverse, V and W its response to its two separators
// three products with a barrier between them. k_line_compact forms D, C, V and W once per operator in
// FP64 (rows regularised by lineShift, as in k_line_factor), and E from C as it is stored; it stores all in FP32
// in the order in which the sweep's threads read them; k_sweep loads them - and its node's off-line couplings - into registers before the
// grid-dependency wait, while the launch before it still runs.
//
// What bounds it: the dependent chain of one line and the boundary between two launches, not bytes (a coarse
// colour launch moves 1 to 5 MB). After the wait there is one L2 round trip (five columns of unknowns, 0.7 us),
// 54 FMAs a thread for the right-hand side (four threads a node, a stencil row each, 0.25 us) and three dots of
// 16 to 32 terms (0.45 us); the next launch's wait returns 1.1 us after the last store. A colour of a 64 x 64
// lattice takes 2.6 us where k_smooth's took 3.3, and 2.9 where 3.5 at 128 x 128.
//
// A sweep is 5e-7 to 1.3e-5 of its result from the FP64 oracle's on sheets at rest, as k_smooth's is, and 2e-5 to 6e-5
// on a taut or torn patch (lineShift says what it is without the reference's shifts).
#pragma once

#include "k_smooth.cuh"

namespace btd {

// Nodes of a chunk and its padded unknowns: 5 nodes keep a chunk's row at four float4 and the
// separators' dense rows at two rounds of eight lanes up to CUT_LINE nodes.
constexpr int CUT_M = 5, CUT_Q = 16, CUT_ROUNDS = 2;
// Lines up to here: 6 (21 + 1) - 1 nodes have 21 separators, whose 63 unknowns fill the two rounds.
constexpr int CUT_LINE = 131;
constexpr int CUT_ROW = CUT_Q / 4 + 2;    // float4 of an interior unknown's row (C, then V and W)
constexpr int CUT_SEP = 2 * CUT_Q / 16;   // float4 a lane of a separator unknown's E row (four lanes)

// Float4 of couplings a thread holds. Coarse rows: five blocks of a stencil row across the line and, lanes
// 0 and 1, the block -2 or +2 along it (lane 3: the majorisation and the fixed flag instead). Fine rows:
// lanes 0 and 1 take the row before the line and lanes 2 and 3 the one after it, the even lane its blocks
// -1 and 0 along, the odd lane its block +1, its scalar two across, the scalar -2 or +2 along, the
// majorisation (lane 3) and the fixed flag.
template <class Rows>
struct CutOf;
template <>
struct CutOf<CoarseRows> {
  static constexpr int RHS = 9;
};
template <>
struct CutOf<FineRows> {
  static constexpr int RHS = 3;
};

// The cut of a line: chunk t starts at node start(t), holds size(t) nodes and is followed by separator t.
struct Cut {
  int P, base, extra;
  float rbe, rb;  // 1 / (base + 2), 1 / (base + 1): cells of a chunk and its separator (see Chunks)
  __host__ __device__ Cut(int P_, int base_, int extra_)
      : P(P_), base(base_), extra(extra_), rbe(1.0f / (float)(base_ + 2)), rb(1.0f / (float)(base_ + 1)) {}
  __host__ __device__ explicit Cut(int len) : Cut(parts(len), (len - parts(len) + 1) / parts(len), (len - parts(len) + 1) % parts(len)) {}
  __host__ __device__ Cut() : Cut(1, 1, 0) {}
  __host__ __device__ static constexpr int parts(int len) { return (len + 1 + CUT_M) / (CUT_M + 1); }
  __device__ int start(int t) const { return t * (base + 1) + min(t, extra); }
  __device__ int size(int t) const { return base + (t < extra ? 1 : 0); }
  __device__ int of(int k) const {
    const int cut = extra * (base + 2);
    return k < cut ? (int)(((float)k + 0.5f) * rbe) : extra + (int)(((float)(k - cut) + 0.5f) * rb);
  }
};

// A line's region (float4): the couplings [RHS][4 len], the interior rows [CUT_ROW][3 I], the
// separators' E [CUT_SEP][3 S][4 lanes] and D [CUT_ROUNDS][3 S][8 lanes]; S = P - 1, I = len - S.
__host__ __device__ constexpr int cutInterior(int len) { return len - Cut::parts(len) + 1; }
__host__ __device__ constexpr int cutSeparators(int len) { return Cut::parts(len) - 1; }
template <class Rows>
__host__ __device__ constexpr int cutRowsAt(int len) {
  return CutOf<Rows>::RHS * 4 * len;
}
template <class Rows>
__host__ __device__ constexpr int cutSepAt(int len) {
  return cutRowsAt<Rows>(len) + CUT_ROW * 3 * cutInterior(len);
}
template <class Rows>
__host__ __device__ constexpr int cutDenseAt(int len) {
  return cutSepAt<Rows>(len) + CUT_SEP * 12 * cutSeparators(len);
}
template <class Rows>
__host__ __device__ constexpr int cutF4(int len) {
  return cutDenseAt<Rows>(len) + CUT_ROUNDS * 24 * cutSeparators(len);
}
// Four threads a node.
__host__ __device__ constexpr int cutThreads(int len) { return (4 * len + 31) / 32 * 32; }

// ------------------------------------------------------------------------------------------ FP64 3x3

struct M3d {
  double a[9];
};
__device__ __forceinline__ M3d m3dZero() { return {{0, 0, 0, 0, 0, 0, 0, 0, 0}}; }
__device__ __forceinline__ M3d m3dSym(const float* s) {
  return {{s[0], s[1], s[2], s[1], s[3], s[4], s[2], s[4], s[5]}};
}
__device__ __forceinline__ M3d m3dMul(const M3d& x, const M3d& y) {
  M3d o;
#pragma unroll
  for (int r = 0; r < 3; ++r)
#pragma unroll
    for (int c = 0; c < 3; ++c) o.a[3 * r + c] = x.a[3 * r] * y.a[c] + x.a[3 * r + 1] * y.a[3 + c] + x.a[3 * r + 2] * y.a[6 + c];
  return o;
}
__device__ __forceinline__ M3d m3dAdd(const M3d& x, const M3d& y, double s = 1.0) {
  M3d o;
#pragma unroll
  for (int q = 0; q < 9; ++q) o.a[q] = x.a[q] + s * y.a[q];
  return o;
}
__device__ __forceinline__ void m3dVec(const M3d& x, const double* v, double* o) {
#pragma unroll
  for (int r = 0; r < 3; ++r) o[r] = x.a[3 * r] * v[0] + x.a[3 * r + 1] * v[1] + x.a[3 * r + 2] * v[2];
}
// The inverse of a pivot block in FP64, with pivotInverse's fallback. The shift of the reference's pivots
// (PIVOT_SHIFT) is added to the line's rows beforehand (lineShift): the cut's pivots are not the reference's.
__device__ __forceinline__ M3d pivotInverseD(const M3d& m) {
  const double s = fmax(fmax(fabs(m.a[0]), fabs(m.a[4])), fabs(m.a[8]));
  const double e = 1e-30;
  const double a00 = m.a[0] + e, a01 = m.a[1], a02 = m.a[2], a10 = m.a[3], a11 = m.a[4] + e, a12 = m.a[5], a20 = m.a[6],
               a21 = m.a[7], a22 = m.a[8] + e;
  const double c00 = a11 * a22 - a12 * a21, c01 = a12 * a20 - a10 * a22, c02 = a10 * a21 - a11 * a20;
  const double id = 1.0 / (a00 * c00 + a01 * c01 + a02 * c02);
  M3d o = {{c00 * id, (a02 * a21 - a01 * a22) * id, (a01 * a12 - a02 * a11) * id, c01 * id, (a00 * a22 - a02 * a20) * id,
            (a02 * a10 - a00 * a12) * id, c02 * id, (a01 * a20 - a00 * a21) * id, (a00 * a11 - a01 * a10) * id}};
  bool ok = true;
#pragma unroll
  for (int q = 0; q < 9; ++q) ok = ok && isfinite(o.a[q]);
  if (!ok) {
    const double d = 1.0 / fmax(s, 1e-30);
    o = {{d, 0, 0, 0, d, 0, 0, 0, d}};
  }
  return o;
}

// ------------------------------------------------------------------------------------------ factor

// Threads of k_line_compact: three CTAs an SM, so that the 256 to 300 lines of a 128 x 128 or 182 x 115 lattice
// are one wave (with four threads a node they were two).
constexpr int CUT_FACTOR_THREADS = 256;

// Shared memory of k_line_compact (doubles): Minv, Minv A and G of every node (27; the dense inverse of the
// separators' system takes their place), first and last rows of V and W of every chunk (36), the separators'
// L, D, U (27); then B, C and the shift of every node in floats (13).
__host__ __device__ constexpr size_t cutFactorSmem(int len) {
  const size_t S = (size_t)cutSeparators(len), a = 27 * (size_t)len, b = 9 * S * S;
  return 8 * ((a > b ? a : b) + 36 * (S + 1) + 27 * S) + 52 * (size_t)len;
}

__device__ __forceinline__ M3d m3dGet(const double* p) {
  M3d m;
#pragma unroll
  for (int q = 0; q < 9; ++q) m.a[q] = p[q];
  return m;
}
__device__ __forceinline__ void m3dPut(double* p, const M3d& m) {
#pragma unroll
  for (int q = 0; q < 9; ++q) p[q] = m.a[q];
}

// One cut of a block-tridiagonal line whose row k is A(k) x_{k-1} + B(k) x_k + C(k) x_{k+1}: its interior rows
// (C, V, W) and E into `out` (float4; E at sepAt), its separators' L, D, U into sR. The whole CTA calls it; it
// ends with a barrier.
template <class GetA, class GetB, class GetC>
__device__ void cutFactor(const Cut& cut, int len, GetA A, GetB B, GetC C, double* sF, double* sVW, double* sR, float4* out, int sepAt) {
  const int P = cut.P, S = P - 1, I3 = 3 * (len - S), tid = threadIdx.x, nt = blockDim.x;
  auto F = [&](int k, int which) { return sF + 27 * k + 9 * which; };
  // chunk interiors: pivot inverses, Minv A and G = Minv C, a thread a chunk
  if (tid < P) {
    const int a = cut.start(tid), b = a + cut.size(tid);
    M3d G = m3dZero();
    for (int k = a; k < b; ++k) {
      const M3d Ak = k > a ? A(k) : m3dZero();
      const M3d Minv = pivotInverseD(m3dAdd(B(k), m3dMul(Ak, G), -1.0));
      G = k + 1 < b ? m3dMul(Minv, C(k)) : m3dZero();
      m3dPut(F(k, 0), Minv);
      m3dPut(F(k, 2), G);
    }
  }
  __syncthreads();
  for (int k = tid; k < len; k += nt) {
    const int t = cut.of(k), p = k - cut.start(t);
    if (p < cut.size(t)) m3dPut(F(k, 1), p > 0 ? m3dMul(m3dGet(F(k, 0)), A(k)) : m3dZero());
  }
  __syncthreads();
  // columns of the chunks' inverses and of their responses to the separators (V: the one before, W: the one
  // after), a thread a column: CUT_Q (padded with zeros) and four each
  float* rows = reinterpret_cast<float*>(out);  // float4 plane p of unknown o: rows[4 (p I3 + o)]
  constexpr int COLS = CUT_Q + 8;
  for (int w = tid; w < P * COLS; w += nt) {
    const int t = w / COLS, col = w % COLS, a = cut.start(t), m = cut.size(t);
    const int o0 = 3 * (a - t);
    // role: 0 interior column, 1 V, 2 W; c its component
    const int role = col < CUT_Q ? 0 : col < CUT_Q + 4 ? 1 : 2, c = role == 0 ? col % 3 : (col - CUT_Q) & 3;
    const bool zero = role == 0 ? col >= 3 * m : (c == 3 || (role == 1 ? t == 0 : t == P - 1));
    double y[3 * CUT_M];
#pragma unroll
    for (int k = 0; k < CUT_M; ++k) {
      double rhs[3] = {0, 0, 0};
      if (!zero && k < m) {
        if (role == 0 && k == col / 3) rhs[0] = c == 0, rhs[1] = c == 1, rhs[2] = c == 2;
        if ((role == 1 && k == 0) || (role == 2 && k == m - 1)) {
          const M3d M = role == 1 ? A(a) : C(a + m - 1);
#pragma unroll
          for (int d = 0; d < 3; ++d) rhs[d] = -(c == 0 ? M.a[3 * d] : c == 1 ? M.a[3 * d + 1] : M.a[3 * d + 2]);
        }
        double u[3], v[3] = {0, 0, 0};
        m3dVec(m3dGet(F(a + k, 0)), rhs, u);
        if (k > 0) m3dVec(m3dGet(F(a + k, 1)), y + 3 * (k > 0 ? k - 1 : 0), v);
        y[3 * k] = u[0] - v[0], y[3 * k + 1] = u[1] - v[1], y[3 * k + 2] = u[2] - v[2];
      } else {
        y[3 * k] = y[3 * k + 1] = y[3 * k + 2] = 0.0;
      }
    }
#pragma unroll
    for (int k = CUT_M - 2; k >= 0; --k) {
      if (k + 1 < m && !zero) {
        double v[3];
        m3dVec(m3dGet(F(a + k, 2)), y + 3 * (k + 1), v);
        y[3 * k] -= v[0], y[3 * k + 1] -= v[1], y[3 * k + 2] -= v[2];
      }
    }
    const int f = role == 0 ? col : CUT_Q + 4 * (role - 1) + c;  // float of the row
#pragma unroll
    for (int q = 0; q < 3 * CUT_M; ++q)
      if (q < 3 * m) rows[4 * ((size_t)(f >> 2) * I3 + o0 + q) + (f & 3)] = (float)y[q];
    if (role > 0 && c < 3) {  // first and last rows of V and W: [chunk][V first, V last, W first, W last][row][column]
      double* vw = sVW + 36 * t + 18 * (role - 1) + c;
#pragma unroll
      for (int d = 0; d < 3; ++d) vw[3 * d] = y[d];
#pragma unroll
      for (int k = 0; k < CUT_M; ++k)
        if (k == m - 1)
#pragma unroll
          for (int d = 0; d < 3; ++d) vw[9 + 3 * d] = y[3 * k + d];
    }
  }
  __syncthreads();
  // the separators' couplings into their chunks, and their Schur complement
  for (int w = tid; w < 3 * S * 2 * CUT_Q; w += nt) {
    const int o = w / (2 * CUT_Q), col = w % (2 * CUT_Q), s = o / 3, c = o % 3;
    const int right = col >= CUT_Q ? 1 : 0, q = col - CUT_Q * right, t = s + right;
    const int sep = cut.start(s) + cut.size(s);
    double v = 0.0;
    if (q < 3 * cut.size(t)) {
      const M3d M = right ? C(sep) : A(sep);
      const int o1 = 3 * ((right ? sep + 1 : sep - 1) - t);  // the chunk's node beside it
#pragma unroll
      for (int d = 0; d < 3; ++d)
        v += (c == 0 ? M.a[d] : c == 1 ? M.a[3 + d] : M.a[6 + d]) * (double)rows[4 * ((size_t)(q >> 2) * I3 + o1 + d) + (q & 3)];
    }
    // lane (col / 4) % 4 of round col / 16
    reinterpret_cast<float*>(out + sepAt)[4 * (((size_t)(col >> 4) * 3 * S + o) * 4 + ((col >> 2) & 3)) + (col & 3)] = (float)v;
  }
  for (int s = tid; s < S; s += nt) {
    const int sep = cut.start(s) + cut.size(s);
    const M3d As = A(sep), Cs = C(sep);
    const double *l = sVW + 36 * s, *r = sVW + 36 * (s + 1);
    m3dPut(sR + 27 * s, m3dMul(As, m3dGet(l + 9)));
    m3dPut(sR + 27 * s + 9, m3dAdd(m3dAdd(B(sep), m3dMul(As, m3dGet(l + 27))), m3dMul(Cs, m3dGet(r))));
    m3dPut(sR + 27 * s + 18, m3dMul(Cs, m3dGet(r + 18)));
  }
  __syncthreads();
}

// The couplings of thread (node n at (i, j), lane) in a line of family fam into c[4 RHS]; the node's
// majorisation is returned (summed over the lanes that hold the +-2 couplings along the line; every lane of
// the warp calls). block(along, across) and the scalars are zero where the neighbour is outside the layer
// or the row is fixed.
template <class Rows>
__device__ __forceinline__ float cutCouplingRow(const DLevel& L, const DLevelLayer& ly, int n, int i, int j, int fam, int lane,
                                                bool fixedNode, float* c) {
  auto inside = [&](int along, int across) {
    const int ii = i + (fam == 0 ? along : across), jj = j + (fam == 0 ? across : along);
    return !fixedNode && ii >= 0 && jj >= 0 && ii < ly.nx && jj < ly.ny;
  };
  const int quad = threadIdx.x & 28;
  if constexpr (CutOf<Rows>::RHS == 9) {
    auto block = [&](int along, int across) {
      if (!inside(along, across)) return symZero();
      return coarseBlock(L.op, L.N, n, ((fam == 0 ? across : along) + 2) * 5 + (fam == 0 ? along : across) + 2);
    };
#pragma unroll
    for (int s = 0; s < 5; ++s) storeSymAt(c, 6 * s, block(s - 2, lane < 2 ? lane - 2 : lane - 1));
    const Sym b5 = lane < 2 ? block(lane == 0 ? -2 : 2, 0) : symZero();
    const float f = lane < 2 ? symFrob(b5) : 0.f;
    const float maj = __shfl_sync(0xffffffffu, f, quad) + __shfl_sync(0xffffffffu, f, quad + 1);
    storeSymAt(c, 30, lane == 3 ? Sym{maj, fixedNode ? 1.f : 0.f, 0, 0, 0, 0} : b5);
    return maj;
  } else {
    const int side = lane < 2 ? -1 : 1;  // the stencil row across the line
    auto block = [&](int along) {
      if (!inside(along, side)) return symZero();
      return fineBlock(L.op, L.N, n, 1 + fineCoupling(fam == 0 ? along : side, fam == 0 ? side : along));
    };
    auto scalar = [&](int along, int across) {
      if (!inside(along, across)) return 0.f;
      return fineScalar(L.op, L.N, n, fineCoupling(fam == 0 ? along : across, fam == 0 ? across : along) - 8);
    };
    const bool odd = (lane & 1) != 0;
    storeSymAt(c, 0, block(odd ? 1 : -1));
    const float s2 = odd ? scalar(2 * side, 0) : 0.f;
    const float f = 1.7320508075688772f * fabsf(s2);
    const float maj = __shfl_sync(0xffffffffu, f, quad + 1) + __shfl_sync(0xffffffffu, f, quad + 3);
    storeSymAt(c, 6, odd ? Sym{scalar(0, 2 * side), s2, lane == 3 ? maj : 0.f, fixedNode ? 1.f : 0.f, 0, 0} : block(0));
    return maj;
  }
}
// A row's diagonal block and its block +1 along the line.
template <class Rows>
__device__ __forceinline__ Sym cutDiagonal(const DLevel& L, int n) {
  return CutOf<Rows>::RHS == 9 ? coarseBlock(L.op, L.N, n, 12) : fineBlock(L.op, L.N, n, 0);
}
template <class Rows>
__device__ __forceinline__ Sym cutNext(const DLevel& L, int n, int fam) {
  return CutOf<Rows>::RHS == 9 ? coarseBlock(L.op, L.N, n, fam == 0 ? 13 : 17) : fineBlock(L.op, L.N, n, fam == 0 ? 1 : 3);
}

template <class Rows>
__global__ void __launch_bounds__(CUT_FACTOR_THREADS, 3) k_line_compact(DLevel L, const int4* __restrict__ lines, const int* __restrict__ base,
                                                      float4* __restrict__ fac) {
  extern __shared__ double smd[];
  const int4 line = lines[blockIdx.x];  // (start node, stride, length, family | layer << 1)
  const int n0 = line.x, st = line.y, len = line.z, fam = line.w & 1;
  const DLevelLayer ly = L.layers[line.w >> 1];
  const Cut cut(len);
  const int S = cut.P - 1, tid = threadIdx.x, nt = blockDim.x;
  double* sF = smd;
  double* sVW = sF + max(27 * len, 9 * S * S);
  double* sR = sVW + 36 * cut.P;
  float* sB = reinterpret_cast<float*>(sR + 27 * S);
  float* sC = sB + 6 * len;
  float* sE = sC + 6 * len;
  float4* out = fac + base[blockIdx.x];
  const int local0 = n0 - ly.offset, i0 = local0 % ly.nx, j0 = local0 / ly.nx;

  // ---- couplings (thread 4 k + lane) and the line's rows: B with the majorisation, C the block +1 along
  constexpr int RHS = CutOf<Rows>::RHS;
  for (int w = tid; w < (4 * len + 31) / 32 * 32; w += nt) {
    const int k = min(w >> 2, len - 1), lane = w & 3;
    const int n = n0 + k * st;
    const bool fixedNode = L.fixed[n] != 0u;
    float c[4 * RHS];
    const float maj = cutCouplingRow<Rows>(L, ly, n, fam == 0 ? i0 + k : i0, fam == 0 ? j0 : j0 + k, fam, lane, fixedNode, c);
    if (w < 4 * len) {
#pragma unroll
      for (int p = 0; p < RHS; ++p) out[(size_t)p * 4 * len + w] = make_float4(c[4 * p], c[4 * p + 1], c[4 * p + 2], c[4 * p + 3]);
      if (lane == 2) storeSymAt(sB, 6 * k, fixedNode ? symId(1.f) : cutDiagonal<Rows>(L, n) + symId(maj));
      if (lane == 3) storeSymAt(sC, 6 * k, k + 1 < len && !fixedNode ? cutNext<Rows>(L, n, fam) : symZero());
    }
  }
  __syncthreads();

  // ---- the cut
  float* piv = reinterpret_cast<float*>(sF);  // not in use yet
  for (int k = tid; k < len; k += nt) {
    const float *B = sB + 6 * k, *C = sC + 6 * k;
    piv[k] = B[0], piv[len + k] = B[3], piv[2 * len + k] = B[5];
    piv[3 * len + k] = C[0] * C[0], piv[4 * len + k] = C[3] * C[3], piv[5 * len + k] = C[5] * C[5];
  }
  __syncthreads();
  linePivots(piv, len);
  for (int k = tid; k < len; k += nt) sE[k] = lineShift(piv, len, k);
  __syncthreads();
  auto row = [&](int k) {
    M3d B = m3dSym(sB + 6 * k);
    B.a[0] += sE[k], B.a[4] += sE[k], B.a[8] += sE[k];
    return B;
  };
  cutFactor(
      cut, len, [&](int k) { return m3dSym(sC + 6 * (k - 1)); }, row,
      [&](int k) { return m3dSym(sC + 6 * k); }, sF, sVW, sR, out + cutRowsAt<Rows>(len), cutSepAt<Rows>(len) - cutRowsAt<Rows>(len));

  // ---- the inverse of the separators' system: block LU by one thread (pivot inverses and G in place of
  // D and U), then column j of the inverse by thread j
  if (tid == 0) {
    M3d G = m3dZero();
    for (int s = 0; s < S; ++s) {
      const M3d Dinv = pivotInverseD(m3dAdd(m3dGet(sR + 27 * s + 9), m3dMul(m3dGet(sR + 27 * s), G), -1.0));
      G = m3dMul(Dinv, m3dGet(sR + 27 * s + 18));
      m3dPut(sR + 27 * s + 9, Dinv);
      m3dPut(sR + 27 * s + 18, G);
    }
  }
  __syncthreads();
  const int D3 = 3 * S;
  double* dense = sF;  // entry (row, column) at row D3 + column
  for (int j = tid; j < D3; j += nt) {
    double y[3] = {0, 0, 0};
    for (int s = 0; s < S; ++s) {
      double b[3], v[3];
      m3dVec(m3dGet(sR + 27 * s), y, v);
#pragma unroll
      for (int d = 0; d < 3; ++d) b[d] = (3 * s + d == j ? 1.0 : 0.0) - v[d];
      m3dVec(m3dGet(sR + 27 * s + 9), b, y);
#pragma unroll
      for (int d = 0; d < 3; ++d) dense[(3 * s + d) * D3 + j] = y[d];
    }
    for (int s = S - 2; s >= 0; --s) {
      double v[3];
      m3dVec(m3dGet(sR + 27 * s + 18), y, v);
#pragma unroll
      for (int d = 0; d < 3; ++d) y[d] = dense[(3 * s + d) * D3 + j] - v[d], dense[(3 * s + d) * D3 + j] = y[d];
    }
  }
  __syncthreads();
  float* dOut = reinterpret_cast<float*>(out + cutDenseAt<Rows>(len));
  for (int w = tid; w < D3 * 32 * CUT_ROUNDS; w += nt) {
    // float w & 3 of lane (w / 4) % 8 of unknown o in a round
    const int ol = w >> 5, o = ol % D3, j = 32 * (ol / D3) + (w & 31);
    dOut[w] = j < D3 ? (float)dense[o * D3 + j] : 0.f;
  }
}

// ------------------------------------------------------------------------------------------ sweep

__device__ __forceinline__ float dot4(float4 a, float4 b) { return fmaf(a.x, b.x, fmaf(a.y, b.y, fmaf(a.z, b.z, a.w * b.w))); }

// The coefficients of a thread: node k = tid / 4, lane = tid % 4 of the right-hand side and interior row;
// separator unknown tid / 4 of E and tid / 8 of D.
template <class Rows>
struct CutRegs {
  float c[4 * CutOf<Rows>::RHS];
  float4 row[CUT_ROW], e[CUT_SEP], d[CUT_ROUNDS];
  int k, lane, t, p;  // the node's chunk and place in it (p = its size: separator t)
  bool fixedNode, interior;
};

template <class Rows>
__device__ __forceinline__ void cutLoad(CutRegs<Rows>& R, const float4* __restrict__ f, int len, const Cut& cut) {
  const int tid = threadIdx.x, S = cut.P - 1, I3 = 3 * (len - S);
  R.lane = tid & 3;
  const bool on = tid < 4 * len;
  R.k = min(tid >> 2, len - 1);
  R.t = cut.of(R.k);
  R.p = R.k - cut.start(R.t);
  R.interior = R.p < cut.size(R.t);
  const int w = 4 * R.k + R.lane;
#pragma unroll
  for (int p = 0; p < CutOf<Rows>::RHS; ++p) {
    const float4 v = on ? __ldg(f + (size_t)p * 4 * len + w) : make_float4(0, 0, 0, 0);
    R.c[4 * p] = v.x, R.c[4 * p + 1] = v.y, R.c[4 * p + 2] = v.z, R.c[4 * p + 3] = v.w;
  }
  const int o = 3 * (R.k - R.t) + R.lane;
  const float4 z = make_float4(0, 0, 0, 0);
#pragma unroll
  for (int p = 0; p < CUT_ROW; ++p) R.row[p] = on && R.interior && R.lane < 3 ? __ldg(f + cutRowsAt<Rows>(len) + (size_t)p * I3 + o) : z;
#pragma unroll
  for (int p = 0; p < CUT_SEP; ++p) R.e[p] = tid < 12 * S ? __ldg(f + cutSepAt<Rows>(len) + (size_t)p * 12 * S + tid) : z;
#pragma unroll
  for (int p = 0; p < CUT_ROUNDS; ++p) R.d[p] = tid < 24 * S ? __ldg(f + cutDenseAt<Rows>(len) + (size_t)p * 24 * S + tid) : z;
}
// Once the loads have landed: lane 3 holds the fixed flag and the majorisation (of the node's own unknown,
// added back). Every lane of the warp calls.
template <class Rows>
__device__ __forceinline__ void cutReady(CutRegs<Rows>& R, int len) {
  const int tid = threadIdx.x;
  const bool on = tid < 4 * len;
  constexpr bool coarse = CutOf<Rows>::RHS == 9;
  const float flag = __shfl_sync(0xffffffffu, R.c[coarse ? 31 : 9], (tid & 28) + 3);
  R.fixedNode = !on || flag != 0.f;
  if constexpr (coarse) {
    if (R.lane == 3) {
      const float m = -R.c[30];
      R.c[30] = m, R.c[31] = 0.f, R.c[32] = 0.f, R.c[33] = m, R.c[34] = 0.f, R.c[35] = m;
    }
  }
}

// A line's scratch in shared memory: interior right-hand sides (P chunks of CUT_Q, zero padded), the
// separators' right-hand sides, reduced (zero padded to the rounds), and unknowns (one float4 each, with
// zeros before and after).
struct CutScratch {
  float* rI;
  float* rS;
  float* rr;
  float4* xS;
};
__host__ __device__ constexpr int cutScratchF4(int len) {
  return CUT_Q / 4 * Cut::parts(len) + (3 * cutSeparators(len) + 3) / 4 + 8 * CUT_ROUNDS + Cut::parts(len) + 1;
}
__device__ __forceinline__ CutScratch cutScratch(float4* sm, int len) {
  const int P = Cut::parts(len);
  CutScratch s;
  s.rI = reinterpret_cast<float*>(sm);
  s.rr = s.rI + CUT_Q * P;
  s.xS = reinterpret_cast<float4*>(s.rr) + 8 * CUT_ROUNDS;
  s.rS = reinterpret_cast<float*>(s.xS + P + 1);
  return s;
}
// Zeroes the scratch's padding (every thread; a barrier follows before its use).
__device__ __forceinline__ void cutClear(float4* sm, int len) {
  for (int q = threadIdx.x; q < cutScratchF4(len); q += blockDim.x) sm[q] = make_float4(0, 0, 0, 0);
}

// The line's solve from the right-hand side of the thread's component (lane < 3), already in the scratch:
// every thread returns its component of its node's unknown. Three barriers.
template <class Rows>
__device__ __forceinline__ float cutSolve(const CutRegs<Rows>& R, const CutScratch& s, int P) {
  const int tid = threadIdx.x, S = P - 1;
  __syncthreads();
  {
    const int o = tid >> 2, l = tid & 3, sep = o / 3;
    float v = 0.f;
    if (tid < 12 * S) {
#pragma unroll
      for (int p = 0; p < CUT_SEP; ++p) v += dot4(R.e[p], *reinterpret_cast<const float4*>(s.rI + sep * CUT_Q + 16 * p + 4 * l));
    }
    v += __shfl_xor_sync(0xffffffffu, v, 1);
    v += __shfl_xor_sync(0xffffffffu, v, 2);
    if (tid < 12 * S && l == 0) s.rr[o] = s.rS[o] - v;
  }
  // the chunk's own part does not wait for the separators
  float x = 0.f;
#pragma unroll
  for (int p = 0; p < CUT_Q / 4; ++p) x += dot4(R.row[p], *reinterpret_cast<const float4*>(s.rI + R.t * CUT_Q + 4 * p));
  __syncthreads();
  {
    const int o = tid >> 3, l = tid & 7;
    float v = 0.f;
    if (tid < 24 * S) {
#pragma unroll
      for (int p = 0; p < CUT_ROUNDS; ++p) v += dot4(R.d[p], *reinterpret_cast<const float4*>(s.rr + 32 * p + 4 * l));
    }
    v += __shfl_xor_sync(0xffffffffu, v, 1);
    v += __shfl_xor_sync(0xffffffffu, v, 2);
    v += __shfl_xor_sync(0xffffffffu, v, 4);
    if (tid < 24 * S && l == 0) reinterpret_cast<float*>(s.xS + 1 + o / 3)[o % 3] = v;
  }
  __syncthreads();
  const float4 xl = s.xS[R.t], xr = s.xS[R.t + 1];
  if (!R.interior) return R.lane == 0 ? xr.x : R.lane == 1 ? xr.y : xr.z;
  const float4 V = R.row[CUT_Q / 4], W = R.row[CUT_Q / 4 + 1];
  x += fmaf(V.x, xl.x, fmaf(V.y, xl.y, V.z * xl.z));
  return x + fmaf(W.x, xr.x, fmaf(W.y, xr.y, W.z * xr.z));
}

// The couplings' part of the thread's node's lagged right-hand side, summed over the four lanes; x the node's
// own unknown in shared memory, at(a) the one a nodes across the line from it (a = -2..2), `along` the step
// along the line.
template <class Rows, class At>
__device__ __forceinline__ float3 cutCouplings(const CutRegs<Rows>& R, const float4* __restrict__ x, At at, int along) {
  auto sym = [&](int f) { return Sym{R.c[f], R.c[f + 1], R.c[f + 2], R.c[f + 3], R.c[f + 4], R.c[f + 5]}; };
  float3 acc = make_float3(0, 0, 0);
  if constexpr (CutOf<Rows>::RHS == 9) {
    const float4* row = at(R.lane < 2 ? R.lane - 2 : R.lane - 1);
#pragma unroll
    for (int s = 0; s < 5; ++s) acc += sym(6 * s) * f3(row[(s - 2) * along]);
    acc += sym(30) * f3(x[(R.lane == 0 ? -2 : R.lane == 1 ? 2 : 0) * along]);
  } else {
    const float4* row = at(R.lane < 2 ? -1 : 1);
    if (R.lane & 1) {
      acc = sym(0) * f3(row[along]);
      acc += R.c[6] * f3(*at(R.lane < 2 ? -2 : 2));
      acc += R.c[7] * f3(x[(R.lane < 2 ? -2 : 2) * along]);
      acc -= R.c[8] * f3(x[0]);
    } else {
      acc = sym(0) * f3(row[-along]);
      acc += sym(6) * f3(row[0]);
    }
  }
#pragma unroll
  for (int m = 1; m <= 2; m <<= 1) {
    acc.x += __shfl_xor_sync(0xffffffffu, acc.x, m);
    acc.y += __shfl_xor_sync(0xffffffffu, acc.y, m);
    acc.z += __shfl_xor_sync(0xffffffffu, acc.z, m);
  }
  return acc;
}

// The five columns of unknowns in shared memory: column a (0..4, the line's own 2) from a multiple of eight
// float4 plus 2, 4, 6 for a = 1, 3, 4, so that the eight threads of a 128-bit access phase (two nodes, four
// lanes, a column each) meet eight different bank groups. Where len + 4 is a multiple of eight, the last two float4 of
// column 1 are the first two of column 2: both are beyond the line's ends, zeros.
__host__ __device__ constexpr int cutColumnStride(int len) { return (len + 4 + 7) / 8 * 8; }
__host__ __device__ constexpr int cutColumn(int a, int len) {
  return a * cutColumnStride(len) + (a == 0 || a == 2 ? 0 : a == 1 ? 2 : a == 3 ? 4 : 6);
}
__host__ __device__ constexpr int cutColumnsF4(int len) { return 5 * cutColumnStride(len) + 6; }

// Shared memory (bytes) of k_sweep: five columns of unknowns (the line and two either side, two nodes more
// at each end) and the solve's scratch.
__host__ __device__ constexpr size_t cutSweepSmem(int len) { return 16 * (size_t)(cutColumnsF4(len) + cutScratchF4(len)); }

// One colour of a sweep, a CTA a line, four threads a node (NT at least that, a multiple of 32).
template <class Rows, int FAM, int NT, int MINB>
__global__ void __launch_bounds__(NT, MINB) k_sweep(DLevel L, LineGeom g, const int4* __restrict__ lines, const int* __restrict__ base,
                                                    const float4* __restrict__ fac) {
  extern __shared__ float4 sm4[];
  int n0, st, len, fb, across0;
  DLevelLayer ly;
  Cut cut;
  if (g.table) {
    const int4 line = lines[g.first + blockIdx.x];
    n0 = line.x, st = line.y, len = line.z;
    ly = L.layers[line.w >> 1];
    fb = base[g.first + blockIdx.x];
    cut = Cut(len);
    across0 = FAM == 0 ? (n0 - ly.offset) / ly.nx : (n0 - ly.offset) % ly.nx;
  } else {
    n0 = g.start0 + blockIdx.x * g.startStep, st = g.stride, len = g.len, ly = g.ly;
    fb = g.base0 + blockIdx.x * g.baseStep;
    cut = Cut(g.P, g.chunkBase, g.chunkExtra);
    across0 = g.across0 + 3 * blockIdx.x;
  }
  const int tid = threadIdx.x, nt = blockDim.x, TX = len + 4;
  const int nAcross = FAM == 0 ? ly.ny : ly.nx, acrossStep = FAM == 0 ? ly.nx : 1;
  CutRegs<Rows> R;
  cutLoad<Rows>(R, fac + fb, len, cut);
  cutReady<Rows>(R, len);
  float4* scratch = sm4 + cutColumnsF4(len);
  cutClear(scratch, len);
  const CutScratch s = cutScratch(scratch, len);
  pdlWait();
  pdlLaunchNext();
  const float b = R.lane < 3 ? __ldcg(reinterpret_cast<const float*>(L.B + n0 + R.k * st) + R.lane) : 0.f;
  for (int q = tid; q < 5 * TX; q += nt) {
    const int a = q / TX, kk = q - a * TX, k = kk - 2, c = across0 + a - 2;
    const bool ok = k >= 0 && k < len && c >= 0 && c < nAcross;
    cpAsync16(sm4 + cutColumn(a, len) + kk, L.X + (ok ? n0 + k * st + (a - 2) * acrossStep : n0), ok);
  }
  cpAsyncWaitAll();
  __syncthreads();
  const float3 acc = cutCouplings(R, sm4 + cutColumn(2, len) + R.k + 2, [&](int q) { return sm4 + cutColumn(q + 2, len) + R.k + 2; }, 1);
  const float r = b - (R.lane == 0 ? acc.x : R.lane == 1 ? acc.y : acc.z);
  if (R.lane < 3 && tid < 4 * len) {
    if (R.interior)
      s.rI[R.t * CUT_Q + 3 * R.p + R.lane] = r;
    else
      s.rS[3 * R.t + R.lane] = r;
  }
  const float x = cutSolve(R, s, cut.P);
  if (R.lane < 3 && !R.fixedNode) reinterpret_cast<float*>(L.X + n0 + R.k * st)[R.lane] = x;
}

}  // namespace btd
