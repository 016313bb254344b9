// Flat vector kernels and float64 bookkeeping of the device-resident GMRES.
//
// Restates jax.scipy.sparse.linalg.gmres (jax/jaxlib >= 0.10.0; called at
// steppers.py:466 and :476): left preconditioning (Krylov space of M A), one
// classical Gram-Schmidt projection per Arnoldi step over the basis, breakdown
// when ||v|| <= eps ||M A v_k||, and either the 'batched' cycle (normal
// equations + Cholesky for the Hessenberg least-squares problem) or the
// 'incremental' cycle (Givens rotations, early exit on the rotated residual).
//
// A classical basis vector V_i is stored unnormalised next to its inverse norm s_i, so
// normalisation never costs a pass over memory: the matvec scales its input
// on load, projections use h_i = s_i <V_i, w>, updates use h_i s_i V_i.
// The classical projection reads the whole basis twice per Arnoldi step (once
// for the inner products, once for the update), which was two thirds of a
// solve.  Here up to GM_S steps share those two reads: the operator is
// applied to its own output s times, Z_1 = (M A - I) V_j, Z_i = (M A - I)
// Z_{i-1}, and the s new vectors are orthogonalised together (s-step Arnoldi
// with a shifted basis; Hoemmen, Communication-avoiding Krylov subspace
// methods, Berkeley 2010).  The shift takes out the identity of M A = I + E:
// E, the horizontal acoustic coupling, is small on smooth vectors, and
// without it Z_i would be V_j over again there.  block_dots forms all products
// of the basis with Z and of Z with itself in one pass over memory,
// block_update the new vectors in a second one, and the Hessenberg columns
// follow from the small matrices (block_finish).  A cycle whose blocks keep
// all their columns spans the same Krylov space and minimises over it as the
// one-step form does; a cycle in which a column is lost to rounding is
// narrow: it is dropped and done over one column at a time, and so are the
// solve's later ones (gmres_run in sisl_api.cu).  256x256x80 float32, restart
// 30: vector passes per cycle 1020 -> 220.
//
// One column at a time is the classical form: the dots and update kernels with
// their one-step bookkeeping, for what follows a narrow cycle.
//
// The block form's stored vectors V carry a small triangular factor per block (GState::B)
// instead of being normalised in memory: the Gram matrix of the vectors as
// stored is summed while they are written and its Cholesky factor is carried
// in the small algebra, so rounding of the stored vectors never enters the
// Arnoldi relation.  Every reduction accumulates in float64; the last block
// of a reduction kernel (ticket counter) finishes the sum and runs the small
// algebra.
#include "sisl_group.cuh"

#include <math.h>

#include <type_traits>

namespace sisl {
namespace {

constexpr int GT = 256;  // threads per block of the flat kernels

template <typename T> struct V16;
template <> struct V16<float> { using type = float4; static constexpr int n = 4; };
template <> struct V16<double> { using type = double2; static constexpr int n = 2; };

template <typename T>
__device__ __forceinline__ void load16(const T* p, T* r) {
  using VT = typename V16<T>::type;
  VT v = __ldg(reinterpret_cast<const VT*>(p));
  const T* q = reinterpret_cast<const T*>(&v);
#pragma unroll
  for (int e = 0; e < V16<T>::n; ++e) r[e] = q[e];
}
// the same through the coherent path: memory this kernel also writes
template <typename T>
__device__ __forceinline__ void load16_rw(const T* p, T* r) {
  using VT = typename V16<T>::type;
  VT v = *reinterpret_cast<const VT*>(p);
  const T* q = reinterpret_cast<const T*>(&v);
#pragma unroll
  for (int e = 0; e < V16<T>::n; ++e) r[e] = q[e];
}
template <typename T>
__device__ __forceinline__ void store16(T* p, const T* r) {
  using VT = typename V16<T>::type;
  VT v;
  T* q = reinterpret_cast<T*>(&v);
#pragma unroll
  for (int e = 0; e < V16<T>::n; ++e) q[e] = r[e];
  *reinterpret_cast<VT*>(p) = v;
}

// Per-thread chunk: CH 16-byte loads (E = CH * 16/sizeof(T) elements).
constexpr int CH = 4;

__device__ __forceinline__ double warp_sum(double s) {
  for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
  return s;
}

// Last-block ticket.  Returns true in exactly one block, after every other
// block's partial results are visible.
__device__ __forceinline__ bool last_block(unsigned int* counter, unsigned int nblk) {
  __shared__ bool am_last;
  __threadfence();
  __syncthreads();
  if (threadIdx.x == 0) {
    unsigned int t = atomicAdd(counter, 1u);
    am_last = (t == nblk - 1);
  }
  __syncthreads();
  if (am_last) __threadfence();
  return am_last;
}

enum DotMode { DM_PROJ = 0, DM_BNORM = 1, DM_MBNORM = 2, DM_RNORM = 3 };

// result_i = <V_i, w> for i < m and <w, w>; finished according to `mode`.
// Per tile, every warp sums its products (float64) with shuffles and lane 0
// adds them to the warp's shared slot acc[q * warps + warp]: (m + 1) x 8
// doubles per block, so shared memory never limits the resident blocks
// (registers do); the block reduces the warps' slots once at the end.
// Block `bid` of `nblk` blocks of one reduction (a member's share of a
// grouped launch, or the whole grid of a standalone one).
template <typename T>
__device__ __forceinline__ void dots_body(const T* __restrict__ Vb, size_t stride, int m, const T* __restrict__ w,
                                          size_t n, double* partial, GState* gs, int mode, int bid, int nblk) {
  extern __shared__ double acc[];  // (m + 1) * warps: per-warp sums
  const int tid = threadIdx.x, nt = blockDim.x;
  const int lane = tid & 31, wp = tid >> 5, nw = nt >> 5;
  for (int q = tid; q < (m + 1) * nw; q += nt) acc[q] = 0.0;
  __syncthreads();
  constexpr int VN = V16<T>::n;
  constexpr int E = CH * VN;
  const size_t tile = (size_t)nt * E;
  for (size_t base = (size_t)bid * tile; base < n; base += (size_t)nblk * tile) {
    T wr[E];
#pragma unroll
    for (int c = 0; c < CH; ++c) {
      const size_t off = base + ((size_t)c * nt + tid) * VN;
      if (off < n) load16(w + off, wr + c * VN);
      else
#pragma unroll
        for (int e = 0; e < VN; ++e) wr[c * VN + e] = T(0);
    }
    double sq = 0.0;
#pragma unroll
    for (int e = 0; e < E; ++e) sq += (double)wr[e] * (double)wr[e];
    sq = warp_sum(sq);
    if (lane == 0) acc[m * nw + wp] += sq;
    // two basis vectors per iteration: both chunks are in flight together
    int i = 0;
    for (; i + 1 < m; i += 2) {
      const T* __restrict__ Va = Vb + (size_t)i * stride;
      const T* __restrict__ Vc = Va + stride;
      T va[E], vc[E];
#pragma unroll
      for (int c = 0; c < CH; ++c) {
        const size_t off = base + ((size_t)c * nt + tid) * VN;
        if (off < n) {
          load16(Va + off, va + c * VN);
          load16(Vc + off, vc + c * VN);
        } else {
#pragma unroll
          for (int e = 0; e < VN; ++e) { va[c * VN + e] = T(0); vc[c * VN + e] = T(0); }
        }
      }
      double pa = 0.0, pc = 0.0;
#pragma unroll
      for (int e = 0; e < E; ++e) {
        pa += (double)va[e] * (double)wr[e];
        pc += (double)vc[e] * (double)wr[e];
      }
      pa = warp_sum(pa);
      pc = warp_sum(pc);
      if (lane == 0) {
        acc[i * nw + wp] += pa;
        acc[(i + 1) * nw + wp] += pc;
      }
    }
    if (i < m) {
      const T* __restrict__ Vi = Vb + (size_t)i * stride;
      T vr[E];
#pragma unroll
      for (int c = 0; c < CH; ++c) {
        const size_t off = base + ((size_t)c * nt + tid) * VN;
        if (off < n) load16(Vi + off, vr + c * VN);
        else
#pragma unroll
          for (int e = 0; e < VN; ++e) vr[c * VN + e] = T(0);
      }
      double p = 0.0;
#pragma unroll
      for (int e = 0; e < E; ++e) p += (double)vr[e] * (double)wr[e];
      p = warp_sum(p);
      if (lane == 0) acc[i * nw + wp] += p;
    }
  }
  __syncthreads();
  // block reduction: thread q sums the warps' slots of result q
  for (int q = tid; q <= m; q += nt) {
    double s_ = 0.0;
    for (int k = 0; k < nw; ++k) s_ += acc[q * nw + k];
    partial[(size_t)bid * (GM_MAXR + 2) + q] = s_;
  }
  if (!last_block(&gs->counter, (unsigned)nblk)) return;
  // finish: sum the partials of all blocks, one warp per result (lanes
  // stride over the blocks, so the loads are independent)
  for (int q = wp; q <= m; q += nw) {
    double s_ = 0.0;
    for (int b = lane; b < nblk; b += 32) s_ += partial[(size_t)b * (GM_MAXR + 2) + q];
    s_ = warp_sum(s_);
    if (lane == 0) acc[q] = s_;
  }
  __syncthreads();
  if (tid == 0) {
    gs->counter = 0;
    const double nrm = sqrt(acc[m]);
    if (mode == DM_PROJ) {
      for (int i = 0; i < m; ++i) gs->h[i] = gs->s[i] * acc[i];
      gs->hn0 = nrm;
    } else if (mode == DM_BNORM) {
      gs->bnorm = nrm;
    } else if (mode == DM_MBNORM) {
      gs->mbnorm = nrm;
    } else {  // DM_RNORM: _safe_normalize of the preconditioned residual
      const bool use = nrm > gs->eps;
      gs->s[0] = use ? 1.0 / nrm : 0.0;
      gs->rnorm = use ? nrm : 0.0;
      gs->B[0][0] = gs->s[0];  // block form: V_0 is a block of its own
      gs->bstart[0] = 0;
      gs->clast[0] = gs->rnorm;
      gs->cstart = 0;
      gs->clen = 1;
    }
  }
  // block form: a cycle's vectors enter the operator unscaled until their block is finished
  if (mode == DM_RNORM && gs->columns > 1)
    for (int q = 1 + tid; q < GM_MAXR + 2; q += nt) gs->s[q] = 1.0;
}

template <typename T>
__global__ void dots_kernel(const T* __restrict__ Vb, size_t stride, int m, const T* __restrict__ w, size_t n,
                            double* partial, GState* gs, int mode, int gated) {
  grid_chain();
  if (gated && gs->active == 0) return;
  dots_body<T>(Vb, stride, m, w, n, partial, gs, mode, blockIdx.x, gridDim.x);
}

enum UpdMode { UM_NONE = 0, UM_ARNOLDI = 1 };

// ---------------------------------------------------------------------------
// block Arnoldi: inner products
// ---------------------------------------------------------------------------
// d += a b on the float64 tensor path (the fifth-generation tensor cores have
// no float64 kind).  Lane l holds A[row l / 4][k l % 4], B[k l % 4][col l / 4]
// and D[row l / 4][cols 2 (l % 4), + 1]; every product and sum is a float64
// fused multiply-add.
__device__ __forceinline__ void dmma(double (&d)[2], double a, double b) {
  asm("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0, %1}, {%2}, {%3}, {%0, %1};"
      : "+d"(d[0]), "+d"(d[1])
      : "d"(a), "d"(b));
}

// One warp per summed matrix row and thread 0 for the s x s factor: the
// coefficients of the block's update from the summed products w[r][i] =
// <row r, Z_i>, rows V_0 .. V_j0 then Z_1 .. Z_s.  r1s: scratch, rows x 8.
//
// Projections in the orthonormal basis: r1 = B^T w.  The part of Z outside
// the basis has the Gram matrix G - r1^T r1 = r2^T r2; a column whose pivot
// there is lost in rounding (Z_i depends on the earlier ones to the
// precision of the stored vectors) ends the block before it, never before its
// first column, which needs no pivot: its norm is taken from the stored
// result.
__device__ __forceinline__ void block_coefs(GState* gs, const double* w, double* r1s, int j0, int s) {
  __shared__ double g[GM_S][GM_S], r2[GM_S][GM_S], u[GM_S][GM_S];
  __shared__ int keep_s;
  const int m = j0 + 1, tid = threadIdx.x, lane = tid & 31, wp = tid >> 5;
  if (tid < GM_S * GM_S) (&r2[0][0])[tid] = (&u[0][0])[tid] = 0.0;
  for (int q = tid; q < m * 8; q += GT) {
    const int l = q >> 3, i = q & 7;
    double v = 0.0;
    if (i < s) {
      const int st = gs->bstart[l];
      for (int p = st; p <= l; ++p) v += gs->B[l][p - st] * w[p * 8 + i];
      gs->r1[l][i] = v;
    }
    r1s[q] = v;
  }
  __syncthreads();
  int pair = 0;
  for (int i = 0; i < s; ++i)
    for (int k = i; k < s; ++k, ++pair) {
      if ((pair & 7) != wp) continue;
      double v = 0.0;
      for (int l = lane; l < m; l += 32) v += r1s[l * 8 + i] * r1s[l * 8 + k];
      v = warp_sum(v);
      if (lane == 0) g[i][k] = w[(m + i) * 8 + k] - v;
    }
  __syncthreads();
  if (tid == 0) {
    int keep = s;
    // what is left of a healthy column, squared and against its length, is 5e-4 or more at six columns: acoustic
    // radius 0.02 to 59, float32 and float64, cosine modes, noise and the states of the workloads
    const double lost = fmax(32.0 * gs->eps, 1e-6);
    for (int i = 0; i < keep; ++i) {
      double piv = g[i][i];
      for (int q = 0; q < i; ++q) {
        double v = g[q][i];
        for (int p = 0; p < q; ++p) v -= r2[p][q] * r2[p][i];
        v /= r2[q][q];
        r2[q][i] = v;
        piv -= v * v;
      }
      const double own = w[(m + i) * 8 + i];  // ||Z_i||^2
      if (piv > lost * own) {
        r2[i][i] = sqrt(piv);
      } else if (i == 0) {  // scaled by its own length; alone in its block
        r2[0][0] = own > 0.0 ? sqrt(own) : 1.0;
        keep = 1;
      } else {
        for (int q = 0; q < i; ++q) r2[q][i] = 0.0;
        keep = i;
      }
    }
    gs->bs = keep;
    keep_s = keep;
  }
  __syncthreads();
  if (tid < keep_s) {  // u = r2^-1, a column per thread
    const int i = tid;
    u[i][i] = 1.0 / r2[i][i];
    for (int q = i - 1; q >= 0; --q) {
      double v = 0.0;
      for (int p = q + 1; p <= i; ++p) v -= r2[q][p] * u[p][i];
      u[q][i] = v / r2[q][q];
    }
  }
  __syncthreads();
  if (tid < GM_S * GM_S) {
    const int i = tid / GM_S, k = tid - i * GM_S;
    gs->r2[i][k] = r2[i][k];
    gs->u[i][k] = u[i][k];
  }
  // r1 u, then back to the stored vectors: cv = B (r1 u)
  double t[GM_S];
  for (int l = tid; l < m; l += GT) {
    for (int i = 0; i < s; ++i) {
      t[i] = 0.0;
      for (int k = 0; k <= i; ++k) t[i] += r1s[l * 8 + k] * u[k][i];
    }
    for (int i = 0; i < s; ++i) r1s[l * 8 + i] = t[i];
  }
  __syncthreads();
  for (int q = tid; q < m * 8; q += GT) {
    const int k = q >> 3, i = q & 7;
    if (i >= s) continue;
    const int st = gs->bstart[k];
    double v = 0.0;
    for (int l = k; l < m && gs->bstart[l] == st; ++l) v += gs->B[l][k - st] * r1s[l * 8 + i];
    gs->cv[k][i] = v;
  }
}

// Products of the m + s stored vectors V_0 .. V_j0, Z_1 .. Z_s (contiguous
// slots, m = j0 + 1) with Z_1 .. Z_s: an (m + s) x s x n contraction, float64
// tensor tiles of 8 rows x 8 columns x 4 elements.  The operands of both
// sides have the same lane layout (row l / 4, element l % 4), so a lane loads
// 16-byte pieces of its row straight from memory and the order of the
// elements within a piece does not matter; NT row tiles stay in registers
// for the whole pass and need no shuffles.  Rows and columns past the end
// repeat the last one and are ignored.
//
// Bound by reading the m + s vectors: the tensor work of a pass (8 of 8
// columns for 6 vectors) stays below the loads' time.  256x256x80 float32,
// the inner products of a cycle of 30: 9.1 ms in one-step form, 2.14 ms here
// (4.7 TB/s of the rows read once), 2.71 with four row tiles loaded and then
// multiplied.  One tile ahead is enough and keeps two blocks' registers: four
// ahead spill (31 rows 893 us against 577), two ahead 807; three blocks an SM
// help only the shortest (7 rows 198 against 263, 31 rows 623).
//
// The partial tiles are summed in two levels (groups of GM_GROUP blocks, then
// the groups), in a fixed order: the same bits on every run.
template <typename T, int NT>
__device__ __forceinline__ void block_dots_body(const T* __restrict__ Vb, size_t stride, int j0, int s, size_t n,
                                                double* partial, GState* gs, int bid, int nblk) {
  constexpr int VN = V16<T>::n;
  constexpr int KW = 8 * VN;  // elements of every row a warp takes per pass: two 16-byte pieces per lane
  constexpr int GRP = NT < 4 ? NT : 4;  // tiles summed over the warps at a time
  __shared__ double red[8][GRP * 64];
  __shared__ double w[NT * 64], r1s[NT * 64];
  const int tid = threadIdx.x, lane = tid & 31, wp = tid >> 5;
  const int m = j0 + 1, rows = m + s;
  const int r = lane >> 2;
  const size_t kq = (size_t)(lane & 3) * VN;
  const T* zp = Vb + (size_t)(m + min(r, s - 1)) * stride + kq;
  const T* v0 = Vb + kq;
  double acc[NT][2];
#pragma unroll
  for (int t = 0; t < NT; ++t) acc[t][0] = acc[t][1] = 0.0;
  // a row tile's loads (at a pass's end the next pass's first ones) are issued while the tile before is multiplied
  const size_t step = (size_t)nblk * 8 * KW;
  T z[2 * VN], zn[2 * VN], a[2 * VN], an[2 * VN];
  auto load = [&](const T* v, T* q) {
    load16(v, q);
    load16(v + 4 * VN, q + VN);
  };
  auto row = [&](int t) { return v0 + (size_t)min(8 * t + r, rows - 1) * stride; };
  size_t k = ((size_t)bid * 8 + wp) * KW;
  if (k < n) {
    load(zp + k, z);
    load(row(0) + k, a);
  }
  for (; k < n; k += step) {
    const size_t kn = k + step < n ? k + step : k;  // the last pass repeats its own loads
#pragma unroll
    for (int t = 0; t < NT; ++t) {
      if (t + 1 < NT) {
        load(row(t + 1) + k, an);
      } else {
        load(zp + kn, zn);
        load(row(0) + kn, an);
      }
#pragma unroll
      for (int e = 0; e < 2 * VN; ++e) dmma(acc[t], (double)a[e], (double)z[e]);
#pragma unroll
      for (int e = 0; e < 2 * VN; ++e) a[e] = an[e];
    }
#pragma unroll
    for (int e = 0; e < 2 * VN; ++e) z[e] = zn[e];
  }
  double* mine = partial + (size_t)bid * (NT * 64);
#pragma unroll
  for (int t0 = 0; t0 < NT; t0 += GRP) {
#pragma unroll
    for (int t = 0; t < GRP; ++t)
      if (t0 + t < NT) {
        red[wp][t * 64 + r * 8 + 2 * (lane & 3)] = acc[t0 + t][0];
        red[wp][t * 64 + r * 8 + 2 * (lane & 3) + 1] = acc[t0 + t][1];
      }
    __syncthreads();
    const int cnt = min(GRP, NT - t0) * 64;
    for (int q = tid; q < cnt; q += GT) {
      double v = 0.0;
#pragma unroll
      for (int k = 0; k < 8; ++k) v += red[k][q];
      mine[t0 * 64 + q] = v;
    }
    __syncthreads();
  }
  const int grp = bid / GM_GROUP, ng = (nblk + GM_GROUP - 1) / GM_GROUP;
  const int gsz = min(GM_GROUP, nblk - grp * GM_GROUP);
  if (!last_block(&gs->group_counter[grp], (unsigned)gsz)) return;
  double* gpart = partial + (size_t)nblk * (NT * 64);
  const double* first = partial + (size_t)grp * GM_GROUP * (NT * 64);
  for (int q = tid; q < NT * 64; q += GT) {
    double v = 0.0;
    for (int b = 0; b < gsz; ++b) v += __ldcg(first + (size_t)b * (NT * 64) + q);
    gpart[(size_t)grp * (NT * 64) + q] = v;
  }
  if (tid == 0) gs->group_counter[grp] = 0;
  __syncthreads();  // every thread has read last_block's verdict before the next one is written
  if (!last_block(&gs->counter, (unsigned)ng)) return;
  for (int q = tid; q < NT * 64; q += GT) {
    double v = 0.0;
    for (int b = 0; b < ng; ++b) v += __ldcg(gpart + (size_t)b * (NT * 64) + q);
    w[q] = v;
  }
  if (tid == 0) gs->counter = 0;
  __syncthreads();
  block_coefs(gs, w, r1s, j0, s);
}

template <typename T, int NT>
__global__ void __launch_bounds__(GT, 2) block_dots_kernel(const T* __restrict__ Vb, size_t stride, int j0, int s,
                                                           size_t n, double* partial, GState* gs) {
  grid_chain();
  if (gs->active == 0) return;
  block_dots_body<T, NT>(Vb, stride, j0, s, n, partial, gs, blockIdx.x, gridDim.x);
}

// ---------------------------------------------------------------------------
// block Arnoldi: update
// ---------------------------------------------------------------------------
// The Hessenberg columns of the block's steps from gram[i][k] = <V_{m+i},
// V_{m+k}> of the new vectors as stored, then the cycle's bookkeeping.
//
// With rc^T rc = gram the new orthonormal vectors are Q_{m+i} = sum_q V_{m+q}
// (rc^-1)[q][i], and in the basis Q the operator's inputs and outputs are
// known columns C: C_0 the scaled V_j0, C_{i+1} = [r1_i; (rc r2)_i] the
// vector Z_{i+1} = (M A - I) (input i).  H C_t = C_{t+1} + C_t gives the new
// columns of H one after the other (a row per thread: a row of column t needs only the
// same row of earlier columns).  For one column this is the classical
// Arnoldi step.
__device__ __forceinline__ void block_finish(GState* gs, const double (&gram)[GM_S][GM_S], int j0, int s) {
  constexpr int P = GM_MAXR + 2;
  __shared__ double C[GM_S + 1][P], hn[GM_S][P], gv[GM_MAXR][2];
  __shared__ double rc[GM_S][GM_S], ri[GM_S][GM_S], t2[GM_S][GM_S], len2[GM_S];
  __shared__ int keep_s, done_s;
  const int m = j0 + 1, R = gs->restart, tid = threadIdx.x, lane = tid & 31, wp = tid >> 5;
  const bool rotate = gs->method != 0;
  if (tid < GM_S * GM_S) (&rc[0][0])[tid] = (&ri[0][0])[tid] = (&t2[0][0])[tid] = 0.0;
  __syncthreads();
  if (tid == 0) {
    int keep = gs->bs;
    for (int i = 0; i < keep; ++i) {
      double piv = gram[i][i];
      for (int q = 0; q < i; ++q) {
        double v = gram[q][i];
        for (int p = 0; p < q; ++p) v -= rc[p][q] * rc[p][i];
        v /= rc[q][q];
        rc[q][i] = v;
        piv -= v * v;
      }
      if (i > 0 && !(piv > 1e-4 * gram[i][i])) {  // not independent of the earlier columns as stored
        for (int q = 0; q < i; ++q) rc[q][i] = 0.0;
        keep = i;
        break;
      }
      rc[i][i] = piv > 0.0 ? sqrt(piv) : 0.0;
      if (!(rc[i][i] > 0.0)) keep = i + 1;  // i = 0: nothing left of Z_1
    }
    keep_s = keep;
  }
  __syncthreads();
  if (tid < keep_s) {  // ri = rc^-1 and t2 = rc r2, a column per thread
    const int i = tid;
    for (int q = 0; q <= i; ++q) {
      double v = 0.0;
      for (int p = q; p <= i; ++p) v += rc[q][p] * gs->r2[p][i];
      t2[q][i] = v;
    }
    ri[i][i] = rc[i][i] > 0.0 ? 1.0 / rc[i][i] : 0.0;
    for (int q = i - 1; q >= 0; --q) {
      double v = 0.0;
      for (int p = q + 1; p <= i; ++p) v -= rc[q][p] * ri[p][i];
      ri[q][i] = v * (rc[q][q] > 0.0 ? 1.0 / rc[q][q] : 0.0);
    }
  }
  for (int q = tid; q < 2 * j0; q += GT) (&gv[0][0])[q] = (&gs->givens[0][0])[q];
  __syncthreads();
  const int keep = keep_s;
  const double start = gs->s[j0];
  const int cst = gs->cstart, cln = gs->clen;
  for (int p = tid; p < m + keep; p += GT) {
    C[0][p] = (p >= cst && p < cst + cln) ? start * gs->clast[p - cst] : 0.0;
    for (int i = 0; i < keep; ++i) C[i + 1][p] = p < m ? gs->r1[p][i] : (p - m <= i ? t2[p - m][i] : 0.0);
  }
  __syncthreads();
  for (int p = tid; p < m + keep; p += GT) {
    double a[GM_S], h[GM_S];
    for (int t = 0; t < GM_S; ++t) a[t] = 0.0;
    for (int c = p > 0 ? p - 1 : 0; c < j0; ++c) {  // known columns (Hessenberg: row p starts at column p - 1)
      const double hv = gs->hraw[c][p];
#pragma unroll
      for (int t = 0; t < GM_S; ++t) a[t] += hv * (t < keep ? C[t][c] : 0.0);
    }
#pragma unroll
    for (int t = 0; t < GM_S; ++t) {
      h[t] = 0.0;
      if (t < keep) {
        double v = C[t + 1][p] + C[t][p] - a[t];
#pragma unroll
        for (int k = 0; k < GM_S; ++k)
          if (k < t) v -= h[k] * C[t][j0 + k];
        h[t] = p <= j0 + t + 1 ? v / C[t][j0 + t] : 0.0;
        hn[t][p] = h[t];
      }
    }
  }
  __syncthreads();
  if (wp < keep) {  // ||M A Q_j||^2
    double v = 0.0;
    for (int p = lane; p < m + keep; p += 32) v += hn[wp][p] * hn[wp][p];
    v = warp_sum(v);
    if (lane == 0) len2[wp] = v;
  }
  __syncthreads();
  // breakdown (jax _kth_arnoldi_iteration): nothing new left of a column
  if (tid < keep && !(hn[tid][m + tid] > gs->eps * sqrt(len2[tid]))) {
    hn[tid][m + tid] = 0.0;
    len2[tid] = -1.0;
  }
  __syncthreads();
  for (int q = tid; q < keep * (R + 1); q += GT) {
    const int t = q / (R + 1), p = q - t * (R + 1);
    gs->hraw[j0 + t][p] = p < m + keep ? hn[t][p] : 0.0;
  }
  __syncthreads();
  if (rotate && tid < keep)  // the cycle's earlier rotations, a column per thread
    for (int i = 0; i < j0; ++i) {
      const double c = gv[i][0], sn = gv[i][1], x1 = hn[tid][i], y1 = hn[tid][i + 1];
      hn[tid][i] = c * x1 - sn * y1;
      hn[tid][i + 1] = sn * x1 + c * y1;
    }
  __syncthreads();
  if (tid == 0) {
    int done = 0, active = 1;
    for (int t = 0; t < keep && active; ++t) {
      const int j = j0 + t;
      done = t + 1;
      if (!rotate) {
        if (len2[t] < 0.0) { gs->breakdown = 1; active = 0; }
        continue;
      }
      double* row = hn[t];
      for (int i = j0; i < j; ++i) {
        const double c = gv[i][0], sn = gv[i][1], x1 = row[i], y1 = row[i + 1];
        row[i] = c * x1 - sn * y1;
        row[i + 1] = sn * x1 + c * y1;
      }
      // _givens_rotation(a, b)
      const double a = row[j], b = row[j + 1];
      double cs, sn;
      if (b == 0.0) {
        cs = 1.0; sn = 0.0;
      } else if (fabs(a) < fabs(b)) {
        const double q = -a / b, r = 1.0 / sqrt(1.0 + q * q);
        cs = r * q; sn = r;
      } else {
        const double q = -b / a, r = 1.0 / sqrt(1.0 + q * q);
        cs = r; sn = r * q;
      }
      gv[j][0] = gs->givens[j][0] = cs;
      gv[j][1] = gs->givens[j][1] = sn;
      row[j] = cs * a - sn * b;
      row[j + 1] = sn * a + cs * b;
      const double b0 = gs->beta[j], b1 = gs->beta[j + 1];
      gs->beta[j] = cs * b0 - sn * b1;
      gs->beta[j + 1] = sn * b0 + cs * b1;
      gs->err = fabs(gs->beta[j + 1]);
      if (!(gs->err > gs->ptol)) active = 0;
    }
    if (keep < s && active) {  // columns lost to rounding, and the cycle not over: see small_solve_state
      gs->narrow = 1;
      active = 0;
    }
    gs->kdone = j0 + done;
    gs->active = active;
    done_s = done;
    // the block's last vector feeds the next one
    const int last = keep - 1;
    gs->s[m + last] = ri[last][last];
    gs->cstart = m;
    gs->clen = keep;
    for (int q = 0; q <= last; ++q) gs->clast[q] = rc[q][last];
  }
  for (int q = tid; q < keep * GM_S; q += GT) {
    const int i = q / GM_S, p = q - i * GM_S;
    gs->B[m + i][p] = p <= i ? ri[p][i] : 0.0;
    if (p == 0) gs->bstart[m + i] = m;
  }
  __syncthreads();
  for (int q = tid; q < done_s * (R + 1); q += GT) {
    const int t = q / (R + 1), p = q - t * (R + 1);
    gs->H[j0 + t][p] = p <= m + t ? hn[t][p] : 0.0;
  }
}

// V_{m+i} <- sum_k u[k][i] Z_k - sum_l cv[l][i] V_l for the S new vectors
// (m = j0 + 1) and the Gram matrix of the results as stored.  One 16-byte
// chunk of all S vectors per thread, four basis vectors' loads in flight.
// Bound by reading m + S and writing S vectors.  Tiles are taken from the end
// of the vectors: block_dots has just walked them from the front, so the
// last tens of MB of every row are still in the 126 MB L2.  256x256x80
// float32, the updates of a cycle of 30: 8.2 ms in one-step form, 2.43 ms
// here (5.4 TB/s).
template <typename T, int S>
__device__ __forceinline__ void block_update_body(T* Vb, size_t stride, int j0, size_t n, double* partial,
                                                  GState* gs, int bid, int nblk) {
  constexpr int VN = V16<T>::n;
  constexpr int NP = S * (S + 1) / 2;
  constexpr int LD = 8;  // coefficients per row, padded for vector loads
  __shared__ __align__(16) T cf[(GM_MAXR + 1) * LD];
  __shared__ double red[NP][GT / 32];
  __shared__ double gram[GM_S][GM_S];
  const int tid = threadIdx.x, lane = tid & 31, wp = tid >> 5;
  const int m = j0 + 1;
  for (int q = tid; q < (m + S) * LD; q += GT) {
    const int l = q / LD, i = q - l * LD;
    cf[q] = i >= S ? T(0) : (T)(l < m ? -gs->cv[l][i] : gs->u[l - m][i]);
  }
  __syncthreads();
  const T* cu = cf + m * LD;
  T* zb = Vb + (size_t)m * stride;
  double g[NP];
#pragma unroll
  for (int q = 0; q < NP; ++q) g[q] = 0.0;
  const size_t tile = (size_t)GT * VN;
  for (long long t = (long long)((n + tile - 1) / tile) - 1 - bid; t >= 0; t -= nblk) {
    const size_t off = (size_t)t * tile + (size_t)tid * VN;
    if (off >= n) continue;
    T acc[S][VN];
    {
      T z[S][VN];
#pragma unroll
      for (int k = 0; k < S; ++k) load16_rw(zb + (size_t)k * stride + off, z[k]);
#pragma unroll
      for (int i = 0; i < S; ++i)
#pragma unroll
        for (int e = 0; e < VN; ++e) {
          T v = cu[i] * z[0][e];
#pragma unroll
          for (int k = 1; k <= i; ++k) v += cu[k * LD + i] * z[k][e];
          acc[i][e] = v;
        }
    }
    const T* v = Vb + off;
    int l = 0;
    for (; l + 4 <= m; l += 4, v += 4 * stride) {
      T x[4][VN];
#pragma unroll
      for (int q = 0; q < 4; ++q) load16_rw(v + (size_t)q * stride, x[q]);
#pragma unroll
      for (int q = 0; q < 4; ++q)
#pragma unroll
        for (int i = 0; i < S; ++i) {
          const T c = cf[(l + q) * LD + i];
#pragma unroll
          for (int e = 0; e < VN; ++e) acc[i][e] += c * x[q][e];
        }
    }
    for (; l < m; ++l, v += stride) {
      T x[VN];
      load16_rw(v, x);
#pragma unroll
      for (int i = 0; i < S; ++i) {
        const T c = cf[l * LD + i];
#pragma unroll
        for (int e = 0; e < VN; ++e) acc[i][e] += c * x[e];
      }
    }
#pragma unroll
    for (int i = 0; i < S; ++i) store16(zb + (size_t)i * stride + off, acc[i]);
#pragma unroll
    for (int e = 0; e < VN; ++e) {
      double d[S];
#pragma unroll
      for (int i = 0; i < S; ++i) d[i] = (double)acc[i][e];
      int q = 0;
#pragma unroll
      for (int i = 0; i < S; ++i)
#pragma unroll
        for (int k = i; k < S; ++k) g[q++] += d[i] * d[k];
    }
  }
#pragma unroll
  for (int q = 0; q < NP; ++q) {
    const double v = warp_sum(g[q]);
    if (lane == 0) red[q][wp] = v;
  }
  __syncthreads();
  if (tid < NP) {
    double v = 0.0;
    for (int k = 0; k < GT / 32; ++k) v += red[tid][k];
    partial[(size_t)bid * NP + tid] = v;
  }
  if (!last_block(&gs->counter, (unsigned)nblk)) return;
  for (int q = wp; q < NP; q += GT / 32) {
    double v = 0.0;
    for (int b = lane; b < nblk; b += 32) v += __ldcg(partial + (size_t)b * NP + q);
    v = warp_sum(v);
    if (lane == 0) {
      int i = 0, r = q;
      while (r >= S - i) { r -= S - i; ++i; }
      gram[i][i + r] = v;
    }
  }
  if (tid == 0) gs->counter = 0;
  __syncthreads();
  block_finish(gs, gram, j0, S);
}

template <typename T, int S>
__global__ void __launch_bounds__(GT, 2) block_update_kernel(T* Vb, size_t stride, int j0, size_t n, double* partial,
                                                             GState* gs) {
  grid_chain();
  if (gs->active == 0) return;
  block_update_body<T, S>(Vb, stride, j0, n, partial, gs, blockIdx.x, gridDim.x);
}

// x64 += sum_{i < min(m, kdone)} coef_i V_i with a float64 solution (the
// end-of-cycle update of GMRES with iterative refinement)
template <typename T>
__device__ __forceinline__ void update_x64_body(const T* __restrict__ Vb, size_t stride, int m,
                                                double* __restrict__ x, size_t n, const GState* gs, int bid,
                                                int nblk) {
  __shared__ double cf[GM_MAXR + 2];
  const int mm = min(m, gs->kdone);
  for (int q = threadIdx.x; q < mm; q += blockDim.x) cf[q] = gs->coef[q];
  __syncthreads();
  // CH 16-byte chunks of T per thread and tile (n is a multiple of 64: the
  // packed fields are padded), every chunk's loads in flight together; per
  // element the sum runs in the order acc = x, acc += coef_i V_i (i = 0, 1, ..)
  constexpr int VN = V16<T>::n;
  constexpr int E = CH * VN;
  const int tid = threadIdx.x, nt = blockDim.x;
  const size_t tile = (size_t)nt * E;
  for (size_t base = (size_t)bid * tile; base < n; base += (size_t)nblk * tile) {
    double acc[E];
    bool ok[CH];
#pragma unroll
    for (int c = 0; c < CH; ++c) {
      const size_t off = base + ((size_t)c * nt + tid) * VN;
      ok[c] = off < n;
#pragma unroll
      for (int e = 0; e < VN; ++e) acc[c * VN + e] = ok[c] ? x[off + e] : 0.0;
    }
    for (int i = 0; i < mm; ++i) {
      const T* __restrict__ Vi = Vb + (size_t)i * stride;
      const double ci = cf[i];
#pragma unroll
      for (int c = 0; c < CH; ++c) {
        if (!ok[c]) continue;
        const size_t off = base + ((size_t)c * nt + tid) * VN;
        T vr[VN];
        load16(Vi + off, vr);
#pragma unroll
        for (int e = 0; e < VN; ++e) acc[c * VN + e] += ci * (double)vr[e];
      }
    }
#pragma unroll
    for (int c = 0; c < CH; ++c) {
      if (!ok[c]) continue;
      const size_t off = base + ((size_t)c * nt + tid) * VN;
#pragma unroll
      for (int e = 0; e < VN; ++e) x[off + e] = acc[c * VN + e];
    }
  }
}
template <typename T>
__global__ void __launch_bounds__(256) update_x64_kernel(const T* __restrict__ Vb, size_t stride, int m,
                                                         double* __restrict__ x, size_t n, const GState* gs) {
  grid_chain();
  update_x64_body<T>(Vb, stride, m, x, n, gs, blockIdx.x, gridDim.x);
}

// w <- w + sign * sum_{i<m'} coef_i V_i with coef from gs->coef (UM_NONE,
// m' = min(m, kdone) when limit_kdone) or coef_i = h_i s_i (UM_ARNOLDI),
// then optionally finish the Arnoldi step j = m - 1.
template <typename T>
__device__ __forceinline__ void update_body(const T* __restrict__ Vb, size_t stride, int m, T* __restrict__ w,
                                            size_t n, double sign, double* partial, GState* gs, int mode,
                                            int limit_kdone, int bid, int nblk) {
  __shared__ double cf[GM_MAXR + 2];
  __shared__ double red[GT / 32];
  int mm = m;
  if (limit_kdone) mm = min(m, gs->kdone);
  for (int q = threadIdx.x; q < mm; q += blockDim.x)
    cf[q] = sign * (mode == UM_ARNOLDI ? gs->h[q] * gs->s[q] : gs->coef[q]);
  __syncthreads();
  constexpr int VN = V16<T>::n;
  constexpr int E = CH * VN;
  const size_t tile = (size_t)GT * E;
  double sq = 0.0;
  for (size_t base = (size_t)bid * tile; base < n; base += (size_t)nblk * tile) {
    T wr[E];
    bool ok[CH];
#pragma unroll
    for (int c = 0; c < CH; ++c) {
      const size_t off = base + ((size_t)c * GT + threadIdx.x) * VN;
      ok[c] = off < n;
      if (ok[c]) load16(w + off, wr + c * VN);
    }
    for (int i = 0; i < mm; ++i) {
      const T* __restrict__ Vi = Vb + (size_t)i * stride;
      const T ci = (T)cf[i];
#pragma unroll
      for (int c = 0; c < CH; ++c) {
        if (!ok[c]) continue;
        const size_t off = base + ((size_t)c * GT + threadIdx.x) * VN;
        T vr[VN];
        load16(Vi + off, vr);
#pragma unroll
        for (int e = 0; e < VN; ++e) wr[c * VN + e] += ci * vr[e];
      }
    }
#pragma unroll
    for (int c = 0; c < CH; ++c) {
      if (!ok[c]) continue;
      const size_t off = base + ((size_t)c * GT + threadIdx.x) * VN;
      store16(w + off, wr + c * VN);
#pragma unroll
      for (int e = 0; e < VN; ++e) sq += (double)wr[c * VN + e] * (double)wr[c * VN + e];
    }
  }
  if (mode != UM_ARNOLDI) return;
  sq = warp_sum(sq);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = sq;
  __syncthreads();
  if (threadIdx.x == 0) {
    double s = 0.0;
    for (int q = 0; q < GT / 32; ++q) s += red[q];
    partial[bid] = s;
  }
  if (!last_block(&gs->counter, (unsigned)nblk)) return;
  if (threadIdx.x >= 32) return;
  double tot = 0.0;  // warp 0 sums the blocks' partials
  for (int b = threadIdx.x; b < nblk; b += 32) tot += partial[b];
  tot = warp_sum(tot);
  if (threadIdx.x != 0) return;
  gs->counter = 0;
  // ---- finish Arnoldi step j (jax _kth_arnoldi_iteration) ----
  const int j = m - 1;
  const int R = gs->restart;
  double vn1 = sqrt(tot);
  const double thresh = gs->eps * gs->hn0;
  if (vn1 > thresh) {
    gs->s[j + 1] = 1.0 / vn1;
  } else {
    gs->s[j + 1] = 0.0;
    vn1 = 0.0;
  }
  double row[GM_MAXR + 1];
  for (int q = 0; q <= R; ++q) row[q] = 0.0;
  for (int q = 0; q <= j; ++q) row[q] = gs->h[q];
  row[j + 1] = vn1;
  gs->kdone = j + 1;
  if (gs->method == 0) {  // batched: H[j, :] = h
    for (int q = 0; q <= R; ++q) gs->H[j][q] = row[q];
    if (vn1 == 0.0) { gs->breakdown = 1; gs->active = 0; }
  } else {  // incremental: rotate into R, update beta
    for (int i = 0; i < j; ++i) {
      const double c = gs->givens[i][0], s = gs->givens[i][1];
      const double x1 = row[i], y1 = row[i + 1];
      row[i] = c * x1 - s * y1;
      row[i + 1] = s * x1 + c * y1;
    }
    // _givens_rotation(a, b)
    const double a = row[j], b = row[j + 1];
    double cs, sn;
    if (b == 0.0) {
      cs = 1.0; sn = 0.0;
    } else if (fabs(a) < fabs(b)) {
      const double t = -a / b, r = 1.0 / sqrt(1.0 + t * t);
      cs = r * t; sn = r;
    } else {
      const double t = -b / a, r = 1.0 / sqrt(1.0 + t * t);
      cs = r; sn = r * t;
    }
    gs->givens[j][0] = cs;
    gs->givens[j][1] = sn;
    row[j] = cs * a - sn * b;
    row[j + 1] = sn * a + cs * b;
    for (int q = 0; q <= R; ++q) gs->H[j][q] = row[q];
    const double b0 = gs->beta[j], b1 = gs->beta[j + 1];
    gs->beta[j] = cs * b0 - sn * b1;
    gs->beta[j + 1] = sn * b0 + cs * b1;
    gs->err = fabs(gs->beta[j + 1]);
    if (!(gs->err > gs->ptol)) gs->active = 0;
  }
}
template <typename T>
__global__ void __launch_bounds__(GT) update_kernel(const T* __restrict__ Vb, size_t stride, int m,
                                                    T* __restrict__ w, size_t n, double sign, double* partial,
                                                    GState* gs, int mode, int gated, int limit_kdone) {
  grid_chain();
  if (gated && gs->active == 0) return;
  update_body<T>(Vb, stride, m, w, n, sign, partial, gs, mode, limit_kdone, blockIdx.x, gridDim.x);
}

__device__ void setup_state(GState* gs, double eps, double tol, double atol_in, int restart, int method, int columns) {
  gs->eps = eps;
  gs->tol = tol;
  gs->atol_in = atol_in;
  gs->restart = restart;
  gs->method = method;
  gs->columns = columns;
  gs->counter = 0;
  for (int q = 0; q < GM_BLOCKS / GM_GROUP + 1; ++q) gs->group_counter[q] = 0;
  gs->active = 1;
  gs->kdone = 0;
  gs->breakdown = 0;
  gs->narrow = 0;
  gs->cycles = 0;
  gs->steps = 0;
  for (int q = 0; q < GM_MAXR + 2; ++q) gs->s[q] = 0.0;
}
__global__ void setup_kernel(GState* gs, double eps, double tol, double atol_in, int restart, int method,
                             int columns) {
  grid_chain();
  setup_state(gs, eps, tol, atol_in, restart, method, columns);
}

// The restart loop runs in the block form (block = 1) until a cycle is narrow
// or it ends, then one column at a time (block = 0).  A narrow cycle is not
// counted.
__device__ __forceinline__ void count_cycle(GState* gs) {
  if (gs->narrow) return;
  gs->cycles += 1;
  gs->steps += gs->kdone;
}
__device__ __forceinline__ bool another_cycle(const GState* gs, int maxiter, int block) {
  return gs->rnorm > gs->atol && gs->cycles < maxiter && (gs->columns > 1) == (block != 0);
}
// Graph mode: after a residual, count the finished cycle and set the WHILE
// condition: another cycle of this form while ||M r|| > atol and cycles < maxiter.
__global__ void gate_kernel(GState* gs, cudaGraphConditionalHandle h, int maxiter, int after_cycle, int block) {
  grid_chain();
  if (after_cycle) count_cycle(gs);
  cudaGraphSetConditional(h, another_cycle(gs, maxiter, block) ? 1u : 0u);
}

__device__ void info_state(const GState* gs, GDevInfo* o) {
  o->cycles = gs->cycles;
  o->arnoldi_steps = gs->steps;
  o->converged = (gs->rnorm <= gs->atol) ? 1 : 0;
  o->pad = 0;
  o->residual_norm = gs->rnorm;
  o->atol = gs->atol;
  o->b_norm = gs->bnorm;
}
__global__ void info_kernel(const GState* gs, GDevInfo* o) { grid_chain(); info_state(gs, o); }

__device__ void init_tol_state(GState* gs) {
  // atol = max(tol ||b||, atol); ptol = ||M b|| min(1, atol / ||b||)
  gs->atol = fmax(gs->tol * gs->bnorm, gs->atol_in);
  gs->ptol = gs->mbnorm * fmin(1.0, gs->atol / gs->bnorm);
}
__global__ void init_tol_kernel(GState* gs) { grid_chain(); init_tol_state(gs); }

__device__ void begin_cycle_state(GState* gs) {
  const int R = gs->restart;
  for (int q = threadIdx.x; q < R * (GM_MAXR + 1); q += blockDim.x) {
    const int r = q / (GM_MAXR + 1), c = q % (GM_MAXR + 1);
    gs->H[r][c] = (r == c) ? 1.0 : 0.0;  // eye(restart, restart + 1)
  }
  for (int q = threadIdx.x; q <= R; q += blockDim.x) gs->beta[q] = 0.0;
  for (int q = threadIdx.x; q < R; q += blockDim.x) { gs->givens[q][0] = 0.0; gs->givens[q][1] = 0.0; }
  __syncthreads();
  if (threadIdx.x == 0) {
    gs->beta[0] = gs->rnorm;
    gs->err = gs->rnorm;
    gs->active = 1;
    gs->kdone = 0;
    gs->breakdown = 0;
    gs->narrow = 0;
  }
}
__global__ void begin_cycle_kernel(GState* gs) {
  grid_chain();
  begin_cycle_state(gs);
}

// y from the cycle's small problem; coef_i = y_i s_i, or B y in the block
// form, whose triangular solves run on one warp.
// Columns of H the least-squares solve stages at a time.
constexpr int SS_C = 32;
// the factorisation of a restart of 100 has work for 32 warps, one of 30 for 8
inline int small_solve_threads(int R) { return R > 32 ? 1024 : 256; }
inline size_t small_solve_smem(int R) { return ((size_t)R * R + (size_t)SS_C * (R | 1)) * sizeof(double); }

// One warp: x <- the solution of T^T x = x for the lower triangle T (row
// stride ld, n <= GM_MAXR rows) with reciprocal diagonal rd, from the last row
// up; a lane keeps every 32nd element, and each solved one is subtracted
// from all the others at once (its row of T is read ahead of it).
__device__ __forceinline__ void triangle_back(const double* t, int ld, int n, const double* rd, double* x) {
  const int lane = threadIdx.x & 31;
  double v[GM_MAXR / 32];
#pragma unroll
  for (int q = 0; q < GM_MAXR / 32; ++q) v[q] = lane + 32 * q < n ? x[lane + 32 * q] : 0.0;
#pragma unroll
  for (int q = GM_MAXR / 32 - 1; q >= 0; --q) {
    for (int i = min(n, 32 * (q + 1)) - 1; i >= 32 * q; --i) {
      const double xi = __shfl_sync(0xffffffffu, v[q], i & 31) * rd[i];
#pragma unroll
      for (int m = 0; m <= q; ++m) {
        const int k = lane + 32 * m;
        if (k < i) v[m] -= t[i * ld + k] * xi;
      }
      if (lane == (i & 31)) v[q] = xi;
    }
  }
#pragma unroll
  for (int q = 0; q < GM_MAXR / 32; ++q)
    if (lane + 32 * q < n) x[lane + 32 * q] = v[q];
}

// The cycle's least-squares problem, one block.  Bound by its serial chain:
// what each pivot and each solved unknown waits for.  Restart 100, batched: 530
// us with strided reads of H, an integer division per updated element and two
// warp sums per unknown, 151 us here (186 with 8 warps); restart 30,
// incremental: 22.5 -> 6.2 us.
__device__ void small_solve_state(GState* gs) {
  extern __shared__ double a2[];  // R * R, then a chunk of columns of H
  const int R = gs->restart, kd = gs->kdone, tid = threadIdx.x, lane = tid & 31, wp = tid >> 5, nw = blockDim.x >> 5;
  __shared__ double b2[GM_MAXR];
  __shared__ double y[GM_MAXR];
  __shared__ double rd[GM_MAXR];  // reciprocal diagonal of a triangular solve
  if (gs->narrow) {  // nothing of the cycle is used: x stays, and it is done over one column at a time
    __syncthreads();
    if (tid == 0) {
      gs->kdone = 0;
      gs->columns = 1;
    }
    return;
  }
  if (gs->method == 0) {
    // _lstsq(H.T, beta): normal equations (H H^T) y = H beta, Cholesky solve, over the cycle's kd steps.  A row past
    // them is an identity row (begin_cycle): as an unknown it would meet the last step's subdiagonal equation for
    // nothing and leave the square Hessenberg system in the least-squares problem's place.  Row p of H ends at column
    // p + 1, and the lower triangle is enough.
    const int P = R | 1;
    double* ht = a2 + (size_t)R * R;  // [SS_C][P]: columns c0 .. of H, transposed
    for (int q = tid; q < kd * R; q += blockDim.x) a2[q] = 0.0;
    for (int p = tid; p < kd; p += blockDim.x) b2[p] = 0.0;
    for (int c0 = 0; c0 <= kd; c0 += SS_C) {
      const int nc = min(SS_C, kd + 1 - c0);
      __syncthreads();
      for (int q = tid; q < kd * SS_C; q += blockDim.x) {
        const int r = q / SS_C, c = q % SS_C;
        if (c < nc) ht[c * P + r] = gs->H[r][c0 + c];
      }
      __syncthreads();
      for (int p = max(c0 - 1, 0) + wp; p < kd; p += nw)
        for (int r = max(c0 - 1, 0) + lane; r <= p; r += 32) {
          double v = a2[p * R + r];
          for (int c = 0; c < min(nc, r + 2 - c0); ++c) v += ht[c * P + p] * ht[c * P + r];
          a2[p * R + r] = v;
        }
      for (int p = tid; p < kd; p += blockDim.x) {
        double v = b2[p];
        for (int c = 0; c < min(nc, p + 2 - c0); ++c) v += ht[c * P + p] * gs->beta[c0 + c];
        b2[p] = v;
      }
    }
    __syncthreads();
    // right-looking Cholesky, lower factor stored in a2; with several columns per block the right-hand side rides
    // along as one more row, which leaves L^-1 b2 in y
    const bool carry = gs->columns > 1;
    for (int k = 0; k < kd; ++k) {
      const double dkk = sqrt(a2[k * R + k]);
      __syncthreads();  // every thread has the pivot
      for (int i = k + 1 + tid; i < kd; i += blockDim.x) a2[i * R + k] /= dkk;
      if (tid == 0) {
        a2[k * R + k] = dkk;
        rd[k] = 1.0 / dkk;
        if (carry) y[k] = b2[k] / dkk;
      }
      __syncthreads();
      for (int i = k + 1 + wp; i < kd; i += nw) {
        const double lik = a2[i * R + k];
        for (int jj = k + 1 + lane; jj <= i; jj += 32) a2[i * R + jj] -= lik * a2[jj * R + k];
      }
      if (carry)
        for (int i = k + 1 + tid; i < kd; i += blockDim.x) b2[i] -= a2[i * R + k] * y[k];
      __syncthreads();
    }
    if (carry) {
      if (wp == 0) triangle_back(a2, R, kd, rd, y);  // L^T y = z
    } else if (tid == 0) {
      for (int i = 0; i < kd; ++i) {  // L z = b2
        double s = b2[i];
        for (int k = 0; k < i; ++k) s -= a2[i * R + k] * y[k];
        y[i] = s / a2[i * R + i];
      }
      for (int i = kd - 1; i >= 0; --i) {  // L^T y = z
        double s = y[i];
        for (int k = i + 1; k < kd; ++k) s -= a2[k * R + i] * y[k];
        y[i] = s / a2[i * R + i];
      }
      for (int i = 0; i < R; ++i) gs->coef[i] = (i < kd) ? y[i] * gs->s[i] : 0.0;
    }
  } else {
    // back substitution with the rotated rows: sum_j R[j][i] y_j = beta_i
    if (gs->columns > 1) {
      for (int q = tid; q < kd * R; q += blockDim.x) {
        const int i = q / R, k = q % R;
        if (k < i) a2[i * R + k] = gs->H[i][k];
      }
      for (int i = tid; i < kd; i += blockDim.x) {
        rd[i] = 1.0 / gs->H[i][i];
        y[i] = gs->beta[i];
      }
      __syncthreads();
      if (wp == 0) triangle_back(a2, R, kd, rd, y);
    } else if (threadIdx.x == 0) {
      for (int i = kd - 1; i >= 0; --i) {
        double s = gs->beta[i];
        for (int jj = i + 1; jj < kd; ++jj) s -= gs->H[jj][i] * y[jj];
        y[i] = s / gs->H[i][i];
      }
      for (int i = 0; i < R; ++i) gs->coef[i] = (i < kd) ? y[i] * gs->s[i] : 0.0;
    }
  }
  if (gs->columns == 1) return;
  __syncthreads();
  for (int k = threadIdx.x; k < R; k += blockDim.x) {
    double v = 0.0;
    if (k < kd) {
      const int st = gs->bstart[k];
      for (int l = k; l < kd && gs->bstart[l] == st; ++l) v += gs->B[l][k - st] * y[l];
    }
    gs->coef[k] = v;
  }
}
__global__ void __launch_bounds__(1024) small_solve_kernel(GState* gs) {
  grid_chain();
  small_solve_state(gs);
}

__global__ void snapshot_kernel(const GState* gs, GHostView* v) {
  grid_chain();
  v->rnorm = gs->rnorm;
  v->atol = gs->atol;
  v->bnorm = gs->bnorm;
  v->kdone = gs->kdone;
  v->narrow = gs->narrow;
}

// ---------------------------------------------------------------------------
// grouped launches over ensemble members: flat block b runs block
// (b - first[m]) of member m's standalone launch (sisl_group.cuh)
// ---------------------------------------------------------------------------
template <typename T>
__device__ __forceinline__ T* gvec(const GroupMember<T>& g, int v) {
  return g.vec + (size_t)v * g.npad;
}

template <typename T>
__global__ void group_dots_kernel(GroupMember<T>* mem, const int* __restrict__ first, int M, int m, int wv,
                                  int mode, int gated) {
  grid_chain();
  const int b = blockIdx.x;
  const int mi = group_find(first, M, b);
  const GroupMember<T>& g = mem[mi];
  if (!g.running || (gated && g.gs->active == 0)) return;
  const int f0 = first[mi];
  dots_body<T>(gvec(g, GV_V0), g.npad, m, gvec(g, wv), g.npad, g.partial, g.gs, mode, b - f0, first[mi + 1] - f0);
}

template <typename T, int NT>
__global__ void __launch_bounds__(GT, 2) group_block_dots_kernel(GroupMember<T>* mem, const int* __restrict__ first,
                                                                 int M, int j0, int s) {
  grid_chain();
  const int b = blockIdx.x;
  const int mi = group_find(first, M, b);
  const GroupMember<T>& g = mem[mi];
  if (!g.running || g.gs->active == 0) return;
  const int f0 = first[mi];
  block_dots_body<T, NT>(gvec(g, GV_V0), g.npad, j0, s, g.npad, g.partial, g.gs, b - f0, first[mi + 1] - f0);
}
template <typename T, int S>
__global__ void __launch_bounds__(GT, 2) group_block_update_kernel(GroupMember<T>* mem, const int* __restrict__ first,
                                                                   int M, int j0) {
  grid_chain();
  const int b = blockIdx.x;
  const int mi = group_find(first, M, b);
  const GroupMember<T>& g = mem[mi];
  if (!g.running || g.gs->active == 0) return;
  const int f0 = first[mi];
  block_update_body<T, S>(gvec(g, GV_V0), g.npad, j0, g.npad, g.partial, g.gs, b - f0, first[mi + 1] - f0);
}
// final_x = 0: Arnoldi projection of V_m out of V_0 .. V_{m-1} (gated);
// final_x = 1: x += sum coef_i V_i over the cycle's basis
template <typename T>
__global__ void __launch_bounds__(GT) group_update_kernel(GroupMember<T>* mem, const int* __restrict__ first, int M,
                                                          int m, int final_x) {
  grid_chain();
  const int b = blockIdx.x;
  const int mi = group_find(first, M, b);
  const GroupMember<T>& g = mem[mi];
  if (!g.running) return;
  const int f0 = first[mi], nb = first[mi + 1] - f0;
  if (final_x) {
    update_body<T>(gvec(g, GV_V0), g.npad, m, gvec(g, GV_X), g.npad, 1.0, g.partial, g.gs, UM_NONE, 1, b - f0, nb);
  } else {
    if (g.gs->active == 0) return;
    update_body<T>(gvec(g, GV_V0), g.npad, m, gvec(g, GV_V0 + m), g.npad, -1.0, g.partial, g.gs, UM_ARNOLDI, 0,
                   b - f0, nb);
  }
}

template <typename T>
__global__ void __launch_bounds__(256) group_update_x64_kernel(GroupMember<T>* mem, const int* __restrict__ first,
                                                               int M, int m) {
  grid_chain();
  const int b = blockIdx.x;
  const int mi = group_find(first, M, b);
  const GroupMember<T>& g = mem[mi];
  if (!g.running) return;
  const int f0 = first[mi];
  update_x64_body<T>(gvec(g, GV_V0), g.npad, m, g.x64, g.npad, g.gs, b - f0, first[mi + 1] - f0);
}

// 0: b64 = b, x64 = x, r64 = 0; 1: residual r64 -> V_0 (u, v) | z (w, pi,
// eta_dot); 2: x = x64 (after the loop: every member); 3: V_1 (u, v) = b (u, v);
// 4: transposed residual r64 -> z
template <typename T>
__global__ void __launch_bounds__(256) group_convert_kernel(GroupMember<T>* mem, const int* __restrict__ first,
                                                            int M, int mode) {
  grid_chain();
  const int b = blockIdx.x;
  const int mi = group_find(first, M, b);
  const GroupMember<T>& g = mem[mi];
  if (mode != 2 && !g.running) return;
  const size_t f0 = first[mi], nb = first[mi + 1] - f0;
  const size_t n = (mode == 3) ? g.off[2] : g.npad;
  const size_t step = nb * blockDim.x;
  T* x = gvec(g, GV_X);
  const T* bv = gvec(g, GV_B);
  T* v0 = gvec(g, GV_V0);
  T* z = gvec(g, GV_Z);
  for (size_t e = (b - f0) * (size_t)blockDim.x + threadIdx.x; e < n; e += step) {
    if (mode == 0) {
      g.b64[e] = (double)bv[e];
      g.x64[e] = (double)x[e];
      g.r64[e] = 0.0;
    } else if (mode == 1) {
      (e < g.off[2] ? v0 : z)[e] = (T)g.r64[e];
    } else if (mode == 2) {
      x[e] = (T)g.x64[e];
    } else if (mode == 4) {
      z[e] = (T)g.r64[e];
    } else {
      v0[g.npad + e] = bv[e];
    }
  }
}

// one thread per member
template <typename T>
__global__ void group_setup_kernel(GroupMember<T>* mem, int M, int R, int method, int transpose, int columns) {
  grid_chain();
  const int m = blockIdx.x * blockDim.x + threadIdx.x;
  if (m >= M) return;
  GroupMember<T>& g = mem[m];
  setup_state(g.gs, g.eps, transpose ? g.tol_t : g.tol, g.atol_in, R, method, columns);
  g.running = 1;
}
template <typename T>
__global__ void group_init_tol_kernel(GroupMember<T>* mem, int M) {
  grid_chain();
  const int m = blockIdx.x * blockDim.x + threadIdx.x;
  if (m < M) init_tol_state(mem[m].gs);
}
template <typename T>
__global__ void group_info_kernel(GroupMember<T>* mem, int M, int solve) {
  grid_chain();
  const int m = blockIdx.x * blockDim.x + threadIdx.x;
  if (m < M && mem[m].info[solve]) info_state(mem[m].gs, mem[m].info[solve]);
}
// one block per member
template <typename T>
__global__ void group_begin_cycle_kernel(GroupMember<T>* mem) {
  grid_chain();
  const GroupMember<T>& g = mem[blockIdx.x];
  if (g.running) begin_cycle_state(g.gs);
}
template <typename T>
__global__ void __launch_bounds__(1024) group_small_solve_kernel(GroupMember<T>* mem) {
  grid_chain();
  const GroupMember<T>& g = mem[blockIdx.x];
  if (g.running) small_solve_state(g.gs);
}
// one block: count the finished cycle of every running member, decide which
// members continue in this form, set the WHILE condition while any does
template <typename T>
__global__ void group_gate_kernel(GroupMember<T>* mem, int M, cudaGraphConditionalHandle h, int after_cycle,
                                  int block) {
  grid_chain();
  int any = 0;
  for (int m = threadIdx.x; m < M; m += blockDim.x) {
    GroupMember<T>& g = mem[m];
    if (after_cycle && g.running) count_cycle(g.gs);
    const int more = (g.running || !after_cycle) && another_cycle(g.gs, g.maxiter, block);
    g.running = more;
    any |= more;
  }
  any = __syncthreads_or(any);
  if (threadIdx.x == 0) cudaGraphSetConditional(h, any ? 1u : 0u);
}

int flat_grid(size_t n, int elems_per_block) {
  size_t b = (n + elems_per_block - 1) / elems_per_block;
  if (b > (size_t)GM_MAXBLOCKS) b = GM_MAXBLOCKS;
  if (b < 1) b = 1;
  return (int)b;
}

// Grid of a grid-stride Krylov kernel: every block resident at once (one
// wave, no tail of a partial second wave), at most GM_MAXBLOCKS.
int resident_grid(const void* fn, int threads, size_t smem, size_t n, int elems_per_block) {
  static std::atomic<int> sms[SMEM_LIMIT_DEVICES];  // SM count per device, found once
  int dev = 0;
  cudaGetDevice(&dev);
  const bool slot = dev >= 0 && dev < SMEM_LIMIT_DEVICES;
  int ns = slot ? sms[dev].load() : 0;
  if (ns == 0) {
    if (cudaDeviceGetAttribute(&ns, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || ns < 1) ns = 148;
    if (slot) sms[dev].store(ns);
  }
  int per_sm = 0;
  if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, fn, threads, smem) != cudaSuccess || per_sm < 1)
    per_sm = 1;
  size_t want = (n + elems_per_block - 1) / elems_per_block;
  size_t cap = (size_t)per_sm * ns;
  if (cap > (size_t)GM_MAXBLOCKS) cap = GM_MAXBLOCKS;
  if (want > cap) want = cap;
  if (want < 1) want = 1;
  return (int)want;
}

}  // namespace

// resident grid of the float64 solution update (tiles of 256 threads x CH 16-byte chunks)
template <typename T>
int gm_x64_blocks_t(size_t n) {
  return resident_grid((const void*)update_x64_kernel<T>, 256, 0, n, 256 * CH * V16<T>::n);
}

// ---------------------------------------------------------------------------
// host wrappers
// ---------------------------------------------------------------------------
// calls f with the row tile count (a compile-time constant) for `rows` rows
template <typename F>
void with_row_tiles(int rows, F&& f) {
  switch (gm_row_tiles(rows)) {
    case 1: f(std::integral_constant<int, 1>{}); break;
    case 2: f(std::integral_constant<int, 2>{}); break;
    case 3: f(std::integral_constant<int, 3>{}); break;
    case 4: f(std::integral_constant<int, 4>{}); break;
    case 5: f(std::integral_constant<int, 5>{}); break;
    case 6: f(std::integral_constant<int, 6>{}); break;
    case 8: f(std::integral_constant<int, 8>{}); break;
    case 10: f(std::integral_constant<int, 10>{}); break;
    case 13: f(std::integral_constant<int, 13>{}); break;
    default: f(std::integral_constant<int, 17>{}); break;
  }
}
// the same for the columns of a block
template <typename F>
void with_columns(int s, F&& f) {
  switch (s) {
    case 1: f(std::integral_constant<int, 1>{}); break;
    case 2: f(std::integral_constant<int, 2>{}); break;
    case 3: f(std::integral_constant<int, 3>{}); break;
    case 4: f(std::integral_constant<int, 4>{}); break;
    case 5: f(std::integral_constant<int, 5>{}); break;
    default: f(std::integral_constant<int, 6>{}); break;
  }
}

int capped(size_t want) { return want < 1 ? 1 : want > (size_t)GM_BLOCKS ? GM_BLOCKS : (int)want; }
// two passes of a block's 8 warps; one chunk per thread
template <typename T>
int gm_block_dots_blocks(size_t n) {
  return capped((n + 128 * V16<T>::n - 1) / (128 * V16<T>::n));
}
template <typename T>
int gm_block_update_blocks(size_t n) {
  return capped((n + GT * V16<T>::n - 1) / (GT * V16<T>::n));
}

template <typename T>
void gm_block_dots(const T* Vb, size_t stride, int j0, int s, size_t n, double* partial, GState* gs,
                   cudaStream_t st) {
  const int g = gm_block_dots_blocks<T>(n);
  with_row_tiles(j0 + 1 + s, [&](auto nt) {
    launch_chained(block_dots_kernel<T, decltype(nt)::value>, g, GT, 0, st, Vb, stride, j0, s, n, partial, gs);
  });
}

template <typename T>
void gm_block_update(T* Vb, size_t stride, int j0, int s, size_t n, double* partial, GState* gs, cudaStream_t st) {
  const int g = gm_block_update_blocks<T>(n);
  with_columns(s, [&](auto sc) {
    launch_chained(block_update_kernel<T, decltype(sc)::value>, g, GT, 0, st, Vb, stride, j0, n, partial, gs);
  });
}

// shared memory of the dots kernel: (m + 1) per-warp slots of 8 warps
constexpr size_t DOTS_SMEM_MAX = (size_t)(GM_MAXR + 1) * 8 * sizeof(double);
constexpr int DOTS_THREADS = 256;

template <typename T>
void gm_dots(const T* Vb, size_t stride, int m, const T* w, size_t n, double* partial, GState* gs, int mode,
             int gated, cudaStream_t st) {
  static SmemLimit attr_bytes;  // per instantiation
  ensure_smem_limit((const void*)dots_kernel<T>, attr_bytes, (size_t)DOTS_SMEM_MAX);
  const int nt = DOTS_THREADS;
  constexpr int E = CH * V16<T>::n;
  const size_t smem = (size_t)(m + 1) * (nt / 32) * sizeof(double);
  const int g = resident_grid((const void*)dots_kernel<T>, nt, smem, n, nt * E);
  launch_chained(dots_kernel<T>, g, nt, smem, st, Vb, stride, m, w, n, partial, gs, mode, gated);
}

template <typename T>
void gm_update(const T* Vb, size_t stride, int m, T* w, size_t n, double sign, double* partial, GState* gs,
               int mode, int gated, int limit_kdone, cudaStream_t st) {
  constexpr int E = CH * V16<T>::n;
  const int g = resident_grid((const void*)update_kernel<T>, GT, 0, n, GT * E);
  launch_chained(update_kernel<T>, g, GT, 0, st, Vb, stride, m, w, n, sign, partial, gs, mode, gated, limit_kdone);
}

template <typename T>
void gm_update_x64(const T* Vb, size_t stride, int m, double* x, size_t n, const GState* gs, cudaStream_t st) {
  launch_chained(update_x64_kernel<T>, gm_x64_blocks_t<T>(n), 256, 0, st, Vb, stride, m, x, n, gs);
}

void gm_setup(GState* gs, double eps, double tol, double atol_in, int restart, int method, int columns,
              cudaStream_t st) {
  launch_chained(setup_kernel, 1, 1, 0, st, gs, eps, tol, atol_in, restart, method, columns);
}
void gm_init_tol(GState* gs, cudaStream_t st) { launch_chained(init_tol_kernel, 1, 1, 0, st, gs); }
void gm_gate(GState* gs, cudaGraphConditionalHandle h, int maxiter, int after_cycle, int block, cudaStream_t st) {
  launch_chained(gate_kernel, 1, 1, 0, st, gs, h, maxiter, after_cycle, block);
}
void gm_info(const GState* gs, GDevInfo* o, cudaStream_t st) { launch_chained(info_kernel, 1, 1, 0, st, gs, o); }
void gm_begin_cycle(GState* gs, cudaStream_t st) { launch_chained(begin_cycle_kernel, 1, 256, 0, st, gs); }
void gm_small_solve(GState* gs, int restart, cudaStream_t st) {
  const size_t smem = small_solve_smem(restart);
  static SmemLimit attr_bytes;
  ensure_smem_limit((const void*)small_solve_kernel, attr_bytes, small_solve_smem(GM_MAXR));
  launch_chained(small_solve_kernel, 1, small_solve_threads(restart), smem, st, gs);
}
void gm_snapshot(const GState* gs, GHostView* v, cudaStream_t st) {
  launch_chained(snapshot_kernel, 1, 1, 0, st, gs, v);
}

// ---------------------------------------------------------------------------
// grouped host wrappers
// ---------------------------------------------------------------------------
template <typename T>
int gm_dots_threads(int m) {
  (void)m;
  return DOTS_THREADS;
}
template <typename T>
int gm_dots_blocks(int m, size_t n) {
  static SmemLimit attr_bytes;
  ensure_smem_limit((const void*)dots_kernel<T>, attr_bytes, (size_t)DOTS_SMEM_MAX);
  const int nt = gm_dots_threads<T>(m);
  constexpr int E = CH * V16<T>::n;
  return resident_grid((const void*)dots_kernel<T>, nt, (size_t)(m + 1) * (nt / 32) * sizeof(double), n, nt * E);
}
template <typename T>
int gm_update_blocks(size_t n) {
  constexpr int E = CH * V16<T>::n;
  return resident_grid((const void*)update_kernel<T>, GT, 0, n, GT * E);
}
int gm_x64_blocks(size_t n) { return gm_x64_blocks_t<float>(n); }
int group_convert_blocks(size_t n) { return flat_grid(n, 256 * 8) < 296 ? flat_grid(n, 256 * 8) : 296; }

template <typename T>
void grp_setup(const GroupLaunch<T>& g, int transpose, cudaStream_t st) {
  launch_chained(group_setup_kernel<T>, (g.M + 127) / 128, 128, 0, st, g.mem, g.M, g.R, g.method, transpose, GM_S);
}
template <typename T>
void grp_dots(const GroupLaunch<T>& g, int m, int w, int mode, int gated, cudaStream_t st) {
  static SmemLimit attr_bytes;
  ensure_smem_limit((const void*)group_dots_kernel<T>, attr_bytes, (size_t)DOTS_SMEM_MAX);
  const int nt = gm_dots_threads<T>(m);
  const size_t smem = (size_t)(m + 1) * (nt / 32) * sizeof(double);
  launch_chained(group_dots_kernel<T>, g.blocks(GT_DOTS0 + m), nt, smem, st, g.mem, g.row(GT_DOTS0 + m), g.M, m, w,
                 mode, gated);
}
template <typename T>
void grp_block_dots(const GroupLaunch<T>& g, int j0, int s, cudaStream_t st) {
  with_row_tiles(j0 + 1 + s, [&](auto nt) {
    launch_chained(group_block_dots_kernel<T, decltype(nt)::value>, g.blocks(GT_BDOT), GT, 0, st, g.mem,
                   g.row(GT_BDOT), g.M, j0, s);
  });
}
template <typename T>
void grp_block_update(const GroupLaunch<T>& g, int j0, int s, cudaStream_t st) {
  with_columns(s, [&](auto sc) {
    launch_chained(group_block_update_kernel<T, decltype(sc)::value>, g.blocks(GT_BUPD), GT, 0, st, g.mem,
                   g.row(GT_BUPD), g.M, j0);
  });
}
template <typename T>
void grp_update_arnoldi(const GroupLaunch<T>& g, int m, cudaStream_t st) {
  launch_chained(group_update_kernel<T>, g.blocks(GT_UPD), GT, 0, st, g.mem, g.row(GT_UPD), g.M, m, 0);
}
template <typename T>
void grp_update_x(const GroupLaunch<T>& g, cudaStream_t st) {
  if (g.refine) launch_chained(group_update_x64_kernel<T>, g.blocks(GT_X64), 256, 0, st, g.mem, g.row(GT_X64), g.M,
                               g.R);
  else launch_chained(group_update_kernel<T>, g.blocks(GT_UPD), GT, 0, st, g.mem, g.row(GT_UPD), g.M, g.R, 1);
}
template <typename T>
void grp_convert(const GroupLaunch<T>& g, int mode, cudaStream_t st) {
  launch_chained(group_convert_kernel<T>, g.blocks(GT_CVT), 256, 0, st, g.mem, g.row(GT_CVT), g.M, mode);
}
template <typename T>
void grp_init_tol(const GroupLaunch<T>& g, cudaStream_t st) {
  launch_chained(group_init_tol_kernel<T>, (g.M + 127) / 128, 128, 0, st, g.mem, g.M);
}
template <typename T>
void grp_begin_cycle(const GroupLaunch<T>& g, cudaStream_t st) {
  launch_chained(group_begin_cycle_kernel<T>, g.M, 256, 0, st, g.mem);
}
template <typename T>
void grp_small_solve(const GroupLaunch<T>& g, cudaStream_t st) {
  static SmemLimit attr_bytes;
  ensure_smem_limit((const void*)group_small_solve_kernel<T>, attr_bytes, small_solve_smem(GM_MAXR));
  launch_chained(group_small_solve_kernel<T>, g.M, small_solve_threads(g.R), small_solve_smem(g.R), st, g.mem);
}
template <typename T>
void grp_gate(const GroupLaunch<T>& g, cudaGraphConditionalHandle h, int after_cycle, int block, cudaStream_t st) {
  launch_chained(group_gate_kernel<T>, 1, 256, 0, st, g.mem, g.M, h, after_cycle, block);
}
template <typename T>
void grp_info(const GroupLaunch<T>& g, int solve, cudaStream_t st) {
  launch_chained(group_info_kernel<T>, (g.M + 127) / 128, 128, 0, st, g.mem, g.M, solve);
}

#define SISL_GROUP_INST(T)                                                                           \
  template int gm_block_dots_blocks<T>(size_t);                                                      \
  template int gm_block_update_blocks<T>(size_t);                                                    \
  template void grp_block_dots<T>(const GroupLaunch<T>&, int, int, cudaStream_t);                    \
  template void grp_block_update<T>(const GroupLaunch<T>&, int, int, cudaStream_t);                  \
  template int gm_dots_threads<T>(int);                                                              \
  template int gm_dots_blocks<T>(int, size_t);                                                       \
  template int gm_update_blocks<T>(size_t);                                                          \
  template void grp_setup<T>(const GroupLaunch<T>&, int, cudaStream_t);                              \
  template void grp_dots<T>(const GroupLaunch<T>&, int, int, int, int, cudaStream_t);                \
  template void grp_update_arnoldi<T>(const GroupLaunch<T>&, int, cudaStream_t);                     \
  template void grp_update_x<T>(const GroupLaunch<T>&, cudaStream_t);                                \
  template void grp_convert<T>(const GroupLaunch<T>&, int, cudaStream_t);                            \
  template void grp_init_tol<T>(const GroupLaunch<T>&, cudaStream_t);                                \
  template void grp_begin_cycle<T>(const GroupLaunch<T>&, cudaStream_t);                             \
  template void grp_small_solve<T>(const GroupLaunch<T>&, cudaStream_t);                             \
  template void grp_gate<T>(const GroupLaunch<T>&, cudaGraphConditionalHandle, int, int, cudaStream_t); \
  template void grp_info<T>(const GroupLaunch<T>&, int, cudaStream_t);
SISL_GROUP_INST(float)
SISL_GROUP_INST(double)
#undef SISL_GROUP_INST

template void gm_block_dots<float>(const float*, size_t, int, int, size_t, double*, GState*, cudaStream_t);
template void gm_block_dots<double>(const double*, size_t, int, int, size_t, double*, GState*, cudaStream_t);
template void gm_block_update<float>(float*, size_t, int, int, size_t, double*, GState*, cudaStream_t);
template void gm_block_update<double>(double*, size_t, int, int, size_t, double*, GState*, cudaStream_t);
template void gm_dots<float>(const float*, size_t, int, const float*, size_t, double*, GState*, int, int,
                             cudaStream_t);
template void gm_dots<double>(const double*, size_t, int, const double*, size_t, double*, GState*, int, int,
                              cudaStream_t);
template void gm_update<float>(const float*, size_t, int, float*, size_t, double, double*, GState*, int, int,
                               int, cudaStream_t);
template void gm_update<double>(const double*, size_t, int, double*, size_t, double, double*, GState*, int,
                                int, int, cudaStream_t);
template void gm_update_x64<float>(const float*, size_t, int, double*, size_t, const GState*, cudaStream_t);
template void gm_update_x64<double>(const double*, size_t, int, double*, size_t, const GState*, cudaStream_t);

}  // namespace sisl
