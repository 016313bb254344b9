// Split-explicit RK3 core (SplitExplicitStepper3D, steppers.py:1076-1737).
//
// One RK3 stage is: the explicit tendencies of the stage state (the explicit
// kernel, mode 1) plus the 3rd-order upwind flux advection of th', u_m,
// v_m, w_m (split_adv_kernel) averaged to the staggers (split_slow_kernel);
// then n acoustic sub-steps of three kernels: the horizontal predictor to
// the midpoint (split_predict_kernel), the vertically implicit pi''/w''
// column solve (split_column_tile_kernel, Thomas in the float arithmetic of
// the tridiagonal solve; split_column_kernel, one thread per column, past its
// shared memory), and the centred corrector with the backward w damping
// (split_correct_kernel); split_end_kernel assembles the stage state and
// split_diag_kernel diagnoses eta_dot and the kinematic w boundaries.
#include "sisl_explicit_dev.cuh"
#include "sisl_split.cuh"

namespace sisl {
namespace {

using dev::Grad;
using dev::Winds;

dim3 box(int ex, int ey, int ez, dim3 blk) {
  return dim3((ex + blk.x - 1) / blk.x, (ey + blk.y - 1) / blk.y, (ez + blk.z - 1) / blk.z);
}

// m_w (u_w z_xi_w + v_w z_eta_w) at w level k of column (i, j)  (steppers.py:1296-1300)
template <typename T>
__device__ __forceinline__ T kinematic(const Dims& d, const Coef<T>& c, const Winds<T>& W, int i, int j, int k) {
  const int p = iw(d, i, j, k);
  return ld(c.mm, h_m(d, i, j)) * (W.uw(i, j, k) * ld(c.zxw, p) + W.vw(i, j, k) * ld(c.zew, p));
}

template <typename T>
__global__ void split_diag_kernel(Dims d, Coef<T> c, const T* __restrict__ u, const T* __restrict__ v,
                                  const T* w_in, T* eta_out, T* w_out) {
  grid_chain();
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  const int j = blockIdx.y * blockDim.y + threadIdx.y;
  const int k = blockIdx.z * blockDim.z + threadIdx.z;
  if (i >= d.nx || j >= d.ny || k > d.nz) return;
  const Winds<T> W{d, c, u, v};
  const int p = iw(d, i, j, k);
  if (k == 0) {
    w_out[p] = kinematic(d, c, W, i, j, 0);  // flow glides over the slope
    eta_out[p] = T(0);
  } else if (k == d.nz) {
    w_out[p] = T(0);
    eta_out[p] = T(0);
  } else {
    const T wv = w_in[p];
    w_out[p] = wv;
    eta_out[p] = (wv - kinematic(d, c, W, i, j, k)) / ld(c.dzw, p);
  }
}


// 3rd-order upwind-biased face value (steppers.py:1312-1360), sg the sign of the flux through the face
template <typename T>
__device__ __forceinline__ T upwind_value(T qm2, T qm1, T q0, T qp1, T sg) {
  const T q4 = T(7.0 / 12.0) * (q0 + qm1) - T(1.0 / 12.0) * (qp1 + qm2);
  const T qb = T(1.0 / 12.0) * ((qp1 - qm2) - T(3) * (q0 - qm1));
  return q4 + sg * qb;
}
template <typename T>
__device__ __forceinline__ T flux_sign(T F, T eps_l) {
  return fabs(F) < eps_l ? T(0) : (F > T(0) ? T(1) : (F < T(0) ? T(-1) : T(0)));
}

// the four advected fields at mass point (i, j, k): th', u_m, v_m, w_m
template <typename T>
struct AdvFields {
  const Dims& d;
  const T* __restrict__ u;
  const T* __restrict__ v;
  const T* __restrict__ w;
  const T* __restrict__ th;
  __device__ __forceinline__ T at(int f, int i, int j, int k) const {
    switch (f) {
      case 0: return ld(th, im(d, i, j, k));
      case 1: return T(0.5) * (ld(u, iu(d, i, j, k)) + ld(u, iu(d, i + 1, j, k)));
      case 2: return T(0.5) * (ld(v, iv(d, i, j, k)) + ld(v, iv(d, i, j + 1, k)));
      default: return T(0.5) * (ld(w, iw(d, i, j, k)) + ld(w, iw(d, i, j, k + 1)));
    }
  }
};

// Blocks of AX x AY columns walk `chunk` levels.  Per level the block forms
// the four fields' values at the (AX + 4) x (AY + 4) cells of its x and y
// stencils once in shared memory (indices wrapped or clamped as the point
// form wraps them; two buffers, one barrier a level); a thread keeps the
// five levels of its z stencil in registers and the face value below its cell
// from the level before.
//
// The flux-form difference less q times the velocity's divergence is taken as
// F1 (q1 - q) - F0 (q0 - q) of the two faces: the fluxes' signs and factors are
// formed once for the four fields, there is no division per field and axis,
// and the two large terms of the direct form no longer cancel.  Bound by the
// issue of arithmetic and shared loads: 256x256x64 float32 598 us a call with
// a block per level, every face twice and three divisions per field.
constexpr int AX = 32, AY = 8;

template <typename T>
__global__ void __launch_bounds__(AX * AY, sizeof(T) == 4 ? 3 : 2) split_adv_kernel(
    Dims d, Coef<T> c, const T* __restrict__ u, const T* __restrict__ v, const T* __restrict__ w,
    const T* __restrict__ eta, const T* __restrict__ th, T eps_l, PtrTable<T> out, int chunk) {
  grid_chain();
  __shared__ T Qt[2][4][AY + 4][AX + 4];
  const int i0 = blockIdx.x * AX, j0 = blockIdx.y * AY;
  const int tx = threadIdx.x, ty = threadIdx.y;
  const int nx = d.nx, ny = d.ny, nz = d.nz;
  const bool live = i0 + tx < nx && j0 + ty < ny;
  const int i = min(i0 + tx, nx - 1), j = min(j0 + ty, ny - 1);
  const int k0 = blockIdx.z * chunk, k1 = min(k0 + chunk, nz);
  const AdvFields<T> F{d, u, v, w, th};
  const int t = tx + AX * ty;
  constexpr int CELLS = (AX + 4) * (AY + 4), FILL = (CELLS + AX * AY - 1) / (AX * AY);
  int ci[FILL], cj[FILL];
#pragma unroll
  for (int n = 0; n < FILL; ++n) {
    const int q = t + n * AX * AY;
    ci[n] = wrap_or_clamp(i0 - 2 + q % (AX + 4), nx, d.px);
    cj[n] = wrap_or_clamp(j0 - 2 + q / (AX + 4), ny, d.py);
  }
  const T mm = ld(c.mm, h_m(d, i, j)), m2 = mm * mm;
  const T sx = mm / (T)d.dx, sy = mm / (T)d.dy;
  const T mu0 = ld(c.mu, h_u(d, i, j)), mu1 = ld(c.mu, h_u(d, i + 1, j));
  const T mv0 = ld(c.mv, h_v(d, i, j)), mv1 = ld(c.mv, h_v(d, i, j + 1));
  auto zat = [&](int f, int k) { return F.at(f, i, j, min(max(k, 0), nz - 1)); };
  T qz[4][5], gb[4];  // levels k - 2 .. k + 2; face value below the cell
  T W0 = ld(eta, iw(d, i, j, k0)) * ld(c.dzw, iw(d, i, j, k0));
  {
    const T sg = flux_sign(W0, eps_l);
#pragma unroll
    for (int f = 0; f < 4; ++f) {
#pragma unroll
      for (int o = 0; o < 4; ++o) qz[f][o + 1] = zat(f, k0 - 2 + o);
      gb[f] = upwind_value(qz[f][1], qz[f][2], qz[f][3], qz[f][4], sg);
    }
  }
#pragma unroll 1
  for (int k = k0, s = 0; k < k1; ++k, s ^= 1) {
#pragma unroll
    for (int n = 0; n < FILL; ++n) {
      const int q = t + n * AX * AY;
      if (q < CELLS) {
#pragma unroll
        for (int f = 0; f < 4; ++f) (&Qt[s][f][0][0])[q] = F.at(f, ci[n], cj[n], k);
      }
    }
    const T U0 = ld(u, iu(d, i, j, k)) / mu0, U1 = ld(u, iu(d, i + 1, j, k)) / mu1;
    const T V0 = ld(v, iv(d, i, j, k)) / mv0, V1 = ld(v, iv(d, i, j + 1, k)) / mv1;
    const T W1 = ld(eta, iw(d, i, j, k + 1)) * ld(c.dzw, iw(d, i, j, k + 1));
    const T sz = T(1) / ld(c.dzm, im(d, i, j, k));
#pragma unroll
    for (int f = 0; f < 4; ++f) {
#pragma unroll
      for (int o = 0; o < 4; ++o) qz[f][o] = qz[f][o + 1];
      qz[f][4] = zat(f, k + 2);
    }
    const T su0 = flux_sign(U0, eps_l), su1 = flux_sign(U1, eps_l), sv0 = flux_sign(V0, eps_l),
            sv1 = flux_sign(V1, eps_l), sw1 = flux_sign(W1, eps_l);
    __syncthreads();  // the other buffer was last read before the previous level's barrier
#pragma unroll
    for (int f = 0; f < 4; ++f) {
      T qx[5], qy[5];
#pragma unroll
      for (int o = 0; o < 5; ++o) {
        qx[o] = Qt[s][f][ty + 2][tx + o];
        qy[o] = Qt[s][f][ty + o][tx + 2];
      }
      const T q = qz[f][2];
      const T ax = U1 * (upwind_value(qx[1], qx[2], qx[3], qx[4], su1) - q) -
                   U0 * (upwind_value(qx[0], qx[1], qx[2], qx[3], su0) - q);
      const T ay = V1 * (upwind_value(qy[1], qy[2], qy[3], qy[4], sv1) - q) -
                   V0 * (upwind_value(qy[0], qy[1], qy[2], qy[3], sv0) - q);
      const T gt = upwind_value(qz[f][1], qz[f][2], qz[f][3], qz[f][4], sw1);
      const T az = W1 * (gt - q) - W0 * (gb[f] - q);
      gb[f] = gt;
      if (live) out.p[f][im(d, i, j, k)] = -m2 * (ax * sx + ay * sy) - az * sz;
    }
    W0 = W1;
  }
}

// slow forcings: tend6 = {tend_u, tend_v, tend_w, tend_pi, tend_th, nl_pi};
// adv4 at mass points averaged to the u faces, v faces and w levels
template <typename T>
__global__ void split_slow_kernel(Dims d, PtrTable<T> t, PtrTable<T> sf) {
  grid_chain();
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  const int j = blockIdx.y * blockDim.y + threadIdx.y;
  const int k = blockIdx.z * blockDim.z + threadIdx.z;
  const int nx = d.nx, ny = d.ny, nz = d.nz;
  if (i > nx || j > ny || k > nz) return;
  // t.p[0..5]: explicit tendencies; t.p[6..9]: advection of th', u_m, v_m, w_m
  if (j < ny && k < nz) {
    int l, r;
    face_pair(i, nx, d.px, l, r);
    const int p = iu(d, i, j, k);
    sf.p[0][p] = t.p[0][p] + T(0.5) * (t.p[7][im(d, l, j, k)] + t.p[7][im(d, r, j, k)]);
  }
  if (i < nx && k < nz) {
    int l, r;
    face_pair(j, ny, d.py, l, r);
    const int p = iv(d, i, j, k);
    sf.p[1][p] = t.p[1][p] + T(0.5) * (t.p[8][im(d, i, l, k)] + t.p[8][im(d, i, r, k)]);
  }
  if (i < nx && j < ny) {
    int l, r;
    level_pair(k, nz, l, r);
    const int p = iw(d, i, j, k);
    sf.p[2][p] = t.p[2][p] + T(0.5) * (t.p[9][im(d, i, j, l)] + t.p[9][im(d, i, j, r)]);
    if (k < nz) {
      const int q = im(d, i, j, k);
      sf.p[3][q] = t.p[3][q] + t.p[5][q];
      sf.p[4][q] = t.p[4][q] + t.p[6][q];
    }
  }
}

template <typename T>
__global__ void split_init_kernel(Dims d, SplitArgs<T> a) {
  grid_chain();
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  const int j = blockIdx.y * blockDim.y + threadIdx.y;
  const int k = blockIdx.z * blockDim.z + threadIdx.z;
  const int nx = d.nx, ny = d.ny, nz = d.nz;
  if (i > nx || j > ny || k > nz) return;
  if (j < ny && k < nz) {
    const int p = iu(d, i, j, k);
    a.upp[p] = a.u0[p] - a.uc[p];
  }
  if (i < nx && k < nz) {
    const int p = iv(d, i, j, k);
    a.vpp[p] = a.v0[p] - a.vc[p];
  }
  if (i < nx && j < ny) {
    const int p = iw(d, i, j, k);
    a.wpp[p] = a.w0[p] - a.wc[p];
    if (k < nz) a.ppp[p] = a.p0[p] - a.pc[p];
  }
}

// Blocks of the predictor and corrector: SX x SY faces of one level.
constexpr int SX = 32, SY = 8;

// What the faces (i, j) of a block read of the cells (i0 - 1 + x, j0 - 1 + y),
// x <= SX, y <= SY, formed once per cell: the horizontal divergence of the
// total winds (stage + perturbation), pi'' and its vertical derivative at the
// mass level (Grad::gzm).  Cell indices beyond the grid wrap on a periodic
// axis and are clamped on an open one, so every interior face (i, j) of
// the block finds the two cells of its gradients at tile columns i - i0,
// i - i0 + 1 (rows j - j0, j - j0 + 1), as face_pair gives them, and the
// periodic duplicate face n its wrapped pair; the open boundary faces take no
// gradient (steppers.py:1528-1538).
template <typename T>
struct FaceTile {
  T div[SY + 1][SX + 1], p[SY + 1][SX + 1], gz[SY + 1][SX + 1];
};
// 1/dx and the map factor in one product, rounded once
template <typename T>
__device__ __forceinline__ T over(T m, double inv) {
  return (T)((double)m * inv);
}

template <typename T>
__device__ __forceinline__ void fill_tile(const Dims& d, const Coef<T>& c, const T* __restrict__ uc,
                                          const T* __restrict__ up, const T* __restrict__ vc,
                                          const T* __restrict__ vp, const T* __restrict__ pp, bool grad, int i0, int j0,
                                          int k, FaceTile<T>& t) {
  const int nx = d.nx, ny = d.ny, nz = d.nz, pm = nx * ny;
  const int kl = k > 0 ? k - 1 : 0, kh = k + 1 < nz ? k + 1 : nz - 1;
  for (int q = threadIdx.x + SX * threadIdx.y; q < (SX + 1) * (SY + 1); q += SX * SY) {
    const int x = q % (SX + 1), y = q / (SX + 1);
    const int ci = wrap_or_clamp(i0 - 1 + x, nx, d.px), cj = wrap_or_clamp(j0 - 1 + y, ny, d.py);
    const int u0 = iu(d, ci, cj, k), v0 = iv(d, ci, cj, k), h = ci + nx * cj;
    const T ca = ld(uc, u0), cb = ld(uc, u0 + 1), ua = ld(up, u0), ub = ld(up, u0 + 1);
    const T da = ld(vc, v0), db = ld(vc, v0 + nx), va = ld(vp, v0), vb = ld(vp, v0 + nx);
    const T mm = ld(c.mm, h);
    if (grad) {
      const T P0 = ld(pp, h + k * pm), Pl = ld(pp, h + kl * pm), Ph = ld(pp, h + kh * pm);
      const T z0 = ld(c.idzw, h + k * pm), z1 = ld(c.idzw, h + (k + 1) * pm);
      t.p[y][x] = P0;
      t.gz[y][x] = T(0.5) * ((k == 0 ? Ph - P0 : P0 - Pl) * z0 + (k + 1 == nz ? P0 - Pl : Ph - P0) * z1);
    }
    t.div[y][x] = ((cb + ub) - (ca + ua)) * over(mm, d.rdx) + ((db + vb) - (da + va)) * over(mm, d.rdy);
  }
}

// PART 1 of the acoustic sub-step (steppers.py:1561-1579): u'' and v'' to
// the midpoint; the boundary faces take the step-start winds (open) or the
// first face (periodic duplicate).  The pressure gradient of the old pi''
// is formed here on the first sub-step of a stage and taken from the
// previous corrector (gx0_ready) on the others.
//
// Predictor and corrector are bound by the issue of their loads; the cell
// tile took two gradients' 28 loads per point to 6.  256x256x64 float32, us:
// predictor 76 -> 74 (gradient ready), corrector 116 -> 90 (walking four levels
// a block, for hoisted indices, costs more in barriers: 80 and 130).
template <typename T>
__global__ void __launch_bounds__(SX * SY) split_predict_kernel(Dims d, Coef<T> c, SplitArgs<T> a) {
  grid_chain();
  __shared__ FaceTile<T> t;
  const int i0 = blockIdx.x * SX, j0 = blockIdx.y * SY, k = blockIdx.z;
  const int tx = threadIdx.x, ty = threadIdx.y;
  const int i = i0 + tx, j = j0 + ty;
  const int nx = d.nx, ny = d.ny;
  const bool ready = a.gx0_ready;
  fill_tile<T>(d, c, a.uc, a.upp, a.vc, a.vpp, a.ppp, !ready, i0, j0, k, t);
  __syncthreads();
  if (i > nx || j > ny) return;
  const T cp = (T)c.s.cp, hdt = T(0.5) * a.dtau;
  const T idx = (T)d.rdx, idy = (T)d.rdy;
  if (j < ny) {
    const int p = iu(d, i, j, k);
    const int ie = (d.px && i == nx) ? 0 : i, pe = iu(d, ie, j, k);
    if (!d.px && (i == 0 || i == nx)) {
      a.uh[p] = ld(a.u0, p) - ld(a.uc, p);
    } else {
      const T mu = ld(c.mu, h_u(d, ie, j)), th = ld(c.thu, pe), sf = ld(a.sfu, pe), old = ld(a.upp, pe);
      T g0;
      if (ready) {
        g0 = ld(a.gx0, p);
      } else {
        const T g = (t.p[ty + 1][tx + 1] - t.p[ty + 1][tx]) * idx * mu;
        g0 = g - ld(c.zxu, pe) * T(0.5) * (t.gz[ty + 1][tx] + t.gz[ty + 1][tx + 1]);
        a.gx0[p] = g0;
      }
      const T dgx = (t.div[ty + 1][tx + 1] - t.div[ty + 1][tx]) * over(mu, d.rdx);
      const T rhs = sf - cp * th * g0 + a.nu_div * dgx;
      a.uh[p] = old + hdt * rhs;
    }
  }
  if (i < nx) {
    const int p = iv(d, i, j, k);
    const int je = (d.py && j == ny) ? 0 : j, pe = iv(d, i, je, k);
    if (!d.py && (j == 0 || j == ny)) {
      a.vh[p] = ld(a.v0, p) - ld(a.vc, p);
    } else {
      const T mv = ld(c.mv, h_v(d, i, je)), th = ld(c.thv, pe), sf = ld(a.sfv, pe), old = ld(a.vpp, pe);
      T g0;
      if (ready) {
        g0 = ld(a.gy0, p);
      } else {
        const T g = (t.p[ty + 1][tx + 1] - t.p[ty][tx + 1]) * idy * mv;
        g0 = g - ld(c.zev, pe) * T(0.5) * (t.gz[ty][tx + 1] + t.gz[ty + 1][tx + 1]);
        a.gy0[p] = g0;
      }
      const T dgy = (t.div[ty + 1][tx + 1] - t.div[ty][tx + 1]) * over(mv, d.rdy);
      const T rhs = sf - cp * th * g0 + a.nu_div * dgy;
      a.vh[p] = old + hdt * rhs;
    }
  }
}

// PART 2 (steppers.py:1584-1605, 1635-1737): the vertically implicit
// acoustic column.  Upward: the explicit w'' (kept in place for the
// correction), the off-centred eta_dot flux, the explicit pi'' increment
// and the forward sweep of the tridiagonal solve for delta pi; downward:
// the back substitution, pi'' += delta pi and the w'' correction by the
// gradient of delta pi.  One thread per column; cpr/dpr hold the sweep.
template <typename T>
__global__ void __launch_bounds__(128) split_column_kernel(Dims d, Coef<T> c, SplitArgs<T> a, T a2cp, T adcp) {
  grid_chain();
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  const int j = blockIdx.y;
  const int nx = d.nx, ny = d.ny, nz = d.nz;
  if (i >= nx || j >= ny) return;
  const T al = a.alpha, dtau = a.dtau, cp = (T)c.s.cp;
  const Winds<T> W{d, c, a.uh, a.vh};
  const Grad<T> G{d, c, a.ppp};
  const T mm = ld(c.mm, h_m(d, i, j));
  const T dx = (T)d.dx, dy = (T)d.dy;
  const T wsfc = kinematic(d, c, W, i, j, 0);
  T fz_lo = T(0), gam_lo = T(0), cprev = T(0), dprev = T(0);
#pragma unroll 4
  for (int k = 0; k < nz; ++k) {
    T fz_hi = T(0), gam_hi = T(0);
    if (k + 1 < nz) {
      const int pw = iw(d, i, j, k + 1);
      const T thw = ld(c.thw, pw), rw = ld(c.rhow, pw);
      const T wold = a.wpp[pw];
      const T wex = wold + dtau * (a.sfw[pw] - cp * thw * G.gzw(i, j, k + 1));
      const T wav = (T(1) - al) * wold + al * wex;
      fz_hi = (wav - kinematic(d, c, W, i, j, k + 1)) * rw * thw;
      gam_hi = a2cp * thw * rw * thw / ld(c.dzw, pw);
      a.wpp[pw] = wex;
    }
    const int p = im(d, i, j, k);
    const T dzm = ld(c.dzm, p), cpidz = ld(c.cpidz, p);
    const int u0 = iu(d, i, j, k), v0 = iv(d, i, j, k);
    const T fx0 = a.uh[u0] * ld(c.rdu, u0) * ld(c.thu, u0);
    const T fx1 = a.uh[u0 + 1] * ld(c.rdu, u0 + 1) * ld(c.thu, u0 + 1);
    const T fy0 = a.vh[v0] * ld(c.rdv, v0) * ld(c.thv, v0);
    const T fy1 = a.vh[v0 + nx] * ld(c.rdv, v0 + nx) * ld(c.thv, v0 + nx);
    const T div_h = mm * ((fx1 - fx0) / dx * mm / dzm + (fy1 - fy0) / dy * mm / dzm);
    const T div_z = (fz_hi - fz_lo) / dzm;
    const T rhs = dtau * (a.sfp[p] - cpidz * dzm * (div_h + div_z));
    const T lower = -cpidz * gam_lo, upper = -cpidz * gam_hi;
    const T mainv = T(1) - lower - upper;
    T cpk, dpk;
    if (k == 0) {
      const T inv = T(1) / mainv;
      cpk = upper * inv;
      dpk = rhs * inv;
    } else {
      const T inv = T(1) / (mainv - lower * cprev);
      cpk = upper * inv;
      dpk = (rhs - lower * dprev) * inv;
    }
    a.cpr[p] = cpk;
    a.dpr[p] = dpk;
    cprev = cpk;
    dprev = dpk;
    fz_lo = fz_hi;
    gam_lo = gam_hi;
  }
  T xh = dprev;
  {
    const int p = im(d, i, j, nz - 1);
    a.ppp[p] = a.ppp[p] + xh;
  }
#pragma unroll 4
  for (int k = nz - 2; k >= 0; --k) {
    const int p = im(d, i, j, k);
    const T x = a.dpr[p] - a.cpr[p] * xh;
    const int pw = iw(d, i, j, k + 1);
    a.wpp[pw] = a.wpp[pw] - adcp * ld(c.thw, pw) * ((xh - x) * ld(c.idzw, pw));
    a.ppp[p] = a.ppp[p] + x;
    xh = x;
  }
  a.wpp[iw(d, i, j, 0)] = wsfc;
  a.wpp[iw(d, i, j, nz)] = T(0);
}

// The same column solve on tiles of PC columns (one block per tile and
// row j) so that every thread works outside the recurrence, each phase's
// loads batched (PU items in flight per thread): A0 the horizontal flux
// divergence and the winds at the mass levels, A1 the w-level terms (explicit
// w'', the eta_dot flux, the coupling gamma), A2 the right-hand sides, B one
// warp runs the Thomas sweeps in shared memory, forming each row (lower,
// upper, main) from gamma and C_pi / dz_m, C the pi'' and w'' updates.  dz_m
// cancels between the divergence and C_pi / dz_m.  Shared memory: (6 nz + 2)
// PC values (c' overwrites the eta_dot fluxes once the right-hand sides are
// formed).  Bound by memory latency: 256x256x64 float32 157 us with a load
// at a time and six divisions a point, 116 here.
template <typename T, int PT, int PC>
__global__ void __launch_bounds__(PT, sizeof(T) == 4 ? 4 : 2) split_column_tile_kernel(Dims d, Coef<T> c,
                                                                                      SplitArgs<T> a, T a2cp,
                                                                                      T adcp) {
  grid_chain();
  extern __shared__ __align__(16) unsigned char smem_raw[];
  T* sm = reinterpret_cast<T*>(smem_raw);
  const int nx = d.nx, ny = d.ny, nz = d.nz, pm = nx * ny;
  T* s_fz = sm;                      // [nz+1][PC]  eta_dot flux -> c'
  T* s_gam = s_fz + (nz + 1) * PC;   // [nz+1][PC]  gamma
  T* s_x = s_gam + (nz + 1) * PC;    // [nz][PC]    flux divergence -> rhs -> d' -> delta pi
  T* s_cz = s_x + nz * PC;           // [nz][PC]    C_pi / dz_m
  T* s_um = s_cz + nz * PC;          // [nz][PC]    winds at mass levels
  T* s_vm = s_um + nz * PC;          // [nz][PC]
  const int j = blockIdx.y, tid = threadIdx.x;
  const int lane = tid % PC, kt = tid / PC;
  constexpr int KS = PT / PC;  // levels per pass of the block
  const int i = blockIdx.x * PC + lane, ic = min(i, nx - 1);
  const bool live = i < nx;
  const int h = ic + nx * j;
  const T al = a.alpha, dtau = a.dtau, cp = (T)c.s.cp;
  const T mm = ld(c.mm, h), m2x = over(mm * mm, d.rdx), m2y = over(mm * mm, d.rdy);
  {  // A0
    constexpr int PU = 2;
    const T* __restrict__ uh = a.uh;
    const T* __restrict__ vh = a.vh;
    for (int k0 = kt; k0 < nz; k0 += PU * KS) {
      T u0[PU], u1[PU], v0[PU], v1[PU], ru0[PU], ru1[PU], rv0[PU], rv1[PU], tu0[PU], tu1[PU], tv0[PU], tv1[PU], cz[PU];
#pragma unroll
      for (int n = 0; n < PU; ++n) {
        const int k = min(k0 + n * KS, nz - 1), pu = iu(d, ic, j, k), pv = iv(d, ic, j, k);
        u0[n] = ld(uh, pu);
        u1[n] = ld(uh, pu + 1);
        v0[n] = ld(vh, pv);
        v1[n] = ld(vh, pv + nx);
        ru0[n] = ld(c.rdu, pu);
        ru1[n] = ld(c.rdu, pu + 1);
        tu0[n] = ld(c.thu, pu);
        tu1[n] = ld(c.thu, pu + 1);
        rv0[n] = ld(c.rdv, pv);
        rv1[n] = ld(c.rdv, pv + nx);
        tv0[n] = ld(c.thv, pv);
        tv1[n] = ld(c.thv, pv + nx);
        cz[n] = ld(c.cpidz, h + k * pm);
      }
#pragma unroll
      for (int n = 0; n < PU; ++n) {
        const int k = k0 + n * KS;
        if (k >= nz) break;
        const int q = k * PC + lane;
        s_um[q] = T(0.5) * (u0[n] + u1[n]);
        s_vm[q] = T(0.5) * (v0[n] + v1[n]);
        s_x[q] = (u1[n] * ru1[n] * tu1[n] - u0[n] * ru0[n] * tu0[n]) * m2x +
                 (v1[n] * rv1[n] * tv1[n] - v0[n] * rv0[n] * tv0[n]) * m2y;
        s_cz[q] = live ? cz[n] : T(0);
      }
    }
  }
  __syncthreads();
  {  // A1
    constexpr int PU = 2;
    const T* __restrict__ pp = a.ppp;
    for (int k0 = kt; k0 <= nz; k0 += PU * KS) {
      T th[PU], rw[PU], wo[PU], sf[PU], iz[PU], dz[PU], zx[PU], ze[PU], pl[PU], ph[PU];
#pragma unroll
      for (int n = 0; n < PU; ++n) {
        const int k = min(k0 + n * KS, nz), pw = h + k * pm;  // an end level's own values: nobody writes them here
        th[n] = ld(c.thw, pw);
        rw[n] = ld(c.rhow, pw);
        wo[n] = a.wpp[pw];
        sf[n] = ld(a.sfw, pw);
        iz[n] = ld(c.idzw, pw);
        dz[n] = ld(c.dzw, pw);
        zx[n] = ld(c.zxw, pw);
        ze[n] = ld(c.zew, pw);
        pl[n] = ld(pp, h + max(k - 1, 0) * pm);
        ph[n] = ld(pp, h + min(k, nz - 1) * pm);
      }
#pragma unroll
      for (int n = 0; n < PU; ++n) {
        const int k = k0 + n * KS;
        if (k > nz) break;
        const int q = k * PC + lane;
        T fz = T(0), gam = T(0);
        if (live && k > 0 && k < nz) {
          const T wex = wo[n] + dtau * (sf[n] - cp * th[n] * ((ph[n] - pl[n]) * iz[n]));
          const T wav = (T(1) - al) * wo[n] + al * wex;
          const T kin = mm * (T(0.5) * (s_um[q - PC] + s_um[q]) * zx[n] + T(0.5) * (s_vm[q - PC] + s_vm[q]) * ze[n]);
          fz = (wav - kin) * rw[n] * th[n];
          gam = a2cp * th[n] * rw[n] * th[n] / dz[n];
          a.wpp[h + k * pm] = wex;
        }
        s_fz[q] = fz;
        s_gam[q] = gam;
      }
    }
  }
  __syncthreads();
#pragma unroll 4
  for (int k = kt; k < nz; k += KS) {  // A2; a column past the grid: a trivial row, lower = upper = 0, main = 1
    const int q = k * PC + lane;
    const T sp = ld(a.sfp, h + k * pm);
    s_x[q] = live ? dtau * (sp - s_cz[q] * (s_x[q] + (s_fz[q + PC] - s_fz[q]))) : T(0);
  }
  __syncthreads();
  if (tid < PC) {  // B
    T cprev = T(0), dprev = T(0);
    for (int k = 0; k < nz; ++k) {
      const int q = k * PC + tid;
      const T cpidz = s_cz[q];
      const T lower = -cpidz * s_gam[q], upper = -cpidz * s_gam[q + PC];
      const T mainv = T(1) - lower - upper;
      T cpk, dpk;
      if (k == 0) {
        const T inv = T(1) / mainv;
        cpk = upper * inv;
        dpk = s_x[q] * inv;
      } else {
        const T inv = T(1) / (mainv - lower * cprev);
        cpk = upper * inv;
        dpk = (s_x[q] - lower * dprev) * inv;
      }
      s_fz[q] = cpk;
      s_x[q] = dpk;
      cprev = cpk;
      dprev = dpk;
    }
    T xh = dprev;
    for (int k = nz - 2; k >= 0; --k) {
      const int q = k * PC + tid;
      xh = s_x[q] - s_fz[q] * xh;
      s_x[q] = xh;
    }
  }
  __syncthreads();
  if (!live) return;
  constexpr int PU = 4;
  for (int k0 = kt; k0 <= nz; k0 += PU * KS) {  // C
    T wx[PU], th[PU], iz[PU], po[PU];
#pragma unroll
    for (int n = 0; n < PU; ++n) {
      const int k = min(k0 + n * KS, nz), pw = h + k * pm;
      wx[n] = a.wpp[pw];
      th[n] = ld(c.thw, pw);
      iz[n] = ld(c.idzw, pw);
      po[n] = a.ppp[h + min(k, nz - 1) * pm];
    }
#pragma unroll
    for (int n = 0; n < PU; ++n) {
      const int k = k0 + n * KS;
      if (k > nz) break;
      const int pw = h + k * pm, q = k * PC + lane;
      if (k == 0) {  // the kinematic ground value: both levels of the padded pair
        const T uw = T(0.5) * (s_um[lane] + s_um[PC + lane]), vw = T(0.5) * (s_vm[lane] + s_vm[PC + lane]);
        a.wpp[pw] = mm * (uw * ld(c.zxw, pw) + vw * ld(c.zew, pw));
      } else if (k == nz) {
        a.wpp[pw] = T(0);
      } else {
        a.wpp[pw] = wx[n] - adcp * th[n] * ((s_x[q] - s_x[q - PC]) * iz[n]);
      }
      if (k < nz) a.ppp[pw] = po[n] + s_x[q];
    }
  }
}

// PART 3 (steppers.py:1607-1626): the centred corrector of u'', v'' into
// upp2/vpp2 (read u'' from upp/vpp), and the backward damping of w''.  The
// gradients of the new pi'' go to gx1/gy1 for the next predictor.
template <typename T>
__global__ void __launch_bounds__(SX * SY) split_correct_kernel(Dims d, Coef<T> c, SplitArgs<T> a,
                                                                T* __restrict__ upp2, T* __restrict__ vpp2) {
  grid_chain();
  __shared__ FaceTile<T> t;
  const int i0 = blockIdx.x * SX, j0 = blockIdx.y * SY, k = blockIdx.z;
  const int tx = threadIdx.x, ty = threadIdx.y;
  const int i = i0 + tx, j = j0 + ty;
  const int nx = d.nx, ny = d.ny, nz = d.nz;
  if (k < nz) fill_tile<T>(d, c, a.uc, a.uh, a.vc, a.vh, a.ppp, true, i0, j0, k, t);
  __syncthreads();
  if (i > nx || j > ny) return;
  const T cp = (T)c.s.cp, dtau = a.dtau;
  const T idx = (T)d.rdx, idy = (T)d.rdy;
  if (j < ny && k < nz) {
    const int p = iu(d, i, j, k);
    if (!d.px && (i == 0 || i == nx)) {
      upp2[p] = ld(a.u0, p) - ld(a.uc, p);
    } else {
      const int ie = (d.px && i == nx) ? 0 : i, pe = iu(d, ie, j, k);
      const T mu = ld(c.mu, h_u(d, ie, j)), zx = ld(c.zxu, pe), th = ld(c.thu, pe), sf = ld(a.sfu, pe), old = ld(a.upp, pe),
              g0 = ld(a.gx0, pe);
      const T g = (t.p[ty + 1][tx + 1] - t.p[ty + 1][tx]) * idx * mu;
      const T g1 = g - zx * T(0.5) * (t.gz[ty + 1][tx] + t.gz[ty + 1][tx + 1]);
      const T dgx = (t.div[ty + 1][tx + 1] - t.div[ty + 1][tx]) * over(mu, d.rdx);
      upp2[p] = old + dtau * (sf - T(0.5) * cp * th * (g0 + g1) + a.nu_div * dgx);
      if (a.gx1) a.gx1[p] = g1;
    }
  }
  if (i < nx && k < nz) {
    const int p = iv(d, i, j, k);
    if (!d.py && (j == 0 || j == ny)) {
      vpp2[p] = ld(a.v0, p) - ld(a.vc, p);
    } else {
      const int je = (d.py && j == ny) ? 0 : j, pe = iv(d, i, je, k);
      const T mv = ld(c.mv, h_v(d, i, je)), ze = ld(c.zev, pe), th = ld(c.thv, pe), sf = ld(a.sfv, pe), old = ld(a.vpp, pe),
              g0 = ld(a.gy0, pe);
      const T g = (t.p[ty + 1][tx + 1] - t.p[ty][tx + 1]) * idy * mv;
      const T g1 = g - ze * T(0.5) * (t.gz[ty][tx + 1] + t.gz[ty + 1][tx + 1]);
      const T dgy = (t.div[ty + 1][tx + 1] - t.div[ty][tx + 1]) * over(mv, d.rdy);
      vpp2[p] = old + dtau * (sf - T(0.5) * cp * th * (g0 + g1) + a.nu_div * dgy);
      if (a.gy1) a.gy1[p] = g1;
    }
  }
  if (i < nx && j < ny) {
    const int p = iw(d, i, j, k);
    const T wc = ld(a.wc, p);
    a.wpp[p] = (wc + a.wpp[p]) / (T(1) + dtau * ld(a.tau, p)) - wc;
  }
}

template <typename T>
__global__ void split_end_kernel(Dims d, SplitArgs<T> a, T dtns, T* u, T* v, T* w, T* eta, T* pp, T* th) {
  grid_chain();
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  const int j = blockIdx.y * blockDim.y + threadIdx.y;
  const int k = blockIdx.z * blockDim.z + threadIdx.z;
  const int nx = d.nx, ny = d.ny, nz = d.nz;
  if (i > nx || j > ny || k > nz) return;
  if (j < ny && k < nz) {
    const int p = iu(d, i, j, k);
    u[p] = a.uc[p] + a.upp[p];
  }
  if (i < nx && k < nz) {
    const int p = iv(d, i, j, k);
    v[p] = a.vc[p] + a.vpp[p];
  }
  if (i < nx && j < ny) {
    const int p = iw(d, i, j, k);
    w[p] = a.wc[p] + a.wpp[p];
    eta[p] = a.ec[p];
    if (k < nz) {
      pp[p] = a.pc[p] + a.ppp[p];
      th[p] = a.th0[p] + dtns * a.sfth[p];
    }
  }
}

template <typename T>
__global__ void split_axpy_kernel(size_t n, const T* __restrict__ b, T* a) {
  grid_chain();
  for (size_t q = blockIdx.x * (size_t)blockDim.x + threadIdx.x; q < n; q += (size_t)gridDim.x * blockDim.x)
    a[q] = a[q] + b[q];
}

}  // namespace

template <typename T>
void launch_split_diag(const Dims& d, const Coef<T>& c, const T* u, const T* v, const T* w_in, T* eta_out,
                       T* w_out, cudaStream_t st) {
  const dim3 blk(32, 4, 2);
  launch_chained(split_diag_kernel<T>, box(d.nx, d.ny, d.nz + 1, blk), blk, 0, st, d, c, u, v, w_in, eta_out, w_out);
}

template <typename T>
void launch_split_adv(const Dims& d, const Coef<T>& c, const T* u, const T* v, const T* w, const T* eta,
                      const T* th, T eps_l, T* const* adv4, cudaStream_t st) {
  const dim3 blk(AX, AY, 1);
  PtrTable<T> o{};
  for (int q = 0; q < 4; ++q) o.p[q] = adv4[q];
  // 16 levels a block where that leaves two blocks an SM, else 8: a chunk's start reads four levels more
  const int tiles = ((d.nx + AX - 1) / AX) * ((d.ny + AY - 1) / AY);
  const int chunk = tiles * ((d.nz + 15) / 16) >= 2 * 148 ? 16 : 8;
  launch_chained(split_adv_kernel<T>, dim3((d.nx + AX - 1) / AX, (d.ny + AY - 1) / AY, (d.nz + chunk - 1) / chunk),
                 blk, 0, st, d, c, u, v, w, eta, th, eps_l, o, chunk);
}

template <typename T>
void launch_split_slow(const Dims& d, const T* const* tend6, const T* const* adv4, T* const* sf5, cudaStream_t st) {
  const dim3 blk(32, 4, 2);
  PtrTable<T> t{}, s{};
  for (int q = 0; q < 6; ++q) t.p[q] = const_cast<T*>(tend6[q]);
  for (int q = 0; q < 4; ++q) t.p[6 + q] = const_cast<T*>(adv4[q]);
  for (int q = 0; q < 5; ++q) s.p[q] = sf5[q];
  launch_chained(split_slow_kernel<T>, box(d.nx + 1, d.ny + 1, d.nz + 1, blk), blk, 0, st, d, t, s);
}

template <typename T>
void launch_split_init(const Dims& d, const SplitArgs<T>& a, cudaStream_t st) {
  const dim3 blk(32, 4, 2);
  launch_chained(split_init_kernel<T>, box(d.nx + 1, d.ny + 1, d.nz + 1, blk), blk, 0, st, d, a);
}

template <typename T>
void launch_split_predict(const Dims& d, const Coef<T>& c, const SplitArgs<T>& a, cudaStream_t st) {
  const dim3 blk(SX, SY, 1);
  launch_chained(split_predict_kernel<T>, box(d.nx + 1, d.ny + 1, d.nz, blk), blk, 0, st, d, c, a);
}

template <typename T, int PC>
static void launch_column_tile(const Dims& d, const Coef<T>& c, const SplitArgs<T>& a, T a2cp, T adcp, size_t smem,
                               cudaStream_t st) {
  constexpr int PT = 256;
  static SmemLimit attr_bytes;  // per instantiation
  ensure_smem_limit((const void*)split_column_tile_kernel<T, PT, PC>, attr_bytes, smem);
  launch_chained(split_column_tile_kernel<T, PT, PC>, dim3((d.nx + PC - 1) / PC, d.ny), PT, smem, st, d, c, a, a2cp,
                 adcp);
}

template <typename T>
void launch_split_column(const Dims& d, const Coef<T>& c, const SplitArgs<T>& a, cudaStream_t st) {
  const double ad = (double)a.alpha * (double)a.dtau;
  const T a2cp = (T)(ad * ad * c.s.cp), adcp = (T)(ad * c.s.cp);
  const size_t level = (size_t)(6 * d.nz + 2) * sizeof(T);  // shared memory of a column
  if (32 * level <= 200 * 1024) {
    launch_column_tile<T, 32>(d, c, a, a2cp, adcp, 32 * level, st);
    return;
  }
  if (16 * level <= 200 * 1024) {  // many levels: half the columns; the one-thread-per-column march beyond
    launch_column_tile<T, 16>(d, c, a, a2cp, adcp, 16 * level, st);
    return;
  }
  launch_chained(split_column_kernel<T>, dim3((d.nx + 127) / 128, d.ny), 128, 0, st, d, c, a, a2cp, adcp);
}

template <typename T>
void launch_split_correct(const Dims& d, const Coef<T>& c, const SplitArgs<T>& a, T* upp2, T* vpp2,
                          cudaStream_t st) {
  const dim3 blk(SX, SY, 1);
  launch_chained(split_correct_kernel<T>, box(d.nx + 1, d.ny + 1, d.nz + 1, blk), blk, 0, st, d, c, a, upp2, vpp2);
}

template <typename T>
void launch_split_end(const Dims& d, const SplitArgs<T>& a, int nsteps, T* u, T* v, T* w, T* eta, T* p, T* th,
                      cudaStream_t st) {
  const dim3 blk(32, 4, 2);
  const T dtns = (T)((double)a.dtau * nsteps);
  launch_chained(split_end_kernel<T>, box(d.nx + 1, d.ny + 1, d.nz + 1, blk), blk, 0, st, d, a, dtns, u, v, w, eta,
                 p, th);
}

template <typename T>
void launch_split_axpy(size_t n, const T* b, T* a, cudaStream_t st) {
  launch_chained(split_axpy_kernel<T>, (unsigned)std::min<size_t>((n + 255) / 256, 148 * 16), 256, 0, st, n, b, a);
}

#define SISL_INST_SPLIT(T)                                                                                       \
  template void launch_split_diag<T>(const Dims&, const Coef<T>&, const T*, const T*, const T*, T*, T*,        \
                                     cudaStream_t);                                                           \
  template void launch_split_adv<T>(const Dims&, const Coef<T>&, const T*, const T*, const T*, const T*,       \
                                    const T*, T, T* const*, cudaStream_t);                                    \
  template void launch_split_slow<T>(const Dims&, const T* const*, const T* const*, T* const*, cudaStream_t); \
  template void launch_split_init<T>(const Dims&, const SplitArgs<T>&, cudaStream_t);                         \
  template void launch_split_predict<T>(const Dims&, const Coef<T>&, const SplitArgs<T>&, cudaStream_t);      \
  template void launch_split_column<T>(const Dims&, const Coef<T>&, const SplitArgs<T>&, cudaStream_t);       \
  template void launch_split_correct<T>(const Dims&, const Coef<T>&, const SplitArgs<T>&, T*, T*,             \
                                        cudaStream_t);                                                        \
  template void launch_split_end<T>(const Dims&, const SplitArgs<T>&, int, T*, T*, T*, T*, T*, T*,            \
                                    cudaStream_t);                                                            \
  template void launch_split_axpy<T>(size_t, const T*, T*, cudaStream_t);
SISL_INST_SPLIT(float)
SISL_INST_SPLIT(double)

}  // namespace sisl
