// Free-surface layers of the fast path: the three top interior layers of a
// stage (freeSurface.cpp:104-256), the PML slabs that reach them
// (pml_deriv.cpp:90-544, pml_freeSurface.cpp:65-337) and the RK combination
// (wave_rk.cpp:13-99, pml_rk.cpp:15-69), for every column of up to
// kSurfBatch scenarios in one launch.
//
// One block computes a 32 x 8 tile of columns of one layer.  It builds, once
// each, the J-weighted traction rows J (xi . T) along x and along y (with the
// one-sided stencils' halo of four) and the velocities of the layer in shared
// memory; the z rows, which no neighbour shares within a layer, and
// everything else a point needs are its thread's own loads.
//
// The layers are a few per cent of a large grid and were up to a third of the
// step on small ones, bound by the latency of chains of loads: a block that
// did three layers in turn had few blocks to fill the GPU, and the loads of
// m, t and the auxiliaries, each behind a store that might alias it, took one
// round trip per field.  Hence one layer per block, every load of a phase
// issued before its first store, and no second launch for the slab columns.
// Measured per stage against the two launches before (three layers per block,
// the exact-order kernel on the slab columns): 64x64x48 40-80 -> 13.5 us,
// 401x401x201 with a 20-cell PML 90-168 -> 61-72 us, 601x601x401 145-263 ->
// 125-149 us (FP32, cold cache).
// At 128 registers the single-scenario form has no spills; the form for several
// scenarios spills (a 72-byte frame, 144 bytes of stores and 72 of loads a
// thread).
// FP32 arithmetic with FMA contraction, equal to the reference up to rounding.
#include <algorithm>

#include "device_common.cuh"
#include "kernels.h"

namespace cgfdm {
namespace {

constexpr int TTX = 32, TTY = 8;  // tile of columns
constexpr int HX = TTX + 4, HY = TTY + 4;
constexpr int NT = TTX * TTY;

// J-weighted traction row of direction dir at q (freeSurface.cpp:128-153).
template <typename S>
__device__ __forceinline__ void jt3(const S *W, const S *cjm, long long fs, long long q, int dir,
                                    float r[3]) {
  const float m0 = ldv(cjm + q + fs * (3 * dir)), m1 = ldv(cjm + q + fs * (3 * dir + 1)),
              m2 = ldv(cjm + q + fs * (3 * dir + 2)), J = ldv(cjm + q + fs * 9);
  const float txx = ldv(W + q + fs * 3), tyy = ldv(W + q + fs * 4), tzz = ldv(W + q + fs * 5);
  const float txy = ldv(W + q + fs * 6), txz = ldv(W + q + fs * 7), tyz = ldv(W + q + fs * 8);
  r[0] = (m0 * txx + m1 * txy + m2 * txz) * J;
  r[1] = (m0 * txy + m1 * tyy + m2 * tyz) * J;
  r[2] = (m0 * txz + m1 * tyz + m2 * tzz) * J;
}

// One-sided 5-point MacCormack sum at p along stride st (already times the
// sign), without the sign and 1/DH.
template <typename T> __device__ __forceinline__ float lsum(const T *p, long long st) {
  return kAm1 * ldv(p - st) + kA0 * ldv(p) + kA1 * ldv(p + st) + kA2 * ldv(p + 2 * st) +
         kA3 * ldv(p + 3 * st);
}

// Stress rows of one direction from its velocity derivatives, added to out.
__device__ __forceinline__ void add_stress(const float m[3], const float dv[3], float mu, float lam,
                                           float out[6]) {
  const float x = m[0] * dv[0], y = m[1] * dv[1], z = m[2] * dv[2];
  const float div = (x + y + z) * lam;
  out[0] += div + 2.0f * mu * x;
  out[1] += div + 2.0f * mu * y;
  out[2] += div + 2.0f * mu * z;
  out[3] += (m[1] * dv[0] + m[0] * dv[1]) * mu;
  out[4] += (m[2] * dv[0] + m[0] * dv[2]) * mu;
  out[5] += (m[2] * dv[1] + m[1] * dv[2]) * mu;
}

struct SurfTile {
  float jx[3][TTY][HX];  // [component][row][column with the x halo]
  float jy[3][HY][TTX];  // [component][row with the y halo][column]
  float v[3][HY][HX];    // [velocity][row][column], x and y halo
};

// Weight and sign-free operand order of the RK combination: see
// StageArgs::lean.  b: what the output adds h to; t: what t adds h to.
struct RkForm {
  float ct, co;
  bool store_t, of_stages, t_from_acc, b_from_acc, b_is_in;
};
__device__ __forceinline__ RkForm rk_form(int irk, int lean) {
  RkForm f;
  f.ct = irk == 0 ? kB1 : irk == 1 ? kB2 : kB3;
  f.co = irk == 0 ? kA2rk : irk == 1 ? kA3rk : irk == 2 ? 1.0f : kB4;
  f.store_t = irk == 3 ? false : lean ? irk == 2 : true;
  f.of_stages = lean && irk == 2;
  f.t_from_acc = !lean && (irk == 1 || irk == 2);
  f.b_from_acc = irk == 3;
  f.b_is_in = irk == 0;
  return f;
}
// New (out, t) of one value; in: stage input, base: m (t in stage 3), acc: t
// or, with of_stages, stage 1's input.
__device__ __forceinline__ void rk_apply(const RkForm &f, float in, float base, float acc, float h,
                                         float &out, float &t) {
  out = base + f.co * h;
  t = f.of_stages ? base + (kT1 * (acc - base) + (kT2 * (in - base) + f.ct * h))
                  : (f.t_from_acc ? acc : base) + f.ct * h;
}

template <typename S> struct OneSurf {
  StageArgs<S> a;
  __device__ __forceinline__ const StageArgs<S> &of(int &) const { return a; }
};
template <typename S> struct ManySurf {
  StageArgs<S> a[kSurfBatch];
  int end[kSurfBatch];  // blocks of scenarios 0..e together
  int n;
  __device__ __forceinline__ const StageArgs<S> &of(int &block) const {
    int e = 0;
    while (e + 1 < n && block >= end[e]) ++e;
    if (e) block -= end[e - 1];
    return a[e];
  }
};

template <typename S, typename Src>
__global__ void __launch_bounds__(NT, 2) stage_surface_kernel(const __grid_constant__ Src src) {
  __shared__ SurfTile sm;
  int block = blockIdx.x;
  const StageArgs<S> &a = src.of(block);
  const Layout L = a.L;
  const long long fs = L.fs;
  const int ntx = (L.nx_ - 2 * HALO + TTX - 1) / TTX, nty = (L.ny_ - 2 * HALO + TTY - 1) / TTY;
  const int l = block / (ntx * nty), tile = block % (ntx * nty);
  const int ktop = L.nz_ - HALO - 1, k = ktop - 2 + l;
  const int ix = HALO + TTX * (tile % ntx), jy = HALO + TTY * (tile / ntx);
  const int tid = threadIdx.x, tx = tid % TTX, ty = tid / TTX;
  const int fb1 = a.fb1, fb2 = a.fb2, fb3 = a.fb3;
  const int bx0 = fb1 > 0 ? 1 : 3, by0 = fb2 > 0 ? 1 : 3;  // halo before the tile
  const S *__restrict__ W = a.win, *__restrict__ cjm = a.cjm;

  // (1) the shared rows; entries outside the padded grid stay unused
#pragma unroll
  for (int g = 0; g < (TTY * HX + NT - 1) / NT; ++g) {
    const int e = tid + g * NT, r = e / HX, c = e % HX;
    const int gi = ix - bx0 + c, gj = jy + r;
    if (e < TTY * HX && gi < L.nx_ && gj < L.ny_) {
      float t[3];
      jt3(W, cjm, fs, L.at(gi, gj, k), 0, t);
      sm.jx[0][r][c] = t[0]; sm.jx[1][r][c] = t[1]; sm.jx[2][r][c] = t[2];
    }
  }
#pragma unroll
  for (int g = 0; g < (HY * TTX + NT - 1) / NT; ++g) {
    const int e = tid + g * NT, r = e / TTX, c = e % TTX;
    const int gi = ix + c, gj = jy - by0 + r;
    if (e < HY * TTX && gi < L.nx_ && gj < L.ny_) {
      float t[3];
      jt3(W, cjm, fs, L.at(gi, gj, k), 1, t);
      sm.jy[0][r][c] = t[0]; sm.jy[1][r][c] = t[1]; sm.jy[2][r][c] = t[2];
    }
  }
#pragma unroll
  for (int g = 0; g < (HY * HX + NT - 1) / NT; ++g) {
    const int e = tid + g * NT, r = e / HX, c = e % HX;
    const int gi = ix - bx0 + c, gj = jy - by0 + r;
    if (e < HY * HX && gi < L.nx_ && gj < L.ny_) {
      const long long q = L.at(gi, gj, k);
      sm.v[0][r][c] = ldv(W + q);
      sm.v[1][r][c] = ldv(W + q + fs);
      sm.v[2][r][c] = ldv(W + q + 2 * fs);
    }
  }

  // (2) the thread's own loads
  const int i = ix + tx, j = jy + ty;
  const bool valid = i < L.nx_ - HALO && j < L.ny_ - HALO;
  const long long c = L.at(valid ? i : HALO, valid ? j : HALO, k);
  const RkForm f = rk_form(a.irk, a.lean);
  float m[3][3], J, mu, lam, bu, in[9], base[9], acc[9], lz[3] = {0.0f, 0.0f, 0.0f};
#pragma unroll
  for (int v = 0; v < 9; ++v) {
    in[v] = ldv(W + c + v * fs);
    base[v] = f.b_is_in ? in[v] : ldv((f.b_from_acc ? (const S *)a.t : a.wm) + c + v * fs);
    acc[v] = f.of_stages ? ldv((const S *)a.wout + c + v * fs)
             : f.t_from_acc ? ldv((const S *)a.t + c + v * fs) : 0.0f;
  }
#pragma unroll
  for (int d = 0; d < 3; ++d)
#pragma unroll
    for (int q = 0; q < 3; ++q) m[d][q] = ldv(cjm + c + fs * (3 * d + q));
  J = ldv(cjm + c + fs * 9);
  mu = ldv(cjm + c + fs * 10);
  lam = ldv(cjm + c + fs * 11);
  bu = ldv(cjm + c + fs * 12) * (float)CRHO_OF<S>::v;
  // z rows: zero at the surface (row ks of the point's seven), above it the
  // negated rows below (freeSurface.cpp:155-183)
  const int ks = 5 - l;
  {
    const float wt[5] = {kAm1, kA0, kA1, kA2, kA3};
#pragma unroll
    for (int q = 0; q < 5; ++q) {
      const int e = 3 + fb3 * (q - 1);
      if (e != ks) {
        const int p = e < ks ? e : 2 * ks - e;
        const float w = e < ks ? wt[q] : -wt[q];
        float t[3];
        jt3(W, cjm, fs, c + (long long)(p - 3) * L.plane, 2, t);
        lz[0] += w * t[0];
        lz[1] += w * t[1];
        lz[2] += w * t[2];
      }
    }
  }
  const float rDH = a.rDH, DT = a.DT;
  const float *px = a.pml, *py = a.pml + 3 * L.nx_, *pz = a.pml + 3 * L.nx_ + 3 * L.ny_;
  const int ic = valid ? i : HALO, jc = valid ? j : HALO;
  const float bx = px[L.nx_ + ic] * (fb1 * rDH), by = py[L.ny_ + jc] * (fb2 * rDH);
  const float gz = fb3 * rDH;
  const long long s2 = ic + (long long)jc * L.nx_;
  const float *DX = a.rdz + s2 * 9, *DY = a.rdz + (long long)L.nx_ * L.ny_ * 9 + s2 * 9;
  float vzt[3];
  if (l < 2) {  // 2- and 3-point operators (axis.h:92-93)
    const long long o = fb3 * L.plane;
#pragma unroll
    for (int v = 0; v < 3; ++v) {
      const float w1 = ldv(W + c + v * fs + o);
      vzt[v] = (l == 1 ? w1 - in[v]
                       : kCf1 * in[v] + kCf2 * w1 + kCf3 * ldv(W + c + v * fs + 2 * o)) * gz;
    }
  }
  __syncthreads();
  if (!valid) return;

  // (3) the increment
  float h[9];
#pragma unroll
  for (int q = 0; q < 3; ++q) {
    const float lx = lsum(&sm.jx[q][ty][tx + bx0], fb1);
    const float ly = lsum(&sm.jy[q][ty + by0][tx], fb2 * TTX);
    h[q] = bu / J * (lx * bx + ly * by + lz[q] * gz) * DT;
  }
  float vxi[3], vet[3];
#pragma unroll
  for (int v = 0; v < 3; ++v) {
    vxi[v] = lsum(&sm.v[v][ty + by0][tx + bx0], fb1) * bx;
    vet[v] = lsum(&sm.v[v][ty + by0][tx + bx0], fb2 * HX) * by;
  }
  if (l == 2) {
#pragma unroll
    for (int q = 0; q < 3; ++q)
      vzt[q] = (DX[3 * q] * vxi[0] + DX[3 * q + 1] * vxi[1] + DX[3 * q + 2] * vxi[2]) +
               (DY[3 * q] * vet[0] + DY[3 * q + 1] * vet[1] + DY[3 * q + 2] * vet[2]);
  }
  float st[6] = {0, 0, 0, 0, 0, 0};
  add_stress(m[0], vxi, mu, lam, st);
  add_stress(m[1], vet, mu, lam, st);
  add_stress(m[2], vzt, mu, lam, st);
#pragma unroll
  for (int v = 0; v < 6; ++v) h[3 + v] = st[v] * DT;

  // (4) the PML slabs of this point, in the order x, y, z; opposite slabs of
  // one axis do not overlap on the fast path
  if (a.nslab) {
    const int np = a.npml;
#pragma unroll 1
    for (int ax = 0; ax < 3; ++ax) {
      const int at = ax == 0 ? i : ax == 1 ? j : k;
      const int nax = ax == 0 ? L.nx_ : ax == 1 ? L.ny_ : L.nz_;
      const int s = at < HALO + np ? ax : ax < 2 && at >= nax - HALO - np ? ax + 3 : -1;
      if (s < 0) continue;
      const SlabDev<float> &sl = a.slab[s];
      const unsigned pos = (unsigned)((i - sl.off0) + (j - sl.off1) * sl.n0 +
                                      (k - sl.off2) * sl.n0 * sl.n1);
      const unsigned snp = (unsigned)sl.np;
      const int fa = ax == 0 ? fb1 : ax == 1 ? fb2 : fb3;
      const long long sa = (ax == 0 ? 1 : ax == 1 ? (long long)L.px : L.plane) * fa;
      const float *prof = ax == 0 ? px : ax == 1 ? py : pz;
      const float dd = prof[2 * nax + at], bt = prof[nax + at], ad = prof[at] + dd;
      const float g = dd * (fa * rDH);
      float av[9], ab[9], aa[9], d[9];
#pragma unroll
      for (int v = 0; v < 9; ++v) {
        const unsigned q = v * snp + pos;
        av[v] = sl.ain[q];
        ab[v] = f.b_is_in ? av[v] : f.b_from_acc ? sl.at[q] : sl.am[q];
        aa[v] = f.of_stages ? sl.aout[q] : f.t_from_acc ? sl.at[q] : 0.0f;
      }
#pragma unroll
      for (int v = 0; v < 9; ++v) d[v] = lsum(W + c + v * fs, sa) * g;
      float ma[3], ha[9];
#pragma unroll
      for (int q = 0; q < 3; ++q) ma[q] = ax == 0 ? m[0][q] : ax == 1 ? m[1][q] : m[2][q];
      ha[0] = (ma[0] * d[3] + ma[1] * d[6] + ma[2] * d[7]) * bu;
      ha[1] = (ma[0] * d[6] + ma[1] * d[4] + ma[2] * d[8]) * bu;
      ha[2] = (ma[0] * d[7] + ma[1] * d[8] + ma[2] * d[5]) * bu;
      float sa6[6] = {0, 0, 0, 0, 0, 0};
      add_stress(ma, d, mu, lam, sa6);
      if (l == 2 && ax != 2) {  // surface-gradient part of the stress auxiliaries
        const float *M = ax == 0 ? DX : DY;
        float vz[3];
#pragma unroll
        for (int q = 0; q < 3; ++q) vz[q] = M[3 * q] * d[0] + M[3 * q + 1] * d[1] + M[3 * q + 2] * d[2];
        add_stress(m[2], vz, mu, lam, sa6);
      }
#pragma unroll
      for (int v = 0; v < 6; ++v) ha[3 + v] = sa6[v];
#pragma unroll
      for (int v = 0; v < 9; ++v) {
        const unsigned q = v * snp + pos;
        h[v] -= bt * av[v] * DT;
        float out, t;
        rk_apply(f, av[v], ab[v], aa[v], (ha[v] - ad * av[v]) * DT, out, t);
        if (f.store_t) sl.at[q] = t;
        sl.aout[q] = out;
      }
    }
  }

  // (5) the RK combination
#pragma unroll
  for (int v = 0; v < 9; ++v) {
    float out, t;
    rk_apply(f, in[v], base[v], acc[v], h[v], out, t);
    if (f.store_t) stv(a.t + c + v * fs, t);
    stv(a.wout + c + v * fs, out);
  }
}

template <typename S> int surface_blocks(const StageArgs<S> &a) {
  return 3 * ((a.L.nx_ - 2 * HALO + TTX - 1) / TTX) * ((a.L.ny_ - 2 * HALO + TTY - 1) / TTY);
}

}  // namespace

template <typename S>
cudaError_t launch_stage_surface(const StageArgs<S> *args, int n, cudaStream_t st, int *nlaunch) {
  static_assert(sizeof(ManySurf<S>) <= 32000, "kernel parameter space");
  for (int e0 = 0; e0 < n; e0 += kSurfBatch) {
    const int ne = std::min(kSurfBatch, n - e0);
    if (ne == 1) {
      const OneSurf<S> one{args[e0]};
      stage_surface_kernel<S, OneSurf<S>><<<surface_blocks(one.a), NT, 0, st>>>(one);
    } else {
      static thread_local ManySurf<S> many;
      many.n = ne;
      int total = 0;
      for (int e = 0; e < ne; ++e) {
        many.a[e] = args[e0 + e];
        many.end[e] = total += surface_blocks(args[e0 + e]);
      }
      stage_surface_kernel<S, ManySurf<S>><<<total, NT, 0, st>>>(many);
    }
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return e;
    if (nlaunch) ++*nlaunch;
  }
  return cudaSuccess;
}

template cudaError_t launch_stage_surface<float>(const StageArgs<float> *, int, cudaStream_t, int *);
template cudaError_t launch_stage_surface<__half>(const StageArgs<__half> *, int, cudaStream_t, int *);
template cudaError_t launch_stage_surface<__nv_bfloat16>(const StageArgs<__nv_bfloat16> *, int,
                                                         cudaStream_t, int *);

}  // namespace cgfdm
