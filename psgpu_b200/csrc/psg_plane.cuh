// psg_plane.cuh -- passes B, C and D of a right-hand side in one kernel, for grids
// up to 64^3: a cluster of CS blocks takes one z plane from the y-inverse through
// the x rows and their products to the y-forward, the plane's rows and columns in
// shared memory.
//
// Bound: at these sizes a pass is a few microseconds of start-up, one tile copy
// and one transform, in a chain of dependent launches (3.9 us a pass at 32^3 FP32,
// 5.9 at 64^3 FP64, against well under 1 us of memory time), so fewer launches is
// the whole gain.  One block holds a plane up to 32^2; a 64^2 plane is split over
// two blocks (128 of the 148 SMs work instead of 64), which exchange lines
// through distributed shared memory as the 2D integrator does (psg_chip2d.cuh,
// whose layouts these are).  From 128^2 on a plane needs four or more blocks'
// shared memory and the passes are bound by bandwidth.
#pragma once
#include "psg_chip2d.cuh"

namespace psg {

template <int N>
struct PlaneShape {
  static constexpr int CS = N <= 32 ? 1 : 2;
  // 64^3: where it is the faster (us a step, passes / plane: FP64 RK4 118 / 104,
  // Boussinesq 143 / 138, FP32 Boussinesq 113 / 108); not for the six FP32
  // Navier-Stokes fields (90 / 96)
  static constexpr bool built(int nf, int elem) { return N <= 32 || (N == 64 && !(nf == 6 && elem == 4)); }
};
constexpr int kPlaneThreads = 384;

// NF as pass C's: 6 (Navier-Stokes), 9 (Boussinesq), 9 + kLinAdj, 12 + kLinTan
template <typename T, int N, int NF>
struct Plane {
  static constexpr int CS = PlaneShape<N>::CS, NI = NF % 100;
  static constexpr int NO = NF == 9 ? 4 : NF == 9 + kLinAdj ? 6 : 3;
  using FI = LineFFTM<N, +1, T>;
  using FO = LineFFTM<N, -1, T>;
  using FX = LineFFTM<N, -1, T, true>;  // consumes FI's output distribution
  static constexpr int G = FI::G, E = FI::E, GPW = 32 / G, EXW = FI::SMEM;
  static constexpr int K = Box<N>::K, X = Box<N>::X, Y = Box<N>::Y, XT = Box<N>::XT, W = kTileW;
  static constexpr int RPC = N / CS, CPC = (X + CS - 1) / CS;  // rows, columns of a block
  static constexpr int RP = RPC | 1, CP = CPC | 1;
  // WIDE: the rows' inverse transforms are dealt over all groups, the physical
  // fields meet in shared memory, and the forward transforms are dealt again, so
  // that a row's five to eight transforms are not one group's chain (32^3 FP32, with
  // a lane group per field in passes A and E: 72 -> 63 us a step; 79 with five
  // passes); a 64^2 plane has no room for the fields
  static constexpr bool WIDE = N <= 32;
  static constexpr int FS = N + 4;  // row stride of the physical fields
  static constexpr size_t smem(int nt) {
    return sizeof(cpx<T>) * (2 * N + (size_t)(nt / G) * EXW + NI * X * RP + NO * N * CP) +
           (WIDE ? sizeof(T) * NI * RPC * FS : 0);
  }
  static constexpr int lines() {
    const int a = NI * CPC, b = WIDE ? (NI + 1) / 2 * RPC : RPC;
    return a > b ? a : b;
  }

  cpx<T>*tw, *ex, *A, *B;
  T* F;  // WIDE: physical fields [NI][RPC][FS]
  int rank, gid, gi, ng, wg;

  __device__ __forceinline__ cpx<T>& row(int f, int y, int k) { return A[(f * X + k) * RP + y]; }
  __device__ __forceinline__ cpx<T>& col(int f, int y, int cl) { return B[(f * N + y) * CP + cl]; }
  static __device__ __forceinline__ constexpr bool dead(int e) {
    return FI::in_index(0, e) > K && FI::in_index(G - 1, e) < N - K;
  }

  // y-inverse of the block's columns
  __device__ __forceinline__ void phase1(const cpx<T>* __restrict__ in, int z, bool all) {
    for (int base = 0; base + wg < NI * CPC; base += ng) {
      // groups past the last line repeat it and store nothing
      const int l = min(base + gid, NI * CPC - 1), f = l / CPC, cl = l % CPC, ikx = rank * CPC + cl;
      const bool live = l == base + gid && ikx < X;
      const int kx = min(ikx, X - 1), xt = kx / W, ym = tile_reach_y<N>(all, xt);
      const cpx<T>* src = in + (((long)f * XT + xt) * N + z) * Y * W + kx % W;
      cpx<T> v[E];
#pragma unroll
      for (int e = 0; e < E; ++e) {
        const int iky = row_to_box(FI::in_index(gi, e), K, N);
        v[e] = (!dead(e) && iky >= K - ym && iky <= K + ym) ? src[iky * W] : czero<T>();
      }
      FI::run(v, gi, tw, ex, WarpSync());
      if (live) {
#pragma unroll
        for (int e = 0; e < E; ++e) {
          const int y = FI::out_index(gi, e);
          chip_store<CS>(&row(f, y % RPC, ikx), y / RPC, v[e]);
        }
      }
    }
  }

  // inverse transform of the real fields fa, fb (fb < 0: fa alone) of row y
  __device__ __forceinline__ void inverse(int fa, int fb, int y, T (&ra)[E], T (&rb)[E]) {
    cpx<T> v[E];
#pragma unroll
    for (int e = 0; e < E; ++e) {
      const int r = FI::in_index(gi, e);
      const bool lo = r <= K, hi = r >= N - K;
      const int k = lo ? r : hi ? N - r : 0;
      v[e] = czero<T>();
      if (dead(e)) continue;
      cpx<T> a = row(fa, y, k), b = fb >= 0 ? row(fb, y, k) : czero<T>();
      if (r == 0) a.y = b.y = (T)0;
      if (hi) { a.y = -a.y; b.y = -b.y; }
      if (lo || hi) v[e] = cpx<T>{a.x - b.y, a.y + b.x};
    }
    FI::run(v, gi, tw, ex, WarpSync());
#pragma unroll
    for (int e = 0; e < E; ++e) { ra[e] = v[e].x; rb[e] = v[e].y; }
  }
  // forward transform of p + i q (both halved) into outputs f, f + 1 of row y, or
  // of p alone into f
  __device__ __forceinline__ void forward_line(const T (&p)[E], const T (&q)[E], int f, int y, bool live,
                                               bool two) {
    cpx<T> v[E];
#pragma unroll
    for (int e = 0; e < E; ++e) v[e] = cpx<T>{p[e], q[e]};
    FX::run(v, gi, tw + N, ex, WarpSync());
#pragma unroll
    for (int e = 0; e < E; ++e) ex[FX::out_index(gi, e)] = v[e];
    __syncwarp();
    if (live) {
#pragma unroll
      for (int e = 0; e < E; ++e) {
        const int k = FX::out_index(gi, e);
        if (k <= K) {
          const cpx<T> a = v[e], b = ex[(N - k) & (N - 1)];
          chip_store<CS>(&col(f, y, k % CPC), k / CPC, two ? cpx<T>{a.x + b.x, a.y - b.y} : a);
          if (two) chip_store<CS>(&col(f + 1, y, k % CPC), k / CPC, cpx<T>{a.y + b.y, b.x - a.x});
        }
      }
    }
    __syncwarp();
  }
  __device__ __forceinline__ void forward(const T (&p)[E], const T (&q)[E], int f, int y, bool live) {
    forward_line(p, q, f, y, live, true);
  }
  __device__ __forceinline__ void forward(const T (&p)[E], int f, int y, bool live) {
    T zero[E];
#pragma unroll
    for (int e = 0; e < E; ++e) zero[e] = (T)0;
    forward_line(p, zero, f, y, live, false);
  }
  // n = -(a x b) sc, or added to n
  static __device__ __forceinline__ void cross(const T (&a)[3][E], const T (&b)[3][E], T (&n)[3][E], T sc,
                                               bool add) {
#pragma unroll
    for (int e = 0; e < E; ++e)
#pragma unroll
      for (int k = 0; k < 3; ++k) {
        const int k1 = (k + 1) % 3, k2 = (k + 2) % 3;
        const T x = -(a[k1][e] * b[k2][e] - a[k2][e] * b[k1][e]) * sc;
        n[k][e] = add ? n[k][e] + x : x;
      }
  }

  // physical field f at x of row y (WIDE)
  __device__ __forceinline__ T fld(int f, int y, int x) { return F[(f * RPC + y) * FS + x]; }
  // output o's product at x of row y, times sc: component o % 3 of the cross
  // products -(a x b), or u . grad rho
  __device__ __forceinline__ T product(int o, int y, int x, T sc) {
    const int k = o % 3, k1 = (k + 1) % 3, k2 = (k + 2) % 3;
    auto cross1 = [&](int a, int b) {
      return -(fld(a + k1, y, x) * fld(b + k2, y, x) - fld(a + k2, y, x) * fld(b + k1, y, x)) * sc;
    };
    if constexpr (NF == 9 + kLinAdj) return o < 3 ? cross1(0, 6) : cross1(6, 3);
    else if constexpr (NF == 12 + kLinTan) return cross1(3, 6) + cross1(9, 0);
    else if (NF == 9 && o == 3)
      return (fld(3, y, x) * fld(6, y, x) + fld(4, y, x) * fld(7, y, x) + fld(5, y, x) * fld(8, y, x)) * sc;
    else return cross1(3, 0);
  }
  // dump: the first dnf physical fields of the plane (as pass C keeps them)
  __device__ __forceinline__ void phase2_wide(T scale, T* __restrict__ dump, int dnf, int z) {
    constexpr int LI = (NI + 1) / 2 * RPC, LO = (NO + 1) / 2 * RPC;
    for (int base = 0; base + wg < LI; base += ng) {
      const int l = min(base + gid, LI - 1), q = l / RPC, y = l % RPC;
      const bool two = 2 * q + 1 < NI;
      T ra[E], rb[E];
      inverse(2 * q, two ? 2 * q + 1 : -1, y, ra, rb);
#pragma unroll
      for (int e = 0; e < E; ++e) {
        T* o = F + (2 * q * RPC + y) * FS + FI::out_index(gi, e);
        *o = ra[e];
        if (two) o[RPC * FS] = rb[e];
      }
    }
    __syncthreads();
    if (dump)
      for (int i = threadIdx.x; i < dnf * RPC * N; i += blockDim.x) {
        const int x = i % N, y = i / N % RPC, f = i / (N * RPC);
        dump[(((long)f * N + z) * N + rank * RPC + y) * N + x] = fld(f, y, x);
      }
    for (int base = 0; base + wg < LO; base += ng) {
      const int l = min(base + gid, LO - 1), q = l / RPC, y = l % RPC;
      const bool live = l == base + gid, two = 2 * q + 1 < NO;
      const T sc = two ? (T)0.5 * scale : scale;
      T a[E], b[E];
#pragma unroll
      for (int e = 0; e < E; ++e) {
        const int x = FX::in_index(gi, e);
        a[e] = product(2 * q, y, x, sc);
        b[e] = two ? product(2 * q + 1, y, x, sc) : (T)0;
      }
      // both kinds of line through one transform: the groups of a warp may differ
      forward_line(a, b, 2 * q, y + rank * RPC, live, two);
    }
  }

  // x rows: the fields and products of pass C
  __device__ __forceinline__ void phase2(T scale) {
    const T h = (T)0.5 * scale;
    for (int base = 0; base + wg < RPC; base += ng) {
      const bool live = base + gid < RPC;
      const int y = live ? base + gid : 0, yg = rank * RPC + y;
      T a[3][E], b[3][E], n[3][E];
      if constexpr (NF == 6 || NF == 9) {  // w = 0..2, u = 3..5: -(u x w)
        inverse(0, 1, y, b[0], b[1]);
        inverse(2, 3, y, b[2], a[0]);
        inverse(4, 5, y, a[1], a[2]);
        cross(a, b, n, h, false);
        if constexpr (NF == 6) {
#pragma unroll
          for (int e = 0; e < E; ++e) n[2][e] *= (T)2;  // alone: no 1/2 of a split
          forward(n[0], n[1], 0, yg, live);
          forward(n[2], 2, yg, live);
        } else {  // u . grad rho
          T n4[E];
          inverse(6, 7, y, b[0], b[1]);
#pragma unroll
          for (int e = 0; e < E; ++e) n4[e] = a[0][e] * b[0][e] + a[1][e] * b[1][e];
          inverse(8, -1, y, b[0], b[1]);
#pragma unroll
          for (int e = 0; e < E; ++e) n4[e] = (n4[e] + a[2][e] * b[0][e]) * h;
          forward(n[0], n[1], 0, yg, live);
          forward(n[2], n4, 2, yg, live);
        }
      } else if constexpr (NF == 9 + kLinAdj) {
        // lines as in pass C: none holds a field of z beside one of x
        T last[E], t[E];
        inverse(6, 7, y, b[0], b[1]);
        inverse(8, -1, y, b[2], t);
        inverse(0, 1, y, a[0], a[1]);
        inverse(2, 3, y, a[2], t);
        cross(a, b, n, h, false);  // -(z x Cx)
        forward(n[0], n[1], 0, yg, live);
#pragma unroll
        for (int e = 0; e < E; ++e) { last[e] = n[2][e]; a[0][e] = t[e]; }
        inverse(4, 5, y, a[1], a[2]);
        cross(b, a, n, h, false);  // -(Cx x Bz)
        forward(last, n[0], 2, yg, live);
        forward(n[1], n[2], 4, yg, live);
      } else {
        T t[E], t2[E];
        inverse(3, 4, y, b[0], b[1]);
        inverse(5, 0, y, b[2], t);
        inverse(6, 7, y, a[0], a[1]);
        inverse(8, 9, y, a[2], t2);
        cross(b, a, n, h, false);  // -(Bz x x)
#pragma unroll
        for (int e = 0; e < E; ++e) { b[0][e] = t[e]; a[0][e] = t2[e]; }
        inverse(1, 2, y, b[1], b[2]);
        inverse(10, 11, y, a[1], a[2]);
        cross(a, b, n, h, true);  // -(Bx x z)
#pragma unroll
        for (int e = 0; e < E; ++e) n[2][e] *= (T)2;
        forward(n[0], n[1], 0, yg, live);
        forward(n[2], 2, yg, live);
      }
    }
  }

  // y-forward of the block's product columns, the kept rows to pass E's tiles
  __device__ __forceinline__ void phase3(cpx<T>* __restrict__ out, int z, bool all) {
    for (int base = 0; base + wg < NO * CPC; base += ng) {
      const int l = min(base + gid, NO * CPC - 1), f = l / CPC, cl = l % CPC, ikx = rank * CPC + cl;
      const bool live = l == base + gid && ikx < X;
      const int kx = min(ikx, X - 1), xt = kx / W, ym = tile_reach_y<N>(all, xt);
      cpx<T> v[E];
#pragma unroll
      for (int e = 0; e < E; ++e) v[e] = col(f, FO::in_index(gi, e), cl);
      FO::run(v, gi, tw, ex, WarpSync());
      if (!live) continue;
      cpx<T>* dst = out + (((long)f * XT + xt) * Y * N + z) * W + kx % W;
#pragma unroll
      for (int e = 0; e < E; ++e) {
        const int iky = row_to_box(FO::out_index(gi, e), K, N);
        if (iky >= K - ym && iky <= K + ym) dst[(long)iky * N * W] = v[e];
      }
    }
  }
};

template <typename T, int N, int NF>
__global__ void __launch_bounds__(kPlaneThreads)
pass_bcd(const cpx<T>* __restrict__ in, cpx<T>* __restrict__ out, const cpx<T>* __restrict__ gtw, T scale,
         const int* __restrict__ full, T* __restrict__ dump, int dnf) {
  using P = Plane<T, N, NF>;
  extern __shared__ __align__(128) unsigned char smem_raw[];
  pdl_trigger();
  P p;
  int rank = 0;
  if (P::CS > 1) asm("mov.u32 %0, %%cluster_ctarank;" : "=r"(rank));
  const int tid = threadIdx.x, z = blockIdx.x / P::CS;
  p.rank = rank;
  p.gid = tid / P::G;
  p.gi = tid % P::G;
  p.ng = blockDim.x / P::G;
  p.wg = p.gid - p.gid % P::GPW;
  p.tw = reinterpret_cast<cpx<T>*>(smem_raw);
  cpx<T>* exs = p.tw + 2 * N;
  p.ex = exs + p.gid * P::EXW;
  p.A = exs + p.ng * P::EXW;
  p.B = p.A + P::NI * P::X * P::RP;
  p.F = reinterpret_cast<T*>(p.B + P::NO * N * P::CP);
  for (int i = tid; i < 2 * N; i += blockDim.x) p.tw[i] = gtw[i];
  const bool all = whole_box(full);
  pdl_wait();
  // the tables are written, and every block of the cluster runs before a line is
  // sent to it
  chip_sync<P::CS>();
  p.phase1(in, z, all);
  chip_sync<P::CS>();
  if constexpr (P::WIDE) p.phase2_wide(scale, dump, dnf, z);
  else p.phase2(scale);
  chip_sync<P::CS>();
  p.phase3(out, z, all);
}

}  // namespace psg
