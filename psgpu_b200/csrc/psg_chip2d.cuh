// psg_chip2d.cuh -- the 2D step with everything between two stages in shared
// memory: one instance per thread-block cluster of CS blocks.
//
// Bound: at these sizes (a 128^2 state is 58 KB in FP64) a step moves no HBM
// traffic worth naming; what costs is latency.  The row scratch of a right-hand
// side in global memory makes every phase wait for L2, and one block per
// instance leaves the rest of the chip idle when there are few instances.
// Here a cluster's blocks split the rows and the columns of the grid and hand the
// intermediate lines to each other through distributed shared memory, so a
// phase never leaves the SMs:
//   1. y-inverse of the fields, one line per lane group, from the block's own
//      columns; the results go to the block that owns the row
//   -- cluster barrier --
//   2. the block's rows: C2R, products, R2C; kx <= K goes to the block that
//      owns the column
//   -- cluster barrier --
//   3. y-forward of the block's product columns, then the spectral finish and
//      the RK4 stage over all of the block's modes (contiguous, no idle lanes)
// Phase 3 and the next stage's phase 1 work on the same columns, so nothing but
// a block barrier lies between them.  Rows and columns are dealt in contiguous runs:
// the lanes that store to another block then cover whole 64- and 128-byte
// segments of its shared memory: rows are stored wavenumber by wavenumber with the
// row index fastest (phase 1's lanes hold consecutive rows of one wavenumber),
// columns row by row (phase 2's lanes hold consecutive wavenumbers of one row).
// Columns dealt round-robin and rows stored row by row scattered every lane's
// value into a segment of its own.  The strides are odd, so that the reads in
// the other direction fall on distinct banks.
// A stage keeps the sum of the increments (z1 + 2 z2 + 2 z3) in place of the
// three of them; 1/k^2 (with the 2/3 mask as its sign) comes from a table.
//
// The arithmetic of the fields, products and stages is psg_ns2d.cuh's and
// psg_tan2d.cuh's (2D_NavierStokes/src_RK4/kernels.h:82-435).
#pragma once
#include <type_traits>

#include "psg_fft2.cuh"
#include "psg_ns2d.cuh"

namespace psg {

// what an instance's launch reads; the kernel of a kind uses the fields it needs
template <typename T>
struct ChipInst {
  int nsteps;
  int mode;     // CHIP_BASE: 2 takes the time derivative of Z into D instead of steps
  T nu, dt;
  cpx<T>* Z;    // state [2K+1][K+1], in / out
  cpx<T>* D;    // perturbation, in / out (CHIP_TANGENT); derivative (mode 2)
  cpx<T>* ZC;   // carried rounding error of the state updates, or null (CHIP_STEP)
  cpx<T>* acc;  // sums of the stage increments, [2K+1][K+1] (twice with a tangent):
                // used when the state arrays do not fit in shared memory
};

// CHIP_STEP: the ensemble's step, final stage as (z - eS z) + (incr - eI incr)
// with the rounding error carried; CHIP_BASE: the UPO search's base step, final
// stage damp2 (damp1 z + incr); CHIP_TANGENT: base and tangent together
enum ChipKind : int { CHIP_STEP = 0, CHIP_BASE = 1, CHIP_TANGENT = 2 };

template <int CS>
__device__ __forceinline__ void chip_sync() {
  if (CS == 1) {
    __syncthreads();
  } else {
    asm volatile(
        "barrier.cluster.arrive.release.aligned;\n\t"
        "barrier.cluster.wait.acquire.aligned;" ::: "memory");
  }
}

// *p of block `rank` of the cluster = v (p: this block's copy of the address)
template <int CS>
__device__ __forceinline__ void chip_store(cpx<double>* p, int rank, cpx<double> v) {
  if (CS == 1) { *p = v; return; }
  uint32_t a;
  asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(a) : "r"((uint32_t)__cvta_generic_to_shared(p)), "r"(rank));
  asm volatile("st.shared::cluster.v2.f64 [%0], {%1, %2};" ::"r"(a), "d"(v.x), "d"(v.y) : "memory");
}
template <int CS>
__device__ __forceinline__ void chip_store(cpx<float>* p, int rank, cpx<float> v) {
  if (CS == 1) { *p = v; return; }
  uint32_t a;
  asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(a) : "r"((uint32_t)__cvta_generic_to_shared(p)), "r"(rank));
  asm volatile("st.shared::cluster.v2.f32 [%0], {%1, %2};" ::"r"(a), "f"(v.x), "f"(v.y) : "memory");
}

// a product that is not contracted into a following sum
__device__ __forceinline__ double mul_rn(double a, double b) { return __dmul_rn(a, b); }
__device__ __forceinline__ float mul_rn(float a, float b) { return __fmul_rn(a, b); }

// The transforms with merged twiddles in FP64 up to 128^2, where they are the faster
// (us a step: 128^2 on 16 blocks 30 -> 25, 64^2 on four 18 -> 16); the tangent's
// registers are at their limit and spill with them (128^2 tangent on 16 blocks 45 ->
// 55).  Not in FP32, although 128^2 on one block takes 107 instead of 97: a path
// through their tables has several rounded factors where LineFFT's has one, the same
// error at every right-hand side, and after 20 steps the FP32 state was 1.23 (16^2 and
// 64^2) and 1.04 (128^2) times as far from 80-bit arithmetic as with LineFFT (FP64: 0.79
// to 0.99).
constexpr bool chip_merged(int elem, int n, int kind) { return elem == 8 && n <= 128 && kind != CHIP_TANGENT; }

template <typename T, int N, int CS, int KIND>
struct ChipShape {
  using FI = LineFFT<N, +1, T>;
  static constexpr int G = FI::G, EXW = FI::SMEM;
  static constexpr int K = N / 3, X = K + 1, Y = 2 * K + 1;
  static constexpr bool TAN = KIND == CHIP_TANGENT;
  static constexpr int NF = TAN ? 6 : 3;  // fields to physical space
  static constexpr int NP = TAN ? 4 : 2;  // products back
  static constexpr int NS = TAN ? 2 : 1;  // states
  static constexpr int RPC = N / CS, CPC = (X + CS - 1) / CS;  // rows, columns of a block
  static constexpr int RP = RPC | 1;                           // wavenumber stride of the physical rows
  static constexpr int CP = CPC | 1;                           // row stride of the product columns
  static constexpr int CO = CPC | 1;                           // row stride of the block's modes
  // rows; columns (one block: in place of the rows, with the stage state apart);
  // one state array
  static constexpr int AW = NF * X * RP, BW = CS == 1 ? NS * Y * CO : NP * N * CP, SW = Y * CPC;
  static constexpr bool CARRY = KIND == CHIP_STEP && sizeof(T) == 4;
  static constexpr int NST = 2 * NS + (CARRY ? 1 : 0);  // state arrays: Z, sum (each state), carried error
  // dynamic shared memory of a block of `nt` threads
  static constexpr size_t smem(int nt, bool state) {
    return sizeof(cpx<T>) * (2 * N + (size_t)(nt / G) * EXW + AW + BW + (state ? (size_t)NST * SW : 0)) +
           sizeof(T) * Y * CO;
  }
  // lane groups the widest phase can use
  static constexpr int lines() {
    const int a = NF * CPC, b = RPC;
    return a > b ? a : b;
  }
};

template <typename T, int N, int CS, int KIND, int PK = 0>
struct Chip2D : ChipShape<T, N, CS, KIND> {
  static_assert(PK == 0 || (sizeof(T) == 4 && KIND == CHIP_STEP), "packed transforms: FP32 steps");
  using S = ChipShape<T, N, CS, KIND>;
  using S::AW; using S::BW; using S::CO; using S::CP; using S::CPC; using S::EXW; using S::G;
  using S::K; using S::NF; using S::NP; using S::NS; using S::RP; using S::RPC; using S::SW; using S::TAN;
  using S::X; using S::Y;
  static constexpr bool M = chip_merged(sizeof(T), N, KIND);
  using FI = std::conditional_t<M, LineFFTM<N, +1, T>, LineFFT<N, +1, T>>;
  using FO = std::conditional_t<M, LineFFTM<N, -1, T>, LineFFT<N, -1, T>>;
  // consumes FI's output distribution
  using FX = std::conditional_t<M, LineFFTM<N, -1, T, true>, LineFFT<N, -1, T, true>>;
  static constexpr int E = FI::E, GPW = 32 / G;  // points per lane, groups per warp

  cpx<T>*tw, *ex, *A, *B;   // twiddles, this group's exchange, rows, columns
  T* wk;                    // [Y][CO]: 1/k^2, negative where the field is zero
  int rank, gid, gi, ng, wg;  // block, lane group, lane, groups, the warp's first group

  __device__ __forceinline__ cpx<T>& row(int f, int y, int k) { return A[(f * X + k) * RP + y]; }
  // product f of the block's column cl
  __device__ __forceinline__ cpx<T>& col(int f, int y, int cl) {
    return CS == 1 ? A[(f * X + cl) * RP + y] : B[(f * N + y) * CP + cl];
  }
  // stage state of part p: with several blocks in the place of product 2p, which
  // the stage update has read by then (phase 1 writes the other blocks' rows only)
  __device__ __forceinline__ cpx<T>& z0(int p, int iky, int cl) {
    return CS == 1 ? B[(p * Y + iky) * CO + cl] : B[(2 * p * N + iky) * CP + cl];
  }

  // field line l = f CPC + cl at box row iky: zero, or w, u = i ky z/k^2,
  // v = -i kx z/k^2 (2D_NavierStokes/src_RK4/kernels.h:126-130), the kx = 0
  // column's lower half from its conjugates.  Selects, no branches: the loads of
  // a line's elements then go out together (a branch on the table's value made
  // each wait for its own: 128^2 FP64, 16 blocks, phase 1 4786 -> 3446 clocks).
  __device__ __forceinline__ cpx<T> field(int f, int cl, int iky) {
    const T t = wk[iky * CO + cl];
    const int ikx = rank * CPC + cl, ff = f % 3;
    const bool cj = ikx == 0 && iky < K;
    const int jky = cj ? 2 * K - iky : iky;
    cpx<T> z = z0(f / 3, jky, cl);
    // u = (i ky t) z, v = (-i kx t) z
    const T m = ff == 1 ? (T)(jky - K) : -(T)ikx;
    cpx<T> r = ff == 0 ? z : cpx<T>{-m * z.y * t, m * z.x * t};
    if (cj) r.y = -r.y;
    return t > (T)0 ? r : czero<T>();
  }

  // the same at transform position r (zero where truncated)
  __device__ __forceinline__ cpx<T> field_at(int f, int cl, int r) {
    const bool lo = r <= K, hi = r >= N - K;
    const cpx<T> v = field(f, cl, lo ? r + K : hi ? r - N + K : 0);
    return (lo || hi) ? v : czero<T>();
  }

  // output y of a column line -> the row's owner
  __device__ __forceinline__ void put_row(int f, int y, int ikx, cpx<T> v) {
    chip_store<CS>(&row(f, y % RPC, ikx), y / RPC, v);
  }
  __device__ __forceinline__ void put_col(int f, int y, int k, cpx<T> v) {
    chip_store<CS>(&col(f, y, k % CPC), k / CPC, v);
  }

  __device__ void phase1() {
    if constexpr (PK != 0) {  // lines 2p, 2p + 1 in one packed transform
      constexpr int NL = (NF * CPC + 1) / 2;
      for (int base = 0; base + wg < NL; base += ng) {
        // lines past the last one repeat it and store nothing
        const int p0 = 2 * (base + gid), p1 = p0 + 1;
        const int l0 = min(p0, NF * CPC - 1), l1 = min(p1, NF * CPC - 1);
        const int f0 = l0 / CPC, c0 = l0 % CPC, f1 = l1 / CPC, c1 = l1 % CPC;
        const bool v0 = p0 == l0 && rank * CPC + c0 < X, v1 = p1 == l1 && rank * CPC + c1 < X;
        Pk v[E];
#pragma unroll
        for (int e = 0; e < E; ++e) {
          const int r = FI::in_index(gi, e);
          const cpx<T> a = dead(e) ? czero<T>() : field_at(f0, c0, r);
          const cpx<T> b = dead(e) ? czero<T>() : field_at(f1, c1, r);
          v[e] = Pk{make_float2(a.x, b.x), make_float2(a.y, b.y)};
        }
        LineFFT2<N, +1>::run(v, gi, tw, reinterpret_cast<float2*>(ex), WarpSync());
#pragma unroll
        for (int e = 0; e < E; ++e) {
          const int y = FI::out_index(gi, e);
          if (v0) put_row(f0, y, rank * CPC + c0, cpx<T>{v[e].re.x, v[e].im.x});
          if (v1) put_row(f1, y, rank * CPC + c1, cpx<T>{v[e].re.y, v[e].im.y});
        }
      }
      return;
    }
    for (int base = 0; base + wg < NF * CPC; base += ng) {
      // groups past the last line repeat it and store nothing
      const int l = min(base + gid, NF * CPC - 1), f = l / CPC, cl = l % CPC, ikx = rank * CPC + cl;
      const bool live = l == base + gid && ikx < X;
      cpx<T> v[E];
#pragma unroll
      for (int e = 0; e < E; ++e) {
        v[e] = dead(e) ? czero<T>() : field_at(f, cl, FI::in_index(gi, e));
      }
      FI::run(v, gi, tw, ex, WarpSync());
      if (live) {
#pragma unroll
        for (int e = 0; e < E; ++e) put_row(f, FI::out_index(gi, e), ikx, v[e]);
      }
    }
  }

  // input element e is truncated for every lane of the group (known at compile
  // time once the caller's loop is unrolled)
  static __device__ __forceinline__ constexpr bool dead(int e) {
    return FI::in_index(0, e) > K && FI::in_index(G - 1, e) < N - K;
  }
  // position r of the line whose inverse transform is a + i b (b: field fb, or
  // none): A + i B up to K, conj(A) + i conj(B) mirrored from N - K; selects
  // instead of branches, as in field()
  __device__ __forceinline__ cpx<T> pair_in(int fa, int fb, int y, int r) {
    const bool lo = r <= K, hi = r >= N - K;
    const int k = lo ? r : hi ? N - r : 0;
    cpx<T> a = row(fa, y, k), b = fb >= 0 ? row(fb, y, k) : czero<T>();
    if (r == 0) a.y = b.y = (T)0;
    if (hi) { a.y = -a.y; b.y = -b.y; }
    return (lo || hi) ? cpx<T>{a.x - b.y, a.y + b.x} : czero<T>();
  }
  __device__ __forceinline__ void inverse_pair(int fa, int fb, int y, cpx<T> (&v)[E]) {
#pragma unroll
    for (int e = 0; e < E; ++e) v[e] = dead(e) ? czero<T>() : pair_in(fa, fb, y, FI::in_index(gi, e));
    FI::run(v, gi, tw, ex, WarpSync());
  }
  // R2C of p + i q and the split into products f, f + 1 of row y0 + y
  __device__ __forceinline__ void forward_pair(cpx<T> (&v)[E], int f, int yg, bool live) {
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
          put_col(f, yg, k, cpx<T>{(T)0.5 * (a.x + b.x), (T)0.5 * (a.y - b.y)});
          put_col(f + 1, yg, k, cpx<T>{(T)0.5 * (a.y + b.y), (T)(-0.5) * (a.x - b.x)});
        }
      }
    }
    __syncwarp();
  }

  __device__ void phase2() {
    const T scale = (T)1 / ((T)N * (T)N);
    for (int base = 0; base + wg < RPC; base += ng) {
      const bool live = base + gid < RPC;
      const int y = live ? base + gid : 0, yg = rank * RPC + y;
      cpx<T> v[E];
      T w[E], u[E];
      if constexpr (PK != 0) {  // (w + i u) and v in one packed transform
        Pk pv[E];
#pragma unroll
        for (int e = 0; e < E; ++e) {
          const int r = FI::in_index(gi, e);
          const cpx<T> a = dead(e) ? czero<T>() : pair_in(0, 1, y, r);
          const cpx<T> b = dead(e) ? czero<T>() : pair_in(2, -1, y, r);
          pv[e] = Pk{make_float2(a.x, b.x), make_float2(a.y, b.y)};
        }
        LineFFT2<N, +1>::run(pv, gi, tw, reinterpret_cast<float2*>(ex), WarpSync());
#pragma unroll
        for (int e = 0; e < E; ++e) { w[e] = pv[e].re.x; u[e] = pv[e].im.x; v[e].x = pv[e].re.y; }
      } else {
        inverse_pair(0, 1, y, v);
#pragma unroll
        for (int e = 0; e < E; ++e) { w[e] = v[e].x; u[e] = v[e].y; }
        inverse_pair(2, TAN ? 5 : -1, y, v);  // (v, dv)
      }
      // products v w, u w (multReal, 2D_NavierStokes/src_RK4/kernels.h:187-201)
      T vv[E], dp[E];
#pragma unroll
      for (int e = 0; e < E; ++e) {
        vv[e] = v[e].x;
        if (TAN) dp[e] = v[e].y * w[e];  // dv w
        v[e] = cpx<T>{vv[e] * w[e] * scale, u[e] * w[e] * scale};
      }
      forward_pair(v, 0, yg, live);
      if constexpr (TAN) {
        inverse_pair(3, 4, y, v);  // (dw, du)
#pragma unroll
        for (int e = 0; e < E; ++e) {
          const T dw = v[e].x, du = v[e].y;
          v[e] = cpx<T>{(dp[e] + vv[e] * dw) * scale, (du * w[e] + u[e] * dw) * scale};
        }
        forward_pair(v, 2, yg, live);
      }
    }
  }

  // y-forward of the block's product columns, kept rows in place of the input
  __device__ void phase3() {
    if constexpr (PK != 0) {  // both products of a column in one packed transform
      for (int base = 0; base + wg < CPC; base += ng) {
        const int cl = base + gid;
        const bool live = cl < CPC && rank * CPC + cl < X;
        Pk v[E];
#pragma unroll
        for (int e = 0; e < E; ++e) {
          const int y = FO::in_index(gi, e);
          const cpx<T> a = live ? col(0, y, cl) : czero<T>(), b = live ? col(1, y, cl) : czero<T>();
          v[e] = Pk{make_float2(a.x, b.x), make_float2(a.y, b.y)};
        }
        LineFFT2<N, -1>::run(v, gi, tw, reinterpret_cast<float2*>(ex), WarpSync());
        if (!live) continue;
#pragma unroll
        for (int e = 0; e < E; ++e) {
          const int iky = row_to_box2(FO::out_index(gi, e), K, N);
          if (iky < 0) continue;
          col(0, iky, cl) = cpx<T>{v[e].re.x, v[e].im.x};
          col(1, iky, cl) = cpx<T>{v[e].re.y, v[e].im.y};
        }
      }
      return;
    }
    for (int base = 0; base + wg < NP * CPC; base += ng) {
      const int l = base + gid, f = l / CPC, cl = l % CPC;
      const bool live = l < NP * CPC && rank * CPC + cl < X;
      cpx<T> v[E];
#pragma unroll
      for (int e = 0; e < E; ++e) v[e] = live ? col(f, FO::in_index(gi, e), cl) : czero<T>();
      FO::run(v, gi, tw, ex, WarpSync());
      if (live) {
#pragma unroll
        for (int e = 0; e < E; ++e) {
          const int iky = row_to_box2(FO::out_index(gi, e), K, N);
          if (iky >= 0) col(f, iky, cl) = v[e];
        }
      }
    }
  }

  // stage s of every mode of the block: increment d = dt (N + forcing), N =
  // -i (kx F(u w) + ky F(v w)) (kernels.h:260-261), forcing -2 at (0, +-4).
  // Four modes at a time, every load before the first store: the arrays may
  // alias as far as the compiler knows, and one mode at a time waited for its own
  // loads (128^2 FP64, 16 blocks: 1498 -> 1010 clocks).
  template <typename IX>
  __device__ void update(const ChipInst<T>& I, int s, cpx<T>* const* Zs, cpx<T>* const* As, cpx<T>* Cs,
                         IX index) {
    constexpr int U = 4, LAST = Y * CPC - 1;
#pragma unroll
    for (int p = 0; p < NS; ++p) {
#pragma unroll 1
      for (int i0 = threadIdx.x; i0 <= LAST; i0 += U * blockDim.x) {
        cpx<T> a[U], b[U], z[U], m[U], c[U];
        int j[U], iky[U], cl[U];
        bool ok[U];
#pragma unroll
        for (int u = 0; u < U; ++u) {
          const int i = i0 + u * blockDim.x, idx = min(i, LAST);
          iky[u] = idx / CPC;
          cl[u] = idx % CPC;
          const int ikx = rank * CPC + cl[u];
          ok[u] = i <= LAST && ikx < X && keep2(ikx, iky[u] - K, K);
          j[u] = index(idx, iky[u], min(ikx, X - 1));
          a[u] = col(2 * p, iky[u], cl[u]);
          b[u] = col(2 * p + 1, iky[u], cl[u]);
          z[u] = Zs[p][j[u]];
          m[u] = As[p][j[u]];
          c[u] = (S::CARRY && s == 3 && Cs) ? Cs[j[u]] : czero<T>();
        }
#pragma unroll
        for (int u = 0; u < U; ++u) {
          if (!ok[u]) continue;
          const int ikx = rank * CPC + cl[u], ky = iky[u] - K;
          const T kx = (T)ikx, kyT = (T)ky;
          T NX = kx * b[u].y + kyT * a[u].y;
          const T NY = -kx * b[u].x - kyT * a[u].x;
          if (p == 0 && ikx == 0 && (ky == 4 || ky == -4)) NX -= (T)2;
          // rounded before it enters a sum, as a stored increment is
          const cpx<T> d = cpx<T>{mul_rn(I.dt, NX), mul_rn(I.dt, NY)};
          cpx<T> zn;
          if (s < 3) {
            As[p][j[u]] = s == 0 ? d : cpx<T>{m[u].x + (T)2 * d.x, m[u].y + (T)2 * d.y};
            if (s == 2) zn = cpx<T>{z[u].x + d.x, z[u].y + d.y};
            else zn = cpx<T>{z[u].x + (T)0.5 * d.x, z[u].y + (T)0.5 * d.y};
          } else {
            const T ix = (m[u].x + d.x) / (T)6, iy = (m[u].y + d.y) / (T)6;
            const T wk2 = kx * kx + kyT * kyT;
            if (KIND == CHIP_STEP) {
              // only the small eS, eI are rounded (see psg_ns2d.cuh)
              const T x = I.dt * I.nu * wk2, hx = (T)0.5 * x;
              const T eS = x / ((T)1 + hx), eI = hx / ((T)1 + hx);
              const T yx = (ix - eI * ix) - eS * z[u].x, yy = (iy - eI * iy) - eS * z[u].y;
              if (S::CARRY && Cs) {  // carry the rounding error of z + y to the next step
                const T ax = yx + c[u].x, ay = yy + c[u].y;
                zn.x = z[u].x + ax;
                zn.y = z[u].y + ay;
                const T bx = zn.x - z[u].x, by = zn.y - z[u].y;
                Cs[j[u]] = cpx<T>{(z[u].x - (zn.x - bx)) + (ax - bx), (z[u].y - (zn.y - by)) + (ay - by)};
              } else {
                zn = cpx<T>{z[u].x + yx, z[u].y + yy};
              }
            } else {
              const T damp1 = (T)1 - (T)0.5 * I.dt * I.nu * wk2;
              const T damp2 = (T)1 / ((T)1 + (T)0.5 * I.dt * I.nu * wk2);
              zn = cpx<T>{damp2 * (damp1 * z[u].x + ix), damp2 * (damp1 * z[u].y + iy)};
            }
            Zs[p][j[u]] = zn;
          }
          z0(p, iky[u], cl[u]) = zn;
        }
      }
    }
  }

  // the stage states from the state arrays
  template <typename IX>
  __device__ void steps(const ChipInst<T>& I, cpx<T>* const* Zs, cpx<T>* const* As, cpx<T>* Cs, IX index) {
    for (int st = 0; st < I.nsteps; ++st) {
#pragma unroll 1
      for (int s = 0; s < 4; ++s) {
        phase1();
        chip_sync<CS>();
        phase2();
        chip_sync<CS>();
        phase3();
        __syncthreads();
        update(I, s, Zs, As, Cs, index);
        __syncthreads();
      }
    }
  }

  __device__ void run(const ChipInst<T>& I, const cpx<T>* __restrict__ gtw, unsigned char* smem, int rank_,
                      bool state) {
    const bool deriv = KIND == CHIP_BASE && I.mode == 2;
    if (!deriv && I.nsteps <= 0) return;
    rank = rank_;
    const int tid = threadIdx.x;
    gid = tid / G; gi = tid % G; ng = blockDim.x / G; wg = gid - gid % GPW;
    tw = reinterpret_cast<cpx<T>*>(smem);
    cpx<T>* exs = tw + 2 * N;
    ex = exs + gid * EXW;
    A = exs + ng * EXW;
    B = A + AW;
    cpx<T>* st = B + BW;
    wk = reinterpret_cast<T*>(st + (state ? S::NST * SW : 0));
    for (int i = tid; i < 2 * N; i += blockDim.x) tw[i] = gtw[i];
    cpx<T>* Zg[2] = {I.Z, I.D};
    for (int idx = tid; idx < Y * CPC; idx += blockDim.x) {
      const int iky = idx / CPC, cl = idx % CPC, ikx = rank * CPC + cl;
      const bool in = ikx < X, keep = in && keep2(ikx, iky - K, K);
      // 1/k^2 of the mode the field takes there (for kx = 0 below ky = 0 its mirror)
      const int my = (ikx == 0 && iky < K) ? 2 * K - iky : iky;
      const T kx = (T)ikx, ky = (T)(my - K);
      const T t = wkinv2(kx * kx + ky * ky);
      wk[iky * CO + cl] = (in && keep2(ikx, my - K, K)) ? t : -t;
#pragma unroll
      for (int p = 0; p < NS; ++p) {
        const cpx<T> z = keep ? Zg[p][iky * X + ikx] : czero<T>();
        if (in) z0(p, iky, cl) = z;
        if (state) st[2 * p * SW + idx] = z;
        else if (in && !keep && !deriv) Zg[p][iky * X + ikx] = z;
      }
      if (S::CARRY && I.ZC) {
        if (state) st[2 * SW + idx] = keep ? I.ZC[iky * X + ikx] : czero<T>();
        else if (in && !keep) I.ZC[iky * X + ikx] = czero<T>();
      }
    }
    // every block of the cluster is running and staged before a line is sent to it
    chip_sync<CS>();
    if (KIND == CHIP_BASE && deriv) {
      phase1();
      chip_sync<CS>();
      phase2();
      chip_sync<CS>();
      phase3();
      __syncthreads();
      for (int idx = tid; idx < Y * CPC; idx += blockDim.x) {
        const int iky = idx / CPC, cl = idx % CPC, ikx = rank * CPC + cl, ky = iky - K;
        if (ikx >= X) continue;
        cpx<T> d = czero<T>();
        if (keep2(ikx, ky, K)) {
          const cpx<T> a = col(0, iky, cl), b = col(1, iky, cl), z = I.Z[iky * X + ikx];
          const T kx = (T)ikx, kyT = (T)ky, wk2 = kx * kx + kyT * kyT;
          T NX = kx * b.y + kyT * a.y;
          const T NY = -kx * b.x - kyT * a.x;
          if (ikx == 0 && ky == 4) NX -= (T)2;
          d = cpx<T>{-I.nu * wk2 * z.x + NX, -I.nu * wk2 * z.y + NY};
        }
        I.D[iky * X + ikx] = d;
      }
      return;
    }
    if (state) {
      cpx<T>* Zs[2] = {st, st + 2 * SW};
      cpx<T>* As[2] = {st + SW, st + 3 * SW};
      steps(I, Zs, As, I.ZC ? st + 2 * SW : nullptr, [](int idx, int, int) { return idx; });
      for (int idx = tid; idx < Y * CPC; idx += blockDim.x) {
        const int iky = idx / CPC, ikx = rank * CPC + idx % CPC;
        if (ikx >= X) continue;
#pragma unroll
        for (int p = 0; p < NS; ++p) Zg[p][iky * X + ikx] = Zs[p][idx];
        if (S::CARRY && I.ZC) I.ZC[iky * X + ikx] = st[2 * SW + idx];
      }
    } else {
      cpx<T>* As[2] = {I.acc, I.acc + X * Y};
      steps(I, Zg, As, I.ZC, [](int, int iky, int ikx) { return iky * X + ikx; });
    }
  }
};

// tables of the merged transforms at grid size n: [plain plan | swapped plan], 2 n
// entries (the others take LineFFT's)
template <typename T>
void chip_tables(int n, cpx<T>* h) {
  switch (n) {
    case 16: LineFFTM<16, 1, T>::host_table(h); LineFFTM<16, 1, T, true>::host_table(h + n); break;
    case 32: LineFFTM<32, 1, T>::host_table(h); LineFFTM<32, 1, T, true>::host_table(h + n); break;
    case 64: LineFFTM<64, 1, T>::host_table(h); LineFFTM<64, 1, T, true>::host_table(h + n); break;
    case 128: LineFFTM<128, 1, T>::host_table(h); LineFFTM<128, 1, T, true>::host_table(h + n); break;
    default: LineFFTM<256, 1, T>::host_table(h); LineFFTM<256, 1, T, true>::host_table(h + n); break;
  }
}

}  // namespace psg
