// FFF (triply periodic Fourier) kernels of the IF-RK4 right-hand side.
//
// Spectral layout (identical to the reference's Blitz arrays, FFF_pencil.cc:209-233):
// one component = complex (Nx, Ny, Hz = Nz/2+1), C order, kx and ky in FFT order;
// a vector field is three components stored back to back.
//
// One right-hand-side evaluation is five launches:
//   inv_x  : dealias on load (+ vorticity for the rotational form), inverse FFT along x
//   y      : inverse FFT along y (in place)
//   z      : C2R along z -> real-space products -> R2C along z (one kernel, lines in registers)
//   y      : forward FFT along y (in place)
//   fwd_x  : forward FFT along x + N_i assembly + force + Leray projection
//            + the IF-RK4 stage update (or a flux reduction / plain N output); one kernel, or an
//            in-place FFT and an elementwise epilogue
#pragma once
#include "ts_common.cuh"
#include "ts_tma.cuh"

namespace ts {

// pass classes of the launch tuning: inverse x, inverse y, z, forward y, forward x
enum { TUNE_X_INV = 0, TUNE_Y_INV = 1, TUNE_Z = 2, TUNE_Y_FWD = 3, TUNE_X_FWD = 4, TUNE_NCLASS = 5, TUNE_NCAND = 6 };

struct Geo {
  int Nx, Ny, Nz, Hz;
  long long S;          // complex elements per component
  // inverse-transformed fields of a right-hand side: complex elements per z line and per
  // component (Hz and S, or the compact lines of Launch::inverse_pitch)
  int Hp;
  long long Sp;
  double kf[3];         // kfactor (reference kfactor[1..3])
  int basis;            // 0 FFF, 1 SFF
  int dealias;          // 0 none, 1 reference corner, 2 two thirds
  // launch tuning per pass class: kernel candidate (0 = the fixed rule) and
  // blocks per SM of the persistent launches (0 = the rule)
  signed char tv[TUNE_NCLASS] = {0, 0, 0, 0, 0};
  signed char tb[TUNE_NCLASS] = {0, 0, 0, 0, 0};
};

// the geometry as the strided passes see the inverse-transformed fields
inline Geo work_geo(const Geo& g) {
  Geo w = g;
  w.Hz = g.Hp;
  w.S = g.Sp;
  return w;
}

// warps per block of the shell-sum kernel k_shell (each warp walks whole z lines)
constexpr int SHELL_WARPS = 4;

// ---------------------------------------------------------------------------
// plain strided-axis FFT (x or y axis) over nf fields, in place
// element (o, row, col) at o*ostride + row*rstride + col, col < inner.
// Persistent and double-buffered: block b walks the work items
// w = b, b + G, ... (w -> field, column tile, outer index); while item w is
// transformed (registers + exchange tile) the tile of its next item streams
// into the other staging tile with cp.async.
// Shared memory: 2 staging tiles + 1 exchange tile of L x CW complex (NT = 3),
// or 2 staging tiles with the consumed one doubling as the exchange tile
// (NT = 2: wider column tiles fit, e.g. 8 columns at L = 1024 in FP32), or
// 3 staging tiles with the consumed one as the exchange tile (NT = 4: the tiles of
// the next two items stream in while one is transformed), or one tile that is also
// the exchange tile (NT = 1: no prefetch inside a block; the blocks sharing an SM
// overlap one another's loads).
// ---------------------------------------------------------------------------
__host__ __device__ constexpr int str_tiles(int nt) { return nt == 4 ? 3 : nt; }
template <typename T, int L, int E, int CW, int DIR, int NT = 3>
__global__ void __launch_bounds__(CW * (L / E), (CW * (L / E)) <= 256 ? 2 : 1)
    k_strided_fft(C<T>* __restrict__ data, int nf, long long fstride, int inner, long long rstride,
                  long long ostride, int nouter, const C<T>* __restrict__ tw, int per, long long mstride,
                  int zero_hi) {
  typedef C<T> V;
  static_assert(NT >= 1 && NT <= 4, "one to three staging tiles");
  constexpr int NBUF = NT == 4 ? 3 : (NT == 1 ? 1 : 2);  // staging tiles: items in flight = NBUF - 1 ahead
  constexpr bool XC = NT != 3;           // exchange in the consumed staging tile
  extern __shared__ __align__(16) unsigned char smraw[];
  V* stage = reinterpret_cast<V*>(smraw);
  const int c = threadIdx.x % CW, t = threadIdx.x / CW;
  const int ntx = (inner + CW - 1) / CW;
  const long long nwork = (long long)nf * ntx * nouter;
  // work item -> (pointer of its column, column valid); field f is field f % per
  // of member f / per (members mstride apart; per = nf for one member)
  auto locate = [&](long long w, bool& ok) -> V* {
    const int f = (int)(w % nf);
    const long long r = w / nf;
    const int tx = (int)(r % ntx);
    const long long o = r / ntx;
    const int col = tx * CW + c;
    ok = col < inner;
    return data + (f / per) * mstride + (f % per) * fstride + o * ostride + (ok ? col : 0);
  };
  auto issue = [&](long long w, int buf) {
    if (w < nwork) {
      bool ok;
      const V* d = locate(w, ok);
      if (ok) {
        V* st = stage + buf * L * CW + c;
#pragma unroll
        for (int s = 0; s < E; ++s) {
          const int r = load_row<L, E>(t, s);
          if (!(zero_hi && 3 * (r < L - r ? r : L - r) > L)) cp_async(st + r * CW, d + r * rstride);
        }
      }
    }
    cp_async_commit();
  };
  // the first NBUF - 1 items; every issue commits one cp.async group (empty past the end)
  issue(blockIdx.x, 0);
  if (NBUF == 3) issue(blockIdx.x + gridDim.x, 1);
  int buf = 0;
  for (long long w = blockIdx.x; w < nwork; w += gridDim.x, buf = (buf + 1 == NBUF ? 0 : buf + 1)) {
    // item w + (NBUF-1) G into the tile item w - G used (every thread passed the
    // barrier after its last exchange read), then wait for item w's group
    issue(w + (NBUF - 1) * (long long)gridDim.x, buf == 0 ? NBUF - 1 : buf - 1);
    cp_async_wait<NBUF - 1>();
    bool ok;
    V* d = locate(w, ok);
    V v[E];
    const V* st = stage + buf * L * CW + c;
#pragma unroll
    for (int s = 0; s < E; ++s) {
      // zero_hi: rows with 3 |k| > L (two-thirds dealiased) are zero and were not loaded
      const int r = load_row<L, E>(t, s);
      v[s] = (ok && !(zero_hi && 3 * (r < L - r ? r : L - r) > L)) ? st[r * CW] : mk<V>(0, 0);
    }
    // each thread read back only what it staged itself; the barrier is for the
    // exchange writes into the consumed tile (NT = 2, 4)
    if (XC) __syncthreads();
    fft_regs<L, E, DIR, 0, 0, false, best_swk(L, E, CW, (int)sizeof(V))>(
        v, t, XC ? stage + buf * L * CW : stage + 2 * L * CW, CW, c, tw, 1);
    if (ok) {
#pragma unroll
      for (int s = 0; s < E; ++s) d[final_row<L, E>(t, s) * rstride] = v[s];
    }
  }
}

// ---------------------------------------------------------------------------
// strided-axis FFT, direct-load form: one tile of CW columns per block, every row of a
// thread loaded straight into its registers (E loads in flight per thread, no staging
// tile), one exchange tile of L x CW complex, so that two to four blocks share an SM and
// overlap one another's loads, exchanges and stores.
// The columns of all fields and outer planes are one run (column q = field, outer index,
// column of the plane), so no tile is cut at a plane's end.  src == dst: in place (a
// block's tile is wholly in registers before its first store).  Outputs are multiplied
// by scl where SCALE.
// ---------------------------------------------------------------------------
template <typename T, int L, int E, int CW, int DIR, int MINB, bool SCALE>
__global__ void __launch_bounds__(CW * (L / E), MINB)
    k_strided_ld(const C<T>* src, C<T>* dst, unsigned ntot, unsigned nplane, unsigned inner, long long fstride,
                 long long rstride, long long ostride, const C<T>* __restrict__ tw, unsigned per, long long mstride,
                 int zero_hi, T scl) {
  chain_begin();
  typedef C<T> V;
  extern __shared__ __align__(16) unsigned char smraw[];
  V* xch = reinterpret_cast<V*>(smraw);
  const int c = threadIdx.x % CW, t = threadIdx.x / CW;
  const unsigned q = blockIdx.x * CW + c;
  const bool ok = q < ntot;
  const unsigned qq = ok ? q : 0;
  const unsigned f = qq / nplane, r = qq - f * nplane, o = r / inner, col = r - o * inner;
  const long long off = (long long)(f / per) * mstride + (long long)(f % per) * fstride + (long long)o * ostride + col;
  const V* a = src + off;
  V v[E];
#pragma unroll
  for (int s = 0; s < E; ++s) {
    // zero_hi: rows with 3 |k| > L (two-thirds dealiased) are zero and were not written
    const int row = load_row<L, E>(t, s);
    v[s] = (ok && !(zero_hi && 3 * (row < L - row ? row : L - row) > L)) ? a[row * rstride] : mk<V>(0, 0);
  }
  fft_regs<L, E, DIR, 0, 0, false, best_swk(L, E, CW, (int)sizeof(V))>(v, t, xch, CW, c, tw, 1);
  if (!ok) return;
  V* d = dst + off;
#pragma unroll
  for (int s = 0; s < E; ++s) d[final_row<L, E>(t, s) * rstride] = SCALE ? scale(v[s], scl) : v[s];
}

// ---------------------------------------------------------------------------
// inverse x pass, all output fields of a column tile in one block (tuning candidates; two
// blocks of 256 threads per SM).
// FORM 0: W_0..2 = D U.  FORM 1: also W_3..5 = D omega.
// ---------------------------------------------------------------------------
__host__ __device__ constexpr int inv_x_nout(int form) { return form == 0 ? 3 : 6; }

template <typename T, int L, int E, int CW, int FORM>
__global__ void __launch_bounds__(CW * (L / E), (CW * (L / E)) <= 256 ? 2 : 1)
    k_inv_x_ld(const C<T>* __restrict__ U, C<T>* __restrict__ W, Geo g, const C<T>* __restrict__ tw, int kept) {
  typedef C<T> V;
  static_assert(FORM == 0 || FORM == 1, "the fluid forms");
  extern __shared__ __align__(16) unsigned char smraw[];
  V* sm = reinterpret_cast<V*>(smraw);
  const int c = threadIdx.x % CW, t = threadIdx.x / CW;
  const int inner = g.Ny * g.Hz;
  int col;
  bool ok;
  if (kept) {
    // two-thirds dealiasing: only the columns with 3|ky| <= Ny and 3 kz <= Nz can be
    // nonzero; block = (kept ly, tile of CW kept lz); the other columns are not
    // written, and the y and z passes treat them as zero without reading them
    const int qy = g.Ny / 3, nzk = g.Nz / 3 + 1, ntz = (nzk + CW - 1) / CW;
    const int iy = blockIdx.x / ntz, lzc = (blockIdx.x % ntz) * CW + c;
    const int ky = iy <= qy ? iy : iy - (2 * qy + 1);
    ok = lzc < nzk;
    col = ((ky + g.Ny) % g.Ny) * g.Hz + (ok ? lzc : 0);
  } else {
    col = blockIdx.x * CW + c;
    ok = col < inner;
  }
  const int ly = ok ? col / g.Hz : 0, lz = ok ? col % g.Hz : 0;
  const T Ky = (T)(kfft(ly, g.Ny) * g.kf[1]), Kz = (T)(lz * g.kf[2]);
  const long long rstride = inner;
  constexpr int nout = inv_x_nout(FORM);
  // FP32 with up to 8 elements per thread: the three (dealiased) components of U
  // are loaded once, up front, and every output field is built from registers
  // (FP64 would spill them)
  constexpr bool UPFRONT = E <= 8 && sizeof(T) == 4;
  V u[UPFRONT ? 3 : 1][UPFRONT ? E : 1];
  if constexpr (UPFRONT) {
#pragma unroll
    for (int s = 0; s < E; ++s) {
      const int lx = load_row<L, E>(t, s);
      const long long off = lx * rstride + col;
      const bool z = !ok || dealias_zero(g.dealias, g.basis, lx, ly, lz, g.Nx, g.Ny, g.Nz);
#pragma unroll
      for (int c = 0; c < 3; ++c) u[c][s] = z ? mk<V>(0, 0) : U[c * g.S + off];
    }
  }
  // unrolled (register path) so that the register-array indices below are compile-time constants
  constexpr int kUnroll = UPFRONT ? nout : 1;
#pragma unroll kUnroll
  for (int f = 0; f < nout; ++f) {
    V v[E];
#pragma unroll
    for (int s = 0; s < E; ++s) {
      const int lx = load_row<L, E>(t, s);
      const long long off = lx * rstride + col;
      V a = mk<V>(0, 0);
      if (UPFRONT) {
        if (f < 3) {
          a = u[f][s];
        } else {
          const T Kx = (T)(kfft(lx, g.Nx) * g.kf[0]);
          const int i = f - 3, i1 = i == 2 ? 0 : i + 1, i2 = i == 0 ? 2 : i - 1;
          const T Ka = i1 == 0 ? Kx : (i1 == 1 ? Ky : Kz);
          const T Kb = i2 == 0 ? Kx : (i2 == 1 ? Ky : Kz);
          a = mul_i<1>(sub(scale(u[i2][s], Ka), scale(u[i1][s], Kb)));
        }
      } else if (ok && !dealias_zero(g.dealias, g.basis, lx, ly, lz, g.Nx, g.Ny, g.Nz)) {
        if (f < 3) {
          a = U[f * g.S + off];
        } else {
          // omega_i = i (K_{i+1} U_{i+2} - K_{i+2} U_{i+1})  (indices mod 3)
          const T Kx = (T)(kfft(lx, g.Nx) * g.kf[0]);
          const int i = f - 3, i1 = i == 2 ? 0 : i + 1, i2 = i == 0 ? 2 : i - 1;
          const T Ka = i1 == 0 ? Kx : (i1 == 1 ? Ky : Kz);
          const T Kb = i2 == 0 ? Kx : (i2 == 1 ? Ky : Kz);
          const V ub = U[i2 * g.S + off], ua = U[i1 * g.S + off];
          a = mul_i<1>(sub(scale(ub, Ka), scale(ua, Kb)));
        }
      }
      v[s] = a;
    }
    fft_regs<L, E, 1, 0, 0, false, best_swk(L, E, CW, (int)sizeof(V))>(v, t, sm, CW, c, tw, 1);
    if (ok) {
      V* d = W + f * g.S + col;
#pragma unroll
      for (int s = 0; s < E; ++s) d[final_row<L, E>(t, s) * rstride] = v[s];
    }
  }
}


// ---------------------------------------------------------------------------
// inverse x pass, one output field per block: every row is loaded straight into registers
// (as in k_strided_ld), a vorticity row is combined from the two components it needs.  The input components are read once per output field
// that needs them; the blocks of a column tile's fields are neighbours (field fastest), so
// all but the first read hit L2.  16 elements per thread and one field keep it at 64-80
// registers and 24-32 warps per SM, where the form with all fields of a tile in one block
// (k_inv_x_ld) holds U in registers, 8 elements per thread and 16 warps.
// FORM 0: W_0..2 = D U.  FORM 1: also W_3..5 = D omega.  FORM 5 (the giver of the per-sphere
// energy flux): W_3..5 = D U inside the sphere |K| <= R (Fill_in_sphere, fill_space.cc:56-64),
// zero outside.
// ---------------------------------------------------------------------------
// rows [lo, hi) of the column (ly, lz) are cleared by dealiasing (dealias_zero, basis 0)
__device__ __forceinline__ void fff_zero_rows(int mode, int ly, int lz, int Nx, int Ny, int Nz, int& lo, int& hi) {
  lo = hi = Nx;
  if (mode == 1) {
    if (ly >= Ny / 3 + 1 && ly <= 2 * Ny / 3 - 1 && lz >= Nz / 3 + 1) lo = Nx / 3 + 1, hi = 2 * Nx / 3;
  } else if (mode == 2) {
    const bool out = 3 * abs(kfft(ly, Ny)) > Ny || 3 * lz > Nz;
    lo = out ? 0 : Nx / 3 + 1;
    hi = out ? Nx : Nx - Nx / 3;
  }
}

template <typename T, int L, int E, int CW, int FORM, int MINB>
__global__ void __launch_bounds__(CW * (L / E), MINB)
    k_inv_x_f(const C<T>* U, C<T>* W, Geo g, const C<T>* __restrict__ tw,
              int kept, double K2max) {
  chain_begin();
  typedef C<T> V;
  static_assert(FORM == 0 || FORM == 1 || FORM == 5, "fluid forms, flux giver");
  constexpr unsigned NF = FORM == 1 ? 6 : 3;
  extern __shared__ __align__(16) unsigned char smraw[];
  V* xch = reinterpret_cast<V*>(smraw);
  const int c = threadIdx.x % CW, t = threadIdx.x / CW;
  const unsigned inner = g.Ny * g.Hz;
  const unsigned f = blockIdx.x % NF, q = (blockIdx.x / NF) * CW + c;
  unsigned ly, lz;
  bool ok;
  if (kept) {
    // two-thirds dealiasing: only the columns with 3|ky| <= Ny and 3 kz <= Nz can be
    // nonzero; they are one run of columns here, the others are not written, and the y and
    // z passes treat them as zero without reading them
    // (kept == 2: compact lines of whole tiles)
    const unsigned qy = g.Ny / 3, nzk = g.Nz / 3 + 1, nzt = kept == 2 ? g.Hp : nzk, iy = q / nzt;
    lz = q - iy * nzt;
    ok = iy <= 2 * qy && lz < nzk;
    ly = iy <= qy ? iy : iy + g.Ny - (2 * qy + 1);
  } else {
    ok = q < inner;
    ly = q / g.Hz;
    lz = q - ly * g.Hz;
  }
  if (!ok) ly = lz = 0;
  const long long col = (long long)ly * g.Hz + lz, rstride = inner;
  const T Ky = (T)(kfft(ly, g.Ny) * g.kf[1]), Kz = (T)(lz * g.kf[2]);
  V v[E];
  int zlo, zhi;
  fff_zero_rows(g.dealias, ly, lz, g.Nx, g.Ny, g.Nz, zlo, zhi);
  if (!ok) zlo = 0, zhi = L;
  if (FORM != 1 || f < 3) {
    const V* src = U + f * g.S + col;
#pragma unroll
    for (int s = 0; s < E; ++s) {
      const int lx = load_row<L, E>(t, s);
      v[s] = (lx >= zlo && lx < zhi) ? mk<V>(0, 0) : src[lx * rstride];
    }
    if (FORM == 5) {
      // inside |K| <= rad: (Kx^2 + Ky^2) + Kz^2 <= K2max in FP64 (Kmagnitude)
      const double Kyd = kfft(ly, g.Ny) * g.kf[1], Kzd = lz * g.kf[2];
#pragma unroll
      for (int s = 0; s < E; ++s) {
        const double Kxd = kfft(load_row<L, E>(t, s), g.Nx) * g.kf[0];
        if (!((Kxd * Kxd + Kyd * Kyd) + Kzd * Kzd <= K2max)) v[s] = mk<V>(0, 0);
      }
    }
  } else {
    // omega_i = i (K_{i+1} U_{i+2} - K_{i+2} U_{i+1})  (indices mod 3)
    const int i = (int)f - 3, i1 = i == 2 ? 0 : i + 1, i2 = i == 0 ? 2 : i - 1;
    const V *sa = U + i1 * g.S + col, *sb = U + i2 * g.S + col;
#pragma unroll
    for (int s = 0; s < E; ++s) {
      const int lx = load_row<L, E>(t, s);
      const bool z = lx >= zlo && lx < zhi;
      const T Kx = (T)(kfft(lx, g.Nx) * g.kf[0]);
      const T Ka = i1 == 0 ? Kx : (i1 == 1 ? Ky : Kz), Kb = i2 == 0 ? Kx : (i2 == 1 ? Ky : Kz);
      const V ua = z ? mk<V>(0, 0) : sa[lx * rstride], ub = z ? mk<V>(0, 0) : sb[lx * rstride];
      v[s] = mul_i<1>(sub(scale(ub, Ka), scale(ua, Kb)));
    }
  }
  fft_regs<L, E, 1, 0, 0, false, best_swk(L, E, CW, (int)sizeof(V))>(v, t, xch, CW, c, tw, 1);
  if (!ok) return;
  V* d = W + (f + (FORM == 5 ? 3 : 0)) * g.Sp + (long long)ly * g.Hp + lz;
  const long long wstride = (long long)g.Ny * g.Hp;
#pragma unroll
  for (int s = 0; s < E; ++s) d[final_row<L, E>(t, s) * wstride] = v[s];
}

// ---------------------------------------------------------------------------
// inverse x pass of the adjoint's cotangent: W_6..8 = IFFT_x(lsc c^-1 P Lam), the
// Leray-projected cotangent divided by the C2R weight c (2 on the planes 0 < kz < Nz/2, else
// 1).  The three components of a column stay in registers from the projection to their
// transforms, one after the other through one exchange tile.
// ---------------------------------------------------------------------------
template <typename T, int L, int E, int CW, int MINB>
__global__ void __launch_bounds__(CW * (L / E), MINB)
    k_inv_x_cot(const C<T>* Lam, C<T>* W, Geo g, const C<T>* __restrict__ tw, T lsc) {
  chain_begin();
  typedef C<T> V;
  extern __shared__ __align__(16) unsigned char smraw[];
  V* xch = reinterpret_cast<V*>(smraw);
  const int c = threadIdx.x % CW, t = threadIdx.x / CW;
  const unsigned inner = g.Ny * g.Hz, q = blockIdx.x * CW + c;
  const bool ok = q < inner;
  const unsigned ly = ok ? q / g.Hz : 0, lz = ok ? q - ly * g.Hz : 0;
  const long long col = (long long)ly * g.Hz + lz, rstride = inner;
  const T Ky = (T)(kfft(ly, g.Ny) * g.kf[1]), Kz = (T)(lz * g.kf[2]);
  const T lw = (lz > 0 && 2 * (int)lz < g.Nz) ? lsc * (T)0.5 : lsc;
  V v[3][E];
#pragma unroll
  for (int i = 0; i < 3; ++i)
#pragma unroll
    for (int s = 0; s < E; ++s) v[i][s] = ok ? Lam[i * g.S + load_row<L, E>(t, s) * rstride + col] : mk<V>(0, 0);
#pragma unroll
  for (int s = 0; s < E; ++s) {
    // (P Lam)_i = Lam_i - K_i (K . Lam) / K^2, identity at K = 0
    const T Kx = (T)(kfft(load_row<L, E>(t, s), g.Nx) * g.kf[0]);
    const T K2 = (Kx * Kx + Ky * Ky) + Kz * Kz;
    const V n = add(add(scale(v[0][s], Kx), scale(v[1][s], Ky)), scale(v[2][s], Kz));
    const V d = quot(n, recip(K2));
    v[0][s] = scale(sub(v[0][s], scale(d, Kx)), lw);
    v[1][s] = scale(sub(v[1][s], scale(d, Ky)), lw);
    v[2][s] = scale(sub(v[2][s], scale(d, Kz)), lw);
  }
#pragma unroll
  for (int i = 0; i < 3; ++i) {
    fft_regs<L, E, 1, 0, 0, false, best_swk(L, E, CW, (int)sizeof(V))>(v[i], t, xch, CW, c, tw, 1);
    if (ok) {
      V* d = W + (6 + i) * g.S + col;
#pragma unroll
      for (int s = 0; s < E; ++s) d[final_row<L, E>(t, s) * rstride] = v[i][s];
    }
  }
}

// ---------------------------------------------------------------------------
// inverse x pass, persistent with a prefetch (FP32, FORM 0 / 1): each block walks the
// column tiles tile = blockIdx.x + k G; every thread stages the dealiased U rows it
// owns (rows load_row(t, s) of its column) with cp.async into its own slots of a
// staging tile, moves them to registers, issues the copies of its next tile into the
// same slots (only it reads them, so no barrier is needed) and then transforms the
// output fields of the current tile from registers while the next tile streams in.
// Same result as k_inv_x_ld.  Shared memory: the staging tile (3 L CW) + the
// exchange tile (L CW).
// ---------------------------------------------------------------------------
template <typename T, int L, int E, int CW, int FORM>
__global__ void __launch_bounds__(CW * (L / E), 1)
    k_inv_x_pf(const C<T>* __restrict__ U, C<T>* __restrict__ W, Geo g, const C<T>* __restrict__ tw, int kept) {
  typedef C<T> V;
  static_assert(FORM == 0 || FORM == 1, "the fluid forms");
  extern __shared__ __align__(16) unsigned char smraw[];
  V* xch = reinterpret_cast<V*>(smraw);  // exchange tile, L x CW
  V* stg = xch + L * CW;                  // staging tile, 3 x L x CW
  const int c = threadIdx.x % CW, t = threadIdx.x / CW;
  const int inner = g.Ny * g.Hz;
  const long long rstride = inner;
  const int qy = g.Ny / 3, nzk = g.Nz / 3 + 1, ntz = (nzk + CW - 1) / CW;
  const int ntiles = kept ? (2 * qy + 1) * ntz : (inner + CW - 1) / CW;
  // column of this thread in tile `tile` (the mapping of k_inv_x_ld's blocks)
  auto column = [&](int tile, bool& ok) -> int {
    if (kept) {
      const int iy = tile / ntz, lzc = (tile % ntz) * CW + c;
      const int ky = iy <= qy ? iy : iy - (2 * qy + 1);
      ok = lzc < nzk;
      return ((ky + g.Ny) % g.Ny) * g.Hz + (ok ? lzc : 0);
    }
    const int col = tile * CW + c;
    ok = col < inner;
    return ok ? col : 0;
  };
  auto issue = [&](int tile) {
    if (tile < ntiles) {
      bool ok;
      const int col = column(tile, ok);
      if (ok) {
        const int ly = col / g.Hz, lz = col % g.Hz;
#pragma unroll
        for (int s = 0; s < E; ++s) {
          const int lx = load_row<L, E>(t, s);
          if (!dealias_zero(g.dealias, g.basis, lx, ly, lz, g.Nx, g.Ny, g.Nz))
#pragma unroll
            for (int q = 0; q < 3; ++q) cp_async(stg + (q * L + lx) * CW + c, U + q * g.S + lx * rstride + col);
        }
      }
    }
    cp_async_commit();
  };
  constexpr int nout = FORM == 0 ? 3 : 6;
  issue(blockIdx.x);
  for (int tile = blockIdx.x; tile < ntiles; tile += gridDim.x) {
    cp_async_wait<0>();
    bool ok;
    const int col = column(tile, ok);
    const int ly = col / g.Hz, lz = col % g.Hz;
    const T Ky = (T)(kfft(ly, g.Ny) * g.kf[1]), Kz = (T)(lz * g.kf[2]);
    V u[3][E];
#pragma unroll
    for (int s = 0; s < E; ++s) {
      const int lx = load_row<L, E>(t, s);
      const bool z = !ok || dealias_zero(g.dealias, g.basis, lx, ly, lz, g.Nx, g.Ny, g.Nz);
#pragma unroll
      for (int q = 0; q < 3; ++q) u[q][s] = z ? mk<V>(0, 0) : stg[(q * L + lx) * CW + c];
    }
    // the slots are this thread's own: the next tile may stream into them now
    issue(tile + gridDim.x);
#pragma unroll
    for (int f = 0; f < nout; ++f) {
      V v[E];
#pragma unroll
      for (int s = 0; s < E; ++s) {
        if (f < 3) {
          v[s] = u[f][s];
        } else {
          // omega_i = i (K_{i+1} U_{i+2} - K_{i+2} U_{i+1})  (indices mod 3)
          const int lx = load_row<L, E>(t, s);
          const T Kx = (T)(kfft(lx, g.Nx) * g.kf[0]);
          const int i = f - 3, i1 = i == 2 ? 0 : i + 1, i2 = i == 0 ? 2 : i - 1;
          const T Ka = i1 == 0 ? Kx : (i1 == 1 ? Ky : Kz);
          const T Kb = i2 == 0 ? Kx : (i2 == 1 ? Ky : Kz);
          v[s] = mul_i<1>(sub(scale(u[i2][s], Ka), scale(u[i1][s], Kb)));
        }
      }
      fft_regs<L, E, 1, 0, 0, false, best_swk(L, E, CW, (int)sizeof(V))>(v, t, xch, CW, c, tw, 1);
      if (ok) {
        V* d = W + f * g.S + col;
#pragma unroll
        for (int s = 0; s < E; ++s) d[final_row<L, E>(t, s) * rstride] = v[s];
      }
    }
  }
  cp_async_wait<0>();  // nothing in flight when the block leaves
}

// ---------------------------------------------------------------------------
// z pass: C2R of the NIN input lines, real-space products, R2C of the NOUT
// product lines.  Lines are contiguous (Hz = M+1 complex, M = Nz/2); a block
// handles `nl` consecutive (x,y) lines of every component, with TPL = M/E
// threads per line.  Each component's line is transformed in registers and
// exchanged through its own padded shared-memory slot (M + M/16 complex);
// after the inverse transforms slot c holds the real line of component c
// packed as M complex (re = even point, im = odd point), the products are
// formed in place per point, and each product line is transformed forward in
// its slot and post-processed straight to global memory.
// In place on P: outputs overwrite the first NOUT components at the same
// lines, after every input line has been read.
// FORM 0 (conservative): in u1,u2,u3 -> out u1u1,u2u2,u3u3,u1u2,u2u3,u3u1
// FORM 1 (rotational):   in u1..3,w1..3 -> out u x w
// ---------------------------------------------------------------------------
template <int M> __host__ __device__ constexpr int zslot() { return M + M / 16 + 1; }

// Real-space product forms of the z pass.
// FORM 0 (conservative, whole tensor): in u1,u2,u3 -> u1u1,u2u2,u3u3,u1u2,u2u3,u3u1
// FORM 7 (conservative step): in u1,u2,u3 -> d2,d3,u1u2,u2u3,u3u1 with d2 = u2u2 - u1u1,
//         d3 = u3u3 - u1u1: taking u1u1 off the diagonal changes N by the gradient of u1u1,
//         which the projection removes, so a step needs one transform less.  It removes it to
//         rounding only: N carries an error of the size of eps |K| u1u1 in the modes with kx = 0,
//         where the whole tensor has none (the other modes have it either way).  u1u1 because x
//         is the bounded axis of SFF and SSF, along which no flow or mean wind is uniform: shear
//         flows and winds along z keep a nonlinear term of exactly zero (with u3u3 taken off, one
//         of 1e-6 at a wind of 10 in FP32); on FFF a flow along x has that error
// FORM 1 (rotational):    in u1..3,w1..3    -> u x w
// FORM 2 (scalar, Boussinesq): in u1,u2,u3,T -> the five of FORM 7, then u1T,u2T,u3T
//                         (compute_diag_offdiag.cc:47-136)
// FORM 3 (adjoint of the rotational form): in u, w, mu -> mu x u, then w x mu
// FORM 5 (MHD):           in u1..3, b1..3 -> the symmetric part S_ij = u_i u_j - b_i b_j of
//         Zp_i Zm_j, Zp = u + b, Zm = u - b, as S22 - S11, S33 - S11, S12, S23, S31, and the
//         antisymmetric part A_ij = b_i u_j - u_i b_j as A12, A23, A31: U.nlin is the
//         divergence of S and B.nlin that of A (compute_nlin_VF_MHD.cc:40-95, MHD.cc:75-84,150-161).
//         Every product is rounded by itself (mul_rn), so that the products of an aligned state,
//         u = b or u = -b, cancel exactly, as Zp_i Zm_j does: with an fma its rounding is left.
//         256^3 FP32 step 4350 us with fma and so (FP64 9150 and 9285); on Zp and Zm held in the
//         registers of u and b 4392 (9330)
// FORM 6 (flux giver):    in u1..3, g1..3   -> u_i g_j (f = 3 i + j), for the giver nonlinear
//                         term N_i = sum_j D_j F[u_j g_i] (compute_nlin_ET_VF.cc:71-87)
__host__ __device__ constexpr int z_nin(int form) {
  return (form == 0 || form == 7) ? 3 : (form == 2 ? 4 : (form == 3 ? 9 : 6));
}
__host__ __device__ constexpr int z_nout(int form) {
  return form == 0 ? 6 : (form == 7 ? 5 : (form == 1 ? 3 : (form == 6 ? 9 : (form == 3 ? 6 : 8))));
}

// component f of a x b for real points packed two per complex (re, im independent)
template <typename V> __device__ __forceinline__ V cross_pk(int f, const V* a, const V* b) {
  const int i = f == 2 ? 0 : f + 1, j = f == 0 ? 2 : f - 1;
  return mk<V>(a[i].x * b[j].x - a[j].x * b[i].x, a[i].y * b[j].y - a[j].y * b[i].y);
}
template <typename V> __device__ __forceinline__ V prod_pk(V a, V b) { return mk<V>(a.x * b.x, a.y * b.y); }
// a c - b d
template <typename V> __device__ __forceinline__ V diff_pk(V a, V c, V b, V d) {
  return mk<V>(a.x * c.x - b.x * d.x, a.y * c.y - b.y * d.y);
}
// a copy that the compiler takes for another value: what is computed from it is computed again
// instead of being kept in registers over the transform of the product before (256^3 FP32 MHD step
// 4410 us with u1u1 kept, which spills 172 bytes a thread, 4348 so)
__device__ __forceinline__ float2 again(float2 a) { asm("" : "+f"(a.x), "+f"(a.y)); return a; }
__device__ __forceinline__ double2 again(double2 a) { asm("" : "+d"(a.x), "+d"(a.y)); return a; }
// product f of a form from its inputs at a point (f known at compile time; not FORM 3)
template <int FORM, typename V> __device__ __forceinline__ V z_product(int f, const V* in) {
  if constexpr (FORM == 1) {
    return cross_pk(f, in, in + 3);
  } else if constexpr (FORM == 0) {
    return f < 3 ? prod_pk(in[f], in[f]) : prod_pk(in[f - 3], in[f == 5 ? 0 : f - 2]);
  } else if constexpr (FORM == 6) {
    return prod_pk(in[f / 3], in[3 + f % 3]);
  } else if constexpr (FORM == 5) {
    auto dif = [&](int a, int c, int b, int d) { return sub(mul_rn(in[a], in[c]), mul_rn(in[b], in[d])); };
    if (f < 2) {
      const V a = f == 0 ? in[0] : again(in[0]), b = f == 0 ? in[3] : again(in[3]);
      return sub(dif(f + 1, f + 1, f + 4, f + 4), sub(mul_rn(a, a), mul_rn(b, b)));
    }
    const int i = (f - 2) % 3, j = (i + 1) % 3;
    return f < 5 ? dif(i, j, 3 + i, 3 + j) : dif(3 + i, j, i, 3 + j);
  } else {
    if (f < 2) {
      const V a = f == 0 ? in[0] : again(in[0]);
      return diff_pk(in[f + 1], in[f + 1], a, a);
    }
    return f < 5 ? prod_pk(in[f - 2], in[(f - 1) % 3]) : prod_pk(in[f - 5], in[3]);
  }
}

template <typename T, int NZ, int E, int FORM>
__global__ void __launch_bounds__(256) k_z_fused(C<T>* __restrict__ P, Geo g, const C<T>* __restrict__ tw, int nl,
                                                 long long msP, int zkeep) {
  typedef C<T> V;
  constexpr int M = NZ / 2, H = M + 1, TPL = M / E, LDS = zslot<M>();
  constexpr int NIN = z_nin(FORM), NOUT = z_nout(FORM);
  extern __shared__ __align__(16) unsigned char smraw[];
  V* sm = reinterpret_cast<V*>(smraw);
  const long long nlines = (long long)g.Nx * g.Ny;
  // member blockIdx.y (P + blockIdx.y * msP holds its fields)
  P += blockIdx.y * msP;
  const long long line0 = (long long)blockIdx.x * nl;
  const int nh = (int)((nlines - line0) < nl ? (nlines - line0) : nl);
  const int l = threadIdx.x / TPL, t = threadIdx.x % TPL;
  const bool live = l < nh;
  const long long lbase = (line0 + (live ? l : 0)) * H;
  auto slot = [&](int c, int ll) { return sm + (c * nl + ll) * LDS; };

  // A. inverse: Z[k] = (X + Y) + i conj(w^k)(X - Y), Y = conj(X[M-k]) (imag of X[0], X[M] dropped),
  //    then the length-M inverse FFT gives z[n] = u[2n] + i u[2n+1]
  for (int c = 0; c < NIN; ++c) {
    const V* X = P + c * g.S + lbase;
    V v[E];
#pragma unroll
    for (int s = 0; s < E; ++s) {
      const int k = load_row<M, E>(t, s);
      V a = mk<V>(0, 0), b = mk<V>(0, 0);
      const int zk = (FORM == 3 && c >= 6) ? M : zkeep;  // the adjoint's cotangent lines are full
      if (live && k <= zk) a = X[k];
      if (live && M - k <= zk) b = conjg(X[M - k]);
      if (k == 0) { a.y = 0; b.y = 0; }
      v[s] = add(add(a, b), mul_i<1>(mul(conjg(tw[k]), sub(a, b))));
    }
    V* sl = slot(c, l < nl ? l : 0);
    fft_regs<M, E, 1, 0, 1>(v, t, sl, 1, 0, tw, 2);
#pragma unroll
    for (int s = 0; s < E; ++s) sl[prow<1>(final_row<M, E>(t, s))] = v[s];
  }
  __syncthreads();
  // B. products, in place per real point pair
  for (int e = threadIdx.x; e < nl * M; e += blockDim.x) {
    const int ll = e / M, m = prow<1>(e % M);
    V in[NIN];
#pragma unroll
    for (int c = 0; c < NIN; ++c) in[c] = slot(c, ll)[m];
    if constexpr (FORM == 3) {
#pragma unroll
      for (int f = 0; f < 3; ++f) {
        slot(f, ll)[m] = cross_pk(f, in + 6, in);
        slot(3 + f, ll)[m] = cross_pk(f, in + 3, in + 6);
      }
    } else {
#pragma unroll
      for (int f = 0; f < NOUT; ++f) slot(f, ll)[m] = z_product<FORM>(f, in);
    }
  }
  __syncthreads();
  // C. forward: length-M FFT of z[n] = p[2n] + i p[2n+1], then
  //    X[k] = 1/2 (Z + Z') - i/2 w^k (Z - Z'), Z' = conj(Z[M-k]), Z[M] = Z[0]
  for (int c = 0; c < NOUT; ++c) {
    V* sl = slot(c, l < nl ? l : 0);
    V v[E];
#pragma unroll
    for (int s = 0; s < E; ++s) v[s] = sl[prow<1>(load_row<M, E>(t, s))];
    __syncthreads();
    fft_regs<M, E, -1, 0, 1>(v, t, sl, 1, 0, tw, 2);
#pragma unroll
    for (int s = 0; s < E; ++s) sl[prow<1>(final_row<M, E>(t, s))] = v[s];
    __syncthreads();
    V* dst = P + c * g.S + line0 * H;
    for (int e = threadIdx.x; e < nh * H; e += blockDim.x) {
      const int ll = e / H, k = e % H;
      const V* z = slot(c, ll);
      const V Z = z[prow<1>(k == M ? 0 : k)];
      const V Zp = conjg(z[prow<1>(k == 0 ? 0 : M - k)]);
      const V s = scale(add(Z, Zp), (T)0.5);
      const V d = mul_i<-1>(mul(tw[k], scale(sub(Z, Zp), (T)0.5)));
      dst[e] = add(s, d);
    }
  }
}

// ---------------------------------------------------------------------------
// z pass, register-resident variant (M = Nz/2 <= 512): one line per group of
// TPL = M/8 consecutive lanes, 8 elements per thread.  The inverse transform
// (forward radix schedule) leaves every component's real line in registers in
// the order the forward transform with the reversed schedule expects, so the
// products are formed in registers and fed straight to the forward FFTs.  The
// real-transform pair terms X[M-k] come from the partner lane by a warp
// shuffle; shared memory holds only one exchange line per line group.
// ---------------------------------------------------------------------------
// threads per block of k_z_reg: up to six components live in registers, so it
// runs 64-thread blocks, six per SM, with a 170-register budget (FP32 only; FP64
// would spill and uses the other z kernels).  On B200 at 256^3 the 64-thread
// blocks streamed 2.88 TB/s against 2.71 for 128-thread blocks.
template <int FORM> __host__ __device__ constexpr int zreg_threads() { return 64; }

// C2R of one line held by TPL lanes (input rows k = t + s*TPL): the pair terms
// X[M-k] come from the partner lane by a warp shuffle (TPL <= 32) or straight
// from global memory (a line spread over several warps; the second read of the
// line hits L1), then the length-M inverse FFT (forward radix schedule) leaves
// the packed real line in registers
// Register layout of a line: with a first radix equal to E (powers of two, and 12), slot
// s of lane t holds row t + s*TPL on input (forward schedule) and on output
// (reversed schedule), and the pair terms X[M-k] sit in the partner lane of the
// same warp (TPL <= 32): warp shuffles.  Otherwise (a line over two warps) the inverse
// reads the pair terms from global memory (L1 hits) and the forward swaps them through
// the line's exchange buffer.
template <int M, int E, int TPL> __host__ __device__ constexpr bool zreg_shfl() {
  return radix_at(M, E, 0) == E && TPL <= 32;
}

// rows of a line into registers (and X[M] on lane t = 0 for the shuffle path);
// issued for every component of a line before any of them is transformed
// (rows above zkeep are zero and not read: two-thirds dealiasing along z)
template <typename T, int M, int E, int TPL>
__device__ __forceinline__ void zreg_load(const C<T>* X, bool live, int t, C<T> (&a)[E], C<T>& XM, int zkeep) {
  typedef C<T> V;
#pragma unroll
  for (int s = 0; s < E; ++s) {
    const int k = load_row<M, E>(t, s);
    a[s] = (live && k <= zkeep) ? X[k] : mk<V>(0, 0);
  }
  XM = (zreg_shfl<M, E, TPL>() && live && t == 0 && M <= zkeep) ? X[M] : mk<V>(0, 0);
}

// C2R of a loaded line (a, XM from zreg_load); the packed real line replaces a
template <typename T, int M, int E, int TPL>
__device__ __forceinline__ void zreg_inverse_loaded(const C<T>* X, bool live, int t, int partner,
                                                    const C<T>* __restrict__ tw, C<T>* xch, C<T> (&a)[E],
                                                    const C<T>& XM, int zkeep) {
  typedef C<T> V;
  V out[E];
#pragma unroll
  for (int s = 0; s < E; ++s) {
    // Z[k] = (X + Y) + i conj(w^k)(X - Y), Y = conj(X[M-k]); imag of X[0], X[M] dropped
    const int k = load_row<M, E>(t, s);
    V b;
    if constexpr (zreg_shfl<M, E, TPL>()) {
      b.x = __shfl_sync(0xffffffffu, a[E - 1 - s].x, partner);
      b.y = __shfl_sync(0xffffffffu, a[E - 1 - s].y, partner);
      if (t == 0) b = (s == 0) ? XM : a[(E - s) % E];
    } else {
      b = (live && M - k <= zkeep) ? X[M - k] : mk<V>(0, 0);
    }
    b = conjg(b);
    V x = a[s];
    if (k == 0) { x.y = 0; b.y = 0; }
    out[s] = add(add(x, b), mul_i<1>(mul(conjg(tw[k]), sub(x, b))));
  }
  fft_regs<M, E, 1, 0, 1, false>(out, t, xch, 1, 0, tw, 2);
#pragma unroll
  for (int s = 0; s < E; ++s) a[s] = out[s];
}

// R2C of one packed real line in registers (reversed radix schedule, so the
// inverse's output order is its input order) and the store of its M+1 rows
template <typename T, int M, int E, int TPL>
__device__ __forceinline__ void zreg_forward_store(C<T> (&p)[E], C<T>* Xo, bool live, int t, int partner,
                                                   const C<T>* __restrict__ tw, C<T>* xch) {
  typedef C<T> V;
  constexpr bool SH = zreg_shfl<M, E, TPL>();
  fft_regs<M, E, -1, 0, 1, true>(p, t, xch, 1, 0, tw, 2);
  // X[k] = 1/2 (Z + Z') - i/2 w^k (Z - Z'), Z' = conj(Z[M-k]), Z[M] = Z[0]
  if constexpr (!SH) {
#pragma unroll
    for (int s = 0; s < E; ++s) xch[prow<1>(final_row<M, E, true>(t, s))] = p[s];
    __syncthreads();
  }
#pragma unroll
  for (int s = 0; s < E; ++s) {
    const int k = final_row<M, E, true>(t, s);
    V zp;
    if constexpr (SH) {
      zp.x = __shfl_sync(0xffffffffu, p[E - 1 - s].x, partner);
      zp.y = __shfl_sync(0xffffffffu, p[E - 1 - s].y, partner);
      if (t == 0) zp = p[(E - s) % E];
    } else {
      zp = xch[prow<1>((M - k) % M)];
    }
    zp = conjg(zp);
    const V z = p[s];
    const V o = add(scale(add(z, zp), (T)0.5), mul_i<-1>(mul(tw[k], scale(sub(z, zp), (T)0.5))));
    if (live) Xo[k] = o;
    if (k == 0 && live) {
      // X[M] = Re Z[0] + Im Z[0] (Z[M] = Z[0])
      const V zc = conjg(z);
      Xo[M] = add(scale(add(z, zc), (T)0.5), mul_i<-1>(mul(tw[M], scale(sub(z, zc), (T)0.5))));
    }
  }
  if constexpr (!SH) __syncthreads();  // the exchange line is reused next
}

// blocks per SM the register z kernel is compiled for: 6 (170 registers), 3 for
// the 12-element lines with a factor 3 (which would spill at 170), 4 for 512-point lines
// (two warps per line, the pair terms through the exchange line; spilled at 170)
// (8 for the 4-element variant)
// (4 for the MHD and flux-giver forms, which hold six lines while they make eight or nine products)
template <int NZ, int EZ = 0, int FORM = 0> __host__ __device__ constexpr int zreg_min_blocks() {
  return EZ == 4 ? 8 : ((NZ / 2) % 3 == 0 ? 3 : ((NZ >= 1024 || FORM == 5 || FORM == 6) ? 4 : 6));
}

// EZ = 0: 8 elements per thread, 12 for a line length with a factor 3 (radices
// 12, 2|4); EZ = 4: 4 elements per thread (twice the lanes per line).
// BATCH: a line over two warps also issues every component's loads before the first
// transform (one load latency per line instead of one per component)
template <typename T, int NZ, int FORM, int EZ = 0, bool BATCH = false>
__global__ void __launch_bounds__(zreg_threads<FORM>(), zreg_min_blocks<NZ, EZ, FORM>())
    k_z_reg(C<T>* P, Geo g, const C<T>* __restrict__ tw, long long msP, int zkeep) {
  chain_begin();
  typedef C<T> V;
  constexpr int M = NZ / 2, H = M + 1, E = EZ ? EZ : ((M % 3 == 0) ? 12 : 8), TPL = M / E, LDX = zslot<M>();
  static_assert(TPL >= 1 && TPL <= 64, "a line spans at most two warps");
  constexpr int NIN = z_nin(FORM), NOUT = z_nout(FORM);
  static_assert(NIN <= 6, "the adjoint form runs in k_z_pair_adj");
  constexpr int LPB = zreg_threads<FORM>() / TPL;
  __shared__ __align__(16) V xch_all[LPB * LDX];
  P += blockIdx.y * msP;  // member blockIdx.y
  const int l = threadIdx.x / TPL, t = threadIdx.x % TPL;
  const int lane = threadIdx.x & 31;
  const int partner = (lane - t) + (TPL - t) % TPL;  // lane holding row M - k
  const long long nlines = (long long)g.Nx * g.Ny;
  const long long line = (long long)blockIdx.x * LPB + l;
  const bool live = line < nlines;
  V* xch = xch_all + l * LDX;

  V in[NIN][E];
  if constexpr (TPL <= 32 || BATCH) {
    // lines within a warp: every component's loads are issued before the first transform
    V XM[NIN];
#pragma unroll
    for (int c = 0; c < NIN; ++c)
      zreg_load<T, M, E, TPL>(P + c * g.S + (live ? line : 0) * H, live, t, in[c], XM[c], zkeep);
#pragma unroll
    for (int c = 0; c < NIN; ++c)
      zreg_inverse_loaded<T, M, E, TPL>(P + c * g.S + (live ? line : 0) * H, live, t, partner, tw, xch, in[c], XM[c],
                                        zkeep);
  } else {
#pragma unroll
    for (int c = 0; c < NIN; ++c) {
      V XM;
      zreg_load<T, M, E, TPL>(P + c * g.S + (live ? line : 0) * H, live, t, in[c], XM, zkeep);
      zreg_inverse_loaded<T, M, E, TPL>(P + c * g.S + (live ? line : 0) * H, live, t, partner, tw, xch, in[c], XM,
                                        zkeep);
    }
  }
  // real-space products; each complex register holds two real points
#pragma unroll
  for (int f = 0; f < NOUT; ++f) {
    V p[E];
#pragma unroll
    for (int s = 0; s < E; ++s) {
      V q[NIN];
#pragma unroll
      for (int c = 0; c < NIN; ++c) q[c] = in[c][s];
      p[s] = z_product<FORM>(f, q);
    }
    zreg_forward_store<T, M, E, TPL>(p, P + f * g.S + (live ? line : 0) * H, live, t, partner, tw, xch);
  }
}

// ---------------------------------------------------------------------------
// z pass, line-pair form: two neighbouring real lines a, b of a component ride in one
// complex transform of the full length N = Nz (z_n = a_n + i b_n), so the real-transform
// pre- and post-processing is additions only:
//   inverse: Z_k = A_k + i B_k, Z_{N-k} = conj(A_k) + i conj(B_k)  (0 < k < M = N/2),
//            Z_0 = Re A_0 + i Re B_0, Z_M = Re A_M + i Re B_M;
//   forward: A_k = (Z_k + conj Z_{N-k}) / 2, B_k = -i (Z_k - conj Z_{N-k}) / 2.
// A pair is held by TPL = N / E lanes, E elements each; the inverse (forward radix
// schedule) leaves the points of every component in the order in which the forward
// transform with the reversed schedule takes them, so the products (re and im: the points
// of the two lines) are formed in registers.  All input components go through each
// exchange together, the products in groups of NB.  A pair within a warp (TPL <= 32)
// needs warp barriers only, and the mirrored rows N - k come from the partner lane by
// shuffles (SH); otherwise they are read again (L1) and, on the way out, taken from the
// exchange line.
// Rounding: both lines carry that of the stronger one (a line of zeros beside another comes out
// as noise of eps times it, and equal lines differ by eps, the modes ky = Ny / 2).  In the norm
// over a field that is the rounding of single lines: the y and x passes mix its lines anyway.
// ---------------------------------------------------------------------------
template <typename T, int NZ, int E> __host__ __device__ constexpr bool zpair_shfl() {
  return radix_at(NZ, E, 0) == E && NZ / E <= 32 && E >= 2;
}
// exchange rows of a pair (prow modes) and the complex values they take
template <typename T> __host__ __device__ constexpr int zpair_pad(int NZ) {
  return sizeof(T) == 4 && NZ >= 128 && NZ % 3 != 0 ? 3 : 2;
}
template <typename T> __host__ __device__ constexpr int zpair_slot(int NZ) { return NZ + NZ / 8; }

// lines of exchange space per pair: the inputs go through it together, the products NB at a time
__host__ __device__ constexpr int zpair_lines(int nin, int nb) { return nin > nb ? nin : nb; }

// the two lines X, X + H (H: line pitch) of NC components (stride cs) as Z rows in registers, rows above zkeep
// zero and not read; every load is issued before any of them is used
template <typename T, int NZ, int E, int NC>
__device__ __forceinline__ void zpair_load(const C<T>* X, int H, long long cs, bool live0, bool live1, int t, int partner,
                                           int zkeep, C<T> (&in)[NC][E]) {
  typedef C<T> V;
  constexpr int M = NZ / 2, TPL = NZ / E;
  if constexpr (zpair_shfl<T, NZ, E>()) {
    // slots s < E/2 hold rows t + s TPL < M, slot E/2 of lane 0 row M
    V a[NC][E / 2], b[NC][E / 2], aM[NC], bM[NC];
#pragma unroll
    for (int c = 0; c < NC; ++c) {
      const V* x = X + c * cs;
#pragma unroll
      for (int s = 0; s < E / 2; ++s) {
        const int k = t + s * TPL;
        a[c][s] = (live0 && k <= zkeep) ? x[k] : mk<V>(0, 0);
        b[c][s] = (live1 && k <= zkeep) ? x[H + k] : mk<V>(0, 0);
      }
      aM[c] = (live0 && t == 0 && M <= zkeep) ? x[M] : mk<V>(0, 0);
      bM[c] = (live1 && t == 0 && M <= zkeep) ? x[H + M] : mk<V>(0, 0);
    }
#pragma unroll
    for (int c = 0; c < NC; ++c) {
      if (t == 0) a[c][0].y = b[c][0].y = 0;
      V w[E / 2];
#pragma unroll
      for (int s = 0; s < E / 2; ++s) {
        in[c][s] = mk<V>(a[c][s].x - b[c][s].y, a[c][s].y + b[c][s].x);
        w[s] = mk<V>(a[c][s].x + b[c][s].y, b[c][s].x - a[c][s].y);  // conj(A) + i conj(B): row N - k
      }
      // slot s >= E/2 of lane t > 0 holds row N - (TPL - t) - (E-1-s) TPL; lane 0 holds row N - (E-s) TPL
#pragma unroll
      for (int s = E / 2; s < E; ++s) {
        V z;
        z.x = __shfl_sync(0xffffffffu, w[E - 1 - s].x, partner);
        z.y = __shfl_sync(0xffffffffu, w[E - 1 - s].y, partner);
        if (t == 0) z = s == E / 2 ? mk<V>(aM[c].x, bM[c].x) : w[(E - s) % (E / 2)];
        in[c][s] = z;
      }
    }
  } else {
#pragma unroll
    for (int c = 0; c < NC; ++c) {
      const V* x = X + c * cs;
#pragma unroll
      for (int s = 0; s < E; ++s) {
        const int r = load_row<NZ, E>(t, s), k = r <= M ? r : NZ - r;
        V a = (live0 && k <= zkeep) ? x[k] : mk<V>(0, 0);
        V b = (live1 && k <= zkeep) ? x[H + k] : mk<V>(0, 0);
        if (k == 0 || k == M) a.y = b.y = 0;
        if (r > M) a.y = -a.y, b.y = -b.y;
        in[c][s] = mk<V>(a.x - b.y, a.y + b.x);
      }
    }
  }
}

// forward transform of NB packed line pairs and the store of their rows 0 .. M
template <typename T, int NZ, int E, int NB>
__device__ __forceinline__ void zpair_forward_store(C<T> (&p)[NB][E], C<T>* X, long long cs, bool live0, bool live1,
                                                    int t, int partner, const C<T>* __restrict__ tw, C<T>* xch,
                                                    int slot) {
  typedef C<T> V;
  constexpr int M = NZ / 2, H = M + 1, TPL = NZ / E;
  constexpr bool WARP = TPL <= 32;
  fft_regs_b<NZ, E, -1, NB, WARP, 0, zpair_pad<T>(NZ), true>(p, t, xch, slot, 1, 0, ct_table<NZ, E, true>(tw));
  if constexpr (zpair_shfl<T, NZ, E>()) {
#pragma unroll
    for (int f = 0; f < NB; ++f) {
      V* Xo = X + f * cs;
#pragma unroll
      for (int s = 0; s < E / 2; ++s) {
        V zp;
        zp.x = __shfl_sync(0xffffffffu, p[f][E - 1 - s].x, partner);
        zp.y = __shfl_sync(0xffffffffu, p[f][E - 1 - s].y, partner);
        if (t == 0) zp = p[f][(E - s) % E];
        const V z = p[f][s];
        const int k = t + s * TPL;
        if (live0) Xo[k] = mk<V>((T)0.5 * (z.x + zp.x), (T)0.5 * (z.y - zp.y));
        if (live1) Xo[H + k] = mk<V>((T)0.5 * (z.y + zp.y), (T)0.5 * (zp.x - z.x));
      }
      if (t == 0) {
        if (live0) Xo[M] = mk<V>(p[f][E / 2].x, (T)0);
        if (live1) Xo[H + M] = mk<V>(p[f][E / 2].y, (T)0);
      }
    }
  } else {
#pragma unroll
    for (int f = 0; f < NB; ++f)
#pragma unroll
      for (int s = 0; s < E; ++s) xch[f * slot + prow<zpair_pad<T>(NZ)>(final_row<NZ, E, true>(t, s))] = p[f][s];
    fft_sync<WARP>();
#pragma unroll
    for (int f = 0; f < NB; ++f) {
      V* Xo = X + f * cs;
      const V* zl = xch + f * slot;
      for (int k = t; k <= M; k += TPL) {
        const V z = zl[prow<zpair_pad<T>(NZ)>(k)], zp = zl[prow<zpair_pad<T>(NZ)>((NZ - k) % NZ)];
        if (live0) Xo[k] = mk<V>((T)0.5 * (z.x + zp.x), (T)0.5 * (z.y - zp.y));
        if (live1) Xo[H + k] = mk<V>((T)0.5 * (z.y + zp.y), (T)0.5 * (zp.x - z.x));
      }
    }
    fft_sync<WARP>();  // the exchange lines are used again by the next group
  }
}

template <typename T, int NZ, int E, int FORM, int NTHR, int MINB, int NB>
__global__ void __launch_bounds__(NTHR, MINB)
    k_z_pair(C<T>* P, Geo g, const C<T>* __restrict__ tw, long long msP, int zkeep, const C<T>* Q,
             const C<T>* X) {
  chain_begin();
  typedef C<T> V;
  constexpr int H = NZ / 2 + 1, TPL = NZ / E, PPB = NTHR / TPL, LDX = zpair_slot<T>(NZ), SLOT = PPB * LDX;
  constexpr int NIN = z_nin(FORM), NOUT = z_nout(FORM);
  constexpr bool WARP = TPL <= 32;
  static_assert(NOUT % NB == 0 && NTHR % TPL == 0 && (!WARP || 32 % TPL == 0), "whole pairs per warp or block");
  extern __shared__ __align__(16) unsigned char smraw[];
  P += blockIdx.y * msP;  // member blockIdx.y
  if (X == nullptr) X = P;
  const int l = threadIdx.x / TPL, t = threadIdx.x % TPL;
  const int lane = threadIdx.x & 31;
  const int partner = (lane - t) + (TPL - t) % TPL;  // lane holding the rows N - k
  const long long nlines = (long long)g.Nx * g.Ny;
  const long long line = 2 * ((long long)blockIdx.x * PPB + l);
  const bool live0 = line < nlines, live1 = line + 1 < nlines;
  V* xch = reinterpret_cast<V*>(smraw) + l * LDX;  // line f of the pair at f * SLOT
  V* Pl = P + (live0 ? line : 0) * H;

  V in[NIN][E];
  if constexpr (FORM == 6) {
    // u from Q (transformed once for all spheres), the giver from P
    const V* Ql = Q + (live0 ? line : 0) * H;
    V a[3][E], b[3][E];
    zpair_load<T, NZ, E, 3>(Ql, H, g.S, live0, live1, t, partner, zkeep, a);
    zpair_load<T, NZ, E, 3>(Pl + 3 * g.S, H, g.S, live0, live1, t, partner, zkeep, b);
#pragma unroll
    for (int c = 0; c < 3; ++c)
#pragma unroll
      for (int s = 0; s < E; ++s) {
        in[c][s] = a[c][s];
        in[c + 3][s] = b[c][s];
      }
  } else {
    zpair_load<T, NZ, E, NIN>(X + (live0 ? line : 0) * g.Hp, g.Hp, g.Sp, live0, live1, t, partner, zkeep, in);
  }
  fft_regs_b<NZ, E, 1, NIN, WARP, 0, zpair_pad<T>(NZ), false>(in, t, xch, SLOT, 1, 0, ct_table<NZ, E, false>(tw));
#pragma unroll
  for (int f0 = 0; f0 < NOUT; f0 += NB) {
    V p[NB][E];
#pragma unroll
    for (int s = 0; s < E; ++s)
#pragma unroll
      for (int f = 0; f < NB; ++f) {
        V q[NIN];
#pragma unroll
        for (int c = 0; c < NIN; ++c) q[c] = in[c][s];
        p[f][s] = z_product<FORM>(f0 + f, q);
      }
    zpair_forward_store<T, NZ, E, NB>(p, Pl + f0 * g.S, g.S, live0, live1, t, partner, tw, xch, SLOT);
  }
}

// z pass of the adjoint right-hand side on line pairs: inputs u (components 0-2), w (3-5),
// mu (6-8); mu x u into components 0-2 and w x mu into 3-5.  The points of mu wait in shared
// memory (each thread reads back only its own), so one vector and one product are in
// registers at a time.
template <typename T, int NZ, int E, int NTHR, int MINB>
__global__ void __launch_bounds__(NTHR, MINB)
    k_z_pair_adj(C<T>* P, Geo g, const C<T>* __restrict__ tw, int zkeep) {
  chain_begin();
  typedef C<T> V;
  constexpr int M = NZ / 2, H = M + 1, TPL = NZ / E, PPB = NTHR / TPL, LDX = zpair_slot<T>(NZ), SLOT = PPB * LDX;
  constexpr bool WARP = TPL <= 32;
  extern __shared__ __align__(16) unsigned char smraw[];
  const int l = threadIdx.x / TPL, t = threadIdx.x % TPL;
  const int lane = threadIdx.x & 31;
  const int partner = (lane - t) + (TPL - t) % TPL;
  const long long nlines = (long long)g.Nx * g.Ny;
  const long long line = 2 * ((long long)blockIdx.x * PPB + l);
  const bool live0 = line < nlines, live1 = line + 1 < nlines;
  V* xch = reinterpret_cast<V*>(smraw) + l * LDX;  // line f of the pair at f * SLOT
  V* mus = reinterpret_cast<V*>(smraw) + PPB * (3 * LDX) + threadIdx.x;  // slot (f, s) at (f E + s) NTHR
  V* Pl = P + (live0 ? line : 0) * H;
  V in[3][E];
  zpair_load<T, NZ, E, 3>(Pl + 6 * g.S, H, g.S, live0, live1, t, partner, M, in);
  fft_regs_b<NZ, E, 1, 3, WARP, 0, zpair_pad<T>(NZ), false>(in, t, xch, SLOT, 1, 0, ct_table<NZ, E, false>(tw));
#pragma unroll
  for (int f = 0; f < 3; ++f)
#pragma unroll
    for (int s = 0; s < E; ++s) mus[(f * E + s) * NTHR] = in[f][s];
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    zpair_load<T, NZ, E, 3>(Pl + 3 * h * g.S, H, g.S, live0, live1, t, partner, zkeep, in);
    fft_regs_b<NZ, E, 1, 3, WARP, 0, zpair_pad<T>(NZ), false>(in, t, xch, SLOT, 1, 0, ct_table<NZ, E, false>(tw));
#pragma unroll
    for (int f = 0; f < 3; ++f) {
      V p[1][E];
#pragma unroll
      for (int s = 0; s < E; ++s) {
        const int i = f == 2 ? 0 : f + 1, j = f == 0 ? 2 : f - 1;
        const V a = h == 0 ? mus[(i * E + s) * NTHR] : in[i][s], b = h == 0 ? in[j][s] : mus[(j * E + s) * NTHR];
        const V c = h == 0 ? mus[(j * E + s) * NTHR] : in[j][s], d = h == 0 ? in[i][s] : mus[(i * E + s) * NTHR];
        p[0][s] = mk<V>(a.x * b.x - c.x * d.x, a.y * b.y - c.y * d.y);
      }
      zpair_forward_store<T, NZ, E, 1>(p, Pl + (3 * h + f) * g.S, g.S, live0, live1, t, partner, tw, xch, SLOT);
    }
  }
}

// ---------------------------------------------------------------------------
// SSS z pass, line-pair form: two neighbouring real lines a, b of a component as one
// complex line p = a + i b.  The sin/cos transform of complex data is the algorithm of the
// x / y passes (one complex FFT of the full length N with the quarter-step twiddles
// w_m = e^{-i pi m / 2N}):
//   inverse: V_m = conj(w_m) (p_m - i p_{N-m}) (cosine, V_0 = p_0), conj(w_m) (p_{N-m} - i p_m)
//            (sine, V_0 = 0); inverse FFT, points left in the reordered order v;
//   forward: Z = FFT(v); p_m = scl (w_m Z_m + conj(w_m) Z_{N-m}) (cosine),
//            i scl (w_m Z_m - conj(w_m) Z_{N-m}) (sine).
// Lines, registers, exchanges, mirrored rows and products as in k_z_pair; the product of two
// reordered lines is the reordered product with the product's own sign pattern (sine x sine =
// cosine, sine x cosine = sine, and the sign flips multiply), so the forward transform takes
// it as it is.  zin / zout: bit c set = input / output c is a sine series along z;
// scl = 1 / (2N).
// ---------------------------------------------------------------------------
template <typename T, int NZ, int E, int FORM, int NTHR, int MINB, int NB>
__global__ void __launch_bounds__(NTHR, MINB)
    k_sss_z_pair(C<T>* P, Geo g, const C<T>* __restrict__ tw, const C<T>* __restrict__ tq, int zin,
                 int zout, T scl) {
  chain_begin();
  typedef C<T> V;
  constexpr int H = NZ / 2 + 1, LD = NZ + 2, TPL = NZ / E, PPB = NTHR / TPL, LDX = zpair_slot<T>(NZ), SLOT = PPB * LDX;
  constexpr int NIN = z_nin(FORM), NOUT = z_nout(FORM);
  constexpr bool WARP = TPL <= 32, SH = zpair_shfl<T, NZ, E>();
  static_assert(FORM == 7 || FORM == 2 || FORM == 6, "conservative products, with or without T, or the flux giver's");
  static_assert(NOUT % NB == 0 && NTHR % TPL == 0, "whole pairs per block");
  extern __shared__ __align__(16) unsigned char smraw[];
  const int l = threadIdx.x / TPL, t = threadIdx.x % TPL;
  const int lane = threadIdx.x & 31;
  const int partner = (lane - t) + (TPL - t) % TPL;  // lane holding the rows N - m (SH)
  const long long nlines = (long long)g.Nx * g.Ny;
  const long long line = 2 * ((long long)blockIdx.x * PPB + l);
  const bool live0 = line < nlines, live1 = line + 1 < nlines;
  V* xch = reinterpret_cast<V*>(smraw) + l * LDX;  // line f of the pair at f * SLOT
  T* Pl = reinterpret_cast<T*>(P + (live0 ? line : 0) * H);  // line a; line b follows at Pl + LD

  V in[NIN][E];
#pragma unroll
  for (int c = 0; c < NIN; ++c) {
    const T* X = Pl + 2 * c * g.S;
#pragma unroll
    for (int s = 0; s < E; ++s) {
      const int m = load_row<NZ, E>(t, s);
      in[c][s] = mk<V>(live0 ? X[m] : (T)0, live1 ? X[LD + m] : (T)0);
    }
  }
#pragma unroll
  for (int c = 0; c < NIN; ++c) {
    const bool sine = (zin >> c) & 1;
    V q[E];  // p_{N-m}
#pragma unroll
    for (int s = 0; s < E; ++s) {
      if constexpr (SH) {
        q[s].x = __shfl_sync(0xffffffffu, in[c][E - 1 - s].x, partner);
        q[s].y = __shfl_sync(0xffffffffu, in[c][E - 1 - s].y, partner);
        if (t == 0) q[s] = in[c][(E - s) % E];
      } else {
        const T* X = Pl + 2 * c * g.S;
        const int m = load_row<NZ, E>(t, s);
        q[s] = m == 0 ? mk<V>(0, 0) : mk<V>(live0 ? X[NZ - m] : (T)0, live1 ? X[LD + NZ - m] : (T)0);
      }
    }
#pragma unroll
    for (int s = 0; s < E; ++s) {
      const int m = load_row<NZ, E>(t, s);
      const V p = in[c][s];
      if (m == 0) in[c][s] = sine ? mk<V>(0, 0) : p;
      else in[c][s] = mul(conjg(tq[m]), sine ? add_i<-1>(q[s], p) : add_i<-1>(p, q[s]));
    }
  }
  fft_regs_b<NZ, E, 1, NIN, WARP, 0, zpair_pad<T>(NZ), false>(in, t, xch, SLOT, 1, 0, ct_table<NZ, E, false>(tw));
#pragma unroll
  for (int f0 = 0; f0 < NOUT; f0 += NB) {
    V p[NB][E];
#pragma unroll
    for (int s = 0; s < E; ++s)
#pragma unroll
      for (int f = 0; f < NB; ++f) {
        V q[NIN];
#pragma unroll
        for (int c = 0; c < NIN; ++c) q[c] = in[c][s];
        p[f][s] = z_product<FORM>(f0 + f, q);
      }
    fft_regs_b<NZ, E, -1, NB, WARP, 0, zpair_pad<T>(NZ), true>(p, t, xch, SLOT, 1, 0, ct_table<NZ, E, true>(tw));
    if constexpr (!SH) {
#pragma unroll
      for (int f = 0; f < NB; ++f)
#pragma unroll
        for (int s = 0; s < E; ++s) xch[f * SLOT + prow<zpair_pad<T>(NZ)>(final_row<NZ, E, true>(t, s))] = p[f][s];
      fft_sync<WARP>();
    }
#pragma unroll
    for (int f = 0; f < NB; ++f) {
      const bool sine = (zout >> (f0 + f)) & 1;
      T* Xo = Pl + 2 * (f0 + f) * g.S;
#pragma unroll
      for (int s = 0; s < E; ++s) {
        const int m = final_row<NZ, E, true>(t, s);
        V zr;
        if constexpr (SH) {
          zr.x = __shfl_sync(0xffffffffu, p[f][E - 1 - s].x, partner);
          zr.y = __shfl_sync(0xffffffffu, p[f][E - 1 - s].y, partner);
          if (t == 0) zr = p[f][(E - s) % E];
        } else {
          zr = xch[f * SLOT + prow<zpair_pad<T>(NZ)>((NZ - m) % NZ)];
        }
        const V w = tq[m], wz = mul(w, p[f][s]), wzr = mul(conjg(w), zr);
        const V o = sine ? mul_i<1>(scale(sub(wz, wzr), scl)) : scale(add(wz, wzr), scl);
        if (live0) Xo[m] = o.x;
        if (live1) Xo[LD + m] = o.y;
      }
      if (t < 2) {  // the two padding reals
        if (live0) Xo[NZ + t] = (T)0;
        if (live1) Xo[LD + NZ + t] = (T)0;
      }
    }
    if constexpr (!SH) fft_sync<WARP>();  // the exchange lines are used again by the next group
  }
}

// ---------------------------------------------------------------------------
// forward x pass + spectral epilogue
// ---------------------------------------------------------------------------
struct StageArgs {
  void* U0;          // state (Vcopy); MODE_ADJ: the adjoint state Lam, overwritten at stage 1
  void* Uout;        // MODE_STEP: where stage 4 writes the new state (U0 for an in-place step)
  void* Ucur;        // stage field; MODE_ADJ: the next stage's cotangent lam
  void* tot;         // RK accumulator; MODE_ADJ: the adjoint accumulator
  void* nout;        // MODE_NLIN: output N (3 comps)
  const void* Ud;    // MODE_FLUX: field whose dealiased copy multiplies N
  double* bins;      // MODE_FLUX: nradii + 1 sums, then per-block partial sums, nradii + 1 per block
  const double* radii;
  int nradii;
  const void* fcube; // force cube (3 comps of (2km+1)^2 (km+1)), nullptr = no force
  int fkm;
  double nu, dt;
  int stage;         // 1..4
  int reality;       // zero the kz = Nz/2 plane at the end of stage 4
  int* err;          // set to 1 when a bounded wait gives up
  const double* ex;  // per-axis integrating factors exp(-nu dt K_i^2 / 2), FP64
  const double* ey;
  const double* ez;
  const float2* exf; // the same as FP32 (hi, lo) pairs (nullptr: split the FP64 product)
  const float2* eyf;
  const float2* ezf;
};

enum { MODE_STEP = 0, MODE_FLUX = 1, MODE_NLIN = 2, MODE_ADJ = 3 };
// MODE_FLUX: at most FLUX_MAX_BINS - 1 radii (each thread keeps one FP64 partial per sphere)
constexpr int FLUX_MAX_BINS = 64;

// Assembly of the stage's spectral vector from forward-transformed product f
// (p already scaled by 1/(Nx Ny Nz)):
//   FORM 0: N_i = sum_j i K_j F[u_i u_j]  (compute_diag_offdiag.cc:47-98)
//   FORM 7: the same from d2, d3, u1u2, u2u3, u3u1 (N up to a gradient, for a step)
//   FORM 1: N = -F[u x omega]
//   FORM 3: A_i + (i K x B)_i  (adjoint; B = products 0-2, A = products 3-5)
template <int FORM, typename V, typename S>
__device__ __forceinline__ void accum_product(int f, V p, S Kx, S Ky, S Kz, V& a0, V& a1, V& a2) {
  if (FORM == 0) {
    switch (f) {
      case 0: a0 = add(a0, ik(Kx, p)); break;
      case 1: a1 = add(a1, ik(Ky, p)); break;
      case 2: a2 = add(a2, ik(Kz, p)); break;
      case 3: a0 = add(a0, ik(Ky, p)); a1 = add(a1, ik(Kx, p)); break;
      case 4: a1 = add(a1, ik(Kz, p)); a2 = add(a2, ik(Ky, p)); break;
      default: a2 = add(a2, ik(Kx, p)); a0 = add(a0, ik(Kz, p)); break;
    }
  } else if (FORM == 7) {
    switch (f) {
      case 0: a1 = add(a1, ik(Ky, p)); break;
      case 1: a2 = add(a2, ik(Kz, p)); break;
      case 2: a0 = add(a0, ik(Ky, p)); a1 = add(a1, ik(Kx, p)); break;
      case 3: a1 = add(a1, ik(Kz, p)); a2 = add(a2, ik(Ky, p)); break;
      default: a2 = add(a2, ik(Kx, p)); a0 = add(a0, ik(Kz, p)); break;
    }
  } else if (FORM == 3) {
    switch (f) {
      case 0: a1 = add(a1, ik(Kz, p)); a2 = sub(a2, ik(Ky, p)); break;
      case 1: a2 = add(a2, ik(Kx, p)); a0 = sub(a0, ik(Kz, p)); break;
      case 2: a0 = add(a0, ik(Ky, p)); a1 = sub(a1, ik(Kx, p)); break;
      case 3: a0 = add(a0, p); break;
      case 4: a1 = add(a1, p); break;
      default: a2 = add(a2, p); break;
    }
  } else {
    if (f == 0) a0 = scale(p, (S)-1);
    else if (f == 1) a1 = scale(p, (S)-1);
    else a2 = scale(p, (S)-1);
  }
}

// ey[ly] ez[lz] from the FP32 pair tables (once per column), for the FP32 step
template <typename T, int MODE>
__device__ __forceinline__ Fac<float> col_pair(const StageArgs& a, int ly, int lz) {
  if constexpr (std::is_same<T, float>::value && MODE == MODE_STEP) {
    if (a.exf) return pair_mul(a.eyf[ly], a.ezf[lz]);
  }
  return Fac<float>{1.0f, 0.0f};
}

// Per-mode epilogue of a right-hand side at spectral element (lx, ly, lz),
// linear offset `off` in a component.  N1..N3 = the assembled vector; the
// state the mode reads comes from st0[i * sstr] (U0 / Lam / the flux field)
// and st1[i * sstr] (tot / the adjoint accumulator), i = component; the
// fused x kernel passes its shared-memory state tiles, the elementwise
// epilogue kernel the global arrays.  exy = ey[ly] ez[lz] (MODE_STEP, MODE_ADJ); pexy = the
// same product from the FP32 pair tables (FP32 MODE_STEP with a.exf; see col_pair).
template <typename T, int MODE>
__device__ __forceinline__ void spec_epilogue(const Geo& g, const StageArgs& a, int lx, int ly, int lz,
                                              long long off, double exy, Fac<float> pexy, C<T> N1, C<T> N2,
                                              C<T> N3, const C<T>* st0, const C<T>* st1, long long sstr,
                                              double* sbins) {
  typedef C<T> V;
  const int kx = kfft(lx, g.Nx), ky = kfft(ly, g.Ny);
  const double Kxd = kx * g.kf[0], Kyd = ky * g.kf[1], Kzd = lz * g.kf[2];
  if (MODE == MODE_NLIN) {
    V* no = reinterpret_cast<V*>(a.nout);
    no[off] = N1; no[g.S + off] = N2; no[2 * g.S + off] = N3;
    return;
  }
  if (MODE == MODE_FLUX) {
    // contribution 2 mult Re(N . conj(D(U))) to the first sphere with |K| <= R
    if (dealias_zero(g.dealias, g.basis, lx, ly, lz, g.Nx, g.Ny, g.Nz)) return;
    const V u1 = st0[0], u2 = st0[sstr], u3 = st0[2 * sstr];
    double re = (double)N1.x * u1.x + (double)N1.y * u1.y + (double)N2.x * u2.x + (double)N2.y * u2.y +
                (double)N3.x * u3.x + (double)N3.y * u3.y;
    double mult = lz > 0 ? 1.0 : 0.5;
    if (kx == g.Nx / 2 || (ky == g.Ny / 2 && g.Ny > 1)) mult *= 2;
    const double Kmag = sqrt((Kxd * Kxd + Kyd * Kyd) + Kzd * Kzd);
    int b = 0;
    while (b < a.nradii && Kmag > a.radii[b]) ++b;
    sbins[b] += 2.0 * mult * re;  // the calling thread's own partials, in a fixed element order
    return;
  }
  if (MODE == MODE_ADJ) {
    const double eh = a.ex[lx] * exy;
    const double e1 = eh * eh;
    const T Eh = (T)eh, E1 = (T)e1;
    const bool dz = dealias_zero(g.dealias, g.basis, lx, ly, lz, g.Nx, g.Ny, g.Nz);
    const T cw = dz ? (T)0 : ((lz > 0 && 2 * lz < g.Nz) ? (T)2 : (T)1);
    V* Lm = reinterpret_cast<V*>(a.U0);
    V* lam = reinterpret_cast<V*>(a.Ucur);
    V* Ac = reinterpret_cast<V*>(a.tot);
    const V Wv[3] = {scale(N1, cw), scale(N2, cw), scale(N3, cw)};
#pragma unroll
    for (int i = 0; i < 3; ++i) {
      const long long o = i * g.S + off;
      const V W = Wv[i];
      if (a.stage == 4) {
        const V Lv = st0[i * sstr];
        Ac[o] = add(scale(Lv, E1), scale(W, E1));
        lam[o] = add(scale(Lv, (T)(a.dt / 3 * eh)), scale(W, (T)(a.dt * eh)));
      } else if (a.stage == 1) {
        Lm[o] = add(st1[i * sstr], W);
      } else {
        const V Lv = st0[i * sstr], Acc = st1[i * sstr];
        Ac[o] = add(Acc, scale(W, Eh));
        lam[o] = a.stage == 3 ? add(scale(Lv, (T)(a.dt / 3 * eh)), scale(W, (T)(0.5 * a.dt)))
                              : add(scale(Lv, (T)(a.dt / 6 * e1)), scale(W, (T)(0.5 * a.dt * eh)));
      }
    }
    return;
  }
  // ---- MODE_STEP ----
  const T Kx = (T)Kxd, Ky = (T)Kyd, Kz = (T)Kzd;
  if (a.fcube) {
    const int km = a.fkm;
    if (abs(kx) <= km && abs(ky) <= km && lz <= km) {
      const V* fc = reinterpret_cast<const V*>(a.fcube);
      const int n = 2 * km + 1;
      const long long fo = ((long long)(kx + km) * n + (ky + km)) * (km + 1) + lz;
      const long long fs = (long long)n * n * (km + 1);
      N1 = sub(N1, fc[fo]); N2 = sub(N2, fc[fs + fo]); N3 = sub(N3, fc[2 * fs + fo]);  // Add_force
    }
  }
  // Leray projection: p = (i K . N)/K^2, p(0)=0; N <- -(N + i K p)
  const double K2 = (Kxd * Kxd + Kyd * Kyd) + Kzd * Kzd;
  const V div = add(add(ik(Kx, N1), ik(Ky, N2)), ik(Kz, N3));
  const V pr = (K2 > 0) ? mk<V>(div.x / (T)K2, div.y / (T)K2) : mk<V>(0, 0);
  const V Rv[3] = {scale(add(N1, ik(Kx, pr)), (T)-1), scale(add(N2, ik(Ky, pr)), (T)-1),
                   scale(add(N3, ik(Kz, pr)), (T)-1)};
  // integrating factors (FP64): E(1/2) = ex ey ez = exp(-nu dt K^2 / 2), E(1) = E(1/2)^2
  Fac<T> Feh, Fe1;
  if constexpr (std::is_same<T, float>::value) {
    if (a.exf) {
      // E(1/2) = ex ey ez and E(1) = E(1/2)^2 as FP32 pair products (about 46 bits; no
      // FP64 operation or conversion per mode)
      Feh = pair_mul(a.exf[lx], pexy);
      Fe1 = pair_mul(Feh, Feh);
    } else {
      const double eh = a.ex[lx] * exy;
      Feh = fac<T>(eh);
      Fe1 = fac<T>(eh * eh);
    }
  } else {
    const double eh = a.ex[lx] * exy;
    Feh = fac<T>(eh);
    Fe1 = fac<T>(eh * eh);
  }
  const Fac<T> Fc1 = fac<T>(a.dt), Fc2 = fac<T>(0.5 * a.dt), Fc3 = fac<T>((1.0 / 3) * a.dt),
               Fc6 = fac<T>((1.0 / 6) * a.dt);
  V* Uc = reinterpret_cast<V*>(a.Ucur);
  V* tot = reinterpret_cast<V*>(a.tot);
  const bool dz = dealias_zero(g.dealias, g.basis, lx, ly, lz, g.Nx, g.Ny, g.Nz);
  // IF-RK4 stage update (RK.cc:91-170 with Single_time_step / Compute_RK4_parts)
#pragma unroll
  for (int i = 0; i < 3; ++i) {
    const long long o = i * g.S + off;
    const V R = Rv[i];
    const V u0 = st0[i * sstr];
    if (a.stage == 1) {
      Uc[o] = rk_u1_c(dz ? mk<V>(0, 0) : u0, R, Feh, Fc2);
      tot[o] = rk_t1_c(R, Fe1, Fc6);
    } else {
      const V tt = st1[i * sstr];
      if (a.stage == 2) {
        Uc[o] = rk_u2_c(u0, R, Feh, Fc2);
        tot[o] = rk_tacc_c(tt, R, Feh, Fc3);
      } else if (a.stage == 3) {
        Uc[o] = rk_u3_c(u0, R, Feh, Fc1);
        tot[o] = rk_tacc_c(tt, R, Feh, Fc3);
      } else {
        const V un = rk_u4_c(u0, tt, R, Fe1, Fc6);
        reinterpret_cast<V*>(a.Uout)[o] = (a.reality && lz == g.Nz / 2) ? mk<V>(0, 0) : un;
        health_mark(nonfinite(un), a.err);
      }
    }
  }
}

// Persistent over column tiles.  Thread 0 streams the product fields of a tile
// through two TMA staging tiles (item = (tile, field); item i+2 is issued as
// soon as every thread has read item i), and the RK state the epilogue needs
// (U0 and tot, or the flux field) into six state tiles at tile start.
// Shared memory: 2 product tiles + 1 exchange tile + 6 state tiles (+ flux bins).
//
// FORM 3 / MODE_ADJ (discrete adjoint of the rotational stage; products
// B = F(mu x u) in fields 0-2 and A = F(w x mu) in 3-5):
//   W = D c (A + i K x B)  = the cotangent of the stage input, and with
//   L = Lam (state tiles 0-2), Acc = tot (tiles 3-5), lam = Ucur:
//   stage 4: Acc = E1 L + E1 W,  lam = dt/3 Eh L + dt Eh W
//   stage 3: Acc += Eh W,        lam = dt/3 Eh L + dt/2 W
//   stage 2: Acc += Eh W,        lam = dt/6 E1 L + dt/2 Eh W
//   stage 1: Lam = Acc + W
template <typename T, int L, int E, int CW, int FORM, int MODE>
__global__ void __launch_bounds__(CW * (L / E), 1)
    k_fwd_x(const __grid_constant__ CUtensorMap mP, const __grid_constant__ CUtensorMap mA,
            const __grid_constant__ CUtensorMap mB, Geo g, StageArgs a, const C<T>* __restrict__ tw) {
  chain_begin();
  typedef C<T> V;
  constexpr int NF = z_nout(FORM);
  constexpr int TILE = L * CW, BR = L < 256 ? L : 256, UNITS = (int)sizeof(V) / 8;
  constexpr int NST = MODE == MODE_NLIN ? 0 : 6;
  extern __shared__ __align__(128) unsigned char smraw_[];
  // TMA destinations: 128-byte aligned (the launcher adds 128 bytes of slack)
  unsigned char* smraw = smraw_ + ((128 - (smem_u32(smraw_) & 127)) & 127);
  V* pst = reinterpret_cast<V*>(smraw);
  V* xch = pst + 2 * TILE;              // exchange tile, row pitch CW (L x (CW + 1) reserved)
  V* sst = xch + L * (CW + 1);
  // MODE_FLUX: per-thread FP64 partials of the spheres (thread-local, fixed element order;
  // summed over the block by block_sum and over blocks by k_bins_finish: reproducible)
  double tb[MODE == MODE_FLUX ? FLUX_MAX_BINS : 1];
  __shared__ __align__(8) uint64_t bar[3];  // product slots 0, 1; state
  const int c = threadIdx.x % CW, t = threadIdx.x / CW;
  const int inner = g.Ny * g.Hz;
  const int ntiles = (inner + CW - 1) / CW;
  const long long rstride = inner;
  const T inv = (T)(1.0 / ((double)g.Nx * g.Ny * g.Nz));
  // state tiles: [0,3) = U0 (or the flux field) from map mA, [3,6) = tot from map mB;
  // tiles [sfirst, nstate) are loaded
  const int nstate = MODE == MODE_FLUX ? 3
                     : (MODE == MODE_STEP ? (a.stage == 1 ? 3 : 6) : (MODE == MODE_ADJ ? (a.stage == 4 ? 3 : 6) : 0));
  const int sfirst = (MODE == MODE_ADJ && a.stage == 1) ? 3 : 0;

  if (MODE == MODE_FLUX)
    for (int i = 0; i <= a.nradii; ++i) tb[i] = 0.0;
  if (threadIdx.x == 0) {
    for (int i = 0; i < 3; ++i) mbar_init(&bar[i], 1);
    fence_mbar_init();
  }
  __syncthreads();
  const long long nitems = (long long)NF * ((ntiles - blockIdx.x + gridDim.x - 1) / gridDim.x);
  auto issue_item = [&](long long i) {
    if (i >= nitems) return;
    const int tile = blockIdx.x + (int)(i / NF) * gridDim.x, f = (int)(i % NF), slot = (int)(i & 1);
    mbar_expect_tx(&bar[slot], (unsigned)TILE * (unsigned)sizeof(V));
    for (int r0 = 0; r0 < L; r0 += BR)
      tma_load_2d(pst + slot * TILE + r0 * CW, &mP, tile * CW * UNITS, f * g.Nx + r0, &bar[slot]);
  };
  auto issue_state = [&](int tile) {
    if (nstate == 0) return;
    mbar_expect_tx(&bar[2], (unsigned)(nstate - sfirst) * TILE * (unsigned)sizeof(V));
    for (int comp = sfirst; comp < nstate; ++comp)
      for (int r0 = 0; r0 < L; r0 += BR)
        tma_load_2d(sst + comp * TILE + r0 * CW, comp < 3 ? &mA : &mB, tile * CW * UNITS, (comp % 3) * g.Nx + r0,
                    &bar[2]);
  };
  if (threadIdx.x == 0) {
    issue_item(0);
    issue_item(1);
  }
  // mbarrier phases of the two product slots and the state barrier (scalars:
  // a runtime-indexed array would live in local memory)
  uint32_t ph0 = 0, ph1 = 0, phs = 0;
  long long item = 0;
  // after a wait gave up: a second bounded wait on every copy still in flight (the
  // product items `item` and item + 1, and this tile's state tiles if pending), so no
  // bulk copy lands in the shared memory of a block that has left
  auto drain = [&](bool state_pending) {
    if (threadIdx.x != 0) return;
    for (long long i = item; i < item + 2 && i < nitems; ++i) mbar_wait(&bar[i & 1], (i & 1) ? ph1 : ph0, nullptr);
    if (state_pending) mbar_wait(&bar[2], phs, nullptr);
  };
  for (int tile = blockIdx.x; tile < ntiles; tile += gridDim.x) {
    if (threadIdx.x == 0) issue_state(tile);
    const int col = tile * CW + c;
    const bool ok = col < inner;
    const int ly = ok ? col / g.Hz : 0, lz = ok ? col % g.Hz : 0;
    const int ky = kfft(ly, g.Ny);
    const double Kyd = ky * g.kf[1], Kzd = lz * g.kf[2];
    const T Ky = (T)Kyd, Kz = (T)Kzd;

    V acc[3][E];
#pragma unroll
    for (int i = 0; i < 3; ++i)
#pragma unroll
      for (int s = 0; s < E; ++s) acc[i][s] = mk<V>(0, 0);

    for (int f = 0; f < NF; ++f, ++item) {
      const int slot = (int)(item & 1);
      const uint32_t phase = slot ? ph1 : ph0;
      const bool got = mbar_wait(&bar[slot], phase, a.err);
      if (__syncthreads_or(!got)) {
        drain(nstate > 0);
        return;
      }
      if (slot) ph1 ^= 1;
      else ph0 ^= 1;
      V v[E];
      const V* st = pst + slot * TILE + c;
#pragma unroll
      for (int s = 0; s < E; ++s) v[s] = ok ? st[load_row<L, E>(t, s) * CW] : mk<V>(0, 0);
      __syncthreads();
      if (threadIdx.x == 0) issue_item(item + 2);
      // exchange rows of pitch CW with the modelled best row swizzle (at 4
      // elements and 8 columns: bit 0 flipped by bit 2, since the first pass stores
      // rows 4 apart from neighbouring threads; 1.0x the minimum wavefronts against
      // 2.0x with the earlier padded pitch CW + 1)
      fft_regs<L, E, -1, 0, 0, false, best_swk(L, E, CW, (int)sizeof(V))>(v, t, xch, CW, c, tw, 1);
#pragma unroll
      for (int s = 0; s < E; ++s) {
        const int lx = final_row<L, E>(t, s);
        const T Kx = (T)(kfft(lx, g.Nx) * g.kf[0]);
        const V p = scale(v[s], inv);
        accum_product<FORM>(f, p, Kx, Ky, Kz, acc[0][s], acc[1][s], acc[2][s]);
      }
    }
    if (nstate) {
      const bool got = mbar_wait(&bar[2], phs, a.err);
      if (__syncthreads_or(!got)) {
        drain(true);
        return;
      }
      phs ^= 1;
    }
    if (ok) {
      const double exy = (MODE == MODE_STEP || MODE == MODE_ADJ) ? a.ey[ly] * a.ez[lz] : 0.0;
      const Fac<float> pexy = col_pair<T, MODE>(a, ly, lz);
#pragma unroll
      for (int s = 0; s < E; ++s) {
        const int lx = final_row<L, E>(t, s);
        const long long off = lx * rstride + col;
        const int so = lx * CW + c;
        spec_epilogue<T, MODE>(g, a, lx, ly, lz, off, exy, pexy, acc[0][s], acc[1][s], acc[2][s], sst + so,
                               sst + 3 * TILE + so, TILE, tb);
      }
    }
    // the next tile's state load overwrites the state tiles
    __syncthreads();
  }
  if (MODE == MODE_FLUX) {
    for (int i = 0; i <= a.nradii; ++i) {
      const double v = block_sum(tb[i]);
      if (threadIdx.x == 0) a.bins[(long long)(blockIdx.x + 1) * (a.nradii + 1) + i] = v;
    }
  }
}

// Stage update of one mode of an IF-RK4 step from its unscaled transforms p (FORM 1, 7), the
// arithmetic of spec_epilogue with the projection folded into the assembly:
//   FORM 1: N = -inv p,        R = -(N - K (K.N) / K^2) = inv (p - K (K.p) / K^2)
//   FORM 7: N = i inv m, m_i = sum_j K_j p_ij,        R = -i inv (m - K (K.m) / K^2)
// (inv is a power of two: every FFF axis is).  STAGE is known at compile time, rK2 = 1 / K^2
// (0 at K = 0), fc the force of the mode (zero outside the band).
template <typename T, int FORM, int STAGE>
__device__ __forceinline__ void step_mode(const C<T>* p, const T (&K)[3], Recip<T> rK2, T inv, const C<T>* fc, bool dz,
                                          bool clear, Fac<T> Feh, Fac<T> Fe1, const Fac<T> (&Fc)[4], const C<T>* u0,
                                          const C<T>* tt, C<T>* Uc, C<T>* tot, C<T>* Uo, long long off, long long S,
                                          int* err) {
  typedef C<T> V;
  V m[3];
  if constexpr (FORM == 1) {
    m[0] = p[0]; m[1] = p[1]; m[2] = p[2];
  } else {
    m[0] = add(scale(p[2], K[1]), scale(p[4], K[2]));
    m[1] = add(add(scale(p[2], K[0]), scale(p[0], K[1])), scale(p[3], K[2]));
    m[2] = add(add(scale(p[4], K[0]), scale(p[3], K[1])), scale(p[1], K[2]));
  }
  if (fc) {
    // N - F: with N = -inv m (FORM 1) m + F / inv, with N = i inv m (FORM 7) m + i F / inv
    const T w = (T)1 / inv;
#pragma unroll
    for (int i = 0; i < 3; ++i) m[i] = FORM == 1 ? add(m[i], scale(fc[i], w)) : add_i<1>(m[i], scale(fc[i], w));
  }
  V d = mk<V>(K[0] * m[0].x + K[1] * m[1].x + K[2] * m[2].x, K[0] * m[0].y + K[1] * m[1].y + K[2] * m[2].y);
  d = quot(d, rK2);
#pragma unroll
  for (int i = 0; i < 3; ++i) {
    const V r = mk<V>((m[i].x - K[i] * d.x) * inv, (m[i].y - K[i] * d.y) * inv);
    const V R = FORM == 1 ? r : mk<V>(r.y, -r.x);
    const long long o = off + i * S;
    if constexpr (STAGE == 1) {
      Uc[o] = rk_u1_c(dz ? mk<V>(0, 0) : u0[i], R, Feh, Fc[1]);
      tot[o] = rk_t1_c(R, Fe1, Fc[3]);
    } else if constexpr (STAGE == 2) {
      Uc[o] = rk_u2_c(u0[i], R, Feh, Fc[1]);
      tot[o] = rk_tacc_c(tt[i], R, Feh, Fc[2]);
    } else if constexpr (STAGE == 3) {
      Uc[o] = rk_u3_c(u0[i], R, Feh, Fc[0]);
      tot[o] = rk_tacc_c(tt[i], R, Feh, Fc[2]);
    } else {
      const V un = rk_u4_c(u0[i], tt[i], R, Fe1, Fc[3]);
      Uo[o] = clear ? mk<V>(0, 0) : un;
      health_mark(nonfinite(un), err);
    }
  }
}

// ---------------------------------------------------------------------------
// forward x pass + epilogue of a step, pipelined form: persistent over column tiles of L x CW.
// The NF product fields of a tile sit in shared memory; NF groups of CW * (L / E) threads
// transform one field each (in registers, the field's own tile as the exchange tile) and
// leave the spectra there, then all threads sweep the tile's modes (assembly, projection,
// stage update), each thread down one column, so everything that depends on the column is
// formed once per tile; what depends on the row comes from shared-memory tables.  While
// tile k is transformed and swept, the products of the block's next tile stream into the
// other buffer (16-byte cp.async, NBUF = 2) and the state its sweep will read is prefetched
// into L2 (PF).  FORM 3: the adjoint's stage.
// ---------------------------------------------------------------------------
__host__ __device__ constexpr size_t pipe_row_bytes() { return 3 * sizeof(double); }
// Mode of the adjoint (FORM 3): W = D c (A + i K x B) and the transposed stage update (see
// k_fwd_x).
template <typename T, int STAGE>
__device__ __forceinline__ void adj_mode(const C<T>* p, const T (&K)[3], T inv, T cw, double eh, double dt, const C<T>* Lv,
                                         const C<T>* Acc, C<T>* lam, C<T>* Ac, C<T>* Lm, long long off, long long S) {
  typedef C<T> V;
  V a[3] = {mk<V>(0, 0), mk<V>(0, 0), mk<V>(0, 0)};
#pragma unroll
  for (int f = 0; f < 6; ++f) accum_product<3>(f, scale(p[f], inv), K[0], K[1], K[2], a[0], a[1], a[2]);
  const double e1 = eh * eh;
  const T Eh = (T)eh, E1 = (T)e1;
#pragma unroll
  for (int i = 0; i < 3; ++i) {
    const long long o = off + i * S;
    const V W = scale(a[i], cw);
    if constexpr (STAGE == 4) {
      Ac[o] = add(scale(Lv[i], E1), scale(W, E1));
      lam[o] = add(scale(Lv[i], (T)(dt / 3 * eh)), scale(W, (T)(dt * eh)));
    } else if constexpr (STAGE == 1) {
      Lm[o] = add(Acc[i], W);
    } else {
      Ac[o] = add(Acc[i], scale(W, Eh));
      lam[o] = STAGE == 3 ? add(scale(Lv[i], (T)(dt / 3 * eh)), scale(W, (T)(0.5 * dt)))
                          : add(scale(Lv[i], (T)(dt / 6 * e1)), scale(W, (T)(0.5 * dt * eh)));
    }
  }
}

template <typename T, int L, int E, int CW, int FORM, int STAGE, int NBUF, bool PF>
__global__ void __launch_bounds__(z_nout(FORM) * CW * (L / E), 1)
    k_fwd_x_pipe(const C<T>* P, Geo g, StageArgs a, const C<T>* __restrict__ tw) {
  chain_begin();
  typedef C<T> V;
  constexpr bool ADJ = FORM == 3, F32 = sizeof(T) == 4 && !ADJ;
  // the state fields the sweep reads at this stage
  constexpr bool LD0 = !(ADJ && STAGE == 1), LD1 = ADJ ? STAGE != 4 : STAGE > 1;
  constexpr int NF = z_nout(FORM), GT = CW * (L / E), NT = NF * GT, TILE = L * CW;
  constexpr int VEC = 16 / (int)sizeof(V), SWK = best_swk(L, E, CW, (int)sizeof(V));
  static_assert(NT % CW == 0 && TILE % VEC == 0, "a thread sweeps one column; 16-byte copies");
  extern __shared__ __align__(16) unsigned char smraw[];
  V* buf0 = reinterpret_cast<V*>(smraw);
  // per row: Kx^2, the x integrating factor (FP32: (hi, lo) pair), Kx
  double* tk2 = reinterpret_cast<double*>(buf0 + NBUF * NF * TILE);
  double* tex = tk2 + L;
  T* tkx = reinterpret_cast<T*>(tex + L);
  const int grp = threadIdx.x / GT, gt = threadIdx.x % GT, c = gt % CW, t = gt / CW;
  const unsigned inner = g.Ny * g.Hz;  // a multiple of CW (Ny is a multiple of 16)
  const unsigned ntiles = inner / CW;
  const T inv = (T)(1.0 / ((double)g.Nx * g.Ny * g.Nz));
  const V* st0 = reinterpret_cast<const V*>(a.U0);
  V* tot = reinterpret_cast<V*>(a.tot);
  V* Uc = reinterpret_cast<V*>(a.Ucur);
  V* Uo = reinterpret_cast<V*>(a.Uout);
  for (int i = threadIdx.x; i < L; i += NT) {
    const double K = kfft(i, g.Nx) * g.kf[0];
    tk2[i] = K * K;
    if constexpr (F32) reinterpret_cast<float2*>(tex)[i] = a.exf[i];
    else tex[i] = a.ex[i];
    tkx[i] = (T)K;
  }
  auto issue = [&](unsigned tile, int b) {
    if (tile < ntiles) {
      V* d = buf0 + b * (NF * TILE);
      for (int i = threadIdx.x; i < NF * TILE / VEC; i += NT) {
        const int f = i / (TILE / VEC), r = (i % (TILE / VEC)) / (CW / VEC), cc = (i % (CW / VEC)) * VEC;
        cp_async16(d + f * TILE + r * CW + cc, P + f * g.S + (long long)r * inner + tile * CW + cc);
      }
      if constexpr (PF) {
        for (int r = threadIdx.x; r < 3 * L; r += NT) {
          const long long off = (r / L) * g.S + (long long)(r % L) * inner + tile * CW;
          if (LD0) asm volatile("prefetch.global.L2 [%0];" ::"l"(st0 + off));
          if (LD1) asm volatile("prefetch.global.L2 [%0];" ::"l"(tot + off));
        }
      }
    }
    cp_async_commit();
  };
  issue(blockIdx.x, 0);
  const Fac<T> Fc[4] = {fac<T>(a.dt), fac<T>(0.5 * a.dt), fac<T>((1.0 / 3) * a.dt), fac<T>((1.0 / 6) * a.dt)};
  const int sc = threadIdx.x % CW, sr0 = threadIdx.x / CW;  // the sweep's column and first row
  constexpr int SR = NT / CW;
  int b = 0;
  for (unsigned tile = blockIdx.x; tile < ntiles; tile += gridDim.x) {
    V* buf = buf0 + b * (NF * TILE);
    cp_async_wait<0>();
    __syncthreads();  // the tile has arrived, and the sweep of the previous one is over
    if (NBUF == 2) issue(tile + gridDim.x, b ^ 1);
    {
      V* ft = buf + grp * TILE;
      V v[E];
#pragma unroll
      for (int s = 0; s < E; ++s) v[s] = ft[load_row<L, E>(t, s) * CW + c];
      __syncthreads();  // every row of the tile is in registers: it is the exchange tile now
      fft_regs<L, E, -1, 0, 0, false, SWK>(v, t, ft, CW, c, tw, 1);
#pragma unroll
      for (int s = 0; s < E; ++s) ft[final_row<L, E>(t, s) * CW + c] = v[s];
    }
    __syncthreads();
    // column constants
    const unsigned col = tile * CW + sc;
    const int ly = col / (unsigned)g.Hz, lz = col - ly * g.Hz, ky = kfft(ly, g.Ny);
    const double Kyd = ky * g.kf[1], Kzd = lz * g.kf[2], c2 = Kyd * Kyd + Kzd * Kzd;
    const T Ky = (T)Kyd, Kz = (T)Kzd;
    const double ecol64 = F32 ? 0.0 : a.ey[ly] * a.ez[lz];
    Fac<T> ecol;
    if constexpr (F32) ecol = pair_mul(a.eyf[ly], a.ezf[lz]);
    else ecol = fac<T>(ecol64);
    int zlo = L, zhi = L;
    if (ADJ || STAGE == 1) fff_zero_rows(g.dealias, ly, lz, g.Nx, g.Ny, g.Nz, zlo, zhi);
    const bool clear = STAGE == 4 && a.reality && lz == g.Nz / 2;
    const bool band = a.fcube && abs(ky) <= a.fkm && lz <= a.fkm;
    const V* fcol = reinterpret_cast<const V*>(a.fcube) + ((long long)a.fkm * (2 * a.fkm + 1) + ky + a.fkm) * (a.fkm + 1) + lz;
    const V *u0p = st0 + col, *ttp = tot + col;
    auto load = [&](int r, V* u0, V* tt) {
#pragma unroll
      for (int i = 0; i < 3; ++i) {
        if (LD0) u0[i] = u0p[i * g.S + (long long)r * inner];
        if (LD1) tt[i] = ttp[i * g.S + (long long)r * inner];
      }
    };
    auto mode = [&](int r, const V* u0, const V* tt) {
      V p[NF];
#pragma unroll
      for (int f = 0; f < NF; ++f) p[f] = buf[f * TILE + r * CW + sc];
      const T K[3] = {tkx[r], Ky, Kz};
      if constexpr (ADJ) {
        const T cw = (r >= zlo && r < zhi) ? (T)0 : ((lz > 0 && 2 * lz < g.Nz) ? (T)2 : (T)1);
        adj_mode<T, STAGE>(p, K, inv, cw, tex[r] * ecol64, a.dt, u0, tt, Uc, tot, const_cast<V*>(st0),
                           (long long)r * inner + col, g.S);
        return;
      }
      const Recip<T> rK2 = recip((T)(tk2[r] + c2));
      Fac<T> Feh, Fe1;
      if constexpr (F32) {
        Feh = pair_mul(reinterpret_cast<const float2*>(tex)[r], ecol);
        if (STAGE == 1 || STAGE == 4) Fe1 = pair_mul(Feh, Feh);
      } else {
        const double eh = tex[r] * ecol64;
        Feh = fac<T>(eh);
        Fe1 = fac<T>(eh * eh);
      }
      V fcv[3];
      bool forced = false;
      if (band) {
        const int kx = kfft(r, g.Nx);
        if (abs(kx) <= a.fkm) {
          forced = true;
          const long long n = 2 * a.fkm + 1, fs = n * n * (a.fkm + 1);
#pragma unroll
          for (int i = 0; i < 3; ++i) fcv[i] = fcol[i * fs + (long long)kx * n * (a.fkm + 1)];
        }
      }
      step_mode<T, FORM, STAGE>(p, K, rK2, inv, forced ? fcv : nullptr, r >= zlo && r < zhi, clear, Feh, Fe1, Fc, u0, tt,
                                Uc, tot, Uo, (long long)r * inner + col, g.S, a.err);
    };
    // the state of the next row is on its way while a row is updated
    V u0[3], tt[3];
    if (sr0 < L) load(sr0, u0, tt);
    for (int r = sr0; r < L; r += SR) {
      V u1[3], t1[3];
      if (r + SR < L) load(r + SR, u1, t1);
      mode(r, u0, tt);
#pragma unroll
      for (int i = 0; i < 3; ++i) {
        u0[i] = u1[i];
        tt[i] = t1[i];
      }
    }
    if (NBUF == 1) {
      __syncthreads();
      issue(tile + gridDim.x, 0);
    } else {
      b ^= 1;
    }
  }
  cp_async_wait<0>();
}

// ---------------------------------------------------------------------------
// Elementwise spectral epilogue of the split form: a step's wherever the pipelined kernel
// has no tile (fwd_x_impl), every mode's where the fused kernel's column tiles would have
// rows narrower than 64 bytes (Nx >= 512).  The NF product fields have already been
// forward-transformed along x in place (k_strided_ld); one thread per spectral element, every
// array access coalesced.  Same arithmetic as k_fwd_x's epilogue (spec_epilogue).
// ---------------------------------------------------------------------------
template <typename T, int FORM, int MODE>
__global__ void __launch_bounds__(256) k_spec_epi(const C<T>* P, Geo g, StageArgs a) {
  chain_begin();
  typedef C<T> V;
  constexpr int NF = z_nout(FORM);
  double tb[MODE == MODE_FLUX ? FLUX_MAX_BINS : 1];  // MODE_FLUX: per-thread sphere partials
  if (MODE == MODE_FLUX)
    for (int i = 0; i <= a.nradii; ++i) tb[i] = 0.0;
  const T inv = (T)(1.0 / ((double)g.Nx * g.Ny * g.Nz));
  const V* st0 = reinterpret_cast<const V*>(MODE == MODE_FLUX ? a.Ud : a.U0);
  const V* st1 = reinterpret_cast<const V*>(a.tot);
  // the state fields the epilogue reads at this stage (U0 / Lam / the flux field; tot)
  const bool ld0 = MODE != MODE_NLIN && !(MODE == MODE_ADJ && a.stage == 1);
  const bool ld1 = (MODE == MODE_STEP && a.stage > 1) || (MODE == MODE_ADJ && a.stage != 4);
  // two elements per thread and iteration (e and e + stride): every load of both is
  // issued before either is used, twice the loads in flight of one element at a time
  // 32-bit index arithmetic (a component holds < 2^31 modes)
  const unsigned n = (unsigned)g.S, stride = gridDim.x * blockDim.x;
  for (unsigned e0 = blockIdx.x * blockDim.x + threadIdx.x; e0 < n; e0 += 2 * stride) {
    const bool has1 = e0 + stride < n;
    V pv[2][NF], s0[2][3], s1[2][3];
#pragma unroll
    for (int j = 0; j < 2; ++j) {
      const unsigned e = e0 + j * stride;
      if (j == 0 || has1) {
#pragma unroll
        for (int f = 0; f < NF; ++f) pv[j][f] = P[f * g.S + e];
#pragma unroll
        for (int i = 0; i < 3; ++i) {
          s0[j][i] = ld0 ? st0[i * g.S + e] : mk<V>(0, 0);
          s1[j][i] = ld1 ? st1[i * g.S + e] : mk<V>(0, 0);
        }
      }
    }
#pragma unroll
    for (int j = 0; j < 2; ++j) {
      const unsigned e = e0 + j * stride;
      if (j == 1 && !has1) break;
      const unsigned r = e / (unsigned)g.Hz;
      const int lz = (int)(e - r * g.Hz), lx = (int)(r / (unsigned)g.Ny), ly = (int)(r - (unsigned)lx * g.Ny);
      const T Kx = (T)(kfft(lx, g.Nx) * g.kf[0]), Ky = (T)(kfft(ly, g.Ny) * g.kf[1]), Kz = (T)(lz * g.kf[2]);
      V a0 = mk<V>(0, 0), a1 = mk<V>(0, 0), a2 = mk<V>(0, 0);
#pragma unroll
      for (int f = 0; f < NF; ++f) accum_product<FORM>(f, scale(pv[j][f], inv), Kx, Ky, Kz, a0, a1, a2);
      const double exy = (MODE == MODE_STEP || MODE == MODE_ADJ) ? a.ey[ly] * a.ez[lz] : 0.0;
      spec_epilogue<T, MODE>(g, a, lx, ly, lz, e, exy, col_pair<T, MODE>(a, ly, lz), a0, a1, a2, s0[j], s1[j], 1, tb);
    }
  }
  if (MODE == MODE_FLUX) {
    for (int i = 0; i <= a.nradii; ++i) {
      const double v = block_sum(tb[i]);
      if (threadIdx.x == 0) a.bins[(long long)(blockIdx.x + 1) * (a.nradii + 1) + i] = v;
    }
  }
}

}  // namespace ts

namespace ts {
// ---------------------------------------------------------------------------
// standalone z transforms for the Forward/Inverse_transform entry points:
// DIR=-1: real padded (Nx,Ny,Nz+2) -> spectral lines (Nx,Ny,Hz), unnormalised
// DIR=+1: spectral lines -> real padded, unnormalised; pads written as 0
// ---------------------------------------------------------------------------
// Line pairs as in k_z_pair (two real lines a, b of component blockIdx.y as a + i b), one
// transform of length N = Nz per pair, 16 elements per thread; the real points go through
// the pair's exchange line so that their stores are contiguous.
template <typename T, int NZ, int E, int DIR, int NTHR, int MINB>
__global__ void __launch_bounds__(NTHR, MINB)
    k_z_single(const C<T>* __restrict__ in, C<T>* __restrict__ out, Geo g, const C<T>* __restrict__ tw) {
  typedef C<T> V;
  constexpr int M = NZ / 2, H = M + 1, LD = NZ + 2, TPL = NZ / E, PPB = NTHR / TPL, LDX = zpair_slot<T>(NZ);
  constexpr bool WARP = TPL <= 32;
  static_assert(NTHR % TPL == 0, "whole pairs per block");
  extern __shared__ __align__(16) unsigned char smraw[];
  const int l = threadIdx.x / TPL, t = threadIdx.x % TPL;
  const long long nlines = (long long)g.Nx * g.Ny;
  const long long line = 2 * ((long long)blockIdx.x * PPB + l);
  const bool live0 = line < nlines, live1 = line + 1 < nlines;
  V* xch = reinterpret_cast<V*>(smraw) + l * LDX;
  // both layouts have H complex (N + 2 reals) per line
  const long long lo = blockIdx.y * g.S + (live0 ? line : 0) * H;
  V v[1][E];
  if constexpr (DIR > 0) {
    const V* X = in + lo;
#pragma unroll
    for (int s = 0; s < E; ++s) {
      const int r = load_row<NZ, E>(t, s), k = r <= M ? r : NZ - r;
      V a = live0 ? X[k] : mk<V>(0, 0), b = live1 ? X[H + k] : mk<V>(0, 0);
      if (k == 0 || k == M) a.y = b.y = 0;
      if (r > M) a.y = -a.y, b.y = -b.y;
      v[0][s] = mk<V>(a.x - b.y, a.y + b.x);
    }
    fft_regs_b<NZ, E, 1, 1, WARP, 0, 1, false>(v, t, xch, LDX, 1, 0, ct_table<NZ, E, false>(tw));
#pragma unroll
    for (int s = 0; s < E; ++s) xch[prow<1>(final_row<NZ, E>(t, s))] = v[0][s];
    fft_sync<WARP>();
    // points 2 i, 2 i + 1 as one store; the pad is slot M
    V* o = out + lo;
    for (int i = t; i <= M; i += TPL) {
      const V p = i < M ? xch[prow<1>(2 * i)] : mk<V>(0, 0), q = i < M ? xch[prow<1>(2 * i + 1)] : mk<V>(0, 0);
      if (live0) o[i] = mk<V>(p.x, q.x);
      if (live1) o[H + i] = mk<V>(p.y, q.y);
    }
  } else {
    const T* X = reinterpret_cast<const T*>(in + lo);
#pragma unroll
    for (int s = 0; s < E; ++s) {
      const int n = load_row<NZ, E>(t, s);
      v[0][s] = mk<V>(live0 ? X[n] : (T)0, live1 ? X[LD + n] : (T)0);
    }
    fft_regs_b<NZ, E, -1, 1, WARP, 0, 1, false>(v, t, xch, LDX, 1, 0, ct_table<NZ, E, false>(tw));
#pragma unroll
    for (int s = 0; s < E; ++s) xch[prow<1>(final_row<NZ, E>(t, s))] = v[0][s];
    fft_sync<WARP>();
    V* o = out + lo;
    for (int k = t; k <= M; k += TPL) {
      const V z = xch[prow<1>(k)], zp = xch[prow<1>((NZ - k) % NZ)];
      if (live0) o[k] = mk<V>((T)0.5 * (z.x + zp.x), (T)0.5 * (z.y - zp.y));
      if (live1) o[H + k] = mk<V>((T)0.5 * (z.y + zp.y), (T)0.5 * (zp.x - z.x));
    }
  }
}

}  // namespace ts
