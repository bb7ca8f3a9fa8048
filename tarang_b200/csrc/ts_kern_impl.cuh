// Launcher definitions, included by the ts_kern_<part>_<precision>.cu files with TS_REAL
// defined to float / double and TS_PART to the group of launchers that the file
// instantiates (one file per group and precision, so that they compile in parallel).
#define TS_PART_STR 1   // strided-axis FFTs
#define TS_PART_IX 2    // FFF inverse x pass
#define TS_PART_Z 3     // z passes
#define TS_PART_FX 4    // FFF forward x pass and epilogue
#define TS_PART_SFF 5   // sin/cos x passes
#define TS_PART_MISC 6  // elementwise, plane-sized and reduction kernels, tuning queries
#include <math.h>
#include <type_traits>
#include "ts_launch.h"
#include "ts_misc.cuh"
#include "ts_radius.h"

namespace ts {

namespace {

typedef TS_REAL T;
typedef C<T> V;

// elements per thread of the register FFTs; columns per block (rows of 128 B)
constexpr int E_REG = std::is_same<T, float>::value ? 16 : 8;
// at L = 1024 the 16-element register FFT would spill under the 512-thread cap
constexpr int e_reg(int L) { return (L >= 1024 ? 8 : E_REG) < L ? (L >= 1024 ? 8 : E_REG) : L; }
// forward-x kernel: 4 elements per thread (3 accumulators each); on B200 at 256^3
// the 512-thread blocks beat the 8-element, 256-thread form by 6 % in FP32 (3.03
// vs 3.09 ms per step) and 2.5 % in FP64 (6.78 vs 6.96 ms)
constexpr int E_ACC = 4;
constexpr int E_ACC_ALT = 8;
constexpr int CWMAX = std::is_same<T, float>::value ? 16 : 8;
constexpr int emin(int a, int b) { return a < b ? a : b; }
constexpr int cw_for(int L, int E) {
  return emin(CWMAX, (512 * E / L) > 0 ? (512 * E / L) : 1);
}
// 8-byte units per complex (TMA boxes are expressed in 8-byte words)
constexpr int UNITS = (int)sizeof(V) / 8;
// column tile width of the TMA x-pass kernels: 64-byte rows, and at least two
// 8-byte units so every tile start is 16-byte aligned
// (the epilogue kernel's 8 tiles + padded exchange tile must fit in 220 KB)
constexpr int xcw_fit(int L, int cw) {
  return (cw > (std::is_same<T, float>::value ? 2 : 1) &&
          (size_t)9 * L * cw * sizeof(V) + (size_t)L * sizeof(V) > 220 * 1024)
             ? xcw_fit(L, cw / 2) : cw;
}
constexpr int xcw(int L) { return xcw_fit(L, std::is_same<T, float>::value ? 8 : 4); }

template <typename Fn> bool dispatch_L(int L, Fn&& fn) {
  switch (L) {
    case 16: fn(std::integral_constant<int, 16>{}); return true;
    case 32: fn(std::integral_constant<int, 32>{}); return true;
    case 64: fn(std::integral_constant<int, 64>{}); return true;
    case 128: fn(std::integral_constant<int, 128>{}); return true;
    case 256: fn(std::integral_constant<int, 256>{}); return true;
    case 512: fn(std::integral_constant<int, 512>{}); return true;
    case 1024: fn(std::integral_constant<int, 1024>{}); return true;
  }
  return false;
}

// SFF launchers also take the non-power-of-two sizes 48 and 96: their FFT
// lengths 3 * 2^k run with 12 elements per thread (radices 4, 2, 3)
template <typename Fn> bool dispatch_L_sff(int L, Fn&& fn) {
  if (dispatch_L(L, fn)) return true;
  {
    switch (L) {
      case 48: fn(std::integral_constant<int, 48>{}); return true;
      case 96: fn(std::integral_constant<int, 96>{}); return true;
    }
  }
  return false;
}
// elements per thread for a length that may carry a factor 3
// (6 where the power-of-two choice is 4 or less: the FP64 SFF forward x kernel
// holds four accumulators per element and spilled at 12)
constexpr int e_mixed(int L, int e_pow2) { return L % 3 == 0 ? (e_pow2 >= 8 ? 12 : 6) : (e_pow2 < L ? e_pow2 : L); }

template <typename K> cudaError_t smem_attr(K kernel, size_t bytes) {
  if (bytes > 48 * 1024) {
    const cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
    if (e != cudaSuccess) cudaGetLastError();  // do not leave the error for a later launch to report
    return e;
  }
  return cudaSuccess;
}

// Launch of a kernel that begins with chain_begin().  Kernels on small fields are launched
// while the preceding kernel of the stream still runs: a pass takes 2-4 us there and the gap
// between two plain launches another 2 us.  Large grids are launched plainly (but for chained_sc):
// their early blocks would take the slots of the running grid's last waves.  B200, plain -> chained: 32^3
// FP32 step 126 -> 77 us, 64^3 FP64 172 -> 161, SSF 96^3 (3.6 MB per component) 329 -> 281, SSS
// 128^3 FP32 (8.5 MB) 653 -> 616, 18-sphere flux 128^3 3278 -> 3084; FP64 adjoint 128^3 (17 MB)
// 12750 -> 13080, 256^3 2711 -> 2715, MHD 256^3 4908 -> 5008.
constexpr long long CHAIN_BYTES = 10000000;
inline bool chained(const Geo& g, int nmem = 1) { return nmem == 1 && g.S * (long long)sizeof(V) <= CHAIN_BYTES; }
// The sin/cos passes: along y (y_as_x: S is one x plane, Sp the component) fields of any size are
// chained.  B200, step, us, plain -> chained: FP32 SSS Boussinesq 64x64x1024 1345 -> 1311,
// 128x256x256 2462 -> 2413, 256^3 4848 -> 4763, SSF fluid 64x64x1024 799 -> 785, 256^3 2988 -> 2973;
// FP64 SSF fluid 128^3 (17 MB) 790 -> 775, 64x64x1024 (34 MB) 1546 -> 1529, 128x256x256 (135 MB) 2969 ->
// 2944, SSF Boussinesq 128x256x256 4391 -> 4415, SSS 256^3 9205 -> 9270.
inline bool chained_sc(const Geo& g, int nmem) { return g.S < g.Sp ? nmem == 1 : chained(g, nmem); }
template <typename... P, typename... A>
cudaError_t launch_chain(bool chain, void (*k)(P...), dim3 grid, unsigned block, size_t sm, cudaStream_t st, A&&... args) {
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[0].val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t c = {};
  c.gridDim = grid;
  c.blockDim = dim3(block);
  c.dynamicSmemBytes = sm;
  c.stream = st;
  c.attrs = at;
  c.numAttrs = chain ? 1 : 0;
  ++g_launches;
  return cudaLaunchKernelEx(&c, k, static_cast<P>(args)...);
}

inline unsigned grid1d(long long n, int threads) {
  long long b = (n + threads - 1) / threads;
  if (b > 148 * 16) b = 148 * 16;
  if (b < 1) b = 1;
  return (unsigned)b;
}

}  // namespace

// persistent strided kernel (the candidates of the y passes; ld_tile is the rule): elements per
// thread, tile columns, staging tiles.  At L = 1024 in FP32 16 elements per thread and 8-column
// tiles (64-byte rows) with the exchange in the consumed staging tile: 2.9 TB/s in the y pass
// against 2.0 with 4-column tiles
constexpr bool wide1024(int L) { return std::is_same<T, float>::value && L == 1024; }
constexpr int str_e(int L) { return wide1024(L) ? 16 : e_mixed(L, e_reg(L)); }
constexpr int str_cw(int L) { return wide1024(L) ? 8 : cw_for(L, str_e(L)); }
constexpr int str_nt(int L) { return wide1024(L) ? 2 : 3; }

// sin/cos x kernel: elements per thread, tile columns, blocks per SM it is compiled for.  Bound by
// DRAM latency: rows of whole 128-byte lines, as many elements per thread as leave two radix
// passes (one exchange), and the blocks per SM at which the registers just do not spill.  B200,
// FP32 forward, us: 128 points 27 (8 elements 35; 8 columns 36; four blocks 31), 256 points 57
// (three blocks 62, 8 elements 117), 96 points with 24 elements 15.1 (12: 17.0, 6: 23.3)
struct LdTile { int E, CW, MINB; };
constexpr LdTile sc_tile(int L, int dir) {
  return std::is_same<T, float>::value
             ? (L == 16 ? LdTile{4, 16, 8} : L == 32 ? LdTile{8, 16, 16} : L == 64 ? LdTile{8, 16, 8}
                : L == 128 ? LdTile{16, 16, 6} : L == 256 ? LdTile{16, 16, dir > 0 ? 2 : 4}
                : L == 512 ? LdTile{16, 16, 1} : L == 96 ? LdTile{24, 16, 8} : LdTile{12, 16, 8})
             : (L == 16 ? LdTile{4, 8, 16} : L == 32 ? LdTile{8, 8, 16} : L == 64 ? LdTile{8, 8, 8}
                : L == 128 ? LdTile{16, 8, 4} : L == 256 ? LdTile{16, 8, 2} : L == 512 ? LdTile{16, 8, 1}
                : LdTile{12, 8, 4});
}

// direct-load strided kernel: elements per thread, tile columns and blocks per SM the
// kernel is compiled for, chosen as for sc_tile.  B200, FP32, us: 256 points forward, three
// fields of 256^3, 72 (8 columns 81, 32 columns 79, 8 elements 101, two blocks 79; the persistent
// cp.async kernel 89-101); 128 points 25 (8 elements 31; persistent 40); 64 points 25 (persistent
// 70); 96 points with 24 elements on 32 columns 49 (16 columns 54, 12 elements 55-60; persistent
// 93); 512 points with 32 elements 165 (16: 189; three blocks 172); 1024 points with 32 elements
// on 8 columns 391 (16 columns 416, 16 elements 455).  FP64: 256 points with 16 elements 72 (8:
// 80; persistent 93), 128 points 35 (8 elements 36), 512 points 83 (32 elements 90, three blocks
// 101), 1024 points on 4 columns 204 (16 elements on 8 columns 220)
constexpr LdTile ld_tile(int L) {
  return std::is_same<T, float>::value
             ? (L == 16 ? LdTile{4, 16, 8} : L == 32 ? LdTile{8, 16, 16} : L == 64 ? LdTile{8, 16, 8}
                : L == 128 ? LdTile{16, 16, 6} : L == 256 ? LdTile{16, 16, 4} : L == 512 ? LdTile{32, 16, 2}
                : L == 1024 ? LdTile{32, 8, 2} : L == 96 ? LdTile{24, 32, 4} : LdTile{12, 16, 8})
             : (L == 16 ? LdTile{4, 8, 16} : L == 32 ? LdTile{8, 8, 16} : L == 64 ? LdTile{8, 8, 6}
                : L == 128 ? LdTile{16, 8, 4} : L == 256 ? LdTile{16, 8, 2} : L == 512 ? LdTile{16, 8, 2}
                : L == 1024 ? LdTile{16, 4, 2} : LdTile{12, 8, 4});
}
// the same for lines whose rows lie FAR_ROW_BYTES or more apart (the x axis of large grids), 0: no
// other tile.  1024 points in FP32: with a page or so per row, 128-byte row segments beat the
// second block per SM (512 x 512 planes, rows 1 MB apart: 1838 -> 1609 us); with nearer rows they
// do not (256 x 256 planes, rows 264 KB apart: 364 -> 420 us).
constexpr long long FAR_ROW_BYTES = 1 << 19;
constexpr LdTile far_tile(int L) {
  return std::is_same<T, float>::value && L == 1024 ? LdTile{32, 16, 1} : LdTile{0, 0, 0};
}
// inverse x kernel (one field per block): the tiles of the strided kernel; three blocks per SM
// at 256 points, where the vorticity's second operand takes registers.  The three fields of a
// group in one block read U once but need 128 registers at 8 elements per thread: 115 us against
// 102 (256^3 rotational)
constexpr LdTile ix_tile(int L) {
  return std::is_same<T, float>::value
             ? (L == 16 ? LdTile{4, 16, 8} : L == 32 ? LdTile{8, 16, 16} : L == 64 ? LdTile{8, 16, 8}
                : L == 128 ? LdTile{16, 16, 6} : L == 256 ? LdTile{16, 16, 3} : L == 512 ? LdTile{32, 16, 2}
                : LdTile{32, 8, 2})
             : (L == 16 ? LdTile{4, 8, 16} : L == 32 ? LdTile{8, 8, 16} : L == 64 ? LdTile{8, 8, 6}
                : L == 128 ? LdTile{16, 8, 4} : L == 256 ? LdTile{16, 8, 2} : L == 512 ? LdTile{16, 8, 2}
                : LdTile{16, 4, 2});
}

// ---------------------------------------------------------------------------
// Launch-tuning candidates.  Candidate 0 of every pass class is the rule; the others are the
// kernels that were the rules before the direct-load, line-pair and pipelined ones, and their
// variants: elements per thread E (the Stockham passes use radix min(E, remaining)), column-tile
// width CW, number of staging tiles NT.  On B200 they are slower than the rules at the sizes
// beside the tile tables (13-60 %); their numbers stay valid for stored tunings.  One that does not fit
// (threads per block, shared memory) or repeats another of the candidates' tables is refused
// (str_cand, ix_cand and sx_cand 0 are the tiles that the tables start from, not the rule's).
// ---------------------------------------------------------------------------
constexpr int NCAND = TUNE_NCAND;
struct Tile { int E, CW, NT; };
constexpr bool tile_eq(Tile a, Tile b) { return a.E == b.E && a.CW == b.CW && a.NT == b.NT; }
constexpr bool tile_fits(int L, Tile c, int tiles) {
  return c.E > 0 && c.CW > 0 && L % c.E == 0 && c.CW * (L / c.E) <= 1024 && c.CW * (L / c.E) >= 32 &&
         (size_t)tiles * L * c.CW * sizeof(V) <= 227 * 1024;
}

// strided passes (y inverse / y forward)
constexpr Tile str_cand(int L, int v) {
  return v == 0 ? Tile{str_e(L), str_cw(L), str_nt(L)}
       : v == 1 ? (L % 3 != 0 && str_e(L) > 4 ? Tile{str_e(L) / 2, str_cw(L), str_nt(L)} : Tile{0, 0, 0})
       : v == 2 ? (str_cw(L) > 1 ? Tile{str_e(L), str_cw(L) / 2, str_nt(L)} : Tile{0, 0, 0})
       : v == 3 ? Tile{str_e(L), str_cw(L), 5 - str_nt(L)}
       : v == 4 ? Tile{str_e(L), str_cw(L), 4}
       : v == 5 ? (wide1024(L) ? Tile{32, 8, 1} : Tile{0, 0, 0})
       : v == 6 ? (wide1024(L) ? Tile{32, 16, 1} : Tile{0, 0, 0})
                : Tile{0, 0, 0};
}
constexpr bool str_valid(int L, int v) {
  return v == 0 || (v == 6 && wide1024(L) && tile_fits(L, str_cand(L, 6), 1)) || (v < NCAND && tile_fits(L, str_cand(L, v), str_tiles(str_cand(L, v).NT)) &&
                    !tile_eq(str_cand(L, v), str_cand(L, 0)) && (v < 2 || !tile_eq(str_cand(L, v), str_cand(L, 1))) &&
                    (v < 3 || !tile_eq(str_cand(L, v), str_cand(L, 2))) &&
                    (v < 4 || !tile_eq(str_cand(L, v), str_cand(L, 3))) &&
                    (v < 5 || !tile_eq(str_cand(L, v), str_cand(L, 4))));
}

// inverse x pass (FFF forms 0, 1): 8 elements per thread in FP32 (U held in
// registers across the output fields; 16 at L = 1024 with per-field loads)
constexpr int ix_e(int L) { return wide1024(L) ? 16 : (std::is_same<T, float>::value ? (8 < L ? 8 : L) : e_reg(L)); }
constexpr int ix_cw(int L) { return wide1024(L) ? 8 : cw_for(L, ix_e(L)); }
constexpr int ix_e_alt(int L) {
  return std::is_same<T, float>::value ? (ix_e(L) == 8 ? (16 <= L ? 16 : 0) : 8) : (ix_e(L) > 4 ? ix_e(L) / 2 : 0);
}
// candidate 3 (FP32): the persistent prefetching kernel k_inv_x_pf, 8 elements per thread
// (the three components of U held in registers), staging + exchange tiles (NT = 4 tiles);
// candidate 4 (FP32, 1024-point lines): 32 elements per thread over 8-column tiles
// (256-thread blocks, two per SM; radix 32 x 32, one exchange per field);
// candidate 5 (FP32, 1024-point lines): 16 elements per thread over 8-column tiles
constexpr Tile ix_cand(int L, int v) {
  return v == 0 ? Tile{ix_e(L), ix_cw(L), 1}
       : v == 1 ? (ix_e_alt(L) > 0 ? Tile{ix_e_alt(L), cw_for(L, ix_e_alt(L)), 1} : Tile{0, 0, 0})
       : v == 2 ? (ix_cw(L) > 1 ? Tile{ix_e(L), ix_cw(L) / 2, 1} : Tile{0, 0, 0})
       : v == 3 ? (std::is_same<T, float>::value ? Tile{8, cw_for(L, 8), 4} : Tile{0, 0, 0})
       : v == 4 ? (wide1024(L) ? Tile{32, 8, 1} : Tile{0, 0, 0})
       : v == 5 ? (wide1024(L) ? Tile{16, 8, 2} : Tile{0, 0, 0})
                : Tile{0, 0, 0};
}
constexpr bool ix_valid(int L, int v) {
  return v == 0 || (v < NCAND && tile_fits(L, ix_cand(L, v), ix_cand(L, v).NT == 4 ? 4 : 1) &&
                    !tile_eq(ix_cand(L, v), ix_cand(L, 0)) && (v < 2 || !tile_eq(ix_cand(L, v), ix_cand(L, 1))) &&
                    (v < 3 || !tile_eq(ix_cand(L, v), ix_cand(L, 2))) &&
                    (v < 4 || !tile_eq(ix_cand(L, v), ix_cand(L, 3))) &&
                    (v < 5 || !tile_eq(ix_cand(L, v), ix_cand(L, 4))));
}

// z candidates (forms 1, 2, 7): 1 = the slot kernel with 8 elements per thread
// (12 with a factor 3), 2 = the slot kernel with 4 (power-of-two lines), 3 = the
// FP32 register kernel with 4 elements per thread (lines of up to 256 points),
// 4 = on 1024-point lines in FP32, the register kernel that loads each component just
// before its transform (the rule there issues every load up front).  Candidate 1 exists where the
// slot kernel was not itself candidate 0 when the numbers were given
template <int NZ, int FORM> constexpr bool z_rule_slots() {
  constexpr int M = NZ / 2;
  return !(std::is_same<T, float>::value && M <= 512) &&
         !(!std::is_same<T, float>::value && M % 3 != 0 && M <= 128);
}
// line-pair kernel: elements per thread, threads per block and blocks per SM the kernel is
// compiled for
struct ZTile { int E, NTHR, MINB, NB; };
constexpr ZTile zp_tile(int NZ, int form) {
  const bool f32 = std::is_same<T, float>::value;
  // FP64 lines: measured as whole steps only, against the shared-memory slot kernel that was the
  // rule before (64x64x512 rotational 1291 -> 712 us, 64x64x1024 2422 -> 1505, MHD 64x64x512 2507 ->
  // 1292, 256^3 17900 -> 9150, SFF 96^3 Boussinesq 1229 -> 627, SSS 64x64x1024 4450 -> 2449); from 256
  // points, at 48 and 96, and in forms 2, 5 and 6 they spill 0.1-1 KB a thread.  The rotational
  // form at 128 points takes 4 elements per thread: 47.5 us against 48.5 with 8, which spill; at 256
  // points it is the other way round (109.9 against 94.2)
  const int E = NZ % 3 == 0 ? 12 : (!f32 && form == 1 && NZ == 128 ? 4 : 8);
  const int tpl = NZ / E, thr = tpl > 64 ? tpl : 64;
  // the three products of the rotational form together: twiddles and barriers shared (138 -> 134 us)
  return ZTile{E, thr, ((f32 && NZ % 3 != 0) || E == 4 ? 6 : 4) * 64 / thr, f32 && form == 1 && NZ % 3 != 0 ? 3 : 1};
}
// FP32 lines of 48, 96 and 1024 points: single lines in registers (k_z_reg) are the rule
template <int NZ, int FORM> constexpr bool zreg_rule() {
  return std::is_same<T, float>::value && FORM != 3 && FORM != 6 && (NZ % 3 == 0 || NZ == 1024);
}
template <int NZ, int FORM> constexpr bool z_valid(int v) {
  constexpr int M = NZ / 2;
  return v == 0 || ((FORM == 1 || FORM == 2 || FORM == 7) && ((v == 1 && !z_rule_slots<NZ, FORM>()) ||
                                  (v == 2 && M % 3 != 0 && M >= 8 && M / 4 <= 256) ||
                                  (v == 3 && std::is_same<T, float>::value && M % 3 != 0 && M >= 8 && M / 4 <= 64) ||
                                  (v == 4 && std::is_same<T, float>::value && M == 512)));
}

// pipelined forward x kernel of a step or of an adjoint step (CW = 0: not used): elements per
// thread, tile columns, buffers, state prefetch into L2.  B200, the four stages' average, us:
// 256x256x256 FP32 rotational 197 (203 without the prefetch, 240 with two buffers; fused TMA
// kernel 235, split 76 + 157), conservative 239 (split 117 + 176); 128x256x256 FP32 91 (99 with
// the prefetch) and 118 (split 35 + 83, 58 + 94); FP64 at 128^3 56 (fused 58, split 18 + 41),
// adjoint 67 (fused 80, split 35 + 51).  FP32 at 512 points (234 against 82 + 160) and FP64 at
// 256 (113 against 36 + 77) gain nothing.
// 32 (FP32) and 64 points: on fields of at most PIPE_SMALL_BYTES, where it saves a launch and the
// products sit in L2.  Steps, us, split -> pipelined, conservative / rotational: FP32 32^3 66 ->
// 64 / 68 -> 65, 64^3 (1 MB per component) 109 -> 93 / 115 -> 102, 32x128x128 (2 MB) 146 -> 127 /
// 147 -> 138; 64x128x128 (4 MB) 196 -> 189 / 193 -> 195, 32x256x256 (9 MB) 328 -> 332 / 326 -> 348;
// FP64 64^3 127 -> 126 / 153 -> 138, but 32^3 75 -> 73 / 92 -> 99
constexpr long long PIPE_SMALL_BYTES = 3000000;
struct PipeTile { int E, CW, NBUF; bool PF; };
constexpr PipeTile pipe_tile(int L, int form) {
  if (form != 3 && L == 64) return PipeTile{8, std::is_same<T, float>::value ? 16 : 8, 1, false};
  if (form != 3 && L == 32 && std::is_same<T, float>::value) return PipeTile{8, 16, 1, false};
  return !std::is_same<T, float>::value
             ? (L == 128 ? (form == 1 ? PipeTile{16, 16, 1, false} : form == 3 ? PipeTile{16, 8, 2, true} : PipeTile{0, 0, 0, false})
                         : PipeTile{0, 0, 0, false})
         : form == 3 ? PipeTile{0, 0, 0, false}
         : L == 256  ? (form == 1 ? PipeTile{16, 16, 1, true} : PipeTile{32, 16, 1, true})
         : L == 128  ? (form == 1 ? PipeTile{16, 32, 2, false} : PipeTile{16, 16, 2, false})
                     : PipeTile{0, 0, 0, false};
}
// lengths whose step takes the split form although the fused kernel's tiles fit: short lines,
// where a fused launch is a serial chain of loads, transforms and updates on few blocks (64^3
// FP64 15 us against 5 + 6, 32^3 FP32 8 against 2 + 2), and FP64 above 128
constexpr bool fx_rule_split(int L) { return L <= 64 || std::is_same<T, float>::value || L > 128; }

// forward x candidates (MODE_STEP): 1 = the split form (strided x FFT, then the
// elementwise epilogue) where the fused TMA kernel's tiles fit (the rule's own form where
// neither the pipelined nor the fused kernel is the rule, see fwd_x_impl); 2 = the fused
// kernel with half-width column tiles (32-byte rows in FP32; where the rule
// splits, the fused kernel at the rule's tile width); 3 = the fused kernel with
// 8 elements per thread (half the threads)
constexpr bool fx_rule_fused(int L) { return xcw(L) * sizeof(V) >= 64; }
constexpr int fx_cw2(int L) { return fx_rule_fused(L) ? xcw(L) / 2 : xcw(L); }
constexpr bool fx_valid(int L, int v) {
  return v == 0 || (v == 1 && fx_rule_fused(L)) || (v == 2 && fx_cw2(L) * sizeof(V) >= 16 && fx_cw2(L) * (L / emin(E_ACC, L)) >= 32) ||
         (v == 3 && fx_rule_fused(L) && emin(E_ACC_ALT, L) != emin(E_ACC, L));
}


// SFF x candidates (k_sff_inv_x, k_sff_fwd_x; the rule is k_sc_x). Inverse: 1 = 4 elements per
// thread (power-of-two lengths), 2 = half-width column tiles. Forward: 1 = fused epilogue from 64
// points on, split below, 2 = half-width column tiles (split from 64 points on, fused below).
constexpr int sx_e(int N, int dir) { return e_mixed(N, dir > 0 ? 8 : (std::is_same<T, float>::value ? 8 : 4)); }
constexpr Tile sx_cand(int N, int dir, int v) {
  return v == 0 ? Tile{sx_e(N, dir), cw_for(N, sx_e(N, dir)), 1}
       : v == 1 ? (dir > 0 ? (N % 3 != 0 && sx_e(N, dir) > 4 ? Tile{4, cw_for(N, 4), 1} : Tile{0, 0, 0})
                           : Tile{sx_e(N, dir), cw_for(N, sx_e(N, dir)), 2})
       : v == 2 ? (cw_for(N, sx_e(N, dir)) > 1 ? Tile{sx_e(N, dir), cw_for(N, sx_e(N, dir)) / 2, 1} : Tile{0, 0, 0})
                : Tile{0, 0, 0};
}
constexpr bool sx_valid(int N, int dir, int v) {
  return v == 0 || (N <= 512 && v < 3 && tile_fits(N, sx_cand(N, dir, v), 3) &&
                    !tile_eq(sx_cand(N, dir, v), sx_cand(N, dir, 0)));
}

#if TS_PART == TS_PART_STR
template <int L, int VV, typename Fn> void with_str_tile(Fn&& fn) {
  if constexpr (str_valid(L, VV)) fn(std::integral_constant<int, VV>{});
  else fn(std::integral_constant<int, 0>{});
}

template <> cudaError_t Launch<T>::strided(const Geo& g, int axis, int dir, void* data, int nf, const void* tw,
                                           cudaStream_t st, int per, long long mstride, int inner_eff,
                                           int zero_hi, void* dst, double scl) {
  if (per <= 0) per = nf;
  cudaError_t err = cudaErrorInvalidValue;
  const int L = axis == 0 ? g.Nx : g.Ny;
  if (L == 1) return cudaSuccess;  // a one-point transform is the identity (two-dimensional runs)
  // the y passes follow the tuning of their class; x passes keep the rule
  const int cls = axis == 1 ? (dir > 0 ? TUNE_Y_INV : TUNE_Y_FWD) : -1;
  const int v = cls >= 0 ? g.tv[cls] : 0, bps = cls >= 0 ? g.tb[cls] : 0;
  // the rule is the direct-load kernel; a tuning candidate or a blocks-per-SM count of a y
  // class launches the persistent kernel (in place, unscaled)
  if (v == 0 && bps == 0) {
    dispatch_L_sff(L, [&](auto Lc) {
      constexpr int LL = decltype(Lc)::value;
      const unsigned inner = inner_eff > 0 ? inner_eff : (axis == 0 ? g.Ny * g.Hz : g.Hz);
      const long long rstride = axis == 0 ? (long long)g.Ny * g.Hz : g.Hz;
      const unsigned nplane = axis == 0 ? inner : inner * (unsigned)g.Nx, ntot = nplane * (unsigned)nf;
      auto tile = [&](auto far) {
        constexpr LdTile c = decltype(far)::value ? far_tile(LL) : ld_tile(LL);
        constexpr size_t sm = (size_t)LL * c.CW * sizeof(V);
        auto launch = [&](auto k) {
          if ((err = smem_attr(k, sm)) != cudaSuccess) return;
          err = launch_chain(chained(g, per == nf ? 1 : nf / per), k, (ntot + c.CW - 1) / c.CW, c.CW * (LL / c.E), sm, st,
                             (const V*)data, (V*)(dst ? dst : data), ntot, nplane, inner, g.S, rstride,
                             (long long)g.Ny * g.Hz, (const V*)tw, (unsigned)per, mstride, zero_hi, (T)scl);
        };
        if (dir > 0) launch(k_strided_ld<T, LL, c.E, c.CW, 1, c.MINB, false>);
        else if (scl == 1.0) launch(k_strided_ld<T, LL, c.E, c.CW, -1, c.MINB, false>);
        else launch(k_strided_ld<T, LL, c.E, c.CW, -1, c.MINB, true>);
      };
      if constexpr (far_tile(LL).CW > 0) {
        if (rstride * (long long)sizeof(V) >= FAR_ROW_BYTES) return tile(std::true_type{});
      }
      tile(std::false_type{});
    });
    return err;
  }
  if ((dst && dst != data) || scl != 1.0) return err;
  dispatch_L_sff(L, [&](auto Lc) {
    constexpr int LL = decltype(Lc)::value;
    auto run = [&](auto vc) {
      constexpr Tile c = str_cand(LL, decltype(vc)::value);
      constexpr int E = c.E, CW = c.CW, NT = c.NT;
      const int inner = inner_eff > 0 ? inner_eff : (axis == 0 ? g.Ny * g.Hz : g.Hz);
      const long long rstride = axis == 0 ? (long long)g.Ny * g.Hz : g.Hz;
      const long long ostride = axis == 0 ? 0 : (long long)g.Ny * g.Hz;
      const int nouter = axis == 0 ? 1 : g.Nx;
      const long long nwork = (long long)nf * ((inner + CW - 1) / CW) * nouter;
      const size_t sm = (size_t)str_tiles(NT) * LL * CW * sizeof(V);
      // persistent grid: as many blocks as fit on the 148 SMs at once (or the tuned count)
      const int cap = (CW * (LL / E)) <= 256 ? 2 : 1;
      const int fit = (int)((227 * 1024) / sm);
      const int per_sm = bps > 0 ? bps : (fit < cap ? fit : cap);
      long long blocks = 148LL * (per_sm > 0 ? per_sm : 1);
      if (blocks > nwork) blocks = nwork;
      auto launch = [&](auto k) {
        if ((err = smem_attr(k, sm)) != cudaSuccess) return;
        k<<<(unsigned)blocks, CW * (LL / E), sm, st>>>((V*)data, nf, g.S, inner, rstride, ostride, nouter,
                                                      (const V*)tw, per, mstride, zero_hi);
        ++g_launches;
        err = cudaGetLastError();
      };
      if (dir < 0) launch(k_strided_fft<T, LL, E, CW, -1, NT>);
      else launch(k_strided_fft<T, LL, E, CW, 1, NT>);
    };
    // 1024 points in FP32: for the y forward pass candidate 5 is the two-tile, 16-element form
    const int vv = wide1024(LL) && v == 0 ? 6 : (wide1024(LL) && dir < 0 && v == 5 ? 0 : v);
    switch (vv) {
      case 6: with_str_tile<LL, 6>(run); break;
      case 1: with_str_tile<LL, 1>(run); break;
      case 2: with_str_tile<LL, 2>(run); break;
      case 3: with_str_tile<LL, 3>(run); break;
      case 4: with_str_tile<LL, 4>(run); break;
      case 5: with_str_tile<LL, 5>(run); break;
      default: run(std::integral_constant<int, 0>{});
    }
  });
  return err;
}
#endif  // TS_PART_STR

#if TS_PART == TS_PART_IX
template <> cudaError_t Launch<T>::inv_x(const Geo& g, int form, const void* U, void* W, const void* tw,
                                         const void* lam, double lsc, cudaStream_t st, int kept, double rad) {
  cudaError_t err_ = cudaErrorInvalidValue;
  // forms 0 and 1 follow the tuning; the adjoint forms keep the rule
  const int v = form <= 1 ? g.tv[TUNE_X_INV] : 0;
  if (v == 0) {
    dispatch_L(g.Nx, [&](auto Lc) {
      constexpr int LL = decltype(Lc)::value;
      constexpr LdTile c = ix_tile(LL);
      const int nzt = g.Hp != g.Hz ? g.Hp : g.Nz / 3 + 1;  // columns of a kept line
      const long long cols = kept ? (long long)(2 * (g.Ny / 3) + 1) * nzt : (long long)g.Ny * g.Hz;
      if (kept) kept = g.Hp != g.Hz ? 2 : 1;
      constexpr size_t sm = (size_t)LL * c.CW * sizeof(V);
      auto run = [&](auto kern, int nf) {
        if ((err_ = smem_attr(kern, sm)) != cudaSuccess) return;
        err_ = launch_chain(chained(g), kern, (unsigned)((cols + c.CW - 1) / c.CW) * nf, c.CW * (LL / c.E), sm, st,
                            (const V*)U, (V*)W, g, (const V*)tw, kept, form == 5 ? k2_limit(rad) : 0.0);
      };
      if (form == 0) run(k_inv_x_f<T, LL, c.E, c.CW, 0, c.MINB>, 3);
      else if (form == 1) run(k_inv_x_f<T, LL, c.E, c.CW, 1, c.MINB>, 6);
      else if (form == 5) run(k_inv_x_f<T, LL, c.E, c.CW, 5, c.MINB>, 3);
      else if (form == 4) {
        // three components in registers: 8 elements per thread
        constexpr int E = 8 < LL ? 8 : 4, CW = cw_for(LL, E), NT = CW * (LL / E);
        constexpr size_t sm4 = (size_t)LL * CW * sizeof(V);
        auto k = k_inv_x_cot<T, LL, E, CW, NT <= 256 ? 256 / NT * (std::is_same<T, float>::value ? 2 : 1) : 1>;
        if ((err_ = smem_attr(k, sm4)) != cudaSuccess) return;
        err_ = launch_chain(chained(g), k, (unsigned)((cols + CW - 1) / CW), NT, sm4, st, (const V*)lam, (V*)W, g,
                            (const V*)tw, (T)lsc);
      }
    });
    return err_;
  }
  dispatch_L(g.Nx, [&](auto Lc) {
    constexpr int LL = decltype(Lc)::value;
    // candidate 5 (1024 points in FP32): tile 0
    const int vv = v == 5 ? 0 : v;
    if constexpr (ix_valid(LL, 3)) {
      if (vv == 3) {
        // persistent, prefetching form: one block per SM
        constexpr Tile c = ix_cand(LL, 3);
        constexpr int E = c.E, CW = c.CW;
        const size_t sm = 4ull * LL * CW * sizeof(V);
        const int nzk = g.Nz / 3 + 1;
        const long long ntiles = kept ? (long long)(2 * (g.Ny / 3) + 1) * ((nzk + CW - 1) / CW)
                                      : (long long)((g.Ny * g.Hz + CW - 1) / CW);
        const unsigned blocks = (unsigned)(ntiles < 148 ? ntiles : 148);
        auto run = [&](auto kern) {
          if ((err_ = smem_attr(kern, sm)) != cudaSuccess) return;
          kern<<<blocks, CW * (LL / E), sm, st>>>((const V*)U, (V*)W, g, (const V*)tw, kept);
          ++g_launches;
          err_ = cudaGetLastError();
        };
        if (form == 0) run(k_inv_x_pf<T, LL, E, CW, 0>);
        else if (form == 1) run(k_inv_x_pf<T, LL, E, CW, 1>);
        return;
      }
    }
    auto tile = [&](auto vc) {
      constexpr Tile c = ix_cand(LL, decltype(vc)::value);
      constexpr int E = c.E, CW = c.CW;
      const int inner = g.Ny * g.Hz;
      const size_t sm = (size_t)LL * CW * sizeof(V);
      const int nzk = g.Nz / 3 + 1;
      const unsigned blocks = kept ? (unsigned)((2 * (g.Ny / 3) + 1) * ((nzk + CW - 1) / CW))
                                   : (unsigned)((inner + CW - 1) / CW);
      auto run = [&](auto kern) {
        if ((err_ = smem_attr(kern, sm)) != cudaSuccess) return;
        kern<<<blocks, CW * (LL / E), sm, st>>>((const V*)U, (V*)W, g, (const V*)tw, kept);
        ++g_launches;
        err_ = cudaGetLastError();
      };
      if (form == 0) run(k_inv_x_ld<T, LL, E, CW, 0>);
      else if (form == 1) run(k_inv_x_ld<T, LL, E, CW, 1>);
    };
    if (vv == 1 && ix_valid(LL, 1)) {
      if constexpr (ix_valid(LL, 1)) tile(std::integral_constant<int, 1>{});
    } else if (vv == 2 && ix_valid(LL, 2)) {
      if constexpr (ix_valid(LL, 2)) tile(std::integral_constant<int, 2>{});
    } else if (vv == 4 && ix_valid(LL, 4)) {
      if constexpr (ix_valid(LL, 4)) tile(std::integral_constant<int, 4>{});
    } else {
      tile(std::integral_constant<int, 0>{});
    }
  });
  return err_;
}
#endif  // TS_PART_IX

#if TS_PART == TS_PART_Z
// shared-memory slot variant of the z pass: E elements per thread, nl lines per
// block within about 106 KB of shared memory
template <int NZ, int FORM, int E>
static cudaError_t z_slots(const Geo& g, void* P, const void* tw, cudaStream_t st, int nmem, long long msP,
                           int zkeep) {
  constexpr int M = NZ / 2;
  constexpr int TPL = M / E;
  constexpr int NIN = z_nin(FORM), NOUT = z_nout(FORM);
  constexpr int NSL = NIN > NOUT ? NIN : NOUT;
  const long long nlines = (long long)g.Nx * g.Ny;
  int nl = 256 / TPL;
  while (nl > 1 && (size_t)NSL * nl * zslot<M>() * sizeof(V) > 106 * 1024) nl /= 2;
  const size_t sm = (size_t)NSL * nl * zslot<M>() * sizeof(V);
  cudaError_t err;
  auto k = k_z_fused<T, NZ, E, FORM>;
  if ((err = smem_attr(k, sm)) != cudaSuccess) return err;
  k<<<dim3((unsigned)((nlines + nl - 1) / nl), nmem), nl * TPL, sm, st>>>((V*)P, g, (const V*)tw, nl, msP, zkeep);
  ++g_launches;
  return cudaGetLastError();
}

template <int NZ, int FORM>
static cudaError_t z_fused_impl(const Geo& g, void* P, const void* tw, int* zerr, cudaStream_t st, int nmem,
                                long long msP, int zkeep, int v, const void* q = nullptr, const void* x = nullptr) {
  constexpr int M = NZ / 2;
  if (zkeep < 0) zkeep = M;
  const long long nlines = (long long)g.Nx * g.Ny;
  cudaError_t err;
  if constexpr (z_valid<NZ, FORM>(1)) {
    if (v == 1) return z_slots<NZ, FORM, e_mixed(M, 8)>(g, P, tw, st, nmem, msP, zkeep);
  }
  if constexpr (z_valid<NZ, FORM>(2)) {
    if (v == 2) return z_slots<NZ, FORM, 4>(g, P, tw, st, nmem, msP, zkeep);
  }
  if constexpr (z_valid<NZ, FORM>(4)) {
    if (v == 4) {
      constexpr int NT = zreg_threads<FORM>(), LPB = NT / (M / 8);
      k_z_reg<T, NZ, FORM, 0, false><<<dim3((unsigned)((nlines + LPB - 1) / LPB), nmem), NT, 0, st>>>(
          (V*)P, g, (const V*)tw, msP, zkeep);
      ++g_launches;
      return cudaGetLastError();
    }
  }
  if constexpr (zreg_rule<NZ, FORM>()) {
    constexpr int E = M % 3 == 0 ? 12 : 8, NT = zreg_threads<FORM>(), LPB = NT / (M / E);
    return launch_chain(chained(g, nmem), k_z_reg<T, NZ, FORM, 0, true>, dim3((unsigned)((nlines + LPB - 1) / LPB), nmem),
                        NT, 0, st, (V*)P, g, (const V*)tw, msP, zkeep);
  }
  if constexpr (z_valid<NZ, FORM>(3)) {
    if (v == 3) {
      constexpr int NT = zreg_threads<FORM>(), LPB = NT / (M / 4);
      k_z_reg<T, NZ, FORM, 4><<<dim3((unsigned)((nlines + LPB - 1) / LPB), nmem), NT, 0, st>>>((V*)P, g, (const V*)tw,
                                                                                              msP, zkeep);
      ++g_launches;
      return cudaGetLastError();
    }
  }
  if constexpr (FORM != 3) {
    // the rule: line pairs
    constexpr ZTile c = zp_tile(NZ, FORM);
    constexpr int PPB = c.NTHR / (NZ / c.E);
    constexpr size_t sm = (size_t)PPB * zpair_lines(z_nin(FORM), c.NB) * zpair_slot<T>(NZ) * sizeof(V);
    const long long npairs = (nlines + 1) / 2;
    auto k = k_z_pair<T, NZ, c.E, FORM, c.NTHR, c.MINB, c.NB>;
    if ((err = smem_attr(k, sm)) != cudaSuccess) return err;
    return launch_chain(chained(g, nmem), k, dim3((unsigned)((npairs + PPB - 1) / PPB), nmem), c.NTHR, sm, st, (V*)P, g,
                        (const V*)tw, msP, zkeep, (const V*)(q ? q : P), (const V*)x);
  }
  if constexpr (FORM == 3) {
    constexpr ZTile c = zp_tile(NZ, FORM);
    constexpr int PPB = c.NTHR / (NZ / c.E);
    constexpr size_t sm = ((size_t)PPB * 3 * zpair_slot<T>(NZ) + 3ull * c.E * c.NTHR) * sizeof(V);
    const long long npairs = (nlines + 1) / 2;
    auto k = k_z_pair_adj<T, NZ, c.E, c.NTHR, c.MINB>;
    if ((err = smem_attr(k, sm)) != cudaSuccess) return err;
    return launch_chain(chained(g), k, (unsigned)((npairs + PPB - 1) / PPB), c.NTHR, sm, st, (V*)P, g, (const V*)tw, zkeep);
  }
}

template <> cudaError_t Launch<T>::z_fused(const Geo& g, int form, void* P, const void* tw, int* zerr,
                                           cudaStream_t st, int nmem, long long msP, int zkeep, const void* q,
                                           const void* x) {
  cudaError_t err = cudaErrorInvalidValue;
  if (form == 3 && nmem != 1) return err;  // the adjoint z pass has no member batching
  if (x && nmem != 1) return err;
  dispatch_L_sff(g.Nz, [&](auto Lc) {
    constexpr int NZ = decltype(Lc)::value;
    const int v = g.tv[TUNE_Z];
    if (form == 7) err = z_fused_impl<NZ, 7>(g, P, tw, zerr, st, nmem, msP, zkeep, v, nullptr, x);
    else if (form == 0) err = z_fused_impl<NZ, 0>(g, P, tw, zerr, st, nmem, msP, zkeep, 0, nullptr, x);
    else if (form == 1) err = z_fused_impl<NZ, 1>(g, P, tw, zerr, st, nmem, msP, zkeep, v, nullptr, x);
    else if (form == 2) err = z_fused_impl<NZ, 2>(g, P, tw, zerr, st, nmem, msP, zkeep, v);
    else if (form == 5) err = z_fused_impl<NZ, 5>(g, P, tw, zerr, st, nmem, msP, zkeep, 0, nullptr, x);
    else if (form == 6) err = z_fused_impl<NZ, 6>(g, P, tw, zerr, st, nmem, msP, zkeep, 0, q);
    else if constexpr (NZ % 3 != 0) err = z_fused_impl<NZ, 3>(g, P, tw, zerr, st, 1, 0, zkeep, 0);
  });
  return err;
}

// SSS z pass (forms 7, 2, 6): line pairs, tiles as the Fourier z pass
template <int NZ, int FORM>
static cudaError_t sss_z_pairs(const Geo& g, void* P, const void* tw, const void* tq, int zin, int zout,
                               cudaStream_t st) {
  constexpr ZTile c = zp_tile(NZ, FORM);
  constexpr int PPB = c.NTHR / (NZ / c.E);
  constexpr size_t sm = (size_t)PPB * zpair_lines(z_nin(FORM), c.NB) * zpair_slot<T>(NZ) * sizeof(V);
  const long long npairs = ((long long)g.Nx * g.Ny + 1) / 2;
  cudaError_t err;
  auto k = k_sss_z_pair<T, NZ, c.E, FORM, c.NTHR, c.MINB, c.NB>;
  if ((err = smem_attr(k, sm)) != cudaSuccess) return err;
  return launch_chain(chained(g), k, (unsigned)((npairs + PPB - 1) / PPB), c.NTHR, sm, st, (V*)P, g, (const V*)tw,
                      (const V*)tq, zin, zout, (T)(1.0 / (2.0 * NZ)));
}

template <> cudaError_t Launch<T>::sss_z_fused(const Geo& g, int form, void* P, const void* tw, const void* tq, int zin,
                                               int zout, cudaStream_t st) {
  cudaError_t err = cudaErrorInvalidValue;
  if (form != 7 && form != 2 && form != 6) return err;
  dispatch_L(g.Nz, [&](auto Lc) {
    constexpr int NZ = decltype(Lc)::value;
    err = form == 7 ? sss_z_pairs<NZ, 7>(g, P, tw, tq, zin, zout, st)
        : form == 2 ? sss_z_pairs<NZ, 2>(g, P, tw, tq, zin, zout, st)
                    : sss_z_pairs<NZ, 6>(g, P, tw, tq, zin, zout, st);
  });
  return err;
}

template <> cudaError_t Launch<T>::z_single(const Geo& g, int dir, const void* in, void* out, int ncomp,
                                            const void* tw, cudaStream_t st) {
  cudaError_t err = cudaErrorInvalidValue;
  dispatch_L(g.Nz, [&](auto Lc) {
    constexpr int NZ = decltype(Lc)::value;
    constexpr int E = emin(16, NZ / 2), TPL = NZ / E, NT = TPL > 128 ? TPL : 128, PPB = NT / TPL;
    constexpr size_t sm = (size_t)PPB * zpair_slot<T>(NZ) * sizeof(V);
    const long long npairs = ((long long)g.Nx * g.Ny + 1) / 2;
    const dim3 grid((unsigned)((npairs + PPB - 1) / PPB), ncomp);
    auto run = [&](auto k) {
      if ((err = smem_attr(k, sm)) != cudaSuccess) return;
      k<<<grid, NT, sm, st>>>((const V*)in, (V*)out, g, (const V*)tw);
      ++g_launches;
      err = cudaGetLastError();
    };
    constexpr int MINB = std::is_same<T, float>::value ? 6 : 3;
    if (dir < 0) run(k_z_single<T, NZ, E, -1, NT, MINB>);
    else run(k_z_single<T, NZ, E, 1, NT, MINB>);
  });
  return err;
}
#endif  // TS_PART_Z

#if TS_PART == TS_PART_FX
template <int FORM, int MODE, int LL, int E, int CW>
static cudaError_t fwd_x_fused(const Geo& g, const void* P, const StageArgs& a, const void* tw, cudaStream_t st);

// pipelined forward x kernel of a step
template <int FORM, int LL>
static cudaError_t fwd_x_pipe(const Geo& g, const void* P, const StageArgs& a, const void* tw, cudaStream_t st) {
  constexpr PipeTile c = pipe_tile(LL, FORM);
  constexpr size_t sm = (size_t)c.NBUF * z_nout(FORM) * LL * c.CW * sizeof(V) + LL * pipe_row_bytes();
  const unsigned ntiles = (unsigned)(g.Ny * g.Hz / c.CW), most = LL <= 64 ? 2 * 148u : 148u, blocks = ntiles < most ? ntiles : most;
  cudaError_t err = cudaErrorInvalidValue;
  auto run = [&](auto k) {
    if ((err = smem_attr(k, sm)) != cudaSuccess) return;
    err = launch_chain(chained(g), k, blocks, z_nout(FORM) * c.CW * (LL / c.E), sm, st, (const V*)P, g, a, (const V*)tw);
  };
  if (a.stage == 1) run(k_fwd_x_pipe<T, LL, c.E, c.CW, FORM, 1, c.NBUF, c.PF>);
  else if (a.stage == 2) run(k_fwd_x_pipe<T, LL, c.E, c.CW, FORM, 2, c.NBUF, c.PF>);
  else if (a.stage == 3) run(k_fwd_x_pipe<T, LL, c.E, c.CW, FORM, 3, c.NBUF, c.PF>);
  else run(k_fwd_x_pipe<T, LL, c.E, c.CW, FORM, 4, c.NBUF, c.PF>);
  return err;
}

template <int FORM, int MODE, int LL>
static cudaError_t fwd_x_impl(const Geo& g, const void* P, const StageArgs& a, const void* tw, cudaStream_t st) {
  constexpr int CW = xcw(LL);
  const int v = MODE == MODE_STEP ? g.tv[TUNE_X_FWD] : 0;
  if constexpr (fx_valid(LL, 2)) {
    if (v == 2) return fwd_x_fused<FORM, MODE, LL, emin(E_ACC, LL), fx_cw2(LL)>(g, P, a, tw, st);
  }
  if constexpr (fx_valid(LL, 3)) {
    if (v == 3) return fwd_x_fused<FORM, MODE, LL, emin(E_ACC_ALT, LL), CW>(g, P, a, tw, st);
  }
  // the rule (a blocks-per-SM count of the tuning launches the fused TMA kernel): the
  // pipelined kernel where it has a tile and the tiles divide the columns, otherwise the split
  // form of a step (fx_rule_split) and the fused kernel of the other modes
  const bool rule = v == 0 && !(MODE == MODE_STEP && g.tb[TUNE_X_FWD] > 0);
  // state pointers as the fused kernel's tensor maps take them
  const void* sA = MODE == MODE_FLUX ? a.Ud : ((MODE == MODE_STEP || MODE == MODE_ADJ) ? a.U0 : P);
  const void* sB = (MODE == MODE_STEP || MODE == MODE_ADJ) ? a.tot : P;
  const bool fused16 = fx_rule_fused(LL) && (((uintptr_t)sA | (uintptr_t)sB) & 15);
  if (fused16 && !(MODE == MODE_STEP && v == 1)) return cudaErrorInvalidValue;
  if constexpr ((MODE == MODE_STEP || MODE == MODE_ADJ) && pipe_tile(LL, FORM).CW > 0) {
    const bool fits = LL > 64 || g.S * (long long)sizeof(V) <= PIPE_SMALL_BYTES;
    if (rule && fits && g.Ny * g.Hz % pipe_tile(LL, FORM).CW == 0) return fwd_x_pipe<FORM, LL>(g, P, a, tw, st);
  }
  const bool split = CW * sizeof(V) < 64 || v == 1 || (rule && MODE == MODE_STEP && fx_rule_split(LL));
  if (split) {
    // tiles narrower than 64-byte rows: forward x FFT in place, then the elementwise epilogue
    constexpr int NF = z_nout(FORM);
    cudaError_t err = Launch<T>::strided(g, 0, -1, const_cast<void*>(P), NF, tw, st);
    if (err != cudaSuccess) return err;
    const unsigned blocks = grid1d(g.S, 256);
    if ((err = launch_chain(chained(g), k_spec_epi<T, FORM, MODE>, blocks, 256, 0, st, (const V*)P, g, a)) != cudaSuccess)
      return err;
    if (MODE == MODE_FLUX) {
      k_bins_finish<<<8, 256, 0, st>>>(a.bins + (a.nradii + 1), (int)blocks, a.nradii + 1, a.bins);
      ++g_launches;
    }
    return cudaGetLastError();
  }
  if constexpr (CW * sizeof(V) >= 64) return fwd_x_fused<FORM, MODE, LL, emin(E_ACC, LL), CW>(g, P, a, tw, st);
  return cudaErrorInvalidValue;
}

template <int FORM, int MODE, int LL, int E, int CW>
static cudaError_t fwd_x_fused(const Geo& g, const void* P, const StageArgs& a, const void* tw, cudaStream_t st) {
  const int inner = g.Ny * g.Hz;
  const int ntiles = (inner + CW - 1) / CW;
  size_t sm = (size_t)(MODE == MODE_NLIN ? 2 : 8) * LL * CW * sizeof(V) + (size_t)LL * (CW + 1) * sizeof(V) + 128;
  const int bps = MODE == MODE_STEP ? g.tb[TUNE_X_FWD] : 0;
  const int per_sm = bps > 0 ? bps : ((int)((220 * 1024) / sm) >= 2 ? 2 : 1);
  const int blocks = ntiles < 148 * per_sm ? ntiles : 148 * per_sm;
  const int br = LL < 256 ? LL : 256;
  CUtensorMap mP, mA, mB;
  cudaError_t err = make_field_map(&mP, P, inner, 6LL * g.Nx, UNITS, CW, br);
  if (err != cudaSuccess) return err;
  const void* A = MODE == MODE_FLUX ? a.Ud : ((MODE == MODE_STEP || MODE == MODE_ADJ) ? a.U0 : P);
  const void* B = (MODE == MODE_STEP || MODE == MODE_ADJ) ? a.tot : P;
  if ((err = make_field_map(&mA, A, inner, 3LL * g.Nx, UNITS, CW, br)) != cudaSuccess) return err;
  if ((err = make_field_map(&mB, B, inner, 3LL * g.Nx, UNITS, CW, br)) != cudaSuccess) return err;
  auto k = k_fwd_x<T, LL, E, CW, FORM, MODE>;
  if ((err = smem_attr(k, sm)) != cudaSuccess) return err;
  if ((err = launch_chain(chained(g), k, blocks, CW * (LL / E), sm, st, mP, mA, mB, g, a, (const V*)tw)) != cudaSuccess)
    return err;
  if (MODE == MODE_FLUX) {
    k_bins_finish<<<8, 256, 0, st>>>(a.bins + (a.nradii + 1), blocks, a.nradii + 1, a.bins);
    ++g_launches;
  }
  return cudaGetLastError();
}

// Line pitch of the inverse-transformed fields of a two-thirds dealiased FFF step of product
// form `form`.  Only the nzk = Nz / 3 + 1 columns kz <= Nz / 3 are ever written there.  In lines
// of Hz = Nz / 2 + 1 elements (odd) they start at any element, a column tile straddles lines,
// and its 128-byte row segments cost five or six sectors of two cache lines each; in compact
// lines of whole 16-column tiles every segment is one aligned cache line, and the z pass writes
// the products elsewhere in lines of Hz.  B200, 256^3 FP32 rotational: inverse x 100 -> 72 us,
// y inverse 112 -> 92.  Lines up to an eighth longer than nzk only (128 points and more: 43 of
// 48, 86 of 96, 171 of 176 columns; at 64 points 22 of 32, and the fields sit in L2), FP32 only
// (in FP64 a segment of unaligned columns costs one sector more of five: 22.1 and 21.9 us), and
// with the rule's kernels in the three inverse passes.
template <> int Launch<T>::inverse_pitch(const Geo& g, int form) {
  if (!std::is_same<T, float>::value || g.basis != 0 || g.dealias != 2) return g.Hz;
  if (form != 0 && form != 1 && form != 5 && form != 7) return g.Hz;
  for (int c : {TUNE_X_INV, TUNE_Y_INV, TUNE_Z})
    if (g.tv[c] || g.tb[c]) return g.Hz;
  if (g.Nz % 3 == 0 || g.Nz == 1024) return g.Hz;  // zreg_rule: in place
  const int nzk = g.Nz / 3 + 1, p = (nzk + 15) / 16 * 16;
  return 8 * p <= 9 * nzk && p < g.Hz ? p : g.Hz;
}

template <> cudaError_t Launch<T>::fwd_x(const Geo& g, int form, int mode, const void* P, const StageArgs& a,
                                         const void* tw, cudaStream_t st) {
  cudaError_t err = cudaErrorInvalidValue;
  dispatch_L(g.Nx, [&](auto Lc) {
    constexpr int LL = decltype(Lc)::value;
    if (form == 3) {
      if (mode == MODE_ADJ) err = fwd_x_impl<3, MODE_ADJ, LL>(g, P, a, tw, st);
    } else if (form == 1) {
      if (mode == MODE_STEP) err = fwd_x_impl<1, MODE_STEP, LL>(g, P, a, tw, st);
      else if (mode == MODE_FLUX) err = fwd_x_impl<1, MODE_FLUX, LL>(g, P, a, tw, st);
      else err = fwd_x_impl<1, MODE_NLIN, LL>(g, P, a, tw, st);
    } else {
      if (mode == MODE_STEP) err = fwd_x_impl<7, MODE_STEP, LL>(g, P, a, tw, st);
      else if (mode == MODE_FLUX) err = fwd_x_impl<0, MODE_FLUX, LL>(g, P, a, tw, st);
      else err = fwd_x_impl<0, MODE_NLIN, LL>(g, P, a, tw, st);
    }
  });
  return err;
}
#endif  // TS_PART_FX

#if TS_PART == TS_PART_SFF
template <> cudaError_t Launch<T>::sc_x(const Geo& g, int dir, const ScArgs& a, const void* tq, cudaStream_t st, int nf,
                                        int nmem) {
  cudaError_t err = cudaErrorInvalidValue;
  dispatch_L_sff(g.Nx, [&](auto Lc) {
    constexpr int NN = decltype(Lc)::value;
    if constexpr (NN <= 512) {
      constexpr LdTile c = sc_tile(NN, 1), cf = sc_tile(NN, -1);
      static_assert(c.E == cf.E && c.CW == cf.CW, "one tile per length");
      const long long cols = (long long)a.nplanes * g.Ny * g.Hz;
      constexpr size_t sm = (size_t)NN * c.CW * sizeof(V);
      const dim3 grid((unsigned)((cols + c.CW - 1) / c.CW), nmem, nf);
      auto run = [&](auto k) {
        if ((err = smem_attr(k, sm)) != cudaSuccess) return;
        err = launch_chain(chained_sc(g, nmem), k, grid, c.CW * (NN / c.E), sm, st, a, g, (const V*)tq);
      };
      if (dir < 0) run(k_sc_x<T, NN, c.E, c.CW, -1, cf.MINB>);
      else run(k_sc_x<T, NN, c.E, c.CW, 1, c.MINB>);
    }
  });
  return err;
}

template <> cudaError_t Launch<T>::sff_inv_x(const Geo& g, const void* U, const void* Tf, void* W, const void* tq,
                                             cudaStream_t st, int nmem, long long msU, long long msT, long long msW) {
  cudaError_t err = cudaErrorInvalidValue;
  const int v = g.tv[TUNE_X_INV];
  if (v == 0) {
    // the rule: one block per column tile and field
    ScArgs a{};
    a.s0 = U;
    a.s3 = Tf;
    a.d = W;
    a.sF = a.dF = a.plane = g.S;
    a.ms0 = msU;
    a.ms3 = msT;
    a.msd = msW;
    a.nplanes = 1;
    a.smask = 0x9;  // u1 and T sine series
    a.scl = 1.0;
    a.deal = g.dealias != 0;
    return sc_x(g, +1, a, tq, st, 4, nmem);
  }
  dispatch_L_sff(g.Nx, [&](auto Lc) {
    constexpr int NN = decltype(Lc)::value;
    if constexpr (NN <= 512) {
      // one NN-point FFT per column and field, 8 elements per thread
      auto run = [&](auto vc) {
        constexpr Tile c = sx_cand(NN, 1, decltype(vc)::value);
        constexpr int E = c.E, CW = c.CW;
        const int inner = g.Ny * g.Hz;
        const size_t sm = 3ull * NN * CW * sizeof(V);  // exchange + 2 staging tiles
        auto k = k_sff_inv_x<T, NN, E, CW>;
        if ((err = smem_attr(k, sm)) != cudaSuccess) return;
        k<<<dim3((inner + CW - 1) / CW, nmem), CW * (NN / E), sm, st>>>((const V*)U, (const V*)Tf, (V*)W, g,
                                                                     (const V*)tq, msU, msT, msW);
        ++g_launches;
        err = cudaGetLastError();
      };
      if (v == 1 && sx_valid(NN, 1, 1)) {
        if constexpr (sx_valid(NN, 1, 1)) run(std::integral_constant<int, 1>{});
      } else if (v == 2 && sx_valid(NN, 1, 2)) {
        if constexpr (sx_valid(NN, 1, 2)) run(std::integral_constant<int, 2>{});
      }
    }
  });
  return err;
}

template <> cudaError_t Launch<T>::sff_fwd_x(const Geo& g, const void* P, const SffArgs& a, const void* tq,
                                             cudaStream_t st, int nmem) {
  cudaError_t err = cudaErrorInvalidValue;
  const int v = g.tv[TUNE_X_FWD];
  if (v == 0) {
    // the rule: the eight products transformed in place, then the elementwise epilogue
    ScArgs s{};
    s.s0 = P;
    s.d = const_cast<void*>(P);
    s.sF = s.dF = s.plane = g.S;
    s.ms0 = s.msd = a.msP;
    s.nplanes = 1;
    for (int f = 0; f < 8; ++f) s.smask |= sff_prod_sine(f) << f;
    s.scl = 1.0 / (2.0 * g.Nx * (double)g.Ny * g.Nz);
    if ((err = sc_x(g, -1, s, tq, st, 8, nmem)) != cudaSuccess) return err;
    return launch_chain(chained(g, nmem), k_sff_prod_epi<T>, dim3(grid1d(g.S, 256), nmem), 256, 0, st, (const V*)P, g, a);
  }
  dispatch_L_sff(g.Nx, [&](auto Lc) {
    constexpr int NN = decltype(Lc)::value;
    if constexpr (NN <= 512) {
      // one NN-point FFT per column and product; four accumulators per element:
      // 8 (FP32) / 4 (FP64) elements per thread
      auto run = [&](auto vc) {
        constexpr Tile c = sx_cand(NN, -1, decltype(vc)::value);
        constexpr int E = c.E, CW = c.CW;
        const int inner = g.Ny * g.Hz;
        const size_t sm = 3ull * NN * CW * sizeof(V);
        // from 64 points on, the x kernel writes the assembled vectors and a coalesced
        // elementwise kernel does the epilogue (its ten state reads stalled the fused form)
        constexpr bool SPLIT = (NN >= 64) != (c.NT == 2);
        auto k = k_sff_fwd_x<T, NN, E, CW, SPLIT>;
        if ((err = smem_attr(k, sm)) != cudaSuccess) return;
        k<<<dim3((inner + CW - 1) / CW, nmem), CW * (NN / E), sm, st>>>((V*)P, g, a, (const V*)tq);
        ++g_launches;
        if ((err = cudaGetLastError()) != cudaSuccess || !SPLIT) return;
        k_sff_epi<T><<<dim3(grid1d(g.S, 256), nmem), 256, 0, st>>>((const V*)P, g, a);
        ++g_launches;
        err = cudaGetLastError();
      };
      if (v == 1 && sx_valid(NN, -1, 1)) {
        if constexpr (sx_valid(NN, -1, 1)) run(std::integral_constant<int, 1>{});
      } else if (v == 2 && sx_valid(NN, -1, 2)) {
        if constexpr (sx_valid(NN, -1, 2)) run(std::integral_constant<int, 2>{});
      }
    }
  });
  return err;
}

template <> cudaError_t Launch<T>::sff_x(const Geo& g, int dir, void* A, int ncomp, int sine, double scl,
                                         const void* tq, cudaStream_t st, int nbatch, long long bstride,
                                         const void* src, int deal) {
  ScArgs a{};
  a.s0 = src ? src : A;
  a.d = A;
  a.sF = a.dF = bstride;
  a.plane = g.S;
  a.nplanes = ncomp;
  a.smask = sine;
  a.scl = scl;
  a.deal = deal;
  return sc_x(g, dir, a, tq, st, nbatch);
}
#endif  // TS_PART_SFF

#if TS_PART == TS_PART_MISC
template <> cudaError_t Launch<T>::reality(const Geo& g, void* A, int ncomp, cudaStream_t st) {
  const long long n = (long long)g.Nx * g.Ny * ncomp;
  return launch_chain(chained(g, (ncomp + 2) / 3), k_reality<T>, (unsigned)((n + 255) / 256), 256, 0, st, (V*)A, ncomp, g);
}

template <> cudaError_t Launch<T>::rbc_slave(const Geo& g, void* U, void* Tf, int slave, double vs, cudaStream_t st) {
  k_rbc_slave<T><<<grid1d(g.S, 256), 256, 0, st>>>((V*)U, (V*)Tf, g, slave, vs);
  ++g_launches;
  return cudaGetLastError();
}

template <> cudaError_t Launch<T>::reality_adj(const Geo& g, void* A, int ncomp, cudaStream_t st) {
  const long long n = (long long)g.Nx * g.Ny * ncomp;
  k_reality_adj<T><<<(unsigned)((n + 255) / 256), 256, 0, st>>>((V*)A, ncomp, g);
  ++g_launches;
  return cudaGetLastError();
}

template <> cudaError_t Launch<T>::carati(const Geo& g, const void* U, void* fc, int km, double rin, double rout,
                                          const double* es, const double* hs, const double* mis, int nsup,
                                          cudaStream_t st) {
  return launch_chain(chained(g), k_carati<T>, 1, 256, 0, st, (const V*)U, (V*)fc, g, km, rin, rout, es, hs, mis, nsup);
}

template <> cudaError_t Launch<T>::energy(const Geo& g, const void* A, const void* B, int ncomp, double* out,
                                          cudaStream_t st) {
  // out[0] = the sum; out[1 .. blocks] hold the per-block partial sums (blocks <= 148 * 16)
  const unsigned blocks = grid1d(g.S, 256);
  k_energy<T><<<blocks, 256, 0, st>>>((const V*)A, (const V*)B, ncomp, g, out);
  k_sum_partials<<<1, 256, 0, st>>>(out, (int)blocks);
  g_launches += 2;
  return cudaGetLastError();
}

template <> cudaError_t Launch<T>::maxdiv(const Geo& g, const void* U, unsigned long long* out, cudaStream_t st) {
  k_maxdiv<T><<<grid1d(g.S, 256), 256, 0, st>>>((const V*)U, g, out);
  ++g_launches;
  return cudaGetLastError();
}

template <> cudaError_t Launch<T>::shell(const Geo& g, const void* A, int ncomp, int nbins, double* bins,
                                         cudaStream_t st, const void* B, unsigned cap) {
  const size_t sm = (size_t)(SHELL_WARPS + 1) * nbins * sizeof(double);
  if (sm > 220 * 1024) return cudaErrorInvalidValue;
  cudaError_t err = smem_attr(k_shell<T>, sm);
  if (err != cudaSuccess) return err;
  const unsigned blocks = shell_blocks(g, cap);
  k_shell<T><<<blocks, 32 * SHELL_WARPS, sm, st>>>((const V*)A, (const V*)B, ncomp, g, nbins, bins + 2 * nbins);
  k_bins_finish<<<(2 * nbins + 7) / 8, 256, 0, st>>>(bins + 2 * nbins, (int)blocks, 2 * nbins, bins);
  g_launches += 2;
  return cudaGetLastError();
}

template <> cudaError_t Launch<T>::expire_wait(int* err, int polls, cudaStream_t st) {
  k_expire_wait<<<1, 32, 0, st>>>(err, polls);
  ++g_launches;
  return cudaGetLastError();
}

template <> cudaError_t Launch<T>::flux_finish(const Geo& g, const double* part, long long pitch, int n_radii, double* res,
                                               cudaStream_t st) {
  k_sum_partials_many<<<n_radii, 256, 0, st>>>(part, pitch, (int)grid1d((g.basis == 3 ? 2 : 1) * g.S, 256), res);
  ++g_launches;
  return cudaGetLastError();
}

template <> cudaError_t Launch<T>::flux_outside(const Geo& g, const void* P, const void* U, double R, double* out,
                                                cudaStream_t st) {
  const unsigned blocks = grid1d(g.S, 256);
  k_flux_outside<T><<<blocks, 256, 0, st>>>((const V*)P, (const V*)U, g, k2_limit(R), out);
  ++g_launches;
  return cudaGetLastError();
}
template <> cudaError_t Launch<T>::ssf_giver(const Geo& g, const void* U, void* P, double R, cudaStream_t st) {
  k_ssf_giver<T><<<grid1d(g.S, 256), 256, 0, st>>>((const V*)U, (V*)P, g, R);
  ++g_launches;
  return cudaGetLastError();
}

template <> cudaError_t Launch<T>::ssf_flux_outside(const Geo& g, const void* P, const void* U, double R, int qx,
                                                    int qy, double* out, cudaStream_t st) {
  const unsigned blocks = grid1d(g.S, 256);
  k_ssf_flux_outside<T><<<blocks, 256, 0, st>>>((const V*)P, (const V*)U, g, R, qx, qy, out);
  ++g_launches;
  return cudaGetLastError();
}

template <> cudaError_t Launch<T>::sss_giver(const Geo& g, const void* U, void* P, double R, cudaStream_t st) {
  k_sss_giver<T><<<grid1d(2 * g.S, 256), 256, 0, st>>>((const T*)U, (T*)P, g, R);
  ++g_launches;
  return cudaGetLastError();
}

template <> cudaError_t Launch<T>::sss_flux_outside(const Geo& g, const void* P, const void* U, double R, int qx,
                                                    int qy, int qz, double* out, cudaStream_t st) {
  const unsigned blocks = grid1d(2 * g.S, 256);
  k_sss_flux_outside<T><<<blocks, 256, 0, st>>>((const T*)P, (const T*)U, g, R, qx, qy, qz, out);
  ++g_launches;
  return cudaGetLastError();
}

template <> cudaError_t Launch<T>::force_scatter(const Geo& g, const void* fc, void* F, int km, cudaStream_t st) {
  const long long n = 3LL * (2 * km + 1) * (2 * km + 1) * (km + 1);
  k_force_scatter<T><<<(unsigned)((n + 255) / 256), 256, 0, st>>>((const V*)fc, (V*)F, g, km);
  ++g_launches;
  return cudaGetLastError();
}

template <> cudaError_t Launch<T>::init_ic(const Geo& g, void* U, const double* Eic, const double* mis, int nsh,
                                           unsigned long long key, cudaStream_t st) {
  k_init_ic<T><<<grid1d(g.S, 256), 256, 0, st>>>((V*)U, g, Eic, mis, nsh, key);
  ++g_launches;
  return cudaGetLastError();
}

template <> cudaError_t Launch<T>::init_temp(const Geo& g, void* A, double amp, double kmax, unsigned long long key,
                                             cudaStream_t st) {
  k_init_temp<T><<<grid1d(g.S, 256), 256, 0, st>>>((V*)A, g, amp, kmax, key);
  ++g_launches;
  return cudaGetLastError();
}

template <> cudaError_t Launch<T>::scale(void* A, long long n, double s, cudaStream_t st) {
  k_scale<T><<<grid1d(n, 256), 256, 0, st>>>((V*)A, n, s);
  ++g_launches;
  return cudaGetLastError();
}

template <> cudaError_t Launch<T>::scalar_epi(const Geo& g, const void* P, const SffArgs& a, cudaStream_t st) {
  return launch_chain(chained(g), k_scalar_epi<T>, grid1d(g.S, 256), 256, 0, st, (const V*)P, g, a);
}

template <> cudaError_t Launch<T>::sss_zperm_fwd(const void* u, void* v, long long nlines, int N, int sine,
                                                cudaStream_t st) {
  k_sss_zperm_fwd<T><<<grid1d(nlines * (N + 2), 256), 256, 0, st>>>((const T*)u, (T*)v, nlines, N, sine);
  ++g_launches;
  return cudaGetLastError();
}
template <> cudaError_t Launch<T>::sss_zpost_fwd(const void* Z, void* c, long long nlines, int N, int sine, double scl,
                                                const void* tq, cudaStream_t st) {
  k_sss_zpost_fwd<T><<<grid1d(nlines * (N + 2), 256), 256, 0, st>>>((const V*)Z, (T*)c, nlines, N, sine, scl,
                                                                     (const V*)tq);
  ++g_launches;
  return cudaGetLastError();
}
template <> cudaError_t Launch<T>::sss_zpre_inv(const void* c, void* Vout, long long nlines, int N, int sine,
                                               const void* tq, cudaStream_t st) {
  k_sss_zpre_inv<T><<<grid1d(nlines * (N / 2 + 1), 256), 256, 0, st>>>((const T*)c, (V*)Vout, nlines, N, sine,
                                                                        (const V*)tq);
  ++g_launches;
  return cudaGetLastError();
}
template <> cudaError_t Launch<T>::sss_zperm_inv(const void* v, void* u, long long nlines, int N, int sine,
                                                cudaStream_t st) {
  k_sss_zperm_inv<T><<<grid1d(nlines * (N + 2), 256), 256, 0, st>>>((const T*)v, (T*)u, nlines, N, sine);
  ++g_launches;
  return cudaGetLastError();
}

template <> cudaError_t Launch<T>::sss_dealias_copy(const Geo& g, const void* A, void* B, int ncomp,
                                                   cudaStream_t st) {
  k_sss_dealias_copy<T><<<dim3(grid1d(g.S, 256), ncomp), 256, 0, st>>>((const T*)A, (T*)B, ncomp, g);
  ++g_launches;
  return cudaGetLastError();
}
template <> cudaError_t Launch<T>::sss_epi(const Geo& g, const void* P, const StageArgs& a, cudaStream_t st) {
  return launch_chain(chained(g), k_sss_epi<T>, grid1d(2 * g.S, 256), 256, 0, st, (const T*)P, g, a);
}


template <> cudaError_t Launch<T>::ssf_epi(const Geo& g, const void* P, const StageArgs& a, cudaStream_t st) {
  return launch_chain(chained(g), k_ssf_epi<T>, grid1d(g.S, 256), 256, 0, st, (const V*)P, g, a);
}

template <> cudaError_t Launch<T>::ssf_rbc_epi(const Geo& g, const void* P, const SffArgs& a, cudaStream_t st) {
  return launch_chain(chained(g), k_ssf_rbc_epi<T>, grid1d(g.S, 256), 256, 0, st, (const V*)P, g, a);
}

template <> cudaError_t Launch<T>::sss_rbc_epi(const Geo& g, const void* P, const SffArgs& a, cudaStream_t st) {
  return launch_chain(chained(g), k_sss_rbc_epi<T>, grid1d(2 * g.S, 256), 256, 0, st, (const T*)P, g, a);
}

template <> cudaError_t Launch<T>::mhd_epi(const Geo& g, const void* P, const SffArgs& a, cudaStream_t st) {
  return launch_chain(chained(g), k_mhd_epi<T>, grid1d(g.S, 256), 256, 0, st, (const V*)P, g, a);
}

template <> cudaError_t Launch<T>::dealias_copy(const Geo& g, const void* A, void* B, int ncomp, cudaStream_t st) {
  k_dealias_copy<T><<<dim3(grid1d(g.S, 256), ncomp), 256, 0, st>>>((const V*)A, (V*)B, ncomp, g);
  ++g_launches;
  return cudaGetLastError();
}

template <> bool Launch<T>::tune_valid(const Geo& g, int form, int cls, int v) {
  if (v == 0) return true;
  if (v < 0 || v >= NCAND) return false;
  const bool sff = g.basis == 1;
  bool ok = false;
  switch (cls) {
    case TUNE_Y_INV:
    case TUNE_Y_FWD:
      dispatch_L_sff(g.Ny, [&](auto Lc) { ok = str_valid(decltype(Lc)::value, v); });
      break;
    case TUNE_X_INV:
      if (sff) dispatch_L_sff(g.Nx, [&](auto Lc) { ok = sx_valid(decltype(Lc)::value, 1, v); });
      else if (form <= 1) dispatch_L(g.Nx, [&](auto Lc) { ok = ix_valid(decltype(Lc)::value, v); });
      break;
    case TUNE_X_FWD:
      if (sff) dispatch_L_sff(g.Nx, [&](auto Lc) { ok = sx_valid(decltype(Lc)::value, -1, v); });
      else if (form <= 1) dispatch_L(g.Nx, [&](auto Lc) { ok = fx_valid(decltype(Lc)::value, v); });
      break;
    case TUNE_Z:
      dispatch_L_sff(g.Nz, [&](auto Lc) {
        constexpr int NZ = decltype(Lc)::value;
        ok = form == 0 ? z_valid<NZ, 7>(v) : form == 1 ? z_valid<NZ, 1>(v) : form == 2 ? z_valid<NZ, 2>(v) : false;
      });
      break;
    default:
      break;
  }
  return ok;
}

template <> bool Launch<T>::tune_blocks(const Geo& g, int form, int cls) {
  if (cls == TUNE_Y_INV || cls == TUNE_Y_FWD) return true;
  bool ok = false;
  if (cls == TUNE_X_FWD && g.basis == 0 && form <= 1)
    dispatch_L(g.Nx, [&](auto Lc) {
      constexpr int LL = decltype(Lc)::value;
      const int v = g.tv[TUNE_X_FWD];
      ok = (v == 0 && fx_rule_fused(LL)) || (v >= 2 && fx_valid(LL, v));
    });
  return ok;
}
#endif  // TS_PART_MISC

}  // namespace ts
