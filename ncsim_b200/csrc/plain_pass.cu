// Tiled passes of the plain path: a run of consecutive gates applied to tiles
// of the register in shared memory, one read and one write of HBM for the run.
//
// A pass picks a window of T <= 11 qubits (the qubits the run's gates move,
// filled up with the lowest other qubits so that tiles load in runs of
// consecutive amplitudes) and streams the register's 2^(n-T) tiles through
// shared memory: a persistent CTA double-buffers its tiles (cp.async copies
// of the next tile land while the current one is worked on) and applies the
// pass's gates to each tile in circuit order, in chains of gates that work on
// amplitudes held in registers, one __syncthreads between chains.
// Gates that only multiply amplitudes by phases (diagonals, phase polynomials)
// join any pass: their phases depend on index bits outside the window only
// through the tile's base index.
//
// Every gate is applied with the arithmetic of the kernel that the gate-by-gate
// path would launch for it (the same dispatch rules, the same cmul/cfma
// expressions on the same operands in the same order), so a run gives the same
// amplitudes either way.  Gates with no tile form (dense gates on two or more
// qubits, permutation tables other than pair swaps, phase polynomials of more
// than MAX_PASS_TERMS terms) run as their own kernels between passes.
//
// What bounds a pass: instruction issue and its latency (random layers at n = 24,
// ncu: issue slots 47% busy, FP64 pipe 27%, shared memory 29%, DRAM 18%), not HBM.
// Measured on random layers of depth 20, complex128, against 8-amplitude cubes on
// 4096-amplitude tiles (one 512-thread CTA per SM): n = 20 0.80 -> 0.44 ms, n = 24
// 11.8 -> 4.9 ms, n = 28 221 -> 93 ms.  An op that does nothing costs about 50
// instructions, so signs that follow one another (a layer's CZs) are one op with a list
// (n = 28 100 -> 96 ms) and a skipped op goes through the dispatch's empty case instead of
// a branch around it (96 -> 93 ms).  Storing the last chain's cubes straight to the
// register instead of through the tile was slower (96 ms).
#include <algorithm>
#include <cmath>
#include <cstring>
#include <memory>
#include <mutex>
#include <string>

#include "engine.cuh"
#include "host/ir.hpp"

namespace ncsim {

namespace {

// Tiles of 2^11 amplitudes: 128 threads with 16 amplitudes each, 64 KB for two complex128
// buffers, three CTAs per SM that drift apart and so overlap one's loads and barriers with
// another's arithmetic.  Tiles of 2^12 (one CTA of 256 threads per SM) take fewer passes but
// run slower (n = 28: 132 ms against 100 ms), tiles of 2^10 take more passes (n = 28: +15%).
constexpr int MAX_TILE_BITS = 11;
// On registers of more than this many qubits a window always holds the two lowest qubits,
// so that a tile is read and written in runs of 64 bytes (complex128).  A window of high
// qubits alone touches single amplitudes: one pass at n = 26 took 1.79 ms against 0.83 ms.
// Smaller registers stay in the L2 and lose more by the extra passes (n = 16: 10 against 8).
constexpr int FREE_WINDOW_QUBITS = 18;
constexpr int LOW_WINDOW_BITS = 2;
constexpr int MAX_TABLE_K = 10;
// longer phase polynomials run as the bit-sliced kernel: evaluated per element
// in a tile they cost a popcount per parity per amplitude
constexpr int MAX_PASS_TERMS = 4;
constexpr int MAX_PASS_PARITIES = 8;
constexpr int MAX_PASS_OPS = 240;  // device ops of one pass (chain heads and flushes included)
constexpr int MAX_PASS_CHAINS = MAX_PASS_OPS / 3;
// A chain's cube: CUBE_BITS tile bits, CUBE amplitudes held by one thread.  Four
// bits: the op fetch and dispatch (about 25 instructions) are shared by 16
// amplitudes, and a layer's 11 window qubits need about 3 shared-memory round
// trips.  The earlier three-bit cubes on 512 threads spent 54% of all issue slots
// with the FP64 pipe 23% busy.
constexpr int CUBE_BITS = 4;
constexpr int CUBE = 1 << CUBE_BITS;

template <class R>
using V = typename VecOf<R>::T;

enum TileKind : uint32_t {
  TK_DENSE1,      // 1-qubit dense matrix (k_dense1)
  TK_DIAG_CONST,  // one phase on the indices with every fixed bit set (k_diag_const)
  TK_DIAG_1Q,     // two phases selected by one bit (k_diag_1q)
  TK_DIAG_TABLE,  // phase table over <= 10 qubits (k_diag)
  TK_PAIRSWAP,    // exchange of i and i ^ x on a fixed-bit sub-cube (k_pairswap)
  TK_PHASEPOLY,   // phase polynomial of the global index (k_phasepoly)
};

// What the device executes.  Inside a chain the element of a cube that an op
// touches is known when the chain is made, so the common ops come in one kind
// per cube bit, with register indices fixed at compile time.
enum DevKind : uint32_t {
  DK_CHAIN = 0,                      // the next k ops, on cubes held in registers
  DK_D1 = 1,                         // + j: dense 2x2 on cube bit j
  DK_D1R = DK_D1 + CUBE_BITS,        // + j: a real matrix (RY): the zero products left out
  DK_D1RE = DK_D1R + CUBE_BITS,      // + j: a real matrix with equal entries in its first column (H): one product for both
  DK_D1X = DK_D1RE + CUBE_BITS,      // + j: real diagonal, imaginary off-diagonal (RX)
  DK_D1E = DK_D1X + CUBE_BITS,       // + j: equal entries in the first column (SQRT_Y)
  DK_D1S = DK_D1E + CUBE_BITS,       // + j: first column (1+i)/2, (1-i)/2 (SQRT_X)
  DK_D1SD = DK_D1S + CUBE_BITS,      // + j: first column (1-i)/2, (1+i)/2 (SQRT_X_DAG)
  DK_PH = DK_D1SD + CUBE_BITS,        // + j: phase on the half of the cube with bit j set
  DK_PH_ALL = DK_PH + CUBE_BITS,     // phase on the whole cube
  DK_PH_MASK,                        // phase on the cube elements of a mask
  DK_TURN,                           // + j: quarter turn (+-i) on the half with bit j set: parts exchanged, one negated
  DK_TURN_ALL = DK_TURN + CUBE_BITS,
  DK_TURN_MASK,
  DK_SIGNS,                          // signs of cube elements, kept pending in a bit mask: em items from item gml on
  DK_FLUSH,                          // the pending signs applied
  DK_RZ,                             // + j: two phases selected by cube bit j
  DK_RZ_OUT = DK_RZ + CUBE_BITS,     // two phases selected by a tile bit outside the cube
  DK_SWAP,                           // + index of the xor mask: exchange inside the cube (no phases)
  DK_SWAPC = DK_SWAP + 10,           // + index of the xor mask: exchange with phases
  DK_POLY_CONST = DK_SWAPC + 10,     // phase polynomial without terms: the same phase on every element
  // outside the chains, sweeps over the tile:
  DK_TABLE,                          // phase table
  DK_POLY,                           // phase polynomial
  DK_TILE_SWAP,                      // exchange across more than two tile bits
  DK_COND = 0x8000,                  // set when the op has fixed bits outside the window (gfix, gval)
};
// the xor masks of an exchange on one or two cube bits, in DK_SWAP's order
constexpr uint32_t SWAP_X[10] = {1, 2, 4, 8, 3, 5, 9, 6, 10, 12};

// One gate of a pass, encoded against the pass's window: "local" masks are
// over the tile's T bits, "global" masks over the bits outside the window.
struct TileOp {
  uint32_t kind;
  uint32_t k;        // qubits (table), terms (phase polynomial)
  uint32_t l0, l1;   // local bit positions (dense1: l0; diag 1q: l0, or l1 = the global qubit outside)
  uint32_t lfix;     // local mask of fixed bits
  uint32_t lones;    // the fixed bits' values at i (pairswap), or lfix (diagonal kinds)
  uint32_t lx;       // local xor mask (pairswap)
  uint32_t flags;    // pairswap: unit_i | unit_j << 1; diag 1q: 1 = the qubit lies outside
  uint64_t gfix;     // fixed bits outside the window ...
  uint64_t gval;     // ... and the values the tile base must have there
  uint64_t gz;       // phase polynomial: offset of its parities
  uint32_t cp;       // complex pool offset
  uint32_t up;       // word pool offset
};

// One device op.  Its head (what it is and what selects its elements) stays in the
// kernel parameters, where a warp reads it into uniform registers: the op loop's
// branches are then uniform ones.  The constants are read from shared memory.
struct OpHead {
  uint32_t kind;
  uint32_t em;        // cube elements (bit b: element b); chain: number of ops
  uint32_t gml, gvl;  // fixed tile bits outside the cube, and their values; chain: cube bits, chain number
};
// One sign: the cube elements em of the threads and tiles whose fixed bits are all one.
struct SignItem {
  uint32_t fix;   // tile bits outside the cube
  uint32_t em;
  uint64_t gfix;  // bits outside the window
};
struct OpCond {
  uint64_t gfix, gval;  // fixed bits outside the window, and the values the tile base must have there
};
template <class R>
struct alignas(16) OpArgs {
  union {
    V<R> c[4];
    uint32_t a[8];    // table: k, up, cp, lfix, lones; polynomial: k, up, cp, parity offset; tile swap: see tile_pairswap;
  };                  // chain: the tile bits of the thread's index, one byte each, in a[0], a[1]
};
struct DevOp {
  OpHead h{};
  OpCond g{};
  OpArgs<double> x{};
};

struct PassGeom {
  int T;                         // tile bits
  int w;                         // low index bits in the window (0..w-1)
  int nh;                        // window bits above them
  uint8_t hq[MAX_TILE_BITS];     // their global positions, ascending
};

// global offset of tile element e (bits 0..w-1 stay, bit w+i goes to hq[i])
__host__ __device__ __forceinline__ uint64_t deposit(uint32_t e, const PassGeom& g) {
  uint64_t off = e & ((1u << g.w) - 1);
  for (int i = 0; i < g.nh; ++i) off |= uint64_t((e >> (g.w + i)) & 1u) << g.hq[i];
  return off;
}
// base index of tile t: t spread over the bits outside the window
__host__ __device__ __forceinline__ uint64_t tile_base_of(uint64_t t, const PassGeom& g) {
  uint64_t v = t << g.w;
  for (int i = 0; i < g.nh; ++i) {
    const int b = g.hq[i];
    v = ((v >> b) << (b + 1)) | (v & ((uint64_t(1) << b) - 1));
  }
  return v;
}

// A tile in shared memory: element e at e ^ (the XOR of e's higher groups of SB
// bits), SB = 3 for 16-byte elements and 4 for 8-byte ones, so tile bit b moves
// the bank group by bit b mod SB.  Lanes whose lowest SB bits sit on tile bits of
// distinct residues mod SB hit distinct banks; chain heads order their thread bits
// that way.  The map is linear over XOR: a thread's and an element's part combine.
template <class R>
__host__ __device__ __forceinline__ uint32_t swz(uint32_t e) {
  if constexpr (sizeof(V<R>) == 16) return e ^ (((e >> 3) ^ (e >> 6) ^ (e >> 9)) & 7u);
  else return e ^ (((e >> 4) ^ (e >> 8)) & 15u);
}
template <class R>
__device__ __forceinline__ V<R>* shared_tile() {
  extern __shared__ __align__(16) unsigned char pass_smem[];
  return reinterpret_cast<V<R>*>(pass_smem);
}
template <class R>
struct SwTile {
  V<R>* p;
  __device__ __forceinline__ V<R>& operator[](uint32_t e) const { return p[swz<R>(e)]; }
};

template <class R>
struct PassParams {
  V<R>* amp;
  uint64_t ntiles;
  PassGeom g;
  uint32_t nops;
  const V<R>* cpool;
  const uint32_t* upool;
  const uint64_t* ppool;  // phase polynomial parities (global masks)
  uint32_t nchains, nsigns;
  SignItem sign[MAX_PASS_OPS];   // copied into shared memory once per CTA, like the arguments
  OpHead head[MAX_PASS_OPS];
  OpCond cond[MAX_PASS_OPS];
  OpArgs<R> args[MAX_PASS_OPS];  // copied into shared memory once per CTA
};

// x with its sign bit xored by s (0 or 0x80000000)
__device__ __forceinline__ double flip(double x, uint32_t s) {
  return __hiloint2double(int(uint32_t(__double2hiint(x)) ^ s), __double2loint(x));
}
__device__ __forceinline__ float flip(float x, uint32_t s) { return __uint_as_float(__float_as_uint(x) ^ s); }

// exchange across three or more tile bits: a: number of fixed bits, pairswap flags, xor mask, values, constants,
// and the fixed bits' positions, four bits each, in a[6], a[7]
template <class R>
__device__ __forceinline__ void tile_pairswap(SwTile<R> t, uint32_t tsz, const OpArgs<R>& op, const V<R>* cpool) {
  const uint32_t nf = op.a[0], pairs = tsz >> nf, x = op.a[2], ones = op.a[3];
  const uint64_t fixed = uint64_t(op.a[7]) << 32 | op.a[6];
  const bool ui = op.a[1] & 1, uj = (op.a[1] >> 1) & 1;
  V<R> ci{}, cj{};
  if (!(ui && uj)) ci = cpool[op.a[4]], cj = cpool[op.a[4] + 1];
  constexpr int N = 8;  // pairs in flight: a thread has eight of a tile's at most
  for (uint32_t p = threadIdx.x; p < pairs; p += N * blockDim.x) {
    uint32_t i[N];
#pragma unroll
    for (int u = 0; u < N; ++u) i[u] = p + u * blockDim.x < pairs ? p + u * blockDim.x : p;  // its own pair again
    uint64_t pos = fixed;
    for (uint32_t f = 0; f < nf; ++f, pos >>= 4) {
      const uint32_t b = uint32_t(pos) & 15u, low = (1u << b) - 1;
#pragma unroll
      for (int u = 0; u < N; ++u) i[u] = ((i[u] & ~low) << 1) | (i[u] & low);
    }
    V<R> vi[N], vj[N];
#pragma unroll
    for (int u = 0; u < N; ++u) {
      i[u] |= ones;
      vi[u] = t[i[u]];
      vj[u] = t[i[u] ^ x];
    }
#pragma unroll
    for (int u = 0; u < N; ++u)
      if (p + u * blockDim.x < pairs) {
        t[i[u]] = ui ? vj[u] : cmul(ci, vj[u]);
        t[i[u] ^ x] = uj ? vi[u] : cmul(cj, vi[u]);
      }
  }
}

__device__ __forceinline__ double2 pass_root(uint64_t f, uint32_t bits) {
  // exp(2 pi i f / 2^bits) with exact quarter and eighth turns (as the gate-by-gate kernel)
  const uint64_t m = uint64_t(1) << bits;
  if (((4 * f) & (m - 1)) == 0) {
    switch ((4 * f / m) & 3) {
      case 0: return make_double2(1.0, 0.0);
      case 1: return make_double2(0.0, 1.0);
      case 2: return make_double2(-1.0, 0.0);
      default: return make_double2(0.0, -1.0);
    }
  }
  if (((8 * f) & (m - 1)) == 0) {
    const double h = 0.70710678118654752440;
    switch ((8 * f / m) & 7) {
      case 1: return make_double2(h, h);
      case 3: return make_double2(-h, h);
      case 5: return make_double2(-h, -h);
      default: return make_double2(h, -h);
    }
  }
  double s, c;
  sincospi(2.0 * double(f) / double(m), &s, &c);
  return make_double2(c, s);
}

// ---- chains: consecutive ops whose coupled bits lie in one cube of CUBE_BITS tile bits ----
// A thread holds the elements of a cube (v[b]: cube pattern b) and applies
// the chain's ops in order to them, one shared-memory round trip for the
// chain.  The ops couple elements only inside a cube, and each element sees
// its ops in circuit order with each op's own arithmetic.  What gives the same
// bits on finite amplitudes more cheaply is used: products with exact zeros are
// left out (real matrices), +-i exchanges the parts, and -1 is a sign flip, which
// commutes with every rounding and so waits in a mask until an op mixes elements.
// (Tiles with other amplitudes are done over with every product: redo_tile.)
// The updates are written so that each result can take the place of an operand
// that has just been read for the last time (both products with a0 first): the
// cases of the op loop then meet on the same registers without copies between.
template <class R, int J>
__device__ __forceinline__ void chain_dense1(V<R> (&v)[CUBE], const V<R>* m) {
  const V<R> m00 = m[0], m01 = m[1], m10 = m[2], m11 = m[3];
#pragma unroll
  for (int b = 0; b < CUBE; ++b)
    if (!((b >> J) & 1)) {
      V<R>&a0 = v[b], &a1 = v[b | (1 << J)];
      V<R> p0 = cmul(m00, a0), p1 = cmul(m10, a0);  // cfma(m01, a1, p0) and cfma(m11, a1, p1):
      p0.x = fma_rn(-m01.y, a1.y, p0.x);
      p0.y = fma_rn(m01.y, a1.x, p0.y);
      a0.x = fma_rn(m01.x, a1.x, p0.x);
      a0.y = fma_rn(m01.x, a1.y, p0.y);
      p1.x = fma_rn(-m11.y, a1.y, p1.x);
      p1.y = fma_rn(m11.y, a1.x, p1.y);
      a1.x = fma_rn(m11.x, a1.x, p1.x);
      a1.y = fma_rn(m11.x, a1.y, p1.y);
    }
}
// A first column (1+i)/2, (1-i)/2 (S = 0), its conjugate (S = 1) or two equal entries
// (S = 2): a product with one half is exact, so the second product is the first turned
// by a quarter (or the same), and four of the sixteen steps go.
template <class R, int J, int S>
__device__ __forceinline__ void chain_dense1_col(V<R> (&v)[CUBE], const V<R>* m) {
  const V<R> m00 = m[0], m01 = m[1], m11 = m[3];
#pragma unroll
  for (int b = 0; b < CUBE; ++b)
    if (!((b >> J) & 1)) {
      V<R>&a0 = v[b], &a1 = v[b | (1 << J)];
      const V<R> p0 = cmul(m00, a0);
      V<R> p1;
      p1.x = S == 0 ? p0.y : S == 1 ? -p0.y : p0.x;
      p1.y = S == 0 ? -p0.x : S == 1 ? p0.x : p0.y;
      a0.x = fma_rn(-m01.y, a1.y, p0.x);
      a0.y = fma_rn(m01.y, a1.x, p0.y);
      a0.x = fma_rn(m01.x, a1.x, a0.x);
      a0.y = fma_rn(m01.x, a1.y, a0.y);
      p1.x = fma_rn(-m11.y, a1.y, p1.x);
      p1.y = fma_rn(m11.y, a1.x, p1.y);
      a1.x = fma_rn(m11.x, a1.x, p1.x);
      a1.y = fma_rn(m11.x, a1.y, p1.y);
    }
}
template <class R, int J>
__device__ __forceinline__ void chain_dense1_real(V<R> (&v)[CUBE], const V<R>* m) {
  const R m00 = m[0].x, m01 = m[1].x, m10 = m[2].x, m11 = m[3].x;
#pragma unroll
  for (int b = 0; b < CUBE; ++b)
    if (!((b >> J) & 1)) {
      V<R>&a0 = v[b], &a1 = v[b | (1 << J)];
      const R px = mul_rn(m10, a0.x), py = mul_rn(m10, a0.y);
      a0.x = mul_rn(m00, a0.x);
      a0.y = mul_rn(m00, a0.y);
      a0.x = fma_rn(m01, a1.x, a0.x);
      a0.y = fma_rn(m01, a1.y, a0.y);
      a1.x = fma_rn(m11, a1.x, px);
      a1.y = fma_rn(m11, a1.y, py);
    }
}
template <class R, int J>
__device__ __forceinline__ void chain_dense1_realcol(V<R> (&v)[CUBE], const V<R>* m) {
  const R m00 = m[0].x, m01 = m[1].x, m11 = m[3].x;
#pragma unroll
  for (int b = 0; b < CUBE; ++b)
    if (!((b >> J) & 1)) {
      V<R>&a0 = v[b], &a1 = v[b | (1 << J)];
      const R px = mul_rn(m00, a0.x), py = mul_rn(m00, a0.y);
      a0.x = fma_rn(m01, a1.x, px);
      a0.y = fma_rn(m01, a1.y, py);
      a1.x = fma_rn(m11, a1.x, px);
      a1.y = fma_rn(m11, a1.y, py);
    }
}
template <class R, int J>
__device__ __forceinline__ void chain_dense1_cross(V<R> (&v)[CUBE], const V<R>* m) {
  const R m00 = m[0].x, i01 = m[1].y, i10 = m[2].y, m11 = m[3].x;
#pragma unroll
  for (int b = 0; b < CUBE; ++b)
    if (!((b >> J) & 1)) {
      V<R>&a0 = v[b], &a1 = v[b | (1 << J)];
      const R px = -mul_rn(i10, a0.y), py = mul_rn(i10, a0.x);
      a0.x = mul_rn(m00, a0.x);
      a0.y = mul_rn(m00, a0.y);
      a0.x = fma_rn(-i01, a1.y, a0.x);
      a0.y = fma_rn(i01, a1.x, a0.y);
      a1.x = fma_rn(m11, a1.x, px);
      a1.y = fma_rn(m11, a1.y, py);
    }
}
template <class R>
__device__ __forceinline__ void phase_in_place(V<R>& u, V<R> c) {  // u = cmul(c, u)
  const R t = mul_rn(c.y, u.y), s = mul_rn(c.y, u.x);
  u.x = fma_rn(c.x, u.x, -t);
  u.y = fma_rn(c.x, u.y, s);
}
template <class R, int J>
__device__ __forceinline__ void chain_phase(V<R> (&v)[CUBE], V<R> c) {
#pragma unroll
  for (int b = 0; b < CUBE; ++b)
    if (J < 0 || ((b >> (J < 0 ? 0 : J)) & 1)) phase_in_place<R>(v[b], c);
}
// u times (0, +1) (sx = sign bit, sy = 0) or (0, -1) (sx = 0, sy = sign bit)
template <class V2>
__device__ __forceinline__ void turn_in_place(V2& u, uint32_t sx, uint32_t sy) {
  const auto x = u.x;
  u.x = flip(u.y, sx);
  u.y = flip(x, sy);
}
template <class R, int J>
__device__ __forceinline__ void chain_turn(V<R> (&v)[CUBE], uint32_t sx, uint32_t sy) {
#pragma unroll
  for (int b = 0; b < CUBE; ++b)
    if (J < 0 || ((b >> (J < 0 ? 0 : J)) & 1)) turn_in_place(v[b], sx, sy);
}
template <class R, int J>
__device__ __forceinline__ void chain_rz(V<R> (&v)[CUBE], const V<R>* c) {
  const V<R> c0 = c[0], c1 = c[1];
#pragma unroll
  for (int b = 0; b < CUBE; ++b) phase_in_place<R>(v[b], ((b >> J) & 1) ? c1 : c0);
}
template <class R, int X>
__device__ __forceinline__ void chain_swap(V<R> (&v)[CUBE], uint32_t em) {  // em: the smaller element of each pair
#pragma unroll
  for (int b = 0; b < CUBE; ++b)
    if (b < (b ^ X))
      if ((em >> b) & 1) {
        const V<R> u = v[b];
        v[b] = v[b ^ X];
        v[b ^ X] = u;
      }
}
template <class R, int X>
__device__ __forceinline__ void chain_swapc(V<R> (&v)[CUBE], uint32_t em, uint32_t flags, const V<R>* c) {
  const V<R> ci = c[0], cj = c[1];
  const bool ui = flags & 1, uj = (flags >> 1) & 1;
#pragma unroll
  for (int b = 0; b < CUBE; ++b)
    if ((em >> b) & 1) {
      const V<R> vi = v[b], vj = v[b ^ X];
      v[b] = ui ? vj : cmul(ci, vj);
      v[b ^ X] = uj ? vi : cmul(cj, vi);
    }
}
// the pending signs applied
template <class R>
__device__ __forceinline__ void chain_flush(V<R> (&v)[CUBE], uint32_t& pend) {
  if (!pend) return;
#pragma unroll
  for (int b = 0; b < CUBE; ++b) {
    const uint32_t s = (pend << (31 - b)) & 0x80000000u;
    v[b].x = flip(v[b].x, s);
    v[b].y = flip(v[b].y, s);
  }
  pend = 0;
}

// v times the phase of the polynomial's value f (u: the polynomial's words)
template <class R>
__device__ __forceinline__ V<R> phase_of_value(V<R> v, uint32_t f, const uint32_t* u, const V<R>* cp) {
  if (is_zero(v)) return v;
  const uint32_t bits = u[0];
  const bool use_table = u[1], s_one = u[2];
  if (bits < 32) f &= (1u << bits) - 1;
  V<R> c;
  if (use_table) {
    c = cp[1 + f];
    if (is_one_v(c)) return v;
  } else {
    if (f == 0 && s_one) return v;
    const double2 rr = pass_root(f, bits);
    c.x = R(rr.x);
    c.y = R(rr.y);
    if (!s_one) c = cmul(cp[0], c);
  }
  return cmul(c, v);
}

// v times the phase of a polynomial at index i
template <class R>
__device__ __forceinline__ V<R> phasepoly_elem(V<R> v, uint64_t i, const OpArgs<R>& op, const PassParams<R>& P) {
  if (is_zero(v)) return v;
  const uint32_t* u = P.upool + op.a[1];
  const V<R>* cp = P.cpool + op.a[2];
  const uint64_t* pp = P.ppool + op.a[3];
  const uint32_t bits = u[0];
  const bool use_table = u[1], s_one = u[2];
  const uint64_t constant = uint64_t(u[3]) | (uint64_t(u[4]) << 32);
  const int nt = int(op.a[0]);
  const uint32_t* start = u + 5;
  const uint32_t* coeff = start + nt + 1;
  uint64_t f = constant;
  for (int tt = 0; tt < nt; ++tt) {
    int all = 1;
    for (uint32_t l = start[tt]; l < start[tt + 1]; ++l) all &= __popcll(pp[l] & i) & 1;
    if (all) f += coeff[tt];
  }
  f &= (uint64_t(1) << bits) - 1;
  V<R> c;
  if (use_table) {
    c = cp[1 + f];
    if (is_one_v(c)) return v;
  } else {
    if (f == 0 && s_one) return v;
    const double2 rr = pass_root(f, bits);
    c.x = R(rr.x);
    c.y = R(rr.y);
    if (!s_one) c = cmul(cp[0], c);
  }
  return cmul(c, v);
}

// The ops outside the chains, one at a time over the tile (element round r of a thread: threadIdx.x + r * blockDim.x).
// Patterns and parities are linear in the index: the thread's part is made once and each round adds its own.
// Evaluated in the chains, element by element with a loop over their qubits or parities, they held up 16 elements at
// once: 30 tables on 8 qubits at n = 10 209 us, here 92 (in chains of 8 elements to each of 512 threads 115), at n = 28
// 53 ms, 28 (47); 30 polynomials of two terms with H between at n = 28 192 ms, 56 (138).  Exchanges across five bits,
// 40 of them at n = 10: 81 us one pair at a time, 61 with all eight in flight.  Not inlined: the op loop keeps its registers.
template <class R>
__device__ __noinline__ void tile_sweep(uint32_t kind, uint32_t buf, uint64_t base, uint64_t dthread, const uint64_t* dround,
                                        const OpArgs<R>& op, const PassParams<R>& P) {
  const SwTile<R> t{shared_tile<R>() + buf};
  const uint32_t tsz = 1u << P.g.T;
  const uint32_t nr = (tsz + blockDim.x - 1) / blockDim.x, lb = 31u - __clz(blockDim.x);  // a round moves tile bits lb and up
  if (kind == DK_TILE_SWAP) {
    tile_pairswap<R>(t, tsz, op, P.cpool);
  } else if (kind == DK_TABLE) {
    const uint32_t k = op.a[0], lfix = op.a[3], lones = op.a[4];
    const uint32_t* qp = P.upool + op.a[1];
    const uint8_t* unit = reinterpret_cast<const uint8_t*>(qp + k);
    const V<R>* c = P.cpool + op.a[2];
    uint32_t x0 = 0, w[CUBE_BITS] = {};
    for (uint32_t j = 0; j < k; ++j) {
      const uint32_t q = qp[j];
      x0 |= (q >= 256 ? uint32_t(base >> (q - 256)) & 1u : (threadIdx.x >> q) & 1u) << j;
#pragma unroll
      for (int i = 0; i < CUBE_BITS; ++i) w[i] |= uint32_t(q == lb + i) << j;
    }
    for (uint32_t r0 = 0; r0 < nr; r0 += 4) {  // four elements in flight
      V<R> u[4], f[4];
      uint32_t leave[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const uint32_t r = r0 + i, e = threadIdx.x + r * blockDim.x;
        uint32_t x = x0;
#pragma unroll
        for (int j = 0; j < CUBE_BITS; ++j) x |= ((r >> j) & 1) ? w[j] : 0u;
        u[i] = t[e];
        f[i] = c[x];
        leave[i] = unit[x] | uint32_t((e & lfix) != lones);
      }
#pragma unroll
      for (int i = 0; i < 4; ++i)
        if (!leave[i]) t[threadIdx.x + (r0 + i) * blockDim.x] = cmul(f[i], u[i]);
    }
  } else {  // DK_POLY
    const uint32_t* u = P.upool + op.a[1];
    const uint64_t* pp = P.ppool + op.a[3];
    const uint32_t nt = op.a[0];
    const uint32_t* start = u + 5;
    const uint32_t* coeff = start + nt + 1;
    const uint64_t i = base | dthread;
    // a parity is one mask over the rounds, a term's rounds are the AND of its parities' masks
    uint32_t in[MAX_PASS_TERMS] = {}, co[MAX_PASS_TERMS] = {};
#pragma unroll
    for (uint32_t k = 0; k < MAX_PASS_TERMS; ++k)
      if (k < nt) {
        uint32_t m = 0xffffu;
        for (uint32_t l = start[k]; l < start[k + 1]; ++l) {
          const uint64_t p = pp[l];
          const auto odd = [&](uint64_t x) { return __popcll(p & x) & 1; };
          m &= (odd(i) ? 0xffffu : 0u) ^ (odd(dround[1]) ? 0xaaaau : 0u) ^ (odd(dround[2]) ? 0xccccu : 0u) ^
               (odd(dround[4]) ? 0xf0f0u : 0u) ^ (nr > 8 && odd(dround[8]) ? 0xff00u : 0u);
        }
        in[k] = m;
        co[k] = coeff[k];
      }
    const uint32_t constant = u[3];  // a value has at most 32 bits
    for (uint32_t r = 0; r < nr; ++r) {
      uint32_t f = constant;
#pragma unroll
      for (uint32_t k = 0; k < MAX_PASS_TERMS; ++k) f += ((in[k] >> r) & 1u) ? co[k] : 0u;
      V<R>& at = t[threadIdx.x + r * blockDim.x];
      at = phase_of_value<R>(at, f, u, P.cpool + op.a[2]);
    }
  }
}

// The chain whose head is op o.  gbase: the tile bits of the thread's cube (its index
// spread over the tile bits outside the cube).  FULL: every product formed (redo_tile).
// With `last` it returns NaN when one of the thread's results is infinite or NaN.
template <class R, bool FULL>
__device__ __forceinline__ R tile_chain(uint32_t tile, uint32_t o, uint32_t gbase, const OpArgs<R>* args,
                                           const SignItem* signs, const PassParams<R>& P, uint64_t base, bool last) {
  V<R>* const t = shared_tile<R>() + tile;  // an index into the shared array, so that accesses stay in the shared space
  const uint32_t nsub = P.head[o].em;
  const uint32_t cbits = P.head[o].gml;  // cube bit j: byte j
  const uint32_t gb = gbase;
  uint32_t lb[CUBE_BITS], sb[CUBE_BITS];
#pragma unroll
  for (int j = 0; j < CUBE_BITS; ++j) {
    lb[j] = 1u << ((cbits >> (8 * j)) & 0xffu);
    sb[j] = swz<R>(lb[j]);
  }
  const uint32_t sg = swz<R>(gb);
  V<R> v[CUBE];
#pragma unroll
  for (int b = 0; b < CUBE; ++b) {
    uint32_t a = 0;
#pragma unroll
    for (int j = 0; j < CUBE_BITS; ++j)
      if ((b >> j) & 1) a ^= sb[j];
    v[b] = t[sg ^ a];
  }
  uint32_t pend = 0;  // elements whose sign is still to be flipped
  for (uint32_t s = o + 1; s <= o + nsub; ++s) {
    const OpHead h = P.head[s];
    const OpArgs<R>& op = args[s];
    const bool skip = (h.kind & DK_COND) && (base & P.cond[s].gfix) != P.cond[s].gval;  // uniform over the CTA
    const bool on = (gb & h.gml) == h.gvl;
    const uint32_t em = h.em;
    uint32_t kind = skip ? 0u : h.kind & ~uint32_t(DK_COND);
    if constexpr (FULL) {
      const auto phase_on = [&](uint32_t elements, V<R> c) {
#pragma unroll
        for (int b = 0; b < CUBE; ++b)
          if ((elements >> b) & 1) phase_in_place<R>(v[b], c);
      };
      if (kind >= DK_D1 && kind < DK_PH) {
        kind = DK_D1 + (kind - DK_D1) % CUBE_BITS;
      } else if (kind >= DK_TURN && kind <= DK_TURN_MASK) {
        uint32_t half = 0;
        for (uint32_t b = 0; b < CUBE; ++b)
          if (kind == DK_TURN_ALL || ((b >> (kind - DK_TURN)) & 1)) half |= 1u << b;
        V<R> c;
        c.x = R(0);
        c.y = op.a[0] ? R(1) : R(-1);
        if (on) phase_on(kind == DK_TURN_MASK ? em : half, c);
        continue;
      } else if (kind == DK_SIGNS) {
        V<R> c;
        c.x = R(-1);
        c.y = R(0);
        for (uint32_t i = 0; i < em; ++i) {
          const SignItem x = signs[h.gml + i];
          if ((gb & x.fix) == x.fix && (base & x.gfix) == x.gfix) phase_on(x.em, c);
        }
        continue;
      }
    }
#define NCSIM_D1(j) \
  case DK_D1 + j: chain_dense1<R, j>(v, op.c); break; \
  case DK_D1R + j: chain_dense1_real<R, j>(v, op.c); break; \
  case DK_D1RE + j: chain_dense1_realcol<R, j>(v, op.c); break; \
  case DK_D1X + j: chain_dense1_cross<R, j>(v, op.c); break; \
  case DK_D1E + j: chain_dense1_col<R, j, 2>(v, op.c); break; \
  case DK_D1S + j: chain_dense1_col<R, j, 0>(v, op.c); break; \
  case DK_D1SD + j: chain_dense1_col<R, j, 1>(v, op.c); break; \
  case DK_PH + j: if (on) chain_phase<R, j>(v, op.c[0]); break; \
  case DK_TURN + j: if (on) chain_turn<R, j>(v, op.a[0], op.a[1]); break; \
  case DK_RZ + j: chain_rz<R, j>(v, op.c); break;
#define NCSIM_SW(i, X) \
  case DK_SWAP + i: if (on) chain_swap<R, X>(v, em); break; \
  case DK_SWAPC + i: if (on) chain_swapc<R, X>(v, em & 0xffffu, em >> 16, op.c); break;
    switch (kind) {
      NCSIM_D1(0)
      NCSIM_D1(1)
      NCSIM_D1(2)
      NCSIM_D1(3)
      NCSIM_SW(0, 1)
      NCSIM_SW(1, 2)
      NCSIM_SW(2, 4)
      NCSIM_SW(3, 8)
      NCSIM_SW(4, 3)
      NCSIM_SW(5, 5)
      NCSIM_SW(6, 9)
      NCSIM_SW(7, 6)
      NCSIM_SW(8, 10)
      NCSIM_SW(9, 12)
      case DK_PH_ALL:
        if (on) chain_phase<R, -1>(v, op.c[0]);
        break;
      case DK_PH_MASK:
        if (on) {
          const V<R> c = op.c[0];
#pragma unroll
          for (int b = 0; b < CUBE; ++b)
            if ((em >> b) & 1) phase_in_place<R>(v[b], c);
        }
        break;
      case DK_TURN_ALL:
        if (on) chain_turn<R, -1>(v, op.a[0], op.a[1]);
        break;
      case DK_TURN_MASK:
        if (on) {
          const uint32_t sx = op.a[0], sy = op.a[1];
#pragma unroll
          for (int b = 0; b < CUBE; ++b)
            if ((em >> b) & 1) turn_in_place(v[b], sx, sy);
        }
        break;
      case DK_SIGNS: {
        const SignItem* const it = signs + h.gml;
#pragma unroll 2
        for (uint32_t i = 0; i < em; ++i) {
          const SignItem x = it[i];
          if ((gb & x.fix) == x.fix && (base & x.gfix) == x.gfix) pend ^= x.em;
        }
        break;
      }
      case DK_FLUSH: chain_flush<R>(v, pend); break;
      case DK_RZ_OUT: chain_phase<R, -1>(v, op.c[on ? 1 : 0]); break;
      case DK_POLY_CONST: {
        // Polynomials with terms are sweeps.  The general form stands here because the compiler lays out the whole
        // switch by it: without this case, or with a short one, it copies a complex128 cube's registers at every op
        // (random layers at n = 28 91 -> 148 and 103 ms).
#pragma unroll
        for (int b = 0; b < CUBE; ++b) {
          uint32_t e = gb;
#pragma unroll
          for (int j = 0; j < CUBE_BITS; ++j)
            if ((b >> j) & 1) e |= lb[j];
          v[b] = phasepoly_elem<R>(v[b], base | deposit(e, P.g), op, P);
        }
        break;
      }
      default: break;
    }
#undef NCSIM_D1
#undef NCSIM_SW
  }
  __syncwarp();  // registers of fewer than 2^9 amplitudes: two threads hold each cube and store the same values
#pragma unroll
  for (int b = 0; b < CUBE; ++b) {
    uint32_t a = 0;
#pragma unroll
    for (int j = 0; j < CUBE_BITS; ++j)
      if ((b >> j) & 1) a ^= sb[j];
    t[sg ^ a] = v[b];
  }
  R odd = R(0);
  if (last) {
    R part[4] = {};  // short dependent chains
#pragma unroll
    for (int b = 0; b < CUBE; ++b) part[b & 3] = fma_rn(v[b].x, R(0), fma_rn(v[b].y, R(0), part[b & 3]));
    odd = (part[0] + part[1]) + (part[2] + part[3]);
  }
  return odd;
}

// A tile whose amplitudes are not all finite, from the register again with every product formed: on an
// infinite or NaN amplitude a product with zero is NaN, and the ops of the chains leave such products out.
// (They keep what is not finite not finite, so the tile's results tell that one was met or made.)
// The last chain's look at its results and a barrier that carries the answer cost 0.8% (n = 28) to 1.4% (n = 20) of
// random layers; the same look in the op loop made its branches divergent ones (10%).
template <class R>
__device__ __noinline__ void redo_tile(uint32_t buf, uint64_t base, const OpArgs<R>* args, const SignItem* signs,
                                       const uint16_t* cubes, uint64_t dthread, const uint64_t* dround, const PassParams<R>& P) {
  const SwTile<R> t{shared_tile<R>() + buf};
  for (uint32_t e = threadIdx.x, r = 0; e < 1u << P.g.T; e += blockDim.x, ++r) t[e] = P.amp[base | dthread | dround[r]];
  __syncthreads();
  for (uint32_t o = 0; o < P.nops; ++o) {
    const OpHead& h = P.head[o];
    if (h.kind == DK_CHAIN) {
      tile_chain<R, true>(buf, o, cubes[h.gvl * blockDim.x + threadIdx.x], args, signs, P, base, false);
      o += h.em;
    } else {
      if ((base & P.cond[o].gfix) != P.cond[o].gval) continue;
      tile_sweep<R>(h.kind & ~uint32_t(DK_COND), buf, base, dthread, dround, args[o], P);
    }
    __syncthreads();
  }
}

// One thread per cube of a tile: 2^(T - CUBE_BITS) threads, at least a warp, at most 128; the
// bound of three times that gives a thread 168 registers, what three CTAs per SM leave it.
// (A bound of 128 threads and four CTAs, 128 registers, spills; the same 168 stated as
// "three CTAs of 128" made ptxas copy the cube's registers at every op, 1.8 times the time.)
constexpr int PASS_THREADS = 1 << (MAX_TILE_BITS - CUBE_BITS);
template <class R>
__global__ void __launch_bounds__(3 * PASS_THREADS) k_plain_pass(const __grid_constant__ PassParams<R> P) {
  const PassGeom& g = P.g;
  const uint32_t tsz = 1u << g.T;
  OpArgs<R>* const args = reinterpret_cast<OpArgs<R>*>(shared_tile<R>() + 2 * tsz);
  SignItem* const signs = reinterpret_cast<SignItem*>(args + P.nops);
  uint16_t* const cubes = reinterpret_cast<uint16_t*>(signs + P.nsigns);  // chain c, thread t: its cube at c * blockDim.x + t
  __shared__ uint64_t dround[CUBE];
  // element round r of a thread: elements threadIdx.x + r * blockDim.x
  const uint32_t nr = (tsz + blockDim.x - 1) / blockDim.x;
  if (threadIdx.x < nr) dround[threadIdx.x] = deposit(threadIdx.x * blockDim.x, g);
  {
    const uint32_t words = P.nops * uint32_t(sizeof(OpArgs<R>) / 16);
    const uint4* src = reinterpret_cast<const uint4*>(P.args);
    uint4* dst = reinterpret_cast<uint4*>(args);
    for (uint32_t i = threadIdx.x; i < words; i += blockDim.x) dst[i] = src[i];
    for (uint32_t i = threadIdx.x; i < P.nsigns; i += blockDim.x) signs[i] = P.sign[i];
  }
  for (uint32_t o = 0; o < P.nops; ++o)
    if (P.head[o].kind == DK_CHAIN) {
      uint32_t gb = 0;
      for (int i = 0; i < g.T - CUBE_BITS; ++i)
        gb |= ((threadIdx.x >> i) & 1u) << ((P.args[o].a[i >> 2] >> (8 * (i & 3))) & 0xffu);
      cubes[P.head[o].gvl * blockDim.x + threadIdx.x] = uint16_t(gb);
    }
  const uint64_t dthread = deposit(threadIdx.x, g);
  __syncthreads();
  // f(element, its offset in the register) for the thread's elements of a tile
  const auto elements = [&](auto f) {
    if (nr == CUBE) {
#pragma unroll
      for (uint32_t r = 0; r < CUBE; ++r) f(threadIdx.x + r * blockDim.x, dround[r]);
    } else {
      for (uint32_t r = 0; r < nr; ++r) f(threadIdx.x + r * blockDim.x, dround[r]);
    }
  };
  const auto load = [&](uint64_t tile, uint32_t buf) {
    const V<R>* src = P.amp + (tile_base_of(tile, g) | dthread);
    V<R>* const dst = shared_tile<R>() + buf;
    elements([&](uint32_t e, uint64_t off) {
      const uint32_t d = static_cast<uint32_t>(__cvta_generic_to_shared(dst + swz<R>(e)));
      if constexpr (sizeof(V<R>) == 16)
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(d), "l"(src + off) : "memory");
      else
        asm volatile("cp.async.ca.shared.global [%0], [%1], 8;\n" ::"r"(d), "l"(src + off) : "memory");
    });
    asm volatile("cp.async.commit_group;\n" ::: "memory");
  };
  // the register passes from the previous launch to this one: everything above overlaps its end
  asm volatile("griddepcontrol.launch_dependents;\n\tgriddepcontrol.wait;" ::: "memory");
  uint64_t tile = blockIdx.x;
  if (tile < P.ntiles) load(tile, 0);
  for (uint32_t buf = 0; tile < P.ntiles; buf ^= tsz, tile += gridDim.x) {
    const uint64_t next = tile + gridDim.x;
    if (next < P.ntiles) {
      load(next, buf ^ tsz);
      asm volatile("cp.async.wait_group 1;\n" ::: "memory");
    } else {
      asm volatile("cp.async.wait_group 0;\n" ::: "memory");
    }
    __syncthreads();
    const uint64_t base = tile_base_of(tile, g);
    R odd = R(0);  // the last chain's
    for (uint32_t o = 0; o < P.nops; ++o) {
      if (o) __syncthreads();
      const OpHead& h = P.head[o];
      if (h.kind == DK_CHAIN) {
        odd = tile_chain<R, false>(buf, o, cubes[h.gvl * blockDim.x + threadIdx.x], args, signs, P, base, h.gvl + 1 == P.nchains);
        o += h.em;
      } else {
        if ((base & P.cond[o].gfix) != P.cond[o].gval) continue;
        tile_sweep<R>(h.kind & ~uint32_t(DK_COND), buf, base, dthread, dround, args[o], P);
      }
    }
    // outside the op loop, whose branches so stay uniform ones
    if (__syncthreads_or(odd != odd)) redo_tile<R>(buf, base, args, signs, cubes, dthread, dround, P);
    V<R>* const dst = P.amp + (base | dthread);
    const V<R>* const from = shared_tile<R>() + buf;
    elements([&](uint32_t e, uint64_t off) { dst[off] = from[swz<R>(e)]; });
    __syncthreads();  // the buffer is refilled two tiles later
  }
}

// ---------------------------------------------------------------------------
// host: how the gate-by-gate path would apply a lowered gate (its dispatch
// rules, kernels_plain.cu launch_*), as a tile op over global qubits
// ---------------------------------------------------------------------------
bool one_c(const CplxD& c) { return c.re == 1.0 && c.im == 0.0; }
bool zero_c(const CplxD& c) { return c.re == 0.0 && c.im == 0.0; }

struct GateForm {
  uint32_t kind = 0;
  bool tileable = false;
  bool nothing = false;
  std::vector<uint32_t> qubits;   // gate qubits (local order)
  uint64_t moving = 0;            // qubits whose amplitudes the gate mixes or moves
  std::vector<CplxD> c;           // matrix / constants / table
  uint64_t fixmask = 0, ones = 0, xmask = 0;
  uint32_t flags = 0;
  std::vector<uint8_t> unit;
  const PolyTerms* poly = nullptr;
};

GateForm form_diag_table(const std::vector<uint32_t>& qubits, const std::vector<CplxD>& diag) {
  GateForm f;
  const int k = int(qubits.size());
  f.qubits = qubits;
  if (k > MAX_TABLE_K) return f;
  const int gd = 1 << k;
  uint32_t fixed = (1u << k) - 1;
  bool any = false;
  int nphased = 0;
  for (int x = 0; x < gd; ++x)
    if (!one_c(diag[x])) fixed &= uint32_t(x), any = true, ++nphased;
  if (!any) {
    f.nothing = true;
    return f;
  }
  f.tileable = true;
  if (nphased == 1 && fixed == uint32_t(gd - 1)) {
    f.kind = TK_DIAG_CONST;
    for (uint32_t q : qubits) f.fixmask |= uint64_t(1) << q;
    f.ones = f.fixmask;
    f.c = {diag[gd - 1]};
    return f;
  }
  if (k == 1) {
    f.kind = TK_DIAG_1Q;
    f.c = {diag[0], diag[1]};
    return f;
  }
  f.kind = TK_DIAG_TABLE;
  for (int j = 0; j < k; ++j)
    if ((fixed >> j) & 1) f.fixmask |= uint64_t(1) << qubits[j];
  f.ones = f.fixmask;
  f.c.assign(diag.begin(), diag.end());
  f.unit.resize(gd);
  for (int x = 0; x < gd; ++x) f.unit[x] = one_c(diag[x]) ? 1 : 0;
  return f;
}

// the share of the register the gate's own kernel reads and writes (its
// algorithmic bytes over a full pass: the sectors that hold an amplitude it changes)
double touched_share(const GateForm& f, int precision) {
  const uint64_t below = precision == NCSIM_C128 ? 1 : 3;  // index bits inside a 32-byte sector
  auto share = [&](uint64_t fixed) { return std::ldexp(1.0, -__builtin_popcountll(fixed & ~below)); };
  switch (f.kind) {
    case TK_DIAG_CONST: case TK_DIAG_TABLE: return share(f.fixmask);
    case TK_PAIRSWAP: {
      const uint64_t ctrl = f.fixmask & ~f.xmask;
      return std::min(1.0, share(ctrl) * 2.0 / double(uint64_t(1) << __builtin_popcountll(f.xmask)));
    }
    default: return 1.0;
  }
}

GateForm form_any(const LoweredOp& op) {
  GateForm f;
  f.qubits = op.qubits;
  switch (op.kind) {
    case LoweredKind::Nothing: f.nothing = true; return f;
    case LoweredKind::Dense: {
      const int k = int(op.qubits.size());
      const int gd = 1 << k;
      bool diag = true;
      for (int r = 0; r < gd && diag; ++r)
        for (int c = 0; c < gd; ++c)
          if (r != c && !zero_c(op.matrix[size_t(r) * gd + c])) {
            diag = false;
            break;
          }
      if (diag && k <= MAX_TABLE_K) {
        std::vector<CplxD> d(gd);
        for (int x = 0; x < gd; ++x) d[x] = op.matrix[size_t(x) * gd + x];
        return form_diag_table(op.qubits, d);
      }
      // circuit text names dense matrices on one qubit only (every named gate on more is monomial)
      if (k > 1) return f;
      f.tileable = true;
      f.kind = TK_DENSE1;
      f.moving = uint64_t(1) << op.qubits[0];
      f.c = op.matrix;
      return f;
    }
    case LoweredKind::Monomial: {
      const int k = int(op.qubits.size());
      const int gd = 1 << k;
      bool diagonal = true;
      for (int x = 0; x < gd; ++x) diagonal &= op.image[x] == uint32_t(x);
      if (diagonal && k <= MAX_TABLE_K) return form_diag_table(op.qubits, op.matrix);
      if (k > MAX_TABLE_K) return f;
      // the pair-swap shape of launch_perm_table; other tables run as their own kernels
      uint32_t d = 0;
      bool ok = true;
      std::vector<uint32_t> moved;
      for (int x = 0; x < gd; ++x)
        if (op.image[x] != uint32_t(x)) {
          moved.push_back(uint32_t(x));
          const uint32_t dx = op.image[x] ^ uint32_t(x);
          if (d == 0) d = dx;
          ok &= dx == d && op.image[op.image[x]] == uint32_t(x);
        } else {
          ok &= one_c(op.matrix[x]);
        }
      if (!ok || !d) return f;
      const uint32_t hbit = 1u << (31 - __builtin_clz(d));
      std::vector<uint32_t> leads;
      for (uint32_t x : moved)
        if (!(x & hbit)) leads.push_back(x);
      uint32_t ones = (1u << k) - 1, zeros = (1u << k) - 1;
      for (uint32_t x : leads) ones &= x, zeros &= ~x;
      const int nfixed = __builtin_popcount(ones) + __builtin_popcount(zeros);
      ok &= leads.size() == (size_t(1) << (k - nfixed)) && (zeros & hbit);
      if (!ok) return f;
      const CplxD c_j = op.matrix[leads[0]], c_i = op.matrix[leads[0] ^ d];
      for (uint32_t x : leads)
        ok &= op.matrix[x].re == c_j.re && op.matrix[x].im == c_j.im && op.matrix[x ^ d].re == c_i.re &&
              op.matrix[x ^ d].im == c_i.im;
      if (!ok) return f;
      f.tileable = true;
      f.kind = TK_PAIRSWAP;
      for (int j = 0; j < k; ++j) {
        if (((ones | zeros) >> j) & 1) f.fixmask |= uint64_t(1) << op.qubits[j];
        if ((ones >> j) & 1) f.ones |= uint64_t(1) << op.qubits[j];
        if ((d >> j) & 1) f.xmask |= uint64_t(1) << op.qubits[j];
      }
      f.moving = f.xmask;
      f.c = {c_i, c_j};
      f.flags = (one_c(c_i) ? 1u : 0u) | (one_c(c_j) ? 2u : 0u);
      return f;
    }
    case LoweredKind::PhasePoly: {
      const PolyTerms& t = op.poly;
      const int nt = int(t.coeffs.size());
      if (nt == 0 && t.scalar_is_one && (t.constant & ((t.bits >= 64 ? 0 : (uint64_t(1) << t.bits)) - 1)) == 0) {
        f.nothing = true;
        return f;
      }
      if (nt > MAX_PASS_TERMS || t.parities.size() > size_t(MAX_PASS_PARITIES) || t.bits > 32) return f;
      f.tileable = true;
      f.kind = TK_PHASEPOLY;
      f.poly = &op.poly;
      return f;
    }
    case LoweredKind::Pauli:  // Pauli gates come only from the API, not from circuit text: own kernel
      if (op.x == 0 && op.z == 0 && (op.phase & 3) == 0) f.nothing = true;
      return f;
  }
  return f;
}

// A gate with an infinite or NaN constant keeps its own kernel, which leaves zero amplitudes alone.
GateForm form_of(const LoweredOp& op) {
  GateForm f = form_any(op);
  for (const auto& c : f.c)
    if (!std::isfinite(c.re) || !std::isfinite(c.im)) f.tileable = false;
  return f;
}

// the window's tile-local position of each global bit (-1: outside)
struct Window {
  PassGeom g{};
  int local[64];
  uint64_t mask = 0;
};

Window make_window(uint32_t n, int T, uint64_t moving) {
  Window W;
  uint64_t m = moving;
  for (uint32_t q = 0; q < n && __builtin_popcountll(m) < T; ++q) m |= uint64_t(1) << q;
  W.mask = m;
  int w = 0;
  while (w < int(n) && ((m >> w) & 1)) ++w;
  W.g.T = __builtin_popcountll(m);
  W.g.w = w;
  W.g.nh = 0;
  for (int i = 0; i < 64; ++i) W.local[i] = -1;
  for (int q = 0; q < w; ++q) W.local[q] = q;
  for (uint32_t q = uint32_t(w); q < n; ++q)
    if ((m >> q) & 1) {
      W.local[q] = w + W.g.nh;
      W.g.hq[W.g.nh++] = uint8_t(q);
    }
  return W;
}

uint32_t local_mask(const Window& W, uint64_t gm) {
  uint32_t l = 0;
  for (int q = 0; q < 64; ++q)
    if (((gm >> q) & 1) && W.local[q] >= 0) l |= 1u << W.local[q];
  return l;
}

}  // namespace

// A planned run of gates: passes and the gates that run as their own kernels.
struct PlainPlan {
  struct Item {
    bool pass = false;
    size_t gate = 0;              // direct: index into `gates`
    Window win;
    std::vector<DevOp> ops;
    std::vector<SignItem> signs;
  };
  int precision = NCSIM_C128;
  std::vector<const LoweredOp*> gates;
  std::vector<Item> items;
  std::vector<double> cpool;      // complex values, interleaved
  std::vector<uint32_t> upool;
  std::vector<uint64_t> ppool;
  int device = -1;
  void* d_cpool = nullptr;
  uint32_t* d_upool = nullptr;
  uint64_t* d_ppool = nullptr;
  size_t passes = 0;
  ~PlainPlan() {
    if (device >= 0) {
      int cur = 0;
      cudaGetDevice(&cur);
      cudaSetDevice(device);
      cudaFree(d_cpool);
      cudaFree(d_upool);
      cudaFree(d_ppool);
      cudaSetDevice(cur);
    }
  }
};

namespace {

int pass_tile_bits(uint32_t n) { return int(std::min<uint32_t>(n, MAX_TILE_BITS)); }

// encode a gate form against a window (appends pool data)
TileOp encode(const GateForm& f, const Window& W, PlainPlan& P) {
  TileOp op{};
  op.kind = f.kind;
  auto push_c = [&](const CplxD& c) {
    P.cpool.push_back(c.re);
    P.cpool.push_back(c.im);
  };
  op.cp = uint32_t(P.cpool.size() / 2);
  op.up = uint32_t(P.upool.size());
  const uint64_t out = ~W.mask;
  switch (f.kind) {
    case TK_DENSE1:
      op.l0 = uint32_t(W.local[f.qubits[0]]);
      for (auto& c : f.c) push_c(c);
      break;
    case TK_DIAG_CONST:
    case TK_PAIRSWAP: {
      op.lfix = local_mask(W, f.fixmask);
      op.lones = local_mask(W, f.ones);
      op.gfix = f.fixmask & out;
      op.gval = f.ones & out;
      op.lx = local_mask(W, f.xmask);
      op.flags = f.flags;
      for (auto& c : f.c) push_c(c);
      break;
    }
    case TK_DIAG_1Q: {
      const uint32_t q = f.qubits[0];
      if (W.local[q] >= 0) {
        op.l0 = uint32_t(W.local[q]);
      } else {
        op.flags = 1;
        op.l1 = q;
      }
      for (auto& c : f.c) push_c(c);
      break;
    }
    case TK_DIAG_TABLE: {
      const int k = int(f.qubits.size());
      op.k = uint32_t(k);
      op.lfix = local_mask(W, f.fixmask);
      op.lones = op.lfix;
      op.gfix = f.fixmask & out;
      op.gval = f.fixmask & out;
      for (uint32_t q : f.qubits) P.upool.push_back(W.local[q] >= 0 ? uint32_t(W.local[q]) : 256u + q);
      const size_t nb = f.unit.size();
      std::vector<uint32_t> words((nb + 3) / 4, 0);
      for (size_t x = 0; x < nb; ++x) words[x / 4] |= uint32_t(f.unit[x]) << (8 * (x % 4));
      P.upool.insert(P.upool.end(), words.begin(), words.end());
      for (auto& c : f.c) push_c(c);
      break;
    }
    case TK_PHASEPOLY: {
      const PolyTerms& t = *f.poly;
      const int nt = int(t.coeffs.size());
      op.k = uint32_t(nt);
      op.gz = uint32_t(P.ppool.size());  // parity offset
      P.upool.push_back(t.bits);
      P.upool.push_back(t.root_table.empty() ? 0u : 1u);
      P.upool.push_back(t.scalar_is_one ? 1u : 0u);
      P.upool.push_back(uint32_t(t.constant));
      P.upool.push_back(uint32_t(t.constant >> 32));
      for (int i = 0; i <= nt; ++i) P.upool.push_back(t.term_start[i]);
      for (int i = 0; i < nt; ++i) P.upool.push_back(uint32_t(t.coeffs[i]));
      P.ppool.insert(P.ppool.end(), t.parities.begin(), t.parities.end());
      push_c(t.scalar);
      for (auto& c : t.root_table) push_c(c);
      break;
    }
  }
  return op;
}

// tile bits an op couples (0 for the ops that act on each element alone)
uint32_t coupled_bits(const TileOp& op) {
  switch (op.kind) {
    case TK_DENSE1: return 1u << op.l0;
    case TK_PAIRSWAP: return op.lx;
    default: return 0;
  }
}

// whether an op goes into a chain: tables, polynomials and exchanges across more than two bits sweep the tile by themselves
bool chainable(const TileOp& op) {
  if (op.kind == TK_DIAG_TABLE) return false;
  if (op.kind == TK_PHASEPOLY) return op.k == 0;
  return op.kind != TK_PAIRSWAP || __builtin_popcount(op.lx) <= 2;
}

// Orders a chain's thread bits: the lowest SB (a quarter warp of 16-byte elements, half a
// warp of 8-byte ones) on tile bits of distinct residues mod SB, so that their accesses
// fall into distinct banks (swz), the rest ascending.
void thread_bits(int T, uint32_t cmask, int SB, uint8_t* at) {
  std::vector<int> free_bits;
  for (int b = 0; b < T; ++b)
    if (!((cmask >> b) & 1)) free_bits.push_back(b);
  std::vector<int> first, rest;
  uint32_t seen = 0;
  for (int b : free_bits) {
    const uint32_t r = 1u << (b % SB);
    if (int(first.size()) < SB && !(seen & r)) first.push_back(b), seen |= r;
    else rest.push_back(b);
  }
  int i = 0;
  for (int b : first) at[i++] = uint8_t(b);
  for (int b : rest) at[i++] = uint8_t(b);
}

// Groups a pass's ops into chains: maximal runs of consecutive ops whose coupled bits fit in
// one cube of CUBE_BITS tile bits, each op encoded against its cube.
std::vector<DevOp> chainify(const std::vector<TileOp>& ops, int T, PlainPlan& P, std::vector<SignItem>& signs) {
  std::vector<DevOp> out;
  const auto cst = [&](uint32_t i) { return make_double2(P.cpool[2 * size_t(i)], P.cpool[2 * size_t(i) + 1]); };
  uint32_t chains = 0;
  size_t i = 0;
  while (i < ops.size()) {
    if (!chainable(ops[i])) {
      const TileOp& op = ops[i++];
      DevOp d{};
      d.g.gfix = op.gfix;
      d.g.gval = op.gval;
      if (op.kind == TK_DIAG_TABLE) {
        d.h.kind = DK_TABLE;
        d.x.a[0] = op.k;
        d.x.a[1] = op.up;
        d.x.a[2] = op.cp;
        d.x.a[3] = op.lfix;
        d.x.a[4] = op.lones;
      } else if (op.kind == TK_PHASEPOLY) {
        d.h.kind = DK_POLY;
        d.x.a[0] = op.k;
        d.x.a[1] = op.up;
        d.x.a[2] = op.cp;
        d.x.a[3] = uint32_t(op.gz);
      } else {
        d.h.kind = DK_TILE_SWAP;
        d.x.a[0] = uint32_t(__builtin_popcount(op.lfix));
        d.x.a[1] = op.flags;
        d.x.a[2] = op.lx;
        d.x.a[3] = op.lones;
        d.x.a[4] = op.cp;
        for (int b = 0, f = 0; b < T; ++b)
          if ((op.lfix >> b) & 1) d.x.a[6 + f / 8] |= uint32_t(b) << (4 * (f & 7)), ++f;
      }
      out.push_back(d);
      continue;
    }
    uint32_t C = 0;
    size_t j = i;
    while (j < ops.size() && chainable(ops[j])) {
      const uint32_t need = coupled_bits(ops[j]);
      if (__builtin_popcount(C | need) > CUBE_BITS) break;
      C |= need;
      ++j;
    }
    // filled with the highest free bits: the low ones stay with the lanes
    for (int b = T - 1; b >= 0 && __builtin_popcount(C) < CUBE_BITS; --b) C |= 1u << b;
    int cpos[CUBE_BITS], nc = 0;
    for (int b = 0; b < T; ++b)
      if ((C >> b) & 1) cpos[nc++] = b;
    auto cube = [&](uint32_t l) {
      for (uint32_t q = 0; q < CUBE_BITS; ++q)
        if (cpos[q] == int(l)) return q;
      return 0u;
    };
    uint32_t loff[CUBE] = {};
    for (int b = 0; b < CUBE; ++b)
      for (int q = 0; q < CUBE_BITS; ++q)
        if ((b >> q) & 1) loff[b] |= 1u << cpos[q];
    // the cube elements b whose cube bits match the op's fixed pattern there
    auto elements = [&](uint32_t lfix, uint32_t lones) {
      uint32_t em = 0;
      for (int b = 0; b < CUBE; ++b)
        if ((loff[b] & lfix) == (lones & C & lfix)) em |= 1u << b;
      return em;
    };
    DevOp head{};
    head.h.kind = DK_CHAIN;
    for (int q = 0; q < CUBE_BITS; ++q) head.h.gml |= uint32_t(cpos[q]) << (8 * q);
    uint8_t tb[MAX_TILE_BITS] = {};
    thread_bits(T, C, P.precision == NCSIM_C128 ? 3 : 4, tb);
    for (int q = 0; q < T - CUBE_BITS; ++q) head.x.a[q >> 2] |= uint32_t(tb[q]) << (8 * (q & 3));
    head.h.gvl = chains++;
    const size_t at_head = out.size();
    out.push_back(head);
    bool pending = false;
    const auto flush = [&] {
      if (!pending) return;
      DevOp d{};
      d.h.kind = DK_FLUSH;
      out.push_back(d);
      pending = false;
    };
    for (size_t o = i; o < j; ++o) {
      const TileOp& op = ops[o];
      DevOp d{};
      d.g.gfix = op.gfix;
      d.g.gval = op.gval;
      d.h.gml = op.lfix & ~C;
      d.h.gvl = op.lones & ~C;
      if (op.kind == TK_DENSE1 || op.kind == TK_PAIRSWAP) flush();
      switch (op.kind) {
        case TK_DENSE1: {
          for (int q = 0; q < 4; ++q) d.x.c[q] = cst(op.cp + uint32_t(q));
          const double2 m00 = d.x.c[0], m01 = d.x.c[1], m10 = d.x.c[2], m11 = d.x.c[3];
          const bool real = m00.y == 0.0 && m01.y == 0.0 && m10.y == 0.0 && m11.y == 0.0;
          const bool col = m00.x == m10.x && m00.y == m10.y;
          const bool half = m00.x == 0.5 && m10.x == 0.5;
          DevKind kind = DK_D1;
          if (real) kind = col ? DK_D1RE : DK_D1R;
          else if (m00.y == 0.0 && m11.y == 0.0 && m01.x == 0.0 && m10.x == 0.0) kind = DK_D1X;
          else if (col) kind = DK_D1E;
          else if (half && m00.y == 0.5 && m10.y == -0.5) kind = DK_D1S;
          else if (half && m00.y == -0.5 && m10.y == 0.5) kind = DK_D1SD;
          d.h.kind = kind + cube(op.l0);
          d.g.gfix = d.g.gval = 0;
          d.h.gml = d.h.gvl = 0;
          break;
        }
        case TK_DIAG_CONST: {
          const double2 c = cst(op.cp);
          d.h.em = elements(op.lfix, op.lones);
          int half = -1;  // the cube bit whose upper half the mask is
          for (int q = 0; q < CUBE_BITS; ++q)
            if (d.h.em == elements(1u << cpos[q], 1u << cpos[q])) half = q;
          const bool all = d.h.em == (1u << CUBE) - 1;
          if (c.x == -1.0 && c.y == 0.0) {
            // signs that follow one another are one op
            pending = true;
            if (out.back().h.kind == DK_SIGNS) {
              ++out.back().h.em;
              d.h.kind = DK_CHAIN;  // nothing more to add
            } else {
              d.h.kind = DK_SIGNS;
              d.h.gml = uint32_t(signs.size());
            }
            signs.push_back({(op.lfix & ~C), d.h.em, op.gfix});
            if (d.h.kind == DK_CHAIN) continue;
            d.h.em = 1;
            d.h.gvl = 0;
            d.g.gfix = d.g.gval = 0;
          } else if (c.x == 0.0 && (c.y == 1.0 || c.y == -1.0)) {
            d.h.kind = half >= 0 ? DK_TURN + uint32_t(half) : all ? DK_TURN_ALL : DK_TURN_MASK;
            d.x.a[0] = c.y > 0 ? 0x80000000u : 0u;  // i u = (-u.y, u.x)
            d.x.a[1] = c.y > 0 ? 0u : 0x80000000u;  // -i u = (u.y, -u.x)
          } else {
            d.h.kind = half >= 0 ? DK_PH + uint32_t(half) : all ? DK_PH_ALL : DK_PH_MASK;
            d.x.c[0] = c;
          }
          break;
        }
        case TK_DIAG_1Q:
          d.x.c[0] = cst(op.cp);
          d.x.c[1] = cst(op.cp + 1);
          d.h.gml = d.h.gvl = 0;
          if (op.flags & 1) {  // outside the window: one of the two phases, by the bit of the tile's base
            d.h.kind = DK_PH_ALL | DK_COND;
            d.g.gfix = uint64_t(1) << op.l1;
            d.g.gval = 0;
            out.push_back(d);
            d.x.c[0] = d.x.c[1];
            d.g.gval = d.g.gfix;
          } else if ((C >> op.l0) & 1) {
            d.h.kind = DK_RZ + cube(op.l0);
          } else {
            d.h.kind = DK_RZ_OUT;
            d.h.gml = d.h.gvl = 1u << op.l0;
          }
          break;
        case TK_PAIRSWAP: {
          uint32_t x = 0;
          for (int b = 0; b < T; ++b)
            if ((op.lx >> b) & 1) x |= 1u << cube(uint32_t(b));
          uint32_t xi = 0;
          while (SWAP_X[xi] != x) ++xi;
          const uint32_t lead = elements(op.lfix, op.lones);
          if ((op.flags & 3) == 3) {
            d.h.kind = DK_SWAP + xi;
            for (uint32_t b = 0; b < CUBE; ++b)
              if ((lead >> b) & 1) d.h.em |= 1u << std::min(b, b ^ x);
          } else {
            d.h.kind = DK_SWAPC + xi;
            d.h.em = lead | (op.flags << 16);
            d.x.c[0] = cst(op.cp);
            d.x.c[1] = cst(op.cp + 1);
          }
          break;
        }
        default:  // TK_PHASEPOLY
          d.h.kind = DK_POLY_CONST;
          d.h.gml = d.h.gvl = 0;
          d.x.a[0] = op.k;
          d.x.a[1] = op.up;
          d.x.a[2] = op.cp;
          d.x.a[3] = uint32_t(op.gz);
          break;
      }
      if (d.g.gfix) d.h.kind |= DK_COND;
      out.push_back(d);
    }
    flush();
    out[at_head].h.em = uint32_t(out.size() - at_head - 1);
    i = j;
  }
  return out;
}

// whether an op of this kind carries constants (else words)
bool has_constants(uint32_t kind) {
  kind &= ~uint32_t(DK_COND);
  return (kind >= DK_D1 && kind <= DK_PH_MASK) || (kind >= DK_RZ && kind <= DK_RZ_OUT) || (kind >= DK_SWAPC && kind < DK_POLY_CONST);
}
void put_args(OpArgs<double>& to, const DevOp& from) { to = from.x; }
void put_args(OpArgs<float>& to, const DevOp& from) {
  to = OpArgs<float>{};
  for (int q = 0; q < 8; ++q) to.a[q] = from.x.a[q];
  if (has_constants(from.h.kind))
    for (int q = 0; q < 4; ++q) to.c[q] = make_float2(float(from.x.c[q].x), float(from.x.c[q].y));
}

}  // namespace

// Plans the gates of a run for one register.  Returns null when no pass would
// carry two or more gates (the gate-by-gate path then runs them as before).
std::shared_ptr<PlainPlan> plan_plain_passes(uint32_t n, int precision, const std::vector<const LoweredOp*>& gates) {
  if (n < 8) return nullptr;
  auto P = std::make_shared<PlainPlan>();
  P->precision = precision;
  P->gates = gates;
  const int T = pass_tile_bits(n);
  std::vector<GateForm> forms(gates.size());
  for (size_t i = 0; i < gates.size(); ++i) forms[i] = form_of(*gates[i]);
  std::vector<size_t> cur;
  const uint64_t low = n > uint32_t(FREE_WINDOW_QUBITS) ? (uint64_t(1) << LOW_WINDOW_BITS) - 1 : 0;
  uint64_t moving = low;  // the window's qubits so far
  auto flush = [&] {
    if (cur.empty()) return;
    // a pass reads and writes the whole register once; gates whose own kernels
    // touch less than that between them stay gate by gate
    double shares = 0.0;
    for (size_t i : cur) shares += touched_share(forms[i], precision);
    if (cur.size() == 1 || shares < 1.25) {
      for (size_t i : cur) {
        PlainPlan::Item it;
        it.gate = i;
        P->items.push_back(it);
      }
    } else {
      PlainPlan::Item it;
      it.pass = true;
      it.win = make_window(n, T, moving);
      std::vector<TileOp> ops;
      for (size_t i : cur) ops.push_back(encode(forms[i], it.win, *P));
      it.ops = chainify(ops, it.win.g.T, *P, it.signs);
      if (it.ops.size() > size_t(MAX_PASS_OPS)) throw Error(NCSIM_ERR_INVALID, "tiled pass: too many ops");
      P->passes += 1;
      P->items.push_back(std::move(it));
    }
    cur.clear();
    moving = low;
  };
  for (size_t i = 0; i < gates.size(); ++i) {
    const GateForm& f = forms[i];
    if (f.nothing) continue;
    if (!f.tileable) {
      flush();
      PlainPlan::Item it;
      it.gate = i;
      P->items.push_back(it);
      continue;
    }
    // a gate makes at most three ops (a chain's head, two phases or a flush and the op; a chain's last
    // flush comes with a sign, which is one op): a pass of MAX_PASS_OPS / 3 gates fits
    if (__builtin_popcountll(moving | f.moving) > T || cur.size() >= size_t(MAX_PASS_OPS / 3)) flush();
    cur.push_back(i);
    moving |= f.moving;
  }
  flush();
  if (P->passes == 0) return nullptr;
  return P;
}

void apply_lowered(ncsim_state* s, const LoweredOp& op);

template <class R>
void launch_pass(ncsim_state* s, const PlainPlan& P, const PlainPlan::Item& it, bool after_pass) {
  PassParams<R> pp;
  pp.amp = reinterpret_cast<V<R>*>(s->amp);
  pp.g = it.win.g;
  pp.ntiles = s->len >> it.win.g.T;
  pp.nops = uint32_t(it.ops.size());
  pp.nchains = 0;
  pp.nsigns = uint32_t(it.signs.size());
  std::copy(it.signs.begin(), it.signs.end(), pp.sign);
  for (size_t i = 0; i < it.ops.size(); ++i) {
    pp.head[i] = it.ops[i].h;
    pp.cond[i] = it.ops[i].g;
    put_args(pp.args[i], it.ops[i]);
    pp.nchains += it.ops[i].h.kind == DK_CHAIN;
  }
  pp.upool = P.d_upool;
  pp.ppool = P.d_ppool;
  // the complex pool as this precision's values
  pp.cpool = reinterpret_cast<const V<R>*>(P.d_cpool);
  const int T = it.win.g.T;
  const unsigned threads = std::max(32u, 1u << (T - CUBE_BITS));
  const size_t smem = 2 * (size_t(1) << T) * sizeof(V<R>) + it.ops.size() * sizeof(OpArgs<R>) + it.signs.size() * sizeof(SignItem) +
                      size_t(pp.nchains) * threads * sizeof(uint16_t);
  {
    // the kernel's shared-memory limit, set once per device and precision (host threads may race here)
    static std::mutex mu;
    static bool done[64][2] = {};
    std::lock_guard<std::mutex> lk(mu);
    const int dev = s->device;
    if (dev < 0 || dev >= 64 || !done[dev][sizeof(R) == 8]) {
      NCSIM_CUDA(cudaFuncSetAttribute(
          k_plain_pass<R>, cudaFuncAttributeMaxDynamicSharedMemorySize,
          int(2 * (size_t(1) << MAX_TILE_BITS) * sizeof(V<R>) + MAX_PASS_OPS * (sizeof(OpArgs<R>) + sizeof(SignItem)) +
              MAX_PASS_CHAINS * (1 << (MAX_TILE_BITS - CUBE_BITS)) * sizeof(uint16_t))));
      if (dev >= 0 && dev < 64) done[dev][sizeof(R) == 8] = true;
    }
  }
  int per_sm = 1;
  NCSIM_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_plain_pass<R>, int(threads), smem));
  const uint64_t grid = std::min<uint64_t>(pp.ntiles, uint64_t(sm_count()) * uint64_t(std::max(per_sm, 1)));
  ProfScope ps(s, K_PLAIN_PASS, 2.0 * double(s->len) * double(s->elem_bytes()));
  // A pass of a few tiles per CTA launches under the end of the pass before it: at n = 16 (8 passes) 200 ->
  // 164 us, n = 20 (14 passes) 443 -> 415; with more tiles the launch is a small part, and CTAs that arrive
  // in the order the last ones leave lose more (n = 22 1248 -> 1264, n = 24 4.92 -> 5.34 ms).
  cudaLaunchAttribute overlap{};
  overlap.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  overlap.val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t launch{};
  launch.gridDim = dim3(unsigned(grid));
  launch.blockDim = dim3(threads);
  launch.dynamicSmemBytes = smem;
  launch.stream = s->stream;
  launch.attrs = &overlap;
  launch.numAttrs = after_pass && pp.ntiles <= 4 * grid ? 1 : 0;
  NCSIM_CUDA(cudaLaunchKernelEx(&launch, k_plain_pass<R>, pp));
}

void run_plain_plan(ncsim_state* s, PlainPlan& P) {
  if (P.device < 0) {
    // The pools go up on the state's own stream and are waited for: a cudaMemcpy from pageable
    // memory runs on the legacy stream and may return before its DMA lands, and the pass
    // kernels run on a non-blocking stream that does not wait for the legacy one.
    cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
    NCSIM_CUDA(cudaStreamIsCapturing(s->stream, &cap));
    if (cap != cudaStreamCaptureStatusNone) throw Error(NCSIM_ERR_DEVICE, "a gate plan is uploaded outside stream capture");
    const bool dbl = s->precision == NCSIM_C128;
    const size_t nc = P.cpool.size() / 2;
    std::vector<float> f;
    if (!dbl) f.assign(P.cpool.begin(), P.cpool.end());
    NCSIM_CUDA(cudaMalloc(&P.d_cpool, std::max<size_t>(nc, 1) * (dbl ? sizeof(double2) : sizeof(float2))));
    NCSIM_CUDA(cudaMalloc(&P.d_upool, std::max<size_t>(P.upool.size(), 1) * sizeof(uint32_t)));
    NCSIM_CUDA(cudaMalloc(&P.d_ppool, std::max<size_t>(P.ppool.size(), 1) * sizeof(uint64_t)));
    P.device = s->device;  // the destructor frees the pools from here on
    if (nc)
      NCSIM_CUDA(cudaMemcpyAsync(P.d_cpool, dbl ? static_cast<const void*>(P.cpool.data()) : f.data(),
                                 nc * (dbl ? sizeof(double2) : sizeof(float2)), cudaMemcpyHostToDevice, s->stream));
    if (!P.upool.empty())
      NCSIM_CUDA(cudaMemcpyAsync(P.d_upool, P.upool.data(), P.upool.size() * sizeof(uint32_t), cudaMemcpyHostToDevice,
                                 s->stream));
    if (!P.ppool.empty())
      NCSIM_CUDA(cudaMemcpyAsync(P.d_ppool, P.ppool.data(), P.ppool.size() * sizeof(uint64_t), cudaMemcpyHostToDevice,
                                 s->stream));
    NCSIM_CUDA(cudaStreamSynchronize(s->stream));
  }
  if (P.device != s->device) throw Error(NCSIM_ERR_DEVICE, "a gate plan stays on the device it was built for");
  bool after_pass = false;
  for (const auto& it : P.items) {
    if (!it.pass) apply_lowered(s, *P.gates[it.gate]);
    else if (s->precision == NCSIM_C128) launch_pass<double>(s, P, it, after_pass);
    else launch_pass<float>(s, P, it, after_pass);
    after_pass = it.pass;
  }
}

}  // namespace ncsim
