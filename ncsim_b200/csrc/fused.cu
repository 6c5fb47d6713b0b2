// Precision form, device side: one kernel launch per pass.
//
// A persistent CTA per SM streams tiles of 2^12 complex64 amplitudes (32 KB)
// through shared memory: two producer warps copy 16-byte chunks with cp.async
// (completion on the tile's mbarrier through cp.async.mbarrier.arrive) into
// five rotating tile buffers, and a third works out what the tile's index bits
// outside the window decide (which diagonal terms apply, the factor of those
// that act on the whole tile).  The CTA takes its tiles in sets of four, and
// four warpgroups run the pass's program, one on each tile of a set, so that a
// group splits amplitudes while the others' MMAs and read-backs run; each group
// writes its finished tile back itself (16-byte stores), so the stores overlap
// the other groups' work and the producers only load.  The unitaries' B
// operands (16 KB bf16 images each) stream from L2 into three rotating slots
// (a fourth producer warp); each group's tcgen05.commit (or release) frees a
// slot.  Per group and tile:
//   unitary op: the tile as 32 rows (the unitary's 5 qubits) x 128 columns;
//     each thread owns a column, splits its 32 amplitudes into bf16 hi/lo
//     and writes them into its own TMEM lane (A = X^T, 128 x 64, K-major,
//     tcgen05.st); one lane of the group's first warp issues 12 tcgen05.mma
//     with A in TMEM (M=128, N=64, K=16, bf16 in, f32 accumulate in the
//     group's 64 TMEM columns):
//       D = Xhi.Rhi + Xlo.Rhi + Xhi.Rlo
//     with R the real form of the fused unitary (bf16 hi/lo images made on the
//     host, output columns ordered so that each row's real and imaginary
//     parts are adjacent); each thread reads its D row back (tcgen05.ld) and
//     writes the 32 new amplitudes into the tile;
//   diagonal op: reduced, where it can be, to a phase per column and a sign
//     mask over the rows of a neighbouring unitary and applied in that
//     unitary's split or read-back; otherwise the tile index splits into two
//     6-bit halves, the active terms fold into a 64-entry phase table per half
//     and a parity table for cross-half signs, and one sweep applies them.
// What bounds it (n = 28, 4.4 unitaries a pass): the CUDA cores' work around the
// MMAs, issue 57% busy, the shared-memory pipe 63%, the tensor pipe 26%, HBM 23%
// (41% of the time the pass's read and write take).  What the layout of that work
// measured, n = 28, 5 passes (10.1 ms before): the MMAs issued under elect.sync
// with warp-uniform operands (12 in 380 cycles, the pipe's own rate; 880 from a
// thread picked by its index), the tile's facts on a warp of their own, addresses by
// one XOR, residuals by sub.f32.bf16, signs by two masks a row: 8.0 ms; column bits
// ordered for free banks and split and read-back loops without conditional updates: 7.65 ms.
// Tried and slower: one warp issuing every group's MMAs (8.5), two accumulator
// reads in flight (spills: 9.9), 16-byte moves where row bit 0 is tile bit 0 (8.2).
// Every wait on an mbarrier is bounded in time: on timeout the CTA records an
// error code and every role stops at its next uniform decision point, waits
// for its own copies and frees its TMEM.
#include <cuda_bf16.h>

#include "engine.cuh"
#include "fused_plan.hpp"

#include <algorithm>
#include <cstring>
#include <memory>

namespace ncsim {
namespace fused {

namespace {

constexpr int GROUP_THREADS = 128;                       // one warpgroup runs the program on one tile
constexpr int GROUPS = 4;                                // four tiles in flight per CTA
constexpr int COMPUTE_THREADS = GROUPS * GROUP_THREADS;  // warps 0-15
constexpr int WARP_TILES = COMPUTE_THREADS / 32;         // warps 16-17: tile loads
constexpr int TILE_THREADS = 64;
constexpr int WARP_OPS = WARP_TILES + 2;                 // warp 18: B operand images
constexpr int WARP_FACTS = WARP_OPS + 1;                 // warp 19: what each tile's index bits decide
constexpr int THREADS = COMPUTE_THREADS + TILE_THREADS + 64;
constexpr int TILE = 1 << TILE_BITS;
constexpr uint32_t TILE_BYTES = uint32_t(TILE) * 8u;
constexpr int OPERAND_BYTES = 16384;  // B: bf16 hi (8 KB) + lo (8 KB)
constexpr int NTILEBUF = GROUPS + 1;  // tile buffers rotating over the CTA's tiles (one loading ahead)
constexpr int NOPSLOT = 3;            // B operand slots rotating over the unitary uses
// Shared memory, from the tiles' base on: the tile buffers sit at multiples of their own size, so
// a tile element's address is one XOR (base ^ column ^ row); one operand slot lies below them, the
// others above.  The small tables (struct Tables) fill what is left at the bottom.
constexpr uint32_t SM_SLOTS = NTILEBUF * TILE_BYTES;
constexpr uint32_t SM_TPHASE = SM_SLOTS + (NOPSLOT - 1) * uint32_t(OPERAND_BYTES);
constexpr int MAX_CHUNKS = 48;  // column-term chunks per pass
constexpr uint32_t SM_END = SM_TPHASE + NTILEBUF * MAX_CHUNKS * uint32_t(sizeof(float2));
constexpr uint32_t SM_DYNAMIC = TILE_BYTES + SM_END;  // the tiles start within TILE_BYTES of the dynamic base
// per group 128 columns: the accumulator D (64), the A operand's bf16 hi (32) and lo (32)
constexpr uint32_t TMEM_COLS = 512;  // 128 per group, rounded up to a power of two
constexpr long long WAIT_CYCLES = 4000000000ll;  // about 2 s at 1.9 GHz
constexpr int HALF = TILE_BITS / 2;              // 6-bit halves of the tile index
constexpr int COL_BITS = TILE_BITS - GROUP_QUBITS;  // a unitary's column index: the tile bits outside its qubits
// Tile layout in shared memory: element e sits at e ^ L(e), where the linear map L folds
// tile bits 4..11 into element bits 1..3 (bit j contributes w[j - 4] below).  A unitary's
// thread owns a column whose 32 lanes step through its lowest non-gate bits; without
// the fold, gate qubits among tile bits 0..3 send those lanes to a few banks (up to
// 16-way conflicts).  The fold keeps bit 0, so 16-byte pairs stay contiguous, and it
// is linear: the address of (column | row) is the XOR of the two parts' addresses.
// The weights minimise the modelled conflicts over the window placements of the
// layered-circuit plans (3.2 -> 2.3 shared-memory wavefronts per warp access; 2 is the
// minimum for 8-byte elements).
__host__ __device__ inline uint32_t swz_fold(uint32_t e) {
  const uint8_t w[TILE_BITS - 4] = {14, 6, 12, 10, 14, 12, 8, 6};
  uint32_t l = 0;
#pragma unroll
  for (int j = 4; j < TILE_BITS; ++j)
    if ((e >> j) & 1u) l ^= w[j - 4];
  return l;
}

enum TermClass : uint8_t { T_LOW = 0, T_HIGH = 1, T_CROSS_SIGN = 2, T_GENERIC = 3 };

struct alignas(16) OpDesc {
  uint8_t kind;  // 0 unitary, 1 terms, 2 terms applied by the next unitary's split, 3 by the previous one's read-back
  uint8_t u;     // unitary index (operand slot)
  // terms [t0, t1) sorted by class: low half [t0,tl), high half [tl,th),
  // cross-half signs [th,tc), the rest [tc,t1)
  uint16_t t0, tl, th, tc, t1;
  uint8_t pc0, pc1;  // unitary: chunks of the preceding terms op, applied while splitting
  uint8_t qc0, qc1;  // unitary: chunks of the following terms op, applied while reading back
};

struct TermDesc {
  uint64_t cmask;  // bits outside the window (constant over a tile)
  uint32_t tmask;  // tile-local bits (for a split-applied term: the unitary's non-gate bits)
  float cr, ci;
};

// Up to 32 terms of a diagonal op applied by a unitary's split or read-back,
// as bit masks over the chunk's terms (bit t = term t0 + t).  A term is active
// on a column when its bits outside the tile are set in the tile's base (a
// per-tile ballot) and its column bits are set in the column index; active
// terms then flip row signs (row[j]: rows with gate bit j set), negate the
// column (neg) or multiply it by their phase (gen; tgen: a phase on every
// column, folded into one factor per tile; only those that open the op's product,
// so that the factors multiply in the terms' order whichever way).
struct alignas(16) ColChunk {
  uint32_t need[COL_BITS];     // terms whose condition includes column bit j
  uint32_t gen;                // other phases on the whole column
  uint32_t row[GROUP_QUBITS];  // sign terms on the rows with gate bit j set
  uint32_t neg;                // -1 on the whole column
  uint32_t tgen;               // phases with no column bit, before any in gen: the same on every column
  uint16_t t0;
  uint16_t cnt;
};

// a pass as the host builds it
struct PassProgram {
  int nops, nu, nterms, nchunks;
  uint8_t pos[MAX_UNITARIES][GROUP_QUBITS];  // tile-local positions of each unitary's qubits (rows)
  uint8_t col[MAX_UNITARIES][COL_BITS];      // and of the other tile bits (columns), see column_order
  OpDesc ops[MAX_OPS];
  TermDesc terms[MAX_TERMS];
  ColChunk chunks[MAX_CHUNKS];
};
struct Terms {
  uint64_t cmask[MAX_TERMS];
  float2 coef[MAX_TERMS];
  uint16_t tmask[MAX_TERMS];
  __device__ __forceinline__ TermDesc get(int k) const { return {cmask[k], tmask[k], coef[k].x, coef[k].y}; }
};
// What a pass's CTAs read with runtime indices: made once with the plan and copied to shared memory
// by one load per thread.  (Built by every CTA from the program in the kernel's parameters, it took
// 5000 of the 11000 cycles before the first tile, as much as two unitaries.)
struct alignas(16) PassTables {
  ColChunk chunks[MAX_CHUNKS];
  OpDesc ops[MAX_OPS];
  alignas(16) uint16_t gbit[MAX_UNITARIES][8];  // byte offset in a tile of each gate bit (row bits)
  uint16_t clo[MAX_UNITARIES][16];              // byte offset of a column: its low four bits' part
  uint16_t chi[MAX_UNITARIES][8];               // and its high three bits'
  uint64_t chunk_off[TILE / 2 / TILE_THREADS];  // byte offset in the register of a tile's 16-byte chunk 64 i
  Terms terms;
  uint8_t swz[1 << (TILE_BITS - 4)];            // L(e) by e >> 4
  uint8_t win[16];                              // tile bit j is index bit win[j], ascending
  uint8_t out[32];                              // bit j of a tile's number is index bit out[j]
};
struct PassArgs {
  float2* amp;
  const PassTables* tables;
  const uint4* rops;  // nu x 16 KB operand images
  int* err;
  uint32_t ntiles;
  int nops, nu, nchunks;
};

// ---- PTX wrappers ----
__device__ __forceinline__ uint32_t smem_u32(const void* p) { return uint32_t(__cvta_generic_to_shared(p)); }

__device__ __forceinline__ void mbar_init(uint32_t bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count) : "memory");
}
__device__ __forceinline__ void mbar_arrive(uint32_t bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
}
__device__ __forceinline__ void mbar_expect_tx(uint32_t bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
}
// try_wait with a suspend-time hint: the thread sleeps (up to about 1 ms) until
// the phase completes instead of spinning
__device__ __forceinline__ bool mbar_try(uint32_t bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2, %3;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t}"
      : "=r"(ok)
      : "r"(bar), "r"(parity), "r"(1000000u)
      : "memory");
  return ok != 0;
}
// one lane of a converged warp; code under it with warp-uniform operands issues tcgen05 at full rate
__device__ __forceinline__ bool elect_one() {
  uint32_t r;
  asm volatile("{\n\t.reg .pred p;\n\telect.sync _|p, 0xffffffff;\n\tselp.u32 %0, 1, 0, p;\n\t}" : "=r"(r));
  return r != 0;
}
// bounded wait: false when the phase did not complete within WAIT_CYCLES
__device__ __forceinline__ bool mbar_wait(uint32_t bar, uint32_t parity) {
  if (mbar_try(bar, parity)) return true;
  const long long t0 = clock64();
  while (!mbar_try(bar, parity)) {
    if (clock64() - t0 > WAIT_CYCLES) return false;
  }
  return true;
}

__device__ __forceinline__ void bulk_load(uint32_t dst, const void* src, uint32_t bytes, uint32_t bar) {
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(dst),
               "l"(src), "r"(bytes), "r"(bar)
               : "memory");
}
__device__ __forceinline__ void cp_async16(uint32_t dst, const void* src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(src) : "memory");
}
// arrives on the mbarrier once this thread's earlier cp.async copies have landed
__device__ __forceinline__ void cp_async_arrive(uint32_t bar) {
  asm volatile("cp.async.mbarrier.arrive.noinc.shared::cta.b64 [%0];" ::"r"(bar) : "memory");
}
// A named barrier that also ORs a flag over its threads: every thread gets the
// same answer, so a stop decided from it is uniform across the barrier's threads.
__device__ __forceinline__ bool bar_any(int id, int count, bool v) {
  uint32_t r;
  asm volatile(
      "{\n\t.reg .pred p, q;\n\t"
      "setp.ne.u32 p, %1, 0;\n\t"
      "bar.red.or.pred q, %2, %3, p;\n\t"
      "selp.u32 %0, 1, 0, q;\n\t}"
      : "=r"(r)
      : "r"(uint32_t(v)), "r"(id), "r"(count)
      : "memory");
  return r != 0;
}

__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }

// K-major, 128-byte swizzle, 8-row atoms 1024 bytes apart (sm100 descriptor version 1)
__device__ __forceinline__ uint64_t sw128_desc(uint32_t saddr) {
  uint64_t d = uint64_t((saddr >> 4) & 0x3FFFu);
  d |= uint64_t(1) << 16;            // leading byte offset (16 B; unused by swizzled K-major)
  d |= uint64_t(1024 >> 4) << 32;    // stride byte offset between 8-row atoms
  d |= uint64_t(1) << 46;            // descriptor version for sm100
  d |= uint64_t(2) << 61;            // SWIZZLE_128B
  return d;
}

constexpr uint32_t NEGATE_A = 1u << 13;  // instruction descriptor: the product with -A

// D (TMEM) += A (TMEM, K-major rows = lanes) x B (shared memory descriptor)
__device__ __forceinline__ void mma_bf16_ta(uint32_t tmem_d, uint32_t tmem_a, uint64_t b, uint32_t idesc, uint32_t acc) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, {%5, %6, %7, %8}, p;\n\t}"
      ::"r"(tmem_d), "r"(tmem_a), "l"(b), "r"(idesc), "r"(acc), "r"(0), "r"(0), "r"(0), "r"(0));
}
// four 32-bit columns of this thread's TMEM lane
__device__ __forceinline__ void tmem_st4(uint32_t taddr, const uint32_t (&v)[4]) {
  asm volatile("tcgen05.st.sync.aligned.32x32b.x4.b32 [%0], {%1, %2, %3, %4};" ::"r"(taddr), "r"(v[0]), "r"(v[1]),
               "r"(v[2]), "r"(v[3])
               : "memory");
}
__device__ __forceinline__ void mma_commit(uint32_t bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar) : "memory");
}

#define NCSIM_TMEM_LD16(taddr, r)                                                                                     \
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];" \
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),        \
                 "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])    \
               : "r"(taddr))

// x, y rounded to bf16, x in the low half
__device__ __forceinline__ uint32_t pack_bf16(float x, float y) {
  uint32_t w;
  asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(w) : "f"(y), "f"(x));
  return w;
}
// bf16(hi - v) for both halves: minus the residual of v = (x, y) rounded to w
__device__ __forceinline__ uint32_t pack_neg_residual(uint32_t w, float x, float y) {
  float a, b;
  asm("{\n\t.reg .b16 p, q;\n\tmov.b32 {p, q}, %2;\n\tsub.f32.bf16 %0, p, %3;\n\tsub.f32.bf16 %1, q, %4;\n\t}"
      : "=f"(a), "=f"(b)
      : "r"(w), "f"(x), "f"(y));
  return pack_bf16(a, b);
}
// an amplitude at a shared-memory address (program order among these and the barriers: volatile)
__device__ __forceinline__ void lds_amp(uint32_t at, float& x, float& y) {
  asm volatile("ld.shared.v2.f32 {%0, %1}, [%2];" : "=f"(x), "=f"(y) : "r"(at));
}
__device__ __forceinline__ void sts_amp(uint32_t at, uint32_t x, uint32_t y) {
  asm volatile("st.shared.v2.b32 [%0], {%1, %2};" ::"r"(at), "r"(x), "r"(y));
}

__device__ __forceinline__ float2 cmulf(float2 a, float2 b) {
  return make_float2(a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x);
}

struct Tables : PassTables {
  uint64_t bars[2 * NTILEBUF + 2 * NOPSLOT + GROUPS];  // tile full, tile done, operand full, operand empty, mma
  float2 tab_lo[GROUPS][1 << HALF], tab_hi[GROUPS][1 << HALF];
  uint8_t tab_cross[GROUPS][1 << HALF];
  uint32_t act[NTILEBUF][MAX_CHUNKS];          // per tile: the chunks' terms active on it
  uint64_t base[NTILEBUF];                     // and its first index
  uint32_t tmem_base;
  volatile int abort;
};
static_assert(sizeof(Tables) + 1024 + uint32_t(OPERAND_BYTES) <= TILE_BYTES, "the small tables fit below the first operand slot");
// The tile's phase tables of a terms op, built by one group's 128 threads: the
// low-half phase products and cross-half sign parities (threads 0-63) and the
// high-half phase products (64-127).
__device__ __forceinline__ void build_tables(const OpDesc& op, uint64_t base, int tg, const Terms& terms,
                                             float2* tab_lo, float2* tab_hi, uint8_t* tab_cross) {
  if (tg < 64) {
    const uint32_t x = uint32_t(tg);
    float2 c = make_float2(1.f, 0.f);
    for (int k = op.t0; k < op.tl; ++k) {
      const TermDesc tm = terms.get(k);
      if ((base & tm.cmask) == tm.cmask && (x & tm.tmask) == tm.tmask) c = cmulf(c, make_float2(tm.cr, tm.ci));
    }
    tab_lo[x] = c;
    uint32_t v = 0;
    for (int k = op.th; k < op.tc; ++k) {
      const TermDesc tm = terms.get(k);
      if ((base & tm.cmask) != tm.cmask) continue;
      if (x & (tm.tmask >> HALF)) v ^= tm.tmask & ((1u << HALF) - 1);
    }
    tab_cross[x] = uint8_t(v);
  } else {
    const uint32_t x = uint32_t(tg - 64);
    float2 c = make_float2(1.f, 0.f);
    for (int k = op.tl; k < op.th; ++k) {
      const TermDesc tm = terms.get(k);
      const uint32_t hm = tm.tmask >> HALF;
      if ((base & tm.cmask) == tm.cmask && (x & hm) == hm) c = cmulf(c, make_float2(tm.cr, tm.ci));
    }
    tab_hi[x] = c;
  }
}

// the phase of tile element e under a terms op (its tables built)
__device__ __forceinline__ float2 term_phase(uint32_t e, const OpDesc& op, uint64_t base, const Terms& terms,
                                             const float2* tab_lo, const float2* tab_hi, const uint8_t* tab_cross) {
  const uint32_t lo = e & ((1u << HALF) - 1), hi = e >> HALF;
  float2 c = cmulf(tab_lo[lo], tab_hi[hi]);
  if (__popc(lo & tab_cross[hi]) & 1) c = make_float2(-c.x, -c.y);
  for (int k = op.tc; k < op.t1; ++k) {
    const TermDesc tm = terms.get(k);
    if ((base & tm.cmask) == tm.cmask && (e & tm.tmask) == tm.tmask) c = cmulf(c, make_float2(tm.cr, tm.ci));
  }
  return c;
}

// The chunks [c0, c1) of a diagonal op applied by a unitary's split or read-back,
// for column tg of that unitary (act: the chunks' terms active on this tile, without the
// tgen ones, whose product is tph).  par: bit j, the rows with gate bit j set change sign;
// bit 5, every row does.  cth: a phase for the whole column (scal: there is one).
__device__ __forceinline__ void column_chunks(const ColChunk* chunks, const uint32_t* act, const float2* tph, int c0, int c1,
                                              uint32_t tg, const float2* coef, uint32_t& par, float2& cth, bool& scal) {
  for (int c = c0; c < c1; ++c) {
    ColChunk ch;
    {
      const uint4* const from = reinterpret_cast<const uint4*>(chunks + c);
      uint4* const to = reinterpret_cast<uint4*>(&ch);
#pragma unroll
      for (int i = 0; i < int(sizeof(ColChunk) / 16); ++i) to[i] = from[i];
    }
    uint32_t a = act[c];
#pragma unroll
    for (int j = 0; j < COL_BITS; ++j) a &= ((tg >> j) & 1u) ? ~0u : ~ch.need[j];
#pragma unroll
    for (int j = 0; j < GROUP_QUBITS; ++j) par ^= (uint32_t(__popc(a & ch.row[j])) & 1u) << j;
    par ^= (uint32_t(__popc(a & ch.neg)) & 1u) << GROUP_QUBITS;
    if (ch.tgen) {
      cth = cmulf(cth, tph[c]);
      scal = true;
    }
    for (uint32_t gb = a & ch.gen; gb; gb &= gb - 1) {
      cth = cmulf(cth, coef[ch.t0 + (__ffs(gb) - 1)]);
      scal = true;
    }
  }
}
// The sign words of 32 rows: row 8 q + i flips by m8[i] ^ m4[q].
__device__ __forceinline__ void sign_words(uint32_t par, uint32_t (&m8)[8], uint32_t (&m4)[4]) {
  uint32_t m[GROUP_QUBITS + 1];
#pragma unroll
  for (int j = 0; j <= GROUP_QUBITS; ++j) m[j] = (0u - ((par >> j) & 1u)) & 0x80000000u;
#pragma unroll
  for (int i = 0; i < 8; ++i) m8[i] = ((i & 1) ? m[0] : 0u) ^ ((i & 2) ? m[1] : 0u) ^ ((i & 4) ? m[2] : 0u);
#pragma unroll
  for (int q = 0; q < 4; ++q) m4[q] = ((q & 1) ? m[3] : 0u) ^ ((q & 2) ? m[4] : 0u) ^ m[5];
}
// The same for packed pairs of bf16: rows 8 q + 2 i (low half) and the next flip by mp[i] ^ m4[q].
__device__ __forceinline__ void sign_pairs(uint32_t par, uint32_t (&mp)[4], uint32_t (&m4)[4]) {
  uint32_t m[GROUP_QUBITS + 1];
#pragma unroll
  for (int j = 0; j <= GROUP_QUBITS; ++j) m[j] = (0u - ((par >> j) & 1u)) & (j ? 0x80008000u : 0x80000000u);
#pragma unroll
  for (int i = 0; i < 4; ++i) mp[i] = m[0] ^ ((i & 1) ? m[1] : 0u) ^ ((i & 2) ? m[2] : 0u);
#pragma unroll
  for (int q = 0; q < 4; ++q) m4[q] = ((q & 1) ? m[3] : 0u) ^ ((q & 2) ? m[4] : 0u) ^ m[5];
}

__device__ __forceinline__ void bar_group(int g) {
  asm volatile("bar.sync %0, %1;" ::"r"(1 + g), "r"(GROUP_THREADS) : "memory");
}

// NG: the warpgroups that work, and so the tiles in a set (a run-time count made the full kernel 7% slower)
template <uint32_t NG>
__global__ void __launch_bounds__(THREADS, 1) k_fused_pass(const __grid_constant__ PassArgs P) {
  extern __shared__ __align__(16) uint8_t smem_raw[];
  Tables& S = *reinterpret_cast<Tables*>(smem_raw);
  const uint32_t sm0 = smem_u32(smem_raw);
  const uint32_t tiles0 = (sm0 + uint32_t(sizeof(Tables)) + uint32_t(OPERAND_BYTES) + TILE_BYTES - 1) & ~(TILE_BYTES - 1);
  if (tiles0 + SM_END > sm0 + SM_DYNAMIC) {  // every thread alike, before anything is held
    if (threadIdx.x == 0) atomicCAS(P.err, 0, 5);
    return;
  }
  // operand slot 0 ends where the tiles begin, the others follow the tiles
  auto slot_addr = [&](uint32_t s) { return s ? tiles0 + SM_SLOTS + (s - 1) * OPERAND_BYTES : tiles0 - OPERAND_BYTES; };
  float2* const tphase_sh = reinterpret_cast<float2*>(smem_raw + (tiles0 - sm0) + SM_TPHASE);

  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  auto bar_tfull = [&](uint32_t b) { return smem_u32(&S.bars[b]); };
  auto bar_tdone = [&](uint32_t b) { return smem_u32(&S.bars[NTILEBUF + b]); };
  auto bar_ofull = [&](uint32_t s) { return smem_u32(&S.bars[2 * NTILEBUF + s]); };
  auto bar_oempty = [&](uint32_t s) { return smem_u32(&S.bars[2 * NTILEBUF + NOPSLOT + s]); };
  auto bar_mma = [&](int g) { return smem_u32(&S.bars[2 * NTILEBUF + 2 * NOPSLOT + g]); };
  auto fail = [&](int code) {
    S.abort = 1;
    atomicCAS(P.err, 0, code);
  };

  if (tid == 0) {
    for (int i = 0; i < NTILEBUF; ++i) {
      mbar_init(bar_tfull(i), TILE_THREADS + 1);  // one cp.async arrival per tile thread, one for the tile's facts
      mbar_init(bar_tdone(i), GROUP_THREADS / 32);
    }
    for (int i = 0; i < NOPSLOT; ++i) {
      mbar_init(bar_ofull(i), 1);
      mbar_init(bar_oempty(i), NG);  // one commit (or release) per group
    }
    for (int g = 0; g < GROUPS; ++g) mbar_init(bar_mma(g), 1);
    S.abort = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 0) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&S.tmem_base)),
                 "r"(TMEM_COLS));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
  }
  for (uint32_t i = uint32_t(tid); i < uint32_t(sizeof(PassTables) / 16); i += THREADS)
    reinterpret_cast<uint4*>(smem_raw)[i] = __ldg(reinterpret_cast<const uint4*>(P.tables) + i);
  // The next pass's launch and tables overlap this one's end; only the register and the error word pass
  // between them, and nothing above touches those but to report a layout that does not fit.  (n = 21, 7
  // passes: 231 -> 215 us; n = 16, 3 passes: 67 -> 63.)
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  asm volatile("griddepcontrol.wait;" ::: "memory");
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = __shfl_sync(0xffffffffu, S.tmem_base, 0);
  // tiles go in sets of NG, one per warpgroup: tile j of this CTA's set p is tile_of(p, j) and
  // the CTA's it-th, in buffer it % NTILEBUF; only the register's last set of tiles can be short,
  // and it is the last one of the CTA that takes it
  const uint32_t ntiles = P.ntiles;
  const uint32_t nsets = (ntiles + NG - 1) / NG;
  const uint32_t my_sets = nsets > blockIdx.x ? (nsets - 1 - blockIdx.x) / gridDim.x + 1 : 0;
  auto tile_of = [&](uint32_t p, uint32_t j) { return NG * (blockIdx.x + p * gridDim.x) + j; };
  float2* tiles = reinterpret_cast<float2*>(smem_raw + (tiles0 - sm0));
  auto at = [&](uint32_t e) { return e ^ uint32_t(S.swz[e >> 4]); };  // stored position of tile element e
  // byte offset in the register of a tile's 16-byte chunk c < 128; chunks of disjoint bits add
  auto chunk_off = [&](uint32_t c) {
    uint64_t g = 0;
#pragma unroll
    for (int j = 0; j < 7; ++j) g |= uint64_t((c >> j) & 1u) << S.win[j + 1];
    return g * sizeof(float2);
  };

  if (warp >= WARP_TILES && warp != WARP_OPS) {
    // ---------------- tiles in order: their loads (64 threads), their facts (a warp) ----------------
    const bool facts = warp == WARP_FACTS;
    const int pt = tid - COMPUTE_THREADS;
    const uint64_t my_off = chunk_off(uint32_t(pt) & (TILE_THREADS - 1));
    const uint32_t my_at = 8u * at(2u * (uint32_t(pt) & (TILE_THREADS - 1)));  // positions of disjoint bits combine by XOR
    const uint64_t lane_bit = uint64_t(1) << S.out[lane];  // the index bit that bit `lane` of a tile number stands for
    uint32_t b = 0, parity = 1;  // buffer it % NTILEBUF, and the parity of its last use
    for (uint32_t it = 0, p = 0, j = 0; p < my_sets; ++it) {
      const uint32_t t = tile_of(p, j);
      if (t >= ntiles) break;  // the CTA's last tiles
      if (++j == NG) j = 0, ++p;
      if (it >= NTILEBUF) {    // the buffer is free once its last tile is written back; each warp stops by itself
        bool ok = true;
        if (lane == 0) {
          ok = mbar_wait(bar_tdone(b), parity);
          if (!ok) fail(3);
          ok = ok && !S.abort;
        }
        if (!__shfl_sync(0xffffffffu, ok, 0)) break;
      }
      const bool on = (t >> lane) & 1u;
      const uint64_t base = uint64_t(__reduce_or_sync(0xffffffffu, on ? uint32_t(lane_bit >> 32) : 0u)) << 32 |
                            __reduce_or_sync(0xffffffffu, on ? uint32_t(lane_bit) : 0u);
      if (!facts) {
        const uint8_t* const src = reinterpret_cast<const uint8_t*>(P.amp) + base * sizeof(float2) + my_off;
        const uint32_t dst = (tiles0 + b * TILE_BYTES) ^ my_at;
#pragma unroll 8
        for (uint32_t i = 0; i < uint32_t(TILE / 2 / TILE_THREADS); ++i) {
          const uint32_t e = 2u * TILE_THREADS * i;
          cp_async16(dst ^ (8u * (e ^ swz_fold(e))), src + S.chunk_off[i]);
        }
        cp_async_arrive(bar_tfull(b));
      } else {
        // which column terms apply on this tile (their bits outside it)
        for (int c = 0; c < P.nchunks; ++c) {
          const ColChunk& ch = S.chunks[c];
          const uint64_t cm = lane < int(ch.cnt) ? S.terms.cmask[ch.t0 + lane] : 0;
          const bool act = lane < int(ch.cnt) && (base & cm) == cm;
          const uint32_t m = __ballot_sync(0xffffffffu, act);
          if (ch.tgen) {  // the same phase on every column: their product, once
            float2 f = make_float2(1.f, 0.f);
            for (uint32_t gb = m & ch.tgen; gb; gb &= gb - 1) f = cmulf(f, S.terms.coef[ch.t0 + (__ffs(gb) - 1)]);
            if (lane == 0) tphase_sh[b * MAX_CHUNKS + c] = f;
          }
          if (lane == 0) S.act[b][c] = m & ~ch.tgen;
        }
        if (lane == 0) {
          S.base[b] = base;
          mbar_arrive(bar_tfull(b));
        }
      }
      if (++b == NTILEBUF) b = 0, parity ^= 1u;
    }
    // copies of this thread still in flight land before the CTA exits
    asm volatile("cp.async.wait_all;" ::: "memory");
  } else if (warp == WARP_OPS) {
    // ---------------- B operand images: use k = set * nu + u, slot k % NOPSLOT ----------------
    const uint32_t nk = my_sets * uint32_t(P.nu);
    uint32_t k = 0, sl = 0, parity = 1, u = 0;
    for (; k < nk; ++k) {
      if (k >= NOPSLOT) {
        bool go = true;
        if (lane == 0) {
          go = mbar_wait(bar_oempty(sl), parity);
          if (!go) fail(4);
          go = go && !S.abort;
        }
        if (!__shfl_sync(0xffffffffu, go, 0)) break;  // lane 0 decides for the warp
      }
      if (lane == 0) {
        mbar_expect_tx(bar_ofull(sl), OPERAND_BYTES);
        bulk_load(slot_addr(sl), P.rops + u * (OPERAND_BYTES / 16), OPERAND_BYTES, bar_ofull(sl));
      }
      __syncwarp();
      if (++u == uint32_t(P.nu)) u = 0;
      if (++sl == NOPSLOT) sl = 0, parity ^= 1u;
    }
    if (k < nk)  // an abort: let the loads already issued land
      for (uint32_t j = k >= NOPSLOT ? k - NOPSLOT : 0; j < k; ++j)
        if (lane == 0) mbar_wait(bar_ofull(j % NOPSLOT), (j / NOPSLOT) & 1);
  } else {
    // ---------------- tensor-core program: group g on its tile of each set ----------------
    const int g = warp / 4, tg = tid & (GROUP_THREADS - 1);
    const uint32_t lane_base = uint32_t((warp & 3) * 32) << 16;
    const uint32_t taddr = tmem + uint32_t(128 * g) + lane_base;  // this warp's lanes: D [0,64), A hi [64,96), A lo [96,128)
    const uint32_t taddr_a = taddr + 64u;
    // the group's first warp issues its MMAs; warp-uniform operands
    const int gu = __shfl_sync(0xffffffffu, g, 0);
    const uint32_t idesc = (1u << 4) | (1u << 7) | (1u << 10) | ((64u >> 3) << 17) | ((128u >> 4) << 24);
    const uint32_t d_tmem = tmem + uint32_t(128 * gu), a_tmem = d_tmem + 64u;
    uint32_t sl = 0, sl_phase = 0;  // the next use's operand slot
    uint32_t mma_phase = 0;
    const uint64_t my_off = chunk_off(uint32_t(tg));
    const uint32_t my_at = 8u * at(2u * uint32_t(tg));
    uint32_t b = uint32_t(g), parity = 0;  // buffer of this group's tile, and the parity of its use
    for (uint32_t p = 0; p < my_sets && uint32_t(g) < NG; ++p) {
      if (tile_of(p, uint32_t(g)) >= ntiles) {  // no tile in the last set: release its operand slots unused
        if (tg == 0)
          for (int u = 0; u < P.nu && !S.abort; ++u) {
            if (!mbar_wait(bar_ofull(sl), sl_phase)) fail(2);
            mbar_arrive(bar_oempty(sl));
            if (++sl == NOPSLOT) sl = 0, sl_phase ^= 1u;
          }
        break;
      }
      if (!mbar_wait(bar_tfull(b), parity)) fail(1);
      const uint64_t base = S.base[b];
      float2* T = tiles + size_t(b) * TILE;
      const uint32_t* const act = S.act[b];
      const float2* const tph = tphase_sh + b * MAX_CHUNKS;
      bool stop = false;
      for (int oi = 0; oi < P.nops; ++oi) {
        const uint4 opw = *reinterpret_cast<const uint4*>(&S.ops[oi]);
        OpDesc op;
        *reinterpret_cast<uint4*>(&op) = opw;
        if (op.kind == 1) {
          // ---- diagonal terms: per-tile tables, then one sweep of the tile ----
          build_tables(op, base, tg, S.terms, S.tab_lo[g], S.tab_hi[g], S.tab_cross[g]);
          bar_group(g);
          {
            // element e = tg + 128 i: its low 6 bits are the thread's, so the low-half
            // phase is one read; the high-half entries are the same across a warp
            const uint32_t lo = uint32_t(tg) & ((1u << HALF) - 1);
            const float2 L = S.tab_lo[g][lo];
            if (op.tc == op.t1) {
              // blocks of 8: every load before any store (the tile and the tables may alias as far
              // as the compiler knows, so a store would hold back the next loads)
              const float2* __restrict__ th = S.tab_hi[g];
              const uint8_t* __restrict__ tx = S.tab_cross[g];
#pragma unroll 1
              for (int i0 = 0; i0 < TILE / GROUP_THREADS; i0 += 8) {
                float2 v[8], h[8];
                uint32_t x[8];
#pragma unroll
                for (int j = 0; j < 8; ++j) {
                  const uint32_t e = uint32_t(tg + GROUP_THREADS * (i0 + j)), hi = e >> HALF;
                  v[j] = T[at(e)];
                  h[j] = th[hi];
                  x[j] = tx[hi];
                }
#pragma unroll
                for (int j = 0; j < 8; ++j) {
                  float2 c = cmulf(L, h[j]);
                  const uint32_t sg = uint32_t(__popc(lo & x[j]) & 1) << 31;
                  c = make_float2(__uint_as_float(__float_as_uint(c.x) ^ sg), __uint_as_float(__float_as_uint(c.y) ^ sg));
                  T[at(uint32_t(tg + GROUP_THREADS * (i0 + j)))] = cmulf(c, v[j]);
                }
              }
            } else {
#pragma unroll 4
              for (int i = 0; i < TILE / GROUP_THREADS; ++i) {
                const uint32_t e = uint32_t(tg + GROUP_THREADS * i);
                T[at(e)] = cmulf(term_phase(e, op, base, S.terms, S.tab_lo[g], S.tab_hi[g], S.tab_cross[g]), T[at(e)]);
              }
            }
          }
          bar_group(g);
          continue;
        }
        // ---- unitary op: this thread owns column tg (A row / TMEM lane) and its 32 rows ----
        const int u = op.u;
        // stored positions (the layout fold is linear: column and row parts combine by XOR)
        const uint32_t cb = (tiles0 + b * TILE_BYTES) ^ uint32_t(S.clo[u][tg & 15]) ^ uint32_t(S.chi[u][tg >> 4]);
        const uint4 gb = *reinterpret_cast<const uint4*>(S.gbit[u]);
        const uint32_t p0 = gb.x & 0xffffu, p1 = gb.x >> 16, p2 = gb.y & 0xffffu, p3 = gb.y >> 16, p4 = gb.z & 0xffffu;
        uint32_t lo8[8];  // rows 0..7 (gate bits 0-2) of this column
#pragma unroll
        for (int i = 0; i < 8; ++i) lo8[i] = cb ^ ((i & 1) ? p0 : 0u) ^ ((i & 2) ? p1 : 0u) ^ ((i & 4) ? p2 : 0u);
        const uint32_t hi4[4] = {0u, p3, p4, p3 ^ p4};  // rows 8q..8q+7
        // a preceding diagonal op, reduced to this column: a sign per row and a phase of the column
        uint32_t par = 0;
        float2 cth = make_float2(1.f, 0.f);
        bool scal = false;
        column_chunks(S.chunks, act, tph, op.pc0, op.pc1, uint32_t(tg), S.terms.coef, par, cth, scal);
        // warp-uniform decisions (a lane without a phase multiplies by exactly 1, one without
        // signs flips nothing), so the unrolled loops carry no divergent branches
        scal = __any_sync(0xffffffffu, scal);
        const bool flip = __any_sync(0xffffffffu, par != 0);
        // the previous op's stores are in, and everyone stops alike
        stop = bar_any(1 + g, GROUP_THREADS, S.abort);
        if (stop) break;
        // A row (this lane): K = row (real parts) and 32 + row (imaginary parts), two bf16 per
        // column, so rows 8q .. 8q+7 are columns 4q .. 4q+3 (re) and 16 + the same (im).  One loop
        // per kind: in one loop, results kept in place past a branch cost a register copy each.
        if (scal) {
          uint32_t mp[4], m4[4];
          sign_pairs(par, mp, m4);
#pragma unroll
          for (int q = 0; q < 4; ++q) {
            float x[8], y[8];  // rows 8q..8q+7, loaded before any other work
#pragma unroll
            for (int i = 0; i < 8; ++i) lds_amp(lo8[i] ^ hi4[q], x[i], y[i]);
#pragma unroll
            for (int i = 0; i < 8; ++i) {
              const float2 c = cmulf(cth, make_float2(x[i], y[i]));
              x[i] = c.x;
              y[i] = c.y;
            }
            uint32_t hr[4], lr[4], hm[4], lm[4];
#pragma unroll
            for (int i = 0; i < 4; ++i) {
              const uint32_t wr = pack_bf16(x[2 * i], x[2 * i + 1]), wm = pack_bf16(y[2 * i], y[2 * i + 1]);
              hr[i] = wr ^ mp[i] ^ m4[q];
              hm[i] = wm ^ mp[i] ^ m4[q];
              lr[i] = pack_neg_residual(wr, x[2 * i], x[2 * i + 1]) ^ mp[i] ^ m4[q];
              lm[i] = pack_neg_residual(wm, y[2 * i], y[2 * i + 1]) ^ mp[i] ^ m4[q];
            }
            tmem_st4(taddr_a + uint32_t(4 * q), hr);
            tmem_st4(taddr_a + uint32_t(16 + 4 * q), hm);
            tmem_st4(taddr_a + uint32_t(32 + 4 * q), lr);
            tmem_st4(taddr_a + uint32_t(48 + 4 * q), lm);
          }
        } else if (flip) {
          uint32_t mp[4], m4[4];
          sign_pairs(par, mp, m4);
#pragma unroll
          for (int q = 0; q < 4; ++q) {
            float x[8], y[8];  // rows 8q..8q+7, loaded before any other work
#pragma unroll
            for (int i = 0; i < 8; ++i) lds_amp(lo8[i] ^ hi4[q], x[i], y[i]);
            uint32_t hr[4], lr[4], hm[4], lm[4];
#pragma unroll
            for (int i = 0; i < 4; ++i) {
              const uint32_t wr = pack_bf16(x[2 * i], x[2 * i + 1]), wm = pack_bf16(y[2 * i], y[2 * i + 1]);
              hr[i] = wr ^ mp[i] ^ m4[q];
              hm[i] = wm ^ mp[i] ^ m4[q];
              lr[i] = pack_neg_residual(wr, x[2 * i], x[2 * i + 1]) ^ mp[i] ^ m4[q];
              lm[i] = pack_neg_residual(wm, y[2 * i], y[2 * i + 1]) ^ mp[i] ^ m4[q];
            }
            tmem_st4(taddr_a + uint32_t(4 * q), hr);
            tmem_st4(taddr_a + uint32_t(16 + 4 * q), hm);
            tmem_st4(taddr_a + uint32_t(32 + 4 * q), lr);
            tmem_st4(taddr_a + uint32_t(48 + 4 * q), lm);
          }
        } else {
#pragma unroll
          for (int q = 0; q < 4; ++q) {
            float x[8], y[8];  // rows 8q..8q+7, loaded before any other work
#pragma unroll
            for (int i = 0; i < 8; ++i) lds_amp(lo8[i] ^ hi4[q], x[i], y[i]);
            uint32_t hr[4], lr[4], hm[4], lm[4];
#pragma unroll
            for (int i = 0; i < 4; ++i) {
              hr[i] = pack_bf16(x[2 * i], x[2 * i + 1]);
              hm[i] = pack_bf16(y[2 * i], y[2 * i + 1]);
              lr[i] = pack_neg_residual(hr[i], x[2 * i], x[2 * i + 1]);
              lm[i] = pack_neg_residual(hm[i], y[2 * i], y[2 * i + 1]);
            }
            tmem_st4(taddr_a + uint32_t(4 * q), hr);
            tmem_st4(taddr_a + uint32_t(16 + 4 * q), hm);
            tmem_st4(taddr_a + uint32_t(32 + 4 * q), lr);
            tmem_st4(taddr_a + uint32_t(48 + 4 * q), lm);
          }
        }
        asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
        tc_fence_before();
        bar_group(g);
        if ((warp & 3) == 0) {
          // all four warps' splits are in TMEM, the operand is in its slot (on a timeout the
          // MMAs read stale operands and the group stops at its next barrier)
          if (!mbar_wait(bar_ofull(sl), sl_phase)) fail(2);
          __syncwarp();
          tc_fence_after();
          const uint32_t slu = __shfl_sync(0xffffffffu, sl, 0);
          const uint32_t b_hi = slot_addr(slu);
          const uint64_t dbh = sw128_desc(b_hi), dbl = sw128_desc(b_hi + OPERAND_BYTES / 2);
          if (elect_one()) {  // K = 16 per MMA: eight A columns, two 16-byte steps of B
#pragma unroll
            for (int s = 0; s < 4; ++s) mma_bf16_ta(d_tmem, a_tmem + 8u * s, dbh + 2 * s, idesc, s > 0);
#pragma unroll
            for (int s = 0; s < 4; ++s) mma_bf16_ta(d_tmem, a_tmem + 32u + 8u * s, dbh + 2 * s, idesc | NEGATE_A, 1);
#pragma unroll
            for (int s = 0; s < 4; ++s) mma_bf16_ta(d_tmem, a_tmem + 8u * s, dbl + 2 * s, idesc, 1);
            mma_commit(bar_mma(gu));
            mma_commit(bar_oempty(slu));  // the slot is free once these MMAs have read it
          }
          __syncwarp();
        }
        if (++sl == NOPSLOT) sl = 0, sl_phase ^= 1u;
        // a following diagonal op, reduced to this column (computed while the MMAs run)
        uint32_t par2 = 0;
        cth = make_float2(1.f, 0.f);
        scal = false;
        column_chunks(S.chunks, act, tph, op.qc0, op.qc1, uint32_t(tg), S.terms.coef, par2, cth, scal);
        scal = __any_sync(0xffffffffu, scal);
        const bool flip2 = __any_sync(0xffffffffu, par2 != 0);
        // every thread waits for the accumulator itself (no group barrier: each warp reads its
        // lanes back as soon as the MMAs land).  A phase cannot be skipped: the next one needs
        // every warp's split after this read-back.  On a timeout the read-back reads stale
        // columns and the group stops at its next barrier.
        if (!mbar_wait(bar_mma(g), mma_phase)) fail(2);
        mma_phase ^= 1u;
        tc_fence_after();
        // D columns 16h .. 16h+15 hold rows 8h .. 8h+7 as (real, imaginary) pairs.  Two loops: in one,
        // results kept in place past a branch cost a register copy each (72 an op).
        if (!scal && !flip2) {
#pragma unroll
          for (int h = 0; h < 4; ++h) {
            uint32_t v[16];
            NCSIM_TMEM_LD16(taddr + uint32_t(16 * h), v);
            asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
            for (int i = 0; i < 8; ++i) sts_amp(lo8[i] ^ hi4[h], v[2 * i], v[2 * i + 1]);
          }
        } else {
          uint32_t m8[8], m4[4];
          sign_words(par2, m8, m4);
#pragma unroll
          for (int h = 0; h < 4; ++h) {
            uint32_t v[16];
            NCSIM_TMEM_LD16(taddr + uint32_t(16 * h), v);
            asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
            for (int i = 0; i < 8; ++i) {
              const float2 c = cmulf(cth, make_float2(__uint_as_float(v[2 * i]), __uint_as_float(v[2 * i + 1])));
              sts_amp(lo8[i] ^ hi4[h], __float_as_uint(c.x) ^ m8[i] ^ m4[h], __float_as_uint(c.y) ^ m8[i] ^ m4[h]);
            }
          }
        }
        tc_fence_before();
      }
      if (stop || bar_any(1 + g, GROUP_THREADS, S.abort)) break;
      // the group writes its tile back; each thread's shared-memory reads are done once its
      // stores are issued, so the buffer is free for the next load after every warp arrives
      uint8_t* const dst = reinterpret_cast<uint8_t*>(P.amp) + base * sizeof(float2) + my_off;
      const uint32_t src = (tiles0 + b * TILE_BYTES) ^ my_at;
#pragma unroll
      for (uint32_t i = 0; i < uint32_t(TILE / 2 / GROUP_THREADS); ++i) {
        const uint32_t e = 2u * GROUP_THREADS * i;
        float4 v;
        asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];"
                     : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w)
                     : "r"(src ^ (8u * (e ^ swz_fold(e)))));
        *reinterpret_cast<float4*>(dst + S.chunk_off[GROUP_THREADS / TILE_THREADS * i]) = v;
      }
      __syncwarp();
      if (lane == 0) mbar_arrive(bar_tdone(b));
      b += NG;
      if (b >= NTILEBUF) b -= NTILEBUF, parity ^= 1u;
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 0) {
    tc_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(TMEM_COLS));
  }
}

// ---------------------------------------------------------------------------
// device copy of a plan: every pass's operand images in one buffer
struct DevicePlan {
  Plan plan;
  std::vector<PassArgs> args;  // per pass, in segment order (amp/err filled per run)
  uint8_t* images = nullptr;   // the operands, then the passes' tables
  int device = -1;
  // The images come from the library's pool: cudaMalloc mapped memory anew for plans that its own chunks had no room
  // for, and cudaFree gave it back (a new circuit's first run at n = 16, depth 12, 2.25 ms, from the pool 1.46).  A
  // run waits for its passes before it lets go of the plan, so nothing reads the images any more.
  ~DevicePlan() {
    if (!images) return;
    int cur = 0;
    cudaGetDevice(&cur);
    if (cur != device) cudaSetDevice(device);
    cudaFreeAsync(images, cudaStreamLegacy);
    if (cur != device) cudaSetDevice(cur);
  }
};

// which device table a term goes to (tile-local mask tm over the two 6-bit halves)
TermClass term_class(uint32_t tm, const CplxD& c) {
  const uint32_t lo = tm & ((1u << HALF) - 1), hi = tm >> HALF;
  if (hi == 0) return T_LOW;
  if (lo == 0) return T_HIGH;
  if (__builtin_popcount(lo) == 1 && __builtin_popcount(hi) == 1 && c.re == -1.0 && c.im == 0.0) return T_CROSS_SIGN;
  return T_GENERIC;
}

// The order of a unitary's column bits.  A warp access moves its amplitudes 16 lanes (8 bytes each)
// at a time, and each lane's bank is linear in the tile bits (a low bit's own, a higher bit's fold):
// there are no conflicts when the four lowest column bits have independent banks.  They are picked
// greedily, the rest follow.  Over the layered circuits' plans (195 unitaries) a warp access takes
// 2.35 wavefronts instead of 2.46 with the bits in ascending order; 2 is the minimum, and the
// unitaries on tile bit 0, whose bank no other bit reaches, take 4.
void column_order(const uint8_t (&pos)[GROUP_QUBITS], uint8_t (&col)[COL_BITS]) {
  uint32_t gm = 0;
  for (uint8_t p : pos) gm |= 1u << p;
  uint32_t span = 1;     // bank vectors (4 bits) reachable by the picked bits, as a set
  uint32_t picked = 0;
  int m = 0;
  for (int b = 0; b < TILE_BITS && m < 4; ++b) {
    if ((gm >> b) & 1) continue;
    const uint32_t v = (b < 4 ? 1u << b : swz_fold(1u << b)) & 15u;
    if ((span >> v) & 1) continue;
    uint32_t next = span;
    for (uint32_t x = 0; x < 16; ++x)
      if ((span >> x) & 1) next |= 1u << (x ^ v);
    span = next;
    picked |= 1u << b;
    col[m++] = uint8_t(b);
  }
  for (int b = 0; b < TILE_BITS; ++b)
    if (!(((gm | picked) >> b) & 1)) col[m++] = uint8_t(b);
}

PassTables build_tables(const PassProgram& P, const std::vector<uint32_t>& window) {
  PassTables T{};
  std::copy(P.chunks, P.chunks + P.nchunks, T.chunks);
  std::copy(P.ops, P.ops + P.nops, T.ops);
  for (int i = 0; i < P.nterms; ++i) {
    T.terms.cmask[i] = P.terms[i].cmask;
    T.terms.coef[i] = make_float2(P.terms[i].cr, P.terms[i].ci);
    T.terms.tmask[i] = uint16_t(P.terms[i].tmask);
  }
  auto stored = [](uint32_t e) { return uint16_t((e ^ swz_fold(e)) * sizeof(float2)); };
  for (int u = 0; u < P.nu; ++u) {
    auto column = [&](uint32_t k) {
      uint32_t e = 0;
      for (int m = 0; m < COL_BITS; ++m) e |= ((k >> m) & 1u) << P.col[u][m];
      return stored(e);
    };
    for (uint32_t k = 0; k < 16; ++k) T.clo[u][k] = column(k);
    for (uint32_t k = 0; k < 8; ++k) T.chi[u][k] = column(k << 4);
    for (int j = 0; j < GROUP_QUBITS; ++j) T.gbit[u][j] = stored(1u << P.pos[u][j]);
  }
  for (uint32_t i = 0; i < uint32_t(TILE / 2 / TILE_THREADS); ++i) {
    const uint32_t e = 2u * TILE_THREADS * i;
    for (int j = 0; j < TILE_BITS; ++j) T.chunk_off[i] |= (uint64_t((e >> j) & 1u) << window[j]) * sizeof(float2);
  }
  for (uint32_t h = 0; h < (1u << (TILE_BITS - 4)); ++h) T.swz[h] = uint8_t(swz_fold(h << 4));
  for (int j = 0; j < TILE_BITS; ++j) T.win[j] = uint8_t(window[j]);
  for (uint32_t q = 0, j = 0, m = 0; m < 32; ++q) {  // the index bits outside the window
    if (j < uint32_t(TILE_BITS) && window[j] == q) ++j;
    else T.out[m++] = uint8_t(q);
  }
  return T;
}

std::unique_ptr<DevicePlan> build_device_plan(const ncsim_circuit& c, uint32_t max_fuse, cudaStream_t stream) {
  auto dp = std::make_unique<DevicePlan>();
  dp->plan = make_plan(c, max_fuse);
  std::vector<uint8_t> images;
  std::vector<size_t> offsets;
  std::vector<PassTables> tables;
  for (const Segment& s : dp->plan.segments) {
    if (!s.fused) continue;
    for (const Pass& ps : s.passes) {
      PassProgram P{};
      uint64_t wmask = 0;
      for (int j = 0; j < TILE_BITS; ++j) wmask |= uint64_t(1) << ps.window[j];
      int wl = 0;
      while (wl < TILE_BITS && ps.window[wl] == uint32_t(wl)) ++wl;
      if (wl < LOW_BITS) throw Error(NCSIM_ERR_INVALID, "fused pass window lacks the low index bits");
      int nu = 0, nt = 0, no = 0;
      for (const FusedOp& op : ps.ops) {
        OpDesc d{};
        if (op.kind == 0) {
          if (nu >= MAX_UNITARIES) throw Error(NCSIM_ERR_INVALID, "fused pass has too many unitaries");
          d.kind = 0;
          d.u = uint8_t(nu);
          for (int j = 0; j < GROUP_QUBITS; ++j) {
            auto it = std::find(ps.window.begin(), ps.window.end(), op.qubits[j]);
            if (it == ps.window.end()) throw Error(NCSIM_ERR_INVALID, "fused unitary outside its window");
            P.pos[nu][j] = uint8_t(it - ps.window.begin());
          }
          column_order(P.pos[nu], P.col[nu]);
          const size_t at = images.size();
          images.resize(at + OPERAND_BYTES);
          build_operand_image(op.u, images.data() + at);
          offsets.push_back(at);
          ++nu;
        } else {
          d.kind = 1;
          if (nt + int(op.terms.size()) > MAX_TERMS) throw Error(NCSIM_ERR_INVALID, "fused pass has too many terms");
          std::vector<std::pair<int, TermDesc>> ts;
          for (const Term& t : op.terms) {
            TermDesc td{};
            uint32_t tm = 0;
            for (int j = 0; j < TILE_BITS; ++j)
              if ((t.mask >> ps.window[j]) & 1) tm |= 1u << j;
            td.tmask = tm;
            td.cmask = t.mask & ~wmask;
            td.cr = float(t.c.re);
            td.ci = float(t.c.im);
            ts.push_back({int(term_class(tm, t.c)), td});
          }
          std::stable_sort(ts.begin(), ts.end(), [](const auto& a, const auto& b) { return a.first < b.first; });
          uint16_t bound[5];  // start of each class, then the end
          bound[0] = uint16_t(nt);
          int cls = 0;
          for (const auto& e : ts) {
            while (cls < e.first) bound[++cls] = uint16_t(nt);
            P.terms[nt++] = e.second;
          }
          while (cls < 4) bound[++cls] = uint16_t(nt);
          d.t0 = bound[0];
          d.tl = bound[1];
          d.th = bound[2];
          d.tc = bound[3];
          d.t1 = bound[4];
        }
        if (no >= MAX_OPS) throw Error(NCSIM_ERR_INVALID, "fused pass has too many ops");
        P.ops[no++] = d;
      }
      P.nops = no;
      P.nu = nu;
      // A terms op right before a unitary whose terms are, relative to that unitary's five
      // qubits, phases of the other bits or signs on one of its qubits is applied while the
      // unitary splits the tile (kind 2); one left after a unitary, by its read-back (kind 3).
      // Their terms go to the device as chunks of bit masks over 32 terms.
      int nch = 0;
      auto fold = [&](OpDesc& t, OpDesc& un, uint8_t kind) -> bool {
        uint32_t gm = 0;
        for (int j = 0; j < GROUP_QUBITS; ++j) gm |= 1u << P.pos[un.u][j];
        for (int k = t.t0; k < t.t1; ++k) {
          const TermDesc& td = P.terms[k];
          const uint32_t gpart = td.tmask & gm;
          if (!(gpart == 0 || (__builtin_popcount(gpart) == 1 && td.cr == -1.0f && td.ci == 0.0f))) return false;
        }
        const int need = (t.t1 - t.t0 + 31) / 32;
        if (nch + need > MAX_CHUNKS) return false;
        int colbit[TILE_BITS];  // tile bit -> column bit of this unitary (-1: a gate bit)
        for (int& cb : colbit) cb = -1;
        for (int m = 0; m < COL_BITS; ++m) colbit[P.col[un.u][m]] = m;
        const uint8_t c0 = uint8_t(nch);
        for (int k0 = t.t0; k0 < t.t1; k0 += 32) {
          ColChunk ch{};
          ch.t0 = uint16_t(k0);
          ch.cnt = uint16_t(std::min(32, t.t1 - k0));
          for (int i = 0; i < ch.cnt; ++i) {
            TermDesc& td = P.terms[k0 + i];
            const uint32_t bit = 1u << i;
            const uint32_t gpart = td.tmask & gm;
            bool rows = false;
            for (int j = 0; j < GROUP_QUBITS; ++j)
              if (gpart == (1u << P.pos[un.u][j])) rows = true, ch.row[j] |= bit;
            td.tmask &= ~gm;
            for (int b = 0; b < TILE_BITS; ++b)
              if ((td.tmask >> b) & 1) ch.need[colbit[b]] |= bit;
            if (!rows) {
              if (td.cr == -1.0f && td.ci == 0.0f) ch.neg |= bit;
              else if (td.tmask == 0 && k0 == t.t0 && !ch.gen) ch.tgen |= bit;
              else ch.gen |= bit;
            }
          }
          P.chunks[nch++] = ch;
        }
        t.kind = kind;
        if (kind == 2) un.pc0 = c0, un.pc1 = uint8_t(nch);
        else un.qc0 = c0, un.qc1 = uint8_t(nch);
        return true;
      };
      for (int i = 0; i + 1 < no; ++i)
        if (P.ops[i].kind == 1 && P.ops[i + 1].kind == 0) fold(P.ops[i], P.ops[i + 1], 2);
      for (int i = 1; i < no; ++i)
        if (P.ops[i].kind == 1 && P.ops[i - 1].kind == 0) fold(P.ops[i], P.ops[i - 1], 3);
      P.nchunks = nch;
      P.nterms = nt;
      P.nops = int(std::remove_if(P.ops, P.ops + no, [](const OpDesc& d) { return d.kind >= 2; }) - P.ops);
      tables.push_back(build_tables(P, ps.window));
      PassArgs a{};
      a.ntiles = uint32_t((uint64_t(1) << c.n) >> TILE_BITS);
      a.nops = P.nops;
      a.nu = P.nu;
      a.nchunks = P.nchunks;
      // the pass's first operand: an offset for now, a device pointer below
      a.rops = reinterpret_cast<const uint4*>(uintptr_t(nu ? offsets[offsets.size() - nu] : 0));
      dp->args.push_back(a);
    }
  }
  const size_t at = images.size();
  images.resize(at + tables.size() * sizeof(PassTables));
  if (!images.empty()) {
    if (!tables.empty()) std::memcpy(images.data() + at, tables.data(), tables.size() * sizeof(PassTables));
    NCSIM_CUDA(cudaGetDevice(&dp->device));
    NCSIM_CUDA(pool_alloc(&dp->images, images.size(), stream));
    // on the state's stream, waited for: a pageable cudaMemcpy may return before its DMA lands,
    // and the pass kernels' non-blocking stream does not wait for the legacy stream
    NCSIM_CUDA(cudaMemcpyAsync(dp->images, images.data(), images.size(), cudaMemcpyHostToDevice, stream));
    NCSIM_CUDA(cudaStreamSynchronize(stream));
  }
  for (size_t i = 0; i < dp->args.size(); ++i) {
    dp->args[i].rops = reinterpret_cast<const uint4*>(dp->images + uintptr_t(dp->args[i].rops));
    dp->args[i].tables = reinterpret_cast<const PassTables*>(dp->images + at) + i;
  }
  NCSIM_CUDA(cudaGetDevice(&dp->device));
  return dp;
}

}  // namespace

}  // namespace fused

int apply_op(ncsim_state* s, const OpIR& op, ncsim_rng& rng);

}  // namespace ncsim

using namespace ncsim;

namespace {
std::mutex g_fused_mu;

// the circuit's device plan for this device and fusion width (built once)
std::shared_ptr<fused::DevicePlan> device_plan_for(const ncsim_circuit* c, uint32_t max_fuse, cudaStream_t stream) {
  std::lock_guard<std::mutex> lk(g_fused_mu);
  int dev = 0;
  NCSIM_CUDA(cudaGetDevice(&dev));
  if (c->fused_plan && c->fused_plan_fuse == max_fuse && c->fused_plan_device == dev)
    return std::static_pointer_cast<fused::DevicePlan>(c->fused_plan);
  std::shared_ptr<fused::DevicePlan> dp(fused::build_device_plan(*c, max_fuse, stream).release());
  c->fused_plan = dp;
  c->fused_plan_fuse = max_fuse;
  c->fused_plan_device = dev;
  return dp;
}
}  // namespace

extern "C" ncsim_status ncsim_sv_run_fused(ncsim_state* s, const ncsim_circuit* c, ncsim_rng* rng, uint32_t max_fuse,
                                           uint8_t* rec, size_t cap, size_t* len, ncsim_fused_stats* stats) {
  return guarded([&] {
    if (!s || !c || !rng) throw Error(NCSIM_ERR_INVALID, "null argument");
    if (s->precision != NCSIM_C64) throw Error(NCSIM_ERR_INVALID, "the fused form runs on complex64 states");
    if (c->n != s->n) throw Error(NCSIM_ERR_INVALID, "circuit on a different register");
    if (c->num_measurements() > cap) throw Error(NCSIM_ERR_INVALID, "record buffer too small");
    if (c->num_measurements()) {
      if (!rec) throw Error(NCSIM_ERR_INVALID, "record is null");
    }
    std::lock_guard<std::recursive_mutex> lk(s->mu);
    std::shared_ptr<fused::DevicePlan> dp = device_plan_for(c, max_fuse ? max_fuse : 5, s->stream);
    struct Passes {  // those launched before an op that is refused still read the plan
      cudaStream_t st;
      bool waited = false;
      ~Passes() {
        if (!waited) cudaStreamSynchronize(st);
      }
    } passes{s->stream};
    int* d_err = s->dev_flag;  // the state's own word: no allocation per run
    NCSIM_CUDA(cudaMemsetAsync(d_err, 0, sizeof(int), s->stream));
    // A tile per warpgroup; a register of fewer tiles than four per SM spreads them first, since
    // groups of one CTA share its tensor core and shared memory: n = 16
    // 94 -> 69 us, n = 19 109 -> 80, n = 20 120 -> 97 against four tiles to a CTA.
    const uint64_t ntiles = s->len >> fused::TILE_BITS, sms = uint64_t(sm_count());
    const uint64_t groups = ntiles <= sms ? 1 : ntiles <= 2 * sms ? 2 : fused::GROUPS;
    const unsigned grid = unsigned(std::min<uint64_t>(sms, (ntiles + groups - 1) / groups));
    const auto kernel = groups == 1 ? fused::k_fused_pass<1> : groups == 2 ? fused::k_fused_pass<2> : fused::k_fused_pass<4>;
    NCSIM_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, fused::SM_DYNAMIC));
    size_t m = 0, pi = 0;
    uint64_t gemm = 0;
    for (const fused::Segment& seg : dp->plan.segments) {
      if (!seg.fused) {
        int r = apply_op(s, c->ops[seg.op], *rng);
        if (r >= 0) rec[m++] = uint8_t(r);
        continue;
      }
      for (size_t k = 0; k < seg.passes.size(); ++k, ++pi) {
        fused::PassArgs P = dp->args[pi];
        P.amp = reinterpret_cast<float2*>(s->amp);
        P.err = d_err;
        ++gemm;  // one pass kernel launch
        ProfScope ps(s, K_FUSED_GEMM, 2.0 * double(s->bytes()));
        cudaLaunchAttribute overlap{};
        overlap.id = cudaLaunchAttributeProgrammaticStreamSerialization;
        overlap.val.programmaticStreamSerializationAllowed = 1;
        cudaLaunchConfig_t launch{};
        launch.gridDim = dim3(grid);
        launch.blockDim = dim3(fused::THREADS);
        launch.dynamicSmemBytes = fused::SM_DYNAMIC;
        launch.stream = s->stream;
        launch.attrs = &overlap;
        launch.numAttrs = k > 0 ? 1 : 0;  // the first pass of a segment follows other kernels
        NCSIM_CUDA(cudaLaunchKernelEx(&launch, kernel, P));
        NCSIM_LAUNCHED("fused pass");
      }
    }
    int h_err = 0;
    NCSIM_CUDA(cudaMemcpyAsync(&h_err, d_err, sizeof(int), cudaMemcpyDeviceToHost, s->stream));
    NCSIM_CUDA(cudaStreamSynchronize(s->stream));
    passes.waited = true;
    if (h_err) throw Error(NCSIM_ERR_DEVICE, "fused pass stopped: a bounded wait timed out (code " + std::to_string(h_err) + ")");
    if (len) *len = m;
    if (stats) {
      stats->source_gates = dp->plan.source_gates;
      stats->fused_unitaries = dp->plan.unitaries;
      stats->passes = dp->plan.passes;
      stats->remap_passes = 0;
      stats->gemm_launches = gemm;
      stats->diagonal_terms = dp->plan.terms;
    }
  });
}

extern "C" ncsim_status ncsim_fused_emulate(const ncsim_circuit* c, uint32_t max_fuse, double* amps, uint64_t len,
                                            ncsim_fused_stats* stats) {
  return guarded([&] {
    if (!c) throw Error(NCSIM_ERR_INVALID, "null circuit");
    fused::Plan p = fused::make_plan(*c, max_fuse ? max_fuse : 5);
    if (amps) {  // without amplitudes: the plan's statistics only
      if (c->n > 22) throw Error(NCSIM_ERR_UNSUPPORTED, "emulation is for registers of at most 22 qubits");
      if (len != (uint64_t(1) << c->n)) throw Error(NCSIM_ERR_INVALID, "amplitude buffer length differs from 2^n");
      std::vector<CplxD> a(len);
      for (uint64_t i = 0; i < len; ++i) a[i] = {amps[2 * i], amps[2 * i + 1]};
      fused::emulate(p, *c, a);
      for (uint64_t i = 0; i < len; ++i) amps[2 * i] = a[i].re, amps[2 * i + 1] = a[i].im;
    }
    if (stats) {
      stats->source_gates = p.source_gates;
      stats->fused_unitaries = p.unitaries;
      stats->passes = p.passes;
      stats->remap_passes = 0;
      stats->gemm_launches = p.passes;
      stats->diagonal_terms = p.terms;
    }
  });
}
