// A run of one-to-one ops of the sparse form in one kernel launch.
//
// Layout.  A warp owns 32 entries and holds their keys transposed: word q (32 bits,
// in shared memory) has qubit q of entry e at bit e.  An op on a few qubits is then a
// few word operations for all 32 entries: CX is one XOR, CCX an AND and a XOR, an
// affine map (MONOMIAL, SWAP) a XOR of words per row, one row per lane.  Phases that
// are fractions of a turn by a power of two are not multiplied op by op: every lane
// counts the turns of the terms that it evaluates in bit planes over the 32 entries
// (a diagonal of 40 terms is two rounds of 32 lanes), and at the end of the run the
// lanes' planes are added and each amplitude is multiplied once.  So a run rounds
// once where its ops one by one would round at each of them.  What has no such
// form (arbitrary phase tables, permutation tables that are not affine) is looked up
// per entry and its new bits balloted back into words.
//
// What bounds it: the chain of the run's dependent ops (shared-memory latency, about
// 60 cycles an op) when the entries are few, instruction issue when they are many.
// One thread per entry walking the ops on keys in registers or shared memory took
// 2.08 ms for the 2000 gates of the n = 31 reversible family on 65 536 entries (1000
// instructions a warp for a 40-term diagonal) and 0.59 ms for the n = 1000 ripple.
#include "sparse_run.hpp"

#include <cstring>
#include <type_traits>

#include "sparse_common.cuh"

namespace {

// ops: 16-byte heads (type | length in 16-byte units << 16, three words), then data
enum : uint32_t {
  OP_END,     // end of a chunk
  OP_NOTS,    // y controlled NOTs, one word each: w[bits 0..9] ^= w[bits 10..19] & w[bits 20..29]; bit 30: an exchange
              // of the first two words instead
  OP_FLIP,    // complements y words: 16-bit list
  OP_TERMS,   // y terms: (three 10-bit qubits, coefficient in 1/256 turns)
  OP_AFFINE,  // y qubits, shift z: 16-bit lists of 10 qubits and 10 rows
  OP_PARITY,  // product of y parities, coefficient z: 16-bit list of (count, qubits)
  OP_BIG,     // start of a polynomial of more than 8 bits: constant y | z << 32
  OP_BIGTERM, // y parities, coefficient z | w << 32: as OP_PARITY
  OP_BIGEND,  // amplitude *= exp(2 pi i f / 2^y)
  OP_TABLE,   // y qubits, first pattern z, w: the image moves bits; 16-bit list
};
constexpr uint32_t CHUNK = 1024;  // words of the stream staged at a time (ops do not straddle chunks)
constexpr uint32_t RUN_WARPS = 8;

struct RunParams {
  uint64_t* key;
  double2* amp;
  uint64_t m;
  uint32_t words, nb;      // 64-bit words per key, 32-qubit blocks of the register
  uint32_t used, changed;  // blocks that the run reads or writes, blocks that it writes
  const uint32_t* stream;
  uint32_t chunks;
  const double2* roots;    // scalar * exp(2 pi i f / 2^B)
  uint32_t trivial;        // every root is 1
  const uint16_t* image;
  const double2* phase;
  const uint8_t* unit;
};

// bit j of lane i's word -> bit i of lane j's
__device__ __forceinline__ uint32_t transpose32(uint32_t x, uint32_t lane) {
  uint32_t m = 0x0000ffffu;
#pragma unroll
  for (uint32_t s = 16; s; s >>= 1) {
    const uint32_t y = __shfl_xor_sync(0xffffffffu, x, s);
    x = (lane & s) ? (x & ~m) | ((y & ~m) >> s) : (x & m) | ((y & m) << s);
    m ^= m << (s >> 1);
  }
  return x;
}

// c / 2^B turns more for the entries of p, in bit planes
template <int B>
__device__ __forceinline__ void count_turns(uint32_t (&pl)[B], uint32_t c, uint32_t p) {
  uint32_t carry = 0;
#pragma unroll
  for (int b = 0; b < B; ++b) {
    const uint32_t t = (c >> b) & 1u ? p : 0u;
    const uint32_t old = pl[b];
    pl[b] = old ^ t ^ carry;
    carry = (old & t) | (carry & (old ^ t));
  }
}

// the AND of `count` parities, each the XOR of a list of words (the lanes share a list)
__device__ __forceinline__ uint32_t parity_product(const uint32_t* w, const uint16_t* list, uint32_t count, uint32_t lane) {
  uint32_t all = ~0u;
  for (uint32_t f = 0; f < count; ++f) {
    const uint32_t cnt = *list++;
    uint32_t x = 0;
    for (uint32_t r = lane; r < cnt; r += 32) x ^= w[list[r]];
    all &= __reduce_xor_sync(0xffffffffu, x);
    list += cnt;
  }
  return all;
}

// B: planes of the turn counters (3: eighths, 8: 1/256)
template <int B>
__global__ void __launch_bounds__(32 * RUN_WARPS) k_sp_run(const RunParams P) {
  extern __shared__ __align__(16) uint32_t run_smem[];
  uint32_t* const stage = run_smem;  // two chunks
  const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5, warps = blockDim.x >> 5;
  uint32_t* const w = run_smem + 2 * CHUNK + warp * P.nb * 32;
  const auto fetch = [&](uint32_t c) {
    if (c < P.chunks) {
      const uint32_t* src = P.stream + uint64_t(c) * CHUNK;
      uint32_t* const dst = stage + (c & 1u) * CHUNK;
      for (uint32_t i = 4 * threadIdx.x; i < CHUNK; i += 4 * blockDim.x)
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(
                         static_cast<uint32_t>(__cvta_generic_to_shared(dst + i))),
                     "l"(src + i)
                     : "memory");
    }
    asm volatile("cp.async.commit_group;\n" ::: "memory");
  };
  for (uint64_t g0 = uint64_t(blockIdx.x) * warps; g0 * 32 < P.m; g0 += uint64_t(gridDim.x) * warps) {
    fetch(0);
    const uint64_t i = (g0 + warp) * 32 + lane;
    const bool live = i < P.m;
    const bool works = (g0 + warp) * 32 < P.m;  // uniform over the warp
    uint32_t* const k32 = reinterpret_cast<uint32_t*>(P.key) + i * 2 * P.words;
    double2 a = make_double2(0.0, 0.0);
    if (works) {
      if (live) a = P.amp[i];
      for (uint32_t b = 0; b < P.nb; ++b)
        if ((P.used >> b) & 1u) w[32 * b + lane] = transpose32(live ? k32[b] : 0u, lane);
      __syncwarp();
    }
    uint32_t pl[B] = {};
    uint64_t big = 0;
    for (uint32_t c = 0; c < P.chunks; ++c) {
      fetch(c + 1);
      asm volatile("cp.async.wait_group 1;\n" ::: "memory");
      __syncthreads();
      const uint4* pc = reinterpret_cast<const uint4*>(stage + (c & 1u) * CHUNK);
      uint4 h = *pc;
      while (works && (h.x & 0xffu) != OP_END) {
        const uint4* const at = pc;
        const uint4 now = h;
        pc += h.x >> 16;
        h = *pc;  // the next op's head, in flight while this one runs
        const uint16_t* const list = reinterpret_cast<const uint16_t*>(at + 1);
        switch (now.x & 0xffu) {
          case OP_NOTS:
            // One lane walks them, so that consecutive ones need no barrier between: the chain through
            // a word is a load, two logic operations and a store.
            if (lane == 0) {
              const uint4* d = at + 1;
              uint4 x = *d;
              for (uint32_t r = 0; r < now.y; r += 4) {
                const uint4 next = *++d;  // at the end: the next op's head
                const auto one = [&](uint32_t o) {
                  const uint32_t t = o & 1023u, c = (o >> 10) & 1023u;
                  const uint32_t vt = w[t], vc = w[c];
                  if (o >> 30) {
                    w[t] = vc;
                    w[c] = vt;
                  } else {
                    w[t] = vt ^ (vc & w[o >> 20]);
                  }
                };
                one(x.x);
                if (r + 1 < now.y) one(x.y);
                if (r + 2 < now.y) one(x.z);
                if (r + 3 < now.y) one(x.w);
                x = next;
              }
            }
            __syncwarp();
            break;
          case OP_FLIP:
            for (uint32_t r = lane; r < now.y; r += 32) w[list[r]] ^= ~0u;  // distinct words
            __syncwarp();
            break;
          case OP_TERMS: {
            const uint2* const t = reinterpret_cast<const uint2*>(at + 1);
            const auto value = [&](uint32_t q) { return w[q & 1023u] & w[(q >> 10) & 1023u] & w[q >> 20]; };
            for (uint32_t r = lane; r < now.y; r += 64) {  // two terms in flight
              const uint2 x = t[r];
              const bool more = r + 32 < now.y;
              const uint2 x2 = more ? t[r + 32] : make_uint2(x.x, 0u);
              const uint32_t p = value(x.x), p2 = value(x2.x);
              count_turns<B>(pl, x.y >> (8 - B), p);
              if (more) count_turns<B>(pl, x2.y >> (8 - B), p2);
            }
            break;
          }
          case OP_AFFINE: {
            // lane j holds qubit j's word and makes row j's
            const uint32_t j0 = lane < now.y ? lane : 0u;
            const uint32_t q = list[j0], row = list[10 + j0];
            const uint32_t u = w[q];
            uint32_t v = (now.z >> lane) & 1u ? ~0u : 0u;
#pragma unroll
            for (uint32_t j = 0; j < SP_MAX_K; ++j) {
              const uint32_t x = __shfl_sync(0xffffffffu, u, j);
              if ((row >> j) & 1u) v ^= x;  // rows have no bits at or past the op's qubits
            }
            __syncwarp();
            if (lane < now.y) w[q] = v;
            __syncwarp();
            break;
          }
          case OP_PARITY: {
            const uint32_t p = parity_product(w, list, now.y, lane);
            count_turns<B>(pl, now.z >> (8 - B), lane == 0 ? p : 0u);
            break;
          }
          case OP_BIG: big = uint64_t(now.y) | uint64_t(now.z) << 32; break;
          case OP_BIGTERM: {
            const uint32_t p = parity_product(w, list, now.y, lane);
            if ((p >> lane) & 1u) big += uint64_t(now.z) | uint64_t(now.w) << 32;
            break;
          }
          case OP_BIGEND:
            poly_finish(big, a, now.y, true, make_double2(1.0, 0.0), false, nullptr);
            break;
          default: {  // OP_TABLE
            uint32_t x = 0;
            for (uint32_t j = 0; j < now.y; ++j) x |= ((w[list[j]] >> lane) & 1u) << j;
            if (!P.unit[now.z + x]) a = zmul(P.phase[now.z + x], a);
            if (now.w) {
              const uint32_t y = P.image[now.z + x];
              __syncwarp();
              for (uint32_t j = 0; j < now.y; ++j) {
                const uint32_t v = __ballot_sync(0xffffffffu, (y >> j) & 1u);
                if (lane == 0) w[list[j]] = v;
              }
              __syncwarp();
            }
            break;
          }
        }
      }
      __syncthreads();  // the chunk's buffer is refilled next
    }
    if (works) {
      if (!P.trivial) {  // the lanes' counts of each entry's turns, added
        uint32_t f = 0;
#pragma unroll
        for (int b = 0; b < B; ++b) f += uint32_t(__popc(transpose32(pl[b], lane))) << b;
        const double2 c = P.roots[f & ((1u << B) - 1)];
        if (!(c.x == 1.0 && c.y == 0.0)) a = zmul(c, a);
      }
      for (uint32_t b = 0; b < P.nb; ++b)
        if ((P.changed >> b) & 1u) {
          const uint32_t v = transpose32(w[32 * b + lane], lane);
          if (live) k32[b] = v;
        }
      if (live) P.amp[i] = a;
      __syncwarp();
    }
  }
}

}  // namespace

namespace ncsim {

void SlicedRun::reset() {
  any_ = moves_ = false;
  stream_.clear();
  nots_ = ~size_t(0);
  pending_.clear();
  std::memset(pending_mask_, 0, sizeof(pending_mask_));
  scalar_ = Phase();
  bits_ = 0;
  used_ = changed_ = 0;
  image_.clear();
  phase_.clear();
  unit_.clear();
}

void SlicedRun::release() {
  reset();
  const auto give_back = [](auto& v) {
    if (v.capacity() * sizeof(v[0]) > KEPT_BYTES) std::remove_reference_t<decltype(v)>().swap(v);
  };
  give_back(stream_);
  give_back(pending_);
  give_back(image_);
  give_back(phase_);
  give_back(unit_);
  blob_.clear();
  give_back(blob_);
}

uint32_t* SlicedRun::put(uint32_t type, uint32_t words) {
  const uint32_t len = 4 + ((words + 3) & ~3u);
  const uint32_t in = uint32_t(stream_.size() % CHUNK);
  if (in + len + 4 > CHUNK) stream_.resize(stream_.size() + CHUNK - in, 0);  // zero words read as OP_END
  const size_t at = stream_.size();
  stream_.resize(at + len, 0);
  stream_[at] = type | (len / 4) << 16;
  return stream_.data() + at;
}

void SlicedRun::touch(uint32_t q, bool write) {
  used_ |= 1u << (q >> 5);
  if (write) {
    changed_ |= 1u << (q >> 5);
    moves_ = true;
  }
}

// Terms wait until an op writes one of their qubits: diagonals that follow one another, or stand
// between ops on other qubits, share their rounds of lanes.
void SlicedRun::term(const std::vector<uint32_t>& f, uint32_t coeff8) {
  Term t{};
  for (size_t j = 0; j < 3; ++j) t.q[j] = uint16_t(f[std::min(j, f.size() - 1)]);
  t.coeff = uint8_t(coeff8);
  pending_.push_back(t);
  for (uint32_t q : f) {
    pending_mask_[q >> 6] |= uint64_t(1) << (q & 63);
    touch(q, false);
  }
}
void SlicedRun::flush_terms() {
  for (size_t i = 0; i < pending_.size();) {
    const uint32_t cnt = uint32_t(std::min<size_t>(pending_.size() - i, 384));
    uint32_t* p = put(OP_TERMS, 2 * cnt);
    p[1] = cnt;
    for (uint32_t r = 0; r < cnt; ++r, ++i) {
      p[4 + 2 * r] = uint32_t(pending_[i].q[0]) | uint32_t(pending_[i].q[1]) << 10 | uint32_t(pending_[i].q[2]) << 20;
      p[5 + 2 * r] = pending_[i].coeff;
    }
  }
  pending_.clear();
  std::memset(pending_mask_, 0, sizeof(pending_mask_));
}
void SlicedRun::before_write(uint32_t q) {
  if ((pending_mask_[q >> 6] >> (q & 63)) & 1) flush_terms();
  touch(q, true);
}

static void put_list(uint32_t* p, const std::vector<uint32_t>& qs, size_t from = 0) {
  uint16_t* l = reinterpret_cast<uint16_t*>(p);
  for (size_t j = 0; j < qs.size(); ++j) l[from + j] = uint16_t(qs[j]);
}

void SlicedRun::flips(const std::vector<uint32_t>& qs) {
  if (qs.empty()) return;
  for (uint32_t q : qs) before_write(q);
  uint32_t* p = put(OP_FLIP, uint32_t(qs.size() + 1) / 2);
  p[1] = uint32_t(qs.size());
  put_list(p + 4, qs);
}
void SlicedRun::control_not(uint32_t t, uint32_t c1, uint32_t c2) {
  before_write(t);
  touch(c1, false);
  touch(c2, false);
  put_not(t | c1 << 10 | c2 << 20);
}
// appended to the stream's last op when that is a list of NOTs with room in its chunk
void SlicedRun::put_not(uint32_t op) {
  if (nots_ < stream_.size() && nots_ + 4 * size_t(stream_[nots_] >> 16) == stream_.size()) {
    const uint32_t n = stream_[nots_ + 1];
    if (n % 4 == 0 && stream_.size() % CHUNK + 8 <= CHUNK && stream_.size() % CHUNK) {
      stream_.resize(stream_.size() + 4, 0);
      stream_[nots_] += 1u << 16;
    }
    if (4 + n < 4 * (stream_[nots_] >> 16)) {
      stream_[nots_ + 4 + n] = op;
      stream_[nots_ + 1] = n + 1;
      return;
    }
  }
  uint32_t* p = put(OP_NOTS, 4);
  nots_ = size_t(p - stream_.data());
  p[1] = 1;
  p[4] = op;
}

// coeff * prod (parity of each factor's qubits): counted in 1/256 turns (big_bits 0) or added to the
// current polynomial of more than 8 bits
void SlicedRun::product(const std::vector<std::vector<uint32_t>>& f, uint64_t coeff, uint32_t big_bits) {
  size_t words = 0;
  for (const auto& l : f) words += l.size() + 1;
  uint32_t* p = put(big_bits ? OP_BIGTERM : OP_PARITY, uint32_t(words + 1) / 2);
  p[1] = uint32_t(f.size());
  p[2] = uint32_t(coeff);
  p[3] = uint32_t(coeff >> 32);
  uint16_t* l = reinterpret_cast<uint16_t*>(p + 4);
  for (const auto& qs : f) {
    *l++ = uint16_t(qs.size());
    for (uint32_t q : qs) *l++ = uint16_t(q), touch(q, false);
  }
}

void SlicedRun::poly(const PhasePolyIR& p, const std::vector<uint32_t>& qubits) {
  const uint64_t mm = p.bits >= 64 ? ~uint64_t(0) : (uint64_t(1) << p.bits) - 1;
  const uint64_t vars = p.nvars >= 64 ? ~uint64_t(0) : (uint64_t(1) << p.nvars) - 1;
  const bool big = p.bits > 8;
  uint64_t constant = p.constant & mm;
  bool open = false;
  for (size_t i = 0; i < p.coeffs.size(); ++i) {
    const uint64_t c = p.coeffs[i] & mm;
    bool single = p.parities[i].size() <= 3, vanishes = c == 0;
    for (uint64_t l : p.parities[i]) {
      vanishes |= (l & vars) == 0;
      single &= __builtin_popcountll(l & vars) == 1;
    }
    if (vanishes) continue;
    if (p.parities[i].empty()) {
      constant = (constant + c) & mm;
      continue;
    }
    if (single && !big) {
      uint32_t f[3], nf = 0;
      for (uint64_t l : p.parities[i]) f[nf++] = qubits[__builtin_ctzll(l & vars)];
      Term t{};
      for (uint32_t j = 0; j < 3; ++j) {
        const uint32_t q = f[std::min(j, nf - 1)];
        t.q[j] = uint16_t(q);
        pending_mask_[q >> 6] |= uint64_t(1) << (q & 63);
        used_ |= 1u << (q >> 5);
      }
      t.coeff = uint8_t(c << (8 - p.bits));
      pending_.push_back(t);
      bits_ = std::max(bits_, p.bits);
      continue;
    }
    std::vector<std::vector<uint32_t>> f;
    for (uint64_t l : p.parities[i]) {
      f.emplace_back();
      for (uint64_t r = l & vars; r; r &= r - 1) f.back().push_back(qubits[__builtin_ctzll(r)]);
    }
    if (big && !open) {
      put(OP_BIG, 0);  // the constant goes with the scalar
      open = true;
    }
    if (!big) bits_ = std::max(bits_, p.bits);
    product(f, big ? c : c << (8 - p.bits), big ? p.bits : 0);
  }
  if (open) put(OP_BIGEND, 0)[1] = p.bits;
  if (constant) scalar_ = scalar_.times(Phase::make(0, int64_t(constant), p.bits));
}

void SlicedRun::table(const std::vector<uint32_t>& qubits, const std::vector<uint32_t>& image, const std::vector<CplxD>& ph) {
  bool moves = false;
  for (size_t x = 0; x < image.size(); ++x) moves |= image[x] != x;
  for (uint32_t q : qubits) {
    if (moves) before_write(q);
    else touch(q, false);
  }
  uint32_t* p = put(OP_TABLE, 5);
  p[1] = uint32_t(qubits.size());
  p[2] = uint32_t(image_.size());
  p[3] = moves;
  put_list(p + 4, qubits);
  for (size_t x = 0; x < image.size(); ++x) {
    image_.push_back(uint16_t(image[x]));
    phase_.push_back(ph[x].re);
    phase_.push_back(ph[x].im);
    unit_.push_back(ph[x].re == 1.0 && ph[x].im == 0.0);
  }
}

void SlicedRun::add_pauli(const std::vector<uint32_t>& qubits, uint64_t x, uint64_t z, uint32_t phase) {
  any_ = true;
  std::vector<uint32_t> fl;
  for (size_t j = 0; j < qubits.size() && j < 64; ++j) {  // Z first: its sign is that of the key before X
    if ((z >> j) & 1) {
      term({qubits[j]}, 128);
      bits_ = std::max(bits_, 1u);
    }
    if ((x >> j) & 1) fl.push_back(qubits[j]);
  }
  flips(fl);
  if (phase & 3u) scalar_ = scalar_.times(Phase::make(0, int64_t(phase & 3u), 2));
}

// whether every term fits in one op of the stream (a product of a great many wide parities does not)
static bool fits(const PhasePolyIR& p) {
  for (const auto& ps : p.parities) {
    size_t n = 0;
    for (uint64_t l : ps) n += 1 + size_t(__builtin_popcountll(l));
    if (n > CHUNK) return false;
  }
  return true;
}

bool SlicedRun::add_gate(const GateIR& g, const std::vector<uint32_t>& qubits, const LoweredOp& low) {
  if ((g.kind == GateKind::Diagonal && !fits(g.poly)) || (g.kind == GateKind::Monomial && !fits(g.mono.phase))) return false;
  switch (low.kind) {
    case LoweredKind::Nothing: return true;
    case LoweredKind::Pauli: add_pauli(qubits, g.pauli.x, g.pauli.z, g.pauli.phase); return true;
    case LoweredKind::PhasePoly:
      if (qubits.size() > 64) throw Error(NCSIM_ERR_UNSUPPORTED, "sparse phase polynomial on more than 64 qubits");
      break;
    case LoweredKind::Monomial:
      if (low.qubits.size() > SP_MAX_K) return false;
      break;
    case LoweredKind::Dense: {
      if (low.qubits.size() > SP_MAX_K) return false;
      std::vector<uint32_t> image;
      std::vector<CplxD> ph;
      if (!permutation_view(low.matrix, size_t(1) << low.qubits.size(), image, ph)) return false;
      any_ = true;
      table(qubits, image, ph);
      return true;
    }
  }
  any_ = true;
  switch (g.kind) {  // the common gates without their general view
    case GateKind::X: flips({qubits[0]}); return true;
    case GateKind::Cx: control_not(qubits[1], qubits[0], qubits[0]); return true;
    case GateKind::Ccx: control_not(qubits[2], qubits[0], qubits[1]); return true;
    case GateKind::Z: term({qubits[0]}, 128); bits_ = std::max(bits_, 1u); return true;
    case GateKind::Cz: term({qubits[0], qubits[1]}, 128); bits_ = std::max(bits_, 1u); return true;
    case GateKind::Ccz: term({qubits[0], qubits[1], qubits[2]}, 128); bits_ = std::max(bits_, 1u); return true;
    case GateKind::Diagonal: poly(g.poly, qubits); return true;
    case GateKind::Swap: {
      before_write(qubits[0]);
      before_write(qubits[1]);
      put_not(qubits[0] | qubits[1] << 10 | 1u << 30);
      return true;
    }
    default: break;
  }
  MonomialIR view;
  if (g.kind != GateKind::Monomial && !monomial_view(g, view)) {  // no affine view: its table
    table(qubits, low.image, low.matrix);
    return true;
  }
  const MonomialIR& mo = g.kind == GateKind::Monomial ? g.mono : view;
  poly(mo.phase, qubits);  // the phase is that of the key before the map
  if (!mo.scalar.is_one()) scalar_ = scalar_.times(mo.scalar);
  if (!mo.affine_identity()) {
    for (uint32_t q : qubits) before_write(q);
    uint32_t* p = put(OP_AFFINE, 10);
    p[1] = mo.k;
    p[2] = uint32_t(mo.shift);
    put_list(p + 4, qubits);
    uint16_t* rows = reinterpret_cast<uint16_t*>(p + 4) + 10;
    const uint64_t vars = (uint64_t(1) << mo.k) - 1;
    for (uint32_t j = 0; j < mo.k; ++j) rows[j] = uint16_t(mo.rows[j] & vars);
  }
  return true;
}

void SlicedRun::launch(ncsim_sparse* s) {
  if (!any_) return;
  flush_terms();
  const uint32_t B = bits_ <= 3 ? 3 : 8;
  bool trivial = true;
  std::vector<double2> roots(size_t(1) << B);
  for (size_t f = 0; f < roots.size(); ++f) {
    const Cd v = scalar_.times(Phase::make(0, int64_t(f), B)).value();
    roots[f] = make_double2(v.re, v.im);
  }
  trivial = bits_ == 0 && scalar_.is_one();
  const bool idle = stream_.empty() && trivial;
  if (s->m && !idle) {
    const uint32_t in = uint32_t(stream_.size() % CHUNK);
    if (in || stream_.empty()) stream_.resize(stream_.size() + CHUNK - in, 0);
    // one upload: stream, roots, phases, images, unit flags
    const size_t ns = stream_.size() * 4, nr = roots.size() * 16, np = phase_.size() * 8, ni = image_.size() * 2;
    blob_.resize(ns + nr + np + ni + unit_.size());
    std::memcpy(blob_.data(), stream_.data(), ns);
    std::memcpy(blob_.data() + ns, roots.data(), nr);
    if (np) std::memcpy(blob_.data() + ns + nr, phase_.data(), np);
    if (ni) std::memcpy(blob_.data() + ns + nr + np, image_.data(), ni);
    if (!unit_.empty()) std::memcpy(blob_.data() + ns + nr + np + ni, unit_.data(), unit_.size());
    cudaStream_t st = s->stream;
    uint8_t* d = upload(blob_, st);
    RunParams P{};
    P.key = s->key;
    P.amp = s->amp;
    P.m = s->m;
    P.words = s->words;
    P.nb = (s->n + 31) / 32;
    P.used = used_;
    P.changed = changed_;
    P.stream = reinterpret_cast<const uint32_t*>(d);
    P.chunks = uint32_t(stream_.size() / CHUNK);
    P.roots = reinterpret_cast<const double2*>(d + ns);
    P.trivial = trivial;
    P.phase = reinterpret_cast<const double2*>(d + ns + nr);
    P.image = reinterpret_cast<const uint16_t*>(d + ns + nr + np);
    P.unit = d + ns + nr + np + ni;
    // warps share a block's staged stream; few entries spread over the SMs one warp each
    const uint64_t groups = (s->m + 31) / 32;
    const uint32_t warps = uint32_t(std::max<uint64_t>(1, std::min<uint64_t>(RUN_WARPS, groups / (2 * uint64_t(sm_count())))));
    const uint64_t blocks = std::min<uint64_t>((groups + warps - 1) / warps, uint64_t(sm_count()) * 16);
    const size_t smem = (2 * CHUNK + size_t(warps) * P.nb * 32) * 4;  // at most 40 KB
    if (B == 3) k_sp_run<3><<<unsigned(blocks), 32 * warps, smem, st>>>(P);
    else k_sp_run<8><<<unsigned(blocks), 32 * warps, smem, st>>>(P);
    NCSIM_LAUNCHED("sparse run");
    dfree(d, st);
  }
  if (moves_) s->sorted = false;
  reset();
}

}  // namespace ncsim
