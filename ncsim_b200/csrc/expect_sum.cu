// Expectations of many Paulis in few passes over the register.
//
// One Pauli at a time, a sum of 100 terms reads the register 100 times and waits for
// the host 100 times.  Here a pass streams the register once in tiles of 2^T
// amplitudes (T <= 11; the tile's bits are a window of qubits) and evaluates every
// term whose X part lies in the window.  Terms with the same X part share their
// products: for a pair (c, d = c ^ x) a Pauli i^k X^x Z^z adds
//   i^k (-1)^{z.c} (s + (-1)^{z.x} conj s),  s = conj(psi(d)) psi(c),
// twice the real or i times twice the imaginary part of s (with x = 0 it is
// (-1)^{z.c} |psi(c)|^2).  A thread makes the products of its 2^(T-7) amplitudes in
// registers and Walsh-Hadamard transforms them over the tile bits that it holds, so
// that a term then costs one lookup and one signed addition per thread, whatever its
// Z part; the sums stay in shared memory until the last tile.
//
// What bounds it: instruction issue, about 14 instructions per term and 150 per X part
// for a thread's 16 amplitudes, against 42 us of HBM per pass at n = 24.
#include <algorithm>
#include <cstring>
#include <map>
#include <vector>

#include "engine.cuh"
#include "host/ir.hpp"

namespace ncsim {

namespace {

constexpr int ES_THREADS = 128;
constexpr int ES_THREAD_BITS = 7;
constexpr int ES_TILE_BITS = 11;
constexpr int ES_MIN_QUBITS = 8;  // smaller registers: one Pauli at a time
constexpr int ES_TERMS = 48;      // terms of one pass (at most 64, a word of signs): 48 KB of sums, two blocks per SM beside a 32 KB tile
constexpr int ES_GROUPS = 32;     // X parts of one pass
constexpr int ES_LOW_BITS = 2;    // lowest qubits kept in every window: runs of 64 bytes

template <class R>
using V = typename VecOf<R>::T;

struct EsTerm {
  uint64_t zout;     // Z bits outside the window
  uint32_t zthread;  // Z bits over the thread's index
  uint32_t row;      // which transformed value: the Z bits over the thread's own amplitudes (+ the imaginary parts' offset)
};
struct EsGroup {
  uint32_t xl;       // X part in the tile (0: diagonal)
  uint32_t h;        // its highest bit
  uint32_t first, count;
  uint32_t parts;    // which parts its terms use: 1 real, 2 imaginary
};
template <class R>
struct EsParams {
  const V<R>* amp;
  uint64_t ntiles;
  int T, w, nh;              // tile bits, low index bits in the window, window bits above them
  uint8_t hq[ES_TILE_BITS];  // and their positions, ascending
  uint32_t groups, terms;
  double* partials;          // [term][block]
  EsGroup g[ES_GROUPS];
  EsTerm t[ES_TERMS];
};

template <int N>
__device__ __forceinline__ void walsh(double (&v)[N]) {
#pragma unroll
  for (int s = 1; s < N; s <<= 1)
#pragma unroll
    for (int b = 0; b < N; ++b)
      if (!(b & s)) {
        const double u = v[b], w = v[b | s];
        v[b] = u + w;
        v[b | s] = u - w;
      }
}

__device__ __forceinline__ uint32_t es_swz(uint32_t e) { return e ^ (((e >> 3) ^ (e >> 6) ^ (e >> 9)) & 7u); }

template <class R, int LOGR>
__global__ void __launch_bounds__(ES_THREADS) k_expect_sum(const __grid_constant__ EsParams<R> P) {
  constexpr int N = 1 << LOGR;  // amplitudes per thread
  extern __shared__ __align__(16) unsigned char es_smem[];
  V<R>* const tile = reinterpret_cast<V<R>*>(es_smem);
  double* const rows = reinterpret_cast<double*>(tile + (ES_THREADS << LOGR));  // [row][thread]
  double* const sums = rows + N * ES_THREADS;                                   // [term][thread]
  const uint32_t tid = threadIdx.x;
  for (uint32_t t = 0; t < P.terms; ++t) sums[t * ES_THREADS + tid] = 0.0;
  const auto offset = [&](uint32_t e) {
    uint64_t o = e & ((1u << P.w) - 1);
    for (int i = 0; i < P.nh; ++i) o |= uint64_t((e >> (P.w + i)) & 1u) << P.hq[i];
    return o;
  };
  uint64_t mine[N];
#pragma unroll
  for (int r = 0; r < N; ++r) mine[r] = offset(tid + r * ES_THREADS);
  uint64_t mine_sign = 0;
  for (uint32_t t = 0; t < P.terms; ++t) mine_sign |= uint64_t(__popc(P.t[t].zthread & tid) & 1u) << t;
  for (uint64_t b = blockIdx.x; b < P.ntiles; b += gridDim.x) {
    uint64_t base = b << P.w;
    for (int i = 0; i < P.nh; ++i) {
      const int q = P.hq[i];
      base = ((base >> q) << (q + 1)) | (base & ((uint64_t(1) << q) - 1));
    }
    V<R> a[N];
#pragma unroll
    for (int r = 0; r < N; ++r) a[r] = P.amp[base + mine[r]];
#pragma unroll
    for (int r = 0; r < N; ++r) tile[es_swz(tid + r * ES_THREADS)] = a[r];
    __syncthreads();
    // bit t: term t's sign for this thread's amplitudes of this tile
    uint64_t sign = mine_sign;
    {
      const uint32_t lane = tid & 31u;
      uint32_t odd[2];
#pragma unroll
      for (uint32_t j = 0; j < 2; ++j) {
        const uint32_t t = min(lane + 32 * j, P.terms - 1);
        odd[j] = __ballot_sync(0xffffffffu, __popcll(P.t[t].zout & base) & 1);
      }
      sign ^= uint64_t(odd[0]) | uint64_t(odd[1]) << 32;
    }
    for (uint32_t g = 0; g < P.groups; ++g) {
      const EsGroup G = P.g[g];
      if (G.xl == 0) {
        double v[N];
#pragma unroll
        for (int r = 0; r < N; ++r) {
          const V<R> c = tile[es_swz(tid + r * ES_THREADS)];
          v[r] = double(c.x) * double(c.x) + double(c.y) * double(c.y);
        }
        walsh<N>(v);
#pragma unroll
        for (int r = 0; r < N; ++r) rows[r * ES_THREADS + tid] = v[r];
      } else {
        // pair r of the thread: its index with a zero at h; spreading, swizzle and x are all XOR-linear
        double re[N / 2], im[N / 2];
        const uint32_t lo = (1u << G.h) - 1;
        const auto at = [&](uint32_t p) { return es_swz(((p & ~lo) << 1) | (p & lo)); };
        const uint32_t mine_at = at(tid), x_at = es_swz(G.xl);
        uint32_t step[LOGR];
#pragma unroll
        for (int j = 0; j + 1 < LOGR; ++j) step[j] = at(ES_THREADS << j);
#pragma unroll
        for (int r = 0; r < N / 2; ++r) {
          uint32_t e = mine_at;
#pragma unroll
          for (int j = 0; j + 1 < LOGR; ++j)
            if ((r >> j) & 1) e ^= step[j];
          const V<R> c = tile[e], d = tile[e ^ x_at];
          const double cx = c.x, cy = c.y, dx = d.x, dy = d.y;
          re[r] = dx * cx + dy * cy;
          im[r] = dx * cy - dy * cx;
        }
        if (G.parts & 1u) {
          walsh<N / 2>(re);
#pragma unroll
          for (int r = 0; r < N / 2; ++r) rows[r * ES_THREADS + tid] = re[r];
        }
        if (G.parts & 2u) {
          walsh<N / 2>(im);
#pragma unroll
          for (int r = 0; r < N / 2; ++r) rows[(N / 2 + r) * ES_THREADS + tid] = im[r];
        }
      }
      // rows and sums are the thread's own: no barrier
#pragma unroll 2
      for (uint32_t t = G.first; t < G.first + G.count; ++t) {
        const double v = rows[P.t[t].row * ES_THREADS + tid];
        const uint32_t flip = uint32_t(sign >> t) << 31;
        sums[t * ES_THREADS + tid] += __hiloint2double(int(uint32_t(__double2hiint(v)) ^ flip), __double2loint(v));
      }
    }
    __syncthreads();  // the tile is overwritten next
  }
  __syncthreads();
  const uint32_t lane = tid & 31u;
  for (uint32_t t = tid >> 5; t < P.terms; t += ES_THREADS / 32) {
    double v = 0.0;
#pragma unroll
    for (int j = 0; j < ES_THREADS / 32; ++j) v += sums[t * ES_THREADS + lane + 32 * j];
#pragma unroll
    for (int o = 16; o; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    if (lane == 0) P.partials[uint64_t(t) * gridDim.x + blockIdx.x] = v;
  }
}

// out[t] = the sum of term t's block partials, in a fixed order (one warp per term)
__global__ void k_expect_sum_blocks(const double* partials, uint32_t blocks, double* out) {
  double v = 0.0;
  for (uint32_t b = threadIdx.x; b < blocks; b += 32) v += partials[uint64_t(blockIdx.x) * blocks + b];
#pragma unroll
  for (int o = 16; o; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  if (threadIdx.x == 0) out[blockIdx.x] = v;
}

// one pass: its window, and the terms it evaluates (indices into the caller's list)
struct EsPass {
  uint64_t window = 0;
  std::vector<std::pair<uint64_t, std::vector<uint32_t>>> groups;
  uint32_t terms = 0;
};

template <class R>
void launch_pass(const ncsim_state* s, const EsPass& pass, const uint64_t* z, double* partials, double* out, unsigned blocks) {
  EsParams<R> P;
  P.amp = static_cast<const V<R>*>(s->amp);
  const int T = __builtin_popcountll(pass.window);
  P.T = T;
  P.ntiles = s->len >> T;
  P.w = 0;
  while (P.w < int(s->n) && ((pass.window >> P.w) & 1)) ++P.w;
  P.nh = 0;
  int local[64];
  for (int q = 0, l = 0; q < 64; ++q) local[q] = ((pass.window >> q) & 1) ? l++ : -1;
  for (int q = P.w; q < int(s->n); ++q)
    if ((pass.window >> q) & 1) P.hq[P.nh++] = uint8_t(q);
  const auto to_local = [&](uint64_t m) {
    uint32_t r = 0;
    for (uint64_t v = m & pass.window; v; v &= v - 1) r |= 1u << local[__builtin_ctzll(v)];
    return r;
  };
  const int logr = T - ES_THREAD_BITS;
  P.groups = uint32_t(pass.groups.size());
  P.terms = 0;
  for (uint32_t g = 0; g < P.groups; ++g) {
    const uint64_t x = pass.groups[g].first;
    EsGroup& G = P.g[g];
    G.xl = to_local(x);
    G.h = G.xl ? 31u - uint32_t(__builtin_clz(G.xl)) : 0u;
    G.first = P.terms;
    G.parts = 0;
    for (uint32_t i : pass.groups[g].second) {
      EsTerm& t = P.t[P.terms++];
      uint32_t zl = to_local(z[i]);
      uint32_t part = 0;
      if (G.xl) {
        const uint32_t lo = (1u << G.h) - 1;
        zl = (zl & lo) | ((zl >> (G.h + 1)) << G.h);  // over the pair's index: bit h is 0 at c
        const uint32_t odd = uint32_t(__builtin_popcountll(z[i] & x) & 1);
        part = odd << (logr - 1);
        G.parts |= 1u << odd;
      }
      t.zout = z[i] & ~pass.window;
      t.zthread = zl & (ES_THREADS - 1);
      t.row = (zl >> ES_THREAD_BITS) + part;
    }
    G.count = P.terms - G.first;
  }
  P.partials = partials;
  const size_t smem = (size_t(ES_THREADS) << logr) * (sizeof(V<R>) + sizeof(double)) + size_t(P.terms) * ES_THREADS * sizeof(double);
  const auto go = [&](auto lr) {
    constexpr int L = decltype(lr)::value;
    // the limit, not this launch's size: threads that race here set the same value
    NCSIM_CUDA(cudaFuncSetAttribute(k_expect_sum<R, L>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                    int((size_t(ES_THREADS) << L) * 24 + ES_TERMS * ES_THREADS * sizeof(double))));
    k_expect_sum<R, L><<<blocks, ES_THREADS, smem, s->stream>>>(P);
  };
  {
    ProfScope ps(s, K_EXPECT, double(s->bytes()));
    if (logr == 1) go(std::integral_constant<int, 1>{});
    else if (logr == 2) go(std::integral_constant<int, 2>{});
    else if (logr == 3) go(std::integral_constant<int, 3>{});
    else go(std::integral_constant<int, 4>{});
    NCSIM_LAUNCHED("k_expect_sum");
  }
  k_expect_sum_blocks<<<P.terms, 32, 0, s->stream>>>(partials, blocks, out);
  NCSIM_LAUNCHED("k_expect_sum_blocks");
}

}  // namespace

// The fewest terms that a pass is made for; fewer go one Pauli at a time.  While the register
// stays in the L2 the wait for a single Pauli outweighs a pass (8 terms in windows of their own,
// n = 20: 178 us one by one, 139 in passes; n = 22 238 and 207).  From 128 MiB on one Pauli streams the
// register faster than a pass (the same terms, n = 23: 338 and 387, n = 28 4.9 and 10.0 ms), two
// do not (n = 26 1.41 and 1.26 ms), unless a window of scattered qubits reads a complex128 register
// of some GiB in short runs (n = 30 19.3 and 22.8 ms; three terms 22.2 and 15.2; a window of low qubits
// 5.2 and 4.7; complex64 16.2 and 13.6).
uint32_t least_terms(const ncsim_state* s, uint64_t window) {
  if (s->bytes() < (size_t(128) << 20)) return 1;
  const bool short_runs = (window & 127) != 127;
  return s->precision == NCSIM_C128 && s->bytes() >= (size_t(4) << 30) && short_runs ? 3 : 2;
}

CplxD state_expectation(const ncsim_state* s, uint64_t x, uint64_t z, uint32_t phase);
void check_pauli_on(const ncsim_state* s, uint64_t x, uint64_t z);

// <psi|P_k|psi> of every term.  Terms whose X part spans more qubits than a window holds, and
// registers of fewer than 8 qubits, go one Pauli at a time; so does a single term, and so do the
// terms of a pass that would have too few (least_terms).
void state_expectations(const ncsim_state* s, uint64_t count, const uint64_t* x, const uint64_t* z, const uint32_t* phase,
                        CplxD* out) {
  for (uint64_t k = 0; k < count; ++k) check_pauli_on(s, x[k], z[k]);
  const int T = int(std::min<uint32_t>(s->n, ES_TILE_BITS));
  const uint64_t low = int(s->n) > T ? (uint64_t(1) << ES_LOW_BITS) - 1 : 0;
  std::map<uint64_t, std::vector<uint32_t>> by_x;
  for (uint64_t k = 0; k < count; ++k) {
    if (count < 2 || s->n < uint32_t(ES_MIN_QUBITS) || __builtin_popcountll(x[k] | low) > T) {
      out[k] = state_expectation(s, x[k], z[k], phase[k] & 3);
      continue;
    }
    by_x[x[k]].push_back(uint32_t(k));
  }
  if (by_x.empty()) return;
  // passes: X parts in ascending order into the first window with room, so that neighbours share one
  std::vector<EsPass> passes;
  std::vector<std::pair<uint64_t, std::vector<uint32_t>>> left(by_x.begin(), by_x.end());
  // the diagonal terms fit any window: last, into what room the others leave
  if (left.front().first == 0) std::rotate(left.begin(), left.begin() + 1, left.end());
  while (!left.empty()) {
    EsPass p;
    p.window = low;
    std::vector<std::pair<uint64_t, std::vector<uint32_t>>> rest;
    for (auto& g : left) {
      const uint64_t w = p.window | g.first;
      const size_t room = size_t(ES_TERMS) - p.terms;
      if (p.groups.size() >= size_t(ES_GROUPS) || room == 0 || __builtin_popcountll(w) > T) {
        rest.push_back(std::move(g));
        continue;
      }
      p.window = w;
      const size_t n = std::min(room, g.second.size());
      p.groups.push_back({g.first, std::vector<uint32_t>(g.second.begin(), g.second.begin() + long(n))});
      p.terms += uint32_t(n);
      if (n < g.second.size()) rest.push_back({g.first, std::vector<uint32_t>(g.second.begin() + long(n), g.second.end())});
    }
    for (int q = 0; __builtin_popcountll(p.window) < T; ++q) p.window |= uint64_t(1) << q;
    left.swap(rest);
    if (p.terms >= least_terms(s, p.window)) {
      passes.push_back(std::move(p));
      continue;
    }
    for (const auto& g : p.groups)
      for (uint32_t k : g.second) out[k] = state_expectation(s, x[k], z[k], phase[k] & 3);
  }
  // Scratch is the state's own, as for a single Pauli: in its reduction scratch the block partials (one
  // pass after another) and behind them the sums, fetched when the room is used up.
  constexpr size_t SLOTS = size_t(MAX_REDUCE_BLOCKS) * PARTIAL_SLOTS;
  const unsigned blocks =
      unsigned(std::min<uint64_t>({s->len >> T, uint64_t(sm_count()) * 2, uint64_t(SLOTS / ES_TERMS - 1)}));
  double* const sums = s->partials + size_t(ES_TERMS) * blocks;
  const size_t room = SLOTS - size_t(ES_TERMS) * blocks;
  for (size_t first = 0; first < passes.size();) {
    size_t end = first, at = 0;
    for (; end < passes.size() && at + passes[end].terms <= room; ++end) {
      if (s->precision == NCSIM_C128) launch_pass<double>(s, passes[end], z, s->partials, sums + at, blocks);
      else launch_pass<float>(s, passes[end], z, s->partials, sums + at, blocks);
      at += passes[end].terms;
    }
    NCSIM_CUDA(cudaMemcpyAsync(s->host_partials, sums, at * sizeof(double), cudaMemcpyDeviceToHost, s->stream));
    NCSIM_CUDA(cudaStreamSynchronize(s->stream));
    const double* v = s->host_partials;
    for (; first < end; ++first)
      for (const auto& g : passes[first].groups)
        for (uint32_t k : g.second) {
          const double a = *v++;
          // i^phase times the sum: 2 Re s, 2 i Im s, or the diagonal's
          const uint32_t odd = uint32_t(__builtin_popcountll(z[k] & g.first) & 1);
          const double m = g.first ? 2.0 * a : a;
          switch ((phase[k] + odd) & 3u) {
            case 0: out[k] = {m, 0.0}; break;
            case 1: out[k] = {0.0, m}; break;
            case 2: out[k] = {-m, 0.0}; break;
            default: out[k] = {0.0, -m}; break;
          }
        }
  }
}

}  // namespace ncsim
