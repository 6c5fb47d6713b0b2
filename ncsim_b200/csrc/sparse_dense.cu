// Dense 1-qubit gates of the sparse form without a sort.
//
// A dense gate on qubit q sends an entry to the two keys that differ in bit q
// (sparse.rs:162-214); the results are then ordered by key, duplicates summed, zeros and
// amplitudes under the cutoff dropped (sparse.rs:114-128).  When the entries are sorted
// and distinct, as they are after every such step, the new order needs no sort: entries
// with the same bits above q are one range of the array, in it those with bit q = 0
// precede those with 1, and both halves are ordered by the bits below.  Merging the two
// halves (an entry's place: two binary searches) brings the partners of every pair side
// by side; each pair gives at most two outputs, and with the running counts S0, S1 of
// outputs kept with bit q = 0 and 1 the output places are
//   key with bit 0:  S0[pair] + S1[start of the range]
//   key with bit 1:  S1[pair] + S0[end of the range].
// A pair's sum has two terms, so it has the same bits in either order.
//
// Which outputs are kept is decided once, by the counting step; the placing step reads
// that decision, so that an output never lands in a place that was not counted for it.
// The values are made twice with the same fixed roundings.
//
// Up to SMALL_OUT outputs one block walks a whole list of gates (the Hadamards that open
// a circuit) with one launch and one wait: 6 us a gate (n = 31, small sets) to 11 (16-word keys), where the sort-based form
// took eleven launches, a wait and some 80 us.  Larger states take five launches a gate
// (merge, count, the scan's two, place).
#include "sparse_dense.hpp"

#include "sparse_common.cuh"

namespace {

constexpr uint32_t SMALL_OUT = 8192;  // outputs of one gate in the one-block form
constexpr uint32_t SMALL_THREADS = 1024;
constexpr uint32_t SMALL_GATES = 64;

template <int W>
struct DKey {
  uint64_t w[W];
};
template <int W>
__device__ __forceinline__ DKey<W> load_key(const uint64_t* k, uint64_t i) {
  DKey<W> r;
#pragma unroll
  for (int w = 0; w < W; ++w) r.w[w] = k[i * W + w];
  return r;
}
template <int W>
__device__ __forceinline__ void store_key(uint64_t* k, uint64_t i, const DKey<W>& v) {
#pragma unroll
  for (int w = 0; w < W; ++w) k[i * W + w] = v.w[w];
}
template <int W>
__device__ __forceinline__ bool equals_at(const uint64_t* k, uint64_t i, const DKey<W>& x) {
#pragma unroll
  for (int w = 0; w < W; ++w)
    if (k[i * W + w] != x.w[w]) return false;
  return true;
}
// the first of m sorted keys that is not below x (W words, word 0 first)
template <int W>
__device__ __forceinline__ uint32_t lower_bound(const uint64_t* k, uint32_t m, const DKey<W>& x) {
  uint32_t lo = 0, hi = m;
  while (lo < hi) {
    const uint32_t mid = (lo + hi) >> 1;
    bool below = false;
#pragma unroll
    for (int w = 0; w < W; ++w) {
      const uint64_t v = k[uint64_t(mid) * W + w];
      if (v != x.w[w]) {
        below = v < x.w[w];
        break;
      }
    }
    if (below) lo = mid + 1;
    else hi = mid;
  }
  return lo;
}

struct Gate1 {
  uint32_t q;
  double2 m[4];
};
template <int W>
struct OnBit {  // the key parts of a gate on qubit q
  uint32_t word;
  uint64_t bit;
  __device__ __forceinline__ explicit OnBit(uint32_t q) : word(q >> 6), bit(uint64_t(1) << (q & 63)) {}
  __device__ __forceinline__ bool one(const DKey<W>& k) const {
    bool r = false;
#pragma unroll
    for (int w = 0; w < W; ++w)
      if (uint32_t(w) == word) r = (k.w[w] & bit) != 0;
    return r;
  }
  __device__ __forceinline__ DKey<W> with(DKey<W> k, bool v) const {
#pragma unroll
    for (int w = 0; w < W; ++w)
      if (uint32_t(w) == word) k.w[w] = v ? (k.w[w] | bit) : (k.w[w] & ~bit);
    return k;
  }
  // the bits above q, then bit q = v, then zeros
  __device__ __forceinline__ DKey<W> prefix(DKey<W> k, bool v) const {
#pragma unroll
    for (int w = 0; w < W; ++w) {
      if (uint32_t(w) == word) k.w[w] = (k.w[w] & ~(2 * bit - 1)) | (v ? bit : 0);
      else if (uint32_t(w) > word) k.w[w] = 0;
    }
    return k;
  }
  // the last key of the range: the bits above q, then ones
  __device__ __forceinline__ DKey<W> last(DKey<W> k) const {
#pragma unroll
    for (int w = 0; w < W; ++w) {
      if (uint32_t(w) == word) k.w[w] |= 2 * bit - 1;
      else if (uint32_t(w) > word) k.w[w] = ~uint64_t(0);
    }
    return k;
  }
};

// entry i's place in the order of the keys without bit q (partners side by side, bit 0 first)
template <int W>
__device__ __forceinline__ uint32_t merged_place(const uint64_t* key, uint32_t m, uint32_t i, const OnBit<W>& B) {
  const DKey<W> k = load_key<W>(key, i);
  const bool one = B.one(k);
  const uint32_t mid = lower_bound<W>(key, m, B.prefix(k, true));
  const DKey<W> other = B.with(k, !one);
  const uint32_t o = lower_bound<W>(key, m, other);
  if (!one) return i + (o - mid);
  return o + (i - mid) + (o < m && equals_at<W>(key, o, other) ? 1u : 0u);
}

// The outputs of the pair whose first entry stands at merged place p (out[r]: the key with bit q = r),
// in a fixed sequence of roundings; false at the second entry of a pair, whose place has none.
template <int W>
__device__ __forceinline__ bool pair_values(const uint64_t* key, const double2* amp, const uint32_t i, bool has_prev,
                                            uint32_t prev, bool has_next, uint32_t next, const OnBit<W>& B,
                                            const double2* g, double2 (&out)[2]) {
  const DKey<W> k = load_key<W>(key, i);
  const bool one = B.one(k);
  const DKey<W> other = B.with(k, !one);
  if (one && has_prev && equals_at<W>(key, prev, other)) return false;
  const double2 v = amp[i];
  const uint32_t col = one ? 1u : 0u;
  out[0] = cmul(g[col], v);
  out[1] = cmul(g[2 + col], v);
  if (!one && has_next && equals_at<W>(key, next, other)) {
    const double2 u = amp[next];
    const double2 a = cmul(g[1], u), b = cmul(g[3], u);
    out[0] = make_double2(__dadd_rn(out[0].x, a.x), __dadd_rn(out[0].y, a.y));
    out[1] = make_double2(__dadd_rn(out[1].x, b.x), __dadd_rn(out[1].y, b.y));
  }
  return true;
}
// which of a pair's outputs stay (bit r: out[r]): nonzero and not under the cutoff
__device__ __forceinline__ uint32_t kept(const double2 (&out)[2], double cut2) {
  uint32_t keep = 0;
#pragma unroll
  for (int r = 0; r < 2; ++r) {
    const double2 a = out[r];
    const bool zero = a.x == 0.0 && a.y == 0.0;
    if (!zero && (cut2 == 0.0 || __fma_rn(a.x, a.x, __dmul_rn(a.y, a.y)) >= cut2)) keep |= 1u << r;
  }
  return keep;
}

// ---- one block, a list of gates ----
struct SmallParams {
  const uint64_t* key0;
  const double2* amp0;
  uint64_t* key[2];  // outputs of the gates, in turn
  double2* amp[2];
  uint32_t m, cap;   // entries, room in each output
  uint32_t gates;
  double cut2;
  uint32_t* result;  // host memory: entries, gates applied
  Gate1 g[SMALL_GATES];
};
template <int W>
__global__ void __launch_bounds__(SMALL_THREADS) k_sp_dense1_small(const __grid_constant__ SmallParams P) {
  __shared__ uint16_t s_at[SMALL_OUT / 2];       // merged place -> entry
  __shared__ uint32_t s_sum[SMALL_OUT / 2 + 1];  // counts of outputs before a place: bit q = 0 | bit q = 1 << 16
  __shared__ uint32_t s_warp[32];
  const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
  const uint64_t* key = P.key0;
  const double2* amp = P.amp0;
  uint32_t m = P.m, done = 0;
  for (; done < P.gates && 2 * m <= P.cap; ++done) {
    const OnBit<W> B(P.g[done].q);
    const double2 g[4] = {P.g[done].m[0], P.g[done].m[1], P.g[done].m[2], P.g[done].m[3]};
    uint64_t* const okey = P.key[done & 1u];
    double2* const oamp = P.amp[done & 1u];
    for (uint32_t i = threadIdx.x; i < m; i += SMALL_THREADS) s_at[merged_place<W>(key, m, i, B)] = uint16_t(i);
    __syncthreads();
    // counts: every thread a range of places, the ranges scanned over the block
    const uint32_t per = (m + SMALL_THREADS - 1) / SMALL_THREADS;
    const uint32_t p0 = min(threadIdx.x * per, m), p1 = min(p0 + per, m);
    const auto pair_at = [&](uint32_t p, double2 (&out)[2]) {
      return pair_values<W>(key, amp, s_at[p], p > 0, s_at[p ? p - 1 : 0], p + 1 < m, s_at[p + 1 < m ? p + 1 : 0], B, g, out);
    };
    uint32_t mine = 0;
    double2 out[2];
    for (uint32_t p = p0; p < p1; ++p) {
      const uint32_t keep = pair_at(p, out) ? kept(out, P.cut2) : 0u;
      s_sum[p] = mine;  // within the range for now
      mine += (keep & 1u) | (keep >> 1) << 16;
    }
    uint32_t inc = mine;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const uint32_t v = __shfl_up_sync(0xffffffffu, inc, o);
      if (lane >= uint32_t(o)) inc += v;
    }
    if (lane == 31) s_warp[warp] = inc;
    __syncthreads();
    if (warp == 0) {
      uint32_t v = s_warp[lane];
      uint32_t t = v;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const uint32_t u = __shfl_up_sync(0xffffffffu, t, o);
        if (lane >= uint32_t(o)) t += u;
      }
      s_warp[lane] = t - v;
      if (lane == 31) s_sum[m] = t;
    }
    __syncthreads();
    const uint32_t before = s_warp[warp] + inc - mine;
    for (uint32_t p = p0; p < p1; ++p) s_sum[p] += before;
    __syncthreads();
    for (uint32_t p = threadIdx.x; p < m; p += SMALL_THREADS) {
      const uint32_t counted = s_sum[p + 1] - s_sum[p];  // the counting step's decision
      const uint32_t keep = (counted & 1u) | (counted >> 16) << 1;
      if (!keep) continue;
      pair_at(p, out);
      const DKey<W> k = load_key<W>(key, s_at[p]);
      const uint32_t lo = lower_bound<W>(key, m, B.prefix(k, false));
      const DKey<W> end = B.last(k);
      uint32_t hi = lower_bound<W>(key, m, end);
      if (hi < m && equals_at<W>(key, hi, end)) ++hi;
      if (keep & 1u) {
        const uint32_t r = (s_sum[p] & 0xffffu) + (s_sum[lo] >> 16);
        store_key<W>(okey, r, B.with(k, false));
        oamp[r] = out[0];
      }
      if (keep & 2u) {
        const uint32_t r = (s_sum[p] >> 16) + (s_sum[hi] & 0xffffu);
        store_key<W>(okey, r, B.with(k, true));
        oamp[r] = out[1];
      }
    }
    __syncthreads();
    const uint32_t total = s_sum[m];
    m = (total & 0xffffu) + (total >> 16);
    key = okey;
    amp = oamp;
    __syncthreads();
  }
  if (threadIdx.x == 0) {
    P.result[0] = m;
    P.result[1] = done;
  }
}

// ---- any number of entries, one gate ----
template <int W>
__global__ void k_sp_dense1_merge(const uint64_t* key, uint32_t m, uint32_t q, uint32_t* at) {
  const OnBit<W> B(q);
  for (uint64_t i = uint64_t(blockIdx.x) * blockDim.x + threadIdx.x; i < m; i += uint64_t(gridDim.x) * blockDim.x)
    at[merged_place<W>(key, m, uint32_t(i), B)] = uint32_t(i);
}
template <int W>
__device__ __forceinline__ bool pair_in(const uint64_t* key, const double2* amp, uint32_t m, const uint32_t* at, uint32_t p,
                                        const OnBit<W>& B, const Gate1& g, double2 (&out)[2]) {
  return pair_values<W>(key, amp, at[p], p > 0, at[p ? p - 1 : 0], p + 1 < m, at[p + 1 < m ? p + 1 : 0], B, g.m, out);
}
template <int W>
__global__ void k_sp_dense1_count(const uint64_t* key, const double2* amp, uint32_t m, const uint32_t* at,
                                  const __grid_constant__ Gate1 g, double cut2, uint64_t* cnt) {
  const OnBit<W> B(g.q);
  for (uint64_t p = uint64_t(blockIdx.x) * blockDim.x + threadIdx.x; p <= m; p += uint64_t(gridDim.x) * blockDim.x) {
    double2 out[2];
    const uint32_t keep = p < m && pair_in<W>(key, amp, m, at, uint32_t(p), B, g, out) ? kept(out, cut2) : 0u;
    cnt[p] = uint64_t(keep & 1u) | uint64_t(keep >> 1) << 32;
  }
}
template <int W>
__global__ void k_sp_dense1_place(const uint64_t* key, const double2* amp, uint32_t m, const uint32_t* at,
                                  const __grid_constant__ Gate1 g, const uint64_t* cnt, const uint64_t* sum, uint64_t* okey,
                                  double2* oamp, uint32_t* result) {
  const OnBit<W> B(g.q);
  for (uint64_t p = uint64_t(blockIdx.x) * blockDim.x + threadIdx.x; p < m; p += uint64_t(gridDim.x) * blockDim.x) {
    if (p == 0) *result = uint32_t(sum[m]) + uint32_t(sum[m] >> 32);
    const uint64_t counted = cnt[p];
    const uint32_t keep = uint32_t(counted & 1u) | uint32_t(counted >> 32) << 1;
    if (!keep) continue;
    double2 out[2];
    pair_in<W>(key, amp, m, at, uint32_t(p), B, g, out);
    const DKey<W> k = load_key<W>(key, at[p]);
    const uint32_t lo = lower_bound<W>(key, m, B.prefix(k, false));
    const DKey<W> end = B.last(k);
    uint32_t hi = lower_bound<W>(key, m, end);
    if (hi < m && equals_at<W>(key, hi, end)) ++hi;
    if (keep & 1u) {
      const uint64_t r = uint64_t(uint32_t(sum[p])) + (sum[lo] >> 32);
      store_key<W>(okey, r, B.with(k, false));
      oamp[r] = out[0];
    }
    if (keep & 2u) {
      const uint64_t r = (sum[p] >> 32) + uint64_t(uint32_t(sum[hi]));
      store_key<W>(okey, r, B.with(k, true));
      oamp[r] = out[1];
    }
  }
}

Gate1 device_gate(const SparseDense1& g) {
  Gate1 r;
  r.q = g.q;
  for (int i = 0; i < 4; ++i) r.m[i] = make_double2(g.m[i].re, g.m[i].im);
  return r;
}

void take(ncsim_sparse* s, uint64_t* key, double2* amp, uint64_t cap, uint64_t m) {
  dfree(s->key, s->stream);
  dfree(s->amp, s->stream);
  s->key = key;
  s->amp = amp;
  s->cap = cap;
  s->m = m;
  s->sorted = true;
}

// the gates from `first` on that fit the one-block form; returns how many were applied
template <int W>
size_t apply_small(ncsim_sparse* s, const std::vector<SparseDense1>& gates, size_t first) {
  cudaStream_t st = s->stream;
  auto P = std::make_unique<SmallParams>();
  P->gates = uint32_t(std::min<size_t>(gates.size() - first, SMALL_GATES));
  for (uint32_t i = 0; i < P->gates; ++i) P->g[i] = device_gate(gates[first + i]);
  uint64_t cap = s->m;
  for (uint32_t i = 0; i < P->gates && cap < SMALL_OUT; ++i) cap *= 2;
  cap = std::min<uint64_t>(cap, SMALL_OUT);
  P->key0 = s->key;
  P->amp0 = s->amp;
  P->m = uint32_t(s->m);
  P->cap = uint32_t(cap);
  P->cut2 = s->cutoff * s->cutoff;
  P->result = reinterpret_cast<uint32_t*>(s->host_partials);  // pinned: written by the kernel
  for (int b = 0; b < 2; ++b) {
    P->key[b] = dalloc<uint64_t>(cap * W, st);
    P->amp[b] = dalloc<double2>(cap, st);
  }
  k_sp_dense1_small<W><<<1, SMALL_THREADS, 0, st>>>(*P);
  NCSIM_LAUNCHED("sparse dense gates");
  NCSIM_CUDA(cudaStreamSynchronize(st));
  const uint32_t m = P->result[0], done = P->result[1];
  const int last = int((done + 1) & 1u);  // the last gate's output (of `done` gates: buffer (done - 1) % 2)
  if (done) {
    take(s, P->key[last], P->amp[last], cap, m);
    dfree(P->key[last ^ 1], st);
    dfree(P->amp[last ^ 1], st);
  } else {
    for (int b = 0; b < 2; ++b) {
      dfree(P->key[b], st);
      dfree(P->amp[b], st);
    }
  }
  return done;
}

template <int W>
void apply_large(ncsim_sparse* s, const SparseDense1& gate) {
  cudaStream_t st = s->stream;
  const uint64_t m = s->m;
  if (2 * m > uint64_t(INT32_MAX)) throw Error(NCSIM_ERR_UNSUPPORTED, "sparse state of more than 2^31 entries");
  const Gate1 g = device_gate(gate);
  const double cut2 = s->cutoff * s->cutoff;
  uint32_t* at = dalloc<uint32_t>(m, st);
  uint64_t* cnt = dalloc<uint64_t>(m + 1, st);
  uint64_t* sum = dalloc<uint64_t>(m + 1, st);
  uint64_t* okey = dalloc<uint64_t>(2 * m * W, st);
  double2* oamp = dalloc<double2>(2 * m, st);
  uint32_t* const result = reinterpret_cast<uint32_t*>(s->host_partials);
  k_sp_dense1_merge<W><<<sp_grid(m), SP_THREADS, 0, st>>>(s->key, uint32_t(m), g.q, at);
  NCSIM_LAUNCHED("sparse dense gate (merge)");
  k_sp_dense1_count<W><<<sp_grid(m + 1), SP_THREADS, 0, st>>>(s->key, s->amp, uint32_t(m), at, g, cut2, cnt);
  NCSIM_LAUNCHED("sparse dense gate (count)");
  size_t tb = 0;
  NCSIM_CUDA(cub::DeviceScan::ExclusiveSum(nullptr, tb, cnt, sum, int(m + 1), st));
  void* tmp = dalloc<uint8_t>(tb, st);
  NCSIM_CUDA(cub::DeviceScan::ExclusiveSum(tmp, tb, cnt, sum, int(m + 1), st));
  k_sp_dense1_place<W><<<sp_grid(m), SP_THREADS, 0, st>>>(s->key, s->amp, uint32_t(m), at, g, cnt, sum, okey, oamp, result);
  NCSIM_LAUNCHED("sparse dense gate (place)");
  dfree(tmp, st);
  dfree(at, st);
  dfree(cnt, st);
  dfree(sum, st);
  NCSIM_CUDA(cudaStreamSynchronize(st));
  take(s, okey, oamp, 2 * m, *result);
}

}  // namespace

namespace ncsim {

bool sparse_dense1(const LoweredOp& low, const std::vector<uint32_t>& qubits, SparseDense1& out) {
  if (low.kind != LoweredKind::Dense || qubits.size() != 1) return false;
  out.q = qubits[0];
  for (int i = 0; i < 4; ++i) {
    out.m[i] = low.matrix[i];
    if (low.matrix[i].re == 0.0 && low.matrix[i].im == 0.0) return false;
  }
  return true;
}

void sparse_apply_dense1(ncsim_sparse* s, const std::vector<SparseDense1>& gates) {
  if (gates.empty()) return;
  sparse_sort(s);
  const auto words = [&](auto f) {
    if (s->words == 1) return f(std::integral_constant<int, 1>{});
    if (s->words == 4) return f(std::integral_constant<int, 4>{});
    return f(std::integral_constant<int, 16>{});
  };
  for (size_t i = 0; i < gates.size() && s->m;) {
    if (2 * s->m <= SMALL_OUT) {
      i += words([&](auto w) { return apply_small<decltype(w)::value>(s, gates, i); });
    } else {
      words([&](auto w) {
        apply_large<decltype(w)::value>(s, gates[i]);
        return size_t(1);
      });
      ++i;
    }
  }
}

}  // namespace ncsim
