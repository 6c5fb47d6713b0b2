// Runs of one-to-one ops of the sparse form (registers of any word count), built
// on the host as an op stream and applied by one kernel launch (sparse_run.cu).
#pragma once

#include <cstdint>
#include <vector>

#include "host/ir.hpp"

struct ncsim_sparse;

namespace ncsim {

// Collects consecutive ops that move every entry to one entry (monomial gates,
// permutations with phases, diagonals, Paulis) and applies them together.
class SlicedRun {
 public:
  bool empty() const { return !any_; }
  // empties the run; its buffers keep their capacity
  void reset();
  // empties the run and gives buffers of more than KEPT_BYTES back: a host thread's run outlives its circuits
  void release();
  // Adds a gate on the register's qubits; false when the gate creates entries or has no such form
  // (it then runs by itself).  `low` is the gate's lowering, on any qubit numbering.
  bool add_gate(const GateIR& g, const std::vector<uint32_t>& qubits, const LoweredOp& low);
  // i^phase X^x Z^z with the masks on `qubits` (bit j: qubits[j])
  void add_pauli(const std::vector<uint32_t>& qubits, uint64_t x, uint64_t z, uint32_t phase);
  // applies the run to the state's entries (queued on its stream) and empties it
  void launch(ncsim_sparse* s);

 private:
  static constexpr size_t KEPT_BYTES = size_t(1) << 20;
  struct Term {
    uint16_t q[3];
    uint8_t coeff;  // in 1/256 turns
  };
  uint32_t* put(uint32_t type, uint32_t words);  // an op of 4 + words words; its first word is set
  void touch(uint32_t q, bool write);
  void term(const std::vector<uint32_t>& factors, uint32_t coeff8);
  void flush_terms();
  void before_write(uint32_t q);
  void poly(const PhasePolyIR& p, const std::vector<uint32_t>& qubits);
  void product(const std::vector<std::vector<uint32_t>>& factors, uint64_t coeff, uint32_t big_bits);
  void flips(const std::vector<uint32_t>& qs);
  void control_not(uint32_t t, uint32_t c1, uint32_t c2);
  void put_not(uint32_t op);
  void table(const std::vector<uint32_t>& qubits, const std::vector<uint32_t>& image, const std::vector<CplxD>& ph);

  bool any_ = false, moves_ = false;
  std::vector<uint32_t> stream_;
  size_t nots_ = ~size_t(0);  // where the last list of NOTs starts
  std::vector<Term> pending_;
  uint64_t pending_mask_[16] = {};
  Phase scalar_;
  uint32_t bits_ = 0;  // of the phases counted so far (at most 8)
  uint32_t used_ = 0, changed_ = 0;  // 32-qubit blocks read or written, and written
  std::vector<uint16_t> image_;
  std::vector<double> phase_;
  std::vector<uint8_t> unit_;
  std::vector<uint8_t> blob_;
};

}  // namespace ncsim
