// Dense 1-qubit gates of the sparse form (registers of any word count).
#pragma once

#include <cstdint>
#include <vector>

#include "host/ir.hpp"

struct ncsim_sparse;

namespace ncsim {

struct SparseDense1 {
  uint32_t q;
  CplxD m[4];  // row-major
};
// the gate as one of these: a 2 x 2 matrix without zero entries, on a qubit of the register
bool sparse_dense1(const LoweredOp& low, const std::vector<uint32_t>& qubits, SparseDense1& out);
// applies them in order (the entries end sorted, duplicates summed, zeros dropped)
void sparse_apply_dense1(ncsim_sparse* s, const std::vector<SparseDense1>& gates);
// sorts the entries (sparse.cu)
void sparse_sort(ncsim_sparse* s);

}  // namespace ncsim
