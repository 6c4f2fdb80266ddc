// Setup-time R1CS data (see r1cs_setup.cpp).
#pragma once
#include <cstdint>
#include <vector>

// A column's row indices are in increasing order: those below 2^13 first, up
// to mid, then the others, each stored modulo 2^13. `order` deals the columns,
// longest first, to the kLcGroups groups in a back-and-forth, so the groups' entry
// counts agree; group g's columns are order[g_ptr[g] .. g_ptr[g + 1]).
constexpr int kLcGroups = 152;
struct HostCsc {
  std::vector<uint32_t> a_ptr, a_mid, b_ptr, b_mid;  // column pointers
  std::vector<uint16_t> a_idx, b_idx;                // row indices modulo 2^13
  std::vector<uint32_t> order, g_ptr;
};

// BLAKE3 statement digest of the BLAKE3 R1CS instance with 2^(m-14) blocks; cached per m.
void flock_statement_digest(int m, uint8_t out[32]);
// Column-major copies of A_0 and B_0 (built once).
const HostCsc& flock_host_csc();
