// FP64 trailing update of the multifrontal factorization on the integer tensor
// pipe (tcgen05 kind::i8), exact to FP64 level by residues (the Ozaki scheme II):
// every row of the outer panel X is scaled by a power of two and rounded to
// integers, the integer product X X^T is formed modulo kOzModuli coprime moduli of
// at most 256 (exact 8-bit products with 32-bit sums), and the tile F -= X X^T is
// put back together from its residues by the Chinese remainder theorem.
#pragma once
#include <cuda_runtime.h>

#include <cstdint>
#include <string>

namespace tdem {

// Device buffers and tensor maps of the residues (one set per factorization
// engine; factorizations using it must not overlap).
struct OzakiBuffers {
  int8_t* residues = nullptr;  // [kOzModuli][rows][kOzK]
  int* exps = nullptr;         // [rows] row exponents
  int64_t rows = 0;
  int sms = 0;                 // SMs of the device: CTAs of the persistent update
  alignas(64) unsigned char map_a[128] = {};  // CUtensorMap of 128-row operand boxes
  alignas(64) unsigned char map_b[128] = {};  // CUtensorMap of 48-row operand boxes
};

// Creates the tensor maps over residues/exps already allocated for `rows` rows and
// sets the kernels' shared-memory limits (current device).
std::string ozaki_setup(OzakiBuffers& ob);

// Reduces the outer-panel rows [J1, m) of every front of a task list (64 rows per
// CTA; aux[i] = the i-th front's first row in the buffer).
void launch_ozaki_residues(const double* L, const int64_t* l_off, const int* m, const int* k, const int* fronts,
                           const int64_t* prefix, const int64_t* aux, int count, int64_t ctas, int j0,
                           const OzakiBuffers& ob, cudaStream_t s);

// F[J1:m, J1:m] -= X X^T for the same fronts; tiles is the prefix total of the list
// (oz_tiles of each front); err[2] is set when a wait inside the kernel gave up.
void launch_ozaki_update(double* L, double* U, const int64_t* l_off, const int64_t* u_off, const int* m,
                         const int* k, const int* fronts, const int64_t* prefix, const int64_t* aux, int count,
                         int64_t tiles, int j0, const OzakiBuffers& ob, int* err, cudaStream_t s);

}  // namespace tdem
