// Lead self-energies on the device for a Hermitian definite coupling H1 = s c 1 (square and cubic
// leads, and multi-orbital leads whose coupling is a multiple of the identity): the fast path of
// caroli-green/src/modes.rs:540-710. The eigenvectors Y of the cell Hamiltonian serve every
// energy; at energy E each transverse mode k has the roots λ of λ² - μ_k λ + 1 = 0 (classified on
// the host, O(n) scalar work), and
//   Σ_R = s c Y diag(λ_R) Y^†,   Σ_L = s c Y diag(1/λ_L) Y^†      (the products of modes.rs:696-713)
//   Γ = i (Σ - Σ^†),             W_R = Y[:, propagating] sqrt(-2 s c Im λ_R)   (W_R W_R^† = Γ_R)
// The O(n³) products Y diag(λ) Y^† are FP64 GEMMs on the tensor cores (ozgemm.cuh; lead_sigma in the engine).
#pragma once
#include <cstdint>

namespace caroli {

// Γ = i (S - S^†), n x n.
__global__ void lead_gamma_kernel(const double2* __restrict__ S, int n, double2* __restrict__ G) {
  const int64_t idx = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (idx >= (int64_t)n * n) return;
  const int i = (int)(idx % n), j = (int)(idx / n);
  const double2 a = S[i + (int64_t)j * n], b = S[j + (int64_t)i * n];
  // i ((a.x - b.x) + i (a.y + b.y)) = -(a.y + b.y) + i (a.x - b.x)
  G[idx] = make_double2(-(a.y + b.y), a.x - b.x);
}

// W[:, c] = Y[:, cols[c]] w[c], n x nc.
__global__ void lead_channels_kernel(const double2* __restrict__ Y, int n, const int32_t* __restrict__ cols,
                                     const double* __restrict__ w, int nc, double2* __restrict__ W) {
  const int64_t idx = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (idx >= (int64_t)n * nc) return;
  const int i = (int)(idx % n), c = (int)(idx / n);
  const double2 y = Y[i + (int64_t)cols[c] * n];
  W[idx] = make_double2(y.x * w[c], y.y * w[c]);
}

}  // namespace caroli
