// Momentum families of VdaggerV: which operators share one pass over the
// eigenvectors.
//
// VdaggerV of momentum p is M_p(i, j) = sum_x e^{-ip.x} conj(V_i(x)) V_j(x)
// (src/OperatorFactory.cpp:292-300).  A family sums the lattice plane by plane,
//   G_h(i, j) = sum_{x in plane h} phase_w(x) conj(V_i(x)) V_j(x),
// and every operator of the family is a Fourier sum over the planes,
//   M_p = sum_h e^{-2 pi i k h / n_planes} G_h,
// so operators that differ only in k cost one pass together.  Without a phase
// (w = 0) G_h is Hermitian and only i <= j is computed.
#pragma once

#include <cstdint>
#include <vector>

namespace slaph {
namespace dev {

constexpr int kVdvFamilyOps = 8;

struct VdvFamily {
  // Planes of constant h along `axis` (0..2): with u, v the other two
  // coordinates in increasing axis order, x_axis = sgn (h - sh_u u - sh_v v)
  // modulo the extent.  axis 3: one plane, the whole lattice.
  int32_t axis, n_planes, sgn, sh_u, sh_v;
  int32_t w[3];  // momentum of the phase that stays inside the plane sums
  int32_t herm;  // w = 0 and B = V: G_h is Hermitian
  int32_t n_ops;
  int32_t op[kVdvFamilyOps];   // operator id
  int32_t k[kVdvFamilyOps];    // Fourier index over the planes
  int32_t dag[kVdvFamilyOps];  // the operator is the conjugate transpose of the sum
};

// Planes with fewer entries than this are not worth a Fourier sum of their own
// (a K step of the kernels holds 16 entries): the lattice is one plane.
constexpr int64_t kVdvMinPlane = 48;
inline bool vdv_planes_along_x(int32_t Ly, int32_t Lz) {
  return 3LL * Ly * Lz >= kVdvMinPlane;
}

// Families of the operators `ids` (momenta mom[3 i..] of ids[i]) on an
// Lx x Ly x Lz lattice.  sheared: the planes may be any {p.x = h}, so that
// every momentum with a component +-1 has a Hermitian family of its own (half
// the work of a phase family); otherwise only planes of constant x.
std::vector<VdvFamily> vdv_families(std::vector<int32_t> const &ids,
                                    std::vector<int32_t> const &mom, int32_t Lx, int32_t Ly,
                                    int32_t Lz, bool sheared, int32_t max_ops);

}  // namespace dev
}  // namespace slaph
