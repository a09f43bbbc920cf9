// Grouping of momenta into VdaggerV families (vdv_families.hpp).
#include "../kernels/vdv_families.hpp"

#include <algorithm>
#include <cstdlib>
#include <map>
#include <utility>

namespace slaph {
namespace dev {

namespace {

VdvFamily family(int32_t axis, int32_t n_planes) {
  VdvFamily f{};
  f.axis = axis;
  f.n_planes = n_planes;
  f.sgn = 1;
  return f;
}

void add(VdvFamily &f, int32_t op, int32_t k, int32_t dag) {
  f.op[f.n_ops] = op;
  f.k[f.n_ops] = k;
  f.dag[f.n_ops] = dag;
  ++f.n_ops;
}

}  // namespace

std::vector<VdvFamily> vdv_families(std::vector<int32_t> const &ids,
                                    std::vector<int32_t> const &mom, int32_t Lx, int32_t Ly,
                                    int32_t Lz, bool sheared, int32_t max_ops) {
  int32_t const L[3] = {Lx, Ly, Lz};
  bool const cubic = Lx == Ly && Lx == Lz;
  auto plane = [&](int a) { return 3LL * Lx * Ly * Lz / L[a]; };
  std::vector<VdvFamily> out;
  struct Member {
    int32_t id, k, dag;
    int32_t p[3];
  };
  // Operators along one axis: Hermitian planes of that axis (x only without
  // sheared planes); the others by the sign class of (py, pz).
  std::vector<Member> along[3];
  std::map<std::pair<int32_t, int32_t>, std::vector<Member>> classes;
  std::vector<Member> whole;
  for (size_t i = 0; i < ids.size(); ++i) {
    int32_t const *p = &mom[3 * i];
    Member m{ids[i], 0, 0, {p[0], p[1], p[2]}};
    int axis = -1;
    for (int a = 0; a < 3; ++a) {
      bool const only = p[(a + 1) % 3] == 0 && p[(a + 2) % 3] == 0;
      if (only && axis < 0 && (a == 0 || sheared) && plane(a) >= kVdvMinPlane) axis = a;
    }
    if (axis >= 0) {
      m.k = p[axis];
      along[axis].push_back(m);
    } else if (!vdv_planes_along_x(Ly, Lz)) {
      whole.push_back(m);
    } else {
      std::pair<int32_t, int32_t> key{p[1], p[2]};
      m.k = p[0];
      if (key < std::make_pair(-p[1], -p[2])) {
        key = {-p[1], -p[2]};
        m.k = -p[0];
        m.dag = 1;
      }
      classes[key].push_back(m);
    }
  }
  size_t const per_family = static_cast<size_t>(std::clamp(max_ops, 1, kVdvFamilyOps));
  auto emit = [&](VdvFamily const &proto, std::vector<Member> const &ms) {
    for (size_t b = 0; b < ms.size(); b += per_family) {
      VdvFamily f = proto;
      for (size_t e = b; e < std::min(ms.size(), b + per_family); ++e)
        add(f, ms[e].id, ms[e].k, ms[e].dag);
      out.push_back(f);
    }
  };
  for (int a = 0; a < 3; ++a)
    if (!along[a].empty()) {
      VdvFamily f = family(a, L[a]);
      f.herm = 1;
      emit(f, along[a]);
    }
  for (auto const &kv : classes) {
    std::vector<Member> rest;
    for (Member const &m : kv.second) {
      // A phase family costs one full pass, a Hermitian one half a pass: one
      // or two operators of a class take sheared planes {p.x = h} each.
      int axis = -1;
      if (sheared && cubic && kv.second.size() < 3)
        for (int a = 0; a < 3 && axis < 0; ++a)
          if (std::abs(m.p[a]) == 1) axis = a;
      if (axis < 0) {
        rest.push_back(m);
        continue;
      }
      VdvFamily f = family(axis, L[axis]);
      f.sgn = m.p[axis];
      f.sh_u = m.p[axis == 0 ? 1 : 0];
      f.sh_v = m.p[axis == 2 ? 1 : 2];
      f.herm = 1;
      add(f, m.id, 1, 0);
      out.push_back(f);
    }
    VdvFamily f = family(0, Lx);
    f.w[1] = kv.first.first;
    f.w[2] = kv.first.second;
    emit(f, rest);
  }
  for (Member const &m : whole) {
    VdvFamily f = family(3, 1);
    for (int a = 0; a < 3; ++a) f.w[a] = m.p[a];
    f.herm = m.p[0] == 0 && m.p[1] == 0 && m.p[2] == 0;
    add(f, m.id, 0, 0);
    out.push_back(f);
  }
  return out;
}

}  // namespace dev
}  // namespace slaph
