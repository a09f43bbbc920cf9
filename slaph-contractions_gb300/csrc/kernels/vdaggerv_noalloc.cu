// slaph_vdaggerv_noalloc: VdaggerV of one operator on one timeslice without
// any device allocation.
//
// Some callers cannot let a library allocate: hosts whose own allocator has
// reserved the device memory up front (a cudaMalloc here would fail or fight
// their pool), and latency-critical loops that cannot afford the device
// synchronisation cudaMalloc/cudaFree may imply.  The FP64 family kernel
// (vdv_fp64.cu) needs no memory beside its operands: the momentum family is a
// kernel argument, phases are formed in registers and the partial sums of a
// tile meet in the distributed shared memory of a cluster.
#include <cuda_runtime.h>

#include <cstdint>
#include <string>
#include <vector>

#include "../host/capi_util.hpp"
#include "kernels.cuh"

namespace {

void check(cudaError_t e, char const *what) {
  if (e != cudaSuccess) throw slaph::CudaError(std::string(what) + ": " + cudaGetErrorString(e));
}

// Largest lattice of the entry point (L^3 up to 64^3): the bound of its
// interface, from the static phase table that it was first built on.
constexpr size_t kMaxVolume = 262144;

}  // namespace

extern "C" int slaph_vdaggerv_noalloc(const slaph_dims *dims, const double *V_t,
                                      const int32_t *momentum, double *out, void *stream) {
  return slaph::guarded([&] {
    if (!dims || !V_t || !momentum || !out) throw slaph::ArgError("null argument");
    if (dims->Lx < 1 || dims->Ly < 1 || dims->Lz < 1 || dims->nev < 1)
      throw slaph::ArgError("invalid lattice or eigenvector count");
    // Each extent is bounded before the product is formed, so the product
    // (at most 2^54) cannot wrap.
    if (static_cast<size_t>(dims->Lx) > kMaxVolume || static_cast<size_t>(dims->Ly) > kMaxVolume ||
        static_cast<size_t>(dims->Lz) > kMaxVolume)
      throw slaph::ArgError("slaph_vdaggerv_noalloc: a lattice extent exceeds the static "
                            "scratch limit of " + std::to_string(kMaxVolume) + " sites (64^3)");
    size_t const vol = static_cast<size_t>(dims->Lx) * dims->Ly * dims->Lz;
    if (vol > kMaxVolume)
      throw slaph::ArgError("slaph_vdaggerv_noalloc: L^3 = " + std::to_string(vol) +
                            " exceeds the static scratch limit of " +
                            std::to_string(kMaxVolume) + " sites (64^3)");
    slaph::dev::Geometry g{};
    g.Lt = 1;
    g.Lx = dims->Lx;
    g.Ly = dims->Ly;
    g.Lz = dims->Lz;
    g.nev = dims->nev;
    g.dilE = dims->dilE > 0 ? dims->dilE : 1;
    g.n_rnd = 1;
    g.nb = 1;
    g.dim_row = 3LL * static_cast<int64_t>(vol);
    std::vector<slaph::dev::VdvFamily> const fam =
        slaph::dev::vdv_families({0}, {momentum[0], momentum[1], momentum[2]}, dims->Lx, dims->Ly,
                                 dims->Lz, true, slaph::dev::kVdvFp64Ops);
    check(slaph::dev::vdaggerv_fp64(reinterpret_cast<double2 *>(out),
                                    reinterpret_cast<double2 const *>(V_t), fam.data(),
                                    static_cast<int32_t>(fam.size()), 0, 1, g,
                                    static_cast<cudaStream_t>(stream)),
          "vdaggerv kernel");
  });
}
