// h2g_resident.cu -- the instantiations of k_resident (rows and plane pairs of a warp, stage, place of b)
// and the launch of the class numbering.
#include "h2g_resident.cuh"

namespace h2g {

namespace {
template <int R, int NP, bool BS>
const void* pick(int vm) {
  if (vm == 0) return (const void*)k_resident<R, NP, 0, BS>;
  if (vm == 1) return (const void*)k_resident<R, NP, 1, BS>;
  return (const void*)k_resident<R, NP, 2, BS>;
}
}  // namespace

// One pair of planes a warp: b in shared memory up to 5 rows, from its vector from 6 on (beside x and b of 6
// rows and 30 planes there is room for 152 classes, and some tiles of the stack have 435); two pairs: b in
// shared memory up to 2 rows.
const void* resident_kernel(int R, int np, int vm) {
  if (np == 1) {
    switch (R) {
      case 1: return pick<1, 1, true>(vm);
      case 2: return pick<2, 1, true>(vm);
      case 3: return pick<3, 1, true>(vm);
      case 4: return pick<4, 1, true>(vm);
      case 5: return pick<5, 1, true>(vm);
      case 6: return pick<6, 1, false>(vm);
      case 7: return pick<7, 1, false>(vm);
      case 8: return pick<8, 1, false>(vm);
      default: return nullptr;
    }
  }
  switch (R) {
    case 1: return pick<1, 2, true>(vm);
    case 2: return pick<2, 2, true>(vm);
    case 3: return pick<3, 2, false>(vm);
    case 4: return pick<4, 2, false>(vm);
    default: return nullptr;
  }
}

const void* resident_sor_kernel(int R, int np) {
  if (np == 1) {
    switch (R) {
      case 1: return (const void*)k_resident_sor<1, 1, true>;
      case 2: return (const void*)k_resident_sor<2, 1, true>;
      case 3: return (const void*)k_resident_sor<3, 1, true>;
      case 4: return (const void*)k_resident_sor<4, 1, true>;
      case 5: return (const void*)k_resident_sor<5, 1, true>;
      case 6: return (const void*)k_resident_sor<6, 1, false>;
      case 7: return (const void*)k_resident_sor<7, 1, false>;
      case 8: return (const void*)k_resident_sor<8, 1, false>;
      default: return nullptr;
    }
  }
  switch (R) {
    case 1: return (const void*)k_resident_sor<1, 2, true>;
    case 2: return (const void*)k_resident_sor<2, 2, true>;
    case 3: return (const void*)k_resident_sor<3, 2, false>;
    case 4: return (const void*)k_resident_sor<4, 2, false>;
    default: return nullptr;
  }
}

cudaError_t launch_tile_classes(cudaStream_t st, const Geo& g, const uint16_t* cls, uint16_t* lcls, uint16_t* list,
                                int* count, int R, int nxb, int ntj) {
  k_tile_classes<<<nxb * ntj, 256, 0, st>>>(g, cls, lcls, list, count, R, nxb);
  return cudaGetLastError();
}

}  // namespace h2g
