// Volume FFT passes (vol3d_fft.cuh): the level sizes of the reference's padded grids.
#include "vol3d_fft.cuh"

namespace nsst {

const V3Ops* v3_ops_grid(int n) {
  switch (n) {
    case 22: {
      static const V3Ops ops = V3Launch<22, true, false>::ops();
      return &ops;
    }
    case 34: {
      static const V3Ops ops = V3Launch<34, true, false>::ops();
      return &ops;
    }
    case 44: {
      static const V3Ops ops = V3Launch<44, true, true>::ops();
      return &ops;
    }
    case 68: {
      static const V3Ops ops = V3Launch<68, true, false>::ops();
      return &ops;
    }
    case 88: {
      static const V3Ops ops = V3Launch<88, true, true>::ops();
      return &ops;
    }
    case 132: {
      static const V3Ops ops = V3Launch<132, true, false>::ops();
      return &ops;
    }
    case 136: {
      static const V3Ops ops = V3Launch<136, true, false>::ops();
      return &ops;
    }
    default:
      return nullptr;
  }
}

}  // namespace nsst
