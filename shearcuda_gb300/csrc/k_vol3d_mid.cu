// Volume FFT passes (vol3d_fft.cuh): 128 and 144 points.
#include "vol3d_fft.cuh"

namespace nsst {

const V3Ops* v3_ops_mid(int n) {
  switch (n) {
    case 128: {
      static const V3Ops ops = V3Launch<128, true, true>::ops();
      return &ops;
    }
    case 144: {
      static const V3Ops ops = V3Launch<144, true, true>::ops();
      return &ops;
    }
    default:
      return nullptr;
  }
}

}  // namespace nsst
