// Volume FFT passes (vol3d_fft.cuh): 192 and 216 points.
#include "vol3d_fft.cuh"

namespace nsst {

const V3Ops* v3_ops_large(int n) {
  switch (n) {
    case 192: {
      static const V3Ops ops = V3Launch<192, true, true>::ops();
      return &ops;
    }
    case 216: {
      static const V3Ops ops = V3Launch<216, false, true>::ops();
      return &ops;
    }
    default:
      return nullptr;
  }
}

}  // namespace nsst
