// Volume FFT passes (vol3d_fft.cuh): 192 points and more.
#include "vol3d_fft.cuh"

namespace nsst {

const V3Ops* v3_ops_large(int n) {
  switch (n) {
    case 192: {
      static const V3Ops ops = V3Launch<192, true, false>::ops();
      return &ops;
    }
    case 204: {
      static const V3Ops ops = V3Launch<204, true, true>::ops();
      return &ops;
    }
    case 216: {
      static const V3Ops ops = V3Launch<216, true, true>::ops();
      return &ops;
    }
    case 256: {  // the convolution of the 216 grid
      static const V3Ops ops = V3Launch<256, false, true>::ops();
      return &ops;
    }
    default:
      return nullptr;
  }
}

}  // namespace nsst
