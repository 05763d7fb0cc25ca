// Volume FFT passes (vol3d_fft.cuh): 100 to 160 points.
#include "vol3d_fft.cuh"

namespace nsst {

const V3Ops* v3_ops_mid(int n) {
  switch (n) {
    case 100: {
      static const V3Ops ops = V3Launch<100, false, true>::ops();
      return &ops;
    }
    case 108: {
      static const V3Ops ops = V3Launch<108, false, true>::ops();
      return &ops;
    }
    case 128: {
      static const V3Ops ops = V3Launch<128, true, false>::ops();
      return &ops;
    }
    case 140: {
      static const V3Ops ops = V3Launch<140, false, true>::ops();
      return &ops;
    }
    case 144: {
      static const V3Ops ops = V3Launch<144, true, true>::ops();
      return &ops;
    }
    case 160: {
      static const V3Ops ops = V3Launch<160, false, true>::ops();
      return &ops;
    }
    default:
      return nullptr;
  }
}

}  // namespace nsst
