// Volume FFT passes (vol3d_fft.cuh): lengths up to 96.
#include "vol3d_fft.cuh"

namespace nsst {

const V3Ops* v3_ops(int n) {
  switch (n) {
    case 16: {
      static const V3Ops ops = V3Launch<16, true, false>::ops();
      return &ops;
    }
    case 24: {
      static const V3Ops ops = V3Launch<24, true, false>::ops();
      return &ops;
    }
    case 32: {
      static const V3Ops ops = V3Launch<32, true, true>::ops();
      return &ops;
    }
    case 48: {
      static const V3Ops ops = V3Launch<48, true, true>::ops();
      return &ops;
    }
    case 56: {
      static const V3Ops ops = V3Launch<56, false, true>::ops();
      return &ops;
    }
    case 64: {
      static const V3Ops ops = V3Launch<64, true, true>::ops();
      return &ops;
    }
    case 72: {
      static const V3Ops ops = V3Launch<72, true, true>::ops();
      return &ops;
    }
    case 80: {
      static const V3Ops ops = V3Launch<80, false, true>::ops();
      return &ops;
    }
    case 96: {
      static const V3Ops ops = V3Launch<96, true, false>::ops();
      return &ops;
    }
    default:
      if (const V3Ops* o = v3_ops_mid(n)) return o;
      if (const V3Ops* o = v3_ops_large(n)) return o;
      return v3_ops_grid(n);
  }
}

}  // namespace nsst
