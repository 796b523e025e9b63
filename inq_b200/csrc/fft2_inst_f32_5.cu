// FFT passes of some line lengths, single precision (spread over files for parallel builds).
#include "fft2.cuh"

namespace inqb {
namespace v2 {
template void launch_n<float, 21>(Ctx &, const Basis &, const PassArgs<float> &, Geom2, int);
template void launch_n<float, 30>(Ctx &, const Basis &, const PassArgs<float> &, Geom2, int);
template void launch_n<float, 40>(Ctx &, const Basis &, const PassArgs<float> &, Geom2, int);
template void launch_n<float, 60>(Ctx &, const Basis &, const PassArgs<float> &, Geom2, int);
template void launch_n<float, 64>(Ctx &, const Basis &, const PassArgs<float> &, Geom2, int);
template void launch_n<float, 105>(Ctx &, const Basis &, const PassArgs<float> &, Geom2, int);
}  // namespace v2
}  // namespace inqb
