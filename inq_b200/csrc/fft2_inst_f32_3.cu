// FFT passes of some line lengths, single precision (spread over files for parallel builds).
#include "fft2.cuh"

namespace inqb {
namespace v2 {
template void launch_n<float, 18>(Ctx &, const Basis &, const PassArgs<float> &, Geom2, int);
template void launch_n<float, 24>(Ctx &, const Basis &, const PassArgs<float> &, Geom2, int);
template void launch_n<float, 35>(Ctx &, const Basis &, const PassArgs<float> &, Geom2, int);
template void launch_n<float, 75>(Ctx &, const Basis &, const PassArgs<float> &, Geom2, int);
template void launch_n<float, 98>(Ctx &, const Basis &, const PassArgs<float> &, Geom2, int);
template void launch_n<float, 126>(Ctx &, const Basis &, const PassArgs<float> &, Geom2, int);
}  // namespace v2
}  // namespace inqb
