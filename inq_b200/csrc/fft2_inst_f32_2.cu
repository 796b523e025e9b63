// FFT passes of some line lengths, single precision (spread over files for parallel builds).
#include "fft2.cuh"

namespace inqb {
namespace v2 {
template void launch_n<float, 16>(Ctx &, const Basis &, const PassArgs<float> &, Geom2, int);
template void launch_n<float, 28>(Ctx &, const Basis &, const PassArgs<float> &, Geom2, int);
template void launch_n<float, 32>(Ctx &, const Basis &, const PassArgs<float> &, Geom2, int);
template void launch_n<float, 48>(Ctx &, const Basis &, const PassArgs<float> &, Geom2, int);
template void launch_n<float, 50>(Ctx &, const Basis &, const PassArgs<float> &, Geom2, int);
template void launch_n<float, 96>(Ctx &, const Basis &, const PassArgs<float> &, Geom2, int);
}  // namespace v2
}  // namespace inqb
