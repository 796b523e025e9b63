// FFT passes of some line lengths, double precision (spread over files for parallel builds).
#include "fft2.cuh"

namespace inqb {
namespace v2 {
template void launch_n<double, 24>(Ctx &, const Basis &, const PassArgs<double> &, Geom2, int);
template void launch_n<double, 42>(Ctx &, const Basis &, const PassArgs<double> &, Geom2, int);
template void launch_n<double, 49>(Ctx &, const Basis &, const PassArgs<double> &, Geom2, int);
template void launch_n<double, 63>(Ctx &, const Basis &, const PassArgs<double> &, Geom2, int);
template void launch_n<double, 81>(Ctx &, const Basis &, const PassArgs<double> &, Geom2, int);
template void launch_n<double, 105>(Ctx &, const Basis &, const PassArgs<double> &, Geom2, int);
template void launch_n<double, 108>(Ctx &, const Basis &, const PassArgs<double> &, Geom2, int);
}  // namespace v2
}  // namespace inqb
