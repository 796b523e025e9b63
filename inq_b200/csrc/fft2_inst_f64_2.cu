// FFT passes of some line lengths, double precision (spread over files for parallel builds).
#include "fft2.cuh"

namespace inqb {
namespace v2 {
template void launch_n<double, 18>(Ctx &, const Basis &, const PassArgs<double> &, Geom2, int);
template void launch_n<double, 30>(Ctx &, const Basis &, const PassArgs<double> &, Geom2, int);
template void launch_n<double, 32>(Ctx &, const Basis &, const PassArgs<double> &, Geom2, int);
template void launch_n<double, 45>(Ctx &, const Basis &, const PassArgs<double> &, Geom2, int);
template void launch_n<double, 70>(Ctx &, const Basis &, const PassArgs<double> &, Geom2, int);
template void launch_n<double, 75>(Ctx &, const Basis &, const PassArgs<double> &, Geom2, int);
template void launch_n<double, 98>(Ctx &, const Basis &, const PassArgs<double> &, Geom2, int);
template void launch_n<double, 120>(Ctx &, const Basis &, const PassArgs<double> &, Geom2, int);
}  // namespace v2
}  // namespace inqb
