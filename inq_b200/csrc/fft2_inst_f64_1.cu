// FFT passes of some line lengths, double precision (spread over files for parallel builds).
#include "fft2.cuh"

namespace inqb {
namespace v2 {
template void launch_n<double, 16>(Ctx &, const Basis &, const PassArgs<double> &, Geom2, int);
template void launch_n<double, 25>(Ctx &, const Basis &, const PassArgs<double> &, Geom2, int);
template void launch_n<double, 40>(Ctx &, const Basis &, const PassArgs<double> &, Geom2, int);
template void launch_n<double, 48>(Ctx &, const Basis &, const PassArgs<double> &, Geom2, int);
template void launch_n<double, 64>(Ctx &, const Basis &, const PassArgs<double> &, Geom2, int);
template void launch_n<double, 72>(Ctx &, const Basis &, const PassArgs<double> &, Geom2, int);
template void launch_n<double, 96>(Ctx &, const Basis &, const PassArgs<double> &, Geom2, int);
template void launch_n<double, 126>(Ctx &, const Basis &, const PassArgs<double> &, Geom2, int);
}  // namespace v2
}  // namespace inqb
