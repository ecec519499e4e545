// fft_int_x.cu -- instances of the integer-pipe x passes (see fft_int.cuh);
// one translation unit per direction so that the two compile in parallel.
#include "fft_int.cuh"

namespace mibm {

bool intfft_x_fwd(Ctx* c, const int4* tw, const double* src, double2* spec) {
  switch (c->g.n1m) {
#define CASE(N) case N: intfft::launch_x_fwd<N>(c, (const intfft::Tw*)tw, src, spec); return true;
    MIBM_INTFFT_SIZES(CASE)
#undef CASE
  }
  return false;
}

bool intfft_x_inv(Ctx* c, const int4* tw, const double2* spec, double* dst) {
  switch (c->g.n1m) {
#define CASE(N) case N: intfft::launch_x_inv<N>(c, (const intfft::Tw*)tw, spec, dst); return true;
    MIBM_INTFFT_SIZES(CASE)
#undef CASE
  }
  return false;
}

}  // namespace mibm
