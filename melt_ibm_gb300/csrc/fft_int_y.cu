// fft_int_y.cu -- instances of the integer-pipe y passes (see fft_int.cuh).
#include "fft_int.cuh"

namespace mibm {

bool intfft_y(Ctx* c, const int4* tw, double2* spec, int sign) {
  switch (c->g.n2m) {
#define CASE(N) case N: intfft::launch_y<N>(c, (const intfft::Tw*)tw, spec, sign); return true;
    MIBM_INTFFT_SIZES(CASE)
#undef CASE
  }
  return false;
}

}  // namespace mibm
