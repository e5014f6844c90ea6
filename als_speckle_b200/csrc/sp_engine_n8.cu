// Engine kernels, standalone 2-D FFT, partial-coherence and registration kernels for
// N = 8 (see sp_engine_launch.cuh, sp_fft2.cuh, sp_coherence.cuh and sp_register.cuh).
#include "sp_engine_launch.cuh"
#include "sp_fft2.cuh"
#include "sp_coherence.cuh"
#include "sp_register.cuh"
namespace sp {
SP_DEFINE_SIZE(8)
SP_DEFINE_FFT2(8)
SP_DEFINE_PC(8)
SP_DEFINE_REG(8)
}  // namespace sp
