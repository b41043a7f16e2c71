// Optional instrumentation of the one-kernel decode step, off unless the library is built with
// -DDF_TIMING: globaltimer stamps at the phase boundaries of CTA 0.  Without that macro everything
// here expands to nothing.  The counters are private to the including translation unit; the
// read-out function (extern "C" tie_debug_df_stamps) is emitted where TIE_TIMING_DF_OWNER is defined
// (decode_fused.cu).
#pragma once

#include <cuda_runtime.h>

namespace tie {

#ifdef DF_TIMING
static __device__ unsigned long long g_df_stamps[16];
#define DF_STAMP(i)                                                                   \
	do {                                                                          \
		if (blockIdx.x == 0 && threadIdx.x == 0) {                            \
			unsigned long long t_;                                        \
			asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t_));        \
			g_df_stamps[i] = t_;                                          \
		}                                                                     \
	} while (0)
#else
#define DF_STAMP(i)
#endif

}  // namespace tie

#if defined(DF_TIMING) && defined(TIE_TIMING_DF_OWNER)
// Debug builds only: globaltimer stamps (ns) of CTA 0 at the phase boundaries of the last launch.
extern "C" int tie_debug_df_stamps(unsigned long long *out)
{
	if (cudaDeviceSynchronize() != cudaSuccess)
		return -1;
	return cudaMemcpyFromSymbol(out, tie::g_df_stamps, sizeof(unsigned long long) * 16) == cudaSuccess ? 0 : -1;
}
#endif
