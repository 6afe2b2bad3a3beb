// What the library's translation units share on the host: errors, launch
// accounting, per-class timing, twiddle tables and the shared-memory opt-in
// (defined in bnufft.cu).
#pragma once

#include <atomic>
#include <utility>

#include <cuda_runtime.h>

#include "../../include/bnufft.h"

namespace bn {

extern std::atomic<long> g_launches;

// sets the thread's error message and returns code
int fail(int code, const char* fmt, ...);

// an event to pass to prof_end when the kernel class is being timed, else null
cudaEvent_t prof_begin(const char* kind, cudaStream_t st);
void prof_end(cudaEvent_t e, cudaStream_t st);

// exp(-2 pi i m / L) on the current device
int get_twiddles(int L, const float2** out);

// opt in to large dynamic shared memory, once per kernel and device
int opt_in_smem(const void* kernel);

template <typename K>
int prep_kernel(K kernel, size_t)
{
	return opt_in_smem((const void*)kernel);
}

// While a solver's loop body is captured (by this thread), its kernels are
// launched so that one may start while the previous one drains (pdl_wait).
extern thread_local bool g_chain;

struct ChainScope {

	bool before;
	ChainScope() : before(g_chain) { g_chain = true; }
	~ChainScope() { g_chain = before; }
};

template <typename... P, typename... A>
void launch_chained(void (*kern)(P...), dim3 grid, dim3 block, size_t smem, cudaStream_t st, A&&... args)
{
	if (!g_chain) {

		kern<<<grid, block, smem, st>>>(std::forward<A>(args)...);
		return;
	}

	cudaLaunchAttribute at = {};
	at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
	at.val.programmaticStreamSerializationAllowed = 1;
	cudaLaunchConfig_t cfg = {};
	cfg.gridDim = grid;
	cfg.blockDim = block;
	cfg.dynamicSmemBytes = smem;
	cfg.stream = st;
	cfg.attrs = &at;
	cfg.numAttrs = 1;
	cudaLaunchKernelEx(&cfg, kern, P(args)...);
}

} // namespace bn

#define CUDA_TRY(call) do { cudaError_t e_ = (call); if (cudaSuccess != e_) \
	return fail(BNUFFT_ERR_CUDA, "%s:%d %s: %s", __FILE__, __LINE__, #call, cudaGetErrorString(e_)); } while (0)

#define LAUNCHED() do { g_launches.fetch_add(1, std::memory_order_relaxed); \
	cudaError_t e_ = cudaGetLastError(); if (cudaSuccess != e_) \
	return fail(BNUFFT_ERR_CUDA, "%s:%d launch: %s", __FILE__, __LINE__, cudaGetErrorString(e_)); } while (0)

#define TRY(call) do { int s_ = (call); if (BNUFFT_OK != s_) return s_; } while (0)
