// Launchers of the FFT passes by length. Each translation unit built from
// passes.cu holds the kernels of one group of lengths behind one table.
#pragma once

#include "fft_passes.cuh"

namespace bn {

// L: FFT length, B: sequences per block; mode: 0 forward, 1 inverse, 2 Toeplitz, 3
// forward with the outputs of four outer sequences (coils) side by side (O: fours)
struct PassTable {

	int (*rows_fwd)(int L, int B, const float2* img, const float2* maps, const float* ax, const float* ayz, int X, long YZ,
			long R, float2* out, cudaStream_t st, const int* done, const Dft& d);
	int (*cols)(int L, int B, int mode, const float2* in, long ies, long ios, int n_in, int wrap_in, float2* out, long oes,
			long oos, int n_out, int wrap_out, int W, long O, const float2* psf, long pes, long pmod, long pos,
			const int* done, cudaStream_t st, const Dft& d);
	int (*rows_inv)(int L, int B, const float2* in, const float2* maps, const float* ax, const float* ayz, int X, long YZ,
			int C, int cpg, float2* out, const float2* pdot, double* dot_part, const int* done, cudaStream_t st,
			const Dft& d);
	int (*rows_fwd_cg)(int L, int B, const float2* bvec, const float2* r, const float2* p_prev, float2* p_cur,
			const float2* maps, const float* ax, const float* ayz, int X, long YZ, long R, float2* out, CgScalars* stt,
			int it, const double* rs_part, int nrs, double* pp_part, cudaStream_t st, const Dft& d);
};

extern const PassTable pass_table_0, pass_table_1, pass_table_2, pass_table_3, pass_table_4, pass_table_5, pass_table_6;

// dynamic shared memory of a column pass (ColLayout) / row pass (RowLayout), twiddles included
inline size_t pass_smem(int L, int B) { return sizeof(float2) * (size_t)L * (size_t)(smem_stride(B) + 1); }
inline size_t rows_smem(int L, int B) { return sizeof(float2) * ((size_t)B * (size_t)(L + L / 8) + (size_t)L); }

// the lengths of each group (balanced by compile time)
#define PASS_LENGTHS_0(X) X(16) X(32) X(64) X(128) X(256)
#define PASS_LENGTHS_1(X) X(512) X(1024)
#define PASS_LENGTHS_2(X) X(2048) X(4096) X(192)
#define PASS_LENGTHS_3(X) X(320) X(448)
#define PASS_LENGTHS_4(X) X(384) X(576)
#define PASS_LENGTHS_5(X) X(640)
#define PASS_LENGTHS_6(X) X(768)

// the table holding length L (one of the lengths above)
inline const PassTable* pass_table(int L)
{
#define PASS_CASE(l) case l:
	switch (L) {
	PASS_LENGTHS_0(PASS_CASE) return &pass_table_0;
	PASS_LENGTHS_1(PASS_CASE) return &pass_table_1;
	PASS_LENGTHS_2(PASS_CASE) return &pass_table_2;
	PASS_LENGTHS_3(PASS_CASE) return &pass_table_3;
	PASS_LENGTHS_4(PASS_CASE) return &pass_table_4;
	PASS_LENGTHS_5(PASS_CASE) return &pass_table_5;
	PASS_LENGTHS_6(PASS_CASE) return &pass_table_6;
	default: return nullptr;
	}
#undef PASS_CASE
}

} // namespace bn
