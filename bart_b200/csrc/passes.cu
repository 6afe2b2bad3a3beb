// The FFT pass kernels of one group of lengths (PASS_GROUP, see passes.cuh).
#include "host.cuh"
#include "passes.cuh"

namespace bn {

namespace {

template <int L, int B>
int launch_rows_fwd_LB(const float2* img, const float2* maps, const float* ax, const float* ayz,
		int X, long YZ, long R, float2* out, cudaStream_t st, const int* done, const Dft& d)
{
	const float2* tw;
	TRY(get_twiddles(L, &tw));
	size_t smem = rows_smem(L, B);
	auto kern = (d.n == L) ? k_rows_fwd<L, B, false> : k_rows_fwd<L, B, true>;
	TRY(prep_kernel(kern, smem));
	cudaEvent_t pe = prof_begin("rows_fwd", st);
	launch_chained(kern, (unsigned)((R + B - 1) / B), B * L / 8, smem, st, img, maps, ax, ayz, X, YZ, R, out, tw, done, d);
	prof_end(pe, st);
	LAUNCHED();
	return BNUFFT_OK;
}

template <int L, int B, int MODE>
int launch_cols_LB(const float2* in, long ies, long ios, int n_in, int wrap_in,
		float2* out, long oes, long oos, int n_out, int wrap_out, int W, long O,
		const float2* psf, long pes, long pmod, long pos, const int* done, cudaStream_t st, const Dft& d)
{
	if constexpr ((3 == MODE) && (16 != B)) {

		return fail(BNUFFT_ERR_ARG, "internal: outputs by four images take 16 columns a block");

	} else {

		const float2* tw;
		TRY(get_twiddles(L, &tw));
		size_t smem = pass_smem(L, B);

		if ((d.n == L) && cols_double_buffered(MODE, false, L, B))
			smem += sizeof(float2) * (size_t)L * (size_t)smem_stride(B);	// the second exchange buffer

		auto kern = k_cols<L, B, MODE, false>;

		if constexpr (3 != MODE)
			kern = (d.n == L) ? kern : k_cols<L, B, MODE, true>;

		TRY(prep_kernel(kern, smem));

		if (O > 65535)
			return fail(BNUFFT_ERR_UNSUPPORTED, "column pass with %ld outer sequences", O);

		dim3 grid((unsigned)((3 == MODE) ? (W + B / 4 - 1) / (B / 4) : (W + B - 1) / B), (unsigned)O);
		cudaEvent_t pe = prof_begin((2 == MODE) ? "cols_toeplitz" : ((1 == MODE) ? "cols_inv" : "cols_fwd"), st);
		launch_chained(kern, grid, B * L / 8, smem, st, in, ies, ios, n_in, wrap_in, out, oes, oos, n_out, wrap_out,
				W, psf, pes, pmod, pos, tw, done, d);
		prof_end(pe, st);
		LAUNCHED();
		return BNUFFT_OK;
	}
}

template <int L, int B>
int launch_rows_inv_LB(const float2* in, const float2* maps, const float* ax, const float* ayz,
		int X, long YZ, int C, int cpg, float2* out, const float2* pdot, double* dot_part, const int* done,
		cudaStream_t st, const Dft& d)
{
	const float2* tw;
	TRY(get_twiddles(L, &tw));
	int groups = (C + cpg - 1) / cpg;
	size_t smem = rows_smem(L, B);
	auto kern = (d.n == L) ? (maps ? k_rows_inv<L, B, false, true> : k_rows_inv<L, B, false, false>)
			: (maps ? k_rows_inv<L, B, true, true> : k_rows_inv<L, B, true, false>);
	TRY(prep_kernel(kern, smem));
	dim3 grid((unsigned)((YZ + B - 1) / B), (unsigned)groups);
	cudaEvent_t pe = prof_begin("rows_inv", st);
	launch_chained(kern, grid, B * L / 8, smem, st, in, maps, ax, ayz, X, YZ, C, cpg, out, tw, pdot, dot_part, done, d);
	prof_end(pe, st);
	LAUNCHED();
	return BNUFFT_OK;
}

template <int L, int B>
int launch_rows_fwd_cg_LB(const float2* bvec, const float2* r, const float2* p_prev, float2* p_cur,
		const float2* maps, const float* ax, const float* ayz, int X, long YZ, long R, float2* out,
		CgScalars* stt, int it, const double* rs_part, int nrs, double* pp_part, cudaStream_t st, const Dft& d)
{
	const float2* tw;
	TRY(get_twiddles(L, &tw));
	size_t smem = rows_smem(L, B);
	auto kern = (d.n == L) ? k_rows_fwd_cg<L, B, false> : k_rows_fwd_cg<L, B, true>;
	TRY(prep_kernel(kern, smem));
	cudaEvent_t pe = prof_begin("rows_fwd", st);
	launch_chained(kern, (unsigned)((R + B - 1) / B), B * L / 8, smem, st, bvec, r, p_prev, p_cur, maps, ax, ayz,
			X, YZ, R, out, tw, stt, it, rs_part, nrs, pp_part, d);
	prof_end(pe, st);
	LAUNCHED();
	return BNUFFT_OK;
}

// run CALL with compile-time LL (FFT length) and BB (sequences per block)
#define DISPATCH_B(B, CALL) \
	switch (B) { \
	case 2: { constexpr int BB = 2; if constexpr (LL >= 4096 && BB * LL / 8 <= 1024) return CALL; break; } \
	case 4: { constexpr int BB = 4; if constexpr (BB * LL / 8 <= 1024 && BB * LL / 8 >= 32) return CALL; break; } \
	case 8: { constexpr int BB = 8; if constexpr (BB * LL / 8 <= 1024 && BB * LL / 8 >= 32) return CALL; break; } \
	case 16: { constexpr int BB = 16; if constexpr (BB * LL / 8 <= 1024 && BB * LL / 8 >= 32) return CALL; break; } \
	} \
	return fail(BNUFFT_ERR_ARG, "no FFT pass instance for L=%d B=%d", L, B);

#define CAT_(a, b) a##b
#define CAT(a, b) CAT_(a, b)

#define DISPATCH_LB(L, B) \
	switch (L) { \
	CAT(PASS_LENGTHS_, PASS_GROUP)(CASE_L) \
	default: break; } \
	return fail(BNUFFT_ERR_ARG, "no FFT pass instance for L=%d B=%d", L, B);

#define CASE_L(l) case l: { constexpr int LL = l; DISPATCH_B(B, PASS_CALL) }

int rows_fwd(int L, int B, const float2* img, const float2* maps, const float* ax, const float* ayz, int X, long YZ,
		long R, float2* out, cudaStream_t st, const int* done, const Dft& d)
{
#define PASS_CALL (launch_rows_fwd_LB<LL, BB>(img, maps, ax, ayz, X, YZ, R, out, st, done, d))
	DISPATCH_LB(L, B)
#undef PASS_CALL
}

template <int MODE>
int cols_mode(int L, int B, const float2* in, long ies, long ios, int n_in, int wrap_in, float2* out, long oes,
		long oos, int n_out, int wrap_out, int W, long O, const float2* psf, long pes, long pmod, long pos,
		const int* done, cudaStream_t st, const Dft& d)
{
#define PASS_CALL (launch_cols_LB<LL, BB, MODE>(in, ies, ios, n_in, wrap_in, out, oes, oos, n_out, wrap_out, W, O, psf, pes, \
		pmod, pos, done, st, d))
	DISPATCH_LB(L, B)
#undef PASS_CALL
}

int cols(int L, int B, int mode, const float2* in, long ies, long ios, int n_in, int wrap_in, float2* out, long oes,
		long oos, int n_out, int wrap_out, int W, long O, const float2* psf, long pes, long pmod, long pos,
		const int* done, cudaStream_t st, const Dft& d)
{
	auto f = (0 == mode) ? cols_mode<0> : ((1 == mode) ? cols_mode<1> : ((2 == mode) ? cols_mode<2> : cols_mode<3>));
	return f(L, B, in, ies, ios, n_in, wrap_in, out, oes, oos, n_out, wrap_out, W, O, psf, pes, pmod, pos, done, st, d);
}

int rows_inv(int L, int B, const float2* in, const float2* maps, const float* ax, const float* ayz, int X, long YZ,
		int C, int cpg, float2* out, const float2* pdot, double* dot_part, const int* done, cudaStream_t st,
		const Dft& d)
{
#define PASS_CALL (launch_rows_inv_LB<LL, BB>(in, maps, ax, ayz, X, YZ, C, cpg, out, pdot, dot_part, done, st, d))
	DISPATCH_LB(L, B)
#undef PASS_CALL
}

int rows_fwd_cg(int L, int B, const float2* bvec, const float2* r, const float2* p_prev, float2* p_cur,
		const float2* maps, const float* ax, const float* ayz, int X, long YZ, long R, float2* out, CgScalars* stt,
		int it, const double* rs_part, int nrs, double* pp_part, cudaStream_t st, const Dft& d)
{
#define PASS_CALL (launch_rows_fwd_cg_LB<LL, BB>(bvec, r, p_prev, p_cur, maps, ax, ayz, X, YZ, R, out, stt, it, rs_part, \
		nrs, pp_part, st, d))
	DISPATCH_LB(L, B)
#undef PASS_CALL
}

} // namespace

extern const PassTable CAT(pass_table_, PASS_GROUP);
const PassTable CAT(pass_table_, PASS_GROUP) = { rows_fwd, cols, rows_inv, rows_fwd_cg };

} // namespace bn
