// Fused FFT passes over the 2x oversampled grid (row passes, column passes,
// the Toeplitz column pass) and what they share with the other kernels: index
// maps, block sums, the device-side CG state. The kernels are templates of the
// FFT length; passes.cu instantiates them. For the grid convention see
// nufft_kernels.cuh.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include "fft_core.cuh"

namespace bn {

// A DFT of logical length n run on the FFT of the kernel's template length L
// (a power of two or a mixed length). n == L: the FFT itself. n < L (any n
// with 2n - 1 <= L):
// Bluestein's chirp-z algorithm (IEEE Trans. Audio Electroacoust. 18(4),
// 1970): with c_j = exp(-i pi j^2 / n), the forward DFT is
//   X_k = c_k sum_j (x_j c_j) conj(c_{k-j}),
// a linear convolution computed as a length-L circular one:
//   X = c . IFFT_L(FFT_L(c . x) . bf),  bf = FFT_L(conj(c) wrapped) / L,
// and the inverse DFT the same with conj(c) and bi = FFT_L(c wrapped) / L.
// Positions j >= n hold zeros before and after.
struct Dft {

	int n;			// logical length
	const float2* chirp;	// [n] c_j (Bluestein only)
	const float2* bf;	// [L] forward filter spectrum / L
	const float2* bi;	// [L] inverse filter spectrum / L
};

// Spectrum-side registers of a pass and their positions: those of the FFT, or
// the input's own ones for Bluestein (whose two transforms chain inside)
__host__ __device__ constexpr int out_regs(int L, bool BLUE) { return BLUE ? 8 : spec_regs(L); }

template <int L, typename LAY, bool BLUE>
__device__ __forceinline__ int out_pos(int m)
{
	if constexpr (BLUE)
		return reg_pos<L, LAY>(m);
	else
		return spec_pos<L, LAY>(m);
}

// Bluestein DFT of v in place; the caller has loaded zeros at positions >= d.n
// and gets zeros there back. Same barrier contract as fft_regs. Its two
// transforms take the shorter twiddle products (twiddle_short), powers of two
// too: the Toeplitz PSF's transforms of 4N points are often Bluestein's, and its
// error stays in every iteration (normal operator at 320^2, 294^2 and 230^2: 4.5e-7,
// 5.8e-7 and 7.8e-7 with chained powers, 3.8e-7, 5.0e-7 and 6.8e-7 so; 1 % slower).
template <int L, typename LAY, bool INV>
__device__ __forceinline__ void bluestein(float2 (&v)[8], float2* s, const float2* tw, const Dft& d)
{
#pragma unroll
	for (int m = 0; m < 8; m++) {

		int p = reg_pos<L, LAY>(m);
		float2 c = (p < d.n) ? d.chirp[p] : make_float2(0.f, 0.f);
		v[m] = INV ? cmulc(v[m], c) : cmul(v[m], c);
	}

	float2 w[spec_regs(L)];
	fft_fwd<L, LAY, true>(v, w, s, tw);
	const float2* b = INV ? d.bi : d.bf;
#pragma unroll
	for (int m = 0; m < spec_regs(L); m++)
		w[m] = cmul(w[m], b[min(spec_pos<L, LAY>(m), L - 1)]);

	fft_inv<L, LAY, true>(w, v, s, tw);
#pragma unroll
	for (int m = 0; m < 8; m++) {

		int p = reg_pos<L, LAY>(m);
		float2 c = (p < d.n) ? d.chirp[p] : make_float2(0.f, 0.f);
		v[m] = INV ? cmulc(v[m], c) : cmul(v[m], c);
	}
}

// forward DFT of v (positions reg_pos(m)) into w (positions out_pos(m)), and
// the inverse from w to v. half_in: registers 2..5 of v are known zeros.
template <int L, typename LAY, bool BLUE>
__device__ __forceinline__ void dft_fwd(float2 (&v)[8], float2 (&w)[out_regs(L, BLUE)], float2* s, const float2* tw,
		const Dft& d, bool half_in = false)
{
	if constexpr (BLUE) {

		bluestein<L, LAY, false>(v, s, tw, d);
#pragma unroll
		for (int m = 0; m < 8; m++)
			w[m] = v[m];

	} else {

		fft_fwd<L, LAY>(v, w, s, tw, half_in);
	}
}

template <int L, typename LAY, bool BLUE>
__device__ __forceinline__ void dft_inv(float2 (&w)[out_regs(L, BLUE)], float2 (&v)[8], float2* s, const float2* tw,
		const Dft& d)
{
	if constexpr (BLUE) {
#pragma unroll
		for (int m = 0; m < 8; m++)
			v[m] = w[m];

		bluestein<L, LAY, true>(v, s, tw, d);

	} else {

		fft_inv<L, LAY>(w, v, s, tw);
	}
}

// Element layouts ------------------------------------------------------------

// smem element stride for B sequences: odd, so 8-byte accesses of a
// half-warp land in distinct banks
__host__ __device__ __forceinline__ int smem_stride(int B) { return B | 1; }

// position of input element n (of n_in) inside the length-L transform
__device__ __forceinline__ int wrap_pos(int n, int n_in, int L)
{
	int p = n - n_in / 2;
	return (p < 0) ? p + L : p;
}

// inverse of wrap_pos: which input element sits at position p (>= n_in: none)
__device__ __forceinline__ int unwrap_pos(int p, int n_in, int L)
{
	int n = p + n_in / 2;
	return (n >= L) ? n - L : n;
}

// float64 block reduction; the result is valid in thread 0. blockDim.x must be
// a multiple of 32.
__device__ __forceinline__ double block_sum_d(double v, double* sh)
{
	for (int o = 16; o > 0; o >>= 1)
		v += __shfl_down_sync(0xffffffffu, v, o);

	__syncthreads();

	if (0 == threadIdx.x % 32)
		sh[threadIdx.x / 32] = v;

	__syncthreads();

	double r = 0.;

	if (threadIdx.x < 32) {

		r = (threadIdx.x < blockDim.x / 32) ? sh[threadIdx.x] : 0.;

		for (int o = 16; o > 0; o >>= 1)
			r += __shfl_down_sync(0xffffffffu, r, o);
	}

	return r;
}

// fixed-order sum of n float64 partials, the same value in every thread
__device__ __forceinline__ double sum_partials_d(const double* part, int n, double* sh)
{
	double v = 0.;

	for (int i = threadIdx.x; i < n; i += blockDim.x)
		v += part[i];

	double r = block_sum_d(v, sh);

	if (0 == threadIdx.x)
		sh[0] = r;

	__syncthreads();
	r = sh[0];
	__syncthreads();
	return r;
}

// flexible CG: largest truncation (directions kept) and ring size
enum { FCG_MAX_M = 16, FCG_RING = FCG_MAX_M + 1 };

// device-side state of the CG solve
struct CgScalars {

	double rs[2];		// ||r||^2 of iteration it in rs[it & 1]
	double eps2;		// stop when ||r||^2 <= eps2
	double b2;		// ||A^H y||^2
	int done;		// set once converged (or p^H A p == 0)
	int iters;		// iterations completed
	int it;			// iteration being run (device-driven loop)
	int maxiter;		// iteration limit of the current solve
	double pap_hist[FCG_RING];	// <p_j, (A^H A + lambda) p_j>, slot j % FCG_RING (flexible CG)
	double best_rs;		// smallest ||r||^2 so far (flexible CG stall test)
	double best_hist[4];	// best_rs after iteration j, slot j % 4
	int best_it;		// iteration count at best_rs
	int net_off;		// learned preconditioner switched off (stall fallback)
	int restart_it;		// flexible CG direction history starts here
	int net_iters;		// learned preconditioner used in iterations < net_iters (0: no limit)
	float rnorm;		// ||r|| of the current residual
	float rinv;		// 1 / ||r|| (0 for r = 0)
	float scale;		// data scaling used
	float inv_scale;	// float(1 / scale)
	int f32;		// plain CG keeps ||r||^2, p^H A p, alpha and beta in float32
};

// iteration index of a CG pass: the host's, or the device counter when the
// loop runs inside a graph (it < 0)
__device__ __forceinline__ int cg_iter(int it, const CgScalars* st) { return (it < 0) ? st->it : it; }

// Plain-CG scalars in the reference's precision when st->f32 is set:
// conjgrad (src/iter/italgos.c:518-554) sums its dot products in float64
// but stores rsold, rsnew, pAp, alpha and beta as float, and divides in
// float. cg_keep rounds a float64 sum as the reference stores it; cg_ratio
// is alpha = rsold / pAp or beta = rsnew / rsold.
__device__ __forceinline__ double cg_keep(const CgScalars* st, double v)
{
	return st->f32 ? (double)(float)v : v;
}

__device__ __forceinline__ float cg_ratio(const CgScalars* st, double num, double den)
{
	return st->f32 ? __fdiv_rn((float)num, (float)den) : (float)(num / den);
}

// three fixed-order float64 sums of partials in one block reduction, the
// same values in every thread (sh: 3 doubles per warp)
__device__ __forceinline__ double3 sum_partials3_d(const double* a, int na, const double* b, int nb,
		const double* c, int nc, double* sh)
{
	double3 v = make_double3(0., 0., 0.);
	const int n = max(na, max(nb, nc));

	for (int i = threadIdx.x; i < n; i += blockDim.x) {

		if (i < na)
			v.x += a[i];

		if (i < nb)
			v.y += b[i];

		if (i < nc)
			v.z += c[i];
	}

	for (int o = 16; o > 0; o >>= 1) {

		v.x += __shfl_down_sync(0xffffffffu, v.x, o);
		v.y += __shfl_down_sync(0xffffffffu, v.y, o);
		v.z += __shfl_down_sync(0xffffffffu, v.z, o);
	}

	__syncthreads();

	if (0 == threadIdx.x % 32) {

		sh[3 * (threadIdx.x / 32) + 0] = v.x;
		sh[3 * (threadIdx.x / 32) + 1] = v.y;
		sh[3 * (threadIdx.x / 32) + 2] = v.z;
	}

	__syncthreads();
	double3 r = make_double3(0., 0., 0.);

	for (int w = 0; w < (int)(blockDim.x / 32); w++) {

		r.x += sh[3 * w + 0];
		r.y += sh[3 * w + 1];
		r.z += sh[3 * w + 2];
	}

	__syncthreads();
	return r;
}

// Row pass, forward, first step of a CG iteration (conjgrad,
// src/iter/italgos.c:538-566, reordered so that the direction update of the
// previous iteration happens while loading):
//   it == 0: p = b;  else: rs = ||r||^2 (from the update's partials),
//   stop if rs <= eps2, beta = rs / rs_prev, p = r + beta p_prev.
// p_prev and p_cur are distinct buffers (blocks of other coils still read
// p_prev while coil 0 writes p_cur); the CG step copies p_cur back to p_prev.
// X <= L / 2 unless Bluestein (the grids are oversampled twofold or more).
// Rows of coil 0 write p and the partial ||p||^2 (for lambda ||p||^2 in
// p^H (A^H A + lambda) p); every row multiplies by its coil's map and runs the
// forward transform like k_rows_fwd.
template <int L, int B, bool BLUE>
__global__ void __launch_bounds__(B * L / 8, (1024 / (B * L / 8)) > 0 ? 1024 / (B * L / 8) : 1) k_rows_fwd_cg(const float2* __restrict__ bvec, const float2* r,
		const float2* p_prev, float2* p_cur, const float2* __restrict__ maps,
		const float* __restrict__ ax, const float* __restrict__ ayz,
		int X, long YZ, long R, float2* out, const float2* __restrict__ twg,
		CgScalars* st, int it, const double* rs_part, int nrs, double* pp_part, Dft d)
{
	pdl_wait();
	using LAY = RowLayout<L, B>;
	const int dn = BLUE ? d.n : L;	// logical DFT length (compile-time for the FFT itself)
	constexpr int NT = B * L / 8;
	extern __shared__ float2 smem[];
	__shared__ double red[32];
	float2* s = smem;
	float2* tw = smem + LAY::SMEM;

	const long row = (long)blockIdx.x * B + LAY::seq();
	const bool valid = (row < R);
	const long yz = valid ? row % YZ : 0;
	const long c = valid ? row / YZ : 0;

	// the inputs are on their way before the scalars are summed (their
	// barriers would otherwise hold the loads back); of a transform that is
	// zero-padded twofold or more only registers 0, 1, 6, 7 have any, of
	// Bluestein's (d.n <= (L + 1) / 2) the first five
	constexpr int NL = BLUE ? 5 : 4;
	auto reg = [](int l) { return BLUE ? l : ((l < 2) ? l : l + 4); };
	float2 rv[NL], po[NL], mv[NL];
	it = cg_iter(it, st);
	const int done = st->done;
	const float2* ri = (0 == it) ? bvec : r;
#pragma unroll
	for (int l = 0; l < NL; l++) {

		int p = reg_pos<L, LAY>(reg(l));
		int n = (p < dn) ? unwrap_pos(p, X, dn) : X;
		const bool in = valid && (n < X);
		const long i = n + X * yz;
		rv[l] = in ? ri[i] : make_float2(0.f, 0.f);
		po[l] = (in && (it > 0)) ? p_prev[i] : make_float2(0.f, 0.f);
		mv[l] = in ? maps[i + X * YZ * c] : make_float2(0.f, 0.f);
	}

	if (done)
		return;

	float beta = 0.f;

	if (it > 0) {

		double rs = cg_keep(st, sum_partials_d(rs_part, nrs, red));
		double rs_prev = st->rs[(it - 1) & 1];
		bool stop = (rs <= st->eps2);

		if (0 == blockIdx.x && 0 == threadIdx.x) {

			st->rs[it & 1] = rs;

			if (stop) {

				st->done = 1;
				st->iters = it;
			}
		}

		if (stop)
			return;

		beta = cg_ratio(st, rs, rs_prev);
	}

	for (int i = threadIdx.x; i < L; i += NT)
		tw[i] = twg[i];

	double pp = 0.;
	float2 v[8];
#pragma unroll
	for (int m = 0; m < 8; m++)
		v[m] = make_float2(0.f, 0.f);
#pragma unroll
	for (int l = 0; l < NL; l++) {

		int p = reg_pos<L, LAY>(reg(l));
		int n = (p < dn) ? unwrap_pos(p, X, dn) : X;

		if (valid && (n < X)) {

			float2 pv = rv[l];

			if (it > 0) {

				pv.x = fmaf(beta, po[l].x, pv.x);
				pv.y = fmaf(beta, po[l].y, pv.y);
			}

			if (0 == c) {

				p_cur[n + X * yz] = pv;
				pp += (double)pv.x * (double)pv.x + (double)pv.y * (double)pv.y;
			}

			float2 w = cmul(pv, mv[l]);
			v[reg(l)] = ax ? cscale(w, ax[n] * ayz[yz]) : w;
		}
	}

	// rows of coil 0 only are in the first blocks
	double t = 0.;

	if ((long)blockIdx.x * B < YZ)
		t = block_sum_d(pp, red);

	if (0 == threadIdx.x)
		pp_part[blockIdx.x] = t;

	float2 w[out_regs(L, BLUE)];
	dft_fwd<L, LAY, BLUE>(v, w, s, tw, d, 2 * X <= L);

	if (valid) {
#pragma unroll
		for (int m = 0; m < out_regs(L, BLUE); m++) {

			int p = out_pos<L, LAY, BLUE>(m);

			if (p < dn)
				out[p + (long)dn * row] = w[m];
		}
	}
}

// Row pass, forward ----------------------------------------------------------
//
// Rows r in [0, R): yz = r % YZ, c = r / YZ. Input row x in [0, X):
//   v = img[x + X*yz (+ X*YZ*c unless maps)] (* maps[x + X*yz + X*YZ*c])
//       * ax[x] * ayz[yz]                          (apodisation, optional)
// placed at wrap_pos(x, X, L), transformed, written to out[p + L*r].
// One block: B rows, B*L/8 threads; a warp reads and writes consecutive
// elements of one row straight from / into the FFT's registers.
template <int L, int B, bool BLUE>
__global__ void __launch_bounds__(B * L / 8, (1024 / (B * L / 8)) > 0 ? 1024 / (B * L / 8) : 1) k_rows_fwd(const float2* img, const float2* __restrict__ maps,
		const float* __restrict__ ax, const float* __restrict__ ayz,
		int X, long YZ, long R, float2* out, const float2* __restrict__ twg, const int* done, Dft d)
{
	pdl_wait();
	using LAY = RowLayout<L, B>;
	const int dn = BLUE ? d.n : L;	// logical DFT length (compile-time for the FFT itself)
	constexpr int NT = B * L / 8;
	extern __shared__ float2 smem[];
	float2* s = smem;
	float2* tw = smem + LAY::SMEM;

	const int stop = done ? *done : 0;	// tested once the loads are under way

	for (int i = threadIdx.x; i < L; i += NT)
		tw[i] = twg[i];

	const long row = (long)blockIdx.x * B + LAY::seq();
	const bool valid = (row < R);
	const long yz = valid ? row % YZ : 0;
	const long c = valid ? row / YZ : 0;
	float2 v[8];

#pragma unroll
	for (int m = 0; m < 8; m++) {

		int p = reg_pos<L, LAY>(m);
		int n = (p < dn) ? unwrap_pos(p, X, dn) : X;
		v[m] = make_float2(0.f, 0.f);

		if (valid && (n < X)) {

			float2 w = maps ? cmul(img[n + X * yz], maps[n + X * yz + X * YZ * c])
					: img[n + X * yz + X * YZ * c];
			v[m] = ax ? cscale(w, ax[n] * ayz[yz]) : w;
		}
	}

	if (stop)
		return;

	float2 w[out_regs(L, BLUE)];
	dft_fwd<L, LAY, BLUE>(v, w, s, tw, d, 2 * X <= L);

	if (valid) {
#pragma unroll
		for (int m = 0; m < out_regs(L, BLUE); m++) {

			int p = out_pos<L, LAY, BLUE>(m);

			if (p < dn)
				out[p + (long)dn * row] = w[m];
		}
	}
}

// Column pass ------------------------------------------------------------------
//
// Sequences (cx, o): cx in [0, W) contiguous columns, o in [0, O) outer index.
// Input element n of sequence (cx, o) is in[cx + n*ies + o*ios] for n < n_in,
// placed at wrap_pos(n, n_in, L) when wrap_in, else at n.
// MODE 0: forward FFT; 1: inverse FFT; 2: forward, * psf, inverse (Toeplitz).
// Output element n' < n_out is taken from position wrap_pos(n', n_out, L)
// when wrap_out, else n', and written to out[cx + n'*oes + o*oos].
// psf element for position p: psf[cx + p*pes + (o % pmod)*pos].
// One block: B columns of one outer index, B*L/8 threads; grid (ceil(W/B), O).
// Global loads go straight into the first FFT stage's registers and results
// leave from the last stage's registers (B consecutive columns per access).
// the Toeplitz column pass of three-stage lengths keeps two exchange buffers
// when they fit (fft_regs_db, mix_fwd)
__host__ __device__ constexpr bool cols_double_buffered(int MODE, bool BLUE, int L, int B)
{
	return (2 == MODE) && !BLUE && (L >= 128) && ((L <= 512) || is_mix(L))
		&& ((2 * L * (B | 1) + L) * 8 <= 200 * 1024);
}

template <int L, int B, int MODE, bool BLUE>
__global__ void __launch_bounds__(B * L / 8, (1024 / (B * L / 8)) > 0 ? 1024 / (B * L / 8) : 1) k_cols(const float2* in, long ies, long ios, int n_in, int wrap_in,
		float2* out, long oes, long oos, int n_out, int wrap_out,
		int W, const float2* __restrict__ psf, long pes, long pmod, long pos,
		const float2* __restrict__ twg, const int* done, Dft d)
{
	pdl_wait();
	using LAY = ColLayout<L, B>;
	const int dn = BLUE ? d.n : L;	// logical DFT length (compile-time for the FFT itself)
	constexpr int NT = B * L / 8;
	constexpr bool DB = cols_double_buffered(MODE, BLUE, L, B);
	extern __shared__ float2 smem[];
	float2* s = smem;
	float2* tw = smem + (DB ? 2 : 1) * LAY::SMEM;

	const int stop = done ? *done : 0;	// tested once the loads are under way

	for (int i = threadIdx.x; i < L; i += NT)
		tw[i] = twg[i];

	constexpr bool BY4 = (3 == MODE), FWD = (0 == MODE) || BY4;
	const int cx = BY4 ? blockIdx.x * (B / 4) + LAY::seq() % (B / 4) : blockIdx.x * B + LAY::seq();
	const bool valid = (cx < W);
	const long o = BY4 ? 4 * (long)blockIdx.y + LAY::seq() / (B / 4) : blockIdx.y;
	const float2* inp = in + o * ios + cx;

	// the input side holds reg_pos positions, the spectrum side out_pos ones:
	// MODE 0 loads the former and stores the latter, MODE 1 the reverse, MODE 2
	// loads and stores the former
	constexpr int NW = out_regs(L, BLUE);
	constexpr int NI = (1 == MODE) ? NW : 8, NO = FWD ? NW : 8;
	auto ipos = [](int m) { return (1 == MODE) ? out_pos<L, LAY, BLUE>(m) : reg_pos<L, LAY>(m); };
	auto opos = [](int m) { return FWD ? out_pos<L, LAY, BLUE>(m) : reg_pos<L, LAY>(m); };
	float2 x[NI], y[NO];
#pragma unroll
	for (int m = 0; m < NI; m++) {

		int p = ipos(m);
		int n = (p >= dn) ? n_in : (wrap_in ? unwrap_pos(p, n_in, dn) : p);
		x[m] = (valid && (n < n_in)) ? inp[n * ies] : make_float2(0.f, 0.f);
	}

	if (stop)
		return;

	const bool half = wrap_in && (2 * n_in <= L);

	if constexpr (FWD) {

		dft_fwd<L, LAY, BLUE>(x, y, s, tw, d, half);

	} else if constexpr (MODE == 1) {

		dft_inv<L, LAY, BLUE>(x, y, s, tw, d);

	} else if constexpr (DB) {	// Toeplitz with double-buffered exchanges; the PSF column loads first

		const float2* pp = psf + (o % pmod) * pos + cx;
		float2 pv[NW];
#pragma unroll
		for (int m = 0; m < NW; m++) {

			int p = out_pos<L, LAY, BLUE>(m);
			pv[m] = (valid && (p < dn)) ? pp[p * pes] : make_float2(0.f, 0.f);
		}

		if constexpr (is_mix(L)) {

			float2 w[NW];
			mix_fwd<L, LAY, true>(x, w, s, s + LAY::SMEM, tw, half);
#pragma unroll
			for (int m = 0; m < NW; m++)
				w[m] = cmul(w[m], pv[m]);

			mix_inv<L, LAY, true>(w, y, s, s + LAY::SMEM, tw);

		} else {

			fft_regs_db<L, LAY, false>(x, s, s + LAY::SMEM, tw, half);
#pragma unroll
			for (int m = 0; m < 8; m++)
				y[m] = cmul(x[m], pv[m]);

			fft_regs_db<L, LAY, true>(y, s, s + LAY::SMEM, tw);
		}

	} else {

		float2 w[NW];
		dft_fwd<L, LAY, BLUE>(x, w, s, tw, d, half);
		const float2* pp = psf + (o % pmod) * pos + cx;
#pragma unroll
		for (int m = 0; m < NW; m++) {

			int p = out_pos<L, LAY, BLUE>(m);

			if (valid && (p < dn))
				w[m] = cmul(w[m], pp[p * pes]);
		}

		dft_inv<L, LAY, BLUE>(w, y, s, tw, d);
	}

	float2* outp = BY4 ? out + 4 * (blockIdx.y * oos + cx) + o % 4 : out + o * oos + cx;
	oes *= BY4 ? 4 : 1;

	if (valid) {
#pragma unroll
		for (int m = 0; m < NO; m++) {

			int p = opos(m);
			int n = (p >= dn) ? n_out : (wrap_out ? unwrap_pos(p, n_out, dn) : p);

			if (n < n_out)
				outp[n * oes] = y[m];
		}
	}
}

// Row pass, inverse --------------------------------------------------------------
//
// Input rows in[p + L*(yz + YZ*c)], p < L. Each block takes B consecutive yz
// rows and coils [c0, c1) (a thread keeps its output pixels in registers
// across the coil loop): inverse FFT per row, keep x < X from
// wrap_pos(x, X, L), scale by ax[x]*ayz[yz] (optional) and either
//   MAPS:      accumulate sum_c conj(maps[x + X*yz + X*YZ*c]) * row
//              into out[x + X*yz + X*YZ*g] (g = blockIdx.y, partial per group)
//   else:      write out[x + X*yz + X*YZ*c] per coil.
// grid (ceil(YZ/B), groups); coils per group cpg.
template <int L, int B, bool BLUE, bool MAPS>
__global__ void __launch_bounds__(B * L / 8, (1024 / (B * L / 8)) > 0 ? 1024 / (B * L / 8) : 1) k_rows_inv(const float2* in, const float2* __restrict__ maps,
		const float* __restrict__ ax, const float* __restrict__ ayz,
		int X, long YZ, int C, int cpg, float2* out, const float2* __restrict__ twg,
		const float2* pdot, double* dot_part, const int* done, Dft d)
{
	pdl_wait();
	using LAY = RowLayout<L, B>;
	const int dn = BLUE ? d.n : L;	// logical DFT length (compile-time for the FFT itself)
	constexpr int NT = B * L / 8;
	constexpr int NW = out_regs(L, BLUE);
	// the coil sums belong to images of at most half the grid's side: all in
	// registers 0, 1, 6 and 7 (the last stage computes no others)
	constexpr int NA = (MAPS && !BLUE) ? 4 : 8;
	auto reg = [](int l) { return ((4 == NA) && (l >= 2)) ? l + 4 : l; };
	// the next coil's row is loaded while this one is transformed, where the
	// registers allow
	constexpr bool AHEAD = MAPS && !BLUE && !is_mix(L);
	extern __shared__ float2 smem[];
	__shared__ double red[32];
	float2* s = smem;
	float2* tw = smem + LAY::SMEM;

	const int stop = done ? *done : 0;	// tested once the loads are under way

	for (int i = threadIdx.x; i < L; i += NT)
		tw[i] = twg[i];

	const long yz = (long)blockIdx.x * B + LAY::seq();
	const bool valid = (yz < YZ);
	const int g = blockIdx.y;
	const int c0 = g * cpg;
	const int c1 = min(C, c0 + cpg);

	// this thread's output pixels: x = unwrap(jt + (L/8) m) where < X
	float2 acc[NA];
#pragma unroll
	for (int l = 0; l < NA; l++)
		acc[l] = make_float2(0.f, 0.f);

	double dot = 0.;
	float2 w[NW], nx[NW], v[8];

	auto load = [&](float2 (&u)[NW], int c) {
#pragma unroll
		for (int m = 0; m < NW; m++) {

			int p = out_pos<L, LAY, BLUE>(m);
			u[m] = (valid && (p < dn)) ? in[p + (long)dn * (yz + YZ * c)] : make_float2(0.f, 0.f);
		}
	};

	if (AHEAD)
		load(w, c0);

	for (int c = c0; c < c1; c++) {

		if (!AHEAD)
			load(w, c);
		else if (c + 1 < c1)
			load(nx, c + 1);

		if (stop)
			return;

		dft_inv<L, LAY, BLUE>(w, v, s, tw, d);

		if (valid) {
#pragma unroll
			for (int l = 0; l < NA; l++) {

				int p = reg_pos<L, LAY>(reg(l));
				int x = (p < dn) ? unwrap_pos(p, X, dn) : X;

				if (x >= X)
					continue;

				float2 t = v[reg(l)];

				if (ax)
					t = cscale(t, ax[x] * ayz[yz]);

				if (MAPS) {

					acc[l] = cadd(acc[l], cmulc(t, maps[x + X * yz + X * YZ * c]));

				} else {

					out[x + X * yz + X * YZ * c] = t;

					if (pdot) {	// Re<pdot, out> per coil (pdot == out: ||out||^2)

						float2 pv = ((const void*)pdot == (const void*)out) ? t : pdot[x + X * yz + X * YZ * c];
						dot += (double)pv.x * (double)t.x + (double)pv.y * (double)t.y;
					}
				}
			}
		}

		if (AHEAD) {
#pragma unroll
			for (int m = 0; m < NW; m++)
				w[m] = nx[m];
		}
	}

	if (MAPS) {

		if (valid) {
#pragma unroll
			for (int l = 0; l < NA; l++) {

				int p = reg_pos<L, LAY>(reg(l));
				int x = (p < dn) ? unwrap_pos(p, X, dn) : X;

				if (x >= X)
					continue;

				out[x + X * yz + X * YZ * g] = acc[l];

				if (pdot) {	// Re<p, partial> for the CG step length

					float2 pv = pdot[x + X * yz];
					dot += (double)pv.x * (double)acc[l].x + (double)pv.y * (double)acc[l].y;
				}
			}
		}
	}

	if (pdot) {

		double t = block_sum_d(dot, red);

		if (0 == threadIdx.x)
			dot_part[blockIdx.x + gridDim.x * blockIdx.y] = t;
	}
}

} // namespace bn
