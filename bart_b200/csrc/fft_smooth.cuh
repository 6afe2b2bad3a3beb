// FFT passes of lengths n = a product of radices 2..13 that are no built
// length (fft_core.cuh): the oversampled grids 2N of ordinary even matrix
// sizes (400 = 8 5 10, 360 = 6 6 10, 308 = 4 7 11). Bluestein's algorithm needs
// two transforms of at least 2n - 1 points for them; here a pass runs the
// Stockham stages of n itself, with the radices as run-time data: every stage
// is a loop of the block's threads over its butterflies from one shared-memory
// buffer to the other, the radix a warp-uniform switch. Twiddle powers come
// from table entries and at most two products each, as in the mixed lengths.
// The row passes keep each sequence contiguous, the column pass interleaves
// the block's columns. A block has read its sequences before it writes them, so
// passes run in place too: in and out (and pdot) may be one array. Same positions, fusions and results (up to rounding) as
// the passes of fft_passes.cuh.
#pragma once

#include "fft_passes.cuh"

namespace bn {

enum { SM_STAGES = 6 };

// stages in order; magic: ceil(2^32 / m), so that j / m = umulhi(j, magic) for
// j m < 2^32, m > 1
struct SmoothPlan {

	int n, nst;
	int radix[SM_STAGES], ns[SM_STAGES];	// ns: product of the earlier radices
	unsigned ns_magic[SM_STAGES];		// of ns (0 for ns = 1)
	unsigned nb_magic[SM_STAGES];		// of the butterflies per sequence, n / radix
	unsigned n_magic;
};

__device__ __forceinline__ int magic_div(int j, unsigned magic) { return magic ? (int)__umulhi((unsigned)j, magic) : j; }

template <bool INV>
__device__ __forceinline__ void dft11(float2 (&x)[11])
{
	constexpr float c1 = 0.84125353283118116886f, c2 = 0.41541501300188642553f, c3 = -0.14231483827328514044f;
	constexpr float c4 = -0.65486073394528506406f, c5 = -0.95949297361449738989f;
	constexpr float s1 = 0.54064081745559758211f, s2 = 0.90963199535451837141f, s3 = 0.98982144188093273238f;
	constexpr float s4 = 0.75574957435425828377f, s5 = 0.28173255684142969771f;
	const float c[11] = { 1.f, c1, c2, c3, c4, c5, c5, c4, c3, c2, c1 };
	const float s[11] = { 0.f, s1, s2, s3, s4, s5, -s5, -s4, -s3, -s2, -s1 };
	dft_odd<11, INV>(x, c, s);
}

template <bool INV>
__device__ __forceinline__ void dft13(float2 (&x)[13])
{
	constexpr float c1 = 0.88545602565320989590f, c2 = 0.56806474673115580251f, c3 = 0.12053668025532305335f;
	constexpr float c4 = -0.35460488704253562597f, c5 = -0.74851074817110109863f, c6 = -0.97094181742605202716f;
	constexpr float s1 = 0.46472317204376854566f, s2 = 0.82298386589365639458f, s3 = 0.99270887409805399280f;
	constexpr float s4 = 0.93501624268541482344f, s5 = 0.66312265824079520238f, s6 = 0.23931566428755776715f;
	const float c[13] = { 1.f, c1, c2, c3, c4, c5, c6, c6, c5, c4, c3, c2, c1 };
	const float s[13] = { 0.f, s1, s2, s3, s4, s5, s6, -s6, -s5, -s4, -s3, -s2, -s1 };
	dft_odd<13, INV>(x, c, s);
}

template <int R, bool INV>
__device__ __forceinline__ void dft_small(float2 (&x)[R])
{
	if constexpr (2 == R)
		dft2<INV>(x);
	else if constexpr (4 == R)
		dft4<INV>(x);
	else if constexpr (8 == R)
		dft8<INV>(x);
	else if constexpr (11 == R)
		dft11<INV>(x);
	else if constexpr (13 == R)
		dft13<INV>(x);
	else
		dft_mix<R, INV>(x);
}

// u[i] *= w^i, w = tw[t] (conjugated for INV); entries t, 2t, 4t, 8t of the
// table of n and products of at most three of them
template <int R, bool INV>
__device__ __forceinline__ void twiddle_small(float2 (&u)[R], const float2* tw, int t)
{
	float2 e[4];
#pragma unroll
	for (int k = 0; k < 4; k++)
		if ((1 << k) < R) {

			e[k] = tw[t << k];

			if (INV)
				e[k].y = -e[k].y;
		}

	float2 w[R];
#pragma unroll
	for (int i = 1; i < R; i++) {

		const int hi = (i >= 8) ? 8 : ((i >= 4) ? 4 : ((i >= 2) ? 2 : 1));
		const float2 top = e[(8 == hi) ? 3 : ((4 == hi) ? 2 : ((2 == hi) ? 1 : 0))];
		w[i] = (i == hi) ? top : cmul(top, w[i - hi]);
		u[i] = cmul(u[i], w[i]);
	}
}

// shared-memory index of element p of sequence b: interleaved columns (COL) or
// padded rows of sl elements
template <bool COL, int B>
__device__ __forceinline__ int sm_idx(int p, int b, int sl)
{
	return COL ? p * (B | 1) + b : b * sl + p + (p >> 3);
}

__host__ __device__ __forceinline__ int sm_row(int n) { return n + n / 8 + 1; }

template <int R, bool INV, bool COL, int B>
__device__ __forceinline__ void sm_stage(const SmoothPlan& d, int s, const float2* src, float2* dst, const float2* tw,
		int sl)
{
	const int nb = d.n / R, ns = d.ns[s], step = nb / ns;

	for (int w = threadIdx.x; w < B * nb; w += blockDim.x) {

		const int b = COL ? w % B : magic_div(w, d.nb_magic[s]);
		const int j = COL ? w / B : w - b * nb;
		const int blk = magic_div(j, d.ns_magic[s]), k = j - blk * ns;
		float2 u[R];
#pragma unroll
		for (int i = 0; i < R; i++)
			u[i] = src[sm_idx<COL, B>(j + i * nb, b, sl)];

		if (ns > 1)
			twiddle_small<R, INV>(u, tw, k * step);

		dft_small<R, INV>(u);
		const int o = blk * ns * R + k;
#pragma unroll
		for (int i = 0; i < R; i++)
			dst[sm_idx<COL, B>(o + i * ns, b, sl)] = u[i];
	}
}

// all stages; the input is in a (complete: begins with a barrier); returns the
// buffer holding the result after a barrier
template <bool INV, bool COL, int B>
__device__ __forceinline__ float2* sm_fft(const SmoothPlan& d, float2* a, float2* b, const float2* tw, int sl)
{
	for (int s = 0; s < d.nst; s++) {

		__syncthreads();

		switch (d.radix[s]) {
#define BN_SM_CASE(r) case r: sm_stage<r, INV, COL, B>(d, s, a, b, tw, sl); break;
		BN_SM_CASE(2) BN_SM_CASE(3) BN_SM_CASE(4) BN_SM_CASE(5) BN_SM_CASE(6) BN_SM_CASE(7) BN_SM_CASE(8) BN_SM_CASE(9)
		BN_SM_CASE(10) BN_SM_CASE(11) BN_SM_CASE(12) BN_SM_CASE(13)
#undef BN_SM_CASE
		default: break;
		}

		float2* t = a;
		a = b;
		b = t;
	}

	__syncthreads();
	return a;
}

enum { SM_THREADS = 256 };

// k_rows_fwd (CG: k_rows_fwd_cg) for a smooth length: B rows per block
template <bool CG, int B>
__global__ void __launch_bounds__(SM_THREADS) k_srows_fwd(const float2* img, const float2* __restrict__ r,
		const float2* __restrict__ p_prev, float2* __restrict__ p_cur, const float2* __restrict__ maps,
		const float* __restrict__ ax, const float* __restrict__ ayz, int X, long YZ, long R, float2* out,
		const float2* __restrict__ twg, const int* done, CgScalars* st, int it, const double* __restrict__ rs_part,
		int nrs, double* __restrict__ pp_part, SmoothPlan d)
{
	extern __shared__ float2 smem[];
	__shared__ double red[32];
	const int sl = sm_row(d.n);
	float2 *s0 = smem, *s1 = smem + B * sl, *tw = smem + 2 * B * sl;
	float beta = 0.f;

	if constexpr (CG) {	// the direction update's scalars, as k_rows_fwd_cg

		if (st->done)
			return;

		it = cg_iter(it, st);

		if (it > 0) {

			const double rs = cg_keep(st, sum_partials_d(rs_part, nrs, red));
			const double rs_prev = st->rs[(it - 1) & 1];
			const bool stop = (rs <= st->eps2);

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

	} else {

		if (done && *done)
			return;
	}

	for (int i = threadIdx.x; i < d.n; i += SM_THREADS)
		tw[i] = twg[i];

	const long row0 = (long)blockIdx.x * B;
	double pp = 0.;

	for (int e = threadIdx.x; e < B * d.n; e += SM_THREADS) {

		const int b = magic_div(e, d.n_magic), p = e - b * d.n;
		const long row = row0 + b;
		const int x = unwrap_pos(p, X, d.n);
		float2 v = make_float2(0.f, 0.f);

		if ((row < R) && (x < X)) {

			const long yz = row % YZ, c = row / YZ, i = x + X * yz;

			if constexpr (CG) {

				float2 pv = img[i];

				if (it > 0) {

					const float2 rv = r[i], po = p_prev[i];
					pv.x = fmaf(beta, po.x, rv.x);
					pv.y = fmaf(beta, po.y, rv.y);
				}

				if (0 == c) {

					p_cur[i] = pv;
					pp += (double)pv.x * (double)pv.x + (double)pv.y * (double)pv.y;
				}

				v = cmul(pv, maps[i + X * YZ * c]);

			} else {

				v = maps ? cmul(img[i], maps[i + X * YZ * c]) : img[i + X * YZ * c];
			}

			if (ax)
				v = cscale(v, ax[x] * ayz[yz]);
		}

		s0[sm_idx<false, B>(p, b, sl)] = v;
	}

	if constexpr (CG) {

		const double t = block_sum_d(pp, red);

		if (0 == threadIdx.x)
			pp_part[blockIdx.x] = t;
	}

	const float2* y = sm_fft<false, false, B>(d, s0, s1, tw, sl);

	for (int e = threadIdx.x; e < B * d.n; e += SM_THREADS) {

		const int b = magic_div(e, d.n_magic), p = e - b * d.n;

		if (row0 + b < R)
			out[p + (long)d.n * (row0 + b)] = y[sm_idx<false, B>(p, b, sl)];
	}
}

// k_cols MODE 0 (forward) or 1 (inverse): B columns of one outer index
template <bool INV, int B>
__global__ void __launch_bounds__(SM_THREADS) k_scols(const float2* in, long ies, long ios, int n_in,
		int wrap_in, float2* out, long oes, long oos, int n_out, int wrap_out, int W,
		const float2* __restrict__ twg, const int* done, SmoothPlan d)
{
	extern __shared__ float2 smem[];
	float2 *s0 = smem, *s1 = smem + d.n * (B | 1), *tw = smem + 2 * d.n * (B | 1);

	if (done && *done)
		return;

	for (int i = threadIdx.x; i < d.n; i += SM_THREADS)
		tw[i] = twg[i];

	const int b = threadIdx.x % B;
	const int cx = blockIdx.x * B + b;
	const bool valid = (cx < W);
	const float2* inp = in + (long)blockIdx.y * ios + cx;

	for (int p = threadIdx.x / B; p < d.n; p += SM_THREADS / B) {

		const int i = wrap_in ? unwrap_pos(p, n_in, d.n) : p;
		s0[sm_idx<true, B>(p, b, 0)] = (valid && (i < n_in)) ? inp[i * ies] : make_float2(0.f, 0.f);
	}

	const float2* y = sm_fft<INV, true, B>(d, s0, s1, tw, 0);
	float2* outp = out + (long)blockIdx.y * oos + cx;

	if (!valid)
		return;

	for (int p = threadIdx.x / B; p < d.n; p += SM_THREADS / B) {

		const int i = wrap_out ? unwrap_pos(p, n_out, d.n) : p;

		if (i < n_out)
			outp[i * oes] = y[sm_idx<true, B>(p, b, 0)];
	}
}

// k_rows_inv: B rows and the coils of one group per block; the coil sums of
// the block's pixels are kept in shared memory, each by its own thread
template <int B>
__global__ void __launch_bounds__(SM_THREADS) k_srows_inv(const float2* in, const float2* __restrict__ maps,
		const float* __restrict__ ax, const float* __restrict__ ayz, int X, long YZ, int C, int cpg,
		float2* out, const float2* __restrict__ twg, const float2* pdot,
		double* __restrict__ dot_part, const int* done, unsigned x_magic, SmoothPlan d)
{
	extern __shared__ float2 smem[];
	__shared__ double red[32];
	const int sl = sm_row(d.n);
	float2 *s0 = smem, *s1 = smem + B * sl, *tw = smem + 2 * B * sl, *acc = tw + d.n;

	if (done && *done)
		return;

	for (int i = threadIdx.x; i < d.n; i += SM_THREADS)
		tw[i] = twg[i];

	const long yz0 = (long)blockIdx.x * B;
	const int c0 = blockIdx.y * cpg, c1 = min(C, c0 + cpg);
	double dot = 0.;

	for (int c = c0; c < c1; c++) {

		__syncthreads();	// the previous coil's result has been read

		for (int e = threadIdx.x; e < B * d.n; e += SM_THREADS) {

			const int b = magic_div(e, d.n_magic), p = e - b * d.n;
			s0[sm_idx<false, B>(p, b, sl)] = (yz0 + b < YZ) ? in[p + (long)d.n * (yz0 + b + YZ * c)] : make_float2(0.f, 0.f);
		}

		const float2* y = sm_fft<true, false, B>(d, s0, s1, tw, sl);

		for (int e = threadIdx.x; e < B * X; e += SM_THREADS) {

			const int b = magic_div(e, x_magic), x = e - b * X;
			const long yz = yz0 + b;

			if (yz >= YZ)
				break;

			float2 t = y[sm_idx<false, B>(wrap_pos(x, X, d.n), b, sl)];

			if (ax)
				t = cscale(t, ax[x] * ayz[yz]);

			const long i = x + X * yz;

			if (maps) {

				t = cmulc(t, maps[i + X * YZ * c]);
				t = (c > c0) ? cadd(acc[e], t) : t;
				acc[e] = t;

				if (c + 1 == c1) {

					out[i + X * YZ * blockIdx.y] = t;

					if (pdot) {

						const float2 pv = pdot[i];
						dot += (double)pv.x * (double)t.x + (double)pv.y * (double)t.y;
					}
				}

			} else {

				out[i + X * YZ * c] = t;

				if (pdot) {

					const float2 pv = ((const void*)pdot == (const void*)out) ? t : pdot[i + X * YZ * c];
					dot += (double)pv.x * (double)t.x + (double)pv.y * (double)t.y;
				}
			}
		}
	}

	if (pdot) {

		const double t = block_sum_d(dot, red);

		if (0 == threadIdx.x)
			dot_part[blockIdx.x + gridDim.x * blockIdx.y] = t;
	}
}

} // namespace bn
