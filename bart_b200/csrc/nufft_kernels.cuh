// NUFFT device kernels: the 512-point Toeplitz column pass (the other FFT passes
// over the 2x oversampled grid are in fft_passes.cuh) and Kaiser-Bessel
// gridding / degridding.
//
// Grid convention. For an image axis of N pixels the oversampled axis has
// L = 2N cells stored in DFT order: cell j' holds the image's Fourier
// transform at frequency j'/2 (j' < N) or (j' - 2N)/2 (j' >= N), in cycles
// per FOV. Image pixel n enters the length-L transform at position
// (n - N/2) mod L (zero elsewhere), which is the reference's centred
// transform (fftmod / linphase chain, src/noncart/nufft.c:196-248, 1410-1423)
// written as an index map instead of phase multiplies. The reference's
// sub-grid s, tap w (src/noncart/nufft.c:158-188) is centred cell
// j = 2w + s, i.e. DFT cell (j + N) mod L.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include "fft_passes.cuh"
#include "fft512.cuh"

namespace bn {

enum { KB_TABLE_N = 1000 };	// kb_size_max, src/noncart/grid.c:38

// Toeplitz column pass for 512-point columns in two-stage transforms
// (fft512_regs): sixteen columns per block, sixteen threads per column, 32
// elements per thread. The same positions, PSF product and crop as k_cols
// MODE 2; one shared-memory exchange and one barrier per transform, plus the
// barrier for the twiddle table and the one between the two transforms.
enum { TOE512_B = 16 };

__global__ void __launch_bounds__(TOE512_B * 16, 2) k_cols_toe512(const float2* in, long ies, long ios,
		int n_in, int wrap_in, float2* out, long oes, long oos, int n_out, int wrap_out,
		int W, const float2* __restrict__ psf, long pes, long pmod, long pos,
		const float2* __restrict__ twg, const int* done)
{
	pdl_wait();
	constexpr int L = 512, SB = TOE512_B;
	extern __shared__ float2 smem[];
	float2* s = smem;
	float2* tw = smem + L * SB;

	const int stop = done ? *done : 0;	// tested once the loads are under way

	for (int i = threadIdx.x; i < L; i += blockDim.x)
		tw[i] = twg[i];

	const int b = threadIdx.x % TOE512_B, t = threadIdx.x / TOE512_B;
	const int cx = blockIdx.x * TOE512_B + b;
	const bool valid = (cx < W);
	const long o = blockIdx.y;
	const float2* inp = in + o * ios + cx;

	float2 v[32];
#pragma unroll
	for (int m = 0; m < 32; m++) {

		const int p = t + 16 * m;
		const int n = wrap_in ? unwrap_pos(p, n_in, L) : p;
		v[m] = (valid && (n < n_in)) ? inp[n * ies] : make_float2(0.f, 0.f);
	}

	if (stop)
		return;

	__syncthreads();	// the twiddle table is complete

	if (wrap_in && (2 * n_in <= L))
		fft512_regs<false, true, SB>(v, s, tw, t, b);
	else
		fft512_regs<false, false, SB>(v, s, tw, t, b);

	const float2* pp = psf + (o % pmod) * pos + cx;
#pragma unroll
	for (int m = 0; m < 32; m++)
		if (valid)
			v[m] = cmul(v[m], pp[(t + 16 * m) * pes]);

	__syncthreads();	// every thread's stage-2 loads are done before s is rewritten
	fft512_regs<true, false, SB>(v, s, tw, t, b);

	if (!valid)
		return;

	float2* outp = out + o * oos + cx;
#pragma unroll
	for (int m = 0; m < 32; m++) {

		const int p = t + 16 * m;
		const int n = wrap_out ? unwrap_pos(p, n_out, L) : p;

		if (n < n_out)
			outp[n * oes] = v[m];
	}
}

// Kaiser-Bessel taps ----------------------------------------------------------------

// intlookup (src/noncart/grid.c:120-149): x *= 2; idx = (int)(x*(n-1));
// lerp in float64 ((1. - c) * a + c * b), rounded to float. Explicit
// round-to-nearest intrinsics keep the compiler from contracting into FMAs,
// so the result is bit-identical to the reference's.
__device__ __forceinline__ float kb_lookup(const float* kb, float x)
{
	x = __fmul_rn(x, 2.0f);
	float xs = __fmul_rn(x, (float)(KB_TABLE_N - 1));
	int idx = (int)xs;
	float fpart = __fsub_rn(xs, (float)idx);
	double a = (double)kb[idx];
	double b = (double)kb[idx + 1];
	double c = (double)fpart;
	double r = __dadd_rn(__dmul_rn(__dsub_rn(1.0, c), a), __dmul_rn(c, b));
	return __double2float_rn(r);
}

enum { MAX_AXIS_TAPS = 10 };

struct AxisTaps {

	int n;
	int cell[MAX_AXIS_TAPS];	// DFT-order cell on the 2N axis
	float w[MAX_AXIS_TAPS];
};

// Taps of one axis for both sub-grid shifts (grid2H_decomp / grid_point_gen,
// src/noncart/nufft.c:158-188, src/noncart/grid.c:403-465):
//   pos_s = float(k + (-s/2)) + float(N/2)   (width hw = w/2 on the N-grid)
//   taps t = ceil(pos_s - hw/2) .. floor(pos_s + hw/2)  (float64 bounds)
//   weight = intlookup(|t - pos_s| / hw)
//   cell: centred j = 2 t + s  ->  DFT order (j + N) mod 2N
// Non-periodic: taps clipped to [0, N-1]; periodic: t mod N.
__device__ __forceinline__ void axis_taps(float k, int N, float hw, int periodic, const float* kb, AxisTaps& t)
{
	t.n = 0;

	if (1 == N) {	// singleton axis: one tap at 0 with intlookup(0)

		t.cell[0] = 0;
		t.w[0] = kb_lookup(kb, 0.f);
		t.n = 1;
		return;
	}

	const int L = 2 * N;
	const float half = (float)(N / 2);
	const double h2 = 0.5 * (double)hw;

#pragma unroll
	for (int s = 0; s < 2; s++) {

		float pos = __fadd_rn(__fadd_rn(k, s ? -0.5f : -0.0f), half);
		int sti = (int)ceil((double)pos - h2);
		int eni = (int)floor((double)pos + h2);

		if (!periodic) {

			sti = max(sti, 0);
			eni = min(eni, N - 1);
		}

		for (int w = sti; (w <= eni) && (t.n < MAX_AXIS_TAPS); w++) {

			float frac = fabsf(__fsub_rn((float)w, pos));
			float val = kb_lookup(kb, __fdiv_rn(frac, hw));
			int wm = periodic ? (((w % N) + N) % N) : w;
			int j = 2 * wm + s + N;

			if (j >= L)
				j -= L;

			t.cell[t.n] = j;
			t.w[t.n] = val;
			t.n++;
		}
	}
}

struct GridGeom {

	int N[3];	// image size per axis
	int G[3];	// grid size per axis (2N, lround(os N) for the chain, or 1)
	long gsz;	// cells per channel
	float hw;	// kernel width on the N-grid (conf.width / 2)
	int periodic;
	// (defaults: the os = 2 gridding, for geometries built field by field)
	int chain = 0;	// os != 2: the chained NUFFT's plain gridding on the G grid
	float os = 2.f;	// its oversampling
	float wg = 6.f;	// its kernel width on the G grid (conf.width)
};

// Taps of one axis of the chained NUFFT (os != 2; nufft_create_chain,
// src/noncart/nufft_chain.c:190-244, gridding by gridH / grid_point_gen,
// src/noncart/grid.c:150-199, 403-465):
//   pos = float(os * k) + float(G/2)   (the centred grid of G cells)
//   taps t = ceil(pos - w/2) .. floor(pos + w/2)  (float64 bounds)
//   weight = intlookup(|t - pos| / w)
//   cell: centred t -> DFT order (t + G/2) mod G (G even)
// Non-periodic: taps clipped to [0, G-1]; periodic: t mod G.
__device__ __forceinline__ void chain_taps(float k, int G, float os, float w, int periodic, const float* kb,
		AxisTaps& t)
{
	t.n = 0;

	if (1 == G) {

		t.cell[0] = 0;
		t.w[0] = kb_lookup(kb, 0.f);
		t.n = 1;
		return;
	}

	const float pos = __fadd_rn(__fmul_rn(os, k), (float)(G / 2));
	int sti = (int)ceil((double)pos - 0.5 * (double)w);
	int eni = (int)floor((double)pos + 0.5 * (double)w);

	if (!periodic) {

		sti = max(sti, 0);
		eni = min(eni, G - 1);
	}

	for (int c = sti; (c <= eni) && (t.n < MAX_AXIS_TAPS); c++) {

		const float frac = fabsf(__fsub_rn((float)c, pos));
		const int cm = periodic ? (((c % G) + G) % G) : c;
		int j = cm + G / 2;

		if (j >= G)
			j -= G;

		t.cell[t.n] = j;
		t.w[t.n] = kb_lookup(kb, __fdiv_rn(frac, w));
		t.n++;
	}
}

// the taps of axis a for either gridding
__device__ __forceinline__ void geom_taps(const GridGeom& g, int a, float k, const float* kb, AxisTaps& t)
{
	if (g.chain)
		chain_taps(k, g.G[a], g.os, g.wg, g.periodic, kb, t);
	else
		axis_taps(k, g.N[a], g.hw, g.periodic, kb, t);
}

// Degridding (forward interpolation), one thread per sample, coils
// [blockIdx.y*cpc, ...). ksp[m + M*c] = sum_taps w * grid[cell + gsz*c].
// The combined weight is ((1*wz)*wy)*wx in float32 as in grid_point_gen.
__global__ void k_degrid(const float4* __restrict__ traj, long M, GridGeom g, int C, int cpc,
		const float2* __restrict__ grid, float2* __restrict__ ksp, const float* __restrict__ kbg)
{
	__shared__ float kb[KB_TABLE_N + 1];

	for (int i = threadIdx.x; i <= KB_TABLE_N; i += blockDim.x)
		kb[i] = kbg[i];

	__syncthreads();

	long m = (long)blockIdx.x * blockDim.x + threadIdx.x;

	if (m >= M)
		return;

	float4 k = traj[m];
	AxisTaps tx, ty, tz;
	geom_taps(g, 0, k.x, kb, tx);
	geom_taps(g, 1, k.y, kb, ty);
	geom_taps(g, 2, k.z, kb, tz);

	const int c0 = blockIdx.y * cpc;
	const int c1 = min(C, c0 + cpc);

	for (int c = c0; c < c1; c++) {

		const float2* gc = grid + g.gsz * c;
		float2 acc = make_float2(0.f, 0.f);

		for (int a = 0; a < tz.n; a++) {

			float dz = tz.w[a];
			long oz = (long)tz.cell[a] * g.G[1];

			for (int bb = 0; bb < ty.n; bb++) {

				float dzy = __fmul_rn(dz, ty.w[bb]);
				long oy = (oz + ty.cell[bb]) * g.G[0];

				for (int cc = 0; cc < tx.n; cc++) {

					float d = __fmul_rn(dzy, tx.w[cc]);
					float2 v = gc[oy + tx.cell[cc]];
					acc.x = fmaf(v.x, d, acc.x);
					acc.y = fmaf(v.y, d, acc.y);
				}
			}
		}

		ksp[m + M * c] = acc;
	}
}

// Gridding (adjoint spreading) with float2 atomics into the grid (must be
// zeroed). One thread per sample, coils as in k_degrid.
__global__ void k_grid_atomic(const float4* __restrict__ traj, long M, GridGeom g, int C, int cpc,
		const float2* __restrict__ ksp, float2* __restrict__ grid, const float* __restrict__ kbg)
{
	__shared__ float kb[KB_TABLE_N + 1];

	for (int i = threadIdx.x; i <= KB_TABLE_N; i += blockDim.x)
		kb[i] = kbg[i];

	__syncthreads();

	long m = (long)blockIdx.x * blockDim.x + threadIdx.x;

	if (m >= M)
		return;

	float4 k = traj[m];
	AxisTaps tx, ty, tz;
	geom_taps(g, 0, k.x, kb, tx);
	geom_taps(g, 1, k.y, kb, ty);
	geom_taps(g, 2, k.z, kb, tz);

	const int c0 = blockIdx.y * cpc;
	const int c1 = min(C, c0 + cpc);

	for (int c = c0; c < c1; c++) {

		float2 val = ksp[m + M * c];

		if ((0.f == val.x) && (0.f == val.y))
			continue;	// grid(): samples that are zero in all channels are skipped

		float2* gc = grid + g.gsz * c;

		for (int a = 0; a < tz.n; a++) {

			float dz = tz.w[a];
			long oz = (long)tz.cell[a] * g.G[1];

			for (int bb = 0; bb < ty.n; bb++) {

				float dzy = __fmul_rn(dz, ty.w[bb]);
				long oy = (oz + ty.cell[bb]) * g.G[0];

				for (int cc = 0; cc < tx.n; cc++) {

					float d = __fmul_rn(dzy, tx.w[cc]);
					atomicAdd(&gc[oy + tx.cell[cc]], make_float2(val.x * d, val.y * d));
				}
			}
		}
	}
}

// Deterministic gridding --------------------------------------------------------
//
// The adjoint interpolation as a sparse matrix in CSR form over grid cells:
// row = cell, entries (sample, weight) in increasing sample order. It is
// built once per trajectory (k_csr_keys + a stable radix sort by
// cell * M + sample + k_csr_fill), after which gridding is a gather per
// cell in that fixed order: no atomics, bit-identical results run to run,
// and every cell is written (no clearing pass). The weights are the same
// float32 products as in k_grid_atomic.

enum { CSR_TAPS_AXIS = 8 };	// per axis: two sub-grids x up to 4 taps (width <= 6)

// one key (cell * M + m, or ~0 for an unused slot) and weight per (sample, tap slot)
__global__ void k_csr_keys(const float4* __restrict__ traj, long M, GridGeom g, const float* __restrict__ kbg,
		unsigned long long* __restrict__ keys, float* __restrict__ vals, int slots_z)
{
	__shared__ float kb[KB_TABLE_N + 1];

	for (int i = threadIdx.x; i <= KB_TABLE_N; i += blockDim.x)
		kb[i] = kbg[i];

	__syncthreads();

	long m = (long)blockIdx.x * blockDim.x + threadIdx.x;

	if (m >= M)
		return;

	float4 k = traj[m];
	AxisTaps tx, ty, tz;
	geom_taps(g, 0, k.x, kb, tx);
	geom_taps(g, 1, k.y, kb, ty);
	geom_taps(g, 2, k.z, kb, tz);

	const int slots = CSR_TAPS_AXIS * CSR_TAPS_AXIS * slots_z;
	unsigned long long* kp = keys + m * slots;
	float* vp = vals + m * slots;
	int t = 0;

	for (int a = 0; a < tz.n; a++) {

		float dz = tz.w[a];
		long oz = (long)tz.cell[a] * g.G[1];

		for (int bb = 0; bb < ty.n; bb++) {

			float dzy = __fmul_rn(dz, ty.w[bb]);
			long oy = (oz + ty.cell[bb]) * g.G[0];

			for (int cc = 0; cc < tx.n; cc++) {

				if (t < slots) {

					kp[t] = (unsigned long long)(oy + tx.cell[cc]) * (unsigned long long)M + (unsigned long long)m;
					vp[t] = __fmul_rn(dzy, tx.w[cc]);
					t++;
				}
			}
		}
	}

	for (; t < slots; t++) {

		kp[t] = ~0ull;
		vp[t] = 0.f;
	}
}

// sorted keys -> column (sample) indices and per-cell counts; unused slots
// (key ~0) sort to the end and are not counted
__global__ void k_csr_fill_valid(const unsigned long long* __restrict__ keys, long nnz, long M, long gsz,
		int* __restrict__ col, int* __restrict__ counts)
{
	for (long i = (long)blockIdx.x * blockDim.x + threadIdx.x; i < nnz; i += (long)gridDim.x * blockDim.x) {

		unsigned long long key = keys[i];

		if (~0ull == key) {

			col[i] = 0;
			continue;
		}

		long cell = (long)(key / (unsigned long long)M);
		col[i] = (int)(key % (unsigned long long)M);

		if (cell < gsz)
			atomicAdd(&counts[cell], 1);	// integer counts: order-independent
	}
}

// grid[cell + gsz*c] = sum over the cell's row of w * ksp[m + M*c]: one warp
// per cell, lane l sums entries l, l+32, ... in order, then a fixed shuffle
// tree combines the lanes, so the summation order is the same every run (and
// long rows at the k-space centre are spread over 32 lanes).
__global__ void k_grid_csr(const long* __restrict__ row_ptr, const int* __restrict__ col, const float* __restrict__ val,
		long gsz, long M, int C, int cpc, const float2* __restrict__ ksp, float2* __restrict__ grid)
{
	const int lane = threadIdx.x % 32;
	long cell = ((long)blockIdx.x * blockDim.x + threadIdx.x) / 32;

	if (cell >= gsz)
		return;

	const long r0 = row_ptr[cell];
	const long r1 = row_ptr[cell + 1];
	const int c0 = blockIdx.y * cpc;
	const int c1 = min(C, c0 + cpc);

	for (int cb = c0; cb < c1; cb += 4) {

		float2 acc[4];
#pragma unroll
		for (int q = 0; q < 4; q++)
			acc[q] = make_float2(0.f, 0.f);

		for (long i = r0 + lane; i < r1; i += 32) {

			float w = val[i];
			long m = col[i];
#pragma unroll
			for (int q = 0; q < 4; q++) {

				if (cb + q < c1) {

					float2 y = ksp[m + M * (cb + q)];
					acc[q].x = fmaf(y.x, w, acc[q].x);
					acc[q].y = fmaf(y.y, w, acc[q].y);
				}
			}
		}

#pragma unroll
		for (int q = 0; q < 4; q++) {

			for (int o = 16; o > 0; o >>= 1) {

				acc[q].x += __shfl_xor_sync(0xffffffffu, acc[q].x, o);
				acc[q].y += __shfl_xor_sync(0xffffffffu, acc[q].y, o);
			}

			if ((0 == lane) && (cb + q < c1))
				grid[cell + gsz * (cb + q)] = acc[q];
		}
	}
}

} // namespace bn
