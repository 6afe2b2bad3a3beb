// Binned Kaiser-Bessel gridding and degridding through shared-memory tiles.
//
// Plan time: every sample gets the bin (tile of BS^d cells of the oversampled
// grid) holding its centre 2k + N per axis; a stable radix sort orders the
// samples by bin, and bins are cut into sub-blocks of at most SUB samples
// (dense bins at the k-space centre become several sub-blocks, so the work
// is balanced). The sorted trajectory is stored as float4 (coalesced loads).
//
// Degridding (gather): four lanes per sample in bin order; neighbouring
// samples read overlapping taps, so the gathers hit L1, and the weights are
// read once per sample for all coils.
// Gridding (scatter): output-stationary tiles for several channels, a quad of
// lanes per sample with global atomics for one (bin order keeps a block's
// atomics within a few L2 lines). Alternative (BNUFFT_GRIDDING=tiles): a block takes one
// sub-block, accumulates its samples' taps into a zeroed shared-memory tile
// (bin plus HALO cells per side, a chunk of coils) with shared-memory atomics
// and flushes touched cells with one global atomic each; on B200 it measured
// slower for radial and kooshball data.
//
// Taps and weights are those of axis_taps (bit-identical to the reference's,
// src/noncart/grid.c:403-465); only the cell index changes from the DFT-order
// grid index to the tile-local index of the same cell.
#pragma once

#include <climits>
#include <cuda_runtime.h>

#include "nufft_kernels.cuh"

namespace bn {

enum { BIN_HALO = 4, BIN_SUB = 512, BIN_THREADS = 256 };

struct BinGeom {

	int bs[3];	// bin size per axis (1 for singleton axes)
	int nb[3];	// bins per axis
	int tile[3];	// tile extent per axis (bs + 2 * halo, or 1)
	long ncells;	// tile cells
};

// centred 2N position of a sample along an axis -> bin index
__device__ __forceinline__ int bin_of(float k, int N, int bs, int nb, int periodic)
{
	if (1 == N)
		return 0;

	float p = 2.f * k + (float)N;

	if (periodic) {

		float L = 2.f * N;
		p = p - L * floorf(p / L);
	}

	int b = (int)floorf(p / (float)bs);
	return min(max(b, 0), nb - 1);
}

// key = bin id of sample m, value = m; samples per bin if wanted
__global__ void k_bin_keys(const float4* __restrict__ traj, long M, GridGeom g, BinGeom bg,
		unsigned* __restrict__ keys, int* __restrict__ vals, int* __restrict__ counts)
{
	for (long m = (long)blockIdx.x * blockDim.x + threadIdx.x; m < M; m += (long)gridDim.x * blockDim.x) {

		float4 k = traj[m];
		int bx = bin_of(k.x, g.N[0], bg.bs[0], bg.nb[0], g.periodic);
		int by = bin_of(k.y, g.N[1], bg.bs[1], bg.nb[1], g.periodic);
		int bz = bin_of(k.z, g.N[2], bg.bs[2], bg.nb[2], g.periodic);
		unsigned key = (unsigned)(bx + bg.nb[0] * (by + bg.nb[1] * bz));
		keys[m] = key;
		vals[m] = (int)m;

		if (counts)
			atomicAdd(&counts[key], 1);
	}
}

// nsub[b] = ceil(count_b / sub), nsub[nbins] = 0
__global__ void k_bin_nsub(const int* __restrict__ bin_start, int nbins, int sub, int* __restrict__ nsub)
{
	for (int b = blockIdx.x * blockDim.x + threadIdx.x; b <= nbins; b += gridDim.x * blockDim.x)
		nsub[b] = (b < nbins) ? (bin_start[b + 1] - bin_start[b] + sub - 1) / sub : 0;
}

// sub-block table: for bin b with n samples starting at bin_start[b],
// ceil(n / sub) entries (bin, first sample, count) starting at sub_start[b]
__global__ void k_sub_fill(const int* __restrict__ bin_start, const int* __restrict__ sub_start, int nbins, int sub,
		int* __restrict__ sub_bin, int* __restrict__ sub_first, int* __restrict__ sub_count)
{
	for (int b = blockIdx.x * blockDim.x + threadIdx.x; b < nbins; b += gridDim.x * blockDim.x) {

		int n = bin_start[b + 1] - bin_start[b];
		int s0 = sub_start[b];

		for (int j = 0; j * sub < n; j++) {

			sub_bin[s0 + j] = b;
			sub_first[s0 + j] = bin_start[b] + j * sub;
			sub_count[s0 + j] = min(sub, n - j * sub);
		}
	}
}

__global__ void k_gather_traj(float4* __restrict__ dst, const float4* __restrict__ src, const int* __restrict__ perm, long M)
{
	for (long i = (long)blockIdx.x * blockDim.x + threadIdx.x; i < M; i += (long)gridDim.x * blockDim.x)
		dst[i] = src[perm[i]];
}

struct TileOrigin {

	int o[3];	// centred 2N index of the tile's first cell per axis
};

__device__ __forceinline__ TileOrigin tile_origin(int bin, const BinGeom& bg, const GridGeom& g)
{
	TileOrigin t;
	int bx = bin % bg.nb[0];
	int by = (bin / bg.nb[0]) % bg.nb[1];
	int bz = bin / (bg.nb[0] * bg.nb[1]);
	t.o[0] = (g.N[0] > 1) ? bx * bg.bs[0] - BIN_HALO : 0;
	t.o[1] = (g.N[1] > 1) ? by * bg.bs[1] - BIN_HALO : 0;
	t.o[2] = (g.N[2] > 1) ? bz * bg.bs[2] - BIN_HALO : 0;
	return t;
}

// grid (DFT order) index of tile cell (lx, ly, lz), or -1 outside a
// non-periodic grid
__device__ __forceinline__ long tile_to_grid(int lx, int ly, int lz, const TileOrigin& to, const GridGeom& g)
{
	int l[3] = { lx, ly, lz };
	long idx = 0;
	long stride = 1;

	for (int a = 0; a < 3; a++) {

		int j = 0;

		if (g.N[a] > 1) {

			const int L = g.G[a];
			j = to.o[a] + l[a];

			if ((j < 0) || (j >= L)) {

				if (!g.periodic)
					return -1;

				j = ((j % L) + L) % L;
			}

			j += g.N[a];

			if (j >= L)
				j -= L;
		}

		idx += j * stride;
		stride *= g.G[a];
	}

	return idx;
}

// Width-6 fast path ------------------------------------------------------------
//
// For the default kernel width 6 (hw = 3 on the N-grid) each sub-grid has
// exactly three taps with weight: the window [pos - 1.5, pos + 1.5] holds
// three integers, or four when pos - 1.5 is an integer, and then both end
// taps sit at |t - pos| = 1.5 where the table is exactly 0 (kb(0.5) = 0,
// src/noncart/grid.c:75-76); the lower one is dropped. Taps clipped by a
// non-periodic grid keep weight 0 and a harmless cell index. The fixed trip
// count lets every tap loop unroll into registers.
struct Taps6 {

	int cell[6];
	float w[6];
};

// MODE 0: cell = DFT-order grid index; MODE 1: cell = tile-local index
template <int MODE>
__device__ __forceinline__ void axis_taps6(float k, int N, int periodic, const float* kb, int origin, Taps6& t)
{
	if (1 == N) {
#pragma unroll
		for (int q = 0; q < 6; q++) {

			t.cell[q] = 0;
			t.w[q] = (0 == q) ? kb_lookup(kb, 0.f) : 0.f;
		}

		return;
	}

	const int L = 2 * N;
	const float half = (float)(N / 2);

#pragma unroll
	for (int s = 0; s < 2; s++) {

		float pos = __fadd_rn(__fadd_rn(k, s ? -0.5f : -0.0f), half);
		double lo = (double)pos - 1.5;
		int sti = (int)ceil(lo);

		if ((double)sti == lo)
			sti += 1;

#pragma unroll
		for (int q = 0; q < 3; q++) {

			int w = sti + q;
			float frac = fabsf(__fsub_rn((float)w, pos));
			float val = kb_lookup(kb, __fdiv_rn(frac, 3.0f));
			bool valid = periodic || ((w >= 0) && (w <= N - 1));
			int cell;

			if (0 == MODE) {

				int wm = periodic ? (((w % N) + N) % N) : min(max(w, 0), N - 1);
				cell = 2 * wm + s + N;

				if (cell >= L)
					cell -= L;

			} else {

				cell = 2 * w + s - origin;

				if (periodic)
					cell = ((cell % L) + L) % L;

				cell = max(cell, 0);	// clipped taps (weight 0) may fall left of the tile
			}

			t.cell[3 * s + q] = cell;
			t.w[3 * s + q] = valid ? val : 0.f;
		}
	}
}

// Gridding, width 6: per sub-block, accumulate into shared-memory tiles of cc
// coils with shared-memory atomics, then flush touched cells with one global
// float2 atomic each. The grid must be zeroed.
template <int TZ>
__global__ void __launch_bounds__(BIN_THREADS, 2) k_grid6_binned(const float4* __restrict__ traj_sorted,
		const int* __restrict__ perm, long M, GridGeom g, BinGeom bg,
		const int* __restrict__ sub_bin, const int* __restrict__ sub_first, const int* __restrict__ sub_count,
		const int* __restrict__ nsub_dev, int C, int cc, const float2* __restrict__ ksp, float2* __restrict__ grid,
		const float* __restrict__ kbg)
{
	extern __shared__ float2 tiles[];	// [cc][ncells]
	__shared__ float kb[KB_TABLE_N + 1];

	const int sb = blockIdx.x;

	if (sb >= *nsub_dev)
		return;

	for (int i = threadIdx.x; i <= KB_TABLE_N; i += blockDim.x)
		kb[i] = kbg[i];

	const int bin = sub_bin[sb];
	const int first = sub_first[sb];
	const int count = sub_count[sb];
	const TileOrigin to = tile_origin(bin, bg, g);
	const int tx = bg.tile[0], ty = bg.tile[1];

	for (int c0 = 0; c0 < C; c0 += cc) {

		const int cn = min(cc, C - c0);

		__syncthreads();

		for (long t = threadIdx.x; t < bg.ncells * cn; t += blockDim.x)
			tiles[t] = make_float2(0.f, 0.f);

		__syncthreads();

		// lanes of a warp take samples 8 apart in bin order: neighbouring
		// samples of a trajectory share taps, so this spreads the
		// shared-memory atomics of one instruction over distinct cells
		const int per = (count + blockDim.x - 1) / blockDim.x;

		for (int r = 0; r < per; r++) {

			int t = threadIdx.x + r * blockDim.x;
			int i = (t % 32) * 8 + (t / 32) % 8 + (t / 256) * 256;

			if (i >= count)
				continue;

			float4 k = traj_sorted[first + i];
			Taps6 ax, ay, az;
			axis_taps6<1>(k.x, g.N[0], g.periodic, kb, to.o[0], ax);
			axis_taps6<1>(k.y, g.N[1], g.periodic, kb, to.o[1], ay);
			axis_taps6<1>(k.z, g.N[2], g.periodic, kb, to.o[2], az);
			const long m = perm[first + i];

			for (int c = 0; c < cn; c++) {

				float2 val = ksp[m + M * (c0 + c)];

				if ((0.f == val.x) && (0.f == val.y))
					continue;

				float* tl = (float*)(tiles + (long)c * bg.ncells);
#pragma unroll 1
				for (int a = 0; a < TZ; a++) {

					float dz = az.w[a];
					int oz = az.cell[a] * ty;
#pragma unroll
					for (int b = 0; b < 6; b++) {

						float dzy = __fmul_rn(dz, ay.w[b]);
						int oy = (oz + ay.cell[b]) * tx;
#pragma unroll
						for (int e = 0; e < 6; e++) {

							float d = __fmul_rn(dzy, ax.w[e]);

							if (0.f != d) {

								int cell = oy + ax.cell[e];
								atomicAdd(&tl[2 * cell + 0], val.x * d);
								atomicAdd(&tl[2 * cell + 1], val.y * d);
							}
						}
					}
				}
			}
		}

		__syncthreads();

		for (long t = threadIdx.x; t < bg.ncells * cn; t += blockDim.x) {

			float2 v = tiles[t];

			if ((0.f == v.x) && (0.f == v.y))
				continue;

			int c = (int)(t / bg.ncells);
			long cell = t - (long)c * bg.ncells;
			int lx = (int)(cell % tx);
			int ly = (int)((cell / tx) % ty);
			int lz = (int)(cell / ((long)tx * ty));
			long gi = tile_to_grid(lx, ly, lz, to, g);

			if (gi >= 0)
				atomicAdd(&grid[gi + g.gsz * (c0 + c)], v);
		}
	}
}

// Footprint record of a sorted sample (built once per trajectory by
// k_foot): float4 0 holds the centred start cells lo of the x, y, z taps
// (as int bits); float4s 1..5 the weights of cells lo .. lo + 5 per axis,
// x then y then z (6 each, the last two slots zero). A singleton axis has
// lo = 0 and the one weight intlookup(0).
enum { FOOT_F4 = 6 };

// Footprint of one axis: the six taps of a sample (two sub-grids x three)
// lie on the centred cells lo .. lo + 5 (2w + s); w7[t] is the weight of
// cell lo + t (0 where a non-periodic grid clips the tap). Singleton axis:
// one tap at 0 with weight intlookup(0).
__device__ __forceinline__ int foot6_lo(float k, int N)
{
	if (1 == N)
		return 0;

	const float half = (float)(N / 2);
	int lo = INT_MAX;
#pragma unroll
	for (int s = 0; s < 2; s++) {

		float pos = __fadd_rn(__fadd_rn(k, s ? -0.5f : -0.0f), half);
		double l = (double)pos - 1.5;
		int sti = (int)ceil(l);

		if ((double)sti == l)
			sti += 1;

		lo = min(lo, 2 * sti + s);
	}

	return lo;
}

__device__ __forceinline__ void foot6_w(float k, int N, int periodic, const float* kb, int lo, float* w7)
{
#pragma unroll
	for (int t = 0; t < 7; t++)
		w7[t] = 0.f;

	if (1 == N) {

		w7[0] = kb_lookup(kb, 0.f);
		return;
	}

	const float half = (float)(N / 2);
#pragma unroll
	for (int s = 0; s < 2; s++) {

		float pos = __fadd_rn(__fadd_rn(k, s ? -0.5f : -0.0f), half);
		double l = (double)pos - 1.5;
		int sti = (int)ceil(l);

		if ((double)sti == l)
			sti += 1;
#pragma unroll
		for (int q = 0; q < 3; q++) {

			int w = sti + q;
			float frac = fabsf(__fsub_rn((float)w, pos));
			float val = kb_lookup(kb, __fdiv_rn(frac, 3.0f));
			bool valid = periodic || ((w >= 0) && (w <= N - 1));
			int t = 2 * w + s - lo;

			if ((t >= 0) && (t < 7))
				w7[t] = valid ? val : 0.f;
		}
	}
}

// footprints of all sorted samples (the weights as axis_taps6 computes them:
// the same kb_lookup of the same float32 distances), a thread per sample and
// axis; lo4 (if given): their start cells once more, for k_tile_hits
__global__ void k_foot(const float4* __restrict__ traj, const int* __restrict__ perm, long M, GridGeom g, const float* __restrict__ kbg,
		float4* __restrict__ foot, short4* __restrict__ lo4)
{
	__shared__ float kb[KB_TABLE_N + 1];

	for (int i = threadIdx.x; i <= KB_TABLE_N; i += blockDim.x)
		kb[i] = kbg[i];

	__syncthreads();

	for (long e = (long)blockIdx.x * blockDim.x + threadIdx.x; e < 3 * M; e += (long)gridDim.x * blockDim.x) {

		const long i = e / 3;
		const int a = (int)(e - 3 * i);
		const float4 k = traj[perm[i]];
		const float ka = (0 == a) ? k.x : ((1 == a) ? k.y : k.z);
		const int N = (0 == a) ? g.N[0] : ((1 == a) ? g.N[1] : g.N[2]);
		float w7[7];
		const int lo = foot6_lo(ka, N);
		foot6_w(ka, N, g.periodic, kb, lo, w7);
		float* f = (float*)(foot + i * FOOT_F4);
		f[a] = __int_as_float(lo);

		if (lo4) {	// for k_tile_hits: cells further out than the grid's edges meet no tile

			const int G = (1 == N) ? 1 : 2 * N;
			int l = lo;

			if (g.periodic) {

				l %= G;
				l = (l < 0) ? l + G : l;

			} else {

				l = min(max(l, -6), G);
			}

			((short*)(lo4 + i))[a] = (short)l;
		}
#pragma unroll
		for (int t = 0; t < 6; t += 2)
			*(float2*)(f + 4 + 6 * a + t) = make_float2(w7[t], w7[t + 1]);

		if (2 == a) {

			f[3] = 0.f;
			*(float2*)(f + 22) = make_float2(0.f, 0.f);
		}
	}
}

// Degridding, width 6: four lanes (a quad) per sample, in bin order. The six x
// taps are at most seven consecutive cells; lane q of the quad reads cells
// 2q, 2q + 1 of the 8-cell window that starts at an even cell, so a tap row is
// one 64-byte access of the quad (a thread per sample needed four separate
// ones, and the gather is bound by the L1's lines per request). Weights come
// from the plan's footprint records and stay in registers for all channels of
// the block (grid.y splits the channels in chunks of cpb where the samples
// alone do not fill the GPU). Four channels are summed side by side and
// exchanged within the quad so that lane q ends up with channel c + q. The
// optional weights multiply (wgt, wgt_c channels) happens on the way out.
// foot, perm: of n samples; M: samples of a channel of ksp.
// Grid sides are even (2N, N even), so the pairs are aligned.
// One B200, 8-coil 128^3 kooshball, 5.12 M samples: 9.17 ms a thread per
// sample, 5.3 ms by quads (3.9 ms from the grid in fours of coils below).
template <int CC, int TZ>
__device__ __forceinline__ void degrid6_quad(const float2* __restrict__ gc, long gsz, long plane,
		const float* __restrict__ f, const int (&zc)[TZ], const int (&row)[6], const float (&wy)[6], float w0, float w1,
		bool act, float2 (&acc)[CC])
{
#pragma unroll
	for (int c = 0; c < CC; c++)
		acc[c] = make_float2(0.f, 0.f);

	if (!act)	// both cells of this lane are outside the footprint
		return;

#pragma unroll 1
	for (int a = 0; a < TZ; a++) {

		const float dz = f[16 + a];
		int z = zc[0];
#pragma unroll
		for (int k = 1; k < TZ; k++)
			z = (k == a) ? zc[k] : z;

		const float2* gz = gc + z * plane;
#pragma unroll
		for (int b = 0; b < 6; b++) {

			const float dzy = __fmul_rn(dz, wy[b]);
			const float d0 = __fmul_rn(dzy, w0), d1 = __fmul_rn(dzy, w1);
#pragma unroll
			for (int c = 0; c < CC; c++) {

				const float4 v = *(const float4*)(gz + gsz * c + row[b]);
				acc[c].x = fmaf(v.x, d0, acc[c].x);
				acc[c].y = fmaf(v.y, d0, acc[c].y);
				acc[c].x = fmaf(v.z, d1, acc[c].x);
				acc[c].y = fmaf(v.w, d1, acc[c].y);
			}
		}
	}
}

__device__ __forceinline__ float2 shfl_xor2(float2 v, int m)
{
	return make_float2(__shfl_xor_sync(0xffffffffu, v.x, m), __shfl_xor_sync(0xffffffffu, v.y, m));
}

// grid cell index of centred cell c of an axis of G = 2N cells; cells outside a
// non-periodic grid (their weight is 0) are moved inside
__device__ __forceinline__ int cell_of(int c, int N, int G, int periodic)
{
	if (1 == G)
		return 0;

	if (periodic) {

		c %= G;
		c = (c < 0) ? c + G : c;

	} else {

		c = min(max(c, 0), G - 1);
	}

	c += N;
	return (c >= G) ? c - G : c;
}

// what a lane of a quad needs of its sample: two x cells and their weights, the
// row offsets and z cells of its taps, the y weights
template <int TZ>
struct Quad {

	const float* f;			// the footprint record (z weights at 16)
	float w0, w1;
	int row[6], zc[TZ];		// x cell included in row
	float wy[6];

	__device__ __forceinline__ Quad(const float4* foot, long i, const GridGeom& g)
	{
		const int q = threadIdx.x & 3;
		const float4 h = foot[i * FOOT_F4];
		f = (const float*)(foot + i * FOOT_F4);

		// this lane's two cells of the x window
		int lo = __float_as_int(h.x);

		if (g.periodic) {

			lo %= g.G[0];
			lo = (lo < 0) ? lo + g.G[0] : lo;

		} else {

			lo = min(max(lo, -6), g.G[0]);	// further out all weights are 0
		}

		// (sides below eight cells hold the window more than once)
		const int u = lo + g.N[0];
		int e = (u & ~1) + 2 * q;
		const int t = e - u;			// -1 .. 6
		e = (e < 0) ? e + 2 * g.G[0] : e;

		while (e >= g.G[0])
			e -= g.G[0];
		w0 = ((t >= 0) && (t < 6)) ? f[4 + t] : 0.f;
		w1 = (t < 5) ? f[5 + t] : 0.f;
#pragma unroll
		for (int b = 0; b < 6; b++) {

			row[b] = cell_of(__float_as_int(h.y) + b, g.N[1], g.G[1], g.periodic) * g.G[0] + e;
			wy[b] = f[10 + b];
		}
#pragma unroll
		for (int a = 0; a < TZ; a++)
			zc[a] = (TZ > 1) ? cell_of(__float_as_int(h.z) + a, g.N[2], g.G[2], g.periodic) : 0;
	}
};

template <int TZ>
__global__ void __launch_bounds__(BIN_THREADS, 3) k_degrid6_quads(const float4* __restrict__ foot,
		const int* __restrict__ perm, long n, long M, GridGeom g, int C, int cpb, const float2* __restrict__ grid,
		float2* __restrict__ ksp, const float2* __restrict__ wgt, int wgt_c)
{
	const int q = threadIdx.x & 3;
	const long s = ((long)blockIdx.x * BIN_THREADS + threadIdx.x) / 4;
	const long i = min(s, n - 1);		// surplus quads repeat the last sample and write nothing
	const long m = perm[i];
	const Quad<TZ> d(foot, i, g);
	const float* f = d.f;
	const float w0 = d.w0, w1 = d.w1;
	const bool act = (0.f != w0) || (0.f != w1);
	const bool valid = (s < n);
	const long plane = (long)g.G[0] * g.G[1];
	const int c0 = blockIdx.y * cpb, c1 = min(C, c0 + cpb);
	int c = c0;

	for (; c + 3 < c1; c += 4) {

		float2 acc[4];
		degrid6_quad<4, TZ>(grid + g.gsz * c, g.gsz, plane, f, d.zc, d.row, d.wy, w0, w1, act, acc);
		float2 k0 = (q & 2) ? acc[2] : acc[0], k1 = (q & 2) ? acc[3] : acc[1];
		k0 = cadd(k0, shfl_xor2((q & 2) ? acc[0] : acc[2], 2));
		k1 = cadd(k1, shfl_xor2((q & 2) ? acc[1] : acc[3], 2));
		float2 r = cadd((q & 1) ? k1 : k0, shfl_xor2((q & 1) ? k0 : k1, 1));

		if (valid) {

			if (wgt)
				r = cmul(r, wgt[m + M * ((c + q) % wgt_c)]);

			ksp[m + M * (c + q)] = r;
		}
	}

	for (; c < c1; c++) {

		float2 acc[1];
		degrid6_quad<1, TZ>(grid + g.gsz * c, g.gsz, plane, f, d.zc, d.row, d.wy, w0, w1, act, acc);
		float2 r = cadd(acc[0], shfl_xor2(acc[0], 2));
		r = cadd(r, shfl_xor2(r, 1));

		if (valid && (0 == q)) {

			if (wgt)
				r = cmul(r, wgt[m + M * (c % wgt_c)]);

			ksp[m + M * c] = r;
		}
	}
}

// Degridding from a grid with four channels of a cell side by side (32 bytes;
// written so by the last column pass): lane q of a sample's quad takes channels
// 2 (q & 1) and the next one, of the even or odd x taps (q >> 1), so a row is
// three 64-byte accesses for four channels, without the window's unused cells
// and mostly within one cache line: 27 lines per sample and channel instead
// of 50 (the gather is bound by the L1's lines per request).
template <int NP>
__device__ __forceinline__ void degrid6_by4(const float4* __restrict__ gp, long group, long plane,
		const float* __restrict__ f, const int (&zc)[6], const int (&row)[6], const float (&wy)[6], const int (&xo)[3], const float (&wx)[3],
		float2 (&acc)[NP][2])
{
#pragma unroll
	for (int p = 0; p < NP; p++)
		acc[p][0] = acc[p][1] = make_float2(0.f, 0.f);
#pragma unroll 1
	for (int a = 0; a < 6; a++) {

		const float dz = f[16 + a];
		int z = zc[0];
#pragma unroll
		for (int k = 1; k < 6; k++)
			z = (k == a) ? zc[k] : z;

		const float4* gz = gp + z * plane;
#pragma unroll
		for (int b = 0; b < 6; b++) {

			const float dzy = __fmul_rn(dz, wy[b]);
			const float4* r = gz + 2 * row[b];
#pragma unroll
			for (int k = 0; k < 3; k++) {

				const float d = __fmul_rn(dzy, wx[k]);
#pragma unroll
				for (int p = 0; p < NP; p++) {

					const float4 v = r[group * p + xo[k]];
					acc[p][0] = cfma(make_float2(v.x, v.y), make_float2(d, d), acc[p][0]);
					acc[p][1] = cfma(make_float2(v.z, v.w), make_float2(d, d), acc[p][1]);
				}
			}
		}
	}
}

__global__ void __launch_bounds__(BIN_THREADS, 3) k_degrid6_by4(const float4* __restrict__ foot,
		const int* __restrict__ perm, long n, long M, GridGeom g, int C, int cpb, const float2* __restrict__ grid,
		float2* __restrict__ ksp, const float2* __restrict__ wgt, int wgt_c)
{
	const int q = threadIdx.x & 3, h = q & 1, odd = q >> 1;
	const long s = ((long)blockIdx.x * BIN_THREADS + threadIdx.x) / 4;
	const long i = min(s, n - 1);		// surplus quads repeat the last sample and write nothing
	const long m = perm[i];
	const float4 lo = foot[i * FOOT_F4];
	const float* f = (const float*)(foot + i * FOOT_F4);
	int zc[6], row[6], xo[3];
	float wy[6], wx[3];
#pragma unroll
	for (int t = 0; t < 6; t++) {

		row[t] = cell_of(__float_as_int(lo.y) + t, g.N[1], g.G[1], g.periodic) * g.G[0];
		zc[t] = cell_of(__float_as_int(lo.z) + t, g.N[2], g.G[2], g.periodic);
		wy[t] = f[10 + t];
	}
#pragma unroll
	for (int k = 0; k < 3; k++) {

		xo[k] = 2 * cell_of(__float_as_int(lo.x) + 2 * k + odd, g.N[0], g.G[0], g.periodic);
		wx[k] = f[4 + 2 * k + odd];
	}

	const int c1 = min(C, (int)blockIdx.y * cpb + cpb);
	const long group = 2 * g.gsz, plane = 2L * g.G[0] * g.G[1];		// in 16-byte words

	// the quad's two halves of a sum are exchanged: lane q keeps channel 2 h + odd
	auto store = [&](const float2 (&a)[2], int c) {
		float2 r = cadd(odd ? a[1] : a[0], shfl_xor2(odd ? a[0] : a[1], 2));
		c += 2 * h + odd;

		if (s < n) {

			if (wgt)
				r = cmul(r, wgt[m + M * (c % wgt_c)]);

			ksp[m + M * c] = r;
		}
	};

	int c = blockIdx.y * cpb;

	for (; c + 7 < c1; c += 8) {

		float2 acc[2][2];
		degrid6_by4<2>((const float4*)grid + group * (c / 4) + h, group, plane, f, zc, row, wy, xo, wx, acc);
		store(acc[0], c);
		store(acc[1], c + 4);
	}

	if (c < c1) {

		float2 acc[1][2];
		degrid6_by4<1>((const float4*)grid + group * (c / 4) + h, group, plane, f, zc, row, wy, xo, wx, acc);
		store(acc[0], c);
	}
}

// Gridding, width 6, with global atomics: a quad per sample in bin order as in
// the degridding, one 16-byte reduction (two cells) per lane and tap row, so a
// quad's reductions of a row fall into one 64-byte piece of the grid. Bound by
// the L2's atomic units. The default for a single channel (one thread per
// sample with four separate 16-byte reductions per row: 256^2 radial, 402
// spokes, 51.8 us; 27 us by quads). The grid must be cleared.
template <int TZ>
__global__ void __launch_bounds__(BIN_THREADS) k_grid6_quads(const float4* __restrict__ foot,
		const int* __restrict__ perm, long n, long M, GridGeom g, int C, const float2* __restrict__ ksp,
		float2* __restrict__ grid)
{
	const long i = ((long)blockIdx.x * BIN_THREADS + threadIdx.x) / 4;

	if (i >= n)
		return;

	const long m = perm[i];
	const Quad<TZ> d(foot, i, g);

	if ((0.f == d.w0) && (0.f == d.w1))
		return;

	for (int c = 0; c < C; c++) {

		const float2 val = ksp[m + M * c];

		if ((0.f == val.x) && (0.f == val.y))
			continue;	// grid(): samples that are zero are skipped

		float2* gc = grid + g.gsz * c;
		const long plane = (long)g.G[0] * g.G[1];
#pragma unroll
		for (int a = 0; a < TZ; a++) {

			const float dz = d.f[16 + a];
#pragma unroll
			for (int b = 0; b < 6; b++) {

				const float dzy = __fmul_rn(dz, d.wy[b]);

				if (0.f == dzy)		// clipped tap
					continue;

				const float d0 = __fmul_rn(dzy, d.w0), d1 = __fmul_rn(dzy, d.w1);
				atomicAdd((float4*)(gc + (d.zc[a] * plane + d.row[b])),
						make_float4(val.x * d0, val.y * d0, val.x * d1, val.y * d1));
			}
		}
	}
}

// Gridding, width 6, output-stationary (the default scatter) ------------------
//
// The grid is cut into tiles of TX x LY x LZ cells of the centred oversampled
// grid. One warp job owns one tile (or a chunk of its samples) and a group of
// coils: lane (line, grp) holds the TX x-cells of tile line (y, z) = line for
// CT coils in registers, so it accumulates without atomics. The samples whose
// footprint meets a tile (their hits: a sample has 2.1 in a 16 x 8 tile, 8.2
// in an 8 x 4 x 4 one) are listed per tile at plan time; before, a job tested
// every sample of the 3^d neighbour bins (9 or 27 per sample), which took half
// of its instructions. A job takes its hits 32 at a time: footprint records
// and coil values (k-space in bin order, a sample's coils side by side) arrive
// by cp.async while the previous batch accumulates, the warp fills a table of
// every hit's weight on every tile line, and then adds hit after hit, the next
// one's weights and values loaded ahead. The x offset of a sample is the same
// for the whole warp, so a switch on it selects a fully unrolled update of
// exactly the taps inside the tile; lanes whose line is outside the sample's
// y/z window skip it. Bound by instruction issue (8-coil 128^3 kooshball, 5.12 M
// samples: 10.1 ms testing candidates, 6.3 ms with hit lists and packed sums).
//
// Work items: tiles with one chunk of hits write their cells with plain stores
// (empty tiles write zeros, so the grid needs no clearing), tiles with several
// chunks (the dense k-space centre) add their chunks with atomics into cells
// that k_zero_tiles cleared, or in deterministic mode (hits listed in sample
// order) leave partial tiles that k_sum_tiles adds in chunk order. Cells travel
// in pairs (16 bytes): tile edges and grid sides are even. Weights are those of axis_taps6 (bit-identical to the
// reference's grid_point_gen, src/noncart/grid.c:403-465) and the combined
// weight the same float32 product ((1 * wz) * wy) * wx.

enum { TG_WARPS = 4 };

struct TileWork {

	const long* hit_start;		// [ntiles + 1]
	const int* hits;		// sorted-sample indices by tile
	const int* work_tile;		// [nwork] tile of a work item
	const int* work_chunk;		// [nwork] chunk of the tile's hits
	const int* nwork_dev;		// number of work items
	const float4* foot;		// [M][FOOT_F4] footprints of the sorted samples
	int chunk;			// hits per work item
	const int* slot;		// deterministic: first partial of each tile with several items
	float2* part;			// [slots][C][cells of a tile] its chunks' partial tiles (null: atomics)
};

__device__ __forceinline__ int dft_index(int c, int N, int G);
__device__ __forceinline__ int foot_rel(int lo, int origin, int G, int periodic);

// The hits of every tile: the samples of its 3^d neighbour bins (bins are tiles;
// a footprint reaches three cells either side of its sample) whose footprint
// meets it, in bin order, so the lists are the same every time. The x neighbours
// of a row of bins are one range of the sorted samples (two where a periodic grid
// wraps), and all ranges are walked as one list of candidates. lo: the footprints'
// start cells. work_start == nullptr: count into nhits; else fill hits from
// hit_start on, and the tile's work items.
// k_tile_hits: a block per tile. k_tile_hits_warp: a warp per tile of at most
// TH_WARP_MOST candidates, the other ones into a list for k_tile_hits. The warps
// serve grids of more than TH_TILES tiles (few tiles are latency, and the blocks'
// form has two launches less) with less than TH_MEAN candidates on average. Plan
// creation by blocks and by warps, radial samples: 128^3, 384 000 samples (79
// candidates) 1025 and 419 us; 5.12 million (1055) 3.30 and 2.94 ms; 64^3, 192 000
// (316) 302 and 267 us; 768 000 (1266) 691 and 712; 256^2, 49 000 in 2048 tiles 101
// and 127; uniform samples on a 1024^3 grid (16) 47 and 8.2 ms.
enum { TH_THREADS = 256, TH_RANGES = 18, TH_WARP_MOST = 1024, TH_MEAN = 1200, TH_TILES = 8192 };

struct TileHits {

	int* nhits;			// count
	const long* hit_start;		// fill
	int* hits;
	const int* work_start;
	int* work_tile;
	int* work_chunk;
};

__device__ __forceinline__ int hit_ranges(const BinGeom& bg) { return 2 * ((bg.nb[1] > 1) ? 3 : 1) * ((bg.nb[2] > 1) ? 3 : 1); }

// range r (first sample, samples) of tile (bx, by, bz): part (0, or 1 past the
// periodic edge) of a neighbour row
__device__ __forceinline__ int2 hit_range(int r, int bx, int by, int bz, const int* bin_start, const GridGeom& g, const BinGeom& bg)
{
	const int ry = (bg.nb[1] > 1) ? 1 : 0, rz = (bg.nb[2] > 1) ? 1 : 0;
	int y = by + (r / 2) % (2 * ry + 1) - ry, z = bz + (r / 2) / (2 * ry + 1) - rz;
	int x0 = bx - 1, x1 = bx + 2;

	if (g.periodic) {

		y = (y < 0) ? y + bg.nb[1] : ((y >= bg.nb[1]) ? y - bg.nb[1] : y);
		z = (z < 0) ? z + bg.nb[2] : ((z >= bg.nb[2]) ? z - bg.nb[2] : z);
	}

	bool ok = (y >= 0) && (y < bg.nb[1]) && (z >= 0) && (z < bg.nb[2]);

	if (0 == r % 2) {

		x0 = max(x0, 0);
		x1 = min(x1, bg.nb[0]);

	} else {

		ok = ok && g.periodic && ((x0 < 0) || (x1 > bg.nb[0]));
		x0 = (x0 < 0) ? bg.nb[0] - 1 : 0;
		x1 = x0 + 1;
	}

	const long row = (long)bg.nb[0] * (y + (long)bg.nb[1] * z);
	const int s0 = ok ? bin_start[row + x0] : 0;
	return make_int2(s0, ok ? bin_start[row + x1] - s0 : 0);
}

// a sample's footprint meets the tile at (ox, oy, oz)
__device__ __forceinline__ bool is_hit(short4 l, int ox, int oy, int oz, const GridGeom& g, const BinGeom& bg)
{
	const int lx = foot_rel(l.x, ox, g.G[0], g.periodic), ly = foot_rel(l.y, oy, g.G[1], g.periodic);
	const int lz = foot_rel(l.z, oz, g.G[2], g.periodic);
	return (lx > -6) && (lx < bg.bs[0]) && (ly > -6) && (ly < bg.bs[1]) && (lz > -6) && (lz < bg.bs[2]);
}

__global__ void __launch_bounds__(TH_THREADS) k_tile_hits_warp(const short4* __restrict__ lo, const int* __restrict__ bin_start,
		GridGeom g, BinGeom bg, long ntiles, TileHits th, int* __restrict__ large, int* __restrict__ nlarge)
{
	const int lane = threadIdx.x % 32, nr = hit_ranges(bg);

	for (long t = ((long)blockIdx.x * TH_THREADS + threadIdx.x) / 32; t < ntiles; t += (long)gridDim.x * (TH_THREADS / 32)) {

		const int bx = (int)(t % bg.nb[0]), by = (int)((t / bg.nb[0]) % bg.nb[1]), bz = (int)(t / ((long)bg.nb[0] * bg.nb[1]));
		const int ox = bx * bg.bs[0], oy = by * bg.bs[1], oz = bz * bg.bs[2];

		if (th.work_start && (th.hit_start[t] == th.hit_start[t + 1])) {	// no hits: one work item

			if (0 == lane) {

				th.work_tile[th.work_start[t]] = (int)t;
				th.work_chunk[th.work_start[t]] = 0;
			}

			continue;
		}

		const int2 range = (lane < nr) ? hit_range(lane, bx, by, bz, bin_start, g, bg) : make_int2(0, 0);
		int end = range.y;		// candidates up to this lane's range

		for (int o = 1; o < 32; o <<= 1) {

			const int u = __shfl_up_sync(0xffffffffu, end, o);
			end += (lane >= o) ? u : 0;
		}

		const int total = __shfl_sync(0xffffffffu, end, 31);

		if (total > TH_WARP_MOST) {

			if (!th.work_start && (0 == lane))
				large[atomicAdd(nlarge, 1)] = (int)t;

			continue;
		}

		int* dst = th.work_start ? th.hits + th.hit_start[t] : nullptr;
		int n = 0;

		for (int base = 0; base < total; base += 32) {

			const int c = base + lane;
			int r = 0;		// the candidate's range: the first that ends after it
#pragma unroll
			for (int step = 16; step > 0; step /= 2)
				r += (c >= __shfl_sync(0xffffffffu, end, r + step - 1)) ? step : 0;

			const int i = __shfl_sync(0xffffffffu, range.x + range.y - end, r) + c;
			const bool hit = (c < total) && is_hit(lo[i], ox, oy, oz, g, bg);
			const unsigned m = __ballot_sync(0xffffffffu, hit);

			if (hit && dst)
				dst[n + __popc(m & ((1u << lane) - 1u))] = i;

			n += __popc(m);
		}

		if (!th.work_start) {

			if (0 == lane)
				th.nhits[t] = n;

		} else {

			const int w0 = th.work_start[t], w1 = th.work_start[t + 1];

			for (int w = w0 + lane; w < w1; w += 32) {

				th.work_tile[w] = (int)t;
				th.work_chunk[w] = w - w0;
			}
		}
	}
}

// LIST: takes the *nlist tiles of list instead of all
template <bool LIST>
__global__ void __launch_bounds__(TH_THREADS, 6) k_tile_hits(const short4* __restrict__ lo, const int* __restrict__ bin_start,
		GridGeom g, BinGeom bg, long ntiles, TileHits th, const int* __restrict__ list, const int* __restrict__ nlist)
{
	__shared__ int wcount[TH_THREADS / 32];
	__shared__ int rs[TH_RANGES], rn[TH_RANGES];	// ranges: first sample, samples
	const int warp = threadIdx.x / 32, lane = threadIdx.x % 32, nr = hit_ranges(bg);
	const long n = LIST ? *nlist : ntiles;

	for (long j = blockIdx.x; j < n; j += gridDim.x) {

		const long t = LIST ? list[j] : j;
		const int bx = (int)(t % bg.nb[0]), by = (int)((t / bg.nb[0]) % bg.nb[1]), bz = (int)(t / ((long)bg.nb[0] * bg.nb[1]));
		const int ox = bx * bg.bs[0], oy = by * bg.bs[1], oz = bz * bg.bs[2];

		if ((int)threadIdx.x < nr) {

			const int2 range = hit_range(threadIdx.x, bx, by, bz, bin_start, g, bg);
			rs[threadIdx.x] = range.x;
			rn[threadIdx.x] = range.y;
		}

		__syncthreads();
		int total = 0;

		for (int r = 0; r < nr; r++)
			total += rn[r];

		int* dst = th.work_start ? th.hits + th.hit_start[t] : nullptr;	// the tile's list
		int pos = 0;
		int count = 0, r = 0, r0 = 0;	// this thread's range and its first candidate

		// candidate c of the list (the thread's next one is loaded ahead)
		auto cand = [&](int c, int& i, short4& l) {
			if (c >= total) {

				i = -1;
				return;
			}

			while (c - r0 >= rn[r])
				r0 += rn[r++];

			i = rs[r] + c - r0;
			l = lo[i];
		};

		int in = -1;
		short4 ln = make_short4(0, 0, 0, 0);
		cand(threadIdx.x, in, ln);

		for (int base = 0; base < total; base += TH_THREADS) {

			const int i = in;
			const short4 l = ln;
			cand(base + TH_THREADS + threadIdx.x, in, ln);
			const bool hit = (i >= 0) && is_hit(l, ox, oy, oz, g, bg);

			if (!th.work_start) {

				count += hit;
				continue;
			}

			const unsigned m = __ballot_sync(0xffffffffu, hit);
			__syncthreads();	// the previous counts have been read

			if (0 == lane)
				wcount[warp] = __popc(m);

			__syncthreads();
			int at = pos + __popc(m & ((1u << lane) - 1u));
#pragma unroll
			for (int w = 0; w < TH_THREADS / 32; w++) {

				at += (w < warp) ? wcount[w] : 0;
				pos += wcount[w];
			}

			if (hit)
				dst[at] = i;
		}

		if (!th.work_start) {

			for (int o = 16; o > 0; o >>= 1)
				count += __shfl_xor_sync(0xffffffffu, count, o);

			if (0 == lane)
				wcount[warp] = count;

			__syncthreads();

			if (0 == threadIdx.x) {

				int sum = 0;

				for (int w = 0; w < TH_THREADS / 32; w++)
					sum += wcount[w];

				th.nhits[t] = sum;
			}

		} else {

			const int w0 = th.work_start[t], w1 = th.work_start[t + 1];

			for (int w = w0 + threadIdx.x; w < w1; w += TH_THREADS) {

				th.work_tile[w] = (int)t;
				th.work_chunk[w] = w - w0;
			}
		}

		__syncthreads();	// before the next tile's ranges
	}
}

// exclusive sum of one value per thread over the block (sh: 33 ints), the total
// in every thread
__device__ __forceinline__ int block_scan(int v, int* sh, int& total)
{
	const int warp = threadIdx.x / 32, lane = threadIdx.x % 32;
	int incl = v;

	for (int o = 1; o < 32; o <<= 1) {

		const int u = __shfl_up_sync(0xffffffffu, incl, o);
		incl += (lane >= o) ? u : 0;
	}

	if (31 == lane)
		sh[warp] = incl;

	__syncthreads();

	if (0 == warp) {

		const int n = (lane < (int)(blockDim.x / 32)) ? sh[lane] : 0;
		int s = n;

		for (int o = 1; o < 32; o <<= 1) {

			const int u = __shfl_up_sync(0xffffffffu, s, o);
			s += (lane >= o) ? u : 0;
		}

		sh[lane] = s - n;

		if (31 == lane)
			sh[32] = s;
	}

	__syncthreads();
	const int r = sh[warp] + incl - v;
	total = sh[32];
	__syncthreads();
	return r;
}

// exclusive sums of n values by one block: out[0 .. n], out[n] the total
__global__ void __launch_bounds__(1024) k_scan(const int* __restrict__ in, int n, int* __restrict__ out)
{
	__shared__ int sh[33];
	int sum = 0;

	for (int base = 0; base < n; base += 1024) {

		const int t = base + threadIdx.x;
		int total;
		const int e = block_scan((t < n) ? in[t] : 0, sh, total);

		if (t < n)
			out[t] = sum + e;

		sum += total;
	}

	if (0 == threadIdx.x)
		out[n] = sum;
}

// What precedes a tile: hits, work items, partial tiles (of tiles with several
// items) and tiles with several items.
struct TileSums {

	long hits;
	int work, slots, multi;
};

// work items of a tile: chunks of its hits, at least one
__device__ __forceinline__ int tile_items(int n, int chunk) { return (n > 0) ? (n - 1) / chunk + 1 : 1; }

// the sums over the block's threads, in every thread (sh: one per warp)
__device__ __forceinline__ TileSums block_sums(TileSums v, TileSums* sh)
{
	for (int o = 16; o > 0; o >>= 1) {

		v.hits += __shfl_xor_sync(0xffffffffu, v.hits, o);
		v.work += __shfl_xor_sync(0xffffffffu, v.work, o);
		v.slots += __shfl_xor_sync(0xffffffffu, v.slots, o);
		v.multi += __shfl_xor_sync(0xffffffffu, v.multi, o);
	}

	if (0 == threadIdx.x % 32)
		sh[threadIdx.x / 32] = v;

	__syncthreads();
	TileSums r = { 0, 0, 0, 0 };

	for (int w = 0; w < (int)(blockDim.x / 32); w++) {

		r.hits += sh[w].hits;
		r.work += sh[w].work;
		r.slots += sh[w].slots;
		r.multi += sh[w].multi;
	}

	__syncthreads();
	return r;
}

// the sums of each segment of seg tiles, a block per segment
__global__ void __launch_bounds__(1024) k_tile_sums(const int* __restrict__ nhits, int ntiles, int chunk, int seg,
		TileSums* __restrict__ sums)
{
	__shared__ TileSums sh[32];
	const int t0 = blockIdx.x * seg, t1 = min(ntiles - t0, seg) + t0;
	TileSums v = { 0, 0, 0, 0 };

	for (int t = t0 + threadIdx.x; t < t1; t += 1024) {

		const int n = nhits[t], k = tile_items(n, chunk);
		v.hits += n;
		v.work += k;
		v.slots += (k > 1) ? k : 0;
		v.multi += (k > 1) ? 1 : 0;
	}

	v = block_sums(v, sh);

	if (0 == threadIdx.x)
		sums[blockIdx.x] = v;
}

// From the hits per tile: where each tile's hits, work items (chunks of hits, at
// least one) and, for tiles with several items, partial tiles begin (slot;
// deterministic mode), and the list of those tiles. A block takes a segment of
// seg tiles; sums: of the segments (not read by a single one).
__global__ void __launch_bounds__(1024) k_tile_plan(const int* __restrict__ nhits, int ntiles, int chunk, int seg,
		const TileSums* __restrict__ sums, long* __restrict__ hit_start, int* __restrict__ work_start,
		int* __restrict__ slot, int* __restrict__ multi)
{
	__shared__ int sh[33];
	__shared__ TileSums shs[32];
	const int t0 = blockIdx.x * seg, t1 = min(ntiles - t0, seg) + t0;
	TileSums before = { 0, 0, 0, 0 };

	if (blockIdx.x > 0) {

		for (int b = threadIdx.x; b < (int)blockIdx.x; b += 1024) {

			const TileSums v = sums[b];
			before.hits += v.hits;
			before.work += v.work;
			before.slots += v.slots;
			before.multi += v.multi;
		}

		before = block_sums(before, shs);
	}

	for (int base = t0; base < t1; base += 1024) {

		const int t = base + threadIdx.x;
		const bool in = (t < t1);
		const int n = in ? nhits[t] : 0;
		const int k = in ? tile_items(n, chunk) : 0;
		const bool several = (k > 1);
		int tl, th, tw, ts, tm;
		const int l = block_scan(n & 0xfffff, sh, tl), h = block_scan(n >> 20, sh, th);	// 1024 counts below 2^31
		const int w = block_scan(k, sh, tw);
		const int s = block_scan(several ? k : 0, sh, ts), m = block_scan(several ? 1 : 0, sh, tm);

		if (in) {

			hit_start[t] = before.hits + l + ((long)h << 20);
			work_start[t] = before.work + w;

			if (slot)
				slot[t] = before.slots + s;

			if (several)
				multi[before.multi + m] = t;
		}

		before.hits += tl + ((long)th << 20);
		before.work += tw;
		before.slots += ts;
		before.multi += tm;
	}

	if ((t1 == ntiles) && (0 == threadIdx.x)) {

		hit_start[ntiles] = before.hits;
		work_start[ntiles] = before.work;

		if (slot)
			slot[ntiles] = before.slots;

		multi[ntiles] = before.multi;
	}
}

// deterministic mode: the tiles with several chunks as the sums of their partial
// tiles in chunk order; a block per tile and channel, a thread per cell (all
// tile shapes of this mode have 128 cells)
enum { TG_DET_CELLS = 128 };

__global__ void __launch_bounds__(TG_DET_CELLS) k_sum_tiles(float2* __restrict__ grid, GridGeom g, BinGeom bg,
		const int* __restrict__ multi, const int* __restrict__ nmulti, const int* __restrict__ work_start,
		const int* __restrict__ slot, const float2* __restrict__ part, int C)
{
	const int e = threadIdx.x;
	const long n = (long)*nmulti * C;

	for (long j = blockIdx.x; j < n; j += gridDim.x) {

		const int t = multi[j / C], c = (int)(j % C);
		const int bx = t % bg.nb[0], by = (t / bg.nb[0]) % bg.nb[1], bz = t / (bg.nb[0] * bg.nb[1]);
		const int chunks = work_start[t + 1] - work_start[t];
		const int cx = bx * bg.bs[0] + e % bg.bs[0];
		const int cy = by * bg.bs[1] + (e / bg.bs[0]) % bg.bs[1];
		const int cz = bz * bg.bs[2] + e / (bg.bs[0] * bg.bs[1]);

		if ((cx >= g.G[0]) || (cy >= g.G[1]) || (cz >= g.G[2]))
			continue;

		const float2* p = part + ((long)slot[t] * C + c) * TG_DET_CELLS + e;
		float2 v = make_float2(0.f, 0.f);
#pragma unroll 8
		for (int k = 0; k < chunks; k++)
			v = cadd(v, p[(long)k * C * TG_DET_CELLS]);

		const long cell = dft_index(cx, g.N[0], g.G[0]) + (long)g.G[0] * (dft_index(cy, g.N[1], g.G[1])
				+ (long)g.G[1] * dft_index(cz, g.N[2], g.G[2]));
		grid[cell + g.gsz * c] = v;
	}
}

// offset of a footprint start relative to a tile origin, along an axis of
// G cells: periodic grids take the representative nearest to the tile
__device__ __forceinline__ int foot_rel(int lo, int origin, int G, int periodic)
{
	int r = lo - origin;

	if (periodic) {

		r %= G;

		if (r > G / 2)
			r -= G;
		else if (r < -G / 2)
			r += G;
	}

	return r;
}

// DFT-order index of centred cell c of an axis (G = 2N cells; 0 for singletons)
__device__ __forceinline__ int dft_index(int c, int N, int G)
{
	if (1 == G)
		return 0;

	c += N;
	return (c >= G) ? c - G : c;
}

// acc[i][c] += (wyz * wx[t]) * v[c] for the taps t whose cell i = RX + t is
// inside the tile (RX a compile-time offset)
template <int TX, int CT, int RX>
__device__ __forceinline__ void tg_accum_x(float2 (&acc)[TX][CT], const float (&wx)[6], float wyz, const float2 (&v)[CT])
{
#pragma unroll
	for (int t = 0; t < 6; t++) {

		if ((RX + t >= 0) && (RX + t < TX)) {

			const float d = __fmul_rn(wyz, wx[t]);
#pragma unroll
			for (int c = 0; c < CT; c++)
				acc[RX + t][c] = cfma(v[c], make_float2(d, d), acc[RX + t][c]);
		}
	}
}

// the update for a sample at x offset rx (-5 .. TX - 1, at most 15)
#define BN_TG_CASE(R) case R: if constexpr (R < TX) tg_accum_x<TX, CT, R>(acc, wx, wyz, v); break;

template <int TX, int CT>
__device__ __forceinline__ void tg_switch(int rx, float2 (&acc)[TX][CT], const float (&wx)[6], float wyz,
		const float2 (&v)[CT])
{
	static_assert(TX <= 16, "x offsets up to 15");

	switch (rx) {
	BN_TG_CASE(-5) BN_TG_CASE(-4) BN_TG_CASE(-3) BN_TG_CASE(-2) BN_TG_CASE(-1)
	BN_TG_CASE(0) BN_TG_CASE(1) BN_TG_CASE(2) BN_TG_CASE(3) BN_TG_CASE(4) BN_TG_CASE(5) BN_TG_CASE(6)
	BN_TG_CASE(7) BN_TG_CASE(8) BN_TG_CASE(9) BN_TG_CASE(10) BN_TG_CASE(11) BN_TG_CASE(12) BN_TG_CASE(13)
	BN_TG_CASE(14) BN_TG_CASE(15)
	default: break;
	}
}

#undef BN_TG_CASE

// grid cells of the tiles that several work items add into: zeroed first, a
// warp per tile and channel
__global__ void k_zero_tiles(float2* __restrict__ grid, GridGeom g, BinGeom bg, const int* __restrict__ multi,
		const int* __restrict__ nmulti, int C)
{
	const int lane = threadIdx.x % 32;
	const long n = (long)*nmulti * C;
	const int half = bg.bs[0] / 2, pairs = half * bg.bs[1] * bg.bs[2];

	for (long j = ((long)blockIdx.x * blockDim.x + threadIdx.x) / 32; j < n; j += (long)gridDim.x * blockDim.x / 32) {

		const int t = multi[j / C], c = (int)(j % C);
		const int bx = t % bg.nb[0], by = (t / bg.nb[0]) % bg.nb[1], bz = t / (bg.nb[0] * bg.nb[1]);

		for (int e = lane; e < pairs; e += 32) {

			const int cx = bx * bg.bs[0] + 2 * (e % half);
			const int cy = by * bg.bs[1] + (e / half) % bg.bs[1];
			const int cz = bz * bg.bs[2] + e / (half * bg.bs[1]);

			if ((cx >= g.G[0]) || (cy >= g.G[1]) || (cz >= g.G[2]))
				continue;

			const long cell = dft_index(cx, g.N[0], g.G[0]) + (long)g.G[0] * (dft_index(cy, g.N[1], g.G[1])
					+ (long)g.G[1] * dft_index(cz, g.N[2], g.G[2]));
			*(float4*)(grid + cell + g.gsz * c) = make_float4(0.f, 0.f, 0.f, 0.f);
		}
	}
}

__device__ __forceinline__ void cp_async(uint32_t dst, const void* src, int bytes)
{
	if (16 == bytes)
		asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" :: "r"(dst), "l"(src));
	else
		asm volatile("cp.async.ca.shared.global [%0], [%1], 8;\n" :: "r"(dst), "l"(src));
}

// shared memory of one warp: two batches of 32 hit records (footprint and CW
// coil values) and the batch's weight table [32][NL]
template <int NL, int CW>
struct TgStage {

	static constexpr int REC = 4 * FOOT_F4 + ((2 * CW + 3) / 4) * 4;	// floats per hit record
	static constexpr int FLOATS = 2 * 32 * REC + 32 * NL;
};

// TX x-cells per lane, LY x LZ lines per tile (LY * LZ divides 32), CT coils
// per lane: a warp job covers CW = (32 / (LY * LZ)) * CT coils. ksp: [M][Cp] in
// bin order, Cp even unless CW = 1, zeros past the last coil.
template <int TX, int LY, int LZ, int CT>
__global__ void __launch_bounds__(32 * TG_WARPS, 4) k_grid6_tiles(long M, GridGeom g, BinGeom bg, TileWork tw, int C,
		int Cp, const float2* __restrict__ ksp, float2* __restrict__ grid)
{
	constexpr int NL = LY * LZ;
	constexpr int GPW = 32 / NL;
	constexpr int CW = GPW * CT;
	static_assert(NL * GPW == 32, "lines per tile must divide 32");
	using ST = TgStage<NL, CW>;
	extern __shared__ __align__(16) float tg_smem[];

	const int warp = threadIdx.x / 32, lane = threadIdx.x % 32;
	const int ncq = (C + CW - 1) / CW;	// coil chunks
	const long job = (long)blockIdx.x * TG_WARPS + warp;
	const long wi = job / ncq;
	const int cq = (int)(job % ncq);

	if (wi >= *tw.nwork_dev)	// warp-uniform; the warps share no barrier
		return;

	float* rec = tg_smem + warp * ST::FLOATS;
	float* wt = rec + 2 * 32 * ST::REC;
	const int tile = tw.work_tile[wi];
	const int bx = tile % bg.nb[0], by = (tile / bg.nb[0]) % bg.nb[1], bz = tile / (bg.nb[0] * bg.nb[1]);
	const int ox = bx * TX, oy = by * LY, oz = bz * LZ;
	const int line = lane % NL, grp = lane / NL;
	const int cw0 = cq * CW;		// first coil of the job
	const int c0 = cw0 + grp * CT;		// first coil of this lane
	const long h0 = tw.hit_start[tile];
	const int nh = (int)(tw.hit_start[tile + 1] - h0);	// (a sample is in a tile's list once)
	const int first = tw.work_chunk[wi] * tw.chunk;
	const int* hits = tw.hits + h0 + first + lane;		// this lane's next hits are 32 apart
	int left = min(nh - first, tw.chunk);

	float2 acc[TX][CT];
#pragma unroll
	for (int i = 0; i < TX; i++)
#pragma unroll
		for (int c = 0; c < CT; c++)
			acc[i][c] = make_float2(0.f, 0.f);

	// lane's record of a batch: footprint and coil values, 16 bytes at a time
	// (8 for a single coil); coils past the padded row stay zero
	const int nv = (1 == CW) ? 1 : min(CW, Cp - cw0);

	if (CW > 1)
		for (int b = 0; b < 2; b++)
			for (int k = nv; k < CW; k++)
				*(float2*)(rec + (b * 32 + lane) * ST::REC + 4 * FOOT_F4 + 2 * k) = make_float2(0.f, 0.f);

	auto fetch = [&](int i, int buf) {
		if (i >= 0) {

			const uint32_t dst = (uint32_t)__cvta_generic_to_shared(rec + (buf * 32 + lane) * ST::REC);
			const float4* f = tw.foot + (long)i * FOOT_F4;
#pragma unroll
			for (int k = 0; k < FOOT_F4; k++)
				cp_async(dst + 16 * k, f + k, 16);

			const float2* v = ksp + (long)i * Cp + cw0;

			if (1 == CW) {

				cp_async(dst + 16 * FOOT_F4, v, 8);

			} else {
#pragma unroll
				for (int k = 0; k < CW; k += 2)
					if (k < nv)
						cp_async(dst + 16 * FOOT_F4 + 8 * k, v + k, 16);
			}
		}

		asm volatile("cp.async.commit_group;\n" ::: "memory");
	};

	int buf = 0;
	int inext = (lane < left) ? hits[0] : -1;
	fetch(inext, 0);
	inext = (32 + lane < left) ? hits[32] : -1;

	for (; left > 0; left -= 32, hits += 32) {

		fetch(inext, buf ^ 1);
		inext = (64 + lane < left) ? hits[64] : -1;
		asm volatile("cp.async.wait_group 1;\n" ::: "memory");
		float* rb = rec + buf * 32 * ST::REC;
		const int n = min(32, left);

		if (lane < n) {	// this lane's own record: offsets relative to the tile

			int* r = (int*)(rb + lane * ST::REC);
			r[0] = foot_rel(r[0], ox, g.G[0], g.periodic);
			r[1] = foot_rel(r[1], oy, g.G[1], g.periodic);
			r[2] = foot_rel(r[2], oz, g.G[2], g.periodic);
		}

		__syncwarp();
#pragma unroll 4
		for (int e = lane; e < n * NL; e += 32) {

			const int l = e % NL;
			const float* r = rb + (e / NL) * ST::REC;
			const int ty = l % LY - __float_as_int(r[1]), tz = l / LY - __float_as_int(r[2]);
			const bool in = (ty >= 0) && (ty < 6) && (tz >= 0) && (tz < 6);
			wt[e] = in ? __fmul_rn(r[16 + tz], r[10 + ty]) : 0.f;
		}

		__syncwarp();

		// one hit's inputs: the line's weight, the x weights and offset, the values
		auto load = [&](int q, float& wyz, float (&wx)[6], int& rx, float2 (&v)[CT]) {
			const float* r = rb + q * ST::REC;
			wyz = wt[q * NL + line];
			rx = __float_as_int(r[0]);
			const float4 a = *(const float4*)(r + 4);
			const float2 b = *(const float2*)(r + 8);
			wx[0] = a.x, wx[1] = a.y, wx[2] = a.z, wx[3] = a.w, wx[4] = b.x, wx[5] = b.y;
			const float2* vp = (const float2*)(r + 4 * FOOT_F4) + grp * CT;

			if constexpr (0 == CT % 2) {
#pragma unroll
				for (int c = 0; c < CT; c += 2) {

					const float4 t = *(const float4*)(vp + c);
					v[c] = make_float2(t.x, t.y);
					v[c + 1] = make_float2(t.z, t.w);
				}

			} else {
#pragma unroll
				for (int c = 0; c < CT; c++)
					v[c] = vp[c];
			}
		};

		// two sets of inputs in turn: one is loaded while the other is added
		float wyz[2], wx[2][6];
		int rx[2];
		float2 v[2][CT];
		load(0, wyz[0], wx[0], rx[0], v[0]);

		for (int q = 0; q < n; q += 2) {

			load(min(q + 1, n - 1), wyz[1], wx[1], rx[1], v[1]);

			if (0.f != wyz[0])
				tg_switch<TX, CT>(rx[0], acc, wx[0], wyz[0], v[0]);

			load(min(q + 2, n - 1), wyz[0], wx[0], rx[0], v[0]);

			if ((0.f != wyz[1]) && (q + 1 < n))
				tg_switch<TX, CT>(rx[1], acc, wx[1], wyz[1], v[1]);
		}

		__syncwarp();	// before the batch after next overwrites this buffer
		buf ^= 1;
	}

	// this lane's line: TX cells from ox along x
	const int cy = oy + line % LY, cz = oz + line / LY;

	if ((cy >= g.G[1]) || (cz >= g.G[2]))
		return;

	const bool add = (nh > tw.chunk);
	const long row = (long)g.G[0] * (dft_index(cy, g.N[1], g.G[1]) + (long)g.G[1] * dft_index(cz, g.N[2], g.G[2]));
#pragma unroll
	for (int i = 0; i < TX; i += 2) {

		const int cx = ox + i;

		if (cx >= g.G[0])
			break;

		const long cell = row + dft_index(cx, g.N[0], g.G[0]);
#pragma unroll
		for (int c = 0; c < CT; c++) {

			if (c0 + c >= C)
				break;

			float4* dst = (float4*)(grid + cell + g.gsz * (c0 + c));
			const float4 v = make_float4(acc[i][c].x, acc[i][c].y, acc[i + 1][c].x, acc[i + 1][c].y);

			if (!add)
				*dst = v;
			else if (tw.part)
				*(float4*)(tw.part + (((long)tw.slot[tile] + tw.work_chunk[wi]) * C + c0 + c) * (TX * NL) + line * TX + i) = v;
			else
				atomicAdd(dst, v);
		}
	}
}

// ksp [M, C] into bin order with a sample's coils side by side:
// dst[i][c] = src[perm[i] + M c], zeros for C <= c < Cp; times the conjugate
// of the weights (w, wc channels) if given. grid (ceil(M / 32), ceil(Cp / 32)).
__global__ void __launch_bounds__(256) k_permute_ksp(float2* __restrict__ dst, const float2* __restrict__ src,
		const int* __restrict__ perm, long M, int C, int Cp, const float2* __restrict__ w, int wc)
{
	__shared__ float2 t[32][33];
	const int warp = threadIdx.x / 32, lane = threadIdx.x % 32;
	const long i0 = (long)blockIdx.x * 32;
	const int cb = blockIdx.y * 32, cn = min(32, Cp - cb);
	const long m = (i0 + lane < M) ? perm[i0 + lane] : 0;

	for (int c = warp; c < cn; c += 8) {

		float2 v = (cb + c < C) ? src[m + M * (cb + c)] : make_float2(0.f, 0.f);

		if (w && (cb + c < C))
			v = cmulc(v, w[m + M * ((cb + c) % wc)]);

		t[c][lane] = v;
	}

	__syncthreads();

	for (int e = threadIdx.x; e < 32 * cn; e += 256) {

		const int i = e / cn, c = e % cn;

		if (i0 + i < M)
			dst[(i0 + i) * Cp + cb + c] = t[c][i];
	}
}

} // namespace bn
