// Max subsampling with 3x3 or 2x2 windows at stride 2, forward and backward, stand-alone and fused behind batch norm ->
// residual add -> ReLU: a thread owns a few adjacent columns of a pair
// (or two) of rows of one plane. Included by
// nnf_maxpool.cu only.
//
// What bounds these layers is HBM. The plane-group kernels of nnf_maxpool.cu, which take every other window and some of these, stage whole planes
// in shared memory between a load phase and a window phase, and spend nine shared-memory reads and their index arithmetic
// on every window; here every element is read into a register once, a row's horizontal maximum is shared by the two windows
// that overlap in that row, the columns a window needs from its right-hand neighbour come by shuffle, and there is no barrier.
// Forward, a window is the horizontal maxima of its rows combined downwards: first row first, later rows only on a strict
// compare, the same winner as the plain backend's row-by-row scan (max_subsampling_layer_updater_plain.cpp:146-159). A NaN can
// win there only as the first element of the window, so row maxima ignore NaNs and the first element is looked at by itself.
// Backward, an element adds the gradients of the (at most four) windows around it whose argmax is the element, in ascending
// output index.
//
// A: the widest access (4, 2 or 1 values) that divides the row and suits the buffers' alignment. Threads follow one another over the
// columns, then the row pairs, then the planes, so no lane idles whatever the width; forward with 3x3 windows the last lane of a warp only
// supplies a column to its neighbour and is served again by the next warp (3 % of the loads, from L1).
// Measured, forward / backward, with the plane-group kernels before: fused 3x3/2 [256,64,56,56] 145 / 113 -> 119 / 110 us, stand-alone
// 3x3/2 [64,96,55,55] 31 / 31 -> 24 / 24 us, 2x2/2 [1024,128,28,28] 109 / 109 -> 93 / 95 us (copy rate: 94 / 94).
#pragma once

namespace nnf
{
	namespace
	{
		struct rows_params
		{
			// forward: x, residual -> z, pooled, argmax; backward: dpooled (in `pooled`), argmax, z -> dx, dres
			const float * x;
			const float * res;
			float * z;
			float * pooled;
			uint32_t * argmax;
			const float * gamma;
			const float * beta;
			const float * mean;
			const float * invsigma;
			float * dx;
			float * dres;
			float slope;
			int add;
			uint32_t c, h, w, hw, oh, ow, ohw;
			uint32_t cols;             // vectors per row
			uint32_t strips;           // strips of a plane
			uint32_t total;            // planes * strips * cols
			fastdiv d_cols, d_c, d_strips;
		};

		// V adjacent values in accesses of A; PARTIAL: only the first `valid` of them exist
		template <int V, int A, bool PARTIAL>
		__device__ __forceinline__ void load_cols(float (&v)[V], const float * p, uint32_t valid)
		{
			#pragma unroll
			for (int j = 0; j < V; j += A)
				if (!PARTIAL || uint32_t(j) < valid)
				{
					if (A == 4)
					{
						const float4 t = __ldcs(reinterpret_cast<const float4 *>(p));
						v[0] = t.x; v[1 % V] = t.y; v[2 % V] = t.z; v[3 % V] = t.w;
					}
					else if (A == 2)
					{
						const float2 t = __ldcs(reinterpret_cast<const float2 *>(p + j));
						v[j] = t.x; v[(j + 1) % V] = t.y;
					}
					else
						v[j] = __ldcs(p + j);
				}
		}

		template <int V, int A, bool PARTIAL>
		__device__ __forceinline__ void store_cols(float * p, const float (&v)[V], uint32_t valid)
		{
			#pragma unroll
			for (int j = 0; j < V; j += A)
				if (!PARTIAL || uint32_t(j) < valid)
				{
					if (A == 4)
						__stcs(reinterpret_cast<float4 *>(p), make_float4(v[0], v[1 % V], v[2 % V], v[3 % V]));
					else if (A == 2)
						__stcs(reinterpret_cast<float2 *>(p + j), make_float2(v[j], v[(j + 1) % V]));
					else
						__stcs(p + j, v[j]);
				}
		}

		template <bool MIN>
		__device__ __forceinline__ bool rows_better(float a, float b) { return MIN ? a < b : a > b; }

		// best of three (or two) adjacent elements of a row, the first of them at offset `off`; NaNs are passed over
		template <int WIN, bool MIN>
		__device__ __forceinline__ void row_best(float a, float b, float c, uint32_t off, float& best, uint32_t& at)
		{
			const float none = __int_as_float(MIN ? 0x7f800000 : 0xff800000);
			best = rows_better<MIN>(a, none) ? a : none;
			at = off;
			if (rows_better<MIN>(b, best)) { best = b; at = off + 1; }
			if (WIN == 3 && rows_better<MIN>(c, best)) { best = c; at = off + 2; }
		}

		constexpr int kRowsThreads = 256;

		// Columns and pairs of rows of a thread, for accesses of A values. Rows of whole float4s: one float4 of two rows (three with the
		// halo row), so that a CTA's accesses cover one contiguous range of memory; with longer strips the same thread count covers
		// more, shorter pieces, and [1024,128,28,28] 2x2/2 forward goes from 93 to 115 us (two pairs) and 125 us (four), walks of
		// whole planes by a thread to 190 us. Other rows: two columns by scalar (or float2) accesses - one column makes every window's work
		// be done twice (stand-alone [64,96,55,55] forward 41 us against 24), four spread a warp's access over four times its width
		// (backward 36 against 24) - and, where there is nothing but the windows to do, two pairs of rows (29 against 24).
		template <int A, bool FUSED>
		struct rows_shape
		{
			static constexpr int columns = A == 4 ? 4 : 2;
			static constexpr int pairs = A == 4 || FUSED ? 1 : 2;
			static constexpr int windows = A == 4 ? 2 : 1;      // that start in a thread's columns
		};

		template <int A, int WIN, bool FUSED, bool MIN>
		__global__ void __launch_bounds__(kRowsThreads) pool_rows_fwd_kernel(const __grid_constant__ rows_params p)
		{
			constexpr int V = rows_shape<A, FUSED>::columns, PAIRS = rows_shape<A, FUSED>::pairs;
			constexpr int NW = rows_shape<A, FUSED>::windows;
			constexpr int OWN = 32 - (WIN == 3 ? 1 : 0);                  // the last lane only supplies a column to its neighbour
			constexpr bool PARTIAL = A < V;                               // the last thread of a row may own fewer columns
			constexpr int ROWS = 2 * PAIRS + (WIN == 3 ? 1 : 0);          // the last windows end in the next strip's first row
			const uint32_t lane = threadIdx.x & 31;
			const uint32_t q = (blockIdx.x * (kRowsThreads / 32) + (threadIdx.x >> 5)) * OWN + lane;
			const uint32_t qc = min(q, p.total - 1);
			const bool own = lane < OWN && q < p.total;
			const uint32_t band = p.d_cols.div(qc);                       // strip of a plane
			const uint32_t k = qc - band * p.cols;
			const uint32_t plane = p.d_strips.div(band);
			const uint32_t m0 = (band - plane * p.strips) * PAIRS;
			const bool last = k + 1 == p.cols;
			const uint32_t valid = p.w - k * V;                           // columns from the thread's first to the row's end
			const uint32_t row0 = 2 * m0;
			const size_t pbase = size_t(plane) * p.hw + row0 * p.w + k * V;
			const float * x = p.x + pbase;
			const float * res = FUSED && p.res ? p.res + pbase : nullptr;
			float * z = FUSED ? p.z + pbase : nullptr;
			const uint32_t ox = NW * k;                                   // the first window that starts in these columns
			const bool w0 = own && ox < p.ow;
			const bool w1 = NW > 1 && own && ox + 1 < p.ow;
			const size_t obase = size_t(plane) * p.ohw + m0 * p.ow + ox;
			float * pooled = p.pooled + obase;
			uint32_t * argmax = p.argmax ? p.argmax + obase : nullptr;
			const uint32_t abs0 = uint32_t(pbase);
			const float none = __int_as_float(MIN ? 0x7f800000 : 0xff800000);
			pdl_begin_early();

			float v[ROWS][V], rv[ROWS][V];
			#pragma unroll
			for (int u = 0; u < ROWS; ++u)
			{
				#pragma unroll
				for (int i = 0; i < V; ++i)
					v[u][i] = rv[u][i] = none;
				if (row0 + u < p.h)
				{
					load_cols<V, A, PARTIAL>(v[u], x + u * p.w, valid);
					if (res)
						load_cols<V, A, PARTIAL>(rv[u], res + u * p.w, valid);
				}
			}
			float mult = 1.0F, shift = 0.0F;
			const bool has_bn = FUSED && p.gamma != nullptr;
			if (has_bn)
			{
				const uint32_t ch = plane - p.d_c.div(plane) * p.c;
				mult = __fmul_rn(__ldg(p.gamma + ch), __ldg(p.invsigma + ch));
				shift = __fsub_rn(__ldg(p.beta + ch), __fmul_rn(mult, __ldg(p.mean + ch)));
			}

			float best[NW];          // the windows that are open
			uint32_t at[NW];
			#pragma unroll
			for (int u = 0; u < ROWS; ++u)
			{
				const bool there = row0 + u < p.h;
				if (FUSED)
				{
					#pragma unroll
					for (int i = 0; i < V; ++i)
					{
						float t = v[u][i];
						if (has_bn)
							t = __fadd_rn(__fmul_rn(t, mult), shift);
						if (res)
							t = __fadd_rn(__fadd_rn(0.0F, t), rv[u][i]); // add layer, alpha = 1: (0 + bn) + residual
						v[u][i] = t >= 0.0F ? t : __fmul_rn(t, p.slope);
						if (PARTIAL && uint32_t(i) >= valid)
							v[u][i] = none;
					}
					if (u < 2 * PAIRS && there && own)
						store_cols<V, A, PARTIAL>(z + u * p.w, v[u], valid);
				}
				// the row's best of every window that starts in these columns; a row or a column past the plane is never better
				float rb[NW];
				uint32_t ra[NW];
				float nx = WIN == 3 ? __shfl_down_sync(0xffffffffu, v[u][0], 1) : 0.0F;
				nx = last ? none : nx;
				#pragma unroll
				for (int i = 0; i < NW; ++i)
					row_best<WIN, MIN>(v[u][2 * i], v[u][2 * i + 1], 2 * i + 2 < V ? v[u][(2 * i + 2) % V] : nx, u * p.w + 2 * i, rb[i], ra[i]);
				auto merge = [&]()
				{
					#pragma unroll
					for (int i = 0; i < NW; ++i)
						if (there && rows_better<MIN>(rb[i], best[i]))
						{
							best[i] = rb[i];
							at[i] = ra[i];
						}
				};
				auto emit = [&](uint32_t m)
				{
					if (m0 + m < p.oh)
					{
						const uint32_t o = m * p.ow;
						if (w0)
						{
							__stcs(pooled + o, best[0]);
							if (argmax) __stcs(argmax + o, abs0 + at[0]);
						}
						if (w1)
						{
							__stcs(pooled + o + 1, best[NW - 1]);
							if (argmax) __stcs(argmax + o + 1, abs0 + at[NW - 1]);
						}
					}
				};
				if ((u & 1) == 0)
				{
					if (WIN == 3 && u > 0)
					{
						merge();                   // third row of the windows above
						emit(u / 2 - 1);
					}
					#pragma unroll
					for (int i = 0; i < NW; ++i)
					{
						const bool stays = v[u][2 * i] != v[u][2 * i];           // a NaN that comes first
						best[i] = stays ? v[u][2 * i] : rb[i];
						at[i] = stays ? u * p.w + 2 * i : ra[i];
					}
				}
				else
				{
					merge();
					if (WIN == 2)
						emit(u / 2);
				}
			}
		}

		template <int A, int WIN, bool FUSED>
		__global__ void __launch_bounds__(kRowsThreads) pool_rows_bwd_kernel(const __grid_constant__ rows_params p)
		{
			constexpr int V = rows_shape<A, FUSED>::columns, PAIRS = rows_shape<A, FUSED>::pairs;
			constexpr int NW = V / 2 + (WIN == 3 ? 1 : 0);                        // windows of one output row around a thread's columns
			constexpr int WROWS = PAIRS + (WIN == 3 ? 1 : 0);                     // rows of windows around a strip
			constexpr bool PARTIAL = A < V;
			constexpr uint32_t nowhere = 0xffffffffu;                             // no element has this offset
			const uint32_t q = blockIdx.x * kRowsThreads + threadIdx.x;
			if (q >= p.total)
				return;
			const uint32_t band = p.d_cols.div(q);
			const uint32_t k = q - band * p.cols;
			const uint32_t plane = p.d_strips.div(band);
			const uint32_t m0 = (band - plane * p.strips) * PAIRS;
			const uint32_t row0 = 2 * m0;
			const uint32_t valid = p.w - k * V;
			const size_t pbase = size_t(plane) * p.hw + row0 * p.w + k * V;
			const uint32_t abs0 = uint32_t(pbase);
			// first of the NW windows: the one that ends in these columns (3x3), else the one that starts there; the same for rows
			const int ox0 = int(k * (V / 2)) - (WIN == 3 ? 1 : 0);
			const int oy0 = int(m0) - (WIN == 3 ? 1 : 0);
			bool wok[NW];
			#pragma unroll
			for (int i = 0; i < NW; ++i)
				wok[i] = ox0 + i >= 0 && uint32_t(ox0 + i) < p.ow;
			const int64_t obase = int64_t(plane) * p.ohw + int64_t(oy0) * p.ow + ox0;
			const float * dyp = p.pooled + obase;
			const uint32_t * idp = p.argmax + obase;
			const float * z = FUSED ? p.z + pbase : nullptr;
			float * dx = p.dx ? p.dx + pbase : nullptr;
			float * dres = FUSED && p.dres ? p.dres + pbase : nullptr;
			pdl_begin_early();

			float v[2 * PAIRS][V];       // z, or what dx holds already
			uint32_t id[WROWS][NW];
			float dy[WROWS][NW];
			#pragma unroll
			for (int u = 0; u < WROWS; ++u)
			{
				const bool rok = oy0 + u >= 0 && uint32_t(oy0 + u) < p.oh;
				#pragma unroll
				for (int i = 0; i < NW; ++i)
				{
					id[u][i] = nowhere;
					dy[u][i] = 0.0F;
					if (rok && wok[i])
					{
						id[u][i] = __ldg(idp + u * p.ow + i);
						dy[u][i] = __ldg(dyp + u * p.ow + i);
					}
				}
			}
			#pragma unroll
			for (int u = 0; u < 2 * PAIRS; ++u)
			{
				#pragma unroll
				for (int j = 0; j < V; ++j)
					v[u][j] = 0.0F;
				if (row0 + u < p.h && (FUSED || p.add))
					load_cols<V, A, PARTIAL>(v[u], (FUSED ? z : dx) + u * p.w, valid);
			}
			float mult = 1.0F;
			const bool has_bn = FUSED && p.gamma != nullptr;
			if (has_bn)
			{
				const uint32_t ch = plane - p.d_c.div(plane) * p.c;
				mult = __fmul_rn(__ldg(p.gamma + ch), __ldg(p.invsigma + ch));
			}
			#pragma unroll
			for (int u = 0; u < 2 * PAIRS; ++u)
			{
				if (row0 + u >= p.h)
					return;
				float acc[V];
				#pragma unroll
				for (int j = 0; j < V; ++j)
					acc[j] = FUSED ? 0.0F : v[u][j];
				const uint32_t a = abs0 + u * p.w;
				// rows of windows that reach this row, in ascending order; u / 2 + 1 is the one that starts at an even row
				#pragma unroll
				for (int t = 0; t < 2; ++t)
				{
					const int wr = WIN == 3 ? u / 2 + t : u / 2;
					if ((WIN == 2 && t == 1) || (WIN == 3 && t == 0 && (u & 1)))
						continue;
					#pragma unroll
					for (int i = 0; i < NW; ++i)
					{
						#pragma unroll
						for (int j = 0; j < V; ++j)
						{
							const int from = 2 * i - (WIN == 3 ? 2 : 0);   // window i's columns relative to the thread's first
							if (j >= from && j < from + WIN)
								if (id[wr][i] == a + j)
									acc[j] = __fadd_rn(acc[j], dy[wr][i]);
						}
					}
				}
				if (!FUSED)
				{
					store_cols<V, A, PARTIAL>(dx + u * p.w, acc, valid);
					continue;
				}
				float odx[V], ores[V];
				#pragma unroll
				for (int j = 0; j < V; ++j)
				{
					// ReLU gate from the sign bit of z; the add layer hands the gradient on; frozen batch norm scales it
					const float ds = (__float_as_uint(v[u][j]) >> 31) ? __fmul_rn(acc[j], p.slope) : acc[j];
					ores[j] = ds;
					odx[j] = has_bn ? __fmul_rn(ds, mult) : ds;
				}
				if (dx)
					store_cols<V, A, PARTIAL>(dx + u * p.w, odx, valid);
				if (dres)
					store_cols<V, A, PARTIAL>(dres + u * p.w, ores, valid);
			}
		}

		// From how many values on the plane-group kernels of nnf_maxpool.cu are the faster ones for small planes whose rows are not whole
		// float4s: their groups of planes start and end on float4s, which counts once the tensors leave L2. us, row / plane-group kernels:
		// Fused, four tensors per value (two-thirds of the instructions). Forward the two meet at 1.5 M values where rows are odd (27x27,
		// 34 M values: 97 against 81) and at 6 M where they are even (18x18: 82 against 76), backward at 12 M where rows are odd (21x21,
		// 34 M values: 97 against 92).
		// Stand-alone forward, the row kernels waste the more of a thread's columns and of a halo row the smaller the plane is; 3x3 windows,
		// odd rows: 9x9 10.4 / 9.0 at 5 M values and 44 / 25 at 25 M, 13x13 14.2 / 11.9 at 8 M, 21x21 26 / 23 at 18 M, 23x23 24.4 / 25.7; even
		// rows: 6x6 8.3 / 7.7 at 5 M, 10x10 23 / 21 at 18 M, 14x14 29.6 / 27.3 at 25 M; 2x2 windows: 9x9 11.7 / 10.0 at 8 M, 21x21 20.9 / 19.5
		// at 18 M, 6x6 53 / 50 at 50 M, 10x10 level.
		// Backward, rows of 4: a warp's accesses to its two rows cover every second 16 bytes (fused, 8 M values: 4x4 23.5 / 19.9, 28x4
		// 23.2 / 20.7; stand-alone only the lowest planes, 4x4 55 / 48 at 50 M). Stand-alone 2x2 with odd rows, which the plane groups walk in
		// chunks of four: 7x7 28 / 24 at 18 M, 300x7 30 / 24, 11x11 38 / 33 at 25 M, 300x11 40 / 33; a fourth chunk element that is mostly
		// missing (9x9, 5x5) puts the point where they meet three times as high, and from 13 columns on rows are the faster ones.
		int64_t plane_groups_from(const pool_geom& g, int access, bool aligned, bool fused, bool backward)
		{
			constexpr int64_t million = 1000000, never = int64_t(1) << 62;
			const bool odd = access == 1, three = g.win_w == 3;
			if (access == 4)
				return !backward || g.w > 4 ? never : fused ? 9 * million / 2 : g.h <= 8 ? 18 * million : never;
			if (fused)
			{
				if (g.hw > 1024)
					return never;
				return backward ? (odd && three ? 12 * million : never) : odd ? 3 * million / 2 : 6 * million;
			}
			if (backward)
				return !odd || three || g.w > 11 ? never : g.w % 4 == 3 ? 15 * million / 2 : 24 * million;
			if (!aligned)
				return never;
			if (odd && g.hw < 36)
				return 2 * million;
			if (three)
				return odd ? (g.hw < 100 ? 5 * million / 2 : g.hw <= 169 ? 5 * million : g.hw <= 441 ? 15 * million : never)
					: (g.hw <= 64 ? 4 * million : g.hw <= 100 ? 12 * million : g.hw <= 256 ? 20 * million : never);
			return odd ? (g.hw <= 169 ? 6 * million : g.hw <= 441 ? 16 * million : never) : g.hw <= 49 ? 35 * million : never;
		}

		// Whether the row kernels take this layer, and the access width. `align`: the common alignment of the full-size buffers in bytes.
		bool plan_rows(rows_params& q, int& access, const pool_geom& g, int64_t planes, size_t align, bool fused, bool backward)
		{
			if (!(g.win_w == g.win_h && (g.win_w == 3 || g.win_w == 2) && g.sw == 2 && g.sh == 2) || tune().pool_staged == 1)
				return false;
			access = (g.w % 4 == 0 && align % 16 == 0) ? 4 : ((g.w % 2 == 0 && align % 8 == 0) ? 2 : 1);
			if (planes * g.hw >= plane_groups_from(g, access, align % 16 == 0, fused, backward))
				return false;
			q.c = g.c; q.h = g.h; q.w = g.w; q.hw = g.hw; q.oh = g.oh; q.ow = g.ow; q.ohw = g.ohw;
			q.cols = (uint32_t)div_up(g.w, access == 4 ? 4 : 2);
			q.strips = (uint32_t)div_up(g.h, access == 4 || fused ? 2 : 4);
			const int64_t total = planes * q.strips * q.cols;
			if (total > kMaxElemsPerLaunch)
				return false;
			q.total = (uint32_t)total;
			q.d_cols = fastdiv(q.cols);
			q.d_c = fastdiv(g.c);
			q.d_strips = fastdiv(q.strips);
			return true;
		}

		template <int A, int WIN, bool FUSED>
		void launch_rows_fwd(const rows_params& q, bool is_min, cudaStream_t s)
		{
			constexpr int OWN = 32 - (WIN == 3 ? 1 : 0);
			const int64_t grid = div_up(div_up(q.total, OWN), kRowsThreads / 32);
			if (is_min)
				launch(pool_rows_fwd_kernel<A, WIN, FUSED, true>, grid, kRowsThreads, 0, s, q);
			else
				launch(pool_rows_fwd_kernel<A, WIN, FUSED, false>, grid, kRowsThreads, 0, s, q);
		}

		template <int A, bool FUSED>
		void rows_fwd(const rows_params& q, int win, bool is_min, cudaStream_t s)
		{
			if (win == 3) launch_rows_fwd<A, 3, FUSED>(q, is_min, s);
			else launch_rows_fwd<A, 2, FUSED>(q, is_min, s);
		}

		template <int A, bool FUSED>
		void rows_bwd(const rows_params& q, int win, cudaStream_t s)
		{
			const int64_t grid = div_up(q.total, kRowsThreads);
			if (win == 3) launch(pool_rows_bwd_kernel<A, 3, FUSED>, grid, kRowsThreads, 0, s, q);
			else launch(pool_rows_bwd_kernel<A, 2, FUSED>, grid, kRowsThreads, 0, s, q);
		}
	}
}
