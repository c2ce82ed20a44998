// Training batch norm (+ activation chain) of channels that fit on chip: one thread-block cluster per channel. Its CTAs share
// the entries; each copies its slice of x (backward: and dy) into shared memory once, the partial sums cross the cluster
// through distributed shared memory, and the result is computed from shared memory: global memory carries every tensor once, and
// a launch has no workspace to clear, no counter, no flag to poll and no second launch behind it.
//
// What bounds it: HBM for tensors that do not fit L2; for small ones the launch and one chain of latencies (copy, cluster
// barrier, store). A plane may start and end anywhere (27x27, 13x13): a row of the tile is the plane's 16-byte frame, that is
// every 16-byte piece that holds an element of it, copied and read as whole float4s; the up to three elements of the neighbouring
// channels at either end are left out of the sums and of the stores. A thread reads back only the pieces that it copied itself
// (cp.async), so there is no barrier between the copies and the sums.
//
// One B200, forward / backward, ReLU, us (the form that took the shape before; 8 and 12 bytes per element at the copy rate):
//   x[128,96,27,27]   22.2 / 34.8   (two kernels per direction 32.6 / 84.8;        11.0 / 16.4)
//   x[32,64,16,16]     4.0 /  6.8   (statistics and apply items 10.4 / 13.4;        0.6 /  1.0)
//   x[256,512,7,7]    17.3 / 26.6   (channel groups 22.1 / 30.1;                    7.9 / 11.8)
//   x[256,512,14,14]  45.2 / 75.2   (statistics and apply items 63.0 / 91.2;       31.4 / 47.1)
// A CTA's life is copies, about 4 us of latencies (sums, barrier, constants, first store) and stores, and the shared memory it
// holds meanwhile is what limits the bytes in flight. Backward, the first CTA of a channel's cluster is held longest: one thread updates
// up to five per-channel gradients, each a round trip to memory behind the one before it, in front of the barrier that the result
// waits for. Persistent clusters with a ring of two to four channels, the next ones'
// copies and sums overlapping a channel's exchange, were slower at every shape (x[256,512,14,14] forward 52.8): about 2 us of
// barriers per channel in series, and clusters of 8 resident on 120 of the SMs only.
#include "nnf_common.cuh"

namespace nnf
{
	namespace
	{
		constexpr int kClusterMaxThreads = 512;
		constexpr uint32_t kClusterMax = 8;       // CTAs per channel (the portable cluster size)
		constexpr int kClusterStages = 4;         // groups of a thread's copies that are waited for one after another

		struct cluster_params
		{
			const float * x;
			const float * dy;        // backward only
			float * out;             // y (forward) or dx (backward)
			const float * gamma;
			const float * beta;
			float * saved;           // forward: written {mean, invstd}; backward: read
			float * sums;            // forward: {sum x, sum x^2} (may be null); backward: bsums[3C]
			float * grad_gamma, * grad_beta, * grad_mean, * grad_invsigma, * grad_slope;
			const float * mean, * invsigma;
			float entry_count;
			act_chain chain;
			uint32_t n, c, hw;
			uint32_t cluster;        // CTAs per channel
			uint32_t entries;        // per CTA
			uint32_t pitch;          // float4s of a row of the tile
			uint32_t row_stride;     // elements from one entry to the next
			uint32_t per_stage;      // float4s of a tile that are copied and waited for together
			fastdiv d_pitch;
			uint32_t total;          // elements of the tensor
			double count, per_count; // elements of a channel, and 1 / that
			float eps;
			uint32_t * report;       // 64 words to be cleared, or null
		};

		__device__ __forceinline__ uint32_t cluster_rank()
		{
			uint32_t r;
			asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
			return r;
		}

		__device__ __forceinline__ void cluster_arrive() { asm volatile("barrier.cluster.arrive.release;" ::: "memory"); }
		__device__ __forceinline__ void cluster_wait() { asm volatile("barrier.cluster.wait.acquire;" ::: "memory"); }

		// stores into the shared memory of another CTA of the cluster, at the address that `p` has in this one
		__device__ __forceinline__ void st_cluster(const double * p, uint32_t rank, double v)
		{
			uint32_t a;
			asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(a) : "r"((uint32_t)__cvta_generic_to_shared(p)), "r"(rank));
			asm volatile("st.shared::cluster.f64 [%0], %1;" :: "r"(a), "d"(v) : "memory");
		}

		// the first `bytes` of a 16-byte piece; the rest of the piece in shared memory is zero
		__device__ __forceinline__ void copy16(float4 * dst, const float * src, uint32_t bytes)
		{
			asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" :: "r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src), "r"(bytes) : "memory");
		}

		template <int N>
		__device__ __forceinline__ void copies_wait() { asm volatile("cp.async.wait_group %0;" :: "n"(N) : "memory"); }

		// A float4 of the tile: where it is in the tensor and which of its four elements belong to the channel.
		template <bool WHOLE>
		struct piece
		{
			uint32_t at;         // its first element in the tensor
			uint32_t lo, hi;     // elements lo .. hi - 1 of the four are the channel's (hi 0: none)

			// the i-th piece of the CTA's tile; `start`: the first element of the channel's plane in the CTA's first entry
			__device__ __forceinline__ piece(const cluster_params& p, uint32_t start, uint32_t i)
			{
				const uint32_t row = p.d_pitch.div(i);
				const uint32_t v = (i - row * p.pitch) * 4;
				const uint32_t plane = start + row * p.row_stride;
				if (WHOLE)
				{
					at = plane + v;
					lo = 0;
					hi = 4;
				}
				else
				{
					const uint32_t skip = plane & 3;
					at = plane - skip + v;
					lo = v == 0 ? skip : 0;
					hi = skip + p.hw > v ? min(skip + p.hw - v, 4u) : 0;
				}
			}

			__device__ __forceinline__ bool whole() const { return WHOLE || hi - lo == 4; }
			__device__ __forceinline__ bool holds(uint32_t j) const { return j >= lo && j < hi; }
		};

		template <int A0, int A1, bool BWD, bool WHOLE>
		__global__ void __launch_bounds__(kClusterMaxThreads, 2) bn_train_cluster_kernel(const cluster_params p)
		{
			constexpr int K = BWD ? 3 : 2;
			constexpr int U = BWD ? 2 : 4;                       // pieces that a thread reads from shared memory at a time
			extern __shared__ float4 tile[];                     // [x, dy][entries][pitch]
			__shared__ double s_warp[kClusterMaxThreads / 32][K];
			__shared__ double s_part[kClusterMax][K];            // the sums of the cluster's CTAs; each CTA has all of them
			__shared__ float s_const[4];
			pdl_begin_early();
			cluster_arrive();                                    // waited for before the first store into another CTA
			if (p.report && blockIdx.x == 0 && threadIdx.x < 64)
				p.report[threadIdx.x] = 0;

			const uint32_t rank = cluster_rank();
			const uint32_t threads = blockDim.x;
			const uint32_t e0 = rank * p.entries;
			const uint32_t rows = e0 < p.n ? min(p.entries, p.n - e0) : 0;
			const uint32_t pieces = rows * p.pitch;
			// the backward launch walks the channels downwards: whatever ran before it (the forward launch walks upwards) left
			// the highest channels of x in L2
			const uint32_t unit = blockIdx.x / p.cluster;
			const uint32_t ch = BWD ? p.c - 1 - unit : unit;
			const uint32_t start = (e0 * p.c + ch) * p.hw;
			float4 * const tile_d = tile + (BWD ? p.entries * p.pitch : 0);

			#pragma unroll
			for (int g = 0; g < kClusterStages; ++g)
			{
				const uint32_t end = min((g + 1) * p.per_stage, pieces);
				#pragma unroll 4
				for (uint32_t i = g * p.per_stage + threadIdx.x; i < end; i += threads)
				{
					const piece<WHOLE> f(p, start, i);
					// a frame may be a piece shorter than the pitch, and the tensor may end inside the last one (the elements that are
					// left are compared before they become bytes, which 32 bits do not hold from 2^30 elements on)
					const uint32_t bytes = WHOLE ? 16 : f.hi > 0 ? min(4u, p.total - f.at) * 4 : 0;
					const uint32_t at = WHOLE || bytes > 0 ? f.at : 0;
					copy16(tile + i, p.x + at, bytes);
					if (BWD)
						copy16(tile_d + i, p.dy + at, bytes);
				}
				asm volatile("cp.async.commit_group;" ::: "memory");
			}

			const float slope = chain_slope(p.chain, ch);
			const float gamma = __ldg(p.gamma + ch), beta = __ldg(p.beta + ch);
			// forward: the sums are taken around the channel's first element, so that a mean far from zero costs no digits
			const float shift = BWD ? 0.0F : __ldcg(p.x + size_t(ch) * p.hw);
			const float mean = BWD ? __ldcg(p.saved + ch) : 0.0F, invstd = BWD ? __ldcg(p.saved + p.c + ch) : 0.0F;
			const float bmult = gamma * invstd;
			float acc[K];
			#pragma unroll
			for (int k = 0; k < K; ++k)
				acc[k] = 0.0F;
			auto sum_stage = [&](uint32_t g)
			{
				const uint32_t end = min((g + 1) * p.per_stage, pieces);
				for (uint32_t first = g * p.per_stage + threadIdx.x; first < end; first += U * threads)
				{
					float4 a[U], d[BWD ? U : 1];
					#pragma unroll
					for (int u = 0; u < U; ++u)
						if (first + u * threads < end)
						{
							a[u] = tile[first + u * threads];
							if (BWD) d[BWD ? u : 0] = tile_d[first + u * threads];
						}
					#pragma unroll
					for (int u = 0; u < U; ++u)
					{
						const uint32_t i = first + u * threads;
						if (i >= end)
							break;
						const piece<WHOLE> f(p, start, i);
						if constexpr (!BWD)
						{
							float v0 = a[u].x - shift, v1 = a[u].y - shift, v2 = a[u].z - shift, v3 = a[u].w - shift;
							if (!WHOLE)
							{
								v0 = f.holds(0) ? v0 : 0.0F;
								v1 = f.holds(1) ? v1 : 0.0F;
								v2 = f.holds(2) ? v2 : 0.0F;
								v3 = f.holds(3) ? v3 : 0.0F;
							}
							acc[0] += (v0 + v1) + (v2 + v3);
							acc[1] = fmaf(v0, v0, fmaf(v1, v1, fmaf(v2, v2, fmaf(v3, v3, acc[1]))));
						}
						else
						{
							const float xs[4] = {a[u].x, a[u].y, a[u].z, a[u].w};
							const float ds[4] = {d[u].x, d[u].y, d[u].z, d[u].w};
							float du[4];
							#pragma unroll
							for (int j = 0; j < 4; ++j)
							{
								float xc = xs[j] - mean;
								float term;
								du[j] = chain_backward_short<A0, A1>(p.chain, fmaf(xc, bmult, beta), ds[j], slope, term);
								if (!WHOLE && !f.holds(j))
									du[j] = xc = term = 0.0F;
								acc[0] += du[j];
								acc[1] = fmaf(du[j], xc, acc[1]);
								acc[K - 1] += term;
							}
							// the second pass needs du, not dy
							tile_d[i] = make_float4(du[0], du[1], du[2], du[3]);
						}
					}
				}
			};
			static_assert(kClusterStages == 4, "one wait per stage");
			copies_wait<3>(); sum_stage(0);
			copies_wait<2>(); sum_stage(1);
			copies_wait<1>(); sum_stage(2);
			copies_wait<0>(); sum_stage(3);

			// the CTA's sums, in warp order, go to every CTA of the cluster
			#pragma unroll
			for (int k = 0; k < K; ++k)
			{
				double t = double(acc[k]);
				#pragma unroll
				for (int o = 16; o > 0; o >>= 1)
					t += __shfl_xor_sync(0xffffffffu, t, o);
				if ((threadIdx.x & 31) == 0)
					s_warp[threadIdx.x >> 5][k] = t;
			}
			__syncthreads();
			cluster_wait();
			if (threadIdx.x < p.cluster * K)
			{
				const uint32_t to = threadIdx.x / K, k = threadIdx.x - to * K;
				double t = 0.0;
				for (uint32_t w = 0; w < threads / 32; ++w)
					t += s_warp[w][k];
				st_cluster(&s_part[rank][k], to, t);
			}
			cluster_arrive();
			cluster_wait();
			if (threadIdx.x == 0)
			{
				double tot[K];
				#pragma unroll
				for (int k = 0; k < K; ++k)
					tot[k] = 0.0;
				for (uint32_t r = 0; r < p.cluster; ++r)
				{
					#pragma unroll
					for (int k = 0; k < K; ++k)
						tot[k] += s_part[r][k];
				}
				if constexpr (!BWD)
				{
					const double sh = double(shift);
					const double ms = tot[0] * p.per_count;        // mean of x - shift
					double var = tot[1] * p.per_count - ms * ms;
					var = var < 0.0 ? 0.0 : var;
					const float fmean = float(sh + ms);
					const float finv = float(rsqrt(var + double(p.eps)));
					const float mult = gamma * finv;
					s_const[0] = mult;
					s_const[1] = fmaf(-mult, fmean, beta);
					if (rank == 0)
					{
						p.saved[ch] = fmean;
						p.saved[p.c + ch] = finv;
						if (p.sums)
						{
							p.sums[ch] = float(tot[0] + p.count * sh);
							p.sums[p.c + ch] = float(tot[1] + 2.0 * sh * tot[0] + p.count * sh * sh);
						}
					}
				}
				else
				{
					const float m0 = float(tot[0]), m1 = float(tot[1] * double(invstd)), m2 = float(tot[K - 1]);
					const float c2 = float(double(m0) * p.per_count), c3 = float(double(m1) * p.per_count);
					// dx = mult * ((du - c2) - xhat * c3) with xhat = (x - mean) * invstd, as two fused multiply-adds
					s_const[0] = bmult;
					s_const[1] = -(bmult * c3 * invstd);
					s_const[2] = -(bmult * c2);
					if (rank == 0)
					{
						p.sums[ch] = m0;
						p.sums[p.c + ch] = m1;
						p.sums[2 * p.c + ch] = m2;
						// per-channel gradients accumulate (batch_norm_layer_updater_cuda.cu:138-139, 167-182)
						if (p.grad_beta) p.grad_beta[ch] += m0;
						if (p.grad_gamma) p.grad_gamma[ch] += m1;
						if (p.grad_slope) p.grad_slope[ch] += m2;
						if (p.grad_mean) p.grad_mean[ch] += p.entry_count * (mean - p.mean[ch]);
						if (p.grad_invsigma) p.grad_invsigma[ch] += p.entry_count * (invstd - p.invsigma[ch]);
					}
				}
			}
			__syncthreads();

			const float k0 = s_const[0], k1 = s_const[1], k2 = BWD ? s_const[2] : 0.0F;
			for (uint32_t first = threadIdx.x; first < pieces; first += U * threads)
			{
				float4 a[U], du[BWD ? U : 1];
				#pragma unroll
				for (int u = 0; u < U; ++u)
					if (first + u * threads < pieces)
					{
						a[u] = tile[first + u * threads];
						if (BWD) du[BWD ? u : 0] = tile_d[first + u * threads];
					}
				#pragma unroll
				for (int u = 0; u < U; ++u)
				{
					const uint32_t i = first + u * threads;
					if (i >= pieces)
						break;
					const piece<WHOLE> f(p, start, i);
					float4 o;
					if constexpr (!BWD)
					{
						o.x = chain_forward<A0, A1>(p.chain, fmaf(a[u].x, k0, k1), slope);
						o.y = chain_forward<A0, A1>(p.chain, fmaf(a[u].y, k0, k1), slope);
						o.z = chain_forward<A0, A1>(p.chain, fmaf(a[u].z, k0, k1), slope);
						o.w = chain_forward<A0, A1>(p.chain, fmaf(a[u].w, k0, k1), slope);
					}
					else
					{
						o.x = fmaf(du[u].x, k0, fmaf(a[u].x - mean, k1, k2));
						o.y = fmaf(du[u].y, k0, fmaf(a[u].y - mean, k1, k2));
						o.z = fmaf(du[u].z, k0, fmaf(a[u].z - mean, k1, k2));
						o.w = fmaf(du[u].w, k0, fmaf(a[u].w - mean, k1, k2));
					}
					float * const out = p.out + f.at;
					if (f.whole())
						st_stream(reinterpret_cast<float4 *>(out), o);
					else
					{
						if (f.holds(0)) st_stream(out, o.x);
						if (f.holds(1)) st_stream(out + 1, o.y);
						if (f.holds(2)) st_stream(out + 2, o.z);
						if (f.holds(3)) st_stream(out + 3, o.w);
					}
				}
			}
		}

		// Most shared memory that a CTA may ask for: what all CTAs of an SM can share, and no more than a CTA may have beside the
		// kernel's static arrays (less than 1 KB).
		int cluster_smem_limit()
		{
			const int optin = running_config().max_shared_memory_per_block_optin - 1024, budget = (int)sm_smem_budget();
			return budget < optin ? budget : optin;
		}

		struct cluster_plan
		{
			int threads;
			size_t smem;
		};

		// CTAs per channel: as few as bring a CTA's slice down to 56 KB (three CTAs on an SM), more while the channels do not fill the
		// SMs. Threads: as many as the CTAs that an SM will hold leave registers for (x[32,256,14,14] forward, two CTAs per SM: 5.6 us
		// with 512 threads, 9.4 with 128; x[256,512,14,14], eight: 44 with 128, 85 with 512).
		bool plan_cluster(cluster_plan& plan, cluster_params& p, int64_t n, int64_t c, int64_t hw, bool backward, size_t slice_limit)
		{
			if (n < 1 || c < 1 || n * c * hw >= (int64_t(1) << 31) || tune().chain_cluster == 99)
				return false;
			const bool whole = hw % 4 == 0;
			const int64_t pitch = whole ? hw / 4 : (hw + 6) / 4;
			const int64_t row_bytes = pitch * 16 * (backward ? 2 : 1);
			// below that the frames of ragged planes are mostly edges (5x5 planes, x[512,512,5,5]: 24.6 / 32.3 us against 24.6 / 34.6)
			if (hw < (whole ? 16 : 25))
				return false;
			auto slice = [&](int64_t k) { return div_up(n, k) * row_bytes; };
			int64_t k = 1;
			const int64_t sms = sm_count();
			if (tune().chain_cluster > 0)
				k = tune().chain_cluster;
			else
			{
				while (k < int64_t(kClusterMax) && slice(k) > 56 * 1024)
					k *= 2;
				while (k < int64_t(kClusterMax) && c * k <= sms && slice(k) > 4 * 1024)
					k *= 2;
			}
			const int64_t bytes = slice(k), room = cluster_smem_limit();
			if (k > int64_t(kClusterMax) || bytes > room || size_t(bytes) > slice_limit)
				return false;
			p.cluster = (uint32_t)k;
			p.entries = (uint32_t)div_up(n, k);
			p.pitch = (uint32_t)pitch;
			plan.smem = (size_t)bytes;
			const int64_t resident = c * k >= sms * (room / bytes) ? room / bytes : div_up(c * k, sms);
			plan.threads = resident <= 2 ? 512 : resident <= 4 ? 256 : 128;
			p.per_stage = (uint32_t)(div_up(p.entries * pitch, kClusterStages * plan.threads) * plan.threads);
			if (p.per_stage < uint32_t(4 * plan.threads))
				p.per_stage = 4 * plan.threads;   // a small tile is one stage: nothing to overlap, and four loads at a time
			p.d_pitch = fastdiv(p.pitch);
			p.row_stride = (uint32_t)(c * hw);
			p.n = (uint32_t)n; p.c = (uint32_t)c; p.hw = (uint32_t)hw;
			p.total = (uint32_t)(n * c * hw);
			p.count = double(n) * double(hw);
			p.per_count = 1.0 / p.count;
			return true;
		}

		template <int A0, int A1, bool BWD, bool WHOLE>
		int launch_cluster(const cluster_params& p, const cluster_plan& plan, cudaStream_t s, const char * what)
		{
			auto kernel = bn_train_cluster_kernel<A0, A1, BWD, WHOLE>;
			// the attribute is the kernel's, not the launch's: the same value whatever the shape, so that host threads with different
			// shapes do not lower it under each other's launches
			const cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, cluster_smem_limit());
			if (e != cudaSuccess)
				return set_error(NNF_ERR_CUDA, "%s: cudaFuncSetAttribute: %s", what, cudaGetErrorString(e));
			cudaLaunchAttribute attr[2];
			attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
			attr[0].val.programmaticStreamSerializationAllowed = 1;
			attr[1].id = cudaLaunchAttributeClusterDimension;
			attr[1].val.clusterDim.x = p.cluster;
			attr[1].val.clusterDim.y = 1;
			attr[1].val.clusterDim.z = 1;
			cudaLaunchConfig_t cfg = {};
			cfg.gridDim = dim3(p.c * p.cluster);
			cfg.blockDim = dim3((unsigned)plan.threads);
			cfg.dynamicSmemBytes = plan.smem;
			cfg.stream = s;
			cfg.attrs = attr;
			cfg.numAttrs = 2;
			cudaLaunchKernelEx(&cfg, kernel, p);   // the error, if any, is picked up by check_launch
			return check_launch(what);
		}

		template <bool BWD, bool WHOLE>
		int dispatch_chain(const cluster_params& p, const cluster_plan& plan, cudaStream_t s, const char * what)
		{
			switch (chain_id(p.chain))
			{
			case 0: return launch_cluster<NNF_ACT_NONE, 0, BWD, WHOLE>(p, plan, s, what);
			case 1: return launch_cluster<NNF_ACT_PRELU, NNF_ACT_ELU, BWD, WHOLE>(p, plan, s, what);
			case 2: return launch_cluster<NNF_ACT_RELU, 0, BWD, WHOLE>(p, plan, s, what);
			default: return launch_cluster<-1, 0, BWD, WHOLE>(p, plan, s, what);
			}
		}
	}

	int cluster_train_fwd(cudaStream_t s, float * y, float * saved, float * sums, const float * x, const float * gamma, const float * beta, float eps,
		const act_chain& chain, int64_t n, int64_t c, int64_t hw, void * report, size_t slice_limit)
	{
		cluster_plan plan;
		cluster_params p = {};
		if (!plan_cluster(plan, p, n, c, hw, false, slice_limit))
			return -1;
		p.x = x; p.out = y; p.gamma = gamma; p.beta = beta; p.saved = saved; p.sums = sums;
		p.eps = eps;
		p.chain = chain;
		p.report = static_cast<uint32_t *>(report);
		const char * what = "bn_train_cluster_kernel (forward)";
		return hw % 4 == 0 ? dispatch_chain<false, true>(p, plan, s, what) : dispatch_chain<false, false>(p, plan, s, what);
	}

	int cluster_train_bwd(cudaStream_t s, float * dx, float * bsums, const float * dy, const float * x, const float * gamma, const float * beta, const float * saved,
		const act_chain& chain, float * grad_gamma, float * grad_beta, float * grad_mean, float * grad_invsigma, float * grad_slope,
		const float * mean, const float * invsigma, float entry_count, int64_t n, int64_t c, int64_t hw, void * report, size_t slice_limit)
	{
		cluster_plan plan;
		cluster_params p = {};
		if (!plan_cluster(plan, p, n, c, hw, true, slice_limit))
			return -1;
		p.x = x; p.dy = dy; p.out = dx; p.gamma = gamma; p.beta = beta; p.saved = const_cast<float *>(saved); p.sums = bsums;
		p.grad_gamma = grad_gamma; p.grad_beta = grad_beta; p.grad_mean = grad_mean; p.grad_invsigma = grad_invsigma; p.grad_slope = grad_slope;
		p.mean = mean; p.invsigma = invsigma; p.entry_count = entry_count;
		p.chain = chain;
		p.report = static_cast<uint32_t *>(report);
		const char * what = "bn_train_cluster_kernel (backward)";
		return hw % 4 == 0 ? dispatch_chain<true, true>(p, plan, s, what) : dispatch_chain<true, false>(p, plan, s, what);
	}
}
