/* The differentiable form: a recurrent network of discrete leaky
 * integrate-and-fire neurons (1 ms Euler step, reset by subtraction) run
 * forward with exact spikes for up to 32 trials at once (one lane per trial),
 * and its backpropagation-through-time adjoint, with a fast-sigmoid surrogate
 * for the derivative of the threshold only. C ABI in include/nemo_b200.h
 * (nemo_b200_lif_*).
 *
 * Model, for neuron i, trial b, step t (v[-1] = 0):
 *   I[t] = sum over in-synapses k of i: w[k] * x_k[t]
 *          x_k[t] = s_j[t-1] for a recurrent synapse from neuron j (0 at t = 0),
 *                   the input channel's spike at t for an input synapse;
 *   u[t] = beta * v[t-1] + I[t];   s[t] = H(u[t] - theta);   v[t] = u[t] - theta * s[t].
 * The output is counts[b][bin] = sum over neurons and the bin's steps of s.
 *
 * Adjoint (backward through time), with s'(u) = 1 / (1 + kappa |u - theta|)^2
 * standing in for the derivative of H:
 *   gs[t]_j = dL/dcounts[b][bin(t)] + sum over recurrent out-synapses (j -> i, w):
 *             w * gu[t+1]_i
 *   gv[t]   = beta * gu[t+1]
 *   gu[t]   = s'(u[t]) * (gs[t] - theta * gv[t]) + gv[t]
 *   dL/dw[k] = sum over t, b of gu[t]_i * x_k[t]
 * The relaxed variant replaces the spike by s = r(u - theta) with
 * r(x) = x / (1 + kappa |x|), whose derivative is the surrogate exactly, so
 * that the adjoint is the true gradient of the relaxed forward (checked
 * against finite differences).
 *
 * Memory: the forward stores every step's spikes (a 32-bit word per neuron:
 * bit b = trial b) and v at every checkpoint (every K steps); the backward
 * recomputes u inside each K-step segment from its checkpoint (the same
 * operations in the same order, so u is bit-identical), then walks the
 * segment backwards. Sums run in a fixed order, so results are reproducible;
 * the weight gradient sums steps segment by segment, so its rounding (not u's)
 * depends on the checkpoint interval. */

#include <cuda_runtime.h>

#include <algorithm>
#include <cstdint>
#include <cstring>
#include <string>

#include <nemo_b200.h>

#include "common.hpp"

namespace nemo_b200 {
namespace lif {
namespace {

const unsigned FULL = 0xffffffffu;
const unsigned THREADS = 256;

struct Net {
	int N, C, B, T, K, binSteps;
	float beta, theta, kappa;
	const int* rowptr;   /* [N + 1] in-synapses of each neuron */
	const int* pre;      /* [nnz] < N: recurrent source; >= N: input channel pre - N */
	const int* colptr;   /* [N + 1] recurrent out-synapses of each neuron */
	const int* post;     /* [nnzRec] target */
	const int* wpos;     /* [nnzRec] index of the synapse in w / pre */
	int nnzRec;          /* colptr[N] */
};

/* spike of presynaptic unit p for the lane's trial at step t */
template<bool RELAXED>
__device__ __forceinline__ float presyn(const Net& n, int p, int t, uint32_t lane, const uint32_t* sBits,
		const float* sF, const uint32_t* inBits)
{
	if(p >= n.N) {
		return float((inBits[size_t(t) * n.C + (p - n.N)] >> lane) & 1u);
	}
	if(t == 0) return 0.0f;
	if(RELAXED) {
		return sF[(size_t(t - 1) * n.N + p) * 32 + lane];
	}
	return float((sBits[size_t(t - 1) * n.N + p] >> lane) & 1u);
}

/* the spike word (bit b = trial b) of presynaptic unit p at step t */
__device__ __forceinline__ uint32_t presynWord(const Net& n, int p, int t, const uint32_t* sBits,
		const uint32_t* inBits)
{
	if(p >= n.N) return inBits[size_t(t) * n.C + (p - n.N)];
	return t == 0 ? 0u : sBits[size_t(t - 1) * n.N + p];
}

/* One forward step for every neuron (warp per neuron, lane per trial).
 * v: [N][32] state, read and written. RECOMPUTE: store u into uOut (a
 * segment buffer [K][N][32]) instead of the spikes and counts. */
template<bool RELAXED, bool RECOMPUTE>
__global__ void __launch_bounds__(THREADS)
k_step(Net n, int t, const float* w, const uint32_t* inBits, uint32_t* sBits, float* sF, float* v,
		float* vCkpt, float* counts, float* uOut, int segStart)
{
	__shared__ float sCount[32];
	const uint32_t lane = threadIdx.x & 31u;
	const bool active = lane < uint32_t(n.B);
	if(!RECOMPUTE) {
		if(threadIdx.x < 32) sCount[threadIdx.x] = 0.0f;
		__syncthreads();
	}
	const int warps = int((gridDim.x * blockDim.x) >> 5);
	for(int i = int((blockIdx.x * blockDim.x + threadIdx.x) >> 5); i < n.N; i += warps) {
		const size_t cell = size_t(i) * 32 + lane;
		const float vPrev = v[cell];
		if(!RECOMPUTE && t % n.K == 0) {
			vCkpt[size_t(t / n.K) * n.N * 32 + cell] = vPrev;
		}
		/* in-synapses in order, 32 at a time: lane L loads synapse base + L
		 * (and, for spikes as bits, the presynaptic word of all trials), then
		 * every lane takes them in turn; a word without spikes adds nothing */
		float I = 0.0f;
		const int k0 = n.rowptr[i], k1 = n.rowptr[i + 1];
		for(int base = k0; base < k1; base += 32) {
			const int k = base + int(lane);
			const int p = k < k1 ? n.pre[k] : 0;
			const float wk = k < k1 ? w[k] : 0.0f;
			const int cnt = min(32, k1 - base);
			if(RELAXED) {
				for(int q = 0; q < cnt; ++q) {
					const int pq = __shfl_sync(FULL, p, q);
					const float wq = __shfl_sync(FULL, wk, q);
					I = __fadd_rn(I, __fmul_rn(wq, presyn<RELAXED>(n, pq, t, lane, sBits, sF, inBits)));
				}
			} else {
				const uint32_t word = k < k1 ? presynWord(n, p, t, sBits, inBits) : 0u;
				uint32_t nz = __ballot_sync(FULL, word != 0u);
				while(nz) {
					const int q = __ffs(int(nz)) - 1;
					nz &= nz - 1u;
					const uint32_t wd = __shfl_sync(FULL, word, q);
					const float wq = __shfl_sync(FULL, wk, q);
					if((wd >> lane) & 1u) I = __fadd_rn(I, wq);
				}
			}
		}
		const float u = __fadd_rn(__fmul_rn(n.beta, vPrev), I);
		const float x = __fsub_rn(u, n.theta);
		float s;
		if(RELAXED) {
			s = __fdiv_rn(x, __fadd_rn(1.0f, __fmul_rn(n.kappa, fabsf(x))));
		} else {
			s = (active && u >= n.theta) ? 1.0f : 0.0f;
		}
		v[cell] = __fsub_rn(u, __fmul_rn(n.theta, s));
		if(RECOMPUTE) {
			uOut[(size_t(t - segStart) * n.N) * 32 + cell] = u;
		} else {
			if(RELAXED) {
				sF[(size_t(t) * n.N + i) * 32 + lane] = active ? s : 0.0f;
			} else {
				const uint32_t word = __ballot_sync(FULL, s != 0.0f);
				if(lane == 0) sBits[size_t(t) * n.N + i] = word;
			}
			if(active && s != 0.0f) atomicAdd(&sCount[lane], s);
		}
	}
	if(!RECOMPUTE) {
		__syncthreads();
		if(threadIdx.x < uint32_t(n.B)) {
			const float c = sCount[threadIdx.x];
			if(c != 0.0f) atomicAdd(&counts[size_t(threadIdx.x) * (n.T / n.binSteps) + t / n.binSteps], c);
		}
	}
}

/* wOut[e] = w[n.wpos[e]]: the recurrent weights in out-synapse order */
__global__ void
k_gather_out(Net n, int nnzRec, const float* w, float* wOut)
{
	for(int e = int(blockIdx.x * blockDim.x + threadIdx.x); e < nnzRec; e += int(gridDim.x * blockDim.x)) {
		wOut[e] = w[n.wpos[e]];
	}
}

/* One backward step: gu[t] of every neuron j from gu[t+1] (guNext, [N][32])
 * and u[t] (uSeg). Warp per neuron (source view), lane per trial; wOut: the
 * recurrent weights in out-synapse order. A chunk's 32 rows of guNext are
 * all loaded before they are summed (in synapse order), so that a warp keeps
 * 32 loads in flight. */
__global__ void __launch_bounds__(THREADS)
k_back(Net n, int t, const float* wOut, const float* uSeg, int segStart, const float* guNext, float* guOut,
		const float* dcounts, bool last)
{
	const uint32_t lane = threadIdx.x & 31u;
	const bool active = lane < uint32_t(n.B);
	const int warps = int((gridDim.x * blockDim.x) >> 5);
	const int bins = n.T / n.binSteps;
	for(int j = int((blockIdx.x * blockDim.x + threadIdx.x) >> 5); j < n.N; j += warps) {
		const size_t cell = size_t(j) * 32 + lane;
		float gs = active ? dcounts[size_t(lane) * bins + t / n.binSteps] : 0.0f;
		float gv = 0.0f;
		if(!last) {
			const int e0 = n.colptr[j], e1 = n.colptr[j + 1];
			for(int base = e0; base < e1; base += 32) {
				const int e = base + int(lane);
				const int i = e < e1 ? n.post[e] : 0;
				const float we = e < e1 ? wOut[e] : 0.0f;
				const int cnt = min(32, e1 - base);
				float g[32];
#pragma unroll
				for(int q = 0; q < 32; ++q) {
					const int iq = __shfl_sync(FULL, i, q);
					g[q] = q < cnt ? guNext[size_t(iq) * 32 + lane] : 0.0f;
				}
#pragma unroll
				for(int q = 0; q < 32; ++q) {
					const float wq = __shfl_sync(FULL, we, q);
					if(q < cnt) gs = __fadd_rn(gs, __fmul_rn(wq, g[q]));
				}
			}
			gv = __fmul_rn(n.beta, guNext[cell]);
		}
		const float u = uSeg[(size_t(t - segStart) * n.N) * 32 + cell];
		const float a = __fadd_rn(1.0f, __fmul_rn(n.kappa, fabsf(__fsub_rn(u, n.theta))));
		const float sp = __fdiv_rn(1.0f, __fmul_rn(a, a));
		const float gu = __fadd_rn(__fmul_rn(sp, __fsub_rn(gs, __fmul_rn(n.theta, gv))), gv);
		guOut[(size_t(t - segStart) * n.N) * 32 + cell] = active ? gu : 0.0f;
	}
}

/* dL/dw over one segment of the relaxed model: for every in-synapse k of
 * neuron i, the sum over the segment's steps and the trials of gu[t]_i *
 * x_k[t]; warp per neuron, lanes summing their trial over the steps, one
 * reduction per synapse. */
__global__ void __launch_bounds__(THREADS)
k_dw_relaxed(Net n, int segStart, int segEnd, const float* guSeg, const float* sF, const uint32_t* inBits, float* dw)
{
	const uint32_t lane = threadIdx.x & 31u;
	const int warps = int((gridDim.x * blockDim.x) >> 5);
	for(int i = int((blockIdx.x * blockDim.x + threadIdx.x) >> 5); i < n.N; i += warps) {
		const int k0 = n.rowptr[i], k1 = n.rowptr[i + 1];
		for(int k = k0; k < k1; ++k) {
			const int p = n.pre[k];
			float acc = 0.0f;
			for(int t = segStart; t < segEnd; ++t) {
				const float g = guSeg[(size_t(t - segStart) * n.N + i) * 32 + lane];
				acc = __fadd_rn(acc, __fmul_rn(g, presyn<true>(n, p, t, lane, nullptr, sF, inBits)));
			}
#pragma unroll
			for(int d = 16; d; d >>= 1) acc = __fadd_rn(acc, __shfl_xor_sync(FULL, acc, d));
			if(lane == 0) dw[k] = __fadd_rn(dw[k], acc);
		}
	}
}

/* ---- event lists (spikes as bits) ----
 *
 * The recompute and the weight gradient of a segment both go over every
 * synapse and every (step, trial) in which its presynaptic unit spikes. The
 * spikes are known, so each unit's (step, trial) pairs of the segment are
 * listed once (k_events) and every synapse walks its unit's list: the work is
 * the number of spikes times the fan-out, where walking words tests every
 * (step, synapse) word and shuffles every one that is not 0 (a gradient step
 * of 10,000 neurons, 2.5e6 synapses, 500 steps and 32 trials on a B200: 62.4 ms
 * with a launch per recomputed step, 48.5 with the lists). A segment is
 * taken in parts of at most PART_STEPS steps, the most for which a neuron's
 * currents of all steps and trials stay in shared memory (8 KB a warp) and a
 * code step * 32 + trial fits 16 bits. */

const int PART_STEPS = 64;
const int PART_WARPS = 8;

/* parts of a segment of `steps` steps and the steps of each (the last one
 * may have fewer) */
static int parts(int steps) { return (steps + PART_STEPS - 1) / PART_STEPS; }
static int partSteps(int steps) { return (steps + parts(steps) - 1) / parts(steps); }

/* The event lists of the steps [c0, c1): for part y (steps from c0 + y L) and
 * presynaptic unit p (neurons, then input channels) the codes (t - part
 * start) * 32 + b of the spikes it delivers, by step, then by trial, in
 * codes[(y * units + p) * L * 32 ...], their number in cnt[y * units + p]. A
 * list is filled up to a multiple of 8 codes with the code L * 32 (a cell
 * that holds 0). A block takes 32 units of one part: their words are read
 * coalesced over the units and turned in shared memory, a warp then has a
 * unit's steps in its lanes. */
__global__ void __launch_bounds__(THREADS)
k_events(Net n, int c0, int c1, int L, const uint32_t* sBits, const uint32_t* inBits, uint16_t* codes, uint32_t* cnt)
{
	__shared__ uint32_t tile[PART_STEPS][33];
	const uint32_t lane = threadIdx.x & 31u;
	const int warp = int(threadIdx.x >> 5);
	const int units = n.N + n.C;
	const int unit0 = int(blockIdx.x) * 32;
	const int t0 = c0 + int(blockIdx.y) * L;
	const int len = min(L, c1 - t0);
	const uint32_t trials = n.B == 32 ? FULL : (1u << n.B) - 1u;
	for(int r = warp; r < len; r += int(THREADS / 32)) {
		const int p = unit0 + int(lane);
		tile[r][lane] = p < units ? presynWord(n, p, t0 + r, sBits, inBits) & trials : 0u;
	}
	__syncthreads();
	for(int q = warp; q < 32; q += int(THREADS / 32)) {
		const int p = unit0 + q;
		if(p >= units) break;
		uint16_t* out = codes + (size_t(blockIdx.y) * units + p) * (size_t(L) * 32);
		uint32_t total = 0;
		for(int r0 = 0; r0 < len; r0 += 32) {
			const int r = r0 + int(lane);
			uint32_t word = r < len ? tile[r][q] : 0u;
			const uint32_t c = uint32_t(__popc(word));
			uint32_t incl = c;
#pragma unroll
			for(int d = 1; d < 32; d <<= 1) {
				const uint32_t x = __shfl_up_sync(FULL, incl, d);
				if(lane >= uint32_t(d)) incl += x;
			}
			uint32_t at = total + incl - c;
			while(word) {
				out[at++] = uint16_t(r * 32 + __ffs(int(word)) - 1);
				word &= word - 1u;
			}
			total += __shfl_sync(FULL, incl, 31);
		}
		const uint32_t fill = (8u - (total & 7u)) & 7u;
		if(lane < fill) out[total + lane] = uint16_t(L * 32);
		if(lane == 0) cnt[size_t(blockIdx.y) * units + p] = total;
	}
}

/* The steps [t0, t1) (one part) from v before them (vIn): u of every step
 * into uOut (segment buffer [K][N][32]), v after them into vOut. Warp per
 * neuron: its currents of all steps and trials are accumulated in shared
 * memory, synapse after synapse in order, a synapse's events over the lanes
 * (distinct cells); a cell so gets its weights in synapse order, as in the
 * forward, and u is bit-identical. The codes of the next synapses are loaded
 * while the last ones are added. */
__global__ void __launch_bounds__(PART_WARPS * 32)
k_recompute(Net n, int t0, int t1, int segStart, int L, const float* w, const uint16_t* codes, const uint32_t* cnt,
		const float* vIn, float* vOut, float* uOut)
{
	extern __shared__ float sCur[];
	const int U = 4;
	const uint32_t lane = threadIdx.x & 31u;
	const bool active = lane < uint32_t(n.B);
	float* cur = sCur + size_t(threadIdx.x >> 5) * (size_t(L) * 32);
	const size_t cap = size_t(L) * 32;
	const int len = t1 - t0;
	const int warps = int((gridDim.x * blockDim.x) >> 5);
	for(int i = int((blockIdx.x * blockDim.x + threadIdx.x) >> 5); i < n.N; i += warps) {
		for(int r = 0; r < len; ++r) cur[r * 32 + int(lane)] = 0.0f;
		__syncwarp();
		const int k0 = n.rowptr[i], k1 = n.rowptr[i + 1];
		for(int base = k0; base < k1; base += 32) {
			const int k = base + int(lane);
			const int p = k < k1 ? n.pre[k] : 0;
			const float wk = k < k1 ? w[k] : 0.0f;
			const uint32_t ck = k < k1 ? cnt[p] : 0u;
			const int nk = min(32, k1 - base);
			uint32_t next[U];
#pragma unroll
			for(int x = 0; x < U; ++x) {
				const uint32_t c = __shfl_sync(FULL, ck, x);
				const int pq = __shfl_sync(FULL, p, x);
				next[x] = lane < c ? codes[size_t(pq) * cap + lane] : 0u;
			}
			for(int q0 = 0; q0 < nk; q0 += U) {
				uint32_t code[U];
#pragma unroll
				for(int x = 0; x < U; ++x) {
					code[x] = next[x];
					const int q = (q0 + U + x) & 31;
					const uint32_t c = q0 + U + x < nk ? __shfl_sync(FULL, ck, q) : 0u;
					const int pq = __shfl_sync(FULL, p, q);
					next[x] = lane < c ? codes[size_t(pq) * cap + lane] : 0u;
				}
#pragma unroll
				for(int x = 0; x < U; ++x) {
					/* past the last synapse: a count of 0 */
					const int q = q0 + x;
					const uint32_t c = __shfl_sync(FULL, ck, q);
					const float wq = __shfl_sync(FULL, wk, q);
					if(lane < c) cur[code[x]] = __fadd_rn(cur[code[x]], wq);
					if(c > 32u) {
						const uint16_t* more = codes + size_t(__shfl_sync(FULL, p, q)) * cap;
						for(uint32_t e = 32u + lane; e < c; e += 32u) cur[more[e]] = __fadd_rn(cur[more[e]], wq);
					}
					__syncwarp();
				}
			}
		}
		const size_t cell = size_t(i) * 32 + lane;
		float v = vIn[cell];
		for(int r = 0; r < len; ++r) {
			const float u = __fadd_rn(__fmul_rn(n.beta, v), cur[r * 32 + int(lane)]);
			const float s = (active && u >= n.theta) ? 1.0f : 0.0f;
			v = __fsub_rn(u, __fmul_rn(n.theta, s));
			uOut[(size_t(t0 - segStart + r) * n.N) * 32 + cell] = u;
		}
		vOut[cell] = v;
		__syncwarp();
	}
}

/* dL/dw of the steps [t0, t1) (one part): warp per neuron, its gu of the
 * part's steps in shared memory, lanes over its in-synapses; each lane sums
 * gu over its presynaptic unit's events, by step, then by trial, eight codes
 * a load. */
__global__ void __launch_bounds__(PART_WARPS * 32)
k_dw_events(Net n, int t0, int t1, int segStart, int L, const float* guSeg, const uint16_t* codes, const uint32_t* cnt,
		float* dw)
{
	extern __shared__ float sGu[];
	const uint32_t lane = threadIdx.x & 31u;
	const size_t cap = size_t(L) * 32;
	float* g = sGu + size_t(threadIdx.x >> 5) * (cap + 32);
	const int len = t1 - t0;
	const int warps = int((gridDim.x * blockDim.x) >> 5);
	g[cap + lane] = 0.0f;
	for(int i = int((blockIdx.x * blockDim.x + threadIdx.x) >> 5); i < n.N; i += warps) {
		for(int r = 0; r < len; ++r) {
			g[r * 32 + int(lane)] = guSeg[(size_t(t0 - segStart + r) * n.N + i) * 32 + lane];
		}
		__syncwarp();
		const int k0 = n.rowptr[i], k1 = n.rowptr[i + 1];
		for(int k = k0 + int(lane); k < k1; k += 32) {
			const int p = n.pre[k];
			const uint32_t c = cnt[p];
			const uint4* list = reinterpret_cast<const uint4*>(codes + size_t(p) * cap);
			float acc = 0.0f;
			uint4 next = c ? list[0] : make_uint4(0u, 0u, 0u, 0u);
			for(uint32_t e = 0; e < c; e += 8u) {
				const uint4 x = next;
				if(e + 8u < c) next = list[(e >> 3) + 1u];
				acc = __fadd_rn(acc, g[x.x & 0xffffu]);
				acc = __fadd_rn(acc, g[x.x >> 16]);
				acc = __fadd_rn(acc, g[x.y & 0xffffu]);
				acc = __fadd_rn(acc, g[x.y >> 16]);
				acc = __fadd_rn(acc, g[x.z & 0xffffu]);
				acc = __fadd_rn(acc, g[x.z >> 16]);
				acc = __fadd_rn(acc, g[x.w & 0xffffu]);
				acc = __fadd_rn(acc, g[x.w >> 16]);
			}
			dw[k] = __fadd_rn(dw[k], acc);
		}
		__syncwarp();
	}
}

static int
grid(int N)
{
	int dev = 0, sms = 148;
	cudaGetDevice(&dev);
	cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
	const long warps = long(N);
	long blocks = (warps * 32 + THREADS - 1) / THREADS;
	const long cap = long(sms) * 8;
	return int(blocks < cap ? blocks : cap);
}

static void
validate(const Net& n)
{
	if(n.N <= 0 || n.T <= 0 || n.K <= 0 || n.binSteps <= 0 || n.C < 0) {
		fail(NEMO_INVALID_INPUT, "lif: sizes must be positive");
	}
	if(n.B < 1 || n.B > 32) {
		fail(NEMO_INVALID_INPUT, "lif: 1 to 32 trials per call (one lane each)");
	}
	if(n.T % n.binSteps != 0) {
		fail(NEMO_INVALID_INPUT, "lif: the steps must be a whole number of bins");
	}
	if(n.nnzRec < 0) {
		fail(NEMO_INVALID_INPUT, "lif: negative recurrent synapse count");
	}
}

} // namespace
} // namespace lif
} // namespace nemo_b200

using namespace nemo_b200;

/* The work buffer: v state [N][32], gu of the step after the segment [N][32],
 * the segment's u and gu [K][N][32], the event lists of its parts (codes, then
 * counts), then the recurrent weights in out-synapse order [nnzRec]. Made
 * from the buffer's start rounded up to 128 bytes (the size has the slack). */
struct LifWork {
	float *v, *guNext, *uSeg, *guSeg;
	uint16_t* codes;
	uint32_t* cnt;
	float* wOut;
	size_t bytes;

	LifWork(const lif::Net& n, float* base)
	{
		const size_t align = 128;
		char* p = reinterpret_cast<char*>((reinterpret_cast<size_t>(base) + align - 1) / align * align);
		char* const p0 = p;
		auto take = [&](size_t bytes) { char* q = p; p += (bytes + align - 1) / align * align; return q; };
		const int K = std::min(n.K, n.T);
		const size_t NS = size_t(n.N) * 32, units = size_t(n.N) + size_t(n.C);
		v = reinterpret_cast<float*>(take(NS * 4));
		guNext = reinterpret_cast<float*>(take(NS * 4));
		uSeg = reinterpret_cast<float*>(take(size_t(K) * NS * 4));
		guSeg = reinterpret_cast<float*>(take(size_t(K) * NS * 4));
		const size_t Y = size_t(lif::parts(K));
		codes = reinterpret_cast<uint16_t*>(take(Y * units * size_t(lif::partSteps(K)) * 32 * 2));
		cnt = reinterpret_cast<uint32_t*>(take(Y * units * 4));
		wOut = reinterpret_cast<float*>(take(size_t(n.nnzRec) * 4));
		bytes = size_t(p - p0) + align;
	}
};

static std::string g_lifError;

#define LIF_CALL(...) \
	try { __VA_ARGS__; return NEMO_OK; } \
	catch(Exception& e) { g_lifError = e.what(); return e.code(); } \
	catch(std::exception& e) { g_lifError = e.what(); return NEMO_UNKNOWN_ERROR; }

extern "C" {

const char* nemo_b200_lif_error(void) { return g_lifError.c_str(); }

size_t
nemo_b200_lif_work_bytes(const nemo_b200_lif_net* net)
{
	lif::Net n;
	static_assert(sizeof(nemo_b200_lif_net) == sizeof(lif::Net), "layout");
	memcpy(&n, net, sizeof(n));
	/* sizes that the calls refuse (validate) need no buffer */
	return n.N > 0 && n.T > 0 && n.K > 0 && n.C >= 0 && n.nnzRec >= 0 ? LifWork(n, nullptr).bytes : 0;
}

int
nemo_b200_lif_forward(const nemo_b200_lif_net* net, const float* w, const uint32_t* in_bits, int relaxed,
		uint32_t* s_bits, float* s_float, float* v_ckpt, float* counts, float* work, void* stream)
{
	LIF_CALL({
		lif::Net n;
		memcpy(&n, net, sizeof(n));
		lif::validate(n);
		cudaStream_t st = static_cast<cudaStream_t>(stream);
		float* v = LifWork(n, work).v;
		NEMO_CUDA(cudaMemsetAsync(v, 0, size_t(n.N) * 32 * 4, st));
		NEMO_CUDA(cudaMemsetAsync(counts, 0, size_t(n.B) * (n.T / n.binSteps) * 4, st));
		const int g = lif::grid(n.N);
		for(int t = 0; t < n.T; ++t) {
			if(relaxed) {
				lif::k_step<true, false><<<g, lif::THREADS, 0, st>>>(n, t, w, in_bits, s_bits, s_float, v, v_ckpt,
						counts, nullptr, 0);
			} else {
				lif::k_step<false, false><<<g, lif::THREADS, 0, st>>>(n, t, w, in_bits, s_bits, s_float, v, v_ckpt,
						counts, nullptr, 0);
			}
		}
		NEMO_CUDA(cudaGetLastError());
	})
}

int
nemo_b200_lif_backward(const nemo_b200_lif_net* net, const float* w, const uint32_t* in_bits, int relaxed,
		const uint32_t* s_bits, const float* s_float, const float* v_ckpt, const float* dcounts, float* dw,
		float* work, void* stream)
{
	LIF_CALL({
		lif::Net n;
		memcpy(&n, net, sizeof(n));
		lif::validate(n);
		cudaStream_t st = static_cast<cudaStream_t>(stream);
		const size_t NS = size_t(n.N) * 32;
		const LifWork k(n, work);
		const int g = lif::grid(n.N);
		/* the recurrent weights in out-synapse order, for k_back */
		if(n.nnzRec) lif::k_gather_out<<<g, lif::THREADS, 0, st>>>(n, n.nnzRec, w, k.wOut);
		const int segments = (n.T + n.K - 1) / n.K;
		const size_t units = size_t(n.N) + size_t(n.C);
		const int L = lif::partSteps(std::min(n.K, n.T));
		const unsigned gp = unsigned((n.N + lif::PART_WARPS - 1) / lif::PART_WARPS);
		const size_t smemU = size_t(lif::PART_WARPS) * L * 32 * 4, smemW = smemU + lif::PART_WARPS * 32 * 4;
		if(!relaxed) {
			NEMO_CUDA(cudaFuncSetAttribute(lif::k_recompute, cudaFuncAttributeMaxDynamicSharedMemorySize, int(smemU)));
			NEMO_CUDA(cudaFuncSetAttribute(lif::k_dw_events, cudaFuncAttributeMaxDynamicSharedMemorySize, int(smemW)));
		}
		for(int sgi = segments - 1; sgi >= 0; --sgi) {
			const int c0 = sgi * n.K, c1 = int(std::min<long>(n.T, long(c0) + n.K));
			const float* ckpt = v_ckpt + size_t(sgi) * NS;
			const int Y = (c1 - c0 + L - 1) / L;
			/* recompute u over the segment from its checkpoint */
			if(relaxed) {
				NEMO_CUDA(cudaMemcpyAsync(k.v, ckpt, NS * 4, cudaMemcpyDeviceToDevice, st));
				for(int t = c0; t < c1; ++t) {
					lif::k_step<true, true><<<g, lif::THREADS, 0, st>>>(n, t, w, in_bits, nullptr,
							const_cast<float*>(s_float), k.v, nullptr, nullptr, k.uSeg, c0);
				}
			} else {
				lif::k_events<<<dim3(unsigned((units + 31) / 32), unsigned(Y)), lif::THREADS, 0, st>>>(n, c0, c1, L, s_bits,
						in_bits, k.codes, k.cnt);
				for(int y = 0; y < Y; ++y) {
					const int t0 = c0 + y * L, t1 = std::min(c1, t0 + L);
					lif::k_recompute<<<gp, lif::PART_WARPS * 32, smemU, st>>>(n, t0, t1, c0, L, w,
							k.codes + size_t(y) * units * L * 32, k.cnt + size_t(y) * units, y ? k.v : ckpt, k.v, k.uSeg);
				}
			}
			/* backwards through the segment */
			for(int t = c1 - 1; t >= c0; --t) {
				const bool last = t == n.T - 1;
				const float* next = t == c1 - 1 ? k.guNext : k.guSeg + size_t(t + 1 - c0) * NS;
				lif::k_back<<<g, lif::THREADS, 0, st>>>(n, t, k.wOut, k.uSeg, c0, next, k.guSeg, dcounts, last);
			}
			if(relaxed) {
				lif::k_dw_relaxed<<<g, lif::THREADS, 0, st>>>(n, c0, c1, k.guSeg, s_float, in_bits, dw);
			} else {
				for(int y = 0; y < Y; ++y) {
					const int t0 = c0 + y * L, t1 = std::min(c1, t0 + L);
					lif::k_dw_events<<<gp, lif::PART_WARPS * 32, smemW, st>>>(n, t0, t1, c0, L, k.guSeg,
							k.codes + size_t(y) * units * L * 32, k.cnt + size_t(y) * units, dw);
				}
			}
			NEMO_CUDA(cudaMemcpyAsync(k.guNext, k.guSeg, NS * 4, cudaMemcpyDeviceToDevice, st));
		}
		NEMO_CUDA(cudaGetLastError());
	})
}

} // extern "C"
