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
#include <map>
#include <memory>
#include <mutex>
#include <string>

#include <nemo_b200.h>

#include "common.hpp"
#include "device_turn.hpp"

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

/* gu[t] of a neuron and trial from its u[t], gs[t] and gv[t] */
__device__ __forceinline__ float guOf(const Net& n, float u, float gs, float gv)
{
	const float a = __fadd_rn(1.0f, __fmul_rn(n.kappa, fabsf(__fsub_rn(u, n.theta))));
	const float sp = __fdiv_rn(1.0f, __fmul_rn(a, a));
	return __fadd_rn(__fmul_rn(sp, __fsub_rn(gs, __fmul_rn(n.theta, gv))), gv);
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
		const float gu = guOf(n, uSeg[(size_t(t - segStart) * n.N) * 32 + cell], gs, gv);
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
 * (step, synapse) word and shuffles every one that is not 0. A segment is
 * taken in parts of at most PART_STEPS steps, the most for which a neuron's
 * currents of all steps and trials stay in shared memory (8 KB a warp) and a
 * code step * 32 + trial fits 16 bits. */

const int PART_STEPS = 64;
const int PART_WARPS = 8;
/* shared memory of a block at PART_STEPS steps (a step's row and a cell a
 * lane), the most a call uses */
const size_t PART_SMEM = size_t(PART_WARPS) * (PART_STEPS * 32 + 32) * 4;

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
 * into uOut (segment buffer [K][N][tw]), v after them into vOut. Warp per
 * neuron: its currents of all steps and trials are accumulated in shared
 * memory, synapse after synapse in order, a synapse's events over the lanes,
 * two a lane (distinct cells); a cell so gets its weights in synapse order, as in the
 * forward, and u is bit-identical. The codes of the next synapses are loaded
 * while the last ones are added. */
__global__ void __launch_bounds__(PART_WARPS * 32)
k_recompute(Net n, int tw, int t0, int t1, int segStart, int L, const float* w, const uint16_t* codes,
		const uint32_t* cnt, const float* vIn, float* vOut, float* uOut)
{
	extern __shared__ float sCur[];
	const int U = 4;
	const uint32_t lane = threadIdx.x & 31u;
	const bool active = lane < uint32_t(n.B);
	const size_t cap = size_t(L) * 32;
	float* cur = sCur + size_t(threadIdx.x >> 5) * (cap + 32);
	const int len = t1 - t0;
	const int warps = int((gridDim.x * blockDim.x) >> 5);
	for(int i = int((blockIdx.x * blockDim.x + threadIdx.x) >> 5); i < n.N; i += warps) {
		for(int r = 0; r < len; ++r) cur[r * 32 + int(lane)] = 0.0f;
		__syncwarp();
		const int k0 = n.rowptr[i], k1 = n.rowptr[i + 1];
		/* the synapses of a group of 32, and those of the next one on their way:
		 * unit and weight during the first half, the unit's count during the
		 * second (past the end: a count of 0) */
		int p = k0 + int(lane) < k1 ? n.pre[k0 + int(lane)] : 0;
		float wk = k0 + int(lane) < k1 ? w[k0 + int(lane)] : 0.0f;
		uint32_t ck = k0 + int(lane) < k1 ? cnt[p] : 0u;
		for(int base = k0; base < k1; base += 32) {
			const int k = base + 32 + int(lane);
			int pNext = 0;
			float wNext = 0.0f;
			uint32_t cNext = 0;
			if(k < k1) {
				pNext = n.pre[k];
				wNext = w[k];
			}
			uint32_t next[U];
#pragma unroll
			for(int x = 0; x < U; ++x) {
				const uint32_t c = __shfl_sync(FULL, ck, x);
				const int pq = __shfl_sync(FULL, p, x);
				next[x] = 2u * lane < c ? *reinterpret_cast<const uint32_t*>(codes + size_t(pq) * cap + 2u * lane) : 0u;
			}
#pragma unroll 1
			for(int q0 = 0; q0 < 32; q0 += U) {
				if(q0 == 16 && k < k1) cNext = cnt[pNext];
				uint32_t code[U];
#pragma unroll
				for(int x = 0; x < U; ++x) {
					code[x] = next[x];
					const int q = (q0 + U + x) & 31;
					const uint32_t c = q0 + U < 32 ? __shfl_sync(FULL, ck, q) : 0u;
					const int pq = __shfl_sync(FULL, p, q);
					next[x] = 2u * lane < c ? *reinterpret_cast<const uint32_t*>(codes + size_t(pq) * cap + 2u * lane) : 0u;
				}
#pragma unroll
				for(int x = 0; x < U; ++x) {
					const int q = q0 + x;
					const uint32_t c = __shfl_sync(FULL, ck, q);
					const float wq = __shfl_sync(FULL, wk, q);
					/* distinct cells: both loads, then both stores; past the end
					 * of the list the cell that is never read */
					float* a = cur + (2u * lane < c ? code[x] & 0xffffu : uint32_t(cap));
					float* b = cur + (2u * lane + 1u < c ? code[x] >> 16 : uint32_t(cap));
					const float va = *a, vb = *b;
					*a = __fadd_rn(va, wq);
					*b = __fadd_rn(vb, wq);
					if(c > 64u) {
						const uint16_t* more = codes + size_t(__shfl_sync(FULL, p, q)) * cap;
						for(uint32_t e = 64u + lane; e < c; e += 32u) cur[more[e]] = __fadd_rn(cur[more[e]], wq);
					}
					__syncwarp();
				}
			}
			p = pNext;
			wk = wNext;
			ck = cNext;
		}
		const size_t cell = size_t(i) * 32 + lane;
		float v = vIn[cell];
		for(int r = 0; r < len; ++r) {
			const float u = __fadd_rn(__fmul_rn(n.beta, v), cur[r * 32 + int(lane)]);
			const float s = (active && u >= n.theta) ? 1.0f : 0.0f;
			v = __fsub_rn(u, __fmul_rn(n.theta, s));
			if(int(lane) < tw) uOut[(size_t(t0 - segStart + r) * n.N + i) * tw + lane] = u;
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
k_dw_events(Net n, int tw, int t0, int t1, int segStart, int L, const float* guSeg, const uint16_t* codes,
		const uint32_t* cnt, const unsigned* error, float* dw)
{
	extern __shared__ float sGu[];
	const uint32_t lane = threadIdx.x & 31u;
	const size_t cap = size_t(L) * 32;
	float* g = sGu + size_t(threadIdx.x >> 5) * (cap + 32);
	const int len = t1 - t0;
	const int warps = int((gridDim.x * blockDim.x) >> 5);
	/* a barrier of the adjoint gave up: the result is NaN */
	const float zero = *error ? __int_as_float(0x7fffffff) : 0.0f;
	g[cap + lane] = 0.0f;
	for(int i = int((blockIdx.x * blockDim.x + threadIdx.x) >> 5); i < n.N; i += warps) {
		for(int r = 0; r < len; ++r) {
			g[r * 32 + int(lane)] = int(lane) < tw ? guSeg[(size_t(t0 - segStart + r) * n.N + i) * tw + lane] : 0.0f;
		}
		__syncwarp();
		const int k0 = n.rowptr[i], k1 = n.rowptr[i + 1];
		/* the next synapse's unit, count and first codes are on their way while
		 * one is summed */
		int k = k0 + int(lane);
		int p = k < k1 ? n.pre[k] : 0;
		uint32_t c = k < k1 ? cnt[p] : 0u;
		int pNext = k + 32 < k1 ? n.pre[k + 32] : 0;
		for(; k < k1; k += 32) {
			const uint4* list = reinterpret_cast<const uint4*>(codes + size_t(p) * cap);
			float acc = zero;
			uint4 n0 = list[0], n1 = list[1];
			const uint32_t cNext = k + 32 < k1 ? cnt[pNext] : 0u;
			const int pAfter = k + 64 < k1 ? n.pre[k + 64] : 0;
			const float old = dw[k];
			for(uint32_t e = 0; e < c; e += 8u) {
				const uint4 x = n0;
				n0 = n1;
				if(e + 16u < c) n1 = list[(e >> 3) + 2u];
				acc = __fadd_rn(acc, g[x.x & 0xffffu]);
				acc = __fadd_rn(acc, g[x.x >> 16]);
				acc = __fadd_rn(acc, g[x.y & 0xffffu]);
				acc = __fadd_rn(acc, g[x.y >> 16]);
				acc = __fadd_rn(acc, g[x.z & 0xffffu]);
				acc = __fadd_rn(acc, g[x.z >> 16]);
				acc = __fadd_rn(acc, g[x.w & 0xffffu]);
				acc = __fadd_rn(acc, g[x.w >> 16]);
			}
			dw[k] = __fadd_rn(old, acc);
			p = pNext;
			c = cNext;
			pNext = pAfter;
		}
		__syncwarp();
	}
}

/* floats of a row of trials: 8, 16 or 32 */
static int rowWidth(int B) { return B <= 8 ? 8 : (B <= 16 ? 16 : 32); }

/* ---- the adjoint of a segment in one launch (spikes as bits) ----
 *
 * A step is gs_j = sum over out-synapses (j -> i) of w * gu[t+1]_i: every
 * synapse reads one row of gu (4 bytes a trial). From L2 that is 256 MB a
 * step for 2e6 synapses and 32 trials, a chain of dependent row gathers a
 * warp (71 us a step). Here the rows are in shared memory, read at 128 bytes
 * a clock and SM:
 *   - the blocks form groups of `parts` blocks (8, or as many as the rows
 *     need); block p of each holds the rows of the p-th part of the neurons,
 *     and every group owns an equal share of the sources, so that each
 *     (source, part) pair has one block;
 *   - a source is worked off by a few lanes (of 32 trials: four lanes, two
 *     float4 each, so that a warp has 8 sources and reads their rows without
 *     bank conflicts), which walk the pair's synapses in order, four a turn. The
 *     synapses are laid out part by part, in a part source by source, as
 *     {row offset, weight} (k_out_fill), every pair filled up to whole turns,
 *     and a lane group has a run of whole sources of about the same length as
 *     every other: the groups of a warp go in step and nothing in a turn is a
 *     branch (a divergent one costs about 75 clocks). A block keeps its
 *     synapses in shared memory when they fit, else they come through a ring
 *     of asynchronous copies a lane group;
 *   - a source's sum over one part goes to global memory (L2) at its last
 *     entry; after a grid barrier the parts are added, in part order, so that
 *     the result does not depend on timing, by the block that finishes the
 *     source and writes its gu[t] row; a second grid barrier ends the step.
 *     (Thread-block clusters of 8 with the sums in distributed shared memory
 *     measured slower: 15 of them run at once, 120 of 148 SMs, their barrier
 *     is no cheaper, and reading the sums took twice as long as from L2.) */

const int ADJ_THREADS = 1024;
const int ADJ_WARPS = ADJ_THREADS / 32;
/* At least 8 parts also where fewer would hold the rows: a part's rows are
 * read from L2 by every group each step, so few parts mean many rows a block;
 * many parts mean sums to add. us a step with at least 2 / 4 / 8 / 16 parts:
 * 300 neurons of 8 trials 4.4 / 4.7 / 4.6 / 5.2, 1,000 of 32 7.5 / 6.1 / 5.4 /
 * 6.6, 2,000 of 32 10.4 / 7.7 / 7.5 / 9.0, 3,000 of 16 8.9 / 7.5 / 8.5 / 8.8,
 * 5,000 of 32 14.0 / 14.0 / 12.2 / 12.5 */
const int ADJ_MIN_PARTS = 8, ADJ_MAX_PARTS = 32;
/* sources of a group (their places in a block's shared memory) */
const size_t ADJ_SOURCES = 8192;
/* rows of gu, the group's sources and the rings (the largest block has 227
 * KB) */
const size_t ADJ_SMEM = 224 * 1024;
/* entries a block may load past its last bucket's end (its rings) */
const size_t ADJ_SLACK = 64;
/* in a bucket's last entry's row offset (a multiple of 32) */
const uint32_t ADJ_LAST = 1u;

struct Adjoint {
	int c0, c1;              /* the segment's steps */
	int parts;               /* blocks per group */
	int partRows;            /* neurons per part */
	int perGroup;            /* sources per group */
	const uint2* bucket;     /* [parts][N] {first entry in the part, count} */
	const uint32_t* total;   /* [parts] entries of each part */
	const uint2* entries;    /* {byte offset of the target's row in its part (| ADJ_LAST), weight}, part after part */
	float* sums;             /* [parts][N][TW] */
	const float* uSeg;       /* [K][N][TW] */
	const float* guNext;     /* [N][TW] gu of step c1 */
	float* guSeg;            /* [K][N][TW] */
	const float* dcounts;
	unsigned* barrier;       /* [0] arrivals, [1] error */
	unsigned barrierBase;    /* arrivals before this launch */
};

/* Synapses of every (source, part) pair, warp per source: cnt[p * N + j] */
__global__ void __launch_bounds__(THREADS)
k_out_count(Net n, int parts, int partRows, uint2* bucket)
{
	const uint32_t lane = threadIdx.x & 31u;
	const int warps = int((gridDim.x * blockDim.x) >> 5);
	for(int j = int((blockIdx.x * blockDim.x + threadIdx.x) >> 5); j < n.N; j += warps) {
		uint32_t mine = 0;   /* lane p: the count of part p */
		const int e0 = n.colptr[j], e1 = n.colptr[j + 1];
		for(int base = e0; base < e1; base += 32) {
			const int e = base + int(lane);
			const int part = e < e1 ? n.post[e] / partRows : -1;
			for(int p = 0; p < parts; ++p) {
				const uint32_t c = uint32_t(__popc(__ballot_sync(FULL, part == p)));
				if(int(lane) == p) mine += c;
			}
		}
		if(int(lane) < parts) bucket[size_t(lane) * n.N + j].y = mine;
	}
}

/* The first entry of every pair in its part (block per part): an exclusive
 * sum of the counts rounded up to a multiple of 4 (at least 4), which
 * k_out_fill fills up with entries that add 0 (the row past the part's last
 * one, weight 0) */
__global__ void __launch_bounds__(1024)
k_out_scan(int N, uint2* bucket, uint32_t* total)
{
	__shared__ uint32_t warpSum[32];
	const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
	uint2* b = bucket + size_t(blockIdx.x) * N;
	const int per = (N + 1023) / 1024;
	const int lo = min(N, int(threadIdx.x) * per), hi = min(N, lo + per);
	uint32_t sum = 0;
	for(int j = lo; j < hi; ++j) sum += max(4u, (b[j].y + 3u) & ~3u);
	uint32_t incl = sum;
#pragma unroll
	for(int d = 1; d < 32; d <<= 1) {
		const uint32_t x = __shfl_up_sync(FULL, incl, d);
		if(lane >= uint32_t(d)) incl += x;
	}
	if(lane == 31) warpSum[warp] = incl;
	__syncthreads();
	if(warp == 0) {
		const uint32_t v = warpSum[lane];
		uint32_t w = v;
#pragma unroll
		for(int d = 1; d < 32; d <<= 1) {
			const uint32_t x = __shfl_up_sync(FULL, w, d);
			if(lane >= uint32_t(d)) w += x;
		}
		warpSum[lane] = w - v;
		if(lane == 31) total[blockIdx.x] = w;
	}
	__syncthreads();
	uint32_t run = warpSum[warp] + incl - sum;
	for(int j = lo; j < hi; ++j) {
		b[j].x = run;
		run += max(4u, (b[j].y + 3u) & ~3u);
	}
}

/* The entries of every source (warp per source), in out-synapse order within
 * a pair */
__global__ void __launch_bounds__(THREADS)
k_out_fill(Net n, int parts, int partRows, int rowBytes, const uint2* bucket, const uint32_t* total, const float* w,
		uint2* entries)
{
	const uint32_t lane = threadIdx.x & 31u;
	const uint32_t lt = (1u << lane) - 1u;
	const int warps = int((gridDim.x * blockDim.x) >> 5);
	uint32_t partBase = 0;   /* lane p: the first entry of part p */
	for(int p = 0; p < int(lane) && p < parts; ++p) partBase += total[p];
	for(int j = int((blockIdx.x * blockDim.x + threadIdx.x) >> 5); j < n.N; j += warps) {
		uint32_t next = int(lane) < parts ? partBase + bucket[size_t(lane) * n.N + j].x : 0u;
		const int e0 = n.colptr[j], e1 = n.colptr[j + 1];
		for(int base = e0; base < e1; base += 32) {
			const int e = base + int(lane);
			const int i = e < e1 ? n.post[e] : 0;
			const int part = e < e1 ? i / partRows : -1;
			for(int p = 0; p < parts; ++p) {
				const uint32_t m = __ballot_sync(FULL, part == p);
				const uint32_t first = __shfl_sync(FULL, next, p);
				if(part == p) {
					entries[first + uint32_t(__popc(m & lt))] = make_uint2(uint32_t(i - p * partRows) * uint32_t(rowBytes),
							__float_as_uint(w[n.wpos[e]]));
				}
				if(int(lane) == p) next += uint32_t(__popc(m));
			}
		}
		__syncwarp();
		if(int(lane) < parts) {
			const uint32_t first = partBase + bucket[size_t(lane) * n.N + j].x;
			while(next == first || (next & 3u)) entries[next++] = make_uint2(uint32_t(partRows) * uint32_t(rowBytes), 0u);
			entries[next - 1u].x |= ADJ_LAST;
		}
	}
}

/* The grid barrier: every block arrives (its writes before are visible to
 * what waits), then waits for `target` arrivals in all. The wait is bounded:
 * after 10 s it sets the error word (the call's results become NaN), and no
 * block waits any more. */
__device__ __forceinline__ void gridArrive(unsigned* bar)
{
	__syncthreads();
	if(threadIdx.x == 0) {
		asm volatile("red.release.gpu.global.add.u32 [%0], 1;" :: "l"(__cvta_generic_to_global(bar)) : "memory");
	}
}

__device__ __forceinline__ void gridWait(unsigned* bar, unsigned target)
{
	if(threadIdx.x == 0) {
		const size_t g = __cvta_generic_to_global(bar);
		unsigned long long start = 0;
		for(unsigned spins = 1;; ++spins) {
			unsigned v;
			asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(g) : "memory");
			if(int(v - target) >= 0) break;
			if((spins & 255u) == 0) {
				unsigned long long now;
				asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(now));
				if(start == 0) start = now;
				if(*(volatile unsigned*) &bar[1]) break;
				if(now - start > 10ull * 1000 * 1000 * 1000) {
					*(volatile unsigned*) &bar[1] = 1u;
					break;
				}
			}
		}
	}
	__syncthreads();
}

/* Row-width constants of k_adjoint */
template<int TW>
struct AdjointShape {
	static const int FLOATS = TW == 32 ? 8 : 4;     /* trials of a lane */
	static const int LANES = TW / FLOATS;           /* lanes of a source */
	static const int GROUPS = 32 / LANES;           /* sources of a warp at once */
	static const int SLOTS = ADJ_WARPS * GROUPS;    /* sources of a block at once */
	static const int RING = 8;                      /* entry pairs on their way to a lane group */
};

/* bytes of the rings of a block */
static size_t
adjointRings(int tw)
{
	const int slots = tw == 32 ? AdjointShape<32>::SLOTS : (tw == 16 ? AdjointShape<16>::SLOTS : AdjointShape<8>::SLOTS);
	return size_t(slots) * AdjointShape<32>::RING * 16;
}

/* Parts of the neurons: 8, or as many as it takes for a part's rows (and the
 * row of zeros) to fit a block beside its sources and rings (from 10,233
 * neurons of 32 trials, 20,473 of 16 and 32,761 of 8 on); 0 past 32 parts */
static int
adjointParts(int N, int tw)
{
	for(int parts = ADJ_MIN_PARTS; parts <= ADJ_MAX_PARTS; ++parts) {
		const size_t rows = size_t((N + parts - 1) / parts) + 1;
		if(rows * tw * 4 + ADJ_SOURCES * 4 + adjointRings(tw) <= ADJ_SMEM) return parts;
	}
	return 0;
}

template<int TW>
__global__ void __launch_bounds__(ADJ_THREADS, 1)
k_adjoint(const __grid_constant__ Net n, const __grid_constant__ Adjoint a)
{
	extern __shared__ __align__(128) char smem[];
	typedef AdjointShape<TW> S;
	const int LANES = S::LANES, RING = S::RING, FLOATS = S::FLOATS;
	const int Q = TW / 4;                     /* float4s of a row */
	const uint32_t lane = threadIdx.x & 31u;
	const int warp = int(threadIdx.x >> 5);
	const int part = int(blockIdx.x) % a.parts;
	/* the part's rows of gu and a row of zeros */
	float* sG = reinterpret_cast<float*>(smem);
	uint32_t* sFirst = reinterpret_cast<uint32_t*>(sG + size_t(a.partRows + 1) * TW);   /* first pair of each source */
	uint4* sEntry = reinterpret_cast<uint4*>(sFirst + (a.perGroup + 1 + 3) / 4 * 4);
	const uint32_t room = uint32_t(ADJ_SMEM - size_t(reinterpret_cast<char*>(sEntry) - smem)) / 16u;

	const int src0 = int(blockIdx.x) / a.parts * a.perGroup;
	const int ns = max(0, min(a.perGroup, n.N - src0));         /* the group's sources */
	const int row0 = part * a.partRows;
	const int rows = max(0, min(a.partRows, n.N - row0));       /* the block's rows */
	const int own = (a.perGroup + a.parts - 1) / a.parts;       /* sources a block finishes */
	const int fin0 = min(ns, part * own), fin1 = min(ns, fin0 + own);
	const int items = (fin1 - fin0) * Q;
	uint32_t partBase = 0;
	for(int p = 0; p < part; ++p) partBase += a.total[p];
	const uint2* bucket = a.bucket + size_t(part) * n.N + src0;
	const uint32_t firstPair = ns ? bucket[0].x / 2u : 0u;
	for(int s = int(threadIdx.x); s < ns; s += ADJ_THREADS) {
		const uint2 b = bucket[s];
		sFirst[s] = b.x / 2u - firstPair;
		if(s == ns - 1) sFirst[ns] = b.x / 2u - firstPair + max(4u, (b.y + 3u) & ~3u) / 2u;
	}
	if(threadIdx.x < uint32_t(TW)) sG[size_t(a.partRows) * TW + threadIdx.x] = 0.0f;
	__syncthreads();
	/* the block's entries in pairs, one run for its sources in order */
	const uint32_t pairs = ns ? sFirst[ns] : 0u;
	const uint4* entries = reinterpret_cast<const uint4*>(a.entries + partBase) + firstPair;
	const bool kept = pairs + 2u <= room;   /* and two pairs of slack */
	if(kept) {
		for(uint32_t q = threadIdx.x; q < pairs; q += ADJ_THREADS) sEntry[q] = __ldg(entries + q);
	}

	/* the lane group's run: the sources that start in its share of the pairs.
	 * A 16-byte load costs a warp the same with one group as with all, so the
	 * groups used fill whole warps: one for a source, from 128 sources on one
	 * for at least five (runs of five sources differ little in length) */
	const int group = int(lane) / LANES;
	const int slot = warp * S::GROUPS + group;
	const int used = min(S::SLOTS, ns <= 128 ? max(ns, 1) : max(128, ns / 5));
	auto sourceAt = [&](uint64_t pair) {
		int lo = 0, hi = ns;   /* the first source that starts at or after it */
		while(lo < hi) {
			const int mid = (lo + hi) / 2;
			if(uint64_t(sFirst[mid]) >= pair) hi = mid;
			else lo = mid + 1;
		}
		return lo;
	};
	int s0 = ns, s1 = ns;
	if(ns <= 128) {
		s0 = min(slot, ns);
		s1 = min(slot + 1, ns);
	} else if(slot < used) {
		s0 = sourceAt((uint64_t(pairs) * slot + used - 1) / used);
		s1 = sourceAt((uint64_t(pairs) * (slot + 1) + used - 1) / used);
	}
	const uint32_t run0 = s0 < s1 ? sFirst[s0] : 0u;
	const uint32_t turns = s0 < s1 ? (sFirst[s1] - run0) / 2u : 0u;
	const uint32_t live = __ballot_sync(FULL, turns != 0u);   /* the lanes with a run */
	const int own0 = int(lane) % LANES;
	/* the lane's float4s of a row: odd groups start with the second one, so
	 * that the two groups of a quarter-warp meet on no bank */
	const int H = FLOATS / 4;
	int at[H];
#pragma unroll
	for(int h = 0; h < H; ++h) at[h] = H == 1 ? own0 * 16 : ((h + group) % H) * 64 + own0 * 16;
	const char* const rowsAt = reinterpret_cast<const char*>(sG);
	const uint32_t zeroAt = uint32_t(a.partRows) * TW * 4u;
	uint4* ring = sEntry + (warp * S::GROUPS + group) * RING;
	const uint32_t ringAt = uint32_t(__cvta_generic_to_shared(ring));
	float* const sums0 = a.sums + (size_t(part) * n.N + size_t(src0 + s0)) * TW;
	const int bins = n.T / n.binSteps;
	unsigned target = a.barrierBase;

	auto fetch = [&](uint32_t pair) {
		asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" :: "r"(ringAt + (pair & uint32_t(RING - 1)) * 16u),
				"l"(__cvta_generic_to_global(entries + pair)) : "memory");
	};
	__syncthreads();

	for(int t = a.c1 - 1; t >= a.c0; --t) {
		const bool last = t == n.T - 1;
		const float* next = t == a.c1 - 1 ? a.guNext : a.guSeg + size_t(t + 1 - a.c0) * n.N * TW;
		const float* uT = a.uSeg + size_t(t - a.c0) * n.N * TW;
		float* out = a.guSeg + size_t(t - a.c0) * n.N * TW;

		if(!last) {
			if(!kept && turns) {
				for(int q = own0; q < RING; q += LANES) fetch(run0 + uint32_t(q));
			}
			/* the rows of gu[t+1], past the L1 cache: other blocks have written
			 * them */
			const uint32_t dst = uint32_t(__cvta_generic_to_shared(sG));
			const char* src = reinterpret_cast<const char*>(next + size_t(row0) * TW);
			for(int q = int(threadIdx.x); q < rows * Q; q += ADJ_THREADS) {
				asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" :: "r"(dst + uint32_t(q) * 16u),
						"l"(__cvta_generic_to_global(src + size_t(q) * 16)) : "memory");
			}
			asm volatile("cp.async.wait_all;" ::: "memory");
			__syncthreads();
			if(turns) {
				const uint32_t most = __reduce_max_sync(live, turns);
				uint32_t pos = run0, filled = run0 + uint32_t(RING);
				float acc[FLOATS];
#pragma unroll
				for(int q = 0; q < FLOATS; ++q) acc[q] = 0.0f;
				/* one entry into the lane's sums; `on` (all bits or none) sends
				 * those of a group that is through to the row of zeros */
				auto add = [&](uint32_t off, uint32_t w, uint32_t on) {
					const char* row = rowsAt + ((off & on & ~31u) | (zeroAt & ~on));
					const float ww = __uint_as_float(w & on);
#pragma unroll
					for(int h = 0; h < H; ++h) {
						const float4 g = *reinterpret_cast<const float4*>(row + at[h]);
						acc[4 * h + 0] = __fmaf_rn(ww, g.x, acc[4 * h + 0]);
						acc[4 * h + 1] = __fmaf_rn(ww, g.y, acc[4 * h + 1]);
						acc[4 * h + 2] = __fmaf_rn(ww, g.z, acc[4 * h + 2]);
						acc[4 * h + 3] = __fmaf_rn(ww, g.w, acc[4 * h + 3]);
					}
				};
				size_t sumAt = __cvta_generic_to_global(sums0);
				auto turn = [&](uint32_t e, const uint4& x, const uint4& y) {
					const uint32_t on = e < turns ? FULL : 0u;
					add(x.x, x.y, on);
					add(x.z, x.w, on);
					add(y.x, y.y, on);
					add(y.z, y.w, on);
					pos += on & 2u;
					/* the source's last entry: its sum, then the next one's */
					const uint32_t done = y.z & on & ADJ_LAST;
#pragma unroll
					for(int h = 0; h < H; ++h) {
						asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.u32 p, %5, 0;\n\t"
								"@p st.global.v4.f32 [%0], {%1, %2, %3, %4};\n\t}" :: "l"(sumAt + size_t(at[h])),
								"f"(acc[4 * h]), "f"(acc[4 * h + 1]), "f"(acc[4 * h + 2]), "f"(acc[4 * h + 3]), "r"(done) : "memory");
					}
					const uint32_t keep = done - 1u;   /* all bits, or none after the last */
#pragma unroll
					for(int q = 0; q < FLOATS; ++q) acc[q] = __uint_as_float(__float_as_uint(acc[q]) & keep);
					sumAt += done * uint32_t(TW * 4);
				};
				if(kept) {
					/* a group that is through may read past its run: inside the
					 * block's entries and the slack behind them */
					for(uint32_t e = 0; e < most; ++e) turn(e, sEntry[pos], sEntry[pos + 1u]);
				} else {
					/* two pairs are used and replaced a turn; this turn's were
					 * asked for RING / 2 - 1 turns ago at the latest */
					for(uint32_t e = 0; e < most; ++e) {
						const uint32_t upTo = pos + uint32_t(RING);
						if(filled + uint32_t(own0) < upTo) fetch(filled + uint32_t(own0));
						filled = upTo;
						asm volatile("cp.async.commit_group;\n\tcp.async.wait_group %0;" :: "n"(RING / 2 - 1) : "memory");
						__syncwarp(live);
						turn(e, ring[pos & uint32_t(RING - 1)], ring[(pos + 1u) & uint32_t(RING - 1)]);
						__syncwarp(live);
					}
					/* the copies asked for past the run's end: the next step
					 * writes the same places, and copies have no order of their
					 * own */
					asm volatile("cp.async.wait_all;" ::: "memory");
				}
			}
		}
		gridArrive(a.barrier);
		/* what finishing the thread's first item needs, on its way during the
		 * barrier (a thread without an item loads some row: a load under a
		 * condition would be waited for at the condition's end) */
		float4 u0, g0;
		float dc[4];
		auto operands = [&](int x, float4& u, float4& g) {
			const size_t cell = size_t(min(src0 + fin0 + x / Q, n.N - 1)) * TW + size_t(x % Q) * 4;
			u = *reinterpret_cast<const float4*>(uT + cell);
			g = __ldcg(reinterpret_cast<const float4*>(next + cell));
		};
		operands(min(int(threadIdx.x), max(items - 1, 0)), u0, g0);
#pragma unroll
		for(int q = 0; q < 4; ++q) {
			const int b = min(int(threadIdx.x) % Q * 4 + q, n.B - 1);
			dc[q] = __ldg(&a.dcounts[size_t(b) * bins + t / n.binSteps]);
		}
		target += gridDim.x;
		gridWait(a.barrier, target);
#pragma unroll 1
		for(int x = int(threadIdx.x); x < items; x += ADJ_THREADS) {
			if(x >= ADJ_THREADS) operands(x, u0, g0);
			const int c = (x % Q) * 4;
			const size_t cell = size_t(src0 + fin0 + x / Q) * TW + c;
			float4 sum = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
			if(last) {
				g0 = sum;
			} else {
				for(int q0 = 0; q0 < a.parts; q0 += 8) {
					float4 y[8];
#pragma unroll
					for(int q = 0; q < 8; ++q) {
						y[q] = __ldcg(reinterpret_cast<const float4*>(a.sums + size_t(min(q0 + q, a.parts - 1)) * n.N * TW + cell));
					}
#pragma unroll
					for(int q = 0; q < 8; ++q) {
						if(q0 + q < a.parts) {
							sum.x = __fadd_rn(sum.x, y[q].x);
							sum.y = __fadd_rn(sum.y, y[q].y);
							sum.z = __fadd_rn(sum.z, y[q].z);
							sum.w = __fadd_rn(sum.w, y[q].w);
						}
					}
				}
			}
			const float us[4] = {u0.x, u0.y, u0.z, u0.w}, gn[4] = {g0.x, g0.y, g0.z, g0.w}, ss[4] = {sum.x, sum.y, sum.z, sum.w};
			float r[4];
#pragma unroll
			for(int q = 0; q < 4; ++q) {
				r[q] = guOf(n, us[q], __fadd_rn(dc[q], ss[q]), __fmul_rn(n.beta, gn[q]));
				if(c + q >= n.B) r[q] = 0.0f;
			}
			const float4 v = make_float4(r[0], r[1], r[2], r[3]);
			*reinterpret_cast<float4*>(out + cell) = v;
		}
		if(t > a.c0) {
			target += gridDim.x;
			gridArrive(a.barrier);
			gridWait(a.barrier, target);
		}
	}
}

/* ---- the forward in one launch (spikes as bits) ----
 *
 * A step needs every neuron's spikes of the step before. One launch runs all
 * steps with a grid barrier between them, where a launch per step costs the
 * launch, the reload of every synapse from L2 (20 MB for 2.5e6) and a lane per
 * trial that takes the synapses one by one. A block owns a contiguous range of
 * neurons: their synapses, v and the step's spike words are in shared memory
 * (synapses past its room are read from L2).
 *
 * A neuron is a warp. Lane L first has the spike word of synapse 31 - L of 32
 * (bit b: trial b); the words are transposed (5 exchanges between lanes), after
 * which lane b has the synapses that spike in trial b, the first one in the
 * highest bit, and adds their weights in synapse order: as many turns as the
 * busiest trial has spikes. What bounds a step is the shared-memory and
 * exchange instructions and, with few neurons a block, their latency (a chain
 * of about 1,000 clocks for 64 synapses): a warp whose block owns more neurons
 * than warps takes two to four of them at once. */

const int FWD_THREADS = 1024;
const int FWD_WARPS = FWD_THREADS / 32;
const size_t FWD_SMEM = 224 * 1024;

struct Forward {
	const float* w;
	const uint32_t* inBits;
	uint32_t* sBits;
	float* vCkpt;
	float* counts;
	int perBlock;            /* neurons a block owns */
	int cached;              /* synapses of a block in shared memory */
	unsigned* barrier;       /* [0] arrivals, [1] error */
};

template<int NN>
__global__ void __launch_bounds__(FWD_THREADS, 1)
k_forward(const __grid_constant__ Net n, const __grid_constant__ Forward a)
{
	extern __shared__ __align__(128) char smem[];
	__shared__ unsigned sCount[32];
	const uint32_t lane = threadIdx.x & 31u;
	const int warp = int(threadIdx.x >> 5);
	const int units = n.N + n.C;
	uint32_t* sWords = reinterpret_cast<uint32_t*>(smem);
	float* sV = reinterpret_cast<float*>(sWords + (units + 31) / 32 * 32);
	float* sW = sV + size_t(a.perBlock) * 32;
	int* sPre = reinterpret_cast<int*>(sW + a.cached);
	int* sRow = sPre + a.cached;   /* first synapse of each owned neuron, from the block's first one */
	/* the transposition's exchange at distance d: keep the bits of keep[d],
	 * take the others from the partner, rotated by turn[d] */
	uint32_t keep[5], turn[5];
	{
		uint32_t m = 0x0000ffffu;
#pragma unroll
		for(int x = 0; x < 5; ++x) {
			const uint32_t d = 16u >> x;
			keep[x] = (lane & d) ? ~m : m;
			turn[x] = (lane & d) ? 32u - d : d;
			m ^= m << (d >> 1);
		}
	}

	const int i0 = int(blockIdx.x) * a.perBlock;
	const int own = max(0, min(a.perBlock, n.N - i0));
	const int kFirst = own > 0 ? n.rowptr[i0] : 0;
	const int kEnd = own > 0 ? n.rowptr[i0 + own] - kFirst : 0;
	const int kCached = min(a.cached, kEnd);
	for(int k = int(threadIdx.x); k < kCached; k += FWD_THREADS) {
		sW[k] = a.w[kFirst + k];
		sPre[k] = n.pre[kFirst + k];
	}
	for(int x = int(threadIdx.x); x < own * 32; x += FWD_THREADS) sV[x] = 0.0f;
	for(int x = int(threadIdx.x); x <= own; x += FWD_THREADS) sRow[x] = own ? n.rowptr[i0 + x] - kFirst : 0;
	if(threadIdx.x < 32) sCount[threadIdx.x] = 0u;

	unsigned target = 0, spikes = 0;
	for(int t = 0; t < n.T; ++t) {
		/* the words this step's synapses deliver: the neurons' of the step
		 * before (past the L1 cache: other blocks wrote them), the inputs' of
		 * this step */
		float* ckpt = t % n.K == 0 ? a.vCkpt + size_t(t / n.K) * n.N * 32 : nullptr;
		const uint32_t* prev = a.sBits + size_t(t - 1) * n.N;
		for(int p0 = int(threadIdx.x); p0 < n.N; p0 += 12 * FWD_THREADS) {
			uint32_t x[12];
#pragma unroll
			for(int q = 0; q < 12; ++q) {
				const int p = p0 + q * FWD_THREADS;
				x[q] = t && p < n.N ? __ldcg(&prev[p]) : 0u;
			}
#pragma unroll
			for(int q = 0; q < 12; ++q) {
				const int p = p0 + q * FWD_THREADS;
				if(p < n.N) sWords[p] = x[q];
			}
		}
		for(int c = int(threadIdx.x); c < n.C; c += FWD_THREADS) sWords[n.N + c] = a.inBits[size_t(t) * n.C + c];
		__syncthreads();
		for(int l0 = warp * NN; l0 < own; l0 += FWD_WARPS * NN) {
			/* NN neurons at once, C groups of 32 synapses of each (a neuron past
			 * the block's last one: no synapses, nothing stored) */
			const int C = NN == 1 ? 2 : 1;
			float I[NN];
			int k0[NN], k1[NN];
			int most = 0;
			bool near = true;
#pragma unroll
			for(int j = 0; j < NN; ++j) {
				const bool in = l0 + j < own;
				I[j] = 0.0f;
				k0[j] = in ? sRow[l0 + j] : 0;
				k1[j] = in ? sRow[l0 + j + 1] : 0;
				most = max(most, k1[j] - k0[j]);
				/* synapses in shared memory, or (some past the block's room)
				 * all from L2 */
				near = near && k1[j] <= kCached;
			}
			for(int base = 0; base < most; base += 32 * C) {
				uint32_t word[NN][C];
				float wk[NN][C];
#pragma unroll
				for(int j = 0; j < NN; ++j) {
#pragma unroll
					for(int c = 0; c < C; ++c) {
						/* past the end: the neuron's last synapse (or the block's
						 * first one), with no spikes */
						const int k = k0[j] + base + c * 32 + 31 - int(lane);
						const int kk = max(min(k, k1[j] - 1), 0);
						const int p = near ? sPre[kk] : __ldg(&n.pre[kFirst + kk]);
						wk[j][c] = near ? sW[kk] : __ldg(&a.w[kFirst + kk]);
						word[j][c] = sWords[p] & (k < k1[j] ? FULL : 0u);
					}
				}
#pragma unroll
				for(int x = 0; x < 5; ++x) {
#pragma unroll
					for(int j = 0; j < NN; ++j) {
#pragma unroll
						for(int c = 0; c < C; ++c) {
							const uint32_t y = __shfl_xor_sync(FULL, word[j][c], 16 >> x);
							word[j][c] = (word[j][c] & keep[x]) | (__funnelshift_l(y, y, turn[x]) & ~keep[x]);
						}
					}
				}
#pragma unroll
				for(int c = 0; c < C; ++c) {
					unsigned spikesMost = 0;
#pragma unroll
					for(int j = 0; j < NN; ++j) spikesMost = max(spikesMost, unsigned(__popc(word[j][c])));
					const unsigned turns = __reduce_max_sync(FULL, spikesMost);
					/* two turns at once */
					for(unsigned x = 0; x < turns; x += 2u) {
#pragma unroll
						for(int j = 0; j < NN; ++j) {
							const uint32_t first = word[j][c];
							const int q0 = 31 - __clz(int(first));
							const uint32_t second = first & ~(1u << (q0 & 31));
							const int q1 = 31 - __clz(int(second));
							word[j][c] = second & ~(1u << (q1 & 31));
							const float w0 = __shfl_sync(FULL, wk[j][c], q0), w1 = __shfl_sync(FULL, wk[j][c], q1);
							if(first) I[j] = __fadd_rn(I[j], w0);
							if(second) I[j] = __fadd_rn(I[j], w1);
						}
					}
				}
			}
#pragma unroll
			for(int j = 0; j < NN; ++j) {
				if(l0 + j >= own) break;
				const int l = l0 + j, i = i0 + l;
				const float vPrev = sV[l * 32 + int(lane)];
				if(ckpt) ckpt[size_t(i) * 32 + lane] = vPrev;
				const float u = __fadd_rn(__fmul_rn(n.beta, vPrev), I[j]);
				const bool s = lane < uint32_t(n.B) && u >= n.theta;
				sV[l * 32 + int(lane)] = __fsub_rn(u, __fmul_rn(n.theta, s ? 1.0f : 0.0f));
				const uint32_t out = __ballot_sync(FULL, s);
				if(lane == 0) a.sBits[size_t(t) * n.N + i] = out;
				spikes += s ? 1u : 0u;
			}
		}
		if((t + 1) % n.binSteps == 0) {
			/* whole numbers: the order does not matter */
			if(spikes) atomicAdd(&sCount[lane], spikes);
			spikes = 0;
			__syncthreads();
			if(threadIdx.x < uint32_t(n.B) && sCount[threadIdx.x]) {
				atomicAdd(&a.counts[size_t(threadIdx.x) * (n.T / n.binSteps) + t / n.binSteps], float(sCount[threadIdx.x]));
				sCount[threadIdx.x] = 0u;
			}
		}
		if(t + 1 < n.T) {
			if(gridDim.x == 1) {
				__syncthreads();
			} else {
				target += gridDim.x;
				gridArrive(a.barrier);
				gridWait(a.barrier, target);
			}
		}
	}
	/* a barrier gave up: the counts become NaN */
	if(threadIdx.x == 0 && *(volatile unsigned*) &a.barrier[1]) {
		for(int x = 0; x < n.B * (n.T / n.binSteps); ++x) atomicAdd(&a.counts[x], __int_as_float(0x7fffffff));
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

static const void*
adjointKernel(int tw)
{
	return tw == 8 ? (const void*) k_adjoint<8> : (tw == 16 ? (const void*) k_adjoint<16> : (const void*) k_adjoint<32>);
}

/* A kernel may use that much dynamic shared memory on the current device:
 * the attribute is the device's, shared by all threads, so it is set once, to
 * the most any call needs, and stays. False: a device with less. */
static bool
allowShared(const void* kernel, size_t smem)
{
	static std::mutex lock;
	static std::map<std::pair<int, const void*>, bool> known;
	int dev = 0;
	NEMO_CUDA(cudaGetDevice(&dev));
	std::lock_guard<std::mutex> guard(lock);
	const std::pair<int, const void*> key(dev, kernel);
	auto it = known.find(key);
	if(it != known.end()) return it->second;
	const cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, int(smem));
	if(e != cudaSuccess) (void) cudaGetLastError();
	return known[key] = e == cudaSuccess;
}

/* blocks of a kernel with that much shared memory that can run at once (one
 * an SM; 0: it does not fit), by device and kernel */
static int
residentBlocks(const void* kernel, int threads, size_t smem)
{
	static std::mutex lock;
	static std::map<std::pair<int, const void*>, int> known;
	int dev = 0;
	NEMO_CUDA(cudaGetDevice(&dev));
	std::lock_guard<std::mutex> guard(lock);
	const std::pair<int, const void*> key(dev, kernel);
	auto it = known.find(key);
	if(it != known.end()) return it->second;
	int perSm = 0, sms = 0, coop = 0;
	NEMO_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
	NEMO_CUDA(cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, dev));
	if(coop && allowShared(kernel, smem)) {
		NEMO_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&perSm, kernel, threads, smem));
	}
	known[key] = perSm > 0 ? sms : 0;
	return known[key];
}

struct AdjointPlan {
	int tw = 32;
	int parts = 0;   /* 0: step by step (k_back) */
	int groups = 0, partRows = 0, perGroup = 0;
};

/* The adjoint in one launch a segment: a group for every 64 sources, as many
 * as run at once. Step by step where a group would have more sources than a
 * block has places for, since many parts leave few groups: past 37,091 neurons
 * of 32 trials (30 parts, four groups), 53,739 of 16, 65,520 of 8 on 148 SMs. */
static AdjointPlan
planAdjoint(const Net& n)
{
	AdjointPlan p;
	const int tw = rowWidth(n.B);
	const int parts = adjointParts(n.N, tw);
	const int most = residentBlocks(adjointKernel(tw), ADJ_THREADS, ADJ_SMEM);
	if(parts == 0 || most < parts) return p;
	const int groups = std::max(1, std::min(most / parts, (n.N + 63) / 64));
	const int per = (n.N + groups - 1) / groups;
	if(size_t(per) + 4 > ADJ_SOURCES) return p;
	p.tw = tw;
	p.parts = parts;
	p.groups = (n.N + per - 1) / per;
	p.partRows = (n.N + parts - 1) / parts;
	p.perGroup = per;
	return p;
}

/* the forward with nn neurons a warp at once */
static const void*
forwardKernel(int nn)
{
	switch(nn) {
		case 1: return (const void*) k_forward<1>;
		case 2: return (const void*) k_forward<2>;
		case 3: return (const void*) k_forward<3>;
		default: return (const void*) k_forward<4>;
	}
}

struct ForwardPlan {
	int blocks = 0;   /* 0: step by step (k_step) */
	int perBlock = 0, cached = 0;
	const void* kernel = nullptr;
};

/* The forward in one launch, unless the spike words and v of a block do not
 * fit its shared memory (past 46,400 to 46,900 neurons, by the channels): eight neurons a block at least,
 * a warp a neuron, a large network's neurons two to four a warp at once. */
static ForwardPlan
planForward(const Net& n)
{
	ForwardPlan p;
	int most = residentBlocks(forwardKernel(1), FWD_THREADS, FWD_SMEM);
	for(int nn = 2; nn <= 4; ++nn) most = std::min(most, residentBlocks(forwardKernel(nn), FWD_THREADS, FWD_SMEM));
	if(most == 0) return p;
	const int blocks = std::min(most, (n.N + 7) / 8);
	const int per = (n.N + blocks - 1) / blocks;
	const size_t fixed = (size_t(n.N) + size_t(n.C) + 31) / 32 * 128 + size_t(per) * 128 + (size_t(per) + 1) * 4;
	if(fixed > FWD_SMEM) return p;
	p.perBlock = per;
	p.blocks = (n.N + per - 1) / per;
	p.cached = int((FWD_SMEM - fixed) / 8);
	p.kernel = forwardKernel(std::min(4, (per + FWD_WARPS - 1) / FWD_WARPS));
	return p;
}

/* A stream that is being captured (or cannot tell) takes the launches whose
 * blocks never wait for one another: two graphs may run at once, and nothing
 * then orders their launches (DeviceTurn). */
static bool
capturing(cudaStream_t st)
{
	cudaStreamCaptureStatus status = cudaStreamCaptureStatusNone;
	if(cudaStreamIsCapturing(st, &status) != cudaSuccess) {
		(void) cudaGetLastError();
		return true;
	}
	return status != cudaStreamCaptureStatusNone;
}

static int
currentDevice()
{
	int dev = 0;
	NEMO_CUDA(cudaGetDevice(&dev));
	return dev;
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
 * counts); the adjoint's synapses (buckets, part totals, entries) and sums or, step by
 * step, the recurrent weights in out-synapse order; the grid barrier. Made
 * from the buffer's start rounded up to 128 bytes (the size has the slack). */
struct LifWork {
	float *v, *guNext, *uSeg, *guSeg;
	uint16_t* codes;
	uint32_t* cnt;
	float* wOut;        /* shares the entries' place */
	uint2 *bucket, *entries;
	uint32_t* total;
	float* sums;
	unsigned* barrier;
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
		const size_t P = size_t(lif::adjointParts(n.N, lif::rowWidth(n.B)));
		bucket = reinterpret_cast<uint2*>(take(P * n.N * 8));
		total = reinterpret_cast<uint32_t*>(take(P * 4));
		entries = reinterpret_cast<uint2*>(take((size_t(n.nnzRec) + 4 * P * n.N + lif::ADJ_SLACK) * 8));
		wOut = reinterpret_cast<float*>(entries);
		sums = reinterpret_cast<float*>(take(P * n.N * lif::rowWidth(n.B) * 4));
		barrier = reinterpret_cast<unsigned*>(take(8));
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
		const LifWork k(n, work);
		float* v = k.v;
		NEMO_CUDA(cudaMemsetAsync(counts, 0, size_t(n.B) * (n.T / n.binSteps) * 4, st));
		const int g = lif::grid(n.N);
		const lif::ForwardPlan plan = relaxed || lif::capturing(st) ? lif::ForwardPlan() : lif::planForward(n);
		if(plan.blocks) {
			NEMO_CUDA(cudaMemsetAsync(k.barrier, 0, 8, st));
			lif::Forward f = {w, in_bits, s_bits, v_ckpt, counts, plan.perBlock, plan.cached, k.barrier};
			std::unique_ptr<DeviceTurn> turn;
			if(plan.blocks > 1) turn.reset(new DeviceTurn(lif::currentDevice(), st));
			void* params[] = {&n, &f};
			NEMO_CUDA(cudaLaunchCooperativeKernel(plan.kernel, dim3(unsigned(plan.blocks)),
					dim3(unsigned(lif::FWD_THREADS)), params, lif::FWD_SMEM, st));
		}
		if(!plan.blocks) NEMO_CUDA(cudaMemsetAsync(v, 0, size_t(n.N) * 32 * 4, st));
		for(int t = 0; t < n.T && !plan.blocks; ++t) {
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
		const lif::AdjointPlan plan = relaxed || lif::capturing(st) ? lif::AdjointPlan() : lif::planAdjoint(n);
		const int tw = plan.tw;
		std::unique_ptr<DeviceTurn> turn;
		NEMO_CUDA(cudaMemsetAsync(k.barrier, 0, 8, st));
		lif::Adjoint adj = {};
		if(plan.parts) {
			lif::k_out_count<<<g, lif::THREADS, 0, st>>>(n, plan.parts, plan.partRows, k.bucket);
			lif::k_out_scan<<<plan.parts, 1024, 0, st>>>(n.N, k.bucket, k.total);
			lif::k_out_fill<<<g, lif::THREADS, 0, st>>>(n, plan.parts, plan.partRows, tw * 4, k.bucket, k.total, w, k.entries);
			adj.parts = plan.parts;
			adj.partRows = plan.partRows;
			adj.perGroup = plan.perGroup;
			adj.sums = k.sums;
			adj.bucket = k.bucket;
			adj.total = k.total;
			adj.entries = k.entries;
			adj.uSeg = k.uSeg;
			adj.guNext = k.guNext;
			adj.guSeg = k.guSeg;
			adj.dcounts = dcounts;
			adj.barrier = k.barrier;
			turn.reset(new DeviceTurn(lif::currentDevice(), st));
		} else if(n.nnzRec) {
			lif::k_gather_out<<<g, lif::THREADS, 0, st>>>(n, n.nnzRec, w, k.wOut);
		}
		const int segments = (n.T + n.K - 1) / n.K;
		const size_t units = size_t(n.N) + size_t(n.C);
		const int L = lif::partSteps(std::min(n.K, n.T));
		const unsigned gp = unsigned((n.N + lif::PART_WARPS - 1) / lif::PART_WARPS);
		const size_t smemP = size_t(lif::PART_WARPS) * (size_t(L) * 32 + 32) * 4;
		if(!relaxed) {
			lif::allowShared((const void*) lif::k_recompute, lif::PART_SMEM);
			lif::allowShared((const void*) lif::k_dw_events, lif::PART_SMEM);
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
					lif::k_recompute<<<gp, lif::PART_WARPS * 32, smemP, st>>>(n, tw, t0, t1, c0, L, w,
							k.codes + size_t(y) * units * L * 32, k.cnt + size_t(y) * units, y ? k.v : ckpt, k.v, k.uSeg);
				}
			}
			/* backwards through the segment */
			if(plan.parts) {
				adj.c0 = c0;
				adj.c1 = c1;
				void* params[] = {&n, &adj};
				NEMO_CUDA(cudaLaunchCooperativeKernel(lif::adjointKernel(tw), dim3(unsigned(plan.parts * plan.groups)),
						dim3(unsigned(lif::ADJ_THREADS)), params, lif::ADJ_SMEM, st));
				adj.barrierBase += unsigned(2 * (c1 - c0) - 1) * unsigned(plan.parts * plan.groups);
			}
			for(int t = c1 - 1; t >= c0 && !plan.parts; --t) {
				const bool last = t == n.T - 1;
				const float* next = t == c1 - 1 ? k.guNext : k.guSeg + size_t(t + 1 - c0) * NS;
				lif::k_back<<<g, lif::THREADS, 0, st>>>(n, t, k.wOut, k.uSeg, c0, next, k.guSeg, dcounts, last);
			}
			if(relaxed) {
				lif::k_dw_relaxed<<<g, lif::THREADS, 0, st>>>(n, c0, c1, k.guSeg, s_float, in_bits, dw);
			} else {
				for(int y = 0; y < Y; ++y) {
					const int t0 = c0 + y * L, t1 = std::min(c1, t0 + L);
					lif::k_dw_events<<<gp, lif::PART_WARPS * 32, smemP, st>>>(n, tw, t0, t1, c0, L, k.guSeg,
							k.codes + size_t(y) * units * L * 32, k.cnt + size_t(y) * units, k.barrier + 1, dw);
				}
			}
			NEMO_CUDA(cudaMemcpyAsync(k.guNext, k.guSeg, size_t(n.N) * tw * 4, cudaMemcpyDeviceToDevice, st));
		}
		NEMO_CUDA(cudaGetLastError());
	})
}

} // extern "C"
