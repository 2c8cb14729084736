// bptt.cu -- differentiable mode: a network of Izhikevich neurons with
// delayed synapses, run forward with checkpoints and differentiated by a
// hand-written backpropagation-through-time adjoint.
//
// Model (per trial b, neuron n, millisecond t; 4 Euler sub-steps per ms as
// in src/nemo/cpu/plugins/Izhikevich.cpp, with a reset after every sub-step
// so that the sub-step chain is differentiable):
//   I(t)  = sum over in-synapses (j, w, d) of w * S_j(t - d)  +  noise(t)
//   sub-step k = 0..3:
//     v1 = v + 1/4 (0.04 v^2 + 5 v + 140 - u + I)
//     u1 = u + 1/4 a (b v1 - u)
//     s  = H(v1 - 30)             (hard)   or  f(v1 - 30)  (smooth)
//     v  = v1 + s (c - v1);  u = u1 + s d;  S(t) += s
//   r(t) = alpha r(t-1) + S(t) for the R readout neurons, alpha = exp(-1/20)
//   loss = sum_t,b,n<R (r - target)^2 / (T R B)
// f(x) = 1/2 (1 + kx / (1 + k|x|)) is the fast sigmoid with slope k = 10,
// and g(x) = f'(x) = k / (2 (1 + k|x|)^2) is the surrogate derivative used
// for H in the backward pass.  Initial state v = -65, u = b v.
//
// Every kernel is a template over the state type Real (float or double):
// the caller's weights, parameters, noise, targets, loss and gradients are
// float32 either way; Real is the type of the neuron state, the stored
// trajectories and the adjoints.  Gradients of this model are sensitive to
// rounding (the spike upstroke amplifies a state perturbation many times
// over), so float32 state gives gradients within about 1e-2 of the exact
// ones, while float64 state reproduces a float64 evaluation.
//
// Layouts: input adjoints lambda_I and the neurons' total inputs I as
// [t][n][b]; noise and targets as PyTorch tensors [T][B][N] and [T][B][R].
// Spikes of the hard threshold are counts of at most 4 per ms: one word of 4
// bits per trial and group of up to 16 trials, [t][group][n].  Checkpoints of
// (v, u) every `ckpt` ms; the backward pass replays each segment from its
// checkpoint and the stored inputs (no synapse is read again) and keeps the
// segment's per-ms start states.
//
// The forward pass and the adjoint each run as one cooperative launch over
// all milliseconds.  A launch per ms (as this file used to have) was bound by
// what it re-read: every (neuron, trial) thread walked its synapses' indices,
// delays and weights in L2 and one 8-byte spike each, 104 us of kernel time
// per gradient ms at 4096 x 200 x 16 trials.  In the loops a CTA owns a run of
// neurons, holds their synapses and state in shared memory, and a barrier
// between the CTAs of a trial group ends each ms.  Groups never exchange
// anything: trials are independent.
#include <cuda_runtime.h>
#include <stdint.h>

#include <algorithm>
#include <cmath>
#include <type_traits>
#include <vector>

#include "../../include/nemo_b200.h"
#include "bptt.hpp"
#include "common.hpp"

namespace nemo_b200 {

#define BP_CUDA(call)                                                              \
	do {                                                                           \
		cudaError_t err_ = (call);                                                 \
		if(err_ != cudaSuccess) {                                                  \
			NB_THROW(NEMO_CUDA_ERROR, "CUDA error %s at %s:%d", cudaGetErrorString(err_), __FILE__, __LINE__); \
		}                                                                          \
	} while(0)

template<typename Real>
__device__ __forceinline__ Real spike_fn(Real x, int smooth)
{
	const Real k = Real(10);
	if(smooth) return Real(0.5) * (Real(1) + k * x / (Real(1) + k * fabs(x)));
	return x >= Real(0) ? Real(1) : Real(0);
}

template<typename Real>
__device__ __forceinline__ Real spike_grad(Real x)
{
	const Real q = Real(1) + Real(10) * fabs(x);
	return Real(0.5) * Real(10) / (q * q);
}

constexpr int BPTT_GROUP = 16;     // trials per group: one 64-bit spike word
constexpr int LOOP_THREADS = 1024; // a warp (or a part of one) gathers a neuron, so as many warps as fit
constexpr int FWD_MIN_CELLS = 16;  // neurons per CTA at least
constexpr int BWD_MIN_CELLS = 16;
constexpr int MASK_HEADER = 16;    // bytes before the masks of a slice
constexpr int SYNC_STRIDE = 32;    // barrier counters 128 bytes apart

// words of BpttState::sync: flags, then a counter per CTA group of the
// forward and of the adjoint loop
enum { SYNC_NONFINITE = 0, SYNC_ERROR = 1 };
__host__ __device__ inline int sync_counter(int group, bool backward, int maxGroups)
{
	return SYNC_STRIDE * (1 + group + (backward ? maxGroups : 0));
}

// Waits give up after this many polls (eleven seconds at 171 ns a poll; a
// millisecond of the loop takes microseconds)
constexpr unsigned LOOP_POLL_LIMIT = 1u << 26;

// One launch of a loop: CTAs and neurons per trial group, the first group,
// and the barrier counters' value when it starts.
struct LoopArgs {
	int ctas, cells, g0, maxGroups;
	unsigned base;
};

// Barrier between the CTAs of one trial group, in two halves so that work
// that needs nothing from the other CTAs can run between them.  The counter
// only grows during a pass; the kernel that ends the pass sets it back to 0.
__device__ __forceinline__ void loop_arrive(unsigned* counter)
{
	__syncthreads();
	if(threadIdx.x == 0) asm volatile("red.release.gpu.global.add.u32 [%0], 1;" :: "l"(counter) : "memory");
}

__device__ __forceinline__ unsigned load_acquire(const unsigned* p)
{
	unsigned v;
	asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
	return v;
}

__device__ __forceinline__ bool loop_wait(unsigned* counter, unsigned target, unsigned* sync, unsigned* hostError)
{
	__shared__ int sOk;
	if(threadIdx.x == 0) {
		int ok = 1;
		for(unsigned polls = 1; load_acquire(counter) < target; ++polls) {
			if(polls > LOOP_POLL_LIMIT || ((polls & 1023u) == 0 && load_acquire(sync + SYNC_ERROR))) {
				atomicExch(sync + SYNC_ERROR, 1u);
				*(volatile unsigned*) hostError = 1u;
				ok = 0;
				break;
			}
		}
		sOk = ok;
	}
	__syncthreads();
	return sOk != 0;
}

// spike words of 1 << wordLog bytes
__device__ __forceinline__ unsigned long long load_word(const unsigned char* words, size_t i, int wordLog)
{
	switch(wordLog) {
		case 0: return words[i];
		case 1: return reinterpret_cast<const uint16_t*>(words)[i];
		case 2: return reinterpret_cast<const uint32_t*>(words)[i];
		default: return reinterpret_cast<const unsigned long long*>(words)[i];
	}
}

__device__ __forceinline__ void store_word(unsigned char* words, size_t i, int wordLog, unsigned long long v)
{
	switch(wordLog) {
		case 0: words[i] = (unsigned char) v; break;
		case 1: reinterpret_cast<uint16_t*>(words)[i] = (uint16_t) v; break;
		case 2: reinterpret_cast<uint32_t*>(words)[i] = (uint32_t) v; break;
		default: reinterpret_cast<unsigned long long*>(words)[i] = v; break;
	}
}

// A neuron's input is summed in four interleaved partial sums: entry k of its
// list of len goes to sum k % 4, the len % 4 last ones to sum 0, and the sums
// combine as (0 + 2) + (1 + 3).  Every forward gather keeps that order, so an
// input does not depend on how the list is spread over lanes (with float32
// state a different order would soon fire different spikes).

// Inputs of one neuron from the spike masks of the last D.ring ms, by one
// warp.  Every lane loads the mask of one synapse's source (a bit per trial);
// at the rates of these networks the mask of 16 trials is nonzero for one
// synapse in seven.  Those are compacted into four short lists, one per
// partial sum, and added: lanes are (sub, trial), and sub-team `sub` of 2 or 4
// takes the lists sub (and sub + 2).
// The window of masks, the lists and the compacted entries sit in shared
// memory when they fit (MODE 2): random 8-byte words from L2 ran at the
// scattered-load rate (819200 a ms at 4096 x 200: 11.4 us a ms), and adding
// the nonzero entries of a round one by one by ballot was bound by
// instruction issue (45k warp instructions per SM and ms, 12 us).
constexpr int FWD_ROUNDS = 8;                        // mask loads in flight per lane
constexpr int FWD_CHUNK = 32 * FWD_ROUNDS;           // synapses per pass over the lists
constexpr int FWD_LIST = FWD_CHUNK / 4 + 4;          // entries of a compacted list (list 0 takes up to 3 more)
constexpr int FWD_LISTS_BYTES = LOOP_THREADS / 32 * 4 * FWD_LIST * 4;

// a synapse of the forward lists in shared memory (MODE 2: at most 65536
// neurons and, as the trials' memory is bounded, fewer ms): source | delay << 16
__device__ __forceinline__ int2 unpack_synapse(int2 e) { return e; }
__device__ __forceinline__ int2 unpack_synapse(unsigned e) { return make_int2((int) (e & 0xffffu), (int) (e >> 16)); }

__device__ __forceinline__ unsigned load_mask(const BpttDev& D, const unsigned char* slice, int src)
{
	slice += MASK_HEADER;
	return D.lanes > 8 ? reinterpret_cast<const uint16_t*>(slice)[src] : slice[src];
}

// the general form: counts from the spike words, every synapse added -- for
// neurons that fired more than once in some ms of the window, and for
// weights that are not finite (inf x 0 is NaN).  Each lane loads the word and
// the weight of one synapse, 32 at a time; the lanes (sub, trial) then take the
// partial sums sub (and sub + 2) from them by shuffles, in order.  (A word at a
// time, every lane loading the same, was bound by one L2 round trip per
// synapse: a gradient of 30000 x 20, 100 ms, one trial 6.6 against 2.3 ms, of 2000 x 100,
// 200 ms, 16 trials 10.6 against 3.9.  Out of line, and called per neuron: the usual path
// beside it lost 1.5% to a second loop over the neurons.)
template<typename Real, typename Entry, typename Weight>
__device__ __noinline__ Real gather_counts(const BpttDev& D, const unsigned char* words, int g, const Entry* list,
		const Weight* w, int len, int t)
{
	const unsigned FULL = 0xffffffffu;
	const int lane = threadIdx.x & 31, b = lane & (D.lanes - 1), main = len & ~3;
	const int sub = (lane >> (31 - __clz(D.lanes))) & 3, subs = D.lanes > 8 ? 2 : 4;
	Real s0 = Real(0), s1 = Real(0);
	for(int k0 = 0; k0 < len; k0 += 32) {
		unsigned long long word = 0;
		Real wk = Real(0);
		if(k0 + lane < len) {
			const int2 e = unpack_synapse(list[k0 + lane]);
			wk = (Real) w[k0 + lane];
			if(t >= e.y) word = load_word(words, ((size_t) (t - e.y) * D.groups + g) * D.N + e.x, D.wordLog);
		}
		auto term = [&](int i, Real sum) {
			const Real x = (Real) ((int) (__shfl_sync(FULL, word, i) >> (4 * b)) & 15);
			return fma(__shfl_sync(FULL, wk, i), x, sum);
		};
		const int n = min(32, len - k0), quads = max(0, min(n, main - k0));
		for(int i = 0; i < quads; i += 4) {
			s0 = term(i + sub, s0);
			if(subs == 2) s1 = term(i + sub + 2, s1);
		}
		for(int i = quads; i < n; ++i) {
			const Real x = term(i, s0);
			if(sub == 0) s0 = x;
		}
	}
	if(subs == 2) s0 += s1;
	else s0 += __shfl_xor_sync(FULL, s0, 2 * D.lanes);
	return s0 + __shfl_xor_sync(FULL, s0, D.lanes);
}

// masks: all slices (global memory); window, slot: the last D.ring of them by
// ms % D.ring and t % D.ring (MODE 2).  (Reading the newest slice from global
// memory instead of waiting for its copy: 8.3 against 7.4 us a ms at
// 4096 x 200 x 16.)  lists: this warp's four lists of FWD_LIST entries (shared
// memory)
template<typename Real, int MODE, typename Entry, typename Weight>
__device__ __forceinline__ Real gather_masks(const BpttDev& D, const unsigned char* masks, const unsigned char* window, int slot,
		int g, const Entry* list, const Weight* w, int len, int t, unsigned* lists)
{
	const unsigned FULL = 0xffffffffu;
	const int lane = threadIdx.x & 31, laneLog = 31 - __clz(D.lanes);
	const int sub = lane >> laneLog, b = lane & (D.lanes - 1), subs = D.lanes > 8 ? 2 : 4;
	const int main = len & ~3;
	const unsigned mineBits = 0x11111111u << (lane & 3), before = mineBits & ((1u << lane) - 1u);
	auto mask_of = [&](int k) -> unsigned {
		const int2 e = unpack_synapse(list[k]);
		if(t < e.y) return 0u;
		if(MODE == 2) {
			int at = slot - e.y;
			at += at < 0 ? D.ring : 0;
			return load_mask(D, window + (unsigned) (at * D.maskStride), e.x);
		}
		const int at = (t - e.y) * D.groups + g;
		return load_mask(D, masks + (size_t) (unsigned) at * D.maskStride, e.x);
	};
	Real s0 = Real(0), s1 = Real(0);
	for(int base = 0; base < len; base += FWD_CHUNK) {
		unsigned m[FWD_ROUNDS];
#pragma unroll
		for(int q = 0; q < FWD_ROUNDS; ++q) {
			const int k = base + 32 * q + lane;
			m[q] = 0u;
			if(base + 32 * q < len && k < len) m[q] = mask_of(k);
		}
		// lane l appends to list l % 4 (the entries k % 4 = l % 4), the last
		// len % 4 entries to list 0
		int count = 0;
#pragma unroll
		for(int q = 0; q < FWD_ROUNDS; ++q) {
			const int k0 = base + 32 * q;
			if(k0 >= len) break;
			const unsigned entry = (unsigned) (32 * q + lane) << 16 | m[q];
			const unsigned live = __ballot_sync(FULL, m[q] != 0);
			if(k0 + 32 <= main) {
				if(m[q]) lists[(lane & 3) * FWD_LIST + count + __popc(live & before)] = entry;
				count += __popc(live & mineBits);
			} else {
				const unsigned tail = main > k0 ? FULL << (main - k0) : FULL;
				const unsigned to0 = live & (0x11111111u | tail), mine = live & mineBits & ~tail, below = (1u << lane) - 1u;
				const int count0 = __shfl_sync(FULL, count, 0);
				if(to0 >> lane & 1u) lists[count0 + __popc(to0 & below)] = entry;
				else if(m[q]) lists[(lane & 3) * FWD_LIST + count + __popc(mine & below)] = entry;
				count += __popc((lane & 3) ? mine : to0);
			}
		}
		__syncwarp();
		const int n0 = __shfl_sync(FULL, count, sub & 3), n1 = __shfl_sync(FULL, count, (sub + 2) & 3);
		const Weight* wb = w + base;
		if(sub < subs) {
			const unsigned* l0 = lists + sub * FWD_LIST;
#pragma unroll 4
			for(int i = 0; i < n0; ++i) {
				const unsigned e = l0[i];
				const Real wk = (Real) wb[e >> 16];
				if((e >> b) & 1u) s0 += wk;
			}
			if(subs == 2) {
				const unsigned* l1 = lists + (sub + 2) * FWD_LIST;
#pragma unroll 4
				for(int i = 0; i < n1; ++i) {
					const unsigned e = l1[i];
					const Real wk = (Real) wb[e >> 16];
					if((e >> b) & 1u) s1 += wk;
				}
			}
		}
		__syncwarp();
	}
	if(subs == 2) s0 += s1;
	else s0 += __shfl_xor_sync(FULL, s0, 2 * D.lanes);
	return s0 + __shfl_xor_sync(FULL, s0, D.lanes);
}

// Sum of w * S[t - delay][n][b] over a list (the smooth threshold), 0 before
// ms 0, by the 4 * lanes (at most 32) threads of a team: SUBS = 4 or 2
// sub-teams of `lanes` trials take the entries k % 4 = sub (and sub + 2), BATCH
// of them in flight per lane.  at: S + b; every lane of the team returns
// the sum.
template<typename Real, int SUBS, int BATCH, typename Entry, typename Weight>
__device__ __forceinline__ Real gather_dense(const BpttDev& D, const Real* at, bool valid, const Entry* sd, const Weight* w,
		int len, int t, int sub)
{
	constexpr int NS = 4 / SUBS;
	const size_t NB = (size_t) D.N * D.B;
	const int main = len & ~3;
	Real sum[NS];
#pragma unroll
	for(int j = 0; j < NS; ++j) sum[j] = Real(0);
	auto term = [&](int k, Real& wk, Real& x) {
		const int2 e = unpack_synapse(sd[k]);
		wk = (Real) w[k];
		x = Real(0);
		if(valid && t >= e.y) x = __ldcg(at + ((size_t) (t - e.y) * NB + (size_t) e.x * D.B));
	};
	for(int k0 = 0; k0 < main; k0 += 4 * (BATCH / NS)) {
		Real wk[BATCH], x[BATCH];
#pragma unroll
		for(int q = 0; q < BATCH; ++q) {
			const int k = k0 + 4 * (q / NS) + sub + SUBS * (q % NS);
			wk[q] = x[q] = Real(0);
			if(k < main) term(k, wk[q], x[q]);
		}
#pragma unroll
		for(int q = 0; q < BATCH; ++q) sum[q % NS] = fma(wk[q], x[q], sum[q % NS]);
	}
	if(sub == 0) {
		for(int k = main; k < len; ++k) {
			Real wk, x;
			term(k, wk, x);
			sum[0] = fma(wk, x, sum[0]);
		}
	}
	Real s = sum[0];
	if(NS == 2) s += sum[NS - 1];
	if(SUBS == 4) s += __shfl_xor_sync(0xffffffffu, s, 2 * D.lanes);
	return s + __shfl_xor_sync(0xffffffffu, s, D.lanes);
}

// V trials of an adjoint row: one 16-byte load where a row's trials allow it
// (V = 2 float64 or 4 float32)
template<typename Real, int V> struct Trials { Real x[V]; };

template<typename Real, int V>
__device__ __forceinline__ Trials<Real, V> load_trials(const Real* p)
{
	Trials<Real, V> r;
	if constexpr(V == 1) {
		r.x[0] = __ldcg(p);
	} else if constexpr(sizeof(Real) == 8) {
		const double2 v = __ldcg(reinterpret_cast<const double2*>(p));
		r.x[0] = v.x;
		r.x[1] = v.y;
	} else {
		const float4 v = __ldcg(reinterpret_cast<const float4*>(p));
		r.x[0] = v.x;
		r.x[1] = v.y;
		r.x[2] = v.z;
		r.x[3] = v.w;
	}
	return r;
}

// Sum of w * lambda_I[t + delay][n][b .. b + V) over a list of element offsets
// (delay x N x B + n x B), by a team of SUBS = 4 or 2 sub-teams that take its
// groups of four entries in turn: one 16-byte shared-memory read gives a lane
// four offsets, and eight 16-byte loads are in flight per lane.  Offsets at or
// beyond `limit` lie after the last ms and count 0 (inside: there are none).
// The lists start on 16 bytes.  now: lambda_I of ms t, at b.
template<typename Real, int V, int SUBS>
__device__ __forceinline__ Trials<Real, V> gather_adjoint(const Real* now, bool valid, bool inside, unsigned limit,
		const unsigned* off, const Real* w, int len, int sub, int lv)
{
	Trials<Real, V> sum;
#pragma unroll
	for(int j = 0; j < V; ++j) sum.x[j] = Real(0);
	const int groups = len >> 2;
	auto add = [&](const Trials<Real, V>& x, Real wk) {
#pragma unroll
		for(int j = 0; j < V; ++j) sum.x[j] = fma(wk, x.x[j], sum.x[j]);
	};
	auto load = [&](unsigned o) -> Trials<Real, V> {
		if(inside || o < limit) return load_trials<Real, V>(now + o);
		Trials<Real, V> x;
#pragma unroll
		for(int j = 0; j < V; ++j) x.x[j] = Real(0);
		return x;
	};
	if(valid) {
		// the last len % 4 entries, one or two a sub-team
		Trials<Real, V> rest[4 / SUBS];
#pragma unroll
		for(int h = 0; h < 4 / SUBS; ++h) {
			const int k = 4 * groups + sub + h * SUBS;
			if(k < len) rest[h] = load(off[k]);
		}
		int g = sub;
		if(inside) {
			for(; g + SUBS < groups; g += 2 * SUBS) {
				const uint4 a = *reinterpret_cast<const uint4*>(off + 4 * g), b = *reinterpret_cast<const uint4*>(off + 4 * (g + SUBS));
				Trials<Real, V> x[8];
				x[0] = load_trials<Real, V>(now + a.x);
				x[1] = load_trials<Real, V>(now + a.y);
				x[2] = load_trials<Real, V>(now + a.z);
				x[3] = load_trials<Real, V>(now + a.w);
				x[4] = load_trials<Real, V>(now + b.x);
				x[5] = load_trials<Real, V>(now + b.y);
				x[6] = load_trials<Real, V>(now + b.z);
				x[7] = load_trials<Real, V>(now + b.w);
				const Real* wa = w + 4 * g;
				const Real* wb = w + 4 * (g + SUBS);
#pragma unroll
				for(int q = 0; q < 4; ++q) add(x[q], wa[q]);
#pragma unroll
				for(int q = 0; q < 4; ++q) add(x[4 + q], wb[q]);
			}
		}
		for(; g < groups; g += SUBS) {
			const uint4 a = *reinterpret_cast<const uint4*>(off + 4 * g);
			const Trials<Real, V> x0 = load(a.x), x1 = load(a.y), x2 = load(a.z), x3 = load(a.w);
			add(x0, w[4 * g]);
			add(x1, w[4 * g + 1]);
			add(x2, w[4 * g + 2]);
			add(x3, w[4 * g + 3]);
		}
#pragma unroll
		for(int h = 0; h < 4 / SUBS; ++h) {
			const int k = 4 * groups + sub + h * SUBS;
			if(k < len) add(rest[h], w[k]);
		}
	}
#pragma unroll
	for(int j = 0; j < V; ++j) {
		if(SUBS == 4) sum.x[j] += __shfl_xor_sync(0xffffffffu, sum.x[j], 2 * lv);
		sum.x[j] += __shfl_xor_sync(0xffffffffu, sum.x[j], lv);
	}
	return sum;
}

// the same from lists in global memory, with offsets of any size, one entry
// per sub-team at a time
template<typename Real, int V, int SUBS>
__device__ __forceinline__ Trials<Real, V> gather_adjoint(const Real* now, bool valid, unsigned long long limit,
		const unsigned long long* off, const float* w, int len, int sub, int lv)
{
	Trials<Real, V> sum;
#pragma unroll
	for(int j = 0; j < V; ++j) sum.x[j] = Real(0);
	if(valid) {
#pragma unroll 4
		for(int k = sub; k < len; k += SUBS) {
			const unsigned long long o = off[k];
			Trials<Real, V> x;
#pragma unroll
			for(int j = 0; j < V; ++j) x.x[j] = Real(0);
			if(o < limit) x = load_trials<Real, V>(now + o);
			const Real wk = (Real) w[k];
#pragma unroll
			for(int j = 0; j < V; ++j) sum.x[j] = fma(wk, x.x[j], sum.x[j]);
		}
	}
#pragma unroll
	for(int j = 0; j < V; ++j) {
		if(SUBS == 4) sum.x[j] += __shfl_xor_sync(0xffffffffu, sum.x[j], 2 * lv);
		sum.x[j] += __shfl_xor_sync(0xffffffffu, sum.x[j], lv);
	}
	return sum;
}

template<int BYTES>
__device__ __forceinline__ void copy_async(void* to, const void* from)
{
	asm volatile("cp.async.ca.shared.global [%0], [%1], %2;" :: "r"((unsigned) __cvta_generic_to_shared(to)), "l"(from),
			"n"(BYTES) : "memory");
}

// one Euler sub-step and its reset; returns s
template<typename Real>
__device__ __forceinline__ Real substep(Real& v, Real& u, Real& v1, Real I, Real a, Real b, Real c, Real d, int smooth)
{
	v1 = v + Real(0.25) * (Real(0.04) * v * v + Real(5) * v + Real(140) - u + I);
	const Real u1 = u + Real(0.25) * a * (b * v1 - u);
	const Real s = spike_fn(v1 - Real(30), smooth);
	v = v1 + s * (c - v1);
	u = u1 + s * d;
	return s;
}

// the four sub-steps of one ms; returns S(t)
template<typename Real>
__device__ __forceinline__ Real substeps(Real& v, Real& u, Real I, Real a, Real b, Real c, Real d, int smooth)
{
	Real St = Real(0), v1;
#pragma unroll
	for(int k = 0; k < 4; ++k) St += substep(v, u, v1, I, a, b, c, d, smooth);
	return St;
}

// weights in list order, for the loops whose lists stay in global memory
__global__ void bptt_list_weights_kernel(size_t M, const int* syn, const float* W, float* out)
{
	for(size_t e = (size_t) blockIdx.x * blockDim.x + threadIdx.x; e < M; e += (size_t) gridDim.x * blockDim.x) {
		out[e] = W[syn[e]];
	}
}

// Forward pass: all T ms.  Per ms a CTA gathers its neurons' inputs (a warp
// per neuron from spike words; with the smooth threshold teams of lanes from
// the stored S), then each thread advances one (neuron, trial).  What a
// thread needs from elsewhere (parameters once, the next ms's noise) is
// loaded ahead of the barrier wait.
// MODE 0: everything in global memory; 1: lists and items in shared memory;
// 2: and the window of spike masks, to which each ms adds the slice that the
// CTAs of the group have just written.
template<typename Real, bool SMOOTH, int MODE>
__global__ void __launch_bounds__(LOOP_THREADS, 1)
bptt_forward_loop(const BpttDev D, const BpttState<Real> X, const BpttParams P, const LoopArgs L)
{
	extern __shared__ __align__(16) unsigned char raw[];
	__shared__ int sAll;
	const int gi = blockIdx.x / L.ctas, g = L.g0 + gi;
	const int n0 = min(D.N, (int) (blockIdx.x % L.ctas) * L.cells), n1 = min(D.N, n0 + L.cells), nc = n1 - n0;
	const int lanes = D.lanes, laneLog = 31 - __clz(lanes);
	const int b0 = g * BPTT_GROUP, nb = min(BPTT_GROUP, D.B - b0);
	const size_t NB = (size_t) D.N * D.B;
	const int first = D.inStart[n0], last = D.inStart[n1];
	// shared memory: items, then (MODE >= 1) weights and synapses, then (MODE
	// 2) the mask window and the warps' compacted lists
	const size_t cap = (size_t) L.cells * lanes;
	using Entry = typename std::conditional<MODE == 2, unsigned, int2>::type;
	using Weight = typename std::conditional<MODE == 0, float, Real>::type;
	Real* in = MODE ? reinterpret_cast<Real*>(raw) : X.scratch + (size_t) blockIdx.x * 5 * cap;
	Real* v = in + cap;
	Real* u = v + cap;
	Real* r = u + cap;
	Real* lossPart = r + cap;
	const Entry* list;
	const Weight* weight;
	const int2* cells = nullptr;
	unsigned char* window = nullptr;
	__shared__ unsigned sLists[LOOP_THREADS / 32 * 4 * FWD_LIST];
	unsigned* lists = sLists + (threadIdx.x >> 5) * 4 * FWD_LIST;
	if constexpr(MODE == 0) {
		list = D.inSd + first;
		weight = X.listW + first;
	} else {
		Real* sw = lossPart + cap;
		Entry* se = reinterpret_cast<Entry*>(raw + ((size_t) (reinterpret_cast<unsigned char*>(sw + (last - first)) - raw) + 7) / 8 * 8);
		for(int e = first + threadIdx.x; e < last; e += LOOP_THREADS) {
			sw[e - first] = (Real) P.W[D.inSyn[e]];
			const int2 sd = D.inSd[e];
			if constexpr(MODE == 2) se[e - first] = (unsigned) sd.x | (unsigned) sd.y << 16;
			else se[e - first] = sd;
		}
		list = se;
		weight = sw;
		// each neuron's place in the lists: read every ms, and L1 does not
		// outlast a barrier
		int2* sc = reinterpret_cast<int2*>(raw + ((size_t) (reinterpret_cast<unsigned char*>(se + (last - first)) - raw) + 7) / 8 * 8);
		for(int cl = threadIdx.x; cl < nc; cl += LOOP_THREADS) {
			const int beg = D.inStart[n0 + cl];
			sc[cl] = make_int2(beg - first, D.inStart[n0 + cl + 1] - beg);
		}
		cells = sc;
		window = raw + ((size_t) (reinterpret_cast<unsigned char*>(sc + nc) - raw) + 15) / 16 * 16;
	}
	auto place = [&](int cl) -> int2 {
		if(MODE) return cells[cl];
		const int beg = D.inStart[n0 + cl];
		return make_int2(beg - first, D.inStart[n0 + cl + 1] - beg);
	};
	unsigned* counter = X.sync + sync_counter(gi, false, L.maxGroups);
	const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;

	if(tid == 0) sAll = 0;
	int lastMulti = -D.ring - 1;  // the last ms in which a neuron of the group fired more than once
	__syncthreads();
	bool odd = false;
	for(int k = tid; k < last - first; k += blockDim.x) odd |= !isfinite(weight[k]);
	if(odd) sAll = 1;
	const int items = nc << laneLog;
	for(int i = tid; i < items; i += blockDim.x) {
		v[i] = Real(-65);
		u[i] = (Real) P.b[n0 + (i >> laneLog)] * Real(-65);
		r[i] = Real(0);
		lossPart[i] = Real(0);
	}
	// this thread's first item: its parameters, and its noise one ms ahead
	const int myN = n0 + (tid >> laneLog), myB = b0 + (tid & (lanes - 1));
	const bool mine = tid < items && (tid & (lanes - 1)) < nb;
	float pa = 0, pb = 0, pc = 0, pd = 0, noise = 0, goal = 0;
	auto ahead = [&](int t) {
		noise = P.noise[((size_t) t * D.B + myB) * D.N + myN];
		if(myN < D.R) goal = P.target[((size_t) t * D.B + myB) * D.R + myN];
	};
	if(mine) {
		pa = P.a[myN];
		pb = P.b[myN];
		pc = P.c[myN];
		pd = P.d[myN];
		ahead(0);
	}
	__syncthreads();
	const bool all = sAll != 0;

	for(int t = 0; t < D.T; ++t) {
		if(!SMOOTH) {
			const int slot = t % D.ring;
			if(t) {
				const unsigned char* slice = X.masks + ((size_t) (t - 1) * D.groups + g) * D.maskStride;
				const unsigned more = __ldcg(reinterpret_cast<const unsigned*>(slice));
				if(MODE == 2) {
					uint4* to = reinterpret_cast<uint4*>(window + (size_t) (slot ? slot - 1 : D.ring - 1) * D.maskStride);
					const uint4* from = reinterpret_cast<const uint4*>(slice);
					for(int k = tid; k < D.maskStride / 16; k += LOOP_THREADS) to[k] = __ldcg(from + k);
					__syncthreads();
				}
				if(more) lastMulti = t - 1;
			}
			const bool counts = all || t - lastMulti <= D.ring;
			for(int cl = warp; cl < nc; cl += LOOP_THREADS / 32) {
				const int2 at = place(cl);
				const Real s = counts ? gather_counts<Real>(D, X.words, g, list + at.x, weight + at.x, at.y, t)
						: gather_masks<Real, MODE>(D, X.masks, window, slot, g, list + at.x, weight + at.x, at.y, t, lists);
				if(lane < lanes) in[(cl << laneLog) + lane] = s;
			}
		} else {
			const int team = min(32, 4 * lanes), sub = (lane & (team - 1)) >> laneLog, b = lane & (lanes - 1);
			const int perWarp = 32 / team, cl0 = warp * perWarp + lane / team;
			for(int cw = warp * perWarp, cl = cl0; cw < nc; cw += LOOP_THREADS / team, cl += LOOP_THREADS / team) {
				const bool cell = cl < nc;
				const int2 p = place(cell ? cl : 0);
				const int beg = p.x, len = cell ? p.y : 0;
				const bool valid = cell && b < nb;
				const Real* at = X.S + b0 + b;
				const Real s = lanes == BPTT_GROUP ? gather_dense<Real, 2, 8>(D, at, valid, list + beg, weight + beg, len, t, sub)
						: gather_dense<Real, 4, 8>(D, at, valid, list + beg, weight + beg, len, t, sub);
				if(cell && sub == 0) in[(cl << laneLog) + b] = s;
			}
		}
		__syncthreads();
		for(int i0 = 0; i0 < items; i0 += LOOP_THREADS) {
			const int i = i0 + tid, bl = i & (lanes - 1), n = n0 + (i >> laneLog), b = b0 + bl;
			const bool act = i < items && bl < nb;
			int count = 0;
			if(act) {
				if(i0) {
					pa = P.a[n];
					pb = P.b[n];
					pc = P.c[n];
					pd = P.d[n];
					noise = P.noise[((size_t) t * D.B + b) * D.N + n];
					if(n < D.R) goal = P.target[((size_t) t * D.B + b) * D.R + n];
				}
				const size_t at = (size_t) n * D.B + b;
				Real vi = v[i], ui = u[i];
				if(t % D.ckpt == 0) {
					const size_t k = (size_t) (t / D.ckpt) * NB + at;
					X.ckV[k] = vi;
					X.ckU[k] = ui;
				}
				const Real I = in[i] + (Real) noise;
				X.I[(size_t) t * NB + at] = I;
				const Real St = substeps(vi, ui, I, (Real) pa, (Real) pb, (Real) pc, (Real) pd, D.smooth);
				v[i] = vi;
				u[i] = ui;
				if(SMOOTH) X.S[(size_t) t * NB + at] = St;
				else count = (int) St;
				if(n < D.R) {
					const Real ri = X.alpha * r[i] + St;
					r[i] = ri;
					X.rHist[((size_t) t * D.R + n) * D.B + b] = ri;
					const Real diff = ri - (Real) goal;
					lossPart[i] += diff * diff;
				}
			}
			if(!SMOOTH) {
				unsigned long long word = 0;
				if(__ballot_sync(0xffffffffu, count != 0)) {
					word = (unsigned long long) count << (4 * bl);
					for(int o = 1; o < lanes; o <<= 1) word |= __shfl_xor_sync(0xffffffffu, word, o);
				}
				const unsigned fired = __ballot_sync(0xffffffffu, count != 0);
				const bool more = __any_sync(0xffffffffu, count > 1);
				if(act && bl == 0) {
					const size_t slice = (size_t) t * D.groups + g;
					store_word(X.words, slice * D.N + n, D.wordLog, word);
					unsigned char* masks = X.masks + slice * D.maskStride;
					const unsigned m = fired >> (lane & ~(lanes - 1)) & ((1u << lanes) - 1u);
					if(lanes > 8) reinterpret_cast<uint16_t*>(masks + MASK_HEADER)[n] = (uint16_t) m;
					else masks[MASK_HEADER + n] = (unsigned char) m;
					// one plain store a warp (every one is a 1): an atomic by each
					// neuron queued 100k of them at one address, 30 us a ms.  (A
					// warp that has fired twice has an item in lane 0.)
					if(more && lane == 0) *reinterpret_cast<volatile unsigned*>(masks) = 1u;
				}
			}
		}
		if(t + 1 < D.T) {
			if(items > LOOP_THREADS && mine) {
				pa = P.a[myN];
				pb = P.b[myN];
				pc = P.c[myN];
				pd = P.d[myN];
			}
			if(L.ctas == 1) {
				if(mine) ahead(t + 1);
				__syncthreads();
			} else {
				loop_arrive(counter);
				if(mine) ahead(t + 1);
				if(!loop_wait(counter, L.base + (unsigned) (t + 1) * L.ctas, X.sync, X.hostError)) return;
			}
		}
	}
	for(int i = tid; i < items; i += LOOP_THREADS) {
		const int bl = i & (lanes - 1), n = n0 + (i >> laneLog);
		if(bl < nb && n < D.R) X.lossPart[(size_t) n * D.B + b0 + bl] = lossPart[i];
	}
}

// deterministic final reduction of the loss (one block of 1024 threads); also
// empties the forward loop's barrier counters and flags.  A pass
// whose barrier gave up has no loss: NaN.
template<typename Real>
__global__ void bptt_loss_kernel(BpttDev D, BpttState<Real> X, float* loss, int maxGroups)
{
	__shared__ Real part[1024];
	for(int i = threadIdx.x; i < maxGroups; i += blockDim.x) X.sync[sync_counter(i, false, maxGroups)] = 0;
	if(threadIdx.x == 0) X.sync[SYNC_NONFINITE] = 0;
	if(X.masks) {
		for(int i = threadIdx.x; i < D.T * D.groups; i += blockDim.x) {
			*reinterpret_cast<unsigned*>(X.masks + (size_t) i * D.maskStride) = 0;
		}
	}
	Real s = Real(0);
	for(int i = threadIdx.x; i < D.R * D.B; i += blockDim.x) s += X.lossPart[i];
	part[threadIdx.x] = s;
	__syncthreads();
	for(int o = blockDim.x / 2; o > 0; o >>= 1) {
		if((int) threadIdx.x < o) part[threadIdx.x] += part[threadIdx.x + o];
		__syncthreads();
	}
	if(threadIdx.x == 0) *loss = X.sync[SYNC_ERROR] ? __int_as_float(0x7fffffff) : (float) (part[0] * X.lossScale);
}

// Adjoint: all T ms from the last to the first.  A segment starts with each
// thread replaying its (neuron, trial) from the checkpoint and the stored
// inputs (the arithmetic of the forward pass).  Per ms t a CTA gathers, for
// its neurons, the input adjoints of their targets -- 8 x 16 bytes per synapse
// and ms from L2 with 16 float64 trials, the bulk of the pass: 105 MB a ms at
// 4096 x 200 -- and each thread reverses the four sub-steps.  The gather is
// bound by the loads in flight: with 512 threads and 8-byte loads (32 KB in
// flight per SM) a ms took 28.5 us at that size; 1024 threads of eight
// 16-byte loads (V trials each) hold 128 KB.  Synapses of delay >= 2 need
// nothing that ms t + 1 wrote, so they are gathered between the two halves
// of the barrier; those of delay 1 follow it.
template<typename Real, int V, bool SM>
__global__ void __launch_bounds__(LOOP_THREADS, 1)
bptt_backward_loop(const BpttDev D, const BpttState<Real> X, const BpttParams P, const LoopArgs L)
{
	extern __shared__ __align__(16) unsigned char raw[];
	const int gi = blockIdx.x / L.ctas, g = L.g0 + gi;
	const int n0 = min(D.N, (int) (blockIdx.x % L.ctas) * L.cells), n1 = min(D.N, n0 + L.cells), nc = n1 - n0;
	const int lanes = D.lanes, laneLog = 31 - __clz(lanes);
	const int b0 = g * BPTT_GROUP, nb = min(BPTT_GROUP, D.B - b0);
	const size_t NB = (size_t) D.N * D.B;
	// shared memory (SM): items, weights, offsets; each neuron's two lists
	// (delays >= 2, delay 1) padded to a multiple of four entries
	const size_t cap = (size_t) L.cells * lanes;
	Real* sum = SM ? reinterpret_cast<Real*>(raw) : X.scratch + (size_t) blockIdx.x * 6 * cap;
	Real* lamV = sum + cap;
	Real* lamU = lamV + cap;
	Real* lamR = lamU + cap;
	Real* gA = lamR + cap;
	Real* gB = gA + cap;
	const int pad0 = D.outPad[n0];
	Real* sw = reinterpret_cast<Real*>(raw + ((11 * cap + 4 * (size_t) L.cells) * sizeof(Real) + 15) / 16 * 16);
	unsigned* so = reinterpret_cast<unsigned*>(sw + (D.outPad[n1] - pad0));
	// each neuron's two lists {start, entries}: read every ms, and L1 does not
	// outlast a barrier
	int4* sc = reinterpret_cast<int4*>(so + (D.outPad[n1] - pad0));
	// a, b, c, d of each neuron, and the items' inputs of the coming ms (start
	// state, input, trace, target), copied while the gathers run
	Real* param = gB + cap;
	Real* inV = param + 4 * L.cells;
	Real* inU = inV + cap;
	Real* inI = inU + cap;
	Real* inR = inI + cap;
	float* inT = reinterpret_cast<float*>(inR + cap);
	if(SM) {
		for(int cl = threadIdx.x; cl < nc; cl += LOOP_THREADS) {
			const int n = n0 + cl, start = D.outStart[n], mid = D.outMid[n], beg = D.outPad[n] - pad0;
			sc[cl] = make_int4(beg, mid - start, beg + (mid - start + 3) / 4 * 4, D.outStart[n + 1] - mid);
			param[4 * cl] = (Real) P.a[n];
			param[4 * cl + 1] = (Real) P.b[n];
			param[4 * cl + 2] = (Real) P.c[n];
			param[4 * cl + 3] = (Real) P.d[n];
		}
		for(int cl = threadIdx.x >> 5; cl < nc; cl += LOOP_THREADS / 32) {
			const int n = n0 + cl, early = D.outMid[n] - D.outStart[n], to = D.outPad[n] - pad0;
			const int gap = (early + 3) / 4 * 4 - early;
			for(int k = threadIdx.x & 31; k < D.outStart[n + 1] - D.outStart[n]; k += 32) {
				const int e = D.outStart[n] + k, at = to + k + (k < early ? 0 : gap);
				so[at] = (unsigned) D.outOff[e];
				sw[at] = (Real) P.W[D.outSyn[e]];
			}
		}
	}
	unsigned* counter = X.sync + sync_counter(gi, true, L.maxGroups);
	const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
	const int items = nc << laneLog;
	for(int i = tid; i < items; i += LOOP_THREADS) lamV[i] = lamU[i] = lamR[i] = gA[i] = gB[i] = Real(0);
	__syncthreads();

	// a team of four sub-teams (or two, of 16 lanes) per neuron, V trials a lane
	const int lv = max(1, lanes / V), team = min(32, 4 * lv), sub = (lane & (team - 1)) / lv, tb = (lane & (lv - 1)) * V;
	const int perWarp = 32 / team, cw0 = warp * perWarp, cl0 = cw0 + lane / team;
	auto gather_all = [&](int t, bool late) {
		const Real* now = X.lamI + (size_t) t * NB + b0 + tb;
		const unsigned long long limit = (unsigned long long) (D.T - t) * NB;
		const bool inside = t + D.ring < D.T;
		for(int cw = cw0, cl = cl0; cw < nc; cw += LOOP_THREADS / team, cl += LOOP_THREADS / team) {
			const bool cell = cl < nc;
			const bool valid = cell && tb < nb;
			Trials<Real, V> s;
			if(SM) {
				const int4 p = sc[cell ? cl : 0];
				const int beg = late ? p.z : p.x, len = !cell ? 0 : late ? p.w : p.y;
				const unsigned lim = (unsigned) min(limit, 0xffffffffull);
				if(V == 1 && lv == BPTT_GROUP) {  // a warp holds two sub-teams of 16 lanes
					s = gather_adjoint<Real, V, 2>(now, valid, inside, lim, so + beg, sw + beg, len, sub, lv);
				} else {
					s = gather_adjoint<Real, V, 4>(now, valid, inside, lim, so + beg, sw + beg, len, sub, lv);
				}
			} else {
				const int n = cell ? n0 + cl : n0;
				const int start = D.outStart[n], mid = D.outMid[n];
				const int len = !cell ? 0 : late ? D.outStart[n + 1] - mid : mid - start;
				const int beg = late ? mid : start;
				if(V == 1 && lv == BPTT_GROUP) {
					s = gather_adjoint<Real, V, 2>(now, valid, limit, D.outOff + beg, X.listW + beg, len, sub, lv);
				} else {
					s = gather_adjoint<Real, V, 4>(now, valid, limit, D.outOff + beg, X.listW + beg, len, sub, lv);
				}
			}
			if(cell && sub == 0) {
				Real* to = sum + (cl << laneLog) + tb;
#pragma unroll
				for(int j = 0; j < V; ++j) to[j] = late ? to[j] + s.x[j] : s.x[j];
			}
		}
	};

	unsigned arrived = L.base;
	bool odd = false;
	for(int t0 = (D.T - 1) / D.ckpt * D.ckpt; t0 >= 0; t0 -= D.ckpt) {
		const int t1 = min(D.T, t0 + D.ckpt);
		for(int i = tid; i < items; i += LOOP_THREADS) {
			const int bl = i & (lanes - 1), n = n0 + (i >> laneLog);
			if(bl >= nb) continue;
			const size_t at = (size_t) n * D.B + b0 + bl;
			const Real a = P.a[n], bb = P.b[n], c = P.c[n], d = P.d[n];
			const size_t k = (size_t) (t0 / D.ckpt) * NB + at;
			Real v = X.ckV[k], u = X.ckU[k];
			constexpr int AHEAD = 8;  // inputs loaded ahead of the sub-steps' chain
			for(int t = t0; t < t1; t += AHEAD) {
				Real I[AHEAD];
#pragma unroll
				for(int q = 0; q < AHEAD; ++q) I[q] = t + q < t1 ? __ldcs(X.I + (size_t) (t + q) * NB + at) : Real(0);
#pragma unroll
				for(int q = 0; q < AHEAD; ++q) {
					if(t + q >= t1) break;
					const size_t s = (size_t) (t + q - t0) * NB + at;
					X.segV[s] = v;
					X.segU[s] = u;
					substeps(v, u, I[q], a, bb, c, d, D.smooth);
				}
			}
		}
		__syncthreads();  // the copies below read what the replay stored
		for(int t = t1 - 1; t >= t0; --t) {
			if(SM) {
				// each thread copies the inputs of its own items
				for(int i = tid; i < items; i += LOOP_THREADS) {
					const int bl = i & (lanes - 1), n = n0 + (i >> laneLog), b = b0 + bl;
					if(bl >= nb) continue;
					const size_t at = (size_t) n * D.B + b, s = (size_t) (t - t0) * NB + at;
					copy_async<sizeof(Real)>(inV + i, X.segV + s);
					copy_async<sizeof(Real)>(inU + i, X.segU + s);
					copy_async<sizeof(Real)>(inI + i, X.I + (size_t) t * NB + at);
					if(n < D.R) {
						copy_async<sizeof(Real)>(inR + i, X.rHist + ((size_t) t * D.R + n) * D.B + b);
						copy_async<4>(inT + i, P.target + ((size_t) t * D.B + b) * D.R + n);
					}
				}
				asm volatile("cp.async.commit_group;" ::: "memory");
			}
			gather_all(t, false);
			if(t + 1 < D.T) {
				if(L.ctas == 1) __syncthreads();
				else if(!loop_wait(counter, arrived, X.sync, X.hostError)) return;
			}
			gather_all(t, true);
			if(SM) asm volatile("cp.async.wait_all;" ::: "memory");
			__syncthreads();
			for(int i = tid; i < items; i += LOOP_THREADS) {
				const int bl = i & (lanes - 1), n = n0 + (i >> laneLog), b = b0 + bl;
				if(bl >= nb) continue;
				const size_t at = (size_t) n * D.B + b;
				Real v, u, I, a, bb, c, d, r = Real(0), goal = Real(0);
				if(SM) {
					const Real* p = param + 4 * (i >> laneLog);
					v = inV[i];
					u = inU[i];
					I = inI[i];
					a = p[0];
					bb = p[1];
					c = p[2];
					d = p[3];
					if(n < D.R) {
						r = inR[i];
						goal = (Real) inT[i];
					}
				} else {
					const size_t s = (size_t) (t - t0) * NB + at;
					v = X.segV[s];
					u = X.segU[s];
					I = __ldcs(X.I + (size_t) t * NB + at);
					a = P.a[n];
					bb = P.b[n];
					c = P.c[n];
					d = P.d[n];
					if(n < D.R) {
						r = X.rHist[((size_t) t * D.R + n) * D.B + b];
						goal = (Real) P.target[((size_t) t * D.B + b) * D.R + n];
					}
				}
				// dL/dS(t): readout trace and the inputs S(t) drives d ms later
				Real lamS = Real(0);
				if(n < D.R) {
					const Real diff = r - goal;
					const Real lr = Real(2) * X.lossScale * diff + X.alpha * lamR[i];
					lamR[i] = lr;
					lamS = lr;
				}
				lamS += sum[i];

				// replay the sub-steps of ms t
				Real vk[4], uk[4], v1k[4];
				{
					Real x = v, y = u;
#pragma unroll
					for(int k = 0; k < 4; ++k) {
						vk[k] = x;
						uk[k] = y;
						substep(x, y, v1k[k], I, a, bb, c, d, D.smooth);
					}
				}

				// reverse through the sub-steps
				Real lv1 = lamV[i], lu = lamU[i];
				Real lamI = Real(0), ga = gA[i], gb = gB[i];
#pragma unroll
				for(int k = 3; k >= 0; --k) {
					const Real v0 = vk[k], u0 = uk[k], v1 = v1k[k], sp = spike_fn(v1 - Real(30), D.smooth);
					// v' = v1 + s (c - v1), u' = u1 + s d
					const Real lams = lamS + lv1 * (c - v1) + lu * d;
					Real lamV1 = lv1 * (Real(1) - sp) + lams * spike_grad(v1 - Real(30));
					const Real lamU1 = lu;
					// u1 = u + a/4 (b v1 - u)
					lamV1 += lamU1 * Real(0.25) * a * bb;
					const Real lamUin = lamU1 * (Real(1) - Real(0.25) * a);
					ga += lamU1 * Real(0.25) * (bb * v1 - u0);
					gb += lamU1 * Real(0.25) * a * v1;
					// v1 = v + 1/4 (0.04 v^2 + 5 v + 140 - u + I)
					lv1 = lamV1 * (Real(1) + Real(0.25) * (Real(0.08) * v0 + Real(5)));
					lu = lamUin - Real(0.25) * lamV1;
					lamI += Real(0.25) * lamV1;
				}
				lamV[i] = lv1;
				lamU[i] = lu;
				gA[i] = ga;
				gB[i] = gb;
				X.lamI[(size_t) t * NB + at] = lamI;
				odd |= !isfinite(lamI);
			}
			if(t > 0) {
				arrived += L.ctas;
				if(L.ctas == 1) __syncthreads();
				else loop_arrive(counter);
			}
		}
	}
	if(odd) X.sync[SYNC_NONFINITE] = 1u;
	for(int i = tid; i < items; i += LOOP_THREADS) {
		const int bl = i & (lanes - 1);
		if(bl >= nb) continue;
		const size_t at = (size_t) (n0 + (i >> laneLog)) * D.B + b0 + bl;
		X.lamU[at] = lamU[i];
		X.gA[at] = gA[i];
		X.gB[at] = gB[i];
	}
}

// readout traces of the last forward pass as [T][B][R]
template<typename Real>
__global__ void bptt_readout_kernel(BpttDev D, BpttState<Real> X, float* out)
{
	const size_t i = (size_t) blockIdx.x * blockDim.x + threadIdx.x;
	const size_t total = (size_t) D.T * D.B * D.R;
	if(i >= total) return;
	const int n = (int) (i % D.R), b = (int) ((i / D.R) % D.B), t = (int) (i / ((size_t) D.R * D.B));
	out[i] = (float) X.rHist[((size_t) t * D.R + n) * D.B + b];
}

// parameter gradients of neuron n: sum over trials, plus u(0) = b v(0) with
// v(0) = -65
template<typename Real>
__device__ __forceinline__ void param_grad(const BpttDev& D, const BpttState<Real>& X, int n, float* da, float* db)
{
	Real sa = Real(0), sb = Real(0);
	for(int b = 0; b < D.B; ++b) {
		const size_t i = (size_t) n * D.B + b;
		sa += X.gA[i];
		sb += X.gB[i] + X.lamU[i] * Real(-65);
	}
	da[n] = (float) sa;
	db[n] = (float) sb;
}

// dL/dW[e] = sum_t,b S_src(t - d) lambda_I,tgt(t) over every (t, b), one warp
// per synapse of source j: spike(k) is S of (t, b) = (k / B, k % B)
template<typename Real, typename Spike>
__device__ __forceinline__ void weight_grad_dense(const BpttDev& D, const BpttState<Real>& X, int j, float* dW, Spike spike)
{
	const size_t NB = (size_t) D.N * D.B;
	const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
	for(int e = D.outStart[j] + warp; e < D.outStart[j + 1]; e += nw) {
		const Real* lam = X.lamI + D.outOff[e];
		const int len = (D.T - (int) (D.outOff[e] / NB)) * D.B;
		Real acc = Real(0);
		for(int k = lane; k < len; k += 32) acc = fma(spike(k), lam[(size_t) (k / D.B) * NB + k % D.B], acc);
#pragma unroll
		for(int o = 16; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
		if(lane == 0) dW[D.outSyn[e]] = (float) acc;
	}
}

// Smooth threshold: every S is nonzero, so the spike train of the source is
// held in shared memory and read against every target's adjoints.  One CTA
// per source; also the parameter gradients of that neuron.
template<typename Real>
__global__ void bptt_weight_grad_smooth(BpttDev D, BpttState<Real> X, float* dW, float* da, float* db, int maxGroups)
{
	extern __shared__ __align__(16) unsigned char raw[];
	Real* sS = reinterpret_cast<Real*>(raw);
	const int j = blockIdx.x;
	const size_t NB = (size_t) D.N * D.B;
	if(j == 0) for(int i = threadIdx.x; i < maxGroups; i += blockDim.x) X.sync[sync_counter(i, true, maxGroups)] = 0;
	if(threadIdx.x == 0) param_grad(D, X, j, da, db);
	for(int k = threadIdx.x; k < D.T * D.B; k += blockDim.x) {
		sS[k] = X.S[(size_t) (k / D.B) * NB + (size_t) j * D.B + k % D.B];
	}
	__syncthreads();
	weight_grad_dense(D, X, j, dW, [&](int k) { return sS[k]; });
}

// Hard threshold: a source fires in few of its T x B (ms, trial) slots (about
// 0.7% at the rates of these networks), so the CTA of a source lists its
// spikes and each thread adds, for one outgoing synapse, the adjoints at
// those spikes: at 4096 x 200 x 500 ms x 16 trials about 50 random 8-byte
// reads per synapse instead of 8000 sequential ones (52 GB of lambda_I, more
// than L2 holds).  Sums run in double over SPIKE_WORDS words at a time.
// When some adjoint is not finite every slot counts (0 x inf is NaN): the
// dense sum, with the spikes decoded on the way.
constexpr int GRAD_THREADS = 256;
constexpr int SPIKE_WORDS = 256;  // words listed per round, at most 16 spikes each

template<typename Real>
__global__ void __launch_bounds__(GRAD_THREADS)
bptt_weight_grad_spikes(BpttDev D, BpttState<Real> X, float* dW, float* da, float* db, int maxGroups)
{
	__shared__ unsigned sSpike[SPIKE_WORDS * BPTT_GROUP];       // t << 16 | b
	__shared__ unsigned char sCount[SPIKE_WORDS * BPTT_GROUP];  // spikes in that ms
	__shared__ int sWarp[GRAD_THREADS / 32];
	const int j = blockIdx.x, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
	const size_t NB = (size_t) D.N * D.B;
	if(j == 0) for(int i = tid; i < maxGroups; i += GRAD_THREADS) X.sync[sync_counter(i, true, maxGroups)] = 0;
	if(tid == 0) param_grad(D, X, j, da, db);
	if(X.sync[SYNC_NONFINITE]) {
		weight_grad_dense(D, X, j, dW, [&](int k) {
			const int t = k / D.B, b = k % D.B;
			const unsigned long long w = load_word(X.words, ((size_t) t * D.groups + b / BPTT_GROUP) * D.N + j, D.wordLog);
			return (Real) (int) ((w >> (4 * (b % BPTT_GROUP))) & 15u);
		});
		return;
	}
	const int words = D.T * D.groups;
	for(int e0 = D.outStart[j]; e0 < D.outStart[j + 1]; e0 += GRAD_THREADS) {
		const int e = e0 + tid;
		const bool mine = e < D.outStart[j + 1];
		const unsigned long long off = mine ? D.outOff[e] : 0;
		const Real* lam = X.lamI + off;
		const int end = D.T - (int) (off / NB);  // spikes from this ms on arrive after the last
		double total = 0;
		for(int w0 = 0; w0 < words; w0 += SPIKE_WORDS) {
			// the spikes of words [w0, w0 + SPIKE_WORDS), in order
			unsigned long long word = 0;
			const int w = w0 + tid;
			if(w < words) word = load_word(X.words, (size_t) w * D.N + j, D.wordLog);
			int n = 0;
			for(unsigned long long m = word; m; ++n) m &= ~(15ull << ((__ffsll((long long) m) - 1) & ~3));
			int incl = n;
#pragma unroll
			for(int o = 1; o < 32; o <<= 1) {
				const int y = __shfl_up_sync(0xffffffffu, incl, o);
				if(lane >= o) incl += y;
			}
			if(lane == 31) sWarp[warp] = incl;
			__syncthreads();
			int pos = incl - n, all = 0;
#pragma unroll
			for(int k = 0; k < GRAD_THREADS / 32; ++k) {
				const int x = sWarp[k];
				if(k < warp) pos += x;
				all += x;
			}
			const unsigned head = ((unsigned) (w / D.groups) << 16) + (unsigned) (w % D.groups) * BPTT_GROUP;
			while(word) {
				const int shift = (__ffsll((long long) word) - 1) & ~3;
				sSpike[pos] = head + (unsigned) (shift >> 2);
				sCount[pos++] = (unsigned char) ((word >> shift) & 15u);
				word &= ~(15ull << shift);
			}
			__syncthreads();
			if(mine) {
				double acc = 0;
#pragma unroll 8
				for(int k = 0; k < all; ++k) {
					const unsigned s = sSpike[k];
					const int t = (int) (s >> 16);
					if(t < end) acc = fma((double) sCount[k], (double) lam[(size_t) t * NB + (s & 0xffffu)], acc);
				}
				total += acc;
			}
			__syncthreads();
		}
		if(mine) dW[D.outSyn[e]] = (float) total;
	}
}

// The launch shape of a loop over the lists `start` with `itemArrays` arrays
// of one Real per (neuron, trial): as many CTAs as there are SMs, one each,
// shared among the trial groups of a launch, each CTA at least minCells
// neurons (fewer CTAs make the barrier cheaper than the work they would
// share).  entry[mode]: bytes of shared memory per list entry besides its
// weight in mode 1 and 2 (0: no such mode); window: those of mode 2 besides.
Bptt::Loop Bptt::planLoop(const std::vector<int>& start, int itemArrays, int minCells, size_t realSize, int sms,
		const size_t entry[3], size_t window) const
{
	Loop p;
	p.groups = std::min(D.groups, sms);
	const int ctas = std::max(1, sms / p.groups);
	p.cells = std::max(std::min(minCells, D.N), (D.N + ctas - 1) / ctas);
	p.ctas = (D.N + p.cells - 1) / p.cells;
	size_t longest = 0;
	for(int n = 0; n < D.N; n += p.cells) {
		longest = std::max(longest, (size_t) (start[std::min(D.N, n + p.cells)] - start[n]));
	}
	const size_t items = (size_t) p.cells * D.lanes * itemArrays * realSize;
	for(int mode = 2; mode > 0; --mode) {
		if(!entry[mode]) continue;
		const size_t bytes = longest * (entry[mode] + realSize) + items + (size_t) p.cells * (16 + 4 * realSize) + 64 + (mode == 2 ? window : 0);
		if(bytes <= m_limit) {
			p.mode = mode;
			p.smem = bytes;
			break;
		}
	}
	return p;
}

Bptt::Bptt(unsigned N, unsigned B, unsigned T, unsigned R, unsigned ckpt, size_t M, const unsigned* src,
		const unsigned* tgt, const unsigned* delay, bool smooth, bool fp64, int device)
{
	if(N == 0 || B == 0 || T == 0 || ckpt == 0) NB_THROW(NEMO_INVALID_INPUT, "empty differentiable network");
	if(R > N) NB_THROW(NEMO_INVALID_INPUT, "more readout neurons than neurons");
	const size_t realSize = fp64 ? 8 : 4;
	if((size_t) T * B * realSize > 227 * 1024) {
		NB_THROW(NEMO_API_UNSUPPORTED, "ms x trials too large for the weight-gradient kernel (%zu bytes of shared memory)",
				(size_t) T * B * realSize);
	}
	if((size_t) N * B > (size_t) INT32_MAX) NB_THROW(NEMO_API_UNSUPPORTED, "neurons x trials too large");
	m_device = device;
	if(device >= 0) BP_CUDA(cudaSetDevice(device));
	else BP_CUDA(cudaGetDevice(&m_device));
	D = BpttDev{};
	D.N = (int) N; D.B = (int) B; D.T = (int) T; D.R = (int) R; D.ckpt = (int) ckpt; D.smooth = smooth ? 1 : 0;
	D.groups = (D.B + BPTT_GROUP - 1) / BPTT_GROUP;
	D.lanes = 1;
	while(D.lanes < std::min(D.B, BPTT_GROUP)) D.lanes *= 2;
	D.maskStride = MASK_HEADER + (D.N * (D.lanes > 8 ? 2 : 1) + 15) / 16 * 16;
	D.ring = 1;
	D.wordLog = D.lanes <= 2 ? 0 : D.lanes == 4 ? 1 : D.lanes == 8 ? 2 : 3;
	m_fp64 = fp64;
	m_M = M;
	// synapses are given source-major: synapse e's weight is W[e]
	std::vector<int> outStart(N + 1, 0), inStart(N + 1, 0), outMid(N, 0), outPad(N + 1, 0);
	for(size_t e = 0; e < M; ++e) {
		if(src[e] >= N || tgt[e] >= N) NB_THROW(NEMO_INVALID_INPUT, "synapse %zu has an invalid neuron", e);
		if(delay[e] < 1) NB_THROW(NEMO_INVALID_INPUT, "synapse %zu has delay 0", e);
		if(e && src[e] < src[e - 1]) NB_THROW(NEMO_INVALID_INPUT, "synapses must be ordered by source");
		outStart[src[e] + 1]++;
		inStart[tgt[e] + 1]++;
		if(delay[e] > 1) outMid[src[e]]++;
	}
	for(unsigned n = 0; n < N; ++n) {
		outPad[n + 1] = outPad[n] + (outMid[n] + 3) / 4 * 4 + (outStart[n + 1] - outMid[n] + 3) / 4 * 4;
		outMid[n] += outStart[n];
		outStart[n + 1] += outStart[n];
		inStart[n + 1] += inStart[n];
	}
	const size_t NB = (size_t) N * B;
	std::vector<int> inSyn(M), outSyn(M);
	std::vector<int2> inSd(M);
	std::vector<unsigned long long> outOff(M);
	std::vector<int> fill(inStart.begin(), inStart.end() - 1), early(outStart.begin(), outStart.end() - 1), late(outMid);
	for(size_t e = 0; e < M; ++e) {
		const int dl = (int) std::min<unsigned>(delay[e], T);
		D.ring = std::max(D.ring, dl);
		const int p = fill[tgt[e]]++;
		inSd[p] = make_int2((int) src[e], dl);
		inSyn[p] = (int) e;
		const int q = delay[e] > 1 ? early[src[e]]++ : late[src[e]]++;
		outOff[q] = (unsigned long long) dl * NB + (unsigned long long) tgt[e] * B;
		outSyn[q] = (int) e;
	}
	try {
		BP_CUDA(cudaStreamCreateWithFlags(&m_filling, cudaStreamNonBlocking));
		D.inStart = upload(inStart);
		D.inSd = upload(inSd);
		D.inSyn = upload(inSyn);
		D.outStart = upload(outStart);
		D.outMid = upload(outMid);
		D.outPad = upload(outPad);
		D.outOff = upload(outOff);
		D.outSyn = upload(outSyn);
		int sms = 1, optin = 0;
		BP_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, m_device));
		BP_CUDA(cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, m_device));
		// the loops' static shared memory: the forward loop's compacted lists
		m_limit = (size_t) std::max(0, optin - 1024 - FWD_LISTS_BYTES);
		const size_t window = (size_t) D.ring * D.maskStride;
		const size_t fwdEntry[3] = { 0, sizeof(int2), smooth || N > 65536 ? 0 : sizeof(unsigned) };
		m_fwd = planLoop(inStart, 5, FWD_MIN_CELLS, realSize, sms, fwdEntry, window);
		// offsets of the adjoint loop's shared lists are 32-bit
		const bool narrow = (unsigned long long) NB * (D.ring + 1ull) <= 0xffffffffull;
		const size_t bwdEntry[3] = { 0, narrow ? sizeof(unsigned) : 0, 0 };
		m_bwd = planLoop(outPad, 11, BWD_MIN_CELLS, realSize, sms, bwdEntry, 0);
		m_maxGroups = sms;
		BP_CUDA(cudaHostAlloc(&m_hostError, 4, cudaHostAllocMapped));
		*m_hostError = 0;
		if(fp64) allocState(X64);
		else allocState(X32);
		// the first pass may come on any stream: its zeros (barrier counters
		// among them) and lists are in place before the handle is out
		BP_CUDA(cudaStreamSynchronize(m_filling));
		BP_CUDA(cudaStreamDestroy(m_filling));
		m_filling = nullptr;
	} catch(...) {
		release();
		throw;
	}
}

template<typename Real>
const void* Bptt::forwardKernel() const
{
	if(D.smooth) {
		return m_fwd.mode ? (const void*) bptt_forward_loop<Real, true, 1> : (const void*) bptt_forward_loop<Real, true, 0>;
	}
	return m_fwd.mode == 2 ? (const void*) bptt_forward_loop<Real, false, 2>
			: m_fwd.mode == 1 ? (const void*) bptt_forward_loop<Real, false, 1> : (const void*) bptt_forward_loop<Real, false, 0>;
}

// 16-byte adjoint loads where every row of B trials starts on 16 bytes
template<typename Real>
const void* Bptt::backwardKernel() const
{
	constexpr int V = 16 / sizeof(Real);
	if(D.B % V == 0) {
		return m_bwd.mode ? (const void*) bptt_backward_loop<Real, V, true> : (const void*) bptt_backward_loop<Real, V, false>;
	}
	return m_bwd.mode ? (const void*) bptt_backward_loop<Real, 1, true> : (const void*) bptt_backward_loop<Real, 1, false>;
}

template<typename Real>
void Bptt::allocState(BpttState<Real>& X)
{
	const size_t NB = (size_t) D.N * D.B, R = (size_t) std::max(1, D.R), B = D.B, T = D.T;
	const size_t nck = (T + D.ckpt - 1) / D.ckpt, seg = (size_t) std::min(D.ckpt, D.T);
	auto a = [&](size_t n) { return static_cast<Real*>(alloc(n * sizeof(Real))); };
	X.alpha = (Real) std::exp(-1.0 / 20.0);
	X.lossScale = Real(1) / ((Real) T * (Real) D.R * (Real) B);
	if(D.smooth) X.S = a(NB * T);
	else {
		X.words = static_cast<unsigned char*>(alloc((T * D.groups * D.N) << D.wordLog));
		X.masks = static_cast<unsigned char*>(alloc(T * D.groups * D.maskStride));
	}
	X.I = a(NB * T);
	X.ckV = a(NB * nck);
	X.ckU = a(NB * nck);
	X.rHist = a(R * T * B);
	X.lossPart = a(R * B);
	X.segV = a(NB * seg);
	X.segU = a(NB * seg);
	X.lamI = a(NB * T);
	X.lamU = a(NB);
	X.gA = a(NB);
	X.gB = a(NB);
	size_t scratch = 0;
	auto global = [&](const Loop& p, int arrays) {
		if(!p.mode) scratch = std::max(scratch, (size_t) p.ctas * p.groups * p.cells * D.lanes * arrays);
	};
	global(m_fwd, 5);
	global(m_bwd, 6);
	if(scratch) {
		X.scratch = a(scratch);
		X.listW = static_cast<float*>(alloc(m_M * sizeof(float)));
	}
	X.sync = static_cast<unsigned*>(alloc((size_t) SYNC_STRIDE * (1 + 2 * m_maxGroups) * sizeof(unsigned)));
	BP_CUDA(cudaHostGetDevicePointer(reinterpret_cast<void**>(&X.hostError), m_hostError, 0));
	auto shared = [&](const void* kernel, size_t bytes) {
		BP_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int) bytes));
	};
	if(m_fwd.mode) shared(forwardKernel<Real>(), m_limit);
	if(m_bwd.mode) shared(backwardKernel<Real>(), m_limit);
	if(D.smooth) shared((const void*) bptt_weight_grad_smooth<Real>, 227 * 1024);
}

Bptt::~Bptt()
{
	release();
}

void Bptt::release() noexcept
{
	if(m_filling) cudaStreamDestroy(m_filling);
	m_filling = nullptr;
	for(void* p : m_allocs) cudaFree(p);
	m_allocs.clear();
	if(m_hostError) cudaFreeHost(m_hostError);
	m_hostError = nullptr;
}

// a barrier of an earlier pass that gave up leaves this model's state undefined
void Bptt::checkError()
{
	if(*(volatile unsigned*) m_hostError) NB_THROW(NEMO_CUDA_ERROR, "differentiable mode: a barrier wait of an earlier pass timed out");
}

template<typename Real>
void Bptt::forwardT(BpttState<Real>& X, const BpttParams& P, float* loss, void* stream)
{
	cudaStream_t st = static_cast<cudaStream_t>(stream);
	if(!m_fwd.mode && m_M) bptt_list_weights_kernel<<<1184, 256, 0, st>>>(m_M, D.inSyn, P.W, X.listW);
	launchLoop(m_fwd, forwardKernel<Real>(), X, P, st);
	bptt_loss_kernel<Real><<<1, 1024, 0, st>>>(D, X, loss, m_maxGroups);
	BP_CUDA(cudaGetLastError());
}

// One cooperative launch (every CTA resident at once: the loop's CTAs wait
// for each other) per set of trial groups.
template<typename Real>
void Bptt::launchLoop(const Loop& p, const void* kernel, BpttState<Real>& X, const BpttParams& P, cudaStream_t st)
{
	LoopArgs a{ p.ctas, p.cells, 0, m_maxGroups, 0u };
	for(; a.g0 < D.groups; a.g0 += p.groups) {
		const int groups = std::min(p.groups, D.groups - a.g0);
		BpttParams params = P;
		void* args[] = { &D, &X, &params, &a };
		BP_CUDA(cudaLaunchCooperativeKernel(kernel, dim3((unsigned) (groups * p.ctas)), dim3(LOOP_THREADS), args,
				p.smem, st));
		a.base += (unsigned) (D.T - 1) * (unsigned) p.ctas;
	}
}

template<typename Real>
void Bptt::backwardT(BpttState<Real>& X, const BpttParams& P, float* dW, float* da, float* db, void* stream)
{
	cudaStream_t st = static_cast<cudaStream_t>(stream);
	if(!m_bwd.mode && m_M) bptt_list_weights_kernel<<<1184, 256, 0, st>>>(m_M, D.outSyn, P.W, X.listW);
	launchLoop(m_bwd, backwardKernel<Real>(), X, P, st);
	if(D.smooth) {
		bptt_weight_grad_smooth<Real><<<D.N, 256, (size_t) D.T * D.B * sizeof(Real), st>>>(D, X, dW, da, db, m_maxGroups);
	} else {
		bptt_weight_grad_spikes<Real><<<D.N, GRAD_THREADS, 0, st>>>(D, X, dW, da, db, m_maxGroups);
	}
	BP_CUDA(cudaGetLastError());
}

template<typename Real>
void Bptt::readoutT(BpttState<Real>& X, float* out, void* stream)
{
	const size_t total = (size_t) D.T * D.B * D.R;
	if(total) {
		bptt_readout_kernel<Real><<<(unsigned) ((total + 255) / 256), 256, 0, static_cast<cudaStream_t>(stream)>>>(D,
				X, out);
	}
	BP_CUDA(cudaGetLastError());
}

void Bptt::forward(const BpttParams& P, float* loss, void* stream)
{
	BP_CUDA(cudaSetDevice(m_device));
	checkError();
	if(m_fp64) forwardT(X64, P, loss, stream);
	else forwardT(X32, P, loss, stream);
}

void Bptt::backward(const BpttParams& P, float* dW, float* da, float* db, void* stream)
{
	BP_CUDA(cudaSetDevice(m_device));
	checkError();
	if(m_fp64) backwardT(X64, P, dW, da, db, stream);
	else backwardT(X32, P, dW, da, db, stream);
}

void Bptt::readout(float* out, void* stream)
{
	BP_CUDA(cudaSetDevice(m_device));
	if(m_fp64) readoutT(X64, out, stream);
	else readoutT(X32, out, stream);
}

void* Bptt::alloc(size_t bytes)
{
	void* p = nullptr;
	bytes = std::max<size_t>(bytes, 4);
	if(cudaMalloc(&p, bytes) != cudaSuccess) {
		NB_THROW(NEMO_CUDA_MEMORY_ERROR, "failed to allocate %zu bytes of device memory", bytes);
	}
	m_allocs.push_back(p);
	BP_CUDA(cudaMemsetAsync(p, 0, bytes, m_filling));
	return p;
}

template<typename V>
const V* Bptt::upload(const std::vector<V>& v)
{
	void* p = nullptr;
	if(cudaMalloc(&p, std::max<size_t>(v.size(), 1) * sizeof(V)) != cudaSuccess) {
		NB_THROW(NEMO_CUDA_MEMORY_ERROR, "failed to allocate device memory");
	}
	m_allocs.push_back(p);
	if(!v.empty()) BP_CUDA(cudaMemcpyAsync(p, v.data(), v.size() * sizeof(V), cudaMemcpyHostToDevice, m_filling));
	return static_cast<const V*>(p);
}

} // namespace nemo_b200
