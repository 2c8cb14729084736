// bptt.hpp -- the differentiable mode (see bptt.cu for the model).
#pragma once

#include <cuda_runtime.h>
#include <stddef.h>

#include <vector>

namespace nemo_b200 {

// sizes and synapse structure (shared by both state types)
struct BpttDev {
	int N, B, T, R, ckpt, smooth;
	int groups;           // trial groups of BPTT_GROUP trials (the last one may be smaller)
	int lanes;            // trials of a group rounded up to a power of two
	int wordLog;          // log2 of a spike word's bytes: 4 bits per trial of a group
	// in-synapses by target, in synapse order, as {source, delay}, delays
	// clamped to T (a longer one never arrives); [N+1] and the synapse index
	const int* inStart;
	const int2* inSd;
	const int* inSyn;
	int ring;             // the longest delay: ms of spikes that a gather reads
	int maskStride;       // bytes of a slice of spike masks: a header, then a mask of `lanes` bits per neuron
	// out-synapses by source, each source's synapses of delay >= 2 before
	// those of delay 1 (outMid), as offsets of their target's trials `delay`
	// ms later in lamI: delay x N x B + target x B
	const int* outStart;  // [N+1] also the synapse range of a source: its weights are W[outStart[n] ..]
	const int* outMid;
	const int* outPad;    // [N+1] start of a source's lists in shared memory, each list padded to four entries
	const unsigned long long* outOff;
	const int* outSyn;    // synapse index
};

// state, trajectory and adjoint arrays in the state type Real
template<typename Real>
struct BpttState {
	Real alpha, lossScale;
	unsigned char* words; // [T][groups][N] spike counts of a group's trials, 4 bits each (hard threshold)
	unsigned char* masks; // [T][groups] slices of maskStride bytes: header (some neuron fired more than once), fired bits
	Real* S;              // [T][N][B] spikes (smooth threshold only)
	Real* I;              // [T][N][B] synaptic input + noise of the last forward pass
	Real* ckV;            // [nck][N][B]
	Real* ckU;
	Real* rHist;          // [T][R][B]
	Real* lossPart;       // [R][B]
	Real* segV;           // [ckpt][N][B] start states of the segment being differentiated
	Real* segU;
	Real* lamI;           // [T][N][B]
	Real* lamU;           // [N][B] adjoint of the initial u
	Real* gA;             // [N][B]
	Real* gB;
	Real* scratch;        // per-item arrays of the two loops when they do not fit in shared memory
	float* listW;         // [M] weights in list order, likewise
	unsigned* sync;       // barrier counters of the loops and the flag words (bptt.cu)
	unsigned* hostError;  // mapped host word: a barrier wait gave up
};

// the caller's float32 tensors (device pointers)
struct BpttParams {
	const float* W;
	const float* a;
	const float* b;
	const float* c;
	const float* d;
	const float* noise;   // [T][B][N]
	const float* target;  // [T][B][R]
};

class Bptt {
public:
	// M synapses, ordered by source; synapse e has weight W[e].  smooth:
	// fast sigmoid in the forward pass; fp64: neuron state, trajectories and
	// adjoints in float64 (inputs and gradients stay float32).
	Bptt(unsigned N, unsigned B, unsigned T, unsigned R, unsigned ckpt, size_t M, const unsigned* src,
			const unsigned* tgt, const unsigned* delay, bool smooth, bool fp64, int device);
	~Bptt();
	// forward pass; *loss (device) receives the loss
	void forward(const BpttParams& P, float* loss, void* stream);
	// gradients of the loss of the last forward pass (device arrays)
	void backward(const BpttParams& P, float* dW, float* da, float* db, void* stream);
	// filtered readout spike trains of the last forward pass, [T][B][R]
	void readout(float* out, void* stream);
	size_t synapses() const { return m_M; }
	unsigned neurons() const { return (unsigned) D.N; }

private:
	// launch shape of the forward or the backward loop: CTAs per trial
	// group, neurons per CTA, groups per launch, shared memory, and what
	// lives there (0: nothing; 1: the CTA's synapses and per-item arrays; 2:
	// and the forward loop's window of spike masks)
	struct Loop {
		int ctas = 1, cells = 1, groups = 1, mode = 0;
		size_t smem = 0;
	};
	BpttDev D;
	bool m_fp64 = false;
	BpttState<float> X32{};
	BpttState<double> X64{};
	Loop m_fwd, m_bwd;
	int m_maxGroups = 1;   // trial groups of one launch at most
	size_t m_limit = 0;    // dynamic shared memory of a loop's CTA at most
	unsigned* m_hostError = nullptr;  // mapped pinned
	cudaStream_t m_filling = nullptr; // of the constructor's zeros and uploads
	int m_device = 0;
	size_t m_M = 0;
	std::vector<void*> m_allocs;
	void release() noexcept;
	void* alloc(size_t bytes);
	template<typename V> const V* upload(const std::vector<V>& v);
	Loop planLoop(const std::vector<int>& start, int itemArrays, int minCells, size_t realSize, int sms,
			const size_t entry[3], size_t window) const;
	void checkError();
	template<typename Real> void allocState(BpttState<Real>& X);
	template<typename Real> void forwardT(BpttState<Real>& X, const BpttParams& P, float* loss, void* stream);
	template<typename Real> void backwardT(BpttState<Real>& X, const BpttParams& P, float* dW, float* da,
			float* db, void* stream);
	template<typename Real> void launchLoop(const Loop& p, const void* kernel, BpttState<Real>& X, const BpttParams& P,
			cudaStream_t st);
	template<typename Real> const void* forwardKernel() const;
	template<typename Real> const void* backwardKernel() const;
	template<typename Real> void readoutT(BpttState<Real>& X, float* out, void* stream);
};

} // namespace nemo_b200
