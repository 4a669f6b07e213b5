// ppc_noalloc.cu — mesh binning that allocates no memory.
//
// Some callers cannot call cudaMalloc at the point where they need the
// mechanics mesh: code that runs under an allocator that forbids hidden
// allocations (a framework's caching allocator or a memory-capped pool),
// real-time loops that must not block on the driver's allocator, or code
// that is not allowed to create a ppc_state at all. ppc_bin_agents_noalloc
// bins agents given in the caller's own device buffers and keeps every
// intermediate (per-voxel chains and prefix, totals of voxel ranges) in
// g_noalloc_scratch below, a fixed-size array in device memory.
// Every GPU that loads this library reserves that array until the process
// exits. All calls on a device share it and it keeps the previous call's
// contents; every entry is rewritten before it is read, apart from the words
// that order a call's work (na_words), which the call before it clears. Calls
// on different streams are ordered one after another by an event. Calls
// captured into graphs are not: replays that overlap with each other or with
// other calls race on the scratch and spoil each other's outputs, though
// nothing beyond those (their words are cleared before every replay, and no
// index read from the scratch is used unchecked).
//
// The result is the one ppc_update_mechanics_mesh + ppc_get_mesh_bins give:
// per-voxel counts and the agents grouped by voxel in voxel order, in
// descending index inside a voxel (the order of a serial run of the
// reference's counting sort).
#include <cuda_runtime.h>

#include <algorithm>
#include <mutex>

#include "ppc_internal.cuh"

namespace {

constexpr int kNaThreads = 1024;
constexpr int kNaBlocks = 1024; // more than any grid has
constexpr int kNaChain = 24;	// agents of a voxel whose order their chain gives; those of larger ones are compared
constexpr int kNaWait = 1 << 22; // polls of a wait before it gives up, about two seconds

// layout of the scratch, in int32 units
constexpr int64_t kOffNext = 0;
constexpr int64_t kOffKey = kOffNext + PPC_NOALLOC_MAX_AGENTS;
constexpr int64_t kOffRank = kOffKey + PPC_NOALLOC_MAX_AGENTS;
constexpr int64_t kOffTmp = kOffRank + PPC_NOALLOC_MAX_AGENTS;
constexpr int64_t kOffHead = kOffTmp + PPC_NOALLOC_MAX_AGENTS;
constexpr int64_t kOffStart = kOffHead + PPC_NOALLOC_MAX_VOXELS;
constexpr int64_t kOffTile = kOffStart + PPC_NOALLOC_MAX_VOXELS;
constexpr int64_t kOffBig = kOffTile + kNaBlocks; // a voxel has more than kNaChain agents
constexpr int64_t kOffWords = kOffBig + 32; // na_words: two that calls use in turn, and the captured calls'
constexpr int64_t kWordsInts = 2 * 32;
constexpr int64_t kScratchInts = kOffWords + 3 * kWordsInts;

static __device__ __align__(256) int32_t g_noalloc_scratch[kScratchInts];

struct na_mesh
{
	double mins[3], maxs[3], shape[3];
	int32_t grid[3];
	int32_t dims;
	int32_t nvox;
};

__device__ __forceinline__ int na_axis(double x, const na_mesh& m, int d)
{
	const double q = (x - m.mins[d]) / m.shape[d];
	if (!(q == q) || q <= 0.0)
		return 0;
	if (q >= (double)m.grid[d])
		return m.grid[d] - 1;
	return (int)q;
}

// The words that order one call's work, a line each: items handed out and
// items done.
struct na_words
{
	int32_t ticket, pad0[31], done, pad1[31];
};
static_assert(sizeof(na_words) == kWordsInts * sizeof(int32_t), "one line per word");

// Thread 0 waits until `want` items are done; false when it gave up. The item
// it then leaves undone makes every block that needs it give up as well, and
// each of them marks the counts with a value that no voxel has as its last
// act, so the mark stands when the launch ends.
__device__ __forceinline__ bool na_wait(na_words* w, int want, int32_t* counts)
{
	int x, polls = 0;
	while (true)
	{
		asm volatile("ld.relaxed.gpu.global.s32 %0, [%1];" : "=r"(x) : "l"(&w->done) : "memory");
		if (x >= want)
			break;
		if (++polls >= kNaWait)
		{
			atomicExch(counts, -1);
			return false;
		}
	}
	asm volatile("fence.acq_rel.gpu;" ::: "memory");
	return true;
}

__device__ __forceinline__ int na_block_scan(int x, int& total)
{
	__shared__ int sums[32];
	const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
	int incl = x;
	for (int o = 1; o < 32; o <<= 1)
	{
		const int y = __shfl_up_sync(0xffffffffu, incl, o);
		if (lane >= o)
			incl += y;
	}
	if (lane == 31)
		sums[warp] = incl;
	__syncthreads();
	const int nw = blockDim.x >> 5;
	if (warp == 0)
	{
		int w = lane < nw ? sums[lane] : 0;
		for (int o = 1; o < 32; o <<= 1)
		{
			const int y = __shfl_up_sync(0xffffffffu, w, o);
			if (lane >= o)
				w += y;
		}
		if (lane < nw)
			sums[lane] = w;
	}
	__syncthreads();
	total = sums[nw - 1];
	const int excl = incl - x + (warp > 0 ? sums[warp - 1] : 0);
	__syncthreads();
	return excl;
}

// The whole call as one launch. The phases clear, count, scan, place and
// compare have an item per block each. A block takes the items in their order
// off a counter, whatever its index, and an item starts once every item of the
// phases before is done. So an item waits only for items that blocks already
// running have taken: the launch needs no set of blocks resident at once, and
// runs beside a kernel that holds some of the SMs. It clears `after`, the words
// of the call behind it.
//
// The call moves 6 MB for 100,003 agents in 884,736 voxels and is bound by its
// dependent phases: a memset and five launches take 34.2 us, one
// launch with grid barriers (which needs all its blocks resident) 20.5, this one
// 20.6 to 21.2 us.
//  count: an agent's voxel, its number there, and its link on the voxel's
//   chain. The chain's last link is whatever the scratch held: whoever walks it
//   knows the count. The totals of the blocks' voxel ranges are formed here too.
//  scan: the starts of a range of voxels.
//  place: descending index inside the voxel, from the agents on its chain.
//   Agents of a voxel of more than kNaChain are gathered by their numbers and
//   compare with one another in the last phase: c^2 loads for c agents, as
//   many as the grid's threads at once. All 131,072 in one voxel take 3.4 ms
//   (a walk along the chain and a block's sort: 380 ms), 3,000 voxels of 30
//   among 31,000 agents 33 us (110 us).
__global__ void __launch_bounds__(kNaThreads, 1)
	k_na_bins(const double* __restrict__ pos, int n, na_mesh m, int32_t* counts, int32_t* scratch, na_words* words,
			  na_words* after, int32_t* agents)
{
	__shared__ int32_t sh[kNaBlocks];
	__shared__ int s_next, s_ok, s_all;
	const int G = gridDim.x, stride = G * kNaThreads;
	const int nvox = m.nvox;
	// voxels per item of the scan, a multiple of four
	const int range = ((nvox + G - 1) / G + 3) & ~3;
	int next = 0;
	if (threadIdx.x == 0)
		next = atomicAdd(&words->ticket, 1);
	while (true)
	{
		if (threadIdx.x == 0)
		{
			const int q = next, phase = q / G;
			s_next = q;
			s_ok = phase == 0 || (phase < 5 && na_wait(words, min(phase, 3) * G, counts));
		}
		__syncthreads();
		const int phase = s_next / G, item = s_next % G, t = item * kNaThreads + threadIdx.x;
		if (!s_ok)
			break;
		if (phase == 0)
		{
			// the caller's buffer is 4-byte aligned at least
			const int head = min(nvox, (int)((16 - (reinterpret_cast<uintptr_t>(counts) & 15)) & 15) / 4);
			const int n4 = (nvox - head) / 4;
			for (int k = t; k < n4; k += stride)
				reinterpret_cast<int4*>(counts + head)[k] = make_int4(0, 0, 0, 0);
			if (t < head)
				counts[t] = 0;
			if (t < nvox - head - 4 * n4)
				counts[head + 4 * n4 + t] = 0;
			if (t < G)
				scratch[kOffTile + t] = 0;
			if (t == 0)
			{
				scratch[kOffBig] = 0;
				if (after)
					after->ticket = after->done = 0;
			}
		}
		else if (phase == 1)
		{
			for (int k = threadIdx.x; k < G; k += kNaThreads)
				sh[k] = 0;
			__syncthreads();
			for (int i = t; i < n; i += stride)
			{
				const int c0 = na_axis(pos[(int64_t)i * m.dims], m, 0);
				const int c1 = m.dims >= 2 ? na_axis(pos[(int64_t)i * m.dims + 1], m, 1) : 0;
				const int c2 = m.dims >= 3 ? na_axis(pos[(int64_t)i * m.dims + 2], m, 2) : 0;
				const int key = c0 + m.grid[0] * (c1 + m.grid[1] * c2);
				const int number = atomicAdd(counts + key, 1);
				const int before = atomicExch(scratch + kOffHead + key, i);
				atomicAdd(sh + key / range, 1);
				scratch[kOffKey + i] = key;
				scratch[kOffRank + i] = number;
				scratch[kOffNext + i] = before;
			}
			__syncthreads();
			for (int k = threadIdx.x; k < G; k += kNaThreads)
				if (sh[k])
					atomicAdd(scratch + kOffTile + k, sh[k]);
		}
		else if (phase == 2)
		{
			int part = 0;
			for (int k = threadIdx.x; k < item; k += kNaThreads)
				part += scratch[kOffTile + k];
			const int lo = item * range, hi = min(nvox, lo + range);
			int c[4];
			auto load = [&](int i) {
#pragma unroll
				for (int q = 0; q < 4; q++)
					c[q] = i + q < hi ? counts[i + q] : 0;
			};
			load(lo + 4 * threadIdx.x);
			int base;
			na_block_scan(part, base);
			for (int b = lo; b < hi; b += 4 * kNaThreads)
			{
				const int i = b + 4 * threadIdx.x;
				if (b > lo)
					load(i);
				int total;
				int4 out;
				out.x = base + na_block_scan(c[0] + c[1] + c[2] + c[3], total);
				out.y = out.x + c[0];
				out.z = out.y + c[1];
				out.w = out.z + c[2];
				if (i + 3 < hi)
					*reinterpret_cast<int4*>(scratch + kOffStart + i) = out; // lo and i are multiples of four
				else
					for (int q = 0; q < 4; q++)
						if (i + q < hi)
							scratch[kOffStart + i + q] = q == 0 ? out.x : q == 1 ? out.y : q == 2 ? out.z : out.w;
				if (max(max(c[0], c[1]), max(c[2], c[3])) > kNaChain)
					scratch[kOffBig] = 1;
				base += total;
			}
		}
		else if (phase == 3)
		{
			for (int i = t; i < n; i += stride)
			{
				const int key = min((unsigned)scratch[kOffKey + i], (unsigned)(nvox - 1));
				const int st = scratch[kOffStart + key], cnt = counts[key];
				if (cnt > kNaChain)
				{
					const int at = st + scratch[kOffRank + i];
					if ((unsigned)at < (unsigned)n)
						scratch[kOffTmp + at] = i;
					continue;
				}
				int j = scratch[kOffHead + key], rank = 0;
				for (int u = 0; u < cnt && (unsigned)j < (unsigned)n; u++)
				{
					rank += j > i;
					if (u + 1 < cnt)
						j = scratch[kOffNext + j];
				}
				if ((unsigned)(st + rank) < (unsigned)n)
					agents[st + rank] = i;
			}
		}
		else
		{
			if (scratch[kOffBig] == 0)
				break; // the same for every block: set by the scan
			if (threadIdx.x == 0)
				s_all = na_wait(words, 4 * G, counts);
			__syncthreads();
			if (!s_all)
				break;
			// warp by warp over the items, so that all of them have the same share
			for (int i = ((threadIdx.x >> 5) * G + item) * 32 + (threadIdx.x & 31); i < n; i += stride)
			{
				const int key = min((unsigned)scratch[kOffKey + i], (unsigned)(nvox - 1));
				const int st = scratch[kOffStart + key], cnt = counts[key];
				if (cnt <= kNaChain || (unsigned)st >= (unsigned)n || cnt > n - st)
					continue;
				const int32_t* all = scratch + kOffTmp + st;
				int rank = 0;
				for (int u = 0; u < cnt; u++)
					rank += all[u] > i;
				agents[st + rank] = i;
			}
		}
		__syncthreads();
		if (threadIdx.x == 0)
		{
			next = atomicAdd(&words->ticket, 1); // its way and that of the item's stores overlap
			asm volatile("red.release.gpu.global.add.s32 [%0], 1;" ::"l"(&words->done) : "memory");
		}
	}
}

std::mutex g_na_mutex;
void* g_na_ptr[256] = {};
int g_na_blocks[256] = {}; // blocks of a whole grid, one per SM
cudaEvent_t g_na_event[256] = {};			// the end of the device's last call...
unsigned long long g_na_stream[256] = {}; // ...and one above the id of its stream (0: none yet)
int g_na_set[256] = {};					  // words of the next call

} // namespace

extern "C" int ppc_bin_agents_noalloc(const ppc_mesh* mesh, const double* positions, int32_t count,
									  int32_t* voxel_counts, int32_t* agents, void* cuda_stream)
{
	if (!mesh || count < 0 || (count > 0 && (!positions || !agents)) || !voxel_counts || mesh->dims < 1
		|| mesh->dims > 3)
	{
		ppc::set_error("ppc_bin_agents_noalloc: null buffer or dims outside 1..3");
		return PPC_ERR_ARG;
	}
	na_mesh m {};
	m.dims = mesh->dims;
	// grid sizes in 64-bit arithmetic, each axis and the running product
	// checked against the scratch's voxel limit before the next multiply, so
	// no extent of the 32-bit mesh fields can wrap the voxel count
	int64_t nvox = 1;
	bool too_many = false;
	for (int d = 0; d < 3; d++)
	{
		m.mins[d] = mesh->bounding_box_mins[d];
		m.maxs[d] = mesh->bounding_box_maxs[d];
		m.shape[d] = mesh->voxel_shape[d];
		int64_t g = 1;
		if (d < mesh->dims)
		{
			if (mesh->voxel_shape[d] <= 0 || mesh->bounding_box_maxs[d] < mesh->bounding_box_mins[d])
			{
				ppc::set_error("ppc_bin_agents_noalloc: invalid mesh");
				return PPC_ERR_ARG;
			}
			const int64_t extent = (int64_t)mesh->bounding_box_maxs[d] - (int64_t)mesh->bounding_box_mins[d];
			g = (extent + mesh->voxel_shape[d] - 1) / mesh->voxel_shape[d];
		}
		g = g < 1 ? 1 : g;
		too_many = too_many || g > PPC_NOALLOC_MAX_VOXELS;
		nvox = too_many ? PPC_NOALLOC_MAX_VOXELS + 1 : nvox * g;
		too_many = too_many || nvox > PPC_NOALLOC_MAX_VOXELS;
		m.grid[d] = (int32_t)(too_many ? 1 : g);
	}
	if (count > PPC_NOALLOC_MAX_AGENTS || too_many)
	{
		ppc::set_error("ppc_bin_agents_noalloc: at most " + std::to_string(PPC_NOALLOC_MAX_AGENTS) + " agents and "
					   + std::to_string(PPC_NOALLOC_MAX_VOXELS) + " voxels fit its fixed scratch (asked for "
					   + std::to_string(count) + " agents, "
					   + (too_many ? std::string("more than the limit of") : std::to_string(nvox)) + " voxels)");
		return PPC_ERR_CAPACITY;
	}
	m.nvox = (int32_t)nvox;

	// the scratch's device address, looked up once per device with that
	// device current (the symbol's host-side name is only a stand-in)
	int dev = 0;
	cudaError_t e = cudaGetDevice(&dev);
	if (e != cudaSuccess || dev < 0 || dev >= 256)
		return e != cudaSuccess ? ppc::cuda_fail(e, "cudaGetDevice") : PPC_ERR_NO_DEVICE;
	cudaStream_t st = static_cast<cudaStream_t>(cuda_stream);
	if (count == 0)
	{
		PPC_CUDA(cudaMemsetAsync(voxel_counts, 0, sizeof(int32_t) * nvox, st));
		return PPC_OK;
	}
	std::lock_guard<std::mutex> lock(g_na_mutex);
	if (!g_na_ptr[dev])
	{
		int sms = 0;
		e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
		if (e == cudaSuccess && !g_na_event[dev])
			e = cudaEventCreateWithFlags(&g_na_event[dev], cudaEventDisableTiming);
		if (e != cudaSuccess)
			return ppc::cuda_fail(e, "ppc_bin_agents_noalloc");
		g_na_blocks[dev] = std::min(sms, kNaBlocks);
		void* p = nullptr;
		e = cudaGetSymbolAddress(&p, g_noalloc_scratch);
		if (e != cudaSuccess)
			return ppc::cuda_fail(e, "cudaGetSymbolAddress(g_noalloc_scratch)");
		g_na_ptr[dev] = p;
	}
	int32_t* scratch = static_cast<int32_t*>(g_na_ptr[dev]);
	na_words* const sets = reinterpret_cast<na_words*>(scratch + kOffWords);
	na_words *words = sets + g_na_set[dev], *after = sets + (g_na_set[dev] ^ 1);
	const int blocks
		= std::min(g_na_blocks[dev], std::max((count + kNaThreads - 1) / kNaThreads, (int)(nvox / (4 * kNaThreads)) + 1));

	// a captured call has words of its own, cleared in the graph; others wait
	// for the call before them where that was on another stream
	cudaStreamCaptureStatus cs = cudaStreamCaptureStatusNone;
	if (cudaStreamIsCapturing(st, &cs) != cudaSuccess)
		cudaGetLastError(); // the launch reports it
	const bool captured = cs != cudaStreamCaptureStatusNone;
	unsigned long long id = 0;
	if (captured)
	{
		words = sets + 2;
		after = nullptr;
		PPC_CUDA(cudaMemsetAsync(words, 0, sizeof(na_words), st));
	}
	else
	{
		PPC_CUDA(cudaStreamGetId(st, &id));
		if (g_na_stream[dev] != 0 && g_na_stream[dev] != id + 1)
			PPC_CUDA(cudaStreamWaitEvent(st, g_na_event[dev], 0));
	}
	// the launch's own status: an error that an earlier call left pending must
	// not pass for one of this launch, whose words are used up
	cudaLaunchConfig_t cfg {};
	cfg.gridDim = dim3(blocks);
	cfg.blockDim = dim3(kNaThreads);
	cfg.stream = st;
	PPC_CUDA(cudaLaunchKernelEx(&cfg, k_na_bins, positions, count, m, voxel_counts, scratch, words, after, agents));
	if (!captured)
	{
		g_na_set[dev] ^= 1;
		PPC_CUDA(cudaEventRecord(g_na_event[dev], st));
		g_na_stream[dev] = id + 1;
	}
	return PPC_OK;
}
