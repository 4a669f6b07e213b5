// ppc_api.cu — the extern "C" entry points of libppc (include/ppc.h).
//
// Host side of the device state: allocation, host <-> device transfer in the
// reference's cell_data layout, the reference solver entry points, and the
// fused step with CUDA-graph replay.
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstdio>
#include <cstring>
#include <exception>
#include <string>
#include <thread>
#include <vector>

#include "ppc_internal.cuh"

namespace ppc {

static thread_local std::string g_last_error;

void set_error(const std::string& msg) { g_last_error = msg; }

int cuda_fail(cudaError_t e, const char* where)
{
	set_error(std::string(where) + ": " + cudaGetErrorString(e));
	return PPC_ERR_CUDA;
}

namespace {

int fail(int rc, const std::string& msg)
{
	set_error(msg);
	return rc;
}

// Device arrays of a state: `want` collects them, `place` carves them out of
// one block and clears those that start at zero with one memset (they lie
// first; on the state's stream, since the legacy stream would not order with
// it). One allocation instead of some eighty.
struct arena
{
	struct item
	{
		void** p;
		size_t bytes;
		bool zero;
	};
	std::vector<item> items;

	template <typename T>
	void want(T*& p, size_t count, bool zero = true)
	{
		items.push_back({ reinterpret_cast<void**>(&p), (std::max<size_t>(count, 1) * sizeof(T) + 255) & ~(size_t)255, zero });
	}

	int place(ppc_state* s)
	{
		size_t total = 0, cleared = 0;
		for (const auto& it : items)
		{
			total += it.bytes;
			cleared += it.zero ? it.bytes : 0;
		}
		char* q = nullptr;
		PPC_CUDA(cudaMalloc(&q, total));
		s->allocations.push_back({ q, total });
		if (cleared)
			PPC_CUDA(cudaMemsetAsync(q, 0, cleared, s->stream));
		char* rest = q + cleared;
		for (const auto& it : items)
		{
			*it.p = it.zero ? q : rest;
			(it.zero ? q : rest) += it.bytes;
		}
		return PPC_OK;
	}
};

#define PPC_TRY(x)                                                                                                     \
	do                                                                                                                 \
	{                                                                                                                  \
		int rc_ = (x);                                                                                                 \
		if (rc_ != PPC_OK)                                                                                             \
			return rc_;                                                                                                \
	} while (0)

int launch_pending(ppc_state* s);

// Staging arena of one transfer call: stage_reset at the start of the call,
// then each field takes its own 256-byte aligned region, so the copy and the
// (un)pack kernel of every field are queued without waiting for the previous
// field's. Growing the arena waits for the queued work (which still reads the
// old buffer) before freeing it.
void stage_reset(ppc_state* s)
{
	s->stage_used = 0;
	s->pending_unpacks.clear();
	s->pending_copies.clear();
	s->pending_host.clear(); // of a call that failed before its data landed
	s->bounce_used = 0;
}

int stage_take(ppc_state* s, size_t bytes, void** out)
{
	size_t off = (s->stage_used + 255) & ~(size_t)255;
	if (off + bytes > s->stage_bytes)
	{
		const size_t want = std::max(off + bytes, 2 * s->stage_bytes);
		if (s->stage)
		{
			// the deferred unpacks and copies still read the old buffer
			PPC_TRY(launch_pending(s));
			PPC_CUDA(cudaStreamSynchronize(s->stream));
			PPC_CUDA(cudaFree(s->stage));
			s->stage = nullptr;
			s->stage_bytes = 0;
		}
		PPC_CUDA(cudaMalloc(&s->stage, want));
		s->stage_bytes = want;
		off = 0;
	}
	*out = static_cast<char*>(s->stage) + off;
	s->stage_used = off + bytes;
	return PPC_OK;
}

int flush_unpacks(ppc_state* s)
{
	for (const auto& u : s->pending_unpacks)
		PPC_TRY(launch_unpack_vec(s, u.dev, u.src, u.r, u.n, u.changed));
	s->pending_unpacks.clear();
	return PPC_OK;
}

const void* mapped(const void* host);

constexpr size_t kBounceMost = (size_t)32 << 20; // page-locked bytes of a state's landing area
constexpr size_t kBounceLeast = (size_t)1 << 20; // smaller copies are left to the driver
constexpr int kHostThreads = 4;

// the queued copies' data, landed and waited for, from the page-locked area
// into the caller's rows
void drain_host(ppc_state* s)
{
	size_t total = 0;
	for (const auto& c : s->pending_host)
		total += c.bytes;
	if (!total)
		return;
	auto part = [s](size_t lo, size_t hi) {
		size_t at = 0;
		for (const auto& c : s->pending_host)
		{
			const size_t a = std::max(lo, at), b = std::min(hi, at + c.bytes);
			if (a < b)
				std::memcpy(static_cast<char*>(c.dst) + (a - at), static_cast<const char*>(c.src) + (a - at), b - a);
			at += c.bytes;
		}
	};
	std::thread helpers[kHostThreads - 1];
	for (int k = 1; k < kHostThreads; k++)
	{
		const size_t lo = total * k / kHostThreads, hi = total * (k + 1) / kHostThreads;
		try
		{
			helpers[k - 1] = std::thread(part, lo, hi);
		}
		catch (const std::exception&)
		{
			part(lo, hi); // no thread to be had
		}
	}
	part(0, total / kHostThreads);
	for (auto& t : helpers)
		if (t.joinable())
			t.join();
	s->pending_host.clear();
	s->bounce_used = 0;
}

// Rows up to this size go between mapped host rows and the device by kernels,
// which cost less than copies' latency: a download's columns in one launch. A
// host loop (upload, step, download) of 2,700 agents, at the line: 67 us, 87
// with copies. Kernels are the faster ones beyond it too (20,000 agents: 105 and
// 128 us) where nothing else runs; larger rows keep the copies, which run on the
// transfer stream beside the device's earlier work.
constexpr size_t kSmallRows = 64 * 1024;

// takes a column of a small download into the launch that follows; false where
// it has to be copied
bool pull_column(ppc_state* s, void* dst, const void* src, size_t bytes, int width)
{
	if (!s->pulling || bytes > kSmallRows || bytes % 4 || (reinterpret_cast<uintptr_t>(dst) | reinterpret_cast<uintptr_t>(src)) % (width ? 8 : 4)
		|| s->pull.count == pull_list::kMost)
		return false;
	void* d = const_cast<void*>(mapped(dst));
	if (!d)
		return false;
	s->pull.job[s->pull.count++] = { d, src, (int32_t)(bytes / (width ? 8 : 4)), width };
	return true;
}

// Queues a device-to-host copy on the stream. Into pageable rows the driver
// copies with one thread, which the host waits for. Where page-locked vectors
// follow (s->landing), a large column lands in the state's page-locked area
// instead, as long as there is room, and drain_host copies it on with a few
// threads beside the vectors' transfer: 1 M agents, ten dividing steps and
// 72 MB, 16 MB of them pageable, 5.33 ms with the driver's copies, 5.06 ms so.
// With nothing to run beside, the driver is the faster one: all fields of
// 300,000 agents into pageable rows 5.4 ms, through the area 15 ms.
int copy_down(ppc_state* s, void* dst, const void* src, size_t bytes)
{
	void* to = dst;
	cudaPointerAttributes at {};
	if (s->landing && bytes >= kBounceLeast && bytes <= s->bounce_bytes - s->bounce_used)
	{
		if (cudaPointerGetAttributes(&at, dst) != cudaSuccess)
			cudaGetLastError();
		if (at.type == cudaMemoryTypeUnregistered)
		{
			to = static_cast<char*>(s->bounce) + s->bounce_used;
			s->pending_host.push_back({ dst, to, bytes });
			s->bounce_used += bytes;
		}
	}
	PPC_CUDA(cudaMemcpyAsync(to, src, bytes, cudaMemcpyDeviceToHost, s->stream));
	return PPC_OK;
}

int flush_copies(ppc_state* s)
{
	for (const auto& c : s->pending_copies)
		PPC_CUDA(cudaMemcpyAsync(c.dst, c.src, c.bytes, cudaMemcpyDeviceToHost, s->stream));
	s->pending_copies.clear();
	return PPC_OK;
}

int launch_pending(ppc_state* s)
{
	PPC_TRY(flush_unpacks(s));
	return flush_copies(s);
}

// status of the device error bits `err`; clears the device word when set
int map_errors(ppc_state* s, int32_t err)
{
	if (err == 0)
		return PPC_OK;
	PPC_CUDA(cudaMemsetAsync(s->v.err, 0, sizeof(int32_t), s->stream));
	PPC_CUDA(cudaStreamSynchronize(s->stream));
	if (err & ERR_TIMEOUT)
	{
		s->lost = true;
		return fail(PPC_ERR_TIMEOUT, "a grid barrier of a step gave up waiting; the state must be uploaded again");
	}
	if (err & ERR_NONFINITE)
		return fail(PPC_ERR_NONFINITE, "an agent position is NaN or infinite");
	if (err & ERR_OUT_OF_MESH)
		return fail(PPC_ERR_OUT_OF_MESH, "an agent lies outside the mechanics mesh");
	if (err & ERR_NEIGHBOR_CAPACITY)
		return fail(PPC_ERR_CAPACITY, "a neighbour list exceeds the neighbour capacity");
	if (err & ERR_AGENT_CAPACITY)
		return fail(PPC_ERR_CAPACITY, "division exceeds the agent capacity of a replicate");
	if (err & ERR_SPRING_CAPACITY)
		return fail(PPC_ERR_ARG, "spring rows are not symmetric");
	if (err & ERR_LIST_CAPACITY)
		return fail(PPC_ERR_CAPACITY, "removal or division list overflow");
	return fail(PPC_ERR_CUDA, "unknown device error");
}

int device_errors(ppc_state* s)
{
	PPC_CUDA(cudaMemcpyAsync(s->pinned_err, s->v.err, sizeof(int32_t), cudaMemcpyDeviceToHost, s->stream));
	PPC_CUDA(cudaStreamSynchronize(s->stream));
	return map_errors(s, *s->pinned_err);
}

// the bins no longer match the positions: the next step rebuilds them
void invalidate_bins(ppc_state* s)
{
	s->skin_lists = false;
	s->bins_valid = false;
	s->bins_cond = false;
}

int finish(ppc_state* s)
{
	PPC_CUDA(cudaGetLastError());
	return device_errors(s);
}

// finish, with the replicates' counts read in the same copy
int finish_counts(ppc_state* s)
{
	PPC_CUDA(cudaGetLastError());
	PPC_CUDA(cudaMemcpyAsync(s->pinned_ctr, s->v.ctr, sizeof(rep_counters) * (s->nreps + 1), cudaMemcpyDeviceToHost,
							 s->stream)); // the counters and the error word
	PPC_CUDA(cudaStreamSynchronize(s->stream));
	for (int32_t k = 0; k < s->nreps; k++)
		s->host_count[k] = s->pinned_ctr[k].count;
	s->counts_known = true;
	return PPC_OK;
}

// rows of a pass over replicate r whose kernels read the live count themselves
int32_t most_rows(ppc_state* s, int32_t r) { return s->counts_known ? s->host_count[r] : s->reps[r].cap; }

bool valid(ppc_state* s, int32_t r) { return s && r >= 0 && r < s->nreps; }

int read_counters(ppc_state* s, std::vector<rep_counters>& c)
{
	c.resize(s->nreps);
	PPC_CUDA(cudaMemcpyAsync(c.data(), s->v.ctr, sizeof(rep_counters) * s->nreps, cudaMemcpyDeviceToHost, s->stream));
	PPC_CUDA(cudaStreamSynchronize(s->stream));
	for (int32_t k = 0; k < s->nreps; k++)
		s->host_count[k] = c[k].count;
	s->counts_known = true;
	return PPC_OK;
}

int release_graph(ppc_state* s)
{
	for (auto& e : s->graphs)
		if (e.exec)
			cudaGraphExecDestroy(e.exec);
	s->graphs.clear();
	return PPC_OK;
}

// ---- host <-> device transfer --------------------------------------------------

template <typename T>
int put_scalar(ppc_state* s, T* dev, const T* host, int32_t base, int32_t n, size_t width, bool defaults, T dflt)
{
	T* dst = dev + (size_t)base * width;
	size_t cnt = (size_t)n * width;
	if (host)
	{
		PPC_CUDA(cudaMemcpyAsync(dst, host, cnt * sizeof(T), cudaMemcpyHostToDevice, s->stream));
	}
	else if (defaults && cnt)
	{
		std::vector<T> tmp(cnt, dflt);
		PPC_CUDA(cudaMemcpyAsync(dst, tmp.data(), cnt * sizeof(T), cudaMemcpyHostToDevice, s->stream));
		PPC_CUDA(cudaStreamSynchronize(s->stream));
	}
	return PPC_OK;
}

template <typename T>
int get_scalar(ppc_state* s, T* host, const T* dev, int32_t base, int32_t first, int32_t n, size_t width)
{
	if (host && n > first
		&& !pull_column(s, host + (size_t)first * width, dev + (size_t)(base + first) * width,
						(size_t)(n - first) * width * sizeof(T), 0))
		PPC_TRY(copy_down(s, host + (size_t)first * width, dev + (size_t)(base + first) * width,
						  (size_t)(n - first) * width * sizeof(T)));
	return PPC_OK;
}

// the device address of a pinned, mapped host buffer (kernels then read or
// write it directly over the bus, without a staging copy), or null
const void* mapped(const void* host)
{
	cudaPointerAttributes at {};
	if (cudaPointerGetAttributes(&at, host) != cudaSuccess)
	{
		cudaGetLastError();
		return nullptr;
	}
	return at.type == cudaMemoryTypeHost ? at.devicePointer : nullptr;
}

// the same for rows of doubles: null where a kernel's loads of them would be
// misaligned (a copy takes any address)
const void* mapped_doubles(const void* host)
{
	return reinterpret_cast<uintptr_t>(host) % sizeof(double) == 0 ? mapped(host) : nullptr;
}

// Host rows (dims doubles per agent) into the double4 device rows. Pinned
// host buffers go through the copy engine into the staging arena (or, in the
// zero-copy transfer mode, are read by the unpack kernel over the bus);
// pageable ones are staged by the copy call itself.
int put_vec(ppc_state* s, double4* dev, const double* host, int32_t r, int32_t n, bool defaults,
			int32_t* changed = nullptr)
{
	if (!host && !defaults)
		return PPC_OK;
	if (n == 0)
		return PPC_OK;
	if (host && (s->zero_copy || s->direct_rows))
		if (const void* d = mapped_doubles(host))
			return launch_unpack_vec(s, dev, static_cast<const double*>(d), r, n, changed);
	const size_t bytes = (size_t)n * s->dims * sizeof(double);
	void* st = nullptr;
	PPC_TRY(stage_take(s, bytes, &st));
	if (host)
		PPC_CUDA(cudaMemcpyAsync(st, host, bytes, cudaMemcpyHostToDevice, s->h2d_stream ? s->h2d_stream : s->stream));
	else
		PPC_CUDA(cudaMemsetAsync(st, 0, bytes, s->stream));
	// the unpack waits until the call's other copies are queued, so the copy
	// engine moves the fields back to back
	s->pending_unpacks.push_back({ dev, static_cast<const double*>(st), r, n, changed });
	return PPC_OK;
}

int get_vec(ppc_state* s, double* host, const double4* dev, int32_t r, int32_t first, int32_t n)
{
	if (!host || n <= first)
		return PPC_OK;
	host += (size_t)first * s->dims;
	dev += first;
	n -= first;
	if (pull_column(s, host, dev + s->reps[r].base, (size_t)n * s->dims * sizeof(double), s->dims))
		return PPC_OK;
	if (s->zero_copy)
		if (const void* d = mapped_doubles(host))
			return launch_pack_vec(s, static_cast<double*>(const_cast<void*>(d)), dev, r, n);
	const size_t bytes = (size_t)n * s->dims * sizeof(double);
	void* st = nullptr;
	PPC_TRY(stage_take(s, bytes, &st));
	PPC_TRY(launch_pack_vec(s, static_cast<double*>(st), dev, r, n));
	// the copy waits until the call's other packs are queued
	s->pending_copies.push_back({ host, st, bytes });
	return PPC_OK;
}

int put_prm(ppc_state* s, int field, const double* host, int32_t r, int32_t n, bool defaults, double dflt)
{
	if ((!host && !defaults) || n == 0)
		return PPC_OK;
	const size_t bytes = (size_t)n * sizeof(double);
	void* st = nullptr;
	PPC_TRY(stage_take(s, bytes, &st));
	if (host)
		PPC_CUDA(cudaMemcpyAsync(st, host, bytes, cudaMemcpyHostToDevice, s->stream));
	else
	{
		std::vector<double> tmp(n, dflt);
		PPC_CUDA(cudaMemcpyAsync(st, tmp.data(), bytes, cudaMemcpyHostToDevice, s->stream));
		PPC_CUDA(cudaStreamSynchronize(s->stream)); // tmp leaves scope
	}
	PPC_TRY(launch_unpack_prm(s, field, static_cast<const double*>(st), r, n));
	return PPC_OK;
}

int get_prm(ppc_state* s, int field, double* host, int32_t r, int32_t first, int32_t n)
{
	if (!host || n <= first)
		return PPC_OK;
	host += first;
	n -= first;
	const size_t bytes = (size_t)n * sizeof(double);
	void* st = nullptr;
	PPC_TRY(stage_take(s, bytes, &st));
	PPC_TRY(launch_pack_prm(s, field, static_cast<double*>(st), s->reps[r].base + first, n));
	return copy_down(s, host, st, bytes);
}

// reference defaults (src/data_storage_phenotype.cpp:62-125,194-214, src/cell.cpp:47-61)
constexpr double kRadius = 8.412710547954228, kNuclearRadius = 5.051670902881889, kSurface = 889.3685284131693;

// true when the view carries no field but positions, velocities, previous
// velocities, pressure and orientation
bool only_kinematic(const ppc_agents* a)
{
	const void* others[] = { a->radius, a->cell_cell_repulsion_strength, a->cell_cell_adhesion_strength,
							 a->relative_maximum_adhesion_distance, a->cell_BM_repulsion_strength,
							 a->attachment_elastic_constant, a->attachment_rate, a->detachment_rate,
							 a->maximum_number_of_attachments, a->cell_adhesion_affinities, a->cell_definition_indices,
							 a->is_movable, a->flags, a->agent_ids, a->total_volume, a->nuclear_volume,
							 a->nuclear_radius, a->surface_area, a->polarity, a->spring_counts, a->springs };
	for (const void* p : others)
		if (p)
			return false;
	return true;
}

double largest(const double* x, int32_t n)
{
	double m = 0;
	for (int32_t i = 0; i < n; i++)
		m = std::max(m, x[i]);
	return m;
}

int transfer_in(ppc_state* s, int32_t r, const ppc_agents* a, bool defaults)
{
	const rep_info& R = s->reps[r];
	const int32_t n = a->count;
	const int32_t base = R.base;
	const int D = s->ndefs;
	view& v = s->v;
	stage_reset(s);
	if (a->cell_definition_indices)
		for (int32_t i = 0; i < n; i++)
			if (a->cell_definition_indices[i] < 0 || a->cell_definition_indices[i] >= D)
				return fail(PPC_ERR_ARG, "cell definition index out of range");

	// the bound on the interaction reach that admits steps over lists
	if (a->radius || defaults)
		s->reach_radius[r] = a->radius ? largest(a->radius, n) : kRadius;
	if (a->relative_maximum_adhesion_distance || defaults)
		s->reach_factor[r]
			= a->relative_maximum_adhesion_distance ? largest(a->relative_maximum_adhesion_distance, n) : 1.25;

	// an upload of kinematic fields only (positions, velocities, previous
	// velocities, pressure, orientation) keeps the mesh when the positions it
	// brings are bit-identical to the resident ones
	// (pos_changed is zero after every rebuild: its copy kernel clears it)
	const bool kinematic = !defaults && only_kinematic(a);
	s->ready_pending = false;
	bool pinned = true;
	for (const void* p : { (const void*)a->positions, (const void*)a->velocities,
						   (const void*)a->previous_velocities, (const void*)a->simple_pressure,
						   (const void*)a->orientation })
		if (p && !mapped(p))
			pinned = false;
	// page-locked kinematic rows are copied into the staging arena on the
	// transfer stream, beside whatever the stream still runs (the last step's
	// mesh rebuild); the arena is free once the stream has unpacked the
	// previous upload, and the unpacks wait for the copies
	const bool small = kinematic && pinned && (size_t)n * s->dims * sizeof(double) <= kSmallRows;
	const bool beside = kinematic && pinned && !small && !s->zero_copy && s->xfer;
	s->direct_rows = small;
	if (beside)
	{
		PPC_CUDA(cudaStreamWaitEvent(s->xfer, s->ev_stage_free, 0));
		s->h2d_stream = s->xfer;
	}
	int rc = put_vec(s, v.pos[s->cur], a->positions, r, n, defaults, kinematic ? v.pos_changed : nullptr);
	if (rc == PPC_OK)
		rc = put_vec(s, v.vel, a->velocities, r, n, defaults);
	if (rc == PPC_OK)
		rc = put_vec(s, v.vprev, a->previous_velocities, r, n, defaults);
	if (rc == PPC_OK)
		rc = put_vec(s, v.orient, a->orientation, r, n, defaults);
	s->h2d_stream = nullptr;
	s->direct_rows = false;
	PPC_TRY(rc);
	if (beside)
	{
		PPC_CUDA(cudaEventRecord(s->ev_h2d, s->xfer));
		PPC_CUDA(cudaStreamWaitEvent(s->stream, s->ev_h2d, 0));
	}
	PPC_TRY(flush_unpacks(s));
	PPC_CUDA(cudaEventRecord(s->ev_stage_free, s->stream));
	PPC_TRY(put_prm(s, 0, a->radius, r, n, defaults, kRadius));
	PPC_TRY(put_prm(s, 1, a->cell_cell_repulsion_strength, r, n, defaults, 10.0));
	PPC_TRY(put_prm(s, 2, a->cell_cell_adhesion_strength, r, n, defaults, 0.4));
	PPC_TRY(put_prm(s, 3, a->cell_BM_repulsion_strength, r, n, defaults, 100.0));
	PPC_TRY(put_scalar(s, v.rmad, a->relative_maximum_adhesion_distance, base, n, 1, defaults, 1.25));
	PPC_TRY(put_scalar(s, v.ec, a->attachment_elastic_constant, base, n, 1, defaults, 0.01));
	PPC_TRY(put_scalar(s, v.arate, a->attachment_rate, base, n, 1, defaults, 0.0));
	PPC_TRY(put_scalar(s, v.drate, a->detachment_rate, base, n, 1, defaults, 0.0));
	PPC_TRY(put_scalar(s, v.pressure, a->simple_pressure, base, n, 1, defaults, 0.0));
	PPC_TRY(put_scalar(s, v.vol, a->total_volume, base, n, 1, defaults, 2494.0));
	PPC_TRY(put_scalar(s, v.nvol, a->nuclear_volume, base, n, 1, defaults, 540.0));
	PPC_TRY(put_scalar(s, v.nrad, a->nuclear_radius, base, n, 1, defaults, kNuclearRadius));
	PPC_TRY(put_scalar(s, v.sarea, a->surface_area, base, n, 1, defaults, kSurface));
	PPC_TRY(put_scalar(s, v.polarity, a->polarity, base, n, 1, defaults, 0.0));
	PPC_TRY(put_scalar(s, v.aff, a->cell_adhesion_affinities, base, n, D, defaults, 1.0));
	PPC_TRY(put_scalar<int32_t>(s, v.def, a->cell_definition_indices, base, n, 1, defaults, 0));
	PPC_TRY(put_scalar<int32_t>(s, v.maxatt, a->maximum_number_of_attachments, base, n, 1, defaults, 12));
	PPC_TRY(put_scalar<uint8_t>(s, v.movable, a->is_movable, base, n, 1, defaults, 1));
	PPC_TRY(put_scalar<uint8_t>(s, v.flags, a->flags, base, n, 1, defaults, 0));

	// ids: given or 0..n-1; the next created agent continues after the largest
	if (a->agent_ids || defaults)
	{
		std::vector<int64_t> ids(n);
		int64_t next = 0;
		for (int32_t i = 0; i < n; i++)
		{
			ids[i] = a->agent_ids ? a->agent_ids[i] : i;
			next = std::max<int64_t>(next, ids[i] + 1);
		}
		PPC_TRY(put_scalar<int64_t>(s, v.ids, ids.data(), base, n, 1, false, 0));
		PPC_CUDA(cudaMemcpyAsync(&v.ctr[r].next_id, &next, sizeof next, cudaMemcpyHostToDevice, s->stream));
		PPC_CUDA(cudaStreamSynchronize(s->stream));
	}

	// springs: host rows hold local indices, device rows hold slots
	if (a->spring_counts || defaults)
	{
		bool any = false;
		if (a->spring_counts)
		{
			for (int32_t i = 0; i < n; i++)
			{
				const int32_t c = a->spring_counts[i];
				if (c < 0 || c > s->scap || c > a->spring_capacity)
					return fail(PPC_ERR_CAPACITY, "spring count exceeds the spring capacity");
				for (int32_t k = 0; k < c; k++)
				{
					const int32_t j = a->springs ? a->springs[(size_t)i * a->spring_capacity + k] : -1;
					if (j < 0 || j >= n)
						return fail(PPC_ERR_ARG, "spring partner index out of range");
				}
				any |= c > 0;
			}
		}
		PPC_TRY(put_scalar<int32_t>(s, v.scnt, a->spring_counts, base, n, 1, true, 0));
		if (any)
		{
			const size_t bytes = (size_t)n * a->spring_capacity * sizeof(int32_t);
			void* st = nullptr;
			PPC_TRY(stage_take(s, bytes, &st));
			PPC_CUDA(cudaMemcpyAsync(st, a->springs, bytes, cudaMemcpyHostToDevice, s->stream));
			PPC_TRY(launch_springs_local(s, r, n, static_cast<int32_t*>(st), a->spring_capacity, 1));
			PPC_CUDA(cudaStreamSynchronize(s->stream));
		}
		s->has_springs = s->has_springs || any;
	}

	if (defaults)
	{
		PPC_CUDA(cudaMemsetAsync(v.ncnt + base, 0, sizeof(int32_t) * std::max(n, 1), s->stream));
		int32_t cnt[2] = { n, n };
		PPC_CUDA(cudaMemcpyAsync(&v.ctr[r].count, cnt, sizeof(int32_t) * 2, cudaMemcpyHostToDevice, s->stream));
		s->host_count[r] = n;
	}

	// host flags that pick kernel variants
	if (a->velocities)
	{
		for (int32_t i = 0; i < n * s->dims && !s->vel_dirty; i++)
			s->vel_dirty = a->velocities[i] != 0.0;
	}
	for (const double* rate : { a->attachment_rate, a->detachment_rate })
		if (rate)
			for (int32_t i = 0; i < n && !s->rates_nonzero; i++)
				s->rates_nonzero = rate[i] != 0.0;
	if (kinematic)
	{
		// the slots still hold the same agents; whether the positions moved is
		// known on the device only: the next rebuild runs there if they did
		if (a->positions && s->bins_valid)
		{
			s->bins_valid = false;
			s->bins_cond = true;
		}
		s->skin_refresh = true;
		// page-locked rows are copied by the queued DMA, so the call returns
		// at once and the next step queues behind the copies; pageable rows
		// are waited for, so the caller may reuse them on return
		if (!pinned)
			PPC_CUDA(cudaStreamSynchronize(s->stream));
		return PPC_OK;
	}
	invalidate_bins(s);
	// slots were rewritten: the next rebuild counts by slot
	PPC_CUDA(cudaMemsetAsync(v.order_valid, 0, sizeof(int32_t), s->stream));
	PPC_CUDA(cudaStreamSynchronize(s->stream));
	return PPC_OK;
}

// whether a download queues copies into vectors, all of them page-locked
bool vectors_page_locked(const ppc_agents* a)
{
	bool any = false;
	for (const double* p : { a->positions, a->velocities, a->previous_velocities, a->orientation })
	{
		if (p && !mapped(p))
			return false;
		any = any || p;
	}
	return any;
}

// queues the copies of agents [first, n) of replicate r into the host view
// (columns that landed are copied on, the rest is not waited for)
int copy_out(ppc_state* s, int32_t r, ppc_agents* a, int32_t first, int32_t n)
{
	const int32_t base = s->reps[r].base;
	const int D = s->ndefs;
	view& v = s->v;
	s->landing = s->bounce && (size_t)(n - first) * sizeof(double) >= kBounceLeast && vectors_page_locked(a);
	PPC_TRY(get_vec(s, a->positions, v.pos[s->cur], r, first, n));
	PPC_TRY(get_vec(s, a->velocities, v.vel, r, first, n));
	PPC_TRY(get_vec(s, a->previous_velocities, v.vprev, r, first, n));
	PPC_TRY(get_vec(s, a->orientation, v.orient, r, first, n));
	PPC_TRY(get_prm(s, 0, a->radius, r, first, n));
	PPC_TRY(get_prm(s, 1, a->cell_cell_repulsion_strength, r, first, n));
	PPC_TRY(get_prm(s, 2, a->cell_cell_adhesion_strength, r, first, n));
	PPC_TRY(get_prm(s, 3, a->cell_BM_repulsion_strength, r, first, n));
	PPC_TRY(get_scalar(s, a->relative_maximum_adhesion_distance, v.rmad, base, first, n, 1));
	PPC_TRY(get_scalar(s, a->attachment_elastic_constant, v.ec, base, first, n, 1));
	PPC_TRY(get_scalar(s, a->attachment_rate, v.arate, base, first, n, 1));
	PPC_TRY(get_scalar(s, a->detachment_rate, v.drate, base, first, n, 1));
	PPC_TRY(get_scalar(s, a->simple_pressure, v.pressure, base, first, n, 1));
	PPC_TRY(get_scalar(s, a->total_volume, v.vol, base, first, n, 1));
	PPC_TRY(get_scalar(s, a->nuclear_volume, v.nvol, base, first, n, 1));
	PPC_TRY(get_scalar(s, a->nuclear_radius, v.nrad, base, first, n, 1));
	PPC_TRY(get_scalar(s, a->surface_area, v.sarea, base, first, n, 1));
	PPC_TRY(get_scalar(s, a->polarity, v.polarity, base, first, n, 1));
	PPC_TRY(get_scalar(s, a->cell_adhesion_affinities, v.aff, base, first, n, D));
	PPC_TRY(get_scalar(s, a->cell_definition_indices, v.def, base, first, n, 1));
	PPC_TRY(get_scalar(s, a->maximum_number_of_attachments, v.maxatt, base, first, n, 1));
	PPC_TRY(get_scalar(s, a->is_movable, v.movable, base, first, n, 1));
	PPC_TRY(get_scalar(s, a->flags, v.flags, base, first, n, 1));
	PPC_TRY(get_scalar(s, a->agent_ids, v.ids, base, first, n, 1));
	// the vectors' copies last, so that the host copies of the columns that
	// landed before them run beside these
	const bool landed = !s->pending_host.empty();
	if (landed)
		PPC_CUDA(cudaEventRecord(s->ev_landed, s->stream));
	PPC_TRY(flush_copies(s));
	if (landed)
	{
		PPC_CUDA(cudaEventSynchronize(s->ev_landed));
		drain_host(s);
	}
	return PPC_OK;
}

int transfer_out_on(ppc_state* s, int32_t r, ppc_agents* a, cudaStream_t main, bool beside)
{
	// Copies as many agents as this host last saw in the replicate, together
	// with the counters and the device error word, and synchronises once; if
	// the device count turns out larger (divisions since), the agents beyond
	// are copied then. Rows between the device count and the
	// previous count, within the host capacity, may be overwritten.
	stage_reset(s);
	const int32_t guess = std::max(0, std::min(s->host_count[r], std::min(a->capacity, s->reps[r].cap)));
	s->pull.count = 0;
	s->pulling = (size_t)guess * s->dims * sizeof(double) <= kSmallRows;
	const size_t head = sizeof(rep_counters) * (s->nreps + 1); // the counters and the error word
	if (!pull_column(s, s->pinned_ctr, s->v.ctr, head, 0))
		PPC_CUDA(cudaMemcpyAsync(s->pinned_ctr, s->v.ctr, head, cudaMemcpyDeviceToHost, s->stream));
	const int rc = copy_out(s, r, a, 0, guess);
	s->pulling = false;
	PPC_TRY(rc);
	PPC_TRY(launch_pull(s));
	PPC_CUDA(cudaStreamSynchronize(s->stream));
	if (beside && *s->pinned_err)
	{
		// the rebuild beside the copies may still set error bits: read the
		// word after the main stream
		s->stream = main;
		PPC_TRY(device_errors(s));
	}
	else
		PPC_TRY(map_errors(s, *s->pinned_err));
	for (int32_t k = 0; k < s->nreps; k++)
		s->host_count[k] = s->pinned_ctr[k].count;
	s->counts_known = true;
	const int32_t n = s->host_count[r];
	a->count = n;
	if (n > a->capacity)
		return fail(PPC_ERR_CAPACITY, "host arrays are smaller than the agent count");
	if (n > guess)
		PPC_TRY(copy_out(s, r, a, guess, n));
	const int32_t base = s->reps[r].base;
	view& v = s->v;
	s->landing = false;
	if (a->spring_counts)
	{
		PPC_TRY(get_scalar(s, a->spring_counts, v.scnt, base, 0, n, 1));
		PPC_CUDA(cudaStreamSynchronize(s->stream));
		int32_t mx = 0;
		for (int32_t i = 0; i < n; i++)
			mx = std::max(mx, a->spring_counts[i]);
		if (mx > a->spring_capacity)
			return fail(PPC_ERR_CAPACITY, "host spring rows are shorter than a spring list");
		if (a->springs && n)
		{
			const size_t bytes = (size_t)n * a->spring_capacity * sizeof(int32_t);
			void* st = nullptr;
			PPC_TRY(stage_take(s, bytes, &st));
			PPC_TRY(launch_springs_local(s, r, n, static_cast<int32_t*>(st), a->spring_capacity, 0));
			PPC_TRY(copy_down(s, a->springs, st, bytes));
		}
	}
	if (n > guess || a->spring_counts)
		PPC_CUDA(cudaStreamSynchronize(s->stream));
	return PPC_OK;
}

// A download right after a step (no kernel launched since) runs on the
// transfer stream once the step's agent fields are final (ev_ready), beside
// the rest of the step's mesh rebuild, which changes none of them; any other
// download runs on the stream.
int transfer_out(ppc_state* s, int32_t r, ppc_agents* a)
{
	const bool beside = s->ready_pending && s->launches == s->ready_launches && s->xfer;
	s->ready_pending = false;
	cudaStream_t main = s->stream;
	if (beside)
	{
		PPC_CUDA(cudaStreamWaitEvent(s->xfer, s->ev_ready, 0));
		s->stream = s->xfer;
	}
	const int rc = transfer_out_on(s, r, a, main, beside);
	s->stream = main;
	return rc;
}

int ensure_bins(ppc_state* s)
{
	if (!s->bins_valid)
	{
		PPC_TRY(launch_bin(s, s->bins_cond));
		s->bins_valid = true;
		s->bins_cond = false;
	}
	return PPC_OK;
}

bool stochastic_springs(ppc_state* s) { return s->params.automated_spring_adhesion && s->rates_nonzero; }

// The fused step recomputes neighbours inside its force pass and does not
// store them; the lists the reference would hold after the step are built
// here when a consumer needs them.
int ensure_lists(ppc_state* s)
{
	if (s->lists_stale)
	{
		PPC_TRY(ensure_bins(s));
		PPC_TRY(launch_neighbors(s));
		s->lists_stale = false;
	}
	return PPC_OK;
}

// one fused mechanics step (+ phenotype container update); `last`: the last
// step of a call, whose agent fields a download may read beside its rebuild
int enqueue_step(ppc_state* s, bool phenotype, double p_divide, double p_death, bool last)
{
	if (s->persistent && !phenotype)
		return launch_step_persistent(s);
	// a compaction leaves its moves to the kernel that visits every agent
	// after it: k_phenotype, or k_bin_count of the rebuild;
	// in a step without the phenotype update the fused passes -3 and -4 also
	// make the count's entries, which hold unless the compaction removes agents
	const bool produce = !phenotype && (s->flat || s->queue);
	s->produce = produce;
	const int rc_fused = launch_fused(s);
	s->produce = false;
	PPC_TRY(rc_fused);
	PPC_TRY(launch_compact(s, false, true, produce));
	if (phenotype)
	{
		PPC_TRY(launch_phenotype(s, true, p_divide, p_death));
		PPC_TRY(launch_compact(s, true, true));
	}
	PPC_TRY(launch_bin(s, false, last, produce));
	return PPC_OK;
}

// One step with stochastic spring attachment: the spring update needs every
// agent's neighbours and its attachments must be settled before the springs
// pull, so the step is a scan, the settlement, and the rest (the order of
// simulator::simulate_mechanics, src/simulator.cpp:173-192, holds within each
// agent's sums). 88,700 agents with every rate on: 114 us a step as the entry
// points' kernels one after another, 83 us so.
int enqueue_step_springs(ppc_state* s, bool phenotype, double p_divide, double p_death, bool last)
{
	s->produce = !phenotype;
	const int rc = launch_spring_step(s);
	s->produce = false;
	PPC_TRY(rc);
	// the scan and k_spring_step read spring rows by slot, so only a call's
	// last rebuild copies their counts into the key order
	if (last)
		PPC_TRY(mark_fields_changed(s));
	PPC_TRY(launch_compact(s, false, true, !phenotype));
	if (phenotype)
	{
		PPC_TRY(launch_phenotype(s, true, p_divide, p_death));
		PPC_TRY(launch_compact(s, true, true));
	}
	PPC_TRY(launch_bin(s, false, last, !phenotype));
	return PPC_OK;
}

constexpr int kGraphSteps = 10; // steps per replay of a long run's graph
constexpr size_t kGraphCache = 8; // captured graphs kept per state

// Replays `k` fused steps from a captured graph, capturing it on first use.
// A graph is keyed by everything its kernels' variants and arguments depend
// on: the step count, the position buffer it starts from, the phenotype
// update and its probabilities, springs, and whether it starts with the
// conditional mesh rebuild an upload of positions leaves for the device.
int replay_steps(ppc_state* s, int k, bool phenotype, double p_divide, double p_death, bool lead_bin)
{
	graph_entry* hit = nullptr;
	for (auto& e : s->graphs)
		if (e.steps == k && e.cur == s->cur && e.sbuf == s->sbuf && e.phenotype == phenotype && e.pdiv == p_divide && e.pdeath == p_death
			&& e.lead_bin == lead_bin && e.springs == s->has_springs)
			hit = &e;
	if (!hit)
	{
		if (s->graphs.size() >= kGraphCache)
			PPC_TRY(release_graph(s));
		graph_entry e {};
		e.steps = k;
		e.cur = s->cur;
		e.sbuf = s->sbuf;
		e.phenotype = phenotype;
		e.pdiv = p_divide;
		e.pdeath = p_death;
		e.lead_bin = lead_bin;
		e.springs = s->has_springs;
		const int cur0 = s->cur;
		const int64_t l0 = s->launches;
		cudaGraph_t g = nullptr;
		PPC_CUDA(cudaStreamBeginCapture(s->stream, cudaStreamCaptureModeThreadLocal));
		int rc = lead_bin ? launch_bin(s, true) : PPC_OK;
		for (int q = 0; q < k && rc == PPC_OK; q++)
			rc = enqueue_step(s, phenotype, p_divide, p_death, q == k - 1);
		e.ready = s->ready_recorded;
		if (s->join_pending)
		{
			// the transfer stream's branch rejoins before the capture ends
			s->join_pending = false;
			if (cudaEventRecord(s->ev_join, s->xfer) != cudaSuccess
				|| cudaStreamWaitEvent(s->stream, s->ev_join, 0) != cudaSuccess)
				rc = fail(PPC_ERR_CUDA, "joining the transfer stream into the step graph failed");
		}
		cudaError_t ec = cudaStreamEndCapture(s->stream, &g);
		s->cur = cur0;
		e.sflip = s->sbuf ^ e.sbuf;
		if (e.sflip)
			flip_sorted_positions(s);
		if (rc != PPC_OK)
		{
			if (g)
				cudaGraphDestroy(g);
			return rc;
		}
		if (ec != cudaSuccess)
			return cuda_fail(ec, "cudaStreamEndCapture");
		ec = cudaGraphInstantiate(&e.exec, g, 0);
		cudaGraphDestroy(g);
		if (ec != cudaSuccess)
			return cuda_fail(ec, "cudaGraphInstantiate");
		e.launches = s->launches - l0;
		s->launches = l0;
		s->graphs.push_back(e);
		hit = &s->graphs.back();
	}
	PPC_CUDA(cudaGraphLaunch(hit->exec, s->stream));
	s->launches += hit->launches;
	s->ready_recorded = hit->ready;
	s->cur ^= k & 1;
	if (hit->sflip)
		flip_sorted_positions(s);
	s->vel_dirty = false;
	return PPC_OK;
}

// The lists' arrays, about 1.2 KB a slot. States of up to kListEarly slots have
// them in the one block of their arrays (120 MB at most), where they cost next to
// nothing to allocate; a second block in the first call that uses them takes 0.4
// to 1 ms, more than a call of 60 steps gains. In larger states, of which many
// never use them (they divide, settle springs, step once a call), they come with
// that call. A device without room for them runs every step through the scanning
// passes.
constexpr int32_t kListEarly = 100000;

void want_lists(ppc_state* s, arena& a)
{
	const size_t C = s->total_cap;
	view& v = s->v;
	// A warp's lists take as many entries a slot as the longest of them: 16 at one
	// agent of radius 7 to 10 um per 8,000 um^3 with the full skin, 20 at one per
	// 6,000, 28 at one per 4,000, whose second attempt, with 0.6 of the skin, takes
	// 23. Denser tissue gets smaller skins, and beyond one per 3,000 none.
	v.nl_pool = 24 * (int64_t)C + 8192;
	a.want(v.nl_used, 1);
	a.want(s->list_bar, 64);
	a.want(v.lpos[0], C, false);
	a.want(v.lpos[1], C, false);
	a.want(v.lvprev, C, false);
	a.want(v.lpress, C, false);
	a.want(v.nlc, C, false);
	a.want(v.nl_slab, C / 32 + 1, false);
	a.want(v.nl, v.nl_pool, false);
	a.want(v.nl_pair, v.nl_pool, false);
	a.want(v.lspr, C * s->scap, false);
	a.want(v.lcoef, C * s->scap, false);
	a.want(v.tpos, C, false);
}

bool lists_allocated(ppc_state* s)
{
	if (s->lists_tried)
		return s->lists_fit;
	s->lists_tried = true;
	arena a;
	want_lists(s, a);
	// a capture on another stream of the program stays valid
	cudaStreamCaptureMode mode = cudaStreamCaptureModeRelaxed;
	cudaThreadExchangeStreamCaptureMode(&mode);
	s->lists_fit = a.place(s) == PPC_OK;
	cudaThreadExchangeStreamCaptureMode(&mode);
	if (!s->lists_fit)
		cudaGetLastError(); // no room is not an error of the state
	return s->lists_fit;
}

static_assert(sizeof(rep_counters) >= 4 * sizeof(int32_t), "the error word and three spare words end the counters");

constexpr int kListLeast = 4;	   // steps of a call that run over lists
constexpr int kListHold = 32;	   // calls at most between two attempts
constexpr float kSkinUnknown = 1e30f;
constexpr int kListSteps = 100000; // steps of one launch over lists

// Whether a call's steps run over neighbour lists: the default launch shape or
// the autotuner's (a caller's choice of another one asks for its own pass), and
// a mesh that leaves a skin beyond the largest reach (by the uploaded fields).
// The launch itself
// costs about 13 us over its steps and making lists about as much as one scanning
// step, so calls of a few steps keep the scanning passes. 88,700 agents, calls of
// four steps in a row: 48 us a call over lists, 125 scanning; each followed by a
// neighbour query, which takes the mesh back: 123 and 159 us.
bool use_lists(ppc_state* s, int32_t steps)
{
	if ((s->lists_tried && !s->lists_fit) || s->scan_only || s->persistent || s->profiling || steps < kListLeast)
		return false;
	double voxel = 1e30;
	for (const auto& R : s->reps)
		for (int d = 0; d < s->dims; d++)
			voxel = std::min(voxel, R.shape[d]);
	for (int32_t r = 0; r < s->nreps; r++)
		if (!(2.0 * s->reach_radius[r] * s->reach_factor[r] + 1.0 < voxel))
			return false;
	// a stream under capture is left to the replayed steps, which refuse it
	cudaStreamCaptureStatus cs = cudaStreamCaptureStatusNone;
	if (cudaStreamIsCapturing(s->stream, &cs) != cudaSuccess || cs != cudaStreamCaptureStatusNone)
		return false;
	// Lists that the device gave up (they did not fit, had no skin or did not
	// pay) are tried again after one call, then two, four and so on: the call
	// that gives them up takes longer than scanning would (20 steps of 14,300
	// agents 1.58 and 1.48 ms, 60 steps 4.5 and 3.5).
	volatile float* skin = s->pinned_skin;
	if (*skin == 0.f)
	{
		s->list_hold = s->list_wait = std::min(kListHold, std::max(1, 2 * s->list_wait));
		*skin = kSkinUnknown;
	}
	else if (*skin < kSkinUnknown)
		s->list_wait = 0;
	if (s->list_hold == 0)
		return lists_allocated(s);
	s->list_hold--;
	return false;
}

int run_list_steps(ppc_state* s, int32_t steps)
{
	if (!s->skin_lists)
	{
		PPC_TRY(ensure_bins(s));
		PPC_TRY(launch_lists(s));
	}
	for (int32_t done = 0; done < steps;)
	{
		const int32_t k = std::min(steps - done, (int32_t)kListSteps);
		PPC_TRY(launch_list_steps(s, k));
		done += k;
	}
	s->bins_valid = false; // the mesh stays that of the lists
	s->bins_cond = false;
	s->lists_stale = true;
	return PPC_OK;
}

// after a call's last step: a download may run beside its rebuild while no
// other kernel is launched
int mark_ready(ppc_state* s)
{
	s->ready_pending = s->ready_recorded;
	s->ready_launches = s->launches;
	return PPC_OK;
}

int run_steps(ppc_state* s, int32_t steps, bool phenotype, double p_divide, double p_death)
{
	if (steps < 0)
		return fail(PPC_ERR_ARG, "negative step count");
	if (s->lost)
		return fail(PPC_ERR_ARG, "a bounded device wait gave up in an earlier step: upload the state again");
	if (steps > 0)
		s->counts_known = false; // compaction and division change the counts
	s->ready_pending = false;
	s->ready_recorded = false;
	if (!phenotype && !stochastic_springs(s) && use_lists(s, steps))
		return run_list_steps(s, steps);
	const bool graphs = s->use_graphs && !s->profiling;
	// a rebuild the device decides on (after an upload of positions) rides
	// at the head of the first replayed graph
	bool lead_bin = graphs && steps > 0 && !s->bins_valid && s->bins_cond && !s->vel_dirty && !stochastic_springs(s);
	if (!lead_bin)
		PPC_TRY(ensure_bins(s));
	s->bins_valid = true;
	s->bins_cond = false;
	if (stochastic_springs(s))
	{
		// non-zero attachment or detachment rates
		s->has_springs = true;
		for (int32_t k = 0; k < steps; k++)
			PPC_TRY(enqueue_step_springs(s, phenotype, p_divide, p_death, k == steps - 1));
		s->lists_stale = steps > 0 || s->lists_stale;
		return mark_ready(s);
	}
	int32_t done = 0;
	// the first step after an upload may read non-zero velocities
	while (done < steps && s->vel_dirty)
	{
		PPC_TRY(enqueue_step(s, phenotype, p_divide, p_death, done == steps - 1));
		done++;
	}
	if (graphs)
	{
		while (steps - done >= kGraphSteps)
		{
			PPC_TRY(replay_steps(s, kGraphSteps, phenotype, p_divide, p_death, lead_bin));
			lead_bin = false;
			done += kGraphSteps;
		}
		while (done < steps)
		{
			PPC_TRY(replay_steps(s, 1, phenotype, p_divide, p_death, lead_bin));
			lead_bin = false;
			done++;
		}
	}
	while (done < steps)
	{
		PPC_TRY(enqueue_step(s, phenotype, p_divide, p_death, done == steps - 1));
		done++;
	}
	s->lists_stale = steps > 0 || s->lists_stale;
	return mark_ready(s);
}

// grid of a mesh (validated: positive voxel shapes, maxs >= mins); sizes in
// 64-bit arithmetic, saturated at INT32_MAX per axis and in the product, so
// an oversized mesh is rejected by the caller's voxel limit instead of
// wrapping
void mesh_info(const ppc_mesh& m, rep_info& R)
{
	R.voxels = 1;
	for (int d = 0; d < 3; d++)
	{
		R.mins[d] = m.bounding_box_mins[d];
		R.maxs[d] = m.bounding_box_maxs[d];
		R.mins_int[d] = m.bounding_box_mins[d];
		R.maxs_int[d] = m.bounding_box_maxs[d];
		R.shape[d] = m.voxel_shape[d];
		int64_t g = 1;
		if (d < m.dims && m.voxel_shape[d] > 0)
			g = ((int64_t)m.bounding_box_maxs[d] - (int64_t)m.bounding_box_mins[d] + m.voxel_shape[d] - 1)
				/ m.voxel_shape[d];
		g = std::min<int64_t>(std::max<int64_t>(g, 1), INT32_MAX);
		R.grid[d] = (int32_t)g;
		R.voxels = std::min<int64_t>(R.voxels * g, (int64_t)INT32_MAX + 1);
	}
}

} // namespace
} // namespace ppc

using namespace ppc;

extern "C" {

const char* ppc_last_error(void) { return g_last_error.c_str(); }

int ppc_abi_version(void) { return PPC_ABI_VERSION; }

int ppc_create_batch(const ppc_mesh* meshes, const int32_t* capacities, int32_t replicates, const ppc_params* params,
					 ppc_state** out)
{
	if (!meshes || !capacities || !params || !out || replicates < 1)
		return fail(PPC_ERR_ARG, "null argument or no replicates");
	const int dims = meshes[0].dims;
	if (dims < 1 || dims > 3 || params->cell_definitions_count < 1 || params->mechanics_time_step <= 0)
		return fail(PPC_ERR_ARG, "dims must be 1..3, cell definitions >= 1, time step > 0");
	int ndev = 0;
	if (cudaGetDeviceCount(&ndev) != cudaSuccess || ndev == 0)
		return fail(PPC_ERR_NO_DEVICE, "no CUDA device");

	auto* s = new ppc_state;
	s->dims = dims;
	s->ndefs = params->cell_definitions_count;
	s->nreps = replicates;
	s->params = *params;
	int64_t vox = 0;
	int64_t cap = 0;
	for (int32_t r = 0; r < replicates; r++)
	{
		if (meshes[r].dims != dims || capacities[r] < 0)
		{
			delete s;
			return fail(PPC_ERR_ARG, "replicates must share dims; capacities must be >= 0");
		}
		for (int d = 0; d < dims; d++)
			if (meshes[r].voxel_shape[d] <= 0 || meshes[r].bounding_box_maxs[d] < meshes[r].bounding_box_mins[d])
			{
				delete s;
				return fail(PPC_ERR_ARG, "invalid mesh");
			}
		rep_info R {};
		mesh_info(meshes[r], R);
		{
			// positions relative to the box minimum reach about the extent; the
			// FP32 filter tolerates 16 float ulps of it per coordinate
			double ext = 1.0;
			for (int d = 0; d < dims; d++)
				ext = std::max(ext, (double)(R.maxs[d] - R.mins[d]) + 2.0 * R.shape[d]);
			int e2 = 0;
			std::frexp(ext, &e2);
			R.fmargin = (float)std::ldexp(16.0, e2 - 24);
		}
		R.inv_grid[0] = 1.0 / R.grid[0];
		R.inv_grid[1] = 1.0 / R.grid[1];
		for (int d = 0; d < 3; d++)
			R.inv_shape[d] = 1.0 / std::max(R.shape[d], 1.0);
		R.base = (int32_t)cap;
		R.cap = capacities[r];
		R.vox_base = vox;
		vox += R.voxels;
		cap += capacities[r];
		s->reps.push_back(R);
		s->meshes.push_back(meshes[r]);
	}
	if (cap > INT32_MAX / 2 || vox > INT32_MAX)
	{
		delete s;
		return fail(PPC_ERR_CAPACITY, "agent capacity or voxel count exceeds 32-bit indexing");
	}
	s->total_cap = (int32_t)std::max<int64_t>(cap, 1);
	s->total_voxels = vox;

	cudaGetDevice(&s->device);
	cudaDeviceGetAttribute(&s->sm_count, cudaDevAttrMultiProcessorCount, s->device);
	int rc = PPC_OK;
	auto try_ = [&](int x) {
		if (rc == PPC_OK)
			rc = x;
	};
	if (cudaStreamCreateWithFlags(&s->own_stream, cudaStreamNonBlocking) != cudaSuccess)
		rc = fail(PPC_ERR_CUDA, "cudaStreamCreate failed");
	s->stream = s->own_stream;
	if (rc == PPC_OK
		&& (cudaStreamCreateWithFlags(&s->xfer, cudaStreamNonBlocking) != cudaSuccess
			|| cudaEventCreateWithFlags(&s->ev_ready, cudaEventDisableTiming) != cudaSuccess
			|| cudaEventCreateWithFlags(&s->ev_h2d, cudaEventDisableTiming) != cudaSuccess
			|| cudaEventCreateWithFlags(&s->ev_stage_free, cudaEventDisableTiming) != cudaSuccess
			|| cudaEventCreateWithFlags(&s->ev_fork, cudaEventDisableTiming) != cudaSuccess
			|| cudaEventCreateWithFlags(&s->ev_join, cudaEventDisableTiming) != cudaSuccess
			|| cudaEventCreateWithFlags(&s->ev_landed, cudaEventDisableTiming) != cudaSuccess))
		rc = fail(PPC_ERR_CUDA, "cudaStreamCreate or cudaEventCreate failed");

	view& v = s->v;
	const size_t C = s->total_cap;
	v.dims = dims;
	v.ndefs = s->ndefs;
	v.nreps = replicates;
	v.total_cap = s->total_cap;
	v.scap = s->scap;
	v.ncap = s->ncap;
	v.dt = params->mechanics_time_step;
	v.walls = params->virtual_wall_at_domain_edges;
	v.auto_springs = params->automated_spring_adhesion != 0;
	rep_info* reps = nullptr;
	arena a;
	a.want(reps, replicates);
	// the error word sits right after the counters, so one copy brings both
	a.want(v.ctr, (size_t)replicates + 1);
	a.want(v.cursor, 1);
	v.nvox = (int32_t)vox;
	{
		// rebuild tiles of about 512 agents at full capacity, 64 to 4096 voxels
		const double want = 512.0 * (double)std::max<int64_t>(vox, 1) / (double)std::max<int64_t>(cap, 1);
		const int sh = (int)std::lround(std::log2(std::max(want, 1.0)));
		v.tshift = std::min(12, std::max(6, sh));
	}
	v.ntiles = (int32_t)((vox + (1 << v.tshift) - 1) >> v.tshift);
	a.want(v.pos[0], C);
	a.want(v.pos[1], C);
	a.want(v.vel, C);
	a.want(v.vprev, C);
	a.want(v.prm, C);
	a.want(v.rmad, C);
	a.want(v.ec, C);
	a.want(v.arate, C);
	a.want(v.drate, C);
	a.want(v.pressure, C);
	a.want(v.vol, C);
	a.want(v.nvol, C);
	a.want(v.nrad, C);
	a.want(v.sarea, C);
	a.want(v.polarity, C);
	a.want(v.orient, C);
	a.want(v.aff, C * s->ndefs);
	a.want(v.def, C);
	a.want(v.maxatt, C);
	a.want(v.scnt, C);
	a.want(v.springs, C * s->scap);
	a.want(v.movable, C);
	a.want(v.flags, C);
	a.want(v.ids, C);
	a.want(v.rid, C);
	a.want(v.vstart, (size_t)vox + 1);
	a.want(v.key, C);
	a.want(v.tmp, C);
	a.want(v.vsc, C);
	a.want(v.tprev, (size_t)v.ntiles);
	a.want(v.tdelta, (size_t)v.ntiles);
	a.want(v.sdelta, ((size_t)v.ntiles + 1023) / 1024);
	a.want(v.skeep, C);
	a.want(v.chead, (size_t)v.ntiles * 32);
	a.want(v.cnext, C);
	a.want(v.porder, C);
	a.want(v.tfresh, C);
	a.want(v.params_changed, 1);
	a.want(v.copy_full, 1);
	a.want(v.recount, 1);
	a.want(v.order_valid, 1);
	a.want(v.binned, replicates);
	a.want(v.moves_pending, 1);
	a.want(v.appended, 1);
	a.want(v.move_src, C); // -1: no pending move into the slot
	a.want(v.sdel, C * s->scap);
	a.want(v.first_end, C);
	a.want(v.pos_changed, 1);
	a.want(v.bin_active, 1);
	a.want(v.barrier, 2);
	a.want(v.sorted, C);
	a.want(v.skey, C);
	a.want(v.spos4, C);
	a.want(v.spos4_next, C);
	a.want(v.sprm4, C);
	a.want(v.sposf, C);
	a.want(v.sposf_next, C);
	a.want(v.sprmf, C);
	a.want(v.safff, C * s->ndefs);
	a.want(v.saff, C * s->ndefs);
	a.want(v.ncnt, C);
	a.want(v.lctl, 16);
	s->reach_radius.assign(replicates, kRadius);
	s->reach_factor.assign(replicates, 1.25);
	a.want(v.bad, C);
	a.want(v.divl, C);
	a.want(v.moves, 2 * C);
	a.want(v.nmoves, replicates);
	a.want(v.draw_epoch, replicates);
	if (rc == PPC_OK && s->total_cap <= kListEarly)
	{
		arena both = a;
		want_lists(s, both);
		s->lists_fit = s->lists_tried = both.place(s) == PPC_OK;
		if (!s->lists_fit)
			cudaGetLastError(); // the state may fit without them
	}
	if (!s->lists_fit)
		try_(rc == PPC_OK ? a.place(s) : rc);
	if (rc == PPC_OK)
	{
		v.reps = reps;
		v.err = reinterpret_cast<int32_t*>(v.ctr + replicates);
		// its own block: ppc_set_neighbor_capacity replaces it
		void* lists = nullptr;
		const size_t bytes = C * s->ncap * sizeof(int32_t);
		if (cudaMalloc(&lists, bytes) != cudaSuccess)
			rc = fail(PPC_ERR_CUDA, "cudaMalloc failed");
		else
		{
			s->allocations.push_back({ lists, bytes });
			v.nidx = static_cast<int32_t*>(lists);
		}
	}
	if (rc == PPC_OK && cudaMemsetAsync(v.chead, 0xff, sizeof(int32_t) * (size_t)v.ntiles * 32, s->stream) != cudaSuccess)
		rc = fail(PPC_ERR_CUDA, "cudaMemset failed");
	if (rc == PPC_OK && cudaMemsetAsync(v.first_end, 0x7f, sizeof(int32_t) * std::max<size_t>(C, 1), s->stream) != cudaSuccess)
		rc = fail(PPC_ERR_CUDA, "cudaMemset failed");
	if (rc == PPC_OK && cudaMemsetAsync(v.move_src, 0xff, sizeof(int32_t) * std::max<size_t>(C, 1), s->stream) != cudaSuccess)
		rc = fail(PPC_ERR_CUDA, "cudaMemset failed");
	s->host_count.assign(replicates, 0);
	if (rc == PPC_OK
		&& cudaHostAlloc(reinterpret_cast<void**>(&s->pinned_ctr), sizeof(rep_counters) * (replicates + 2),
						 cudaHostAllocMapped)
			   != cudaSuccess)
		rc = fail(PPC_ERR_CUDA, "cudaHostAlloc failed");
	if (rc == PPC_OK)
	{
		// a landing area for states whose columns are large enough to use it
		const size_t column = sizeof(double) * C;
		if (column >= kBounceLeast)
		{
			s->bounce_bytes = std::min(kBounceMost, 2 * column);
			if (cudaHostAlloc(&s->bounce, s->bounce_bytes, cudaHostAllocDefault) != cudaSuccess)
			{
				cudaGetLastError(); // downloads then leave the copies to the driver
				s->bounce = nullptr;
			}
		}
		s->pinned_err = reinterpret_cast<int32_t*>(s->pinned_ctr + replicates);
		s->pinned_skin = reinterpret_cast<float*>(s->pinned_ctr + replicates + 1);
		*s->pinned_skin = kSkinUnknown;
	}
	if (rc == PPC_OK)
	{
		std::vector<int32_t> rid(C, 0);
		for (int32_t r = 0; r < replicates; r++)
			for (int32_t k = 0; k < s->reps[r].cap; k++)
				rid[s->reps[r].base + k] = r;
		if (cudaMemcpyAsync(v.rid, rid.data(), C * sizeof(int32_t), cudaMemcpyHostToDevice, s->stream) != cudaSuccess
			|| cudaMemcpyAsync(reps, s->reps.data(), sizeof(rep_info) * replicates, cudaMemcpyHostToDevice, s->stream)
				   != cudaSuccess
			|| cudaStreamSynchronize(s->stream) != cudaSuccess)
			rc = fail(PPC_ERR_CUDA, "initial copy failed");
	}
	if (rc != PPC_OK)
	{
		ppc_destroy(s);
		return rc;
	}
	*out = s;
	return PPC_OK;
}

int ppc_create(const ppc_mesh* mesh, const ppc_params* params, int32_t agent_capacity, ppc_state** out)
{
	return ppc_create_batch(mesh, &agent_capacity, 1, params, out);
}

int ppc_destroy(ppc_state* s)
{
	if (!s)
		return PPC_OK;
	if (s->stream)
		cudaStreamSynchronize(s->stream);
	if (s->xfer)
		cudaStreamSynchronize(s->xfer);
	release_graph(s);
	for (auto e : s->prof_events)
		cudaEventDestroy(e);
	for (auto e : { s->ev_ready, s->ev_h2d, s->ev_stage_free, s->ev_fork, s->ev_join, s->ev_landed })
		if (e)
			cudaEventDestroy(e);
	if (s->xfer)
		cudaStreamDestroy(s->xfer);
	for (auto& b : s->allocations)
		cudaFree(b.p);
	if (s->stage)
		cudaFree(s->stage);
	if (s->ix_scratch)
		cudaFree(s->ix_scratch);
	for (auto& b : { s->ix_store.p, s->mot_store.p })
		if (b)
			cudaFree(b);
	for (auto& g : s->gradients)
		if (g.p)
			cudaFree(g.p);
	if (s->pinned_ctr)
		cudaFreeHost(s->pinned_ctr);
	if (s->bounce)
		cudaFreeHost(s->bounce);
	if (s->own_stream)
		cudaStreamDestroy(s->own_stream);
	delete s;
	return PPC_OK;
}

int ppc_set_stream(ppc_state* s, void* stream)
{
	if (!s)
		return fail(PPC_ERR_ARG, "null state");
	PPC_CUDA(cudaStreamSynchronize(s->stream));
	release_graph(s);
	s->stream = stream ? static_cast<cudaStream_t>(stream) : s->own_stream;
	return PPC_OK;
}

int ppc_set_precision(ppc_state* s, int32_t precision)
{
	if (!s || (precision != PPC_FP64 && precision != PPC_FP32_FORCE))
		return fail(PPC_ERR_ARG, "precision must be PPC_FP64 or PPC_FP32_FORCE");
	if (precision == PPC_FP32_FORCE && s->ndefs > 65535)
		return fail(PPC_ERR_UNSUPPORTED, "the FP32-force form packs definition indices in 16 bits");
	PPC_CUDA(cudaStreamSynchronize(s->stream));
	s->precision = precision;
	s->v.f32 = precision == PPC_FP32_FORCE ? 1 : 0;
	invalidate_bins(s); // the single-precision copies are written by the binning
	PPC_TRY(mark_fields_changed(s));
	release_graph(s);
	return PPC_OK;
}

int ppc_set_random_seed(ppc_state* s, uint64_t seed)
{
	if (!s)
		return fail(PPC_ERR_ARG, "null state");
	s->seed = seed;
	s->v.seed = seed;
	release_graph(s);
	return PPC_OK;
}

int ppc_set_launch_shape(ppc_state* s, int32_t tile_edge, int32_t threads, int32_t smem_bytes)
{
	if (!s)
		return fail(PPC_ERR_ARG, "null state");
	if (tile_edge < -4 || tile_edge > 0 || threads < 32 || threads > 256 || threads % 32 != 0 || smem_bytes < 0
		|| smem_bytes > 160 * 1024)
		return fail(PPC_ERR_ARG, "tile edge 0, -1, -2, -3 or -4, threads 32..256 (multiple of 32), smem <= 160 KiB");
	PPC_CUDA(cudaStreamSynchronize(s->stream));
	release_graph(s);
	s->flat = tile_edge == -3;
	s->queue = tile_edge == -4;
	s->scan_only = !s->queue; // a caller's own choice; ppc_autotune's leaves the lists on
	s->staged = tile_edge == 0;
	s->coop = tile_edge == 0 || tile_edge == -2;
	s->tile_threads = threads;
	s->tile_smem = smem_bytes;
	return PPC_OK;
}

int ppc_set_step_form(ppc_state* s, int32_t form)
{
	if (!s || (form != PPC_STEP_KERNELS && form != PPC_STEP_PERSISTENT))
		return fail(PPC_ERR_ARG, "form must be PPC_STEP_KERNELS or PPC_STEP_PERSISTENT");
	int coop = 0;
	if (form == PPC_STEP_PERSISTENT
		&& (cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, s->device) != cudaSuccess || !coop))
		return fail(PPC_ERR_UNSUPPORTED, "the device has no cooperative launch");
	PPC_CUDA(cudaStreamSynchronize(s->stream));
	release_graph(s);
	s->persistent = form == PPC_STEP_PERSISTENT;
	return PPC_OK;
}

int ppc_set_wait_limit(ppc_state* s, int64_t polls)
{
	if (!s || polls < 1)
		return fail(PPC_ERR_ARG, "the wait limit must be at least one poll");
	PPC_CUDA(cudaStreamSynchronize(s->stream));
	release_graph(s);
	s->wait_limit = polls;
	return PPC_OK;
}

int ppc_set_host_transfer(ppc_state* s, int32_t mode)
{
	if (!s || (mode != PPC_TRANSFER_COPY_ENGINE && mode != PPC_TRANSFER_ZERO_COPY))
		return fail(PPC_ERR_ARG, "mode must be PPC_TRANSFER_COPY_ENGINE or PPC_TRANSFER_ZERO_COPY");
	s->zero_copy = mode == PPC_TRANSFER_ZERO_COPY;
	return PPC_OK;
}

int ppc_set_neighbor_capacity(ppc_state* s, int32_t per_agent)
{
	if (!s || per_agent < 1)
		return fail(PPC_ERR_ARG, "neighbour capacity must be >= 1");
	if (per_agent == s->ncap)
		return PPC_OK;
	PPC_CUDA(cudaStreamSynchronize(s->stream));
	int32_t* p = nullptr;
	size_t bytes = (size_t)s->total_cap * per_agent * sizeof(int32_t);
	PPC_CUDA(cudaMalloc(&p, bytes));
	for (auto& b : s->allocations)
		if (b.p == s->v.nidx)
		{
			cudaFree(b.p);
			b.p = p;
			b.bytes = bytes;
		}
	s->v.nidx = p;
	s->v.ncap = s->ncap = per_agent;
	PPC_CUDA(cudaMemsetAsync(s->v.ncnt, 0, sizeof(int32_t) * s->total_cap, s->stream));
	release_graph(s);
	return PPC_OK;
}

} // extern "C"

namespace ppc {
namespace {

// What a step left that gave up at a barrier: arrivals at the barriers, movers
// on the tiles' chains, planned moves, and removal candidates.
int reset_interrupted(ppc_state* s)
{
	const view& v = s->v;
	const size_t C = s->total_cap, tiles = v.ntiles, word = sizeof(int32_t);
	if (s->lists_fit)
		PPC_CUDA(cudaMemsetAsync(s->list_bar, 0, 64 * sizeof(unsigned long long), s->stream));
	PPC_CUDA(cudaMemsetAsync(v.chead, 0xff, 32 * tiles * word, s->stream));
	PPC_CUDA(cudaMemsetAsync(v.tdelta, 0, tiles * word, s->stream));
	PPC_CUDA(cudaMemsetAsync(v.sdelta, 0, (tiles + 1023) / 1024 * word, s->stream));
	PPC_CUDA(cudaMemsetAsync(v.move_src, 0xff, C * word, s->stream));
	for (int32_t* flag : { v.moves_pending, v.appended, v.recount })
		PPC_CUDA(cudaMemsetAsync(flag, 0, word, s->stream));
	for (int32_t r = 0; r < s->nreps; r++)
		PPC_CUDA(cudaMemsetAsync(&v.ctr[r].nbad, 0, word, s->stream));
	return PPC_OK;
}

} // namespace
} // namespace ppc

extern "C" {

int ppc_upload(ppc_state* s, int32_t r, const ppc_agents* a)
{
	if (!valid(s, r) || !a || a->count < 0)
		return fail(PPC_ERR_ARG, "invalid state, replicate or agents");
	if (a->count > s->reps[r].cap)
		return fail(PPC_ERR_CAPACITY, "agent count exceeds the replicate's capacity");
	// a fresh upload resets the replicate's counters except the event totals
	// and the spring-draw epoch
	std::vector<rep_counters> all;
	PPC_TRY(read_counters(s, all));
	rep_counters c {};
	c.divisions = all[r].divisions;
	c.deaths = all[r].deaths;
	c.spring_epoch = all[r].spring_epoch; // the draw streams continue, as in the reference's generator
	PPC_CUDA(cudaMemcpyAsync(&s->v.ctr[r], &c, sizeof c, cudaMemcpyHostToDevice, s->stream));
	PPC_CUDA(cudaStreamSynchronize(s->stream));
	s->lists_stale = false;
	s->skin_reset = true;
	if (s->lost)
		PPC_TRY(reset_interrupted(s));
	s->lost = false;
	return transfer_in(s, r, a, true);
}

int ppc_upload_fields(ppc_state* s, int32_t r, const ppc_agents* a)
{
	if (!valid(s, r) || !a)
		return fail(PPC_ERR_ARG, "invalid state, replicate or agents");
	// the count is read from the device unless no count-changing work was
	// queued since it was last read (a download, typically)
	if (!s->counts_known)
	{
		std::vector<rep_counters> c;
		PPC_TRY(read_counters(s, c));
	}
	if (a->count != s->host_count[r])
		return fail(PPC_ERR_ARG, "count differs from the device count");
	return transfer_in(s, r, a, false);
}

int ppc_download(ppc_state* s, int32_t r, ppc_agents* a)
{
	if (!valid(s, r) || !a)
		return fail(PPC_ERR_ARG, "invalid state, replicate or agents");
	PPC_CUDA(cudaGetLastError());
	return transfer_out(s, r, a); // reads the device error word with the counters
}

int ppc_get_count(ppc_state* s, int32_t r, int32_t* count)
{
	if (!valid(s, r) || !count)
		return fail(PPC_ERR_ARG, "invalid state or replicate");
	std::vector<rep_counters> c;
	PPC_TRY(read_counters(s, c));
	*count = c[r].count;
	return finish(s);
}

int ppc_get_event_counts(ppc_state* s, int32_t r, int64_t* divisions, int64_t* deaths)
{
	if (!valid(s, r))
		return fail(PPC_ERR_ARG, "invalid state or replicate");
	std::vector<rep_counters> c;
	PPC_TRY(read_counters(s, c));
	if (divisions)
		*divisions = c[r].divisions;
	if (deaths)
		*deaths = c[r].deaths;
	return PPC_OK;
}

int ppc_synchronize(ppc_state* s)
{
	if (!s)
		return fail(PPC_ERR_ARG, "null state");
	return finish(s);
}

void* ppc_host_alloc(size_t bytes)
{
	void* p = nullptr;
	if (cudaHostAlloc(&p, std::max<size_t>(bytes, 1), cudaHostAllocDefault) != cudaSuccess)
		return nullptr;
	return p;
}

void ppc_host_free(void* p)
{
	if (p)
		cudaFreeHost(p);
}

int ppc_update_mechanics_mesh(ppc_state* s)
{
	if (!s)
		return fail(PPC_ERR_ARG, "null state");
	PPC_TRY(launch_bin(s, false));
	s->bins_valid = true;
	s->bins_cond = false;
	return finish(s);
}

int ppc_update_cell_neighbors(ppc_state* s)
{
	if (!s)
		return fail(PPC_ERR_ARG, "null state");
	PPC_TRY(ensure_bins(s));
	PPC_TRY(launch_neighbors(s));
	s->lists_stale = false;
	return finish(s);
}

int ppc_update_cell_forces(ppc_state* s)
{
	if (!s)
		return fail(PPC_ERR_ARG, "null state");
	PPC_TRY(ensure_lists(s));
	PPC_TRY(launch_forces(s));
	return finish(s);
}

int ppc_update_motility(ppc_state* s)
{
	if (!s)
		return fail(PPC_ERR_ARG, "null state");
	return PPC_OK;
}

int ppc_update_basement_membrane_interactions(ppc_state* s)
{
	if (!s)
		return fail(PPC_ERR_ARG, "null state");
	if (!s->params.virtual_wall_at_domain_edges)
		return PPC_OK;
	PPC_TRY(launch_membrane(s));
	return finish(s);
}

int ppc_update_spring_attachments(ppc_state* s)
{
	if (!s)
		return fail(PPC_ERR_ARG, "null state");
	if (!s->params.automated_spring_adhesion)
		return PPC_OK;
	// detachment and attachment draws (they advance the draw epoch even when
	// every rate is zero, as the reference's loop does), then the pull
	PPC_TRY(ensure_lists(s));
	PPC_TRY(launch_spring_updates(s));
	s->has_springs = s->has_springs || s->rates_nonzero;
	if (s->has_springs)
		PPC_TRY(launch_springs(s));
	return finish(s);
}

int ppc_update_positions(ppc_state* s)
{
	if (!s)
		return fail(PPC_ERR_ARG, "null state");
	PPC_TRY(launch_positions(s));
	invalidate_bins(s);
	return finish(s);
}

int ppc_update_cell_container_for_mechanics(ppc_state* s)
{
	if (!s)
		return fail(PPC_ERR_ARG, "null state");
	s->counts_known = false;
	PPC_TRY(ensure_lists(s));
	PPC_TRY(launch_mark_remove(s));
	PPC_TRY(launch_compact(s, false));
	invalidate_bins(s);
	return finish(s);
}

int ppc_update_cell_container_for_phenotype(ppc_state* s)
{
	if (!s)
		return fail(PPC_ERR_ARG, "null state");
	s->counts_known = false;
	PPC_TRY(ensure_lists(s));
	PPC_TRY(launch_phenotype(s, false, 0, 0));
	PPC_TRY(launch_compact(s, true));
	invalidate_bins(s);
	return finish(s);
}

int ppc_count_flags(ppc_state* s, int32_t r, int32_t flag, int32_t* count)
{
	if (!valid(s, r) || !count)
		return fail(PPC_ERR_ARG, "invalid arguments");
	int32_t* d = reinterpret_cast<int32_t*>(s->v.err) + 1; // the word after the error word, spare
	PPC_CUDA(cudaMemsetAsync(d, 0, sizeof(int32_t), s->stream));
	PPC_TRY(launch_count_flags(s, r, flag, d));
	PPC_CUDA(cudaMemcpyAsync(s->pinned_err + 1, d, sizeof(int32_t), cudaMemcpyDeviceToHost, s->stream));
	PPC_CUDA(cudaStreamSynchronize(s->stream));
	*count = s->pinned_err[1];
	return finish(s);
}

int ppc_flag_by_draws(ppc_state* s, double p_divide, double p_death)
{
	if (!s)
		return fail(PPC_ERR_ARG, "null state");
	PPC_TRY(launch_flag_by_draws(s, p_divide, p_death));
	return finish(s);
}

// device scratch for the phenotype fields of a per-call entry point, kept
// between calls
static int ensure_field_scratch(ppc_state* s, size_t bytes)
{
	if (bytes <= s->ix_scratch_bytes)
		return PPC_OK;
	if (s->ix_scratch)
	{
		PPC_CUDA(cudaStreamSynchronize(s->stream));
		PPC_CUDA(cudaFree(s->ix_scratch));
		s->ix_scratch = nullptr;
		s->ix_scratch_bytes = 0;
	}
	PPC_CUDA(cudaMalloc(&s->ix_scratch, bytes));
	s->ix_scratch_bytes = bytes;
	return PPC_OK;
}

} // extern "C"

namespace ppc {
namespace {

// one resident column: its device base, the caller's host rows, bytes per
// value and values per agent
struct column
{
	void* dev;
	const void* host;
	size_t elem;
	size_t width;
};

// the interaction columns of `x` paired with the host rows of `f`, in one order
std::vector<column> ix_column_list(const ix_columns& x, const ppc_interactions* f, int D)
{
	const size_t S = (size_t)x.S, d = (size_t)D, e = sizeof(double);
	return {
		{ x.dead, f ? f->dead : nullptr, 1, 1 },
		{ x.dead_phago, f ? f->dead_phagocytosis_rate : nullptr, e, 1 },
		{ x.damage_rate, f ? f->damage_rate : nullptr, e, 1 },
		{ x.live_phago, f ? f->live_phagocytosis_rates : nullptr, e, d },
		{ x.attack, f ? f->attack_rates : nullptr, e, d },
		{ x.fusion, f ? f->fusion_rates : nullptr, e, d },
		{ x.immuno, f ? f->immunogenicities : nullptr, e, d },
		{ x.frac, f ? f->fraction_transferred_when_ingested : nullptr, e, S },
		{ x.damage, f ? f->damage : nullptr, e, 1 },
		{ x.attack_time, f ? f->total_attack_time : nullptr, e, 1 },
		{ x.nuclei, f ? f->number_of_nuclei : nullptr, sizeof(int32_t), 1 },
		{ x.fluid, f ? f->fluid : nullptr, e, 1 },
		{ x.solid, f ? f->solid : nullptr, e, 1 },
		{ x.cyto, f ? f->cytoplasmic : nullptr, e, 1 },
		{ x.cyto_fluid, f ? f->cytoplasmic_fluid : nullptr, e, 1 },
		{ x.cyto_solid, f ? f->cytoplasmic_solid : nullptr, e, 1 },
		{ x.nuc_fluid, f ? f->nuclear_fluid : nullptr, e, 1 },
		{ x.nuc_solid, f ? f->nuclear_solid : nullptr, e, 1 },
		{ x.fluid_fraction, f ? f->fluid_fraction : nullptr, e, 1 },
		{ x.c2n, f ? f->cytoplasmic_to_nuclear_ratio : nullptr, e, 1 },
		{ x.target_cyto, f ? f->target_solid_cytoplasmic : nullptr, e, 1 },
		{ x.target_nuc, f ? f->target_solid_nuclear : nullptr, e, 1 },
		{ x.isub, f ? f->internalized_substrates : nullptr, e, S },
	};
}

std::vector<column> mot_column_list(const mot_columns& m, const ppc_motility* f, int dims)
{
	const size_t e = sizeof(double), d = (size_t)dims;
	return {
		{ m.motile, f ? f->is_motile : nullptr, 1, 1 },
		{ m.restrict2d, f ? f->restrict_to_2d : nullptr, 1, 1 },
		{ m.persistence, f ? f->persistence_time : nullptr, e, 1 },
		{ m.speed, f ? f->migration_speed : nullptr, e, 1 },
		{ m.bias, f ? f->migration_bias : nullptr, e, 1 },
		{ m.direction, f ? f->migration_bias_direction : nullptr, e, d },
		{ m.vector, f ? f->motility_vector : nullptr, e, d },
		{ m.rule, f ? f->direction_rule : nullptr, 1, 1 },
		{ m.chemo_index, f ? f->chemotaxis_index : nullptr, sizeof(int32_t), 1 },
		{ m.chemo_dir, f ? f->chemotaxis_direction : nullptr, e, 1 },
		{ m.sens, f ? f->chemotactic_sensitivities : nullptr, e, (size_t)m.S },
	};
}

// carves the columns out of one zeroed block of C rows; the view changes, so
// captured step graphs are released
int alloc_columns(ppc_state* s, store_block& b, std::vector<std::pair<void**, size_t>> cols)
{
	PPC_CUDA(cudaStreamSynchronize(s->stream));
	PPC_TRY(release_graph(s));
	if (b.p)
	{
		PPC_CUDA(cudaFree(b.p));
		b.p = nullptr;
	}
	size_t total = 0;
	for (auto& c : cols)
		total += (c.second + 255) & ~(size_t)255;
	PPC_CUDA(cudaMalloc(&b.p, std::max<size_t>(total, 1)));
	PPC_CUDA(cudaMemsetAsync(b.p, 0, std::max<size_t>(total, 1), s->stream));
	b.bytes = total;
	char* q = static_cast<char*>(b.p);
	for (auto& c : cols)
	{
		*c.first = q;
		q += (c.second + 255) & ~(size_t)255;
	}
	return PPC_OK;
}

int ensure_ix_store(ppc_state* s, int32_t S)
{
	if (s->ix_store.p && s->v.ix.S == S)
		return PPC_OK;
	const size_t C = s->total_cap, D = s->ndefs, e = sizeof(double);
	ix_columns& x = s->v.ix;
	const int32_t halve = x.halve_sub;
	x = ix_columns {};
	x.S = S;
	x.halve_sub = halve;
	std::vector<std::pair<void**, size_t>> cols = {
		{ (void**)&x.dead, C }, { (void**)&x.nuclei, C * 4 }, { (void**)&x.dead_phago, C * e },
		{ (void**)&x.damage_rate, C * e }, { (void**)&x.live_phago, C * D * e }, { (void**)&x.attack, C * D * e },
		{ (void**)&x.fusion, C * D * e }, { (void**)&x.immuno, C * D * e }, { (void**)&x.frac, C * S * e },
		{ (void**)&x.damage, C * e }, { (void**)&x.attack_time, C * e }, { (void**)&x.fluid, C * e },
		{ (void**)&x.solid, C * e }, { (void**)&x.cyto, C * e }, { (void**)&x.cyto_fluid, C * e },
		{ (void**)&x.cyto_solid, C * e }, { (void**)&x.nuc_fluid, C * e }, { (void**)&x.nuc_solid, C * e },
		{ (void**)&x.fluid_fraction, C * e }, { (void**)&x.c2n, C * e }, { (void**)&x.target_cyto, C * e },
		{ (void**)&x.target_nuc, C * e }, { (void**)&x.isub, C * S * e },
	};
	return alloc_columns(s, s->ix_store, cols);
}

int ensure_mot_store(ppc_state* s, int32_t S)
{
	if (s->mot_store.p && s->v.mot.S == S)
		return PPC_OK;
	const size_t C = s->total_cap, d = s->dims, e = sizeof(double);
	mot_columns& m = s->v.mot;
	const int32_t per_agent = m.per_agent;
	m = mot_columns {};
	m.per_agent = per_agent;
	m.S = S;
	std::vector<std::pair<void**, size_t>> cols = {
		{ (void**)&m.motile, C }, { (void**)&m.restrict2d, C }, { (void**)&m.rule, C },
		{ (void**)&m.persistence, C * e }, { (void**)&m.speed, C * e }, { (void**)&m.bias, C * e },
		{ (void**)&m.direction, C * d * e }, { (void**)&m.vector, C * d * e }, { (void**)&m.chemo_index, C * 4 },
		{ (void**)&m.chemo_dir, C * e }, { (void**)&m.sens, C * (size_t)S * e },
	};
	return alloc_columns(s, s->mot_store, cols);
}

// rows [base, base + n) of the columns from (to_device) or to the host rows
int move_columns(ppc_state* s, const std::vector<column>& cols, int32_t base, int32_t n, bool to_device)
{
	s->landing = false;
	for (const auto& c : cols)
	{
		if (!c.host || c.width == 0 || n == 0)
			continue;
		char* dev = static_cast<char*>(c.dev) + (size_t)base * c.width * c.elem;
		const size_t bytes = (size_t)n * c.width * c.elem;
		if (to_device)
			PPC_CUDA(cudaMemcpyAsync(dev, c.host, bytes, cudaMemcpyHostToDevice, s->stream));
		else
			PPC_TRY(copy_down(s, const_cast<void*>(c.host), dev, bytes));
	}
	PPC_CUDA(cudaStreamSynchronize(s->stream));
	return PPC_OK;
}

int check_ix_fields(const ppc_interactions* f)
{
	const void* all[] = { f->dead, f->dead_phagocytosis_rate, f->damage_rate, f->live_phagocytosis_rates,
						  f->attack_rates, f->fusion_rates, f->immunogenicities, f->damage, f->total_attack_time,
						  f->number_of_nuclei, f->fluid, f->solid, f->cytoplasmic, f->cytoplasmic_fluid,
						  f->cytoplasmic_solid, f->nuclear_fluid, f->nuclear_solid, f->fluid_fraction,
						  f->cytoplasmic_to_nuclear_ratio, f->target_solid_cytoplasmic, f->target_solid_nuclear };
	for (const void* p : all)
		if (!p)
			return fail(PPC_ERR_ARG, "a ppc_interactions field is NULL");
	if (f->substrates > 0 && (!f->internalized_substrates || !f->fraction_transferred_when_ingested))
		return fail(PPC_ERR_ARG, "a ppc_interactions substrate field is NULL");
	return PPC_OK;
}

int check_mot_fields(const ppc_motility* f)
{
	if (!f->is_motile || !f->restrict_to_2d || !f->persistence_time || !f->migration_speed || !f->migration_bias
		|| !f->migration_bias_direction || !f->motility_vector)
		return fail(PPC_ERR_ARG, "a ppc_motility field is NULL");
	if (f->substrates < 0)
		return fail(PPC_ERR_ARG, "negative substrate count");
	if (f->direction_rule
		&& (!f->chemotaxis_index || !f->chemotaxis_direction || (f->substrates > 0 && !f->chemotactic_sensitivities)))
		return fail(PPC_ERR_ARG, "a direction-rule field of ppc_motility is NULL");
	return PPC_OK;
}

// the replicate's live count, read from the device unless already known
int live_count(ppc_state* s, int32_t r, int32_t& n)
{
	if (!s->counts_known)
	{
		std::vector<rep_counters> c;
		PPC_TRY(read_counters(s, c));
	}
	n = s->host_count[r];
	return PPC_OK;
}

} // namespace
} // namespace ppc

extern "C" {

int ppc_upload_interactions(ppc_state* s, int32_t r, const ppc_interactions* f, int32_t compute_internalized_substrates)
{
	if (!valid(s, r) || !f || f->substrates < 0)
		return fail(PPC_ERR_ARG, "invalid arguments");
	int32_t n = 0;
	PPC_TRY(live_count(s, r, n));
	if (f->count != n)
		return fail(PPC_ERR_ARG, "fields.count differs from the replicate's agent count");
	PPC_TRY(check_ix_fields(f));
	if (s->ix_store.p && f->substrates != s->v.ix.S)
		return fail(PPC_ERR_ARG, "substrates differ from the resident interaction fields'");
	PPC_TRY(ensure_ix_store(s, f->substrates));
	if (s->v.ix.halve_sub != (compute_internalized_substrates != 0))
	{
		PPC_CUDA(cudaStreamSynchronize(s->stream));
		PPC_TRY(release_graph(s));
		s->v.ix.halve_sub = compute_internalized_substrates != 0;
	}
	return move_columns(s, ix_column_list(s->v.ix, f, s->ndefs), s->reps[r].base, n, true);
}

int ppc_download_interactions(ppc_state* s, int32_t r, ppc_interactions* f)
{
	if (!valid(s, r) || !f)
		return fail(PPC_ERR_ARG, "invalid arguments");
	if (!s->ix_store.p || f->substrates != s->v.ix.S)
		return fail(PPC_ERR_ARG, "no resident interaction fields with these substrates");
	PPC_CUDA(cudaGetLastError());
	std::vector<rep_counters> c;
	PPC_TRY(read_counters(s, c));
	const int32_t n = c[r].count;
	f->count = n;
	PPC_TRY(check_ix_fields(f));
	return move_columns(s, ix_column_list(s->v.ix, f, s->ndefs), s->reps[r].base, n, false);
}

int ppc_upload_motility(ppc_state* s, int32_t r, const ppc_motility* f)
{
	if (!valid(s, r) || !f)
		return fail(PPC_ERR_ARG, "invalid arguments");
	int32_t n = 0;
	PPC_TRY(live_count(s, r, n));
	if (f->count != n)
		return fail(PPC_ERR_ARG, "fields.count differs from the replicate's agent count");
	PPC_TRY(check_mot_fields(f));
	const int32_t S = f->direction_rule ? f->substrates : (s->mot_store.p ? s->v.mot.S : 0);
	PPC_TRY(ensure_mot_store(s, S));
	if (s->v.mot.per_agent != (f->restrict_per_agent != 0))
	{
		PPC_CUDA(cudaStreamSynchronize(s->stream));
		PPC_TRY(release_graph(s));
		s->v.mot.per_agent = f->restrict_per_agent != 0;
	}
	if (!f->direction_rule && n > 0) // no rules: every agent keeps the caller's direction
		PPC_CUDA(cudaMemsetAsync(s->v.mot.rule + s->reps[r].base, PPC_DIRECTION_NONE, (size_t)n, s->stream));
	return move_columns(s, mot_column_list(s->v.mot, f, s->dims), s->reps[r].base, n, true);
}

int ppc_download_motility(ppc_state* s, int32_t r, ppc_motility* f)
{
	if (!valid(s, r) || !f)
		return fail(PPC_ERR_ARG, "invalid arguments");
	if (!s->mot_store.p)
		return fail(PPC_ERR_ARG, "no resident motility fields");
	PPC_CUDA(cudaGetLastError());
	std::vector<rep_counters> c;
	PPC_TRY(read_counters(s, c));
	const int32_t n = c[r].count;
	f->count = n;
	PPC_TRY(check_mot_fields(f));
	return move_columns(s, mot_column_list(s->v.mot, f, s->dims), s->reps[r].base, n, false);
}

int ppc_update_motility_fields(ppc_state* s, int32_t r, ppc_motility* f)
{
	if (!valid(s, r))
		return fail(PPC_ERR_ARG, "invalid arguments");
	if (f)
		PPC_TRY(ppc_upload_motility(s, r, f)); // fields travel with the call
	else if (!s->mot_store.p)
		return fail(PPC_ERR_ARG, "no resident motility fields: upload them or pass fields");
	const int32_t n = most_rows(s, r); // known where the fields came with the call
	if ((int32_t)s->mot_epoch.size() < s->nreps)
		s->mot_epoch.resize(s->nreps, 0);
	const uint64_t epoch = s->mot_epoch[r]++;
	if (n > 0)
	{
		const int32_t base = s->reps[r].base;
		const mot_columns& mc = s->v.mot;
		const size_t d = (size_t)s->dims;
		mot_fields m {};
		m.n = n;
		m.replicate = r;
		m.base = base;
		m.dt = s->params.mechanics_time_step;
		m.per_agent = mc.per_agent;
		m.cur = s->cur;
		m.epoch = epoch;
		m.motile = mc.motile + base;
		m.restrict2d = mc.restrict2d + base;
		m.rule = mc.rule + base;
		m.persistence = mc.persistence + base;
		m.speed = mc.speed + base;
		m.bias = mc.bias + base;
		m.direction = mc.direction + (size_t)base * d;
		m.vector = mc.vector + (size_t)base * d;
		m.chemo_index = mc.chemo_index + base;
		m.chemo_dir = mc.chemo_dir + base;
		m.S = mc.S;
		m.sens = mc.sens + (size_t)base * mc.S;
		if ((int32_t)s->gradients.size() > r && s->gradients[r].p)
		{
			const auto& g = s->gradients[r];
			m.grad = static_cast<const double*>(g.p);
			m.gS = g.S;
			for (int q = 0; q < 3; q++)
			{
				m.ggrid[q] = g.grid[q];
				m.gshape[q] = g.shape[q];
				m.gmins[q] = s->reps[r].mins[q];
			}
		}
		PPC_TRY(launch_motility(s, m));
		s->vel_dirty = true; // the next fused step reads the velocities
	}
	if (f)
		PPC_TRY(move_columns(s,
							 { { s->v.mot.vector, f->motility_vector, sizeof(double), (size_t)s->dims },
							   { s->v.mot.direction, f->migration_bias_direction, sizeof(double), (size_t)s->dims } },
							 s->reps[r].base, n, false));
	PPC_TRY(finish_counts(s));
	return map_errors(s, *s->pinned_err);
}

int ppc_upload_gradients(ppc_state* s, int32_t r, const ppc_gradient_field* g)
{
	if (!valid(s, r) || !g || g->substrates < 0 || (g->substrates > 0 && !g->gradients))
		return fail(PPC_ERR_ARG, "invalid gradient field");
	ppc_state::gradient_field f;
	f.S = g->substrates;
	int64_t voxels = 1;
	const ppc_mesh& m = s->meshes[r];
	for (int d = 0; d < 3; d++)
	{
		int64_t n = 1;
		if (d < m.dims)
		{
			if (g->voxel_shape[d] <= 0)
				return fail(PPC_ERR_ARG, "diffusion voxel edges must be positive");
			n = ((int64_t)m.bounding_box_maxs[d] - m.bounding_box_mins[d] + g->voxel_shape[d] - 1) / g->voxel_shape[d];
			f.shape[d] = g->voxel_shape[d];
		}
		f.grid[d] = (int32_t)std::max<int64_t>(1, std::min<int64_t>(n, INT32_MAX));
		voxels *= f.grid[d];
		if (voxels > ((int64_t)1 << 31))
			return fail(PPC_ERR_CAPACITY, "the diffusion mesh has too many voxels");
	}
	if ((int32_t)s->gradients.size() < s->nreps)
		s->gradients.resize(s->nreps);
	PPC_CUDA(cudaStreamSynchronize(s->stream));
	if (s->gradients[r].p)
		PPC_CUDA(cudaFree(s->gradients[r].p));
	s->gradients[r] = ppc_state::gradient_field {};
	const size_t bytes = (size_t)voxels * f.S * 3 * sizeof(double);
	if (bytes)
	{
		PPC_CUDA(cudaMalloc(&f.p, bytes));
		PPC_CUDA(cudaMemcpyAsync(f.p, g->gradients, bytes, cudaMemcpyHostToDevice, s->stream));
		PPC_CUDA(cudaStreamSynchronize(s->stream));
	}
	s->gradients[r] = f;
	return PPC_OK;
}

int ppc_update_cell_cell_interactions(ppc_state* s, int32_t r, ppc_interactions* f)
{
	if (!valid(s, r) || (f && f->substrates < 0))
		return fail(PPC_ERR_ARG, "invalid arguments");
	if (f)
	{
		// fields travel with the call: resident for its duration
		if (s->ix_store.p && f->substrates != s->v.ix.S)
			PPC_TRY(ensure_ix_store(s, f->substrates));
		PPC_TRY(ppc_upload_interactions(s, r, f, s->v.ix.halve_sub));
	}
	else if (!s->ix_store.p)
		return fail(PPC_ERR_ARG, "no resident interaction fields: upload them or pass fields");
	// The scratch has a row per live agent and some to spare. Where the host
	// does not know the count the pass runs over the rows there are, and does
	// nothing if the agents are more.
	const size_t row = sizeof(int32_t) * (4 + (size_t)s->ncap);
	int32_t n = (int32_t)std::min<size_t>(s->ix_scratch_bytes / row, s->reps[r].cap);
	if (s->counts_known) // also where the fields came with the call
		n = s->host_count[r];
	else if (n == 0)
		PPC_TRY(live_count(s, r, n));
	if ((int32_t)s->ix_epoch.size() < s->nreps)
		s->ix_epoch.resize(s->nreps, 0);
	const uint64_t epoch = s->ix_epoch[r]++;
	if (n == 0)
		return PPC_OK;
	PPC_TRY(ensure_lists(s));
	const int32_t base = s->reps[r].base;
	const ix_columns& c = s->v.ix;
	const size_t D = s->ndefs, S = c.S;
	ix_fields x {};
	x.substrates = c.S;
	x.replicate = r;
	x.base = base;
	x.dt = s->params.mechanics_time_step;
	x.epoch = epoch;
	x.status = s->v.err + 1; // the words after the error word, spare
	x.dead = c.dead + base;
	x.dead_phago = c.dead_phago + base;
	x.damage_rate = c.damage_rate + base;
	x.live_phago = c.live_phago + base * D;
	x.attack = c.attack + base * D;
	x.fusion = c.fusion + base * D;
	x.immuno = c.immuno + base * D;
	x.frac = c.frac + base * S;
	x.damage = c.damage + base;
	x.attack_time = c.attack_time + base;
	x.nuclei = c.nuclei + base;
	x.fluid = c.fluid + base;
	x.solid = c.solid + base;
	x.cyto = c.cyto + base;
	x.cyto_fluid = c.cyto_fluid + base;
	x.cyto_solid = c.cyto_solid + base;
	x.nuc_fluid = c.nuc_fluid + base;
	x.nuc_solid = c.nuc_solid + base;
	x.fluid_fraction = c.fluid_fraction + base;
	x.c2n = c.c2n + base;
	x.target_cyto = c.target_cyto + base;
	x.target_nuc = c.target_nuc + base;
	x.isub = c.isub + base * S;
	for (;; n = s->host_count[r])
	{
		if (n * row > s->ix_scratch_bytes)
			PPC_TRY(ensure_field_scratch(s, row * std::min<int64_t>(s->reps[r].cap, (int64_t)n + n / 8 + 1024)));
		int32_t* ip = static_cast<int32_t*>(s->ix_scratch);
		const size_t nd = (size_t)n;
		x.n = n;
		x.ncand = ip;
		x.dep = ip + nd;
		x.walk = ip + 2 * nd;
		x.order = ip + 3 * nd;
		x.cand = ip + 4 * nd;
		PPC_CUDA(cudaMemsetAsync(x.status, 0, 3 * sizeof(int32_t), s->stream));
		PPC_TRY(launch_interactions(s, x));
		// the call's status, the device error word and the counts in one copy
		PPC_TRY(finish_counts(s));
		if (!(s->pinned_err[1] & 2))
			break;
	}
	if (s->pinned_err[1])
		return fail(PPC_ERR_CAPACITY, "a neighbour list exceeds the neighbour capacity: no interaction ran");
	// positions and radii may have changed: the next mesh update rebuilds the
	// bins where they did (the device knows); the neighbour lists stay those
	// the interactions used, as in the reference
	s->bins_cond = s->bins_cond || s->bins_valid;
	s->bins_valid = false;
	if (f)
	{
		std::vector<column> back;
		for (const auto& col : ix_column_list(s->v.ix, f, s->ndefs))
			back.push_back(col);
		PPC_TRY(move_columns(s, back, base, s->host_count[r], false));
		return finish(s);
	}
	return map_errors(s, s->pinned_err[0]);
}

int ppc_step(ppc_state* s, int32_t steps)
{
	if (!s)
		return fail(PPC_ERR_ARG, "null state");
	return run_steps(s, steps, false, 0, 0);
}

int ppc_autotune(ppc_state* s, int32_t steps, int32_t* tile_edge, int32_t* threads)
{
	if (!s || steps < 1)
		return fail(PPC_ERR_ARG, "autotune needs a state and steps >= 1");
	struct shape
	{
		int edge, threads, smem;
	};
	const shape cand[] = { { -4, 128, 0 }, { -3, 128, 0 }, { -1, 128, 0 }, { -2, 128, 0 }, { 0, 128, 32 * 1024 },
							 { 0, 64, 16 * 1024 } };
	const int ncand = (int)(sizeof cand / sizeof cand[0]);
	cudaEvent_t e0 = nullptr, e1 = nullptr;
	PPC_CUDA(cudaEventCreate(&e0));
	PPC_CUDA(cudaEventCreate(&e1));
	int best = -1;
	float best_ms = 0.f;
	int rc = PPC_OK;
	for (int k = 0; k < ncand && rc == PPC_OK; k++)
	{
		rc = ppc_set_launch_shape(s, cand[k].edge, cand[k].threads, cand[k].smem);
		s->scan_only = true; // the shapes' own passes are compared
		if (rc == PPC_OK)
			rc = run_steps(s, steps, false, 0, 0); // warm-up: graph capture of this shape
		if (rc != PPC_OK)
			break;
		float ms = 0.f;
		if (cudaEventRecord(e0, s->stream) != cudaSuccess)
			rc = fail(PPC_ERR_CUDA, "cudaEventRecord failed");
		if (rc == PPC_OK)
			rc = run_steps(s, steps, false, 0, 0);
		if (rc == PPC_OK
			&& (cudaEventRecord(e1, s->stream) != cudaSuccess || cudaEventSynchronize(e1) != cudaSuccess
				|| cudaEventElapsedTime(&ms, e0, e1) != cudaSuccess))
			rc = fail(PPC_ERR_CUDA, "timing the candidate shape failed");
		if (rc == PPC_OK && (best < 0 || ms < best_ms))
		{
			best = k;
			best_ms = ms;
		}
	}
	cudaEventDestroy(e0);
	cudaEventDestroy(e1);
	s->scan_only = false;
	PPC_TRY(rc);
	PPC_TRY(ppc_set_launch_shape(s, cand[best].edge, cand[best].threads, cand[best].smem));
	s->scan_only = false;
	if (tile_edge)
		*tile_edge = cand[best].edge;
	if (threads)
		*threads = cand[best].threads;
	return PPC_OK;
}

int ppc_step_with_phenotype(ppc_state* s, int32_t steps, double p_divide, double p_death)
{
	if (!s)
		return fail(PPC_ERR_ARG, "null state");
	return run_steps(s, steps, true, p_divide, p_death);
}

int ppc_get_neighbors(ppc_state* s, int32_t r, int32_t* counts, int32_t* lists, int32_t list_capacity)
{
	if (!valid(s, r) || !counts || !lists || list_capacity < 1)
		return fail(PPC_ERR_ARG, "invalid arguments");
	PPC_TRY(ensure_lists(s));
	std::vector<rep_counters> c;
	PPC_TRY(read_counters(s, c));
	const int32_t n = c[r].count;
	if (n == 0)
		return PPC_OK;
	int32_t* d = nullptr;
	const size_t bytes = (size_t)n * (list_capacity + 1) * sizeof(int32_t);
	PPC_CUDA(cudaMalloc(&d, bytes));
	int rc = launch_neighbors_local(s, r, n, d, d + n, list_capacity);
	if (rc == PPC_OK)
	{
		cudaMemcpyAsync(counts, d, n * sizeof(int32_t), cudaMemcpyDeviceToHost, s->stream);
		cudaMemcpyAsync(lists, d + n, (size_t)n * list_capacity * sizeof(int32_t), cudaMemcpyDeviceToHost, s->stream);
		cudaStreamSynchronize(s->stream);
	}
	cudaFree(d);
	PPC_TRY(rc);
	for (int32_t i = 0; i < n; i++)
		if (counts[i] > list_capacity || counts[i] > s->ncap)
			return fail(PPC_ERR_CAPACITY, "a neighbour list is longer than the capacity");
	return finish(s);
}

int ppc_get_voxel_count(ppc_state* s, int32_t r, int64_t* voxel_count)
{
	if (!valid(s, r) || !voxel_count)
		return fail(PPC_ERR_ARG, "invalid arguments");
	*voxel_count = s->reps[r].voxels;
	return PPC_OK;
}

int ppc_get_mesh_bins(ppc_state* s, int32_t r, int32_t* voxel_counts, int32_t* agents)
{
	if (!valid(s, r) || !voxel_counts || !agents)
		return fail(PPC_ERR_ARG, "invalid arguments");
	PPC_TRY(ensure_bins(s));
	const rep_info& R = s->reps[r];
	std::vector<int32_t> starts(R.voxels + 1);
	PPC_CUDA(cudaMemcpyAsync(starts.data(), s->v.vstart + R.vox_base, (R.voxels + 1) * 4, cudaMemcpyDeviceToHost,
							 s->stream));
	PPC_CUDA(cudaStreamSynchronize(s->stream));
	const int32_t first = starts[0], n = starts[R.voxels] - starts[0];
	std::vector<int32_t> sorted(std::max(n, 1));
	if (n > 0)
	{
		PPC_CUDA(cudaMemcpyAsync(sorted.data(), s->v.sorted + first, (size_t)n * 4, cudaMemcpyDeviceToHost, s->stream));
		PPC_CUDA(cudaStreamSynchronize(s->stream));
	}
	for (int64_t k = 0; k < R.voxels; k++)
		voxel_counts[k] = starts[k + 1] - starts[k];
	for (int32_t u = 0; u < n; u++)
		agents[u] = sorted[u] - R.base;
	return finish(s);
}

int ppc_get_mesh_position(const ppc_mesh* mesh, const double* position, int32_t* c)
{
	if (!mesh || !position || !c)
		return fail(PPC_ERR_ARG, "null argument");
	rep_info R {};
	mesh_info(*mesh, R);
	for (int d = 0; d < 3; d++)
	{
		c[d] = 0;
		if (d >= mesh->dims)
			continue;
		const double q = (position[d] - R.mins[d]) / R.shape[d];
		c[d] = (q == q && q > 0) ? (q >= R.grid[d] ? R.grid[d] - 1 : (int32_t)q) : 0;
	}
	return PPC_OK;
}

int ppc_get_mesh_index(const ppc_mesh* mesh, const int32_t* c, int32_t* index)
{
	if (!mesh || !c || !index)
		return fail(PPC_ERR_ARG, "null argument");
	rep_info R {};
	mesh_info(*mesh, R);
	*index = c[0] + R.grid[0] * (c[1] + R.grid[1] * c[2]);
	return PPC_OK;
}

int ppc_set_profiling(ppc_state* s, int32_t on)
{
	if (!s)
		return fail(PPC_ERR_ARG, "null state");
	PPC_CUDA(cudaStreamSynchronize(s->stream));
	s->profiling = on != 0;
	s->prof_used = 0;
	return PPC_OK;
}

int ppc_get_profile(ppc_state* s, double* fused_ms, int64_t* fused_launches)
{
	if (!s || !fused_ms || !fused_launches)
		return fail(PPC_ERR_ARG, "null argument");
	PPC_CUDA(cudaStreamSynchronize(s->stream));
	double total = 0;
	for (size_t k = 0; k + 1 < s->prof_used; k += 2)
	{
		float ms = 0;
		PPC_CUDA(cudaEventElapsedTime(&ms, s->prof_events[k], s->prof_events[k + 1]));
		total += ms;
	}
	*fused_ms = total;
	*fused_launches = (int64_t)(s->prof_used / 2);
	return PPC_OK;
}

int ppc_get_launch_count(ppc_state* s, int64_t* launches)
{
	if (!s || !launches)
		return fail(PPC_ERR_ARG, "null argument");
	*launches = s->launches;
	return PPC_OK;
}

} // extern "C"
