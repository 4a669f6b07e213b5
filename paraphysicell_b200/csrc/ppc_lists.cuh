// ppc_lists.cuh — mechanics steps over neighbour lists that outlive a step.
// Included by ppc_kernels.cu, whose binning, pair and container code it uses.
//
// The passes that scan the mechanics mesh look at every agent of 27 voxels
// and rebuild the mesh after every step, although agents move hundredths of
// a micrometre per step. Here the mesh of one step gives each agent the list
// of the agents within its interaction reach plus a skin (L. Verlet, Phys.
// Rev. 159, 1967), and the steps after it read only that list, until some
// agent has moved half the skin since the lists were made. Up to then every
// neighbour of an agent is on its list, and the exact FP64 test picks them.
//
// The reference adds a neighbour's terms in the order of the current mesh:
// ascending voxel key, descending slot inside a voxel. Every agent carries
// that order as one word (current key, complement of the slot) beside its
// position, and the accepted neighbours are taken in its order. So the sums
// round as they do with the mesh rebuilt every step.
//
// All steps of a call run in one cooperative launch: the grid stays resident
// and a grid barrier separates the steps. The barrier's word also carries
// the events of the step, so the blocks learn of them without another round
// trip: agents to remove (the container update runs in the kernel and the
// removed agents' entries go dead), or lists past their skin (mesh and lists
// are rebuilt). The agents' positions and previous velocities live in key
// order while the lists hold and are stored to the slot-ordered arrays by the
// call's last step, and before any rebuild.
//
// What bounds a step: while the grid holds all agents, one thread each, the
// barrier and a chain of one gather and the FP64 pair code, all latency (so
// each agent's rows and list stay on chip between the steps); beyond that the
// latency of the gathers under too few warps, then the bytes of the agents'
// rows. Measured on one B200, 60 steps and the download of their result, with
// the mesh rebuilt and searched every step and so: 900 agents in 2-D 1.02 and
// 0.27 ms, 14,300 in 3-D 1.98 and 0.60 ms, 88,700 with springs 1.92 and 0.67
// ms, 96 replicates with 1.03 M agents 55 and 22 ms. Of a step's
// 7,900 cycles for 900 agents the barrier takes 3,300 (of which 2,700 remain
// with nothing stored before it) and the agents' chain 4,300.

constexpr int kListThreads = 640; // one block per SM: 148 arrivals per barrier; 96 registers a thread (in 3-D 66
								  // bytes of them spilled, in 2-D 114)
constexpr int kListLoop = 512;	  // the same where a thread takes several agents: 128 registers
constexpr size_t kListSmem = 200 * 1024; // shared bytes of a block, most of them cached list entries
constexpr int kListHits = 12;	  // accepted neighbours a lane orders in shared memory
constexpr int kListFew = 256;	  // block size up to which a thread has registers to spare
constexpr int kListMost = 255;	  // entries of one list
// um; the lists of the default cell radius then hold about twice its neighbours.
// 60 steps of 14,300 agents placed at random, and after 120 steps: 1.05 and 0.62
// ms with 3 um, 0.85 and 0.55 with 5, the same with 8, which the pool of 24
// entries a slot admits in sparse tissue only.
constexpr float kSkinMax = 5.0f;
constexpr float kSkinMin = 0.5f;  // below it there are no lists
// Where agents move fast, the lists are soon past their skin. Mesh and lists made
// anew by the grid cost about as much as five steps over lists save against
// scanning (2,000 to 80,000 agents: 86 to 145 us against 16 to 24 us a step), so
// each rebuild adds five steps less those its lists lasted to a debt, and a call
// whose debt is past the limit goes on without lists. The limit, eight steps or
// three quarters of the call's, admits the first steps of a relaxing tissue: 60
// steps of 14,300 overlapping agents that repel ten times as hard as usual take
// 2.16 ms, 3.95 with a limit of eight, 3.53 scanning. Where agents stay fast it
// makes 60 steps 1.3 times as long as scanning (2.2 without a limit), once: the
// calls after it scan.
constexpr int kListPays = 5, kListDebt = 8;
__device__ __forceinline__ int list_debt_limit(int steps) { return max(kListDebt, steps / 4 * 3); }
constexpr int32_t kStill = 1 << 30; // list entries: the neighbour is not movable

// events in the upper half of a barrier word
constexpr unsigned long long kEventRebuild = 1ull << 32, kEventRemove = 1ull << 48;

struct list_args
{
	unsigned long long* bar;	  // this launch's two barrier words, 16 words apart
	unsigned long long* bar_next; // the next launch's, zeroed by this one
	long long limit;			  // polls of a barrier wait before it gives up
	int32_t opts;				  // FUSED_WALLS | FUSED_SPRINGS | FUSED_VEL (of the first step)
	int32_t steps;
	int32_t p;		 // lpos buffer that holds the positions
	int32_t cur;	 // slot-ordered position buffer
	int32_t refresh; // slot-ordered positions or velocities were uploaded since the lists' copies were made
	int32_t springs; // removals are replayed on the spring rows
	int32_t cached;	 // list entries per agent kept in shared memory
	float voxel;	 // smallest voxel edge of the meshes
	float* skin_out; // host-mapped: the skin of the lists in use
};

__device__ __forceinline__ unsigned long long order_word(int32_t key, int slot)
{
	return ((unsigned long long)(uint32_t)key << 32) | (uint32_t)~slot;
}

// axis_coord_quiet through the reciprocal of the voxel edge: the product is
// within two ulps of the quotient, so both truncate alike unless the product
// is that close to an integer, where the division decides
__device__ __forceinline__ int axis_coord_fast(double x, const rep_info& R, int d)
{
	const double q = (x - R.mins[d]) * R.inv_shape[d];
	const double near = rint(q);
	if (fabs(q - near) <= 1e-9 * fabs(q) || !(q < 1e9))
		return axis_coord_quiet(x, R, d);
	if (!(q > 0.0))
		return 0;
	return min((int)q, R.grid[d] - 1);
}

template <int DIMS>
__device__ __forceinline__ int32_t quiet_key(const rep_info& R, const double4& p)
{
	const int c0 = axis_coord_fast(p.x, R, 0);
	const int c1 = DIMS >= 2 ? axis_coord_fast(p.y, R, 1) : 0;
	const int c2 = DIMS >= 3 ? axis_coord_fast(p.z, R, 2) : 0;
	return (int32_t)(R.vox_base + c0 + (int64_t)R.grid[0] * (c1 + (int64_t)R.grid[1] * c2));
}

__device__ __forceinline__ float lctl_float(const view& v, int word)
{
	return __int_as_float(ld_relaxed_i32(v.lctl + word));
}

// A 32-byte row in one load or store: a warp's gather of rows costs the L1
// one tag lookup per row, not one per 16-byte half. Rows are 32-byte aligned.
__device__ __forceinline__ double4 row_load(const double4* p)
{
	double4 x;
	asm volatile("ld.global.v4.f64 {%0, %1, %2, %3}, [%4];"
				 : "=d"(x.x), "=d"(x.y), "=d"(x.z), "=d"(x.w)
				 : "l"(p)
				 : "memory");
	return x;
}

__device__ __forceinline__ void row_store(double4* p, const double4& x)
{
	asm volatile("st.global.v4.f64 [%0], {%1, %2, %3, %4};" ::"l"(p), "d"(x.x), "d"(x.y), "d"(x.z), "d"(x.w)
				 : "memory");
}

// the skin of lists over agents whose largest reach is known: a pair within
// its reaches plus the skin must lie in adjacent voxels of the mesh the lists
// are made from; 0 when no useful skin is left
__device__ __forceinline__ float list_skin(const view& v, float voxel)
{
	const float skin = fminf(voxel * 0.99999f - 2.0f * lctl_float(v, LCTL_REACH), lctl_float(v, LCTL_CAP));
	return skin >= kSkinMin ? skin : 0.0f;
}

// the largest reach of the agents in the key order, from the threads' own
__device__ __forceinline__ void list_reach(const view& v, double w)
{
	const float f = w > 0.0 ? __double2float_ru(w) : 0.0f;
	const int m = __reduce_max_sync(0xffffffffu, __float_as_int(f)); // non-negative floats order as integers
	if ((threadIdx.x & 31) == 0 && m > ld_relaxed_i32(v.lctl + LCTL_REACH))
		atomicMax(v.lctl + LCTL_REACH, m);
}

// ---- making the lists -------------------------------------------------------

struct __align__(16) list_warp
{
	int2 rows[9][32];  // per agent and stencil row: first candidate number, array position - number
	int32_t first[33]; // each agent's first candidate in the warp's list; first[32]: the total
	int32_t cnt[32];   // entries on each agent's list
	float margin[32];
	float4 pf[32];
};

// What the pair code needs of two agents' fields (a change of any rebuilds the
// lists): the sum of the radii, the reach of the pair, and the square roots of
// the repulsion and adhesion products, rounded as in pair_fp64::add_pair
// (pair_fp32::add).
template <bool F32>
__device__ __forceinline__ double4 list_pair(const view& v, int t, int u, const double4& qi, const double4& qj,
											 double wi, double wj, int def_i, int def_j)
{
	const int64_t D = v.ndefs;
	if (F32)
	{
		const float4 fj = v.sprmf[u];
		return make_double4((float)qi.x + fj.x, (float)wi + (float)wj, sqrtf((float)qi.y * fj.y),
							sqrtf((float)qi.z * fj.z * v.safff[t * D + def_j] * v.safff[u * D + def_i]));
	}
	return make_double4(qi.x + qj.x, wi + wj, sqrt(qi.y * qj.y),
						sqrt(qi.z * qj.z * v.saff[t * D + def_j] * v.saff[u * D + def_i]));
}

// entry e of the lists: neighbour u of the agent at t
__device__ __forceinline__ void list_entry(const view& v, int64_t e, int t, int u)
{
	const double4 qi = v.sprm4[t], qj = v.sprm4[u];
	const double wi = v.spos4[t].w, wj = v.spos4[u].w;
	int def_i, def_j;
	bool mov_i, mov_j;
	unpack_bits(qi.w, def_i, mov_i);
	unpack_bits(qj.w, def_j, mov_j);
	v.nl[e] = make_int2(u | (mov_j ? 0 : kStill), __float_as_int((float)(wi + wj)));
	if (v.f32)
	{
		const double4 f = list_pair<true>(v, t, u, qi, qj, wi, wj, def_i, def_j);
		reinterpret_cast<float4*>(v.nl_pair)[e] = make_float4((float)f.x, (float)f.y, (float)f.z, (float)f.w);
	}
	else
		v.nl_pair[e] = list_pair<false>(v, t, u, qi, qj, wi, wj, def_i, def_j);
}

// The lists of the warp's agents (key-ordered positions tw .. tw + 31), and
// their copies in key order. The candidates of the agents are laid end to end
// and shared out over the lanes (as in the queue pass), so the filter runs on
// full warps; it runs twice, first to count the entries, then to store them
// in candidate order, which is that of the mesh. A warp's lists take one slab
// of the pool, entry k of lane l at k * 32 + l; where a warp finds the pool
// full, the lists are made again with a smaller skin. The
// single-precision filter with the replicate's margin never drops a pair
// within reach plus skin. Every lane calls it.
// ROUNDS: candidate rounds whose loads are in flight together.
template <int DIMS, int ROUNDS>
__device__ __forceinline__ void list_build(const view& v, int cur, int p, int tw, int n, float skin, int springs_on,
										   list_warp& w)
{
	constexpr int NR = DIMS == 3 ? 9 : (DIMS == 2 ? 3 : 1);
	const int lane = threadIdx.x & 31;
	const int64_t C = v.total_cap;
	const int t = tw + lane;
	const bool act = t < n;
	int s = 0, r = 0, def_i = 0;
	bool mov_i = false;
	int32_t key = 0;
	double4 pi = make_double4(0, 0, 0, 0), qi = pi;
	float4 pf = make_float4(0, 0, 0, 0);
	int lo[NR], hi[NR];
#pragma unroll
	for (int k = 0; k < NR; k++)
		lo[k] = hi[k] = 0;
	if (act)
	{
		s = v.sorted[t];
		key = v.skey[t];
		pi = v.spos4[t];
		pf = v.sposf[t];
		qi = v.sprm4[t];
		r = rep_of(v, s);
		unpack_bits(qi.w, def_i, mov_i);
		stencil_bounds<DIMS>(v, v.reps[r], key, lo, hi);
	}
	int c = 0;
#pragma unroll
	for (int k = 0; k < NR; k++)
	{
		w.rows[k][lane] = make_int2(c, lo[k] - c);
		c += hi[k] - lo[k];
	}
	int incl = c;
#pragma unroll
	for (int o = 1; o < 32; o <<= 1)
	{
		const int y = __shfl_up_sync(0xffffffffu, incl, o);
		if (lane >= o)
			incl += y;
	}
	const int total = skin > 0.0f ? __shfl_sync(0xffffffffu, incl, 31) : 0;
	w.first[lane] = incl - c;
	if (lane == 31)
		w.first[32] = incl;
	w.cnt[lane] = 0;
	w.margin[lane] = v.reps[r].fmargin + skin;
	w.pf[lane] = pf;
	if (act)
	{
		// the agent's rows in key order, and its springs as (position in the
		// key order, coefficient)
		v.lpos[p][t] = make_double4(pi.x, pi.y, pi.z, __longlong_as_double((long long)order_word(key, s)));
		v.lvprev[t] = v.vprev[s];
		const int ns = (springs_on && mov_i) ? unpack_springs(qi.w) : 0;
		const int D = v.ndefs;
		for (int k = 0; k < ns; k++)
		{
			const int j = v.springs[(int64_t)s * v.scap + k];
			v.lspr[k * C + t] = v.tpos[j];
			v.lcoef[k * C + t]
				= sqrt(v.ec[s] * v.ec[j] * v.aff[(int64_t)s * D + v.def[j]] * v.aff[(int64_t)j * D + def_i]);
		}
	}
	__syncwarp();
	int64_t slab = -1;
	for (int pass = 0; pass < 2; pass++)
	{
		for (int base = 0; base < total; base += 32 * ROUNDS)
		{
			float4 cand[ROUNDS];
			int cu[ROUNDS], own[ROUNDS];
#pragma unroll
			for (int q = 0; q < ROUNDS; q++)
			{
				const int x = base + q * 32 + lane;
				own[q] = -1;
				cu[q] = 0;
				if (x < total)
				{
					int i = 0;
#pragma unroll
					for (int step = 16; step >= 1; step >>= 1)
						if (w.first[i + step] <= x)
							i += step;
					const int cc = x - w.first[i];
					int k = 0;
#pragma unroll
					for (int kk = 1; kk < NR; kk++)
						k += w.rows[kk][i].x <= cc;
					own[q] = i;
					cu[q] = w.rows[k][i].y + cc;
					cand[q] = v.sposf[cu[q]];
				}
			}
#pragma unroll
			for (int q = 0; q < ROUNDS; q++)
			{
				bool keep = false;
				if (own[q] >= 0)
					keep = cu[q] != tw + own[q] && filter_keep<DIMS>(w.pf[own[q]], cand[q], w.margin[own[q]]);
				const unsigned kept = __ballot_sync(0xffffffffu, keep);
				if (!kept)
					continue;
				const unsigned mine = __match_any_sync(0xffffffffu, own[q]) & kept;
				int at = 0;
				if (keep)
				{
					at = w.cnt[own[q]] + __popc(mine & ((1u << lane) - 1));
					if (pass == 1)
					{
						const int64_t e = slab + 32 * at + own[q];
						list_entry(v, e, tw + own[q], cu[q]);
					}
				}
				__syncwarp();
				if (keep && (mine >> lane) == 1u) // the last of its agent's entries in this round
					w.cnt[own[q]] = at + 1;
				__syncwarp();
			}
		}
		if (pass == 1)
			break;
		// the slab for the longest of the warp's lists
		const int most = (int)__reduce_max_sync(0xffffffffu, (unsigned)w.cnt[lane]);
		if (skin <= 0.0f)
			break;
		unsigned long long at = 0;
		if (lane == 0 && most <= kListMost)
			at = atomicAdd(v.nl_used, 32ull * most);
		at = __shfl_sync(0xffffffffu, at, 0);
		if (most > kListMost || (int64_t)at + 32 * most > v.nl_pool)
		{
			if (lane == 0)
				atomicMin(v.lctl + LCTL_WANT, __float_as_int(0.6f * skin));
			break;
		}
		slab = (int64_t)at;
		if (act)
			v.nlc[t] = w.cnt[lane];
		__syncwarp();
		w.cnt[lane] = 0;
		__syncwarp();
	}
	if (lane == 0 && tw < n)
	{
		v.nl_slab[tw >> 5] = slab;
		if (slab < 0)
			v.lctl[LCTL_FIT] = 0;
	}
	__syncwarp();
}

// position of each slot in the key order
__device__ __forceinline__ void list_positions(const view& v, int t, int n)
{
	if (t < n)
		v.tpos[v.sorted[t]] = t;
}

// reach and slot positions, the lists' inputs, after a rebuild by its own kernels
__global__ void __launch_bounds__(kThreads) k_list_prepare(view v, int reset)
{
	grid_wait();
	const int t = blockIdx.x * blockDim.x + threadIdx.x;
	const int n = *v.cursor;
	if (t == 0)
	{
		if (reset)
		{
			v.lctl[LCTL_WANT] = __float_as_int(kSkinMax);
			v.lctl[LCTL_DEBT] = 0;
		}
		v.lctl[LCTL_CAP] = v.lctl[LCTL_WANT];
		v.lctl[LCTL_FIT] = 1;
		v.lctl[LCTL_AGE] = 0;
		*v.nl_used = 0;
	}
	list_reach(v, t < n ? v.spos4[t].w : 0.0);
	list_positions(v, t, n);
}

template <int DIMS>
__global__ void __launch_bounds__(128) k_list_build(view v, int cur, int p, int springs_on, float voxel, float* skin_out)
{
	grid_wait();
	__shared__ list_warp w[4];
	const float skin = list_skin(v, voxel);
	if (blockIdx.x == 0 && threadIdx.x == 0)
	{
		v.lctl[LCTL_DIRTY] = 0;
		v.lctl[LCTL_BUILT] = __float_as_int(skin);
		*skin_out = skin;
	}
	list_build<DIMS, 4>(v, cur, p, blockIdx.x * 128 + (threadIdx.x & ~31), *v.cursor, skin, springs_on,
					 w[threadIdx.x >> 5]);
}

// ---- a step -------------------------------------------------------------------

// The reference's neighbour test, distance <= rmad_i r_i + rmad_j r_j, in
// squares: 1 within, 0 beyond, -1 where the reach's rounding to float (or the
// square root's, 1e-16) decides and list_near has to.
template <int DIMS>
__device__ __forceinline__ int list_test(const double4& pi, const double4& q, float reach)
{
	const double ddx = pi.x - q.x;
	const double ddy = DIMS >= 2 ? pi.y - q.y : 0.0;
	const double ddz = DIMS >= 3 ? pi.z - q.z : 0.0;
	double d2 = ddx * ddx;
	if (DIMS >= 2)
		d2 = d2 + ddy * ddy;
	if (DIMS >= 3)
		d2 = d2 + ddz * ddz;
	const double r2 = (double)reach * (double)reach;
	if (reach > 0.0f && d2 < r2 * (1.0 - 1e-6))
		return 1;
	return d2 > r2 * (1.0 + 1e-6) ? 0 : -1;
}

template <int DIMS>
__device__ __forceinline__ bool list_near(const double4& pi, const double4& q, double reach)
{
	const double ddx = pi.x - q.x;
	const double ddy = DIMS >= 2 ? pi.y - q.y : 0.0;
	const double ddz = DIMS >= 3 ? pi.z - q.z : 0.0;
	double d2 = ddx * ddx;
	if (DIMS >= 2)
		d2 = d2 + ddy * ddy;
	if (DIMS >= 3)
		d2 = d2 + ddz * ddz;
	// exact early reject: d2 > reach^2 (1 + 1e-12) implies sqrt(d2) > reach
	if (d2 > reach * reach * (1.0 + 1e-12))
		return false;
	const double dist = DIMS == 1 ? fabs(ddx) : sqrt(d2);
	return dist <= reach;
}

// one pair's terms for agent i at pi, its neighbour at q: the arithmetic of
// pair_fp64::add_pair (pair_fp32::add) with the entry's products
template <int DIMS, bool F32>
__device__ __forceinline__ double4 list_terms(const double4& pi, const double4& q, bool mov_i, const double4& pair)
{
	const double ddx = pi.x - q.x;
	const double ddy = DIMS >= 2 ? pi.y - q.y : 0.0;
	const double ddz = DIMS >= 3 ? pi.z - q.z : 0.0;
	double4 out = make_double4(0, 0, 0, 0);
	if (F32)
	{
		const float dx = (float)ddx, dy = (float)ddy, dz = (float)ddz;
		float d2f = dx * dx;
		if (DIMS >= 2)
			d2f = d2f + dy * dy;
		if (DIMS >= 3)
			d2f = d2f + dz * dz;
		const float distf = DIMS == 1 ? fabsf(dx) : sqrtf(d2f);
		const float d = distf < 0.00001f ? 0.00001f : distf;
		float rep = 1.f - d / (float)pair.x;
		rep = rep < 0.f ? 0.f : rep;
		rep = rep * rep;
		const float term = rep * 36.64504274775163f;
		out.w = term;
		if (mov_i)
		{
			rep = rep * (float)pair.z;
			float adh = 1.f - d / (float)pair.y;
			adh = adh * adh;
			adh = adh * (float)pair.w;
			const float force = (rep - adh) / d;
			out.x = force * dx;
			out.y = force * dy;
			out.z = force * dz;
		}
	}
	else
	{
		double d2 = ddx * ddx;
		if (DIMS >= 2)
			d2 = d2 + ddy * ddy;
		if (DIMS >= 3)
			d2 = d2 + ddz * ddz;
		const double dist = DIMS == 1 ? fabs(ddx) : sqrt(d2);
		const double d = dist < 0.00001 ? 0.00001 : dist;
		double rep = 1.0 - d / pair.x;
		rep = rep < 0 ? 0 : rep;
		rep = rep * rep;
		out.w = rep * simple_pressure_coefficient;
		if (mov_i)
		{
			rep = rep * pair.z;
			double adh = 1.0 - d / pair.y;
			adh = adh * adh;
			adh = adh * pair.w;
			const double force = (rep - adh) / d;
			out.x = force * ddx;
			out.y = force * ddy;
			out.z = force * ddz;
		}
	}
	return out;
}

// the sums of one agent over its neighbours, terms added in call order
template <bool F32>
struct list_sum
{
	double vx = 0, vy = 0, vz = 0, pressure = 0;
	nsum fx, fy, fz, fp;

	__device__ __forceinline__ void add(double tx, double ty, double tz, double term, bool mov_i, bool mov_j)
	{
		if (F32)
		{
			if (mov_i)
				fp.add((float)term);
			if (mov_j)
				fp.add((float)term);
			if (mov_i)
			{
				fx.add((float)tx);
				fy.add((float)ty);
				fz.add((float)tz);
			}
		}
		else
		{
			if (mov_i)
				pressure = pressure + term;
			if (mov_j)
				pressure = pressure + term;
			if (mov_i)
			{
				vx = vx + tx;
				vy = vy + ty;
				vz = vz + tz;
			}
		}
	}

	__device__ __forceinline__ void finish()
	{
		if (F32)
		{
			vx = vx + fx.value();
			vy = vy + fy.value();
			vz = vz + fz.value();
			pressure = fp.value();
		}
	}
};

// what a thread keeps of its agent between the steps: its place, and (in its
// warp's shared columns, which unlike spilled registers stay on the SM when a
// barrier drops the L1) its rows
struct list_own
{
	int64_t slab;		   // the warp's slab of list entries, or -1
	int s, r, cnt, springs; // s < 0: no agent, or removed
	bool mov;
};

struct __align__(16) list_step_warp
{
	double px[32], py[32], pz[32];			 // the agents' positions
	double vx[32], vy[32], vz[32];			 // previous velocities
	double radius[32], bm[32];
	double tx[32], ty[32], tz[32], tp[32]; // the pair terms of a round
	float rx[32], ry[32], rz[32];			 // positions the lists were made at
	int32_t first[33];					 // each agent's first accepted neighbour in the warp's list
	int2 hit[kListHits][32];			 // per agent: its accepted neighbours in order (list entry, neighbour)
};

__device__ __forceinline__ list_own list_load(const view& v, const list_args& a, list_step_warp& w, int p, int t, int n)
{
	const int lane = threadIdx.x & 31;
	list_own o {};
	o.s = -1;
	o.slab = (t & ~31) < n ? v.nl_slab[t >> 5] : -1; // the warp's, also for its lanes without an agent
	if (t >= n)
		return o;
	o.s = v.sorted[t];
	o.cnt = v.nlc[t];
	const double4 pos = row_load(v.lpos[p] + t);
	const double4 vp = row_load(v.lvprev + t);
	const float4 ref = v.sposf[t];
	const double4 q = row_load(v.sprm4 + t);
	const long long bits = __double_as_longlong(q.w);
	w.px[lane] = pos.x;
	w.py[lane] = pos.y;
	w.pz[lane] = pos.z;
	w.vx[lane] = vp.x;
	w.vy[lane] = vp.y;
	w.vz[lane] = vp.z;
	w.radius[lane] = q.x;
	w.rx[lane] = ref.x;
	w.ry[lane] = ref.y;
	w.rz[lane] = ref.z;
	o.mov = ((bits >> 32) & 1) != 0;
	o.springs = ((a.opts & FUSED_SPRINGS) && o.mov) ? unpack_springs(q.w) : 0;
	if (o.s < 0)
		return o;
	o.r = v.nreps == 1 ? 0 : (v.nreps <= 65536 ? (int)((bits >> 48) & 0xffff) : v.rid[o.s]);
	if (a.opts & FUSED_WALLS)
		w.bm[lane] = v.prm[o.s].w;
	return o;
}

// The block's cached list entries: entry k of thread i at k * T + i.
struct list_cache
{
	double4* pair; // (float4 in the FP32-force form)
	int2* entry;
	int n; // entries cached per agent
	int T, t0; // threads of the block, and the key-ordered position of its first
};

// entry k of the agent at t, in its warp's slab; where entries are cached, the
// agent's thread is t less the block's first
__device__ __forceinline__ int2 list_get(const view& v, const list_cache& lc, int64_t slab, int t, int k)
{
	return k < lc.n ? lc.entry[k * lc.T + t - lc.t0] : v.nl[slab + (t & 31) + 32 * k];
}

// what the pair code needs of the agent at t and its entry k
template <bool F32>
__device__ __forceinline__ double4 list_get_pair(const view& v, const list_cache& lc, int64_t slab, int t, int k)
{
	const int64_t e = slab + (t & 31) + 32 * k;
	if (F32)
	{
		const float4 f = k < lc.n ? reinterpret_cast<const float4*>(lc.pair)[k * lc.T + t - lc.t0]
								  : reinterpret_cast<const float4*>(v.nl_pair)[e];
		return make_double4(f.x, f.y, f.z, f.w);
	}
	return k < lc.n ? lc.pair[k * lc.T + t - lc.t0] : row_load(v.nl_pair + e);
}

// The end of a step for the agent at t with its neighbours' sums: membrane,
// springs, Adams-Bashforth, its rows in lpos[p ^ 1], and the step's events.
template <int DIMS, bool F32>
__device__ __forceinline__ unsigned long long list_finish(const view& v, const list_args& a, const rep_info* reps,
														  list_step_warp& w, const list_own& o, int p, int t, bool first,
														  bool last, float skin, list_sum<F32>& sum)
{
	const int64_t C = v.total_cap;
	const int lane = threadIdx.x & 31;
	const double4* pos = v.lpos[p];
	sum.finish();
	const rep_info& R = reps[o.r];
	double4 pn = make_double4(w.px[lane], w.py[lane], w.pz[lane], 0.0);
	if (o.mov)
	{
		double4 vel = make_double4(sum.vx, sum.vy, sum.vz, 0.0);
		if (a.opts & FUSED_WALLS)
			walls<DIMS>(v, R, pn, w.radius[lane], w.bm[lane], vel);
		for (int k = 0; k < o.springs; k++)
		{
			const double coef = v.lcoef[k * C + t];
			const double4 pj = pos[v.lspr[k * C + t]];
			for (int d = 0; d < DIMS; d++)
				set_comp(vel, d, comp(vel, d) + coef * (comp(pj, d) - comp(pn, d)));
		}
		double4 vp = make_double4(w.vx[lane], w.vy[lane], w.vz[lane], 0.0);
		ab2<DIMS>(v.dt, pn, vel, vp);
		row_store(v.lvprev + t, vp);
		if (last)
			v.vprev[o.s] = vp;
		w.px[lane] = pn.x;
		w.py[lane] = pn.y;
		w.pz[lane] = pn.z;
		w.vx[lane] = vp.x;
		w.vy[lane] = vp.y;
		w.vz[lane] = vp.z;
		if (first && (a.opts & FUSED_VEL))
			v.vel[o.s] = make_double4(0, 0, 0, 0);
	}
	if (last)
	{
		v.pos[a.cur][o.s] = pn;
		v.pressure[o.s] = sum.pressure;
	}
	else
		v.lpress[t] = sum.pressure;
	pn.w = __longlong_as_double((long long)order_word(quiet_key<DIMS>(R, pn), o.s));
	row_store(v.lpos[p ^ 1] + t, pn);
	unsigned long long ev = 0;
	if (!(pn.x == pn.x && pn.y == pn.y && pn.z == pn.z))
		atomicOr(v.err, ERR_NONFINITE);
	if (to_remove<DIMS>(R, pn, first ? v.flags[o.s] : PPC_FLAG_NONE))
	{
		append_bad(v, o.r, o.s - R.base);
		ev = kEventRemove;
	}
	// moved half the skin since the lists were made (both float positions
	// carry the rounding the margin covers); without a skin, every step
	const float fx = (float)(pn.x - R.mins[0]) - w.rx[lane];
	const float fy = DIMS >= 2 ? (float)(pn.y - R.mins[1]) - w.ry[lane] : 0.f;
	const float fz = DIMS >= 3 ? (float)(pn.z - R.mins[2]) - w.rz[lane] : 0.f;
	const float half = 0.5f * skin - R.fmargin;
	if (!(half > 0.f) || fx * fx + fy * fy + fz * fz > half * half * 0.9999f)
		ev |= kEventRebuild;
	return ev;
}

// the velocity an agent enters a call's first step with
template <bool F32>
__device__ __forceinline__ void list_enter(const view& v, const list_args& a, const list_own& o, bool first,
										   list_sum<F32>& sum)
{
	if (first && (a.opts & FUSED_VEL) && o.s >= 0 && o.mov)
	{
		const double4 v0 = v.vel[o.s];
		sum.vx = v0.x;
		sum.vy = v0.y;
		sum.vz = v0.z;
	}
}

// One step of the warp's agents (this lane's at key-ordered position t, its
// rows in `w` and `o`): neighbours, forces, then list_finish. Each lane picks
// its neighbours from its list and puts up to kListHits of them in order;
// their pair terms are evaluated by full warps, whatever lane they belong to,
// and each lane adds its own in their order; lanes with more neighbours go
// on after the last one in the order. `first`: flags and entry velocities
// count; `last`: the slot-ordered rows are stored. Returns the step's events.
// Every lane calls it.
template <int DIMS, bool F32, int BATCH>
__device__ __forceinline__ unsigned long long list_step(const view& v, const list_args& a, const rep_info* reps,
														const list_cache& lc, list_step_warp& w, const list_own& o,
														int p, int t, int n, bool first, bool last, float skin)
{
	const int lane = threadIdx.x & 31;
	const double4* pos = v.lpos[p];
	const bool act = o.s >= 0;
	list_sum<F32> sum;
	list_enter<F32>(v, a, o, first, sum);
	const int cnt = act ? o.cnt : 0;
	unsigned long long done = 0; // order word of the last neighbour added
	bool more = true;
	do
	{
		int nh = 0;
		if (more)
		{
			more = false;
			const double4 pi = make_double4(w.px[lane], w.py[lane], w.pz[lane], 0.0);
			unsigned long long tail = done; // order word of the last hit
			auto word = [&](int h) { // order word of hit h
				return (unsigned long long)__double_as_longlong(pos[w.hit[h][lane].y & ~kStill].w);
			};
			int2 next[BATCH];
			for (int k0 = -BATCH; k0 < cnt; k0 += BATCH)
			{
				// the batch's rows and the next batch's entries in flight together
				double4 q[BATCH];
				int2 e[BATCH];
#pragma unroll
				for (int j = 0; j < BATCH; j++)
				{
					e[j] = next[j];
					if (k0 >= 0 && k0 + j < cnt)
						q[j] = row_load(pos + (e[j].x & ~kStill));
				}
#pragma unroll
				for (int j = 0; j < BATCH; j++)
					if (k0 + BATCH + j < cnt)
						next[j] = list_get(v, lc, o.slab, t, k0 + BATCH + j);
				if (k0 < 0)
					continue;
#pragma unroll
				for (int j = 0; j < BATCH; j++)
				{
					if (k0 + j >= cnt)
						continue;
					const int u = e[j].x & ~kStill;
					const int in = list_test<DIMS>(pi, q[j], __int_as_float(e[j].y));
					if (in == 0 || (in < 0 && !list_near<DIMS>(pi, q[j], v.spos4[t].w + v.spos4[u].w)))
						continue;
					const unsigned long long ow = (unsigned long long)__double_as_longlong(q[j].w);
					if (ow <= done)
						continue;
					more = more || nh == kListHits;
					if (nh == kListHits && ow > tail)
						continue;
					if (k0 + j >= lc.n)
						prefetch_l1(v.nl_pair + o.slab + lane + 32 * (k0 + j));
					// at the end of the hits, or, where agents crossed voxels
					// since the lists were made, at its place among them
					int g = nh < kListHits ? nh++ : kListHits - 1;
					if (ow < tail)
						for (; g > 0 && word(g - 1) > ow; g--)
							w.hit[g][lane] = w.hit[g - 1][lane];
					w.hit[g][lane] = make_int2(k0 + j, e[j].x);
					tail = ow > tail ? ow : word(nh - 1);
				}
			}
			done = tail;
		}
		int off = nh;
#pragma unroll
		for (int d = 1; d < 32; d <<= 1)
		{
			const int y = __shfl_up_sync(0xffffffffu, off, d);
			if (lane >= d)
				off += y;
		}
		const int total = __shfl_sync(0xffffffffu, off, 31);
		if (total == 0)
			break;
		off -= nh;
		w.first[lane] = off;
		const unsigned movs = __ballot_sync(0xffffffffu, o.mov);
		__syncwarp();
		for (int base = 0; base < total; base += 32)
		{
			const int x = base + lane;
			bool mov_j = false;
			if (x < total)
			{
				int i = 0;
#pragma unroll
				for (int step = 16; step >= 1; step >>= 1)
					if (w.first[i + step] <= x)
						i += step;
				const int2 hit = w.hit[x - w.first[i]][i];
				const int u = hit.y;
				const double4 pair = list_get_pair<F32>(v, lc, o.slab, t - lane + i, hit.x); // one slab per warp
				mov_j = (u & kStill) == 0;
				const double4 tm = list_terms<DIMS, F32>(make_double4(w.px[i], w.py[i], w.pz[i], 0.0),
														 row_load(pos + (u & ~kStill)),
														 (movs >> i) & 1, pair);
				w.tx[lane] = tm.x;
				w.ty[lane] = tm.y;
				w.tz[lane] = tm.z;
				w.tp[lane] = tm.w;
			}
			const unsigned movj = __ballot_sync(0xffffffffu, mov_j);
			__syncwarp();
			const int hi = min(off + nh, base + 32) - base;
			for (int q = max(off, base) - base; q < hi; q++)
				sum.add(w.tx[q], w.ty[q], w.tz[q], w.tp[q], o.mov, (movj >> q) & 1);
			__syncwarp();
		}
	} while (__any_sync(0xffffffffu, more));
	if (!act)
	{
		if (t < n)
			v.lpos[p ^ 1][t] = v.lpos[p][t]; // a removed agent's entry stays out of reach
		return 0;
	}
	return list_finish<DIMS, F32>(v, a, reps, w, o, p, t, first, last, skin, sum);
}

// Asks L2 for what the warp needs of the agents from position tw on: lane by
// lane one 128-byte line of their rows, and of their list entries.
__device__ __forceinline__ void list_prefetch(const view& v, int p, int tw, int n)
{
	if (tw >= n)
		return;
	const int lane = threadIdx.x & 31;
	const int64_t slab = v.nl_slab[tw >> 5];
	const char* row;
	if (lane < 8)
		row = reinterpret_cast<const char*>(v.lpos[p] + tw) + 128 * lane;
	else if (lane < 16)
		row = reinterpret_cast<const char*>(v.lvprev + tw) + 128 * (lane - 8);
	else if (lane < 24)
		row = reinterpret_cast<const char*>(v.sprm4 + tw) + 128 * (lane - 16);
	else if (lane < 28)
		row = reinterpret_cast<const char*>(v.sposf + tw) + 128 * (lane - 24);
	else
		row = reinterpret_cast<const char*>(lane & 1 ? v.sorted + tw : v.nlc + tw);
	prefetch_l2(row);
	if (slab >= 0)
		prefetch_l2(reinterpret_cast<const char*>(v.nl + slab) + 128 * lane);
}

// The slot-ordered rows of the agent at t from its key-ordered ones in lpos[p].
__device__ __forceinline__ void list_flush(const view& v, int cur, int p, int t)
{
	const int s = v.sorted[t];
	if (s < 0)
		return;
	const double4 pn = v.lpos[p][t];
	v.pos[cur][s] = make_double4(pn.x, pn.y, pn.z, 0.0);
	v.pressure[s] = v.lpress[t];
	if ((__double_as_longlong(v.sprm4[t].w) >> 32) & 1)
		v.vprev[s] = v.lvprev[t];
}

// Uploaded positions and previous velocities into the key-ordered rows. A
// moved agent's key is computed with the mesh's error reports.
template <int DIMS>
__device__ __forceinline__ unsigned long long list_refresh(const view& v, int cur, int p, int t, float skin)
{
	const int s = v.sorted[t];
	if (s < 0)
		return 0;
	const double4 x = v.pos[cur][s];
	const double4 old = v.lpos[p][t];
	v.lvprev[t] = v.vprev[s];
	if (__double_as_longlong(x.x) == __double_as_longlong(old.x)
		&& __double_as_longlong(x.y) == __double_as_longlong(old.y)
		&& __double_as_longlong(x.z) == __double_as_longlong(old.z))
		return 0;
	const int r = rep_of(v, s);
	const rep_info& R = v.reps[r];
	v.lpos[p][t]
		= make_double4(x.x, x.y, x.z, __longlong_as_double((long long)order_word(voxel_key(v, cur, s, r), s)));
	const float4 ref = v.sposf[t];
	const float fx = (float)(x.x - R.mins[0]) - ref.x;
	const float fy = DIMS >= 2 ? (float)(x.y - R.mins[1]) - ref.y : 0.f;
	const float fz = DIMS >= 3 ? (float)(x.z - R.mins[2]) - ref.z : 0.f;
	const float half = 0.5f * skin - R.fmargin;
	return !(half > 0.f) || !(fx * fx + fy * fy + fz * fz <= half * half * 0.9999f) ? kEventRebuild : 0;
}

// move_agent with the loads of some fields at a time before their stores: a
// few round trips instead of one per field (the arrays could alias for all
// the compiler knows), which counts where a grid waits for the moves: 96
// replicates' removals of a step took 150,000 cycles with move_agent and the
// serial plan, 14,000 with this and list_remove_rep's. The rebuild's count
// keeps move_agent, whose few registers suit a kernel that hardly ever moves
// an agent.
__device__ __forceinline__ void list_move(const view& v, int cur, int d, int s)
{
	copy_columns(v, v.dims, d, s);
	double4* rows[] = { v.pos[cur], v.vel, v.vprev, v.prm, v.orient };
	double4 row[5];
#pragma unroll
	for (int k = 0; k < 5; k++)
		row[k] = rows[k][s];
#pragma unroll
	for (int k = 0; k < 5; k++)
		rows[k][d] = row[k];
	double* ones[] = { v.rmad, v.ec, v.arate, v.drate, v.pressure, v.vol, v.nvol, v.nrad, v.sarea, v.polarity };
	double one[10];
#pragma unroll
	for (int k = 0; k < 10; k++)
		one[k] = ones[k][s];
	const int32_t def = v.def[s], maxatt = v.maxatt[s], ncnt = v.ncnt[s];
	const uint8_t movable = v.movable[s], flags = v.flags[s];
	const int64_t id = v.ids[s];
#pragma unroll
	for (int k = 0; k < 10; k++)
		ones[k][d] = one[k];
	v.def[d] = def;
	v.maxatt[d] = maxatt;
	v.movable[d] = movable;
	v.flags[d] = flags;
	v.ids[d] = id;
#pragma unroll 1
	for (int q = 0; q < v.ndefs; q++)
		v.aff[(int64_t)d * v.ndefs + q] = v.aff[(int64_t)s * v.ndefs + q];
	const int nn = min(ncnt, v.ncap);
#pragma unroll 1
	for (int q = 0; q < nn; q++)
		v.nidx[(int64_t)d * v.ncap + q] = v.nidx[(int64_t)s * v.ncap + q];
	v.ncnt[d] = ncnt;
}

// The container update of replicate r after a step, one block, without a
// rebuild (and without springs): update_cell_container_internal's loop
// (reference: containers_solver.cpp:81-120) removes every marked agent, and the
// k-th hole below the new count, ascending, takes the k-th unmarked agent
// from the end. The removed agents' entries go dead, out of every agent's
// reach, and the moved agents keep their place in the key order under their
// new slot.
__device__ __forceinline__ void list_remove_rep(const view& v, int r, int cur, int p, int32_t* sh)
{
	rep_counters& C = v.ctr[r];
	const int base = v.reps[r].base;
	const int nb = min(C.nbad, v.reps[r].cap);
	if (nb == 0)
		return;
	const int count = C.count, left = count - nb;
	int32_t* bad = v.bad + base;
	block_sort(bad, nb, sh);
	__syncthreads();
	int deaths = 0;
	for (int i = threadIdx.x; i < nb; i += blockDim.x)
	{
		const int t = v.tpos[base + bad[i]];
		deaths += v.flags[base + bad[i]] == PPC_FLAG_TO_REMOVE;
		v.sorted[t] = -1;
		v.lpos[p][t].x = 1e150;
		v.tmp[base + i] = 1; // the unmarked agents of the tail [left, count), from the end
	}
	__syncthreads();
	for (int i = threadIdx.x; i < nb; i += blockDim.x)
		if (bad[i] >= left)
			v.tmp[base + count - 1 - bad[i]] = 0;
	__syncthreads();
	int before = 0;
	for (int c = 0; c < nb; c += blockDim.x)
	{
		const int i = c + threadIdx.x;
		const int is = i < nb ? v.tmp[base + i] : 0;
		int total;
		const int k = before + block_exclusive_scan(is, total);
		if (is)
		{
			const int h = base + bad[k], q = base + count - 1 - i;
			list_move(v, cur, h, q);
			const int t = v.tpos[q];
			v.sorted[t] = h;
			v.tpos[h] = t;
			const long long word = __double_as_longlong(v.lpos[p][t].w);
			v.lpos[p][t].w = __longlong_as_double((long long)order_word((int32_t)(word >> 32), h));
		}
		before += total;
	}
	deaths = __reduce_add_sync(0xffffffffu, deaths);
	if ((threadIdx.x & 31) == 0 && deaths)
		atomicAdd(reinterpret_cast<unsigned long long*>(&C.deaths), (unsigned long long)deaths);
	__syncthreads();
	if (threadIdx.x == 0)
	{
		C.count = left;
		C.nbad = 0;
		v.binned[r] = left;
	}
	__syncthreads();
}

__device__ __forceinline__ unsigned long long ld_relaxed_u64(const unsigned long long* p)
{
	unsigned long long x;
	asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];" : "=l"(x) : "l"(p) : "memory");
	return x;
}

// The grid barriers of one launch. Barrier k uses word k & 1: a block can
// reach barrier k + 2 only after every block has left barrier k, so the word
// a slow block still polls does not change under it and all blocks read the
// same arrivals and events. Words count up over the launch. The state lives
// in shared memory and is thread 0's.
struct list_barrier
{
	unsigned k;					// barriers passed
	unsigned long long seen[2]; // each word's events so far
	unsigned long long ev, out;
};

// Waits for every block; returns the events the blocks brought, or all ones
// when a wait gave up (the state is then lost).
__device__ __forceinline__ unsigned long long list_wait(const view& v, const list_args& a, list_barrier& b,
														unsigned long long ev)
{
	if (__syncthreads_or(ev != 0))
	{
		if (threadIdx.x == 0)
			b.ev = 0;
		__syncthreads();
		if (ev)
			atomicOr(&b.ev, ev);
		__syncthreads();
		ev = b.ev;
	}
	if (threadIdx.x == 0)
	{
		// release and acquire order the whole block's accesses through the
		// block barriers around them
		const unsigned k = b.k++;
		unsigned long long* w = a.bar + 16 * (k & 1);
		const unsigned target = (k / 2 + 1) * gridDim.x;
		asm volatile("red.release.gpu.global.add.u64 [%0], %1;" ::"l"(w), "l"(1ull + ev) : "memory");
		unsigned long long x = ld_relaxed_u64(w);
		long long polls = 0;
		bool ok = true;
		while ((unsigned)x < target)
		{
			if (++polls > a.limit || ((polls & 1023) == 0 && (ld_relaxed_i32(v.err) & ERR_TIMEOUT)))
			{
				atomicOr(v.err, ERR_TIMEOUT);
				ok = false;
				break;
			}
			x = ld_relaxed_u64(w);
		}
		asm volatile("fence.acq_rel.gpu;" ::: "memory");
		x &= ~0xffffffffull;
		b.out = ok ? x - b.seen[k & 1] : ~0ull;
		b.seen[k & 1] = x;
	}
	__syncthreads();
	return b.out;
}

// Container update (after a removal), mesh and (`lists`) lists rebuilt by the
// whole grid; the new key-ordered rows go to lpos[p]. `flushed`: the
// slot-ordered rows are current. Returns false when a barrier gave up.
template <int DIMS>
__device__ __forceinline__ bool list_rebuild(const view& v, const list_args& a, list_barrier& bar, int p, bool remove,
										  bool flushed, bool lists, unsigned char* smem)
{
	const int T = blockDim.x, t0 = blockIdx.x * T + threadIdx.x, step = gridDim.x * T;
	const int cur = a.cur;
	if (!flushed)
	{
		const int n = *v.cursor;
		for (int t = t0; t < n; t += step)
			list_flush(v, cur, p, t);
		if (list_wait(v, a, bar, 0) == ~0ull)
			return false;
	}
	if (remove)
	{
		for (int r = blockIdx.x; r < v.nreps; r += gridDim.x)
		{
			compact_plan_rep(v, r, 0, a.springs, 1, 0, reinterpret_cast<int32_t*>(smem));
			__syncthreads(); // thread 0 finishes the serial plan before the next sort
		}
		if (list_wait(v, a, bar, 0) == ~0ull)
			return false;
	}
	while (true)
	{
		if (blockIdx.x == 0 && threadIdx.x == 0)
		{
			*v.bin_active = 1;
			v.lctl[LCTL_REACH] = 0;
			v.lctl[LCTL_DIRTY] = 0;
			v.lctl[LCTL_CAP] = v.lctl[LCTL_WANT];
			v.lctl[LCTL_FIT] = lists ? 1 : 0;
			*v.nl_used = 0;
		}
		for (int t = blockIdx.x * T; t < v.total_cap; t += step)
			bin_count_body(v, cur, t + threadIdx.x);
		if (list_wait(v, a, bar, 0) == ~0ull)
			return false;
		for (int b = blockIdx.x; b < v.ntiles; b += gridDim.x)
			bin_order_tile<0>(v, b, *reinterpret_cast<place_smem*>(smem), 1);
		if (list_wait(v, a, bar, 0) == ~0ull)
			return false;
		const int n = *v.cursor;
		for (int tb = blockIdx.x * T; tb < v.total_cap; tb += step)
		{
			const int t = tb + threadIdx.x;
			bin_copy_agent(v, cur, t, 0, v.spos4, v.sposf, 1);
			list_reach(v, t < n ? v.spos4[t].w : 0.0);
			list_positions(v, t, n);
		}
		bin_finish(v, t0, step);
		if (list_wait(v, a, bar, 0) == ~0ull)
			return false;
		const float skin = lists ? list_skin(v, a.voxel) : 0.0f;
		if (blockIdx.x == 0 && threadIdx.x == 0)
		{
			*a.skin_out = skin;
			v.lctl[LCTL_BUILT] = __float_as_int(skin);
		}
		if (!lists)
			return list_wait(v, a, bar, 0) != ~0ull;
		list_warp& w = reinterpret_cast<list_warp*>(smem)[threadIdx.x >> 5];
		for (int tb = blockIdx.x * T; tb < n; tb += step)
			list_build<DIMS, 2>(v, cur, p, tb + (threadIdx.x & ~31), n, skin, a.opts & FUSED_SPRINGS, w);
		if (list_wait(v, a, bar, 0) == ~0ull)
			return false;
		if (lctl_float(v, LCTL_WANT) >= skin)
			return true;
		if (list_wait(v, a, bar, 0) == ~0ull) // lists that did not fit are made again with the smaller skin
			return false;
	}
}

// The steps of a call. RESIDENT: the grid has a thread for every agent, which
// keeps the agent's rows and the first entries of its list in shared memory
// between the steps. The launch runs while every warp has its lists; where
// some do not fit, no skin is left, or they do not pay (kListDebt), it leaves
// the rest of the call (LCTL_LEFT), with the mesh current, to k_list_rest
// behind it.
template <int DIMS, bool F32, bool RESIDENT, int MOST>
__global__ void __launch_bounds__(MOST, 1)
	k_list_steps(const __grid_constant__ view v, const __grid_constant__ list_args a)
{
	// list entries whose loads are in flight together: as many as the
	// registers of MOST threads hold
	constexpr int BATCH = MOST > kListFew ? 2 : 4;
	extern __shared__ __align__(16) unsigned char smem[];
	__shared__ rep_info s_rep;
	if (ld_relaxed_i32(v.err) & ERR_TIMEOUT)
		return; // an earlier launch gave up: wait for the host
	if (blockIdx.x == 0 && threadIdx.x < 2)
		a.bar_next[16 * threadIdx.x] = 0;
	const int T = blockDim.x, t0 = blockIdx.x * T + threadIdx.x, step = gridDim.x * T;
	if (v.nreps == 1 && threadIdx.x == 0)
		s_rep = v.reps[0];
	const rep_info* reps = v.nreps == 1 ? &s_rep : v.reps;
	list_step_warp& w = reinterpret_cast<list_step_warp*>(smem)[threadIdx.x >> 5];
	list_cache lc;
	lc.T = T;
	lc.t0 = blockIdx.x * T;
	lc.n = RESIDENT ? a.cached : 0;
	lc.pair = reinterpret_cast<double4*>(smem + (T / 32) * sizeof(list_step_warp));
	lc.entry = reinterpret_cast<int2*>(lc.pair + (size_t)lc.n * T);
	__shared__ list_barrier bar;
	__shared__ int s_made, s_debt; // step that the lists in use were made before; their debt
	if (threadIdx.x == 0)
	{
		bar = list_barrier {};
		s_made = -v.lctl[LCTL_AGE];
		s_debt = v.lctl[LCTL_DEBT];
	}
	__syncthreads();
	int n = *v.cursor;
	int p = a.p;
	float skin = lctl_float(v, LCTL_BUILT);
	bool rebuild = v.lctl[LCTL_DIRTY] != 0;
	const bool cut = lctl_float(v, LCTL_WANT) < skin; // lists that did not fit
	if (a.refresh)
	{
		unsigned long long ev = 0;
		for (int t = t0; t < n; t += step)
			ev |= list_refresh<DIMS>(v, a.cur, p, t, skin);
		ev = list_wait(v, a, bar, ev);
		if (ev == ~0ull)
			return;
		rebuild = rebuild || ev != 0;
	}
	auto charge = [&](int k) { // the lists are to be made anew before step k
		if (threadIdx.x == 0)
		{
			s_debt = max(0, s_debt + kListPays - (k - s_made));
			s_made = k;
		}
	};
	if (rebuild)
		charge(0);
	rebuild = rebuild || cut;
	// past this barrier no block reads the control words of the old lists
	if (rebuild && list_wait(v, a, bar, 0) == ~0ull)
		return;
	list_own own;
	auto reload = [&]() {
		own = list_load(v, a, w, p, t0, n);
		const int m = own.s >= 0 && own.slab >= 0 ? min(own.cnt, lc.n) : 0;
		for (int k = 0; k < m; k++)
		{
			const int64_t e = own.slab + 32 * k + (threadIdx.x & 31);
			const int i = k * T + threadIdx.x;
			lc.entry[i] = v.nl[e];
			if (F32)
				reinterpret_cast<float4*>(lc.pair)[i] = reinterpret_cast<const float4*>(v.nl_pair)[e];
			else
				lc.pair[i] = v.nl_pair[e];
		}
		__syncwarp();
	};
	bool flushed = true, replay = false; // of the rebuild: the slot-ordered rows are current; removals are due
	for (int k = 0;; k++)
	{
		if (rebuild)
		{
			__syncthreads(); // the debt is thread 0's
			if (!list_rebuild<DIMS>(v, a, bar, p, replay, flushed, s_debt <= list_debt_limit(a.steps),
									smem))
				return;
			n = *v.cursor;
			skin = lctl_float(v, LCTL_BUILT);
		}
		if (k == 0 || rebuild)
		{
			const bool fit = v.lctl[LCTL_FIT] != 0;
			if (t0 == 0)
				v.lctl[LCTL_LEFT] = fit ? 0 : a.steps - k;
			if (!fit && k < a.steps)
				return;
		}
		if (k == a.steps)
			break;
		if (RESIDENT && (k == 0 || rebuild))
			reload();
		const bool last = k == a.steps - 1;
		unsigned long long ev = 0;
		if (RESIDENT)
			ev = list_step<DIMS, F32, BATCH>(v, a, reps, lc, w, own, p, t0, n, k == 0, last, skin);
		else
			for (int tb = blockIdx.x * T; tb < n; tb += step)
			{
				const int t = tb + threadIdx.x;
				own = list_load(v, a, w, p, t, n);
				list_prefetch(v, p, (t & ~31) + step, n);
				ev |= list_step<DIMS, F32, BATCH>(v, a, reps, lc, w, own, p, t, n, k == 0, last, skin);
			}
		p ^= 1;
		ev = list_wait(v, a, bar, ev);
		if (ev == ~0ull)
			return;
		rebuild = false;
		if (ev == 0)
			continue;
		const bool remove = ev >= kEventRemove, past = (unsigned)(ev >> 32 & 0xffff) != 0;
		replay = remove && a.springs;
		rebuild = replay || (past && !last);
		if (rebuild)
			charge(k + 1);
		flushed = last;
		if (past && last && !replay && t0 == 0)
			v.lctl[LCTL_DIRTY] = 1; // the next call rebuilds first
		if (remove && !replay)
		{
			for (int r = blockIdx.x; r < v.nreps; r += gridDim.x)
				list_remove_rep(v, r, a.cur, p, reinterpret_cast<int32_t*>(smem));
			if (list_wait(v, a, bar, 0) == ~0ull)
				return;
			if (RESIDENT && !rebuild && !last)
				reload();
		}
	}
	if (t0 == 0)
	{
		v.lctl[LCTL_AGE] = a.steps - s_made;
		v.lctl[LCTL_DEBT] = s_debt;
	}
	if (blockIdx.x == 0 && v.auto_springs)
		for (int r = threadIdx.x; r < v.nreps; r += T)
			v.ctr[r].spring_epoch += a.steps;
}

// The steps that k_list_steps left, without lists: the queue pass over the
// mesh, the container update and the mesh rebuild, separated by grid barriers,
// as in the persistent step (whose registers and blocks per SM bound it the
// same way). Its own kernel, since one with both bodies spilled registers in
// the steps over lists (29,000 cycles a step on 88,700 agents instead of
// 22,000); where nothing is left the launch costs a call about 3 us. The slot-
// ordered positions end in pos[a.cur], and the next lists start from a
// rebuild.
template <int DIMS, bool F32>
__global__ void __launch_bounds__(kPersistThreads)
	k_list_rest(const __grid_constant__ view v, const __grid_constant__ list_args a)
{
	extern __shared__ __align__(16) unsigned char smem[];
	if (ld_relaxed_i32(v.err) & ERR_TIMEOUT)
		return; // an earlier launch gave up: wait for the host
	if (blockIdx.x == 0 && threadIdx.x < 2)
		a.bar_next[16 * threadIdx.x] = 0;
	const int steps = v.lctl[LCTL_LEFT];
	if (steps == 0)
		return;
	__shared__ list_barrier bar;
	if (threadIdx.x == 0)
		bar = list_barrier {};
	__syncthreads();
	const int T = kPersistThreads, t0 = blockIdx.x * T, step = gridDim.x * T;
	int cur = a.cur;
	for (int k = a.steps - steps; k < a.steps; k++)
	{
		const int opts = k == 0 ? a.opts : a.opts & ~FUSED_VEL, nxt = cur ^ 1;
		for (int t = t0; t < v.total_cap; t += step)
			fused_queue_agent<DIMS, F32>(v, cur, opts, t + threadIdx.x,
										 reinterpret_cast<queue_smem*>(smem)->w[threadIdx.x >> 5]);
		if (list_wait(v, a, bar, 0) == ~0ull)
			return;
		for (int r = blockIdx.x; r < v.nreps; r += gridDim.x)
		{
			compact_plan_rep(v, r, 0, a.springs, 1, 0, reinterpret_cast<int32_t*>(smem));
			__syncthreads(); // thread 0 finishes the serial plan before the next sort
		}
		if (blockIdx.x == 0 && threadIdx.x == 0)
			*v.bin_active = 1;
		if (list_wait(v, a, bar, 0) == ~0ull)
			return;
		for (int t = t0; t < v.total_cap; t += step)
			bin_count_body(v, nxt, t + threadIdx.x);
		if (list_wait(v, a, bar, 0) == ~0ull)
			return;
		for (int b = blockIdx.x; b < v.ntiles; b += gridDim.x)
			bin_order_tile<kPersistThreads>(v, b, *reinterpret_cast<place_smem*>(smem), 1);
		if (list_wait(v, a, bar, 0) == ~0ull)
			return;
		for (int t = t0; t < v.total_cap; t += step)
			bin_copy_agent(v, nxt, t + threadIdx.x, 0, v.spos4, v.sposf, 1);
		bin_finish(v, t0 + threadIdx.x, step);
		if (list_wait(v, a, bar, 0) == ~0ull)
			return;
		cur = nxt;
	}
	if (cur != a.cur)
		for (int t = t0 + threadIdx.x; t < v.total_cap; t += step)
			v.pos[a.cur][t] = v.pos[cur][t];
	if (blockIdx.x == 0 && threadIdx.x == 0)
	{
		v.lctl[LCTL_DIRTY] = 1;
		v.lctl[LCTL_AGE] = kListPays; // the rebuild that the next lists start from is not theirs
		v.lctl[LCTL_DEBT] = 0;
	}
	if (blockIdx.x == 0 && v.auto_springs)
		for (int r = threadIdx.x; r < v.nreps; r += T)
			v.ctr[r].spring_epoch += a.steps;
}
