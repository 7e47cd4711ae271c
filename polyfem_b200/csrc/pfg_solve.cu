// Linear solve on the device: conjugate gradient with the diagonal (Jacobi)
// preconditioner on the context's assembled Hessian (full or Dirichlet-reduced
// CSC), the hand-off the Newton step makes to its linear solver after every
// assembly: the Hessian NLProblem::hessian returns (solver/NLProblem.cpp:615-621)
// goes to polysolve's linear::Solver (analyze_pattern / factorize / solve),
// called inside the Newton solver of polysolve@47dc48d (external).
//
// The iteration is Eigen's ConjugateGradient with DiagonalPreconditioner (Eigen
// 3.4, the version the reference pins in cmake/recipes/eigen.cmake), restated:
//   r = b - H x, rhs2 = |b|^2;  rhs2 == 0: x = 0, done
//   threshold = max(tol^2 rhs2, smallest normal double)
//   |r|^2 < threshold: done after 0 iterations
//   p = D^-1 r, rz = r.p, i = 0
//   while i < max_iter:
//     q = H p;  alpha = rz / p.q;  x += alpha p;  r -= alpha q
//     |r|^2 < threshold: stop
//     z = D^-1 r;  rz' = r.z;  beta = rz' / rz;  rz = rz';  p = z + beta p;  i += 1
//   iterations = i, relative residual = sqrt(|r|^2 / rhs2)
// with D^-1 = 1 / diag(H) where the diagonal is non-zero, else 1.
// One persistent cooperative kernel (k_cg) runs the iterations: the matrix streams
// through each warp's shared-memory stages, filled by bulk copies, the vectors live in
// 32-byte slots of one node each (its up to three free dofs, zero-padded), and two or
// three grid-wide exchanges per iteration separate H p with p.q, the step with r.r and
// r.z, and the new direction.  Every CTA forms the scalars from the same partials in the same order,
// so the stop test needs no host; the host reads the state once per batch.
//
// H is structurally and numerically symmetric (the reduction sums both triangles of
// every block in the same element order), so column j of the CSC is row j and
// q = H p is a gather: one warp per node's columns, no atomics.  Every dot product is a
// fixed-order reduction (warp butterfly, warps in order, CTAs in order), so the
// iterates are bitwise deterministic.
#include "pfg_bulk_span.h"
#include "pfg_internal.h"

#include <algorithm>
#include <vector>

namespace pfg
{

namespace
{

constexpr int CG_NT = 256;      // threads per block of every kernel here
constexpr int CG_MAX_GRID = 1184; // 148 SMs x 8: blocks of the grid-stride kernels
#ifndef PFG_SPMV_MINB
#define PFG_SPMV_MINB 8 // 64 warps per SM at 32 registers (a few spill): measured best
#endif

__device__ __forceinline__ double warp_sum(double v)
{
#pragma unroll
	for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
	return v;
}

// sum over the block's threads in a fixed order; the result is valid in thread 0
__device__ __forceinline__ double block_sum(double v)
{
	__shared__ double ws[CG_NT / 32];
	v = warp_sum(v);
	if ((threadIdx.x & 31) == 0) ws[threadIdx.x >> 5] = v;
	__syncthreads();
	double s = 0.0;
	if (threadIdx.x == 0)
#pragma unroll
		for (int w = 0; w < CG_NT / 32; ++w) s += ws[w];
	__syncthreads();
	return s;
}

__global__ void __launch_bounds__(CG_NT) k_diag_inv(int n, const int *__restrict__ outer, const int *__restrict__ inner,
													const double *__restrict__ vals, double *__restrict__ invd)
{
	for (int j = blockIdx.x * CG_NT + threadIdx.x; j < n; j += gridDim.x * CG_NT)
	{
		// rows of a column are sorted: binary search for the diagonal entry
		int lo = __ldg(outer + j), hi = __ldg(outer + j + 1);
		double d = 0.0;
		while (lo < hi)
		{
			const int mid = (lo + hi) >> 1;
			const int r = __ldg(inner + mid);
			if (r == j)
			{
				d = __ldg(vals + mid);
				break;
			}
			if (r < j)
				lo = mid + 1;
			else
				hi = mid;
		}
		invd[j] = d != 0.0 ? 1.0 / d : 1.0;
	}
}

// q = H p, one warp per column group (m <= 3 consecutive columns with the same rows,
// a node's dofs): each row index is loaded and p gathered once for the m columns.
__global__ void __launch_bounds__(CG_NT, PFG_SPMV_MINB) k_spmv(int ngroups, const int *__restrict__ groups,
												const int *__restrict__ outer, const int *__restrict__ inner,
												const double *__restrict__ vals, const double *__restrict__ p,
												double *__restrict__ q)
{
	const int lane = threadIdx.x & 31;
	const int wpb = CG_NT / 32;
	for (int g = blockIdx.x * wpb + (threadIdx.x >> 5); g < ngroups; g += gridDim.x * wpb)
	{
		int c0 = 3 * g, m = 3;
		if (groups)
		{
			const int code = __ldg(groups + g);
			c0 = code >> 2;
			m = code & 3;
		}
		const int k0 = __ldg(outer + c0), len = __ldg(outer + c0 + 1) - k0;
		const int o1 = m > 1 ? __ldg(outer + c0 + 1) : k0, o2 = m > 2 ? __ldg(outer + c0 + 2) : k0;
		double s0 = 0.0, s1 = 0.0, s2 = 0.0;
		for (int t = lane; t < len; t += 32)
		{
			const double pv = __ldg(p + __ldg(inner + k0 + t));
			s0 = fma(__ldg(vals + k0 + t), pv, s0);
			if (m > 1) s1 = fma(__ldg(vals + o1 + t), pv, s1);
			if (m > 2) s2 = fma(__ldg(vals + o2 + t), pv, s2);
		}
		s0 = warp_sum(s0);
		if (m > 1) s1 = warp_sum(s1);
		if (m > 2) s2 = warp_sum(s2);
		if (lane == 0)
		{
			q[c0] = s0;
			if (m > 1) q[c0 + 1] = s1;
			if (m > 2) q[c0 + 2] = s2;
		}
	}
}

// Plan of a system (CgPlan): neighbour blocks.  group_of[dof] = its column group.
__global__ void __launch_bounds__(CG_NT) k_group_of(int ngroups, const int *__restrict__ groups, int *__restrict__ group_of)
{
	for (int g = blockIdx.x * CG_NT + threadIdx.x; g < ngroups; g += gridDim.x * CG_NT)
	{
		const int code = groups ? __ldg(groups + g) : 12 * g + 3;
		for (int c = 0; c < (code & 3); ++c) group_of[(code >> 2) + c] = g;
	}
}

// A warp per group: its rows are runs of one neighbour group's dofs each.  count: the
// number of runs (dst == NULL), else dst[at[g] + k] = neighbour group * 4 + run length.
__global__ void __launch_bounds__(CG_NT) k_group_rows(int ngroups, const int *__restrict__ groups,
													  const int *__restrict__ outer, const int *__restrict__ inner,
													  const int *__restrict__ group_of, int *__restrict__ count,
													  const long long *__restrict__ at, int *__restrict__ dst)
{
	const int lane = threadIdx.x & 31, wpb = CG_NT / 32;
	for (int g = blockIdx.x * wpb + (threadIdx.x >> 5); g < ngroups; g += gridDim.x * wpb)
	{
		const int c0 = groups ? __ldg(groups + g) >> 2 : 3 * g;
		const int k0 = __ldg(outer + c0), len = __ldg(outer + c0 + 1) - k0;
		int runs = 0;
		for (int t0 = 0; t0 < len; t0 += 32)
		{
			const int t = t0 + lane;
			const int me = t < len ? __ldg(group_of + __ldg(inner + k0 + t)) : -1;
			const int before = t > 0 && t < len ? __ldg(group_of + __ldg(inner + k0 + t - 1)) : -1;
			const bool first = t < len && me != before;
			const unsigned starts = __ballot_sync(0xffffffffu, first);
			if (dst && first)
			{
				int m = 1;
				while (m < 3 && t + m < len && __ldg(group_of + __ldg(inner + k0 + t + m)) == me) ++m;
				dst[at[g] + runs + __popc(starts & ((1u << lane) - 1u))] = me * 4 + m;
			}
			runs += __popc(starts);
		}
		if (!dst && lane == 0) count[g] = runs;
	}
}

// dense vectors -> slots: r = b - q (q = H x of a starting guess, or NULL), x, D^-1,
// z = p = D^-1 r; part = (r.z, r.r, b.b) per block
__global__ void __launch_bounds__(CG_NT) k_cg_start(int ngroups, const int *__restrict__ groups,
													const double *__restrict__ invd, const double *__restrict__ b,
													const double *__restrict__ q, const double *__restrict__ x, CgWork w,
													double *__restrict__ part)
{
	double rz = 0.0, rr = 0.0, bb = 0.0;
	for (int g = blockIdx.x * CG_NT + threadIdx.x; g < ngroups; g += gridDim.x * CG_NT)
	{
		const int code = groups ? __ldg(groups + g) : 12 * g + 3;
		const int c0 = code >> 2, m = code & 3;
#pragma unroll
		for (int c = 0; c < 4; ++c)
		{
			const size_t k = 4 * (size_t)g + c;
			const bool on = c < m;
			const double bj = on ? b[c0 + c] : 0.0, dj = on ? invd[c0 + c] : 0.0;
			const double rj = on && q ? bj - q[c0 + c] : bj, zj = dj * rj;
			w.x[k] = on && q ? x[c0 + c] : 0.0;
			w.r[k] = rj;
			w.invd[k] = dj;
			w.z[k] = zj;
			w.p[k] = zj;
			rz = fma(rj, zj, rz);
			rr = fma(rj, rj, rr);
			bb = fma(bj, bj, bb);
		}
	}
	const double s0 = block_sum(rz), s1 = block_sum(rr), s2 = block_sum(bb);
	if (threadIdx.x == 0)
	{
		part[blockIdx.x] = s0;
		part[gridDim.x + blockIdx.x] = s1;
		part[2 * gridDim.x + blockIdx.x] = s2;
	}
}

// one block: the starting scalars from the per-block partials in block order
__global__ void __launch_bounds__(CG_NT) k_cg_start_scalars(const double *__restrict__ part, int count, double tol,
															double *__restrict__ sc)
{
	double s[3];
	for (int c = 0; c < 3; ++c)
	{
		double v = 0.0;
		for (int i = threadIdx.x; i < count; i += CG_NT) v += part[c * count + i];
		s[c] = block_sum(v);
	}
	if (threadIdx.x != 0) return;
	sc[CG_RZ] = s[0];
	sc[CG_RR] = s[1];
	sc[CG_RHS2] = s[2];
	const double thr = fmax(tol * tol * s[2], 2.2250738585072014e-308);
	sc[CG_THR] = thr;
	sc[CG_DONE] = (s[2] == 0.0 || s[1] < thr) ? 1.0 : 0.0;
	sc[CG_ITER] = 0.0;
	sc[CG_ERR] = 0.0;
}

__global__ void __launch_bounds__(CG_NT) k_cg_unpack(int ngroups, const int *__restrict__ groups,
													 const double *__restrict__ xs, double *__restrict__ x)
{
	for (int g = blockIdx.x * CG_NT + threadIdx.x; g < ngroups; g += gridDim.x * CG_NT)
	{
		const int code = groups ? __ldg(groups + g) : 12 * g + 3;
		for (int c = 0; c < (code & 3); ++c) x[(code >> 2) + c] = xs[4 * (size_t)g + c];
	}
}

// ------------------------------------------------------------------ the iterations
// k_cg: one CTA of 16 warps per SM, 128 registers a thread.
//
// H p.  Every warp owns a run of chunks (CgPlan: a few groups, at most CG_COST values) and
// feeds itself: two stages, one bulk copy for a chunk's values and one for its
// descriptors and neighbour codes, the next chunk on its way while one is multiplied.
// Nothing waits across warps: a ring shared by the CTA with a producer warp spent 1,300
// cycles a chunk on its barriers and copies (85 us an iteration at P2 24^3).  A run of at
// most two chunks is copied once and stays.  Odd iterations walk the runs backwards: the
// chunks read last are still in L2.
// A warp takes a group's 3 x 3 blocks a lane each, two groups at a time: per block one
// 32-byte slot of p and nine values from shared memory (a lane per row gathered p in 8-byte
// pieces and read an index per row instead of per block).
//
// Per iteration at P2 24^3 / P1 13^3: 115 / 24.8 us with five launches, 75 / 10.1 us here
// (before CG_PITCH 79 / 12.0; then 8 and 20 warps, or stages of 500 values: 105, 96 and 96 us
// at P2 24^3).  What is left at P2 24^3 is 41 us of streaming (240 MB, half of it from L2), the
// products that do not overlap it, and three exchanges; at P1 13^3 two exchanges and the chains
// behind them.
constexpr int CG_W = 16, CG_CTA = 32 * CG_W;
// doubles of values a stage holds: three whole groups of 27 3 x 3 blocks, an inner node of a
// hexahedral mesh (640 values, two of them: Q1 64^3 / 96^3 181 / 622 us an iteration, 169 / 543
// with three; P2 24^3 80.4, 78.9)
constexpr int CG_COST = 736;
constexpr int CG_BLOB = 180;              // ints of a chunk's descriptors and codes
constexpr int CG_SPIN = 1 << 22;          // bound of every wait (an exchange: about a second)
constexpr int CG_PK = 5, CG_MAX_CTAS = 32 * CG_PK; // packets per lane of an exchange; CTAs
// uint4 from one CTA's packet to the next.  Packets side by side share the L2 slices that all
// CTAs poll, and what an exchange takes then hangs on where the array lies: P1 13^3 9.7 to
// 13.3 us an iteration at 19 places within 512 KB, 256 bytes apart 9.8 to 10.3 (P1 8^3 8.0 to
// 10.7, 6.9 to 7.8); streaming P2 20^3 49.5 to 51.9, 128 bytes apart 47.1 to 48.4, 256 47.9 to 48.8
constexpr int CG_PITCH = 16;
constexpr int CG_OWN = 256;               // own groups whose q (and, FUSED, p) stay in shared memory
// a chunk's blob: head (first group, groups, -, -), a descriptor per group (first column * 4 +
// columns, first value in the chunk, rows | all blocks 3 x 3 << 30, first code in the blob)
// with an end entry, the codes (neighbour group * 4 + its dofs)
struct __align__(16) CgStage
{
	double v[CG_COST + 2]; // + 2: the copies move whole 16-byte units (bulk_span)
	int4 blob[CG_BLOB / 4];
};
struct CgSmem // 224 KB
{
	CgStage st[CG_W][2];
	unsigned long long full[CG_W][2];
	double q[4 * CG_OWN], p[4 * CG_OWN];
	double red[2][32], sum[2];
	int stop;
};

__device__ __forceinline__ unsigned smem_u32(const void *p) { return (unsigned)__cvta_generic_to_shared(p); }
__device__ __forceinline__ bool mbar_test(unsigned long long *b, unsigned parity)
{
	unsigned ok;
	asm volatile("{\n.reg .pred p;\nmbarrier.try_wait.parity.acquire.cta.shared::cta.b64 p, [%1], %2;\nselp.u32 %0, 1, 0, p;\n}"
				 : "=r"(ok)
				 : "r"(smem_u32(b)), "r"(parity)
				 : "memory");
	return ok;
}
__device__ __forceinline__ void bulk_load(void *dst, const void *src, unsigned bytes, unsigned long long *bar)
{
	asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(smem_u32(dst)),
				 "l"(src), "r"(bytes), "r"(smem_u32(bar))
				 : "memory");
}

// Sums of a and b over the warp, written to *sa and *sb: the first step folds the two into
// one value per half warp (6 double shuffles for 10)
__device__ __forceinline__ void warp_sum2(double a, double b, double *sa, double *sb)
{
	const int lane = threadIdx.x & 31;
	const bool up = lane & 16;
	double v = __shfl_xor_sync(0xffffffffu, up ? a : b, 16) + (up ? b : a);
#pragma unroll
	for (int o = 8; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
	if ((lane & 15) == 0) *(up ? sb : sa) = v;
}
// The sum over the warp of s[0], s[1], s[2] in lanes 0, 8 and 16 (lane 24: nothing): 7 double
// shuffles for 15
__device__ __forceinline__ double warp_sum3(const double (&s)[3])
{
	const int lane = threadIdx.x & 31;
	const bool h16 = lane & 16, h8 = lane & 8;
	double v = __shfl_xor_sync(0xffffffffu, h16 ? s[0] : s[2], 16) + (h16 ? s[2] : s[0]);
	double u = s[1] + __shfl_xor_sync(0xffffffffu, s[1], 16);
	// lanes with bit 3 clear keep v (s0 below lane 16, s2 above), the others u (s1)
	double t = __shfl_xor_sync(0xffffffffu, h8 ? v : u, 8) + (h8 ? u : v);
#pragma unroll
	for (int o = 4; o > 0; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
	return t;
}

// Grid-wide sums in one exchange of packets, a barrier as well (cooperative launch: all
// CTAs resident), entered by all threads.  Every CTA publishes its partial sums of
// a and b over its threads in a fixed order, each 8-byte word carrying half a double and
// the exchange's number; one warp of every CTA reads all packets until all carry it, and
// adds them in CTA order: one store and one poll round trip, against three trips for a
// counter, a generation word and the partials.  DATA: what the CTAs wrote before the
// exchange is visible to all after it (the two fences, ~1 us; only needed where others'
// vector entries are read next).  Three packet arrays in turn: a CTA can only overwrite
// one after all have read it.  Bounded: false once any wait has given up.  A CTA that gives up
// can leave others an exchange ahead, so every launch has numbers of its own (CgPlan::gen): the
// packets such a launch leaves behind match nothing later.
struct Sums
{
	double a, b;
};
__device__ __forceinline__ uint4 ld_packet(const uint4 *p)
{
	uint4 v;
	asm volatile("ld.relaxed.gpu.global.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(p) : "memory");
	return v;
}
template <int NV, bool DATA, int PITCH>
__device__ __forceinline__ bool exchange(CgSmem &S, uint4 *pk, int G, unsigned gen, double a, double b, int *err, Sums &out)
{
	const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
	if (NV > 1)
		warp_sum2(a, b, S.red[0] + warp, S.red[1] + warp);
	else if (NV > 0)
	{
		a = warp_sum(a);
		if (lane == 0) S.red[0][warp] = a;
	}
	__syncthreads();
	if (warp == 0)
	{
		if (NV > 0) a = warp_sum(lane < CG_W ? S.red[0][lane] : 0.0);
		if (NV > 1) b = warp_sum(lane < CG_W ? S.red[1][lane] : 0.0);
		if (lane == 0)
		{
			if (DATA) __threadfence(); // the CTA's writes before its packet
			uint4 *mine = pk + PITCH * blockIdx.x;
			asm volatile("st.relaxed.gpu.global.v4.u32 [%0], {%1, %2, %3, %2};" ::"l"(mine), "r"(__double2loint(a)), "r"(gen),
						 "r"(__double2hiint(a))
						 : "memory");
			if (NV > 1)
				asm volatile("st.relaxed.gpu.global.v4.u32 [%0], {%1, %2, %3, %2};" ::"l"(mine + 1), "r"(__double2loint(b)),
							 "r"(gen), "r"(__double2hiint(b))
							 : "memory");
		}
		// a lane's packets are read together, so a round is one trip to L2
		double sa = 0.0, sb = 0.0;
		uint4 u[CG_PK], v[NV > 1 ? CG_PK : 1];
		bool wait = true;
		for (int spin = 0; spin < CG_SPIN && wait; ++spin)
		{
#pragma unroll
			for (int j = 0; j < CG_PK; ++j)
			{
				const int i = min(lane + 32 * j, G - 1);
				u[j] = ld_packet(pk + PITCH * i);
				if (NV > 1) v[j] = ld_packet(pk + PITCH * i + 1);
			}
			wait = false;
#pragma unroll
			for (int j = 0; j < CG_PK; ++j)
			{
				wait |= u[j].y != gen || u[j].w != gen;
				if (NV > 1) wait |= v[j].y != gen || v[j].w != gen;
			}
		}
		bool bad = wait;
#pragma unroll
		for (int j = 0; j < CG_PK; ++j)
			if (lane + 32 * j < G)
			{
				if (NV > 0) sa += __hiloint2double((int)u[j].z, (int)u[j].x);
				if (NV > 1) sb += __hiloint2double((int)v[j].z, (int)v[j].x);
			}
		if (DATA) __threadfence(); // the other CTAs' writes before what follows
		if (NV > 0) sa = warp_sum(sa);
		if (NV > 1) sb = warp_sum(sb);
		bad = __any_sync(0xffffffffu, bad);
		if (lane == 0)
		{
			S.sum[0] = sa;
			S.sum[1] = sb;
			if (bad)
			{
				atomicExch(err, 1);
				S.stop = 1;
			}
		}
	}
	__syncthreads();
	out.a = S.sum[0];
	out.b = S.sum[1];
	return *(volatile int *)&S.stop == 0;
}

// a slot in one 32-byte load
struct Slot
{
	double x, y, z;
};
__device__ __forceinline__ Slot ld_slot(const double *v, int g)
{
	Slot s;
	[[maybe_unused]] double pad;
	asm volatile("ld.global.v4.f64 {%0, %1, %2, %3}, [%4];" : "=d"(s.x), "=d"(s.y), "=d"(s.z), "=d"(pad) : "l"(v + 4 * (size_t)g));
	return s;
}
// the search direction of group g: p, or (FUSED) z + beta p_old
template <bool FUSED>
__device__ __forceinline__ Slot direction(const double *p, const double *z, double beta, int g)
{
	Slot s = ld_slot(p, g);
	if (FUSED)
	{
		const Slot t = ld_slot(z, g);
		s.x = fma(beta, s.x, t.x);
		s.y = fma(beta, s.y, t.y);
		s.z = fma(beta, s.z, t.z);
	}
	return s;
}

// The lane's share of one group's sums over its rows of H(row, c0 + c) p(row), c = 0, 1, 2.
// sv, sn: its values (columns len apart) and neighbour codes; a lane per block.
template <bool FUSED>
__device__ __forceinline__ void group_product(const double *sv, const int *sn, int nblk, int len, int m, const double *p,
											  const double *z, double beta, int lane, double (&s)[3])
{
	int base = 0;
	for (int k0 = 0; k0 < nblk; k0 += 32)
	{
		const int k = k0 + lane;
		const int code = k < nblk ? sn[k] : 0, mr = code & 3;
		Slot d = {0.0, 0.0, 0.0};
		if (k < nblk) d = direction<FUSED>(p, z, beta, code >> 2);
		int incl = mr; // rows of the blocks up to this one
#pragma unroll
		for (int o = 1; o < 32; o *= 2)
		{
			const int y = __shfl_up_sync(0xffffffffu, incl, o);
			if (lane >= o) incl += y;
		}
		const double *v = sv + base + incl - mr;
#pragma unroll
		for (int c = 0; c < 3; ++c)
			if (c < m)
			{
				if (mr > 0) s[c] = fma(v[c * len], d.x, s[c]);
				if (mr > 1) s[c] = fma(v[c * len + 1], d.y, s[c]);
				if (mr > 2) s[c] = fma(v[c * len + 2], d.z, s[c]);
			}
		base += __shfl_sync(0xffffffffu, incl, 31);
	}
}

// The lanes' shares of NG groups of a chunk (descriptors d, at most 32 blocks each, all
// 3 x 3) at once
template <bool FUSED, int NG>
__device__ __forceinline__ void group_products(const double *sv, const int *blob, const int4 (&d)[NG], const int (&nblk)[NG],
											   const double *p, const double *z, double beta, int lane, double (&s)[NG][3])
{
	Slot g[NG];
#pragma unroll
	for (int h = 0; h < NG; ++h)
	{
		g[h] = {0.0, 0.0, 0.0};
		if (lane < nblk[h]) g[h] = direction<FUSED>(p, z, beta, blob[d[h].w + lane] >> 2);
	}
#pragma unroll
	for (int h = 0; h < NG; ++h)
	{
		const int len = d[h].z & 0x3fffffff;
		const double *v = sv + d[h].y + 3 * min(lane, nblk[h] - 1); // past the end: the last block, times zero
#pragma unroll
		for (int c = 0; c < 3; ++c)
			s[h][c] = lane < nblk[h] ? fma(v[c * len + 2], g[h].z, fma(v[c * len + 1], g[h].y, v[c * len] * g[h].x)) : 0.0;
	}
}

// EDGE: the array of values does not end on 16-byte units; the warps that own its first and
// last chunk clip their copies.  A variant, because the test alone costs the streaming kernel
// 0.7% (P2 24^3 79.3 -> 79.9 us an iteration); a resident run copies once, and always tests.
// FUSED (all runs resident): the new direction z + beta p_old is formed where H p gathers
// it, which reads two slots per block but saves the third exchange of an iteration.
template <bool FUSED, bool EDGE>
__global__ void __launch_bounds__(CG_CTA, 1) k_cg(CgPlan pl, const double *vals, CgWork w, int iters)
{
	extern __shared__ __align__(16) unsigned char cg_raw[];
	CgSmem &S = *reinterpret_cast<CgSmem *>(cg_raw);
	const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
	double *sc = w.sc;
	int *err = reinterpret_cast<int *>(sc + CG_ERR);
	if (sc[CG_DONE] != 0.0) return; // the same for every CTA: written before this launch
	const int it0 = (int)sc[CG_ITER];
	if (tid == 0)
	{
		for (int i = 0; i < 2 * CG_W; ++i)
			asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_u32(&S.full[0][0] + i)) : "memory");
		S.stop = 0;
		asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
	}
	// this warp's run of chunks, this CTA's groups: what it multiplies is what it steps, so
	// q, x and r stay its own
	const int2 *run = pl.run + blockIdx.x * CG_W;
	const int ch0 = run[warp].x, nch = run[warp + 1].x - ch0;
	const int g0 = run[0].y, nown = run[CG_W].y - g0;
	const bool resident = nch <= 2;
	const bool edge = EDGE && ((blockIdx.x == 0 && warp == 0) || ch0 + nch == pl.chunks);
	__syncthreads();
	// the chunks' entries (blob in 16-byte units, its size in them, first value, values; no
	// values: too large to stage), 32 at a time, a lane each
	int have = -1;
	int4 ent = make_int4(0, 0, 0, 0);
	unsigned par[2] = {0u, 0u}; // parity of the stages' next completion
	int load = 0, used = 0;     // chunks requested and taken, for the stage of each
	const auto request = [&](int i) {
		if ((i >> 5) != have)
		{
			have = i >> 5;
			ent = __ldg(pl.chunk + ch0 + min(32 * have + lane, nch - 1));
		}
		const int b0 = __shfl_sync(0xffffffffu, ent.x, i & 31), bn = __shfl_sync(0xffffffffu, ent.y, i & 31);
		const int v0 = __shfl_sync(0xffffffffu, ent.z, i & 31), nv = __shfl_sync(0xffffffffu, ent.w, i & 31);
		const int st = load++ & 1;
		if (lane == 0)
		{
			CgStage &T = S.st[warp][st];
			unsigned long long *full = &S.full[warp][st];
			const double *v = vals + v0;
			const int mv = (int)(((size_t)v >> 3) & 1);
			unsigned bv = nv ? (unsigned)((nv + mv + 1) / 2) * 16u : 0u;
			const double *src = v - mv;
			double *dst = T.v;
			if (EDGE && edge) // see bulk_span
			{
				const BulkSpan sp = bulk_span(v0, nv, pl.nnz, mv);
				if (sp.lo) T.v[mv] = __ldg(v);
				if (sp.hi) T.v[mv + nv - 1] = __ldg(v + nv - 1);
				bv = (unsigned)(sp.end - sp.begin) * 8u;
				src = v + sp.begin;
				dst = T.v + mv + sp.begin;
			}
			asm volatile("mbarrier.arrive.expect_tx.release.cta.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(full)),
						 "r"(bv + (unsigned)bn * 16u)
						 : "memory");
			if (bv) bulk_load(dst, src, bv, full);
			bulk_load(T.blob, pl.blob + b0, (unsigned)bn * 16u, full);
		}
		return make_int2(v0, nv);
	};
	int2 vq[2] = {make_int2(0, 0), make_int2(0, 0)}; // first value and count of the chunk in each stage
	const auto back = [&](int it) { return !resident && ((it0 + it) & 1); };
	for (int i = 0; i < min(nch, 2); ++i) vq[i] = request(back(0) ? nch - 1 - i : i);
	// the next chunk requested is here; false: gave up, nothing more is taken or requested
	const auto take = [&]() {
		const int st = used & 1;
		bool here = false;
		for (int spin = 0; !here && spin < CG_SPIN; ++spin) here = mbar_test(&S.full[warp][st], par[st]);
		here = __all_sync(0xffffffffu, here);
		if (here)
		{
			par[st] ^= 1u;
			++used;
		}
		else if (lane == 0)
		{
			atomicExch(err, 1);
			S.stop = 1;
		}
		return here;
	};
	int own_chunks = nch; // to multiply: none when a resident one did not come
	if (resident)
		while (used < load)
			if (!take())
			{
				own_chunks = 0;
				break;
			}
	const int G = gridDim.x + pl.missing; // (pl.ctas, the same, from the parameters: 0.1 us an iteration slower at P1 13^3)
	double *q = nown <= CG_OWN ? S.q : w.q + 4 * (size_t)g0, *po = S.p;
	unsigned gen = pl.gen; // exchange numbers given to earlier launches
	uint4 *pk = pl.packets;
	constexpr int PITCH = FUSED ? CG_PITCH : CG_PITCH / 2;
	const double thr = sc[CG_THR];
	double rz = sc[CG_RZ], rr = sc[CG_RR], alpha = 0.0, beta = it0 ? sc[CG_BETA] : 0.0;
	bool done = false, ok = true;
	int it = 0;
	for (; it < iters; ++it)
	{
		// q = H p, p.q; FUSED: p_old and p alternate between two buffers
		const bool odd = (it0 + it) & 1;
		const double *pin = FUSED && odd ? w.p2 : w.p;
		double *pout = FUSED ? (odd ? w.p : w.p2) : w.p;
		double pq = 0.0;
		const int comp = lane >> 3; // lanes 0, 8, 16, 24: entries 0, 1, 2 and the padding, as warp_sum3 leaves the sums
		const bool mine = (lane & 7) == 0;
		const auto own_direction = [&](int g) {
			double pv = 0.0;
			if (mine && comp < 3)
			{
				const size_t o = 4 * (size_t)g + comp;
				pv = *(const volatile double *)(pin + o);
				if (FUSED) pv = fma(beta, pv, *(const volatile double *)(w.z + o));
			}
			return pv;
		};
		const auto put = [&](int g, double pv, double s) {
			if (!mine) return;
			const double qc = comp < 3 ? s : 0.0;
			q[4 * (g - g0) + comp] = qc;
			if (FUSED)
			{
				pout[4 * (size_t)g + comp] = pv;
				if (nown <= CG_OWN) po[4 * (g - g0) + comp] = pv;
			}
			pq = fma(pv, qc, pq);
		};
		for (int i = 0; i < own_chunks; ++i)
		{
			const int st = resident ? i : used & 1;
			if (!resident && !take()) break;
			const CgStage &T = S.st[warp][st];
			const int *blob = reinterpret_cast<const int *>(T.blob);
			const int4 head = T.blob[0];
			const int4 *desc = T.blob + 1;
			const int v0 = st ? vq[1].x : vq[0].x, nv = st ? vq[1].y : vq[0].y;
			const double *sv = nv ? T.v + (((size_t)(vals + v0) >> 3) & 1) : vals + v0; // one group too large to stage: from memory
			// once the chunk's last values are read (before they are summed over the lanes): the
			// chunk two ahead into the stage, of this iteration's walk or the next's
			const auto next = [&]() {
				if (resident) return;
				__syncwarp();
				int n = i + 2, ni = it;
				if (n >= nch)
				{
					n -= nch;
					++ni;
				}
				if (ni < iters)
				{
					const int2 r = request(back(ni) ? nch - 1 - n : n);
					if (st) vq[1] = r;
					else vq[0] = r;
				}
			};
			int j = 0;
			for (; j + 1 < head.y; j += 2)
			{
				const int4 d[2] = {desc[j], desc[j + 1]};
				const int nb[2] = {d[1].w - d[0].w, desc[j + 2].w - d[1].w};
				if (!(d[0].z & d[1].z & (1 << 30)) || max(nb[0], nb[1]) > 32) break;
				const double p0 = own_direction(head.x + j), p1 = own_direction(head.x + j + 1);
				double s[2][3];
				group_products<FUSED, 2>(sv, blob, d, nb, pin, w.z, beta, lane, s);
				if (j + 2 == head.y) next();
				const double s0 = warp_sum3(s[0]), s1 = warp_sum3(s[1]);
				put(head.x + j, p0, s0);
				put(head.x + j + 1, p1, s1);
			}
			for (; j < head.y; ++j)
			{
				const int4 d[1] = {desc[j]};
				const int nb[1] = {desc[j + 1].w - d[0].w};
				const double p0 = own_direction(head.x + j);
				double s[1][3] = {};
				if ((d[0].z & (1 << 30)) && nb[0] <= 32 && nv)
					group_products<FUSED, 1>(sv, blob, d, nb, pin, w.z, beta, lane, s);
				else
					group_product<FUSED>(sv + d[0].y, nv ? blob + d[0].w : pl.big + d[0].w, nb[0], d[0].z & 0x3fffffff, d[0].x & 3, pin, w.z,
										 beta, lane, s[0]);
				if (j + 1 == head.y) next();
				put(head.x + j, p0, warp_sum3(s[0]));
			}
		}
		Sums sum;
		if (!(ok = exchange<1, false, PITCH>(S, pk, G, ++gen, pq, 0.0, err, sum))) break;
		alpha = rz / sum.a;
		// x += alpha p, r -= alpha q, z = D^-1 r
		const double *pown = FUSED && nown <= CG_OWN ? po : pout + 4 * (size_t)g0;
		double srr = 0.0, srz = 0.0;
		for (int g = tid; g < nown; g += CG_CTA)
		{
			const size_t o = 4 * (size_t)(g0 + g);
#pragma unroll
			for (int h = 0; h < 4; h += 2)
			{
				const double2 p = *reinterpret_cast<const double2 *>(pown + 4 * g + h), qv = *reinterpret_cast<const double2 *>(q + 4 * g + h);
				const double2 iv = *reinterpret_cast<const double2 *>(w.invd + o + h);
				double2 x = *reinterpret_cast<const double2 *>(w.x + o + h), r = *reinterpret_cast<const double2 *>(w.r + o + h);
				x.x = fma(alpha, p.x, x.x);
				x.y = fma(alpha, p.y, x.y);
				r.x = fma(-alpha, qv.x, r.x);
				r.y = fma(-alpha, qv.y, r.y);
				if (h) x.y = r.y = 0.0; // the slot's padding
				const double2 z = make_double2(iv.x * r.x, h ? 0.0 : iv.y * r.y);
				*reinterpret_cast<double2 *>(w.x + o + h) = x;
				*reinterpret_cast<double2 *>(w.r + o + h) = r;
				*reinterpret_cast<double2 *>(w.z + o + h) = z;
				srr = fma(r.y, r.y, fma(r.x, r.x, srr));
				srz = fma(r.y, z.y, fma(r.x, z.x, srz));
			}
		}
		if (!(ok = exchange<2, FUSED, PITCH>(S, pk + PITCH * G, G, ++gen, srr, srz, err, sum))) break;
		rr = sum.a;
		if (rr < thr)
		{
			done = true; // converged: x and r stay as they are, the count is not advanced
			break;
		}
		beta = sum.b / rz;
		rz = sum.b;
		if (!FUSED)
		{
			for (int g = tid; g < nown; g += CG_CTA)
			{
				const size_t o = 4 * (size_t)(g0 + g);
#pragma unroll
				for (int h = 0; h < 4; h += 2)
				{
					const double2 z = *reinterpret_cast<const double2 *>(w.z + o + h);
					double2 p = *reinterpret_cast<const double2 *>(w.p + o + h);
					p.x = fma(beta, p.x, z.x);
					p.y = fma(beta, p.y, z.y);
					*reinterpret_cast<double2 *>(w.p + o + h) = p;
				}
			}
			if (!(ok = exchange<0, true, PITCH>(S, pk + 2 * PITCH * G, G, ++gen, 0.0, 0.0, err, sum))) break;
		}
	}
	// copies still in flight (the solve stopped, or a wait gave up): wait for them before leaving
	for (; used < load; ++used)
	{
		const int st = used & 1;
		for (int spin = 0; spin < CG_SPIN && !mbar_test(&S.full[warp][st], par[st]); ++spin)
			;
		par[st] ^= 1u;
	}
	if (tid == 0 && blockIdx.x == 0)
	{
		sc[CG_ALPHA] = alpha;
		sc[CG_BETA] = beta;
		sc[CG_RZ] = rz;
		sc[CG_RR] = rr;
		sc[CG_ITER] = (double)(it0 + it);
		sc[CG_DONE] = !ok ? 2.0 : done ? 1.0 : 0.0;
	}
}

int grid_vec(int n) { return n <= 0 ? 1 : (int)std::min<long long>(CG_MAX_GRID, ((long long)n + CG_NT - 1) / CG_NT); }
int grid_spmv(int ngroups) { return ngroups <= 0 ? 1 : (int)std::min<long long>(CG_MAX_GRID, ((long long)ngroups + 7) / 8); }

} // namespace

size_t cg_partials_doubles() { return 3 * (size_t)CG_MAX_GRID; } // three per block of k_cg_start

cudaError_t launch_hessian_apply(int n_nodes, const int *outer, const int *inner, const double *vals, const double *p,
								 double *q, cudaStream_t s)
{
	if (n_nodes > 0)
		k_spmv<<<grid_spmv(n_nodes), CG_NT, 0, s>>>(n_nodes, nullptr, outer, inner, vals, p, q);
	return cudaGetLastError();
}

cudaError_t launch_cg_diag_inv(int n, const int *outer, const int *inner, const double *vals, double *invd,
							   cudaStream_t s)
{
	if (n > 0) k_diag_inv<<<grid_vec(n), CG_NT, 0, s>>>(n, outer, inner, vals, invd);
	return cudaGetLastError();
}

// The plan of a system, from its device pattern: descriptors, chunks and runs on the host
// (a few words per group), neighbour codes on the device.
cudaError_t build_cg_plan(int n, int ngroups, const int *groups, const int *outer, const int *inner, int max_ctas, CgPlan *pl,
						  cudaStream_t s)
{
	*pl = CgPlan();
	if (ngroups <= 0) return cudaSuccess;
	int dev = 0, sms = 0;
	cudaError_t e;
	if ((e = cudaGetDevice(&dev)) != cudaSuccess) return e;
	if ((e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev)) != cudaSuccess) return e;
	std::vector<int> ho((size_t)n + 1), hg, cnt(ngroups);
	int *d_of = nullptr, *d_cnt = nullptr;
	const int gs = grid_spmv(ngroups);
	if ((e = cudaMalloc(&d_of, sizeof(int) * (size_t)std::max(n, 1))) == cudaSuccess &&
		(e = cudaMalloc(&d_cnt, sizeof(int) * (size_t)ngroups)) == cudaSuccess)
	{
		k_group_of<<<grid_vec(ngroups), CG_NT, 0, s>>>(ngroups, groups, d_of);
		k_group_rows<<<gs, CG_NT, 0, s>>>(ngroups, groups, outer, inner, d_of, d_cnt, nullptr, nullptr);
		if (groups) hg.resize(ngroups);
		if ((e = cudaGetLastError()) == cudaSuccess &&
			(e = cudaMemcpyAsync(cnt.data(), d_cnt, sizeof(int) * (size_t)ngroups, cudaMemcpyDeviceToHost, s)) == cudaSuccess &&
			(e = cudaMemcpyAsync(ho.data(), outer, sizeof(int) * ((size_t)n + 1), cudaMemcpyDeviceToHost, s)) == cudaSuccess &&
			(!groups ||
			 (e = cudaMemcpyAsync(hg.data(), groups, sizeof(int) * (size_t)ngroups, cudaMemcpyDeviceToHost, s)) == cudaSuccess))
			e = cudaStreamSynchronize(s);
	}
	long long *d_at = nullptr;
	if (e == cudaSuccess)
	{
		const auto code_of = [&](int g) { return groups ? hg[g] : 12 * g + 3; };
		const auto values_of = [&](int g) {
			const int code = code_of(g);
			return (long long)(code & 3) * (ho[(code >> 2) + 1] - ho[code >> 2]);
		};
		long long total = 0;
		for (int g = 0; g < ngroups; ++g) total += values_of(g);
		// two groups for a warp at least: each CTA more costs every exchange
		const int ctas = std::min({sms, max_ctas, CG_MAX_CTAS, (ngroups + 2 * CG_W - 1) / (2 * CG_W)}), warps = ctas * CG_W;
		std::vector<int4> chunk, blob; // blob: codes are filled in on the device
		std::vector<int2> run;
		std::vector<long long> at(ngroups);
		long long nbig = 0, done = 0;
		std::vector<int> cur; // groups of the open chunk
		long long cur_v = 0, cur_n = 0;
		const auto close = [&]() {
			if (cur.empty()) return;
			const size_t b0 = blob.size();
			const int v0 = ho[code_of(cur[0]) >> 2], ng = (int)cur.size();
			const bool huge = cur_v > CG_COST || 8 + 4 * ng + cur_n > CG_BLOB; // one group
			blob.push_back(make_int4(cur[0], ng, 0, 0));
			int n0 = huge ? 0 : 4 * (ng + 2);
			if (huge) at[cur[0]] = -1 - nbig; // its codes go to the overflow array
			for (int g : cur)
			{
				const int code = code_of(g), c0 = code >> 2, len = ho[c0 + 1] - ho[c0];
				const bool full = (code & 3) == 3 && len == 3 * cnt[g];
				if (!huge) at[g] = 4 * (long long)b0 + n0;
				blob.push_back(make_int4(code, ho[c0] - v0, len | (full ? 1 << 30 : 0), huge ? (int)nbig : n0));
				n0 += cnt[g];
			}
			blob.push_back(make_int4(0, 0, 0, huge ? (int)nbig + cnt[cur[0]] : n0));
			if (huge) nbig += cnt[cur[0]];
			else blob.resize(b0 + (size_t)(n0 + 3) / 4);
			chunk.push_back(make_int4((int)b0, (int)(blob.size() - b0), v0, huge ? 0 : (int)cur_v));
			cur.clear();
			cur_v = cur_n = 0;
		};
		// boundaries of the warps' runs at even shares of the values
		int w = 0;
		for (int g = 0; g < ngroups; ++g)
		{
			while (w < warps && (double)done >= (double)w * (double)total / warps)
			{
				close();
				run.push_back(make_int2((int)chunk.size(), g));
				++w;
			}
			const long long nv = values_of(g);
			if (!cur.empty() && (cur_v + nv > CG_COST || 4 * ((long long)cur.size() + 3) + cur_n + cnt[g] > CG_BLOB)) close();
			cur.push_back(g);
			cur_v += nv;
			cur_n += cnt[g];
			done += nv;
			if (cur_v > CG_COST || 4 * ((long long)cur.size() + 2) + cur_n > CG_BLOB) close();
		}
		close();
		while ((int)run.size() <= warps) run.push_back(make_int2((int)chunk.size(), ngroups));
		pl->ctas = ctas;
		pl->nnz = ho[n];
		pl->chunks = (int)chunk.size();
		pl->resident = true;
		for (int i = 0; i < warps; ++i) pl->resident = pl->resident && run[i + 1].x - run[i].x <= 2;
		// the overflow codes sit behind the blobs
		const long long big0 = 4 * (long long)blob.size();
		for (long long &x : at)
			if (x < 0) x = big0 + (-1 - x);
		blob.resize(blob.size() + (size_t)(nbig + 3) / 4);
		const size_t packet_bytes = 3 * sizeof(uint4) * CG_PITCH * (size_t)ctas;
		if ((e = cudaMalloc(&pl->run, sizeof(int2) * run.size())) == cudaSuccess &&
			(e = cudaMalloc(&pl->chunk, sizeof(int4) * chunk.size())) == cudaSuccess &&
			(e = cudaMalloc(&pl->blob, sizeof(int4) * blob.size())) == cudaSuccess &&
			(e = cudaMalloc(&d_at, sizeof(long long) * at.size())) == cudaSuccess &&
			(e = cudaMalloc(&pl->packets, packet_bytes)) == cudaSuccess &&
			(e = cudaMemsetAsync(pl->packets, 0, packet_bytes, s)) == cudaSuccess &&
			(e = cudaMemcpyAsync(pl->run, run.data(), sizeof(int2) * run.size(), cudaMemcpyHostToDevice, s)) == cudaSuccess &&
			(e = cudaMemcpyAsync(pl->chunk, chunk.data(), sizeof(int4) * chunk.size(), cudaMemcpyHostToDevice, s)) == cudaSuccess &&
			(e = cudaMemcpyAsync(pl->blob, blob.data(), sizeof(int4) * blob.size(), cudaMemcpyHostToDevice, s)) == cudaSuccess &&
			(e = cudaMemcpyAsync(d_at, at.data(), sizeof(long long) * at.size(), cudaMemcpyHostToDevice, s)) == cudaSuccess)
		{
			pl->big = reinterpret_cast<int *>(pl->blob) + big0;
			k_group_rows<<<gs, CG_NT, 0, s>>>(ngroups, groups, outer, inner, d_of, d_cnt, d_at, reinterpret_cast<int *>(pl->blob));
			if ((e = cudaGetLastError()) == cudaSuccess) e = cudaStreamSynchronize(s);
		}
	}
	cudaFree(d_of);
	cudaFree(d_cnt);
	cudaFree(d_at);
	if (e != cudaSuccess) free_cg_plan(pl);
	return e;
}

void free_cg_plan(CgPlan *pl)
{
	void *ptrs[] = {pl->run, pl->chunk, pl->blob, pl->packets};
	for (void *p : ptrs)
		if (p) cudaFree(p);
	*pl = CgPlan();
}

cudaError_t launch_cg_start(int n, int ngroups, const int *groups, const int *outer, const int *inner,
							const double *vals, const double *b, bool guess, double tol, const double *x, const CgWork &w,
							cudaStream_t s)
{
	const int gv = grid_vec(ngroups);
	double *invd = w.dense, *q = w.dense + n;
	cudaError_t e = launch_cg_diag_inv(n, outer, inner, vals, invd, s);
	if (e != cudaSuccess) return e;
	if (guess)
		k_spmv<<<grid_spmv(ngroups), CG_NT, 0, s>>>(ngroups, groups, outer, inner, vals, x, q);
	k_cg_start<<<gv, CG_NT, 0, s>>>(ngroups, groups, invd, b, guess ? q : nullptr, x, w, w.part);
	k_cg_start_scalars<<<1, CG_NT, 0, s>>>(w.part, gv, tol, w.sc);
	return cudaGetLastError();
}

cudaError_t launch_cg_iterations(int count, CgPlan &pl, const double *vals, bool padded, const CgWork &w, cudaStream_t s,
								 int missing)
{
	const bool edge = ((size_t)vals & 15) || ((pl.nnz & 1) && !padded);
	// resident runs: the matrix's latency is gone and the exchanges are the cost
	const void *kernel = pl.resident ? (const void *)k_cg<true, true> : edge ? (const void *)k_cg<false, true> : (const void *)k_cg<false, false>;
	cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(CgSmem));
	if (e != cudaSuccess) return e;
	CgPlan p = pl;
	p.missing = missing;
	pl.gen += 3u * (unsigned)count; // at most three exchanges an iteration
	CgWork ww = w;
	void *args[] = {&p, &vals, &ww, &count};
	return cudaLaunchCooperativeKernel(kernel, dim3(pl.ctas - missing), dim3(CG_CTA), args, sizeof(CgSmem), s);
}

cudaError_t launch_cg_probe(int ctas, CgPlan &pl, const double *vals, const CgWork &w, cudaStream_t s)
{
	const cudaError_t e = cudaMemsetAsync(w.sc + CG_DONE, 0xff, sizeof(double), s); // not zero: k_cg returns at once
	return e == cudaSuccess ? launch_cg_iterations(0, pl, vals, true, w, s, pl.ctas - ctas) : e;
}

cudaError_t launch_cg_unpack(int ngroups, const int *groups, const CgWork &w, double *x, cudaStream_t s)
{
	k_cg_unpack<<<grid_vec(ngroups), CG_NT, 0, s>>>(ngroups, groups, w.x, x);
	return cudaGetLastError();
}

} // namespace pfg
