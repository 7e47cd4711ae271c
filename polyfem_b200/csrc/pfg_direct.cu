// Sparse direct solve on the device: a multifrontal Cholesky factorisation
// P A P^T = L L^T of a symmetric positive definite matrix in the assembler's CSC
// pattern, and the triangular solves.  PolyFEM's Newton step hands each assembled
// Hessian to a polysolve linear::Solver (analyzePattern, factorize, solve) inside
// the Newton solver of polysolve@47dc48d (external); the direct choices its call
// sites name are sparse LDL^T / Cholesky factorisations (Eigen::SimplicialLDLT,
// Cholmod, Pardiso: mesh/remesh/L2Projection.cpp:25-29, State.cpp:1562-1565).
// This is that family's algorithm laid out for the GPU:
//   analysis (host, once per pattern): columns with identical patterns (the dofs
//     of one node) are grouped; the group graph is ordered by nested dissection:
//     of all cuts across the groups' positions along x, y and z, where these are
//     known, and along a breadth-first order the one with the smallest vertex
//     separator, weighted by balance.  P2 24^3: 2.29 TFLOP against 3.31 with the
//     middle breadth-first level (whose surfaces bend around the start corner),
//     Q1 24^3: 37 against 134 GFLOP.  The cuts across positions find the planes of a
//     body that lies along the axes, the breadth-first ones do not depend on how it
//     lies: turned by 0.5 rad about (1, 2, 3) 2.63 TFLOP and 84 GFLOP, without them
//     8.51 and 92.  The dissection tree is the assembly
//     tree: every separator (and every leaf part) is one front whose columns are
//     eliminated together, after its two halves.  Row structures, front sizes,
//     the scatter of A's entries into the fronts and the extend-add maps are
//     precomputed.
//   factorisation (device): fronts of equal height in the tree are processed by
//     the same launches, leaves first: A's lower entries are scattered into the
//     zeroed fronts, the children's update matrices are added in child order,
//     and each front is partially factorised in pairs of 64-column panels
//     (Cholesky of each diagonal block, the triangular solve of the rows below, the
//     first panel's update of the second, then one rank-128 update of the trailing
//     lower triangle, all products on the FP64 tensor pipe); the
//     trailing block is the update matrix the parent adds.
//   solve (device): forward substitution leaves first (each front adds its
//     children's update vectors in child order), backward substitution from the
//     root, then the inverse permutation; each panel step is one launch.
// Every sum is taken in a fixed order, so factor and solution are bitwise
// deterministic.  Fronts are dense lower triangles of m (m + 1) / 2 doubles
// (packed columns), all resident for the factor's lifetime.
#include "pfg_device.cuh"
#include "pfgpu.h"

#include <algorithm>
#include <cmath>
#include <cstring>
#include <numeric>
#include <string>
#include <vector>

namespace pfg
{

namespace
{

constexpr int NBF = 64;         // panel width
constexpr int LEAF_DOFS = 96;   // dissection stops at parts of at most this many dofs
constexpr double MAX_HALF = 0.7; // largest share of a part that one side of a cut may keep
constexpr double BALANCE = 1.0;  // weight of the imbalance in a cut's cost
// A breadth-first cut has to be a tenth smaller than one across the positions, whose halves
// have planes for their next cuts.  At 1.0 P2 24^3 takes 0.6% fewer operations but a level
// more, 115.5 ms against 113; at 1.2 turned cubes of hexahedra take up to 2.6 times as many.
constexpr double BFS_COST = 1.1;
constexpr int ROWS_TILE = 64;   // rows per CTA of the panel solve and of the forward substitution

struct DevFront
{
	long long foff; // front in the front buffer (doubles): m (m + 1) / 2, packed lower columns
	long long woff; // m doubles of solve workspace
	long long roff; // rows of this front's update in the parent (relpos), m - k entries
	long long ioff; // permuted positions of the m - k rows below the front's columns
	int col0;       // first permuted column
	int k;          // columns eliminated in this front
	int m;          // k + rows below
	int child0;     // children in child_list[child0 .. child0 + nchild)
	int nchild;
	int pad;
};

// Fronts are stored as packed lower columns: column j of an order-m front holds
// rows j .. m-1, and entry (i, j), i >= j, sits at pk(m, j) + i.
__host__ __device__ __forceinline__ long long pk(int m, int j) { return (long long)j * m - (long long)j * (j + 1) / 2; }

struct Panel
{
	int lvl, j0;
	int rows_grid, upd_grid, tiles_grid; // CTAs per front: rows below, update of the second panel, trailing update
};

} // namespace

struct DirectFactor
{
	int n = 0;
	long long nnz = 0;
	int ns = 0;
	std::vector<int> perm;             // permuted position -> dof
	std::vector<DevFront> fr;          // fronts in postorder
	std::vector<int> lvl_start;        // fronts of height h: lvl_list[lvl_start[h] .. lvl_start[h+1])
	std::vector<int> lvl_list;
	std::vector<long long> lvl_fbeg;   // front doubles of each level [lvl_fbeg[h], lvl_fbeg[h+1])
	std::vector<long long> lvl_abeg;   // A-map entries of each level
	std::vector<int> lvl_maxchild, lvl_maxrc, lvl_maxk;
	std::vector<Panel> panels;         // 64-column panels, level by level, in order
	long long front_doubles = 0, work_doubles = 0, amap_n = 0;
	// host maps between the analysis and the upload
	std::vector<int> h_child, h_relpos, h_rows, h_amap_src;
	std::vector<long long> h_amap_dst;
	// device
	DevFront *d_fr = nullptr;
	int *d_lvl_list = nullptr, *d_child = nullptr, *d_relpos = nullptr, *d_rows = nullptr, *d_perm = nullptr;
	int *d_amap_src = nullptr;
	long long *d_amap_dst = nullptr;
	double *d_front = nullptr, *d_work = nullptr, *d_vec = nullptr; // d_vec: 2 n (permuted rhs, solution)
	double *d_io = nullptr;                                          // n: b and x of a host-memory solve
	int *d_err = nullptr;
	bool factorized = false;
};

// ------------------------------------------------------------------ analysis

namespace
{

struct NdBuilder
{
	// group graph
	int nv = 0;
	std::vector<int> off, adj, wt;
	std::vector<double> xyz; // vertex positions (3 per vertex), or empty
	// dissection tree (created in postorder: every node after its descendants)
	std::vector<std::vector<int>> cols;     // groups of each node
	std::vector<std::vector<int>> children;
	std::vector<int> mark, vis, lev;
	int label = 0, stamp = 0;

	int make_node(std::vector<int> g, std::vector<int> ch)
	{
		std::sort(g.begin(), g.end());
		cols.push_back(std::move(g));
		children.push_back(std::move(ch));
		return (int)cols.size() - 1;
	}

	// breadth-first levels from root over vertices marked `lab`; returns the visit
	// order and fills level starts; vis[] = stamp for visited, lev[] = level
	void bfs(int root, int lab, std::vector<int> &order, std::vector<int> &ls)
	{
		++stamp;
		order.clear();
		ls.clear();
		order.push_back(root);
		vis[root] = stamp;
		lev[root] = 0;
		ls.push_back(0);
		size_t head = 0;
		int cur = 0;
		while (head < order.size())
		{
			const int v = order[head];
			if (lev[v] != cur)
			{
				cur = lev[v];
				ls.push_back((int)head);
			}
			++head;
			for (int t = off[v]; t < off[v + 1]; ++t)
			{
				const int u = adj[t];
				if (mark[u] == lab && vis[u] != stamp)
				{
					vis[u] = stamp;
					lev[u] = lev[v] + 1;
					order.push_back(u);
				}
			}
		}
		ls.push_back((int)order.size());
	}

	int degree_in(int v, int lab) const
	{
		int d = 0;
		for (int t = off[v]; t < off[v + 1]; ++t) d += mark[adj[t]] == lab;
		return d;
	}

	// A part of the graph: its vertices sorted by x, y and z where they have positions, and in
	// the pattern's order in ord[3] (the breadth-first orders start from it, as they do for a
	// pattern without positions).
	struct Part
	{
		std::vector<int> ord[4];
	};

	// Best vertex separator over every cut of one order: the vertices of rank >= c with
	// a neighbour of rank < c (or of rank < c with one of rank >= c) separate the rest.
	// A vertex is in the first set exactly for the cuts in (least neighbour rank, rank]
	// and in the second for those in (rank, greatest neighbour rank], so one pass over
	// the edges gives the separator weight of all cuts as a running sum.
	struct Cut
	{
		double cost = 1e300;
		int axis = -1, at = 0;
		bool upper = false; // the separator's vertices have rank >= at
	};
	void try_order(const std::vector<int> &ord, int axis, int lab, Cut &best)
	{
		const int ns = (int)ord.size();
		for (int r = 0; r < ns; ++r) lev[ord[r]] = r;
		std::vector<long long> up(ns + 2, 0), lo(ns + 2, 0);
		long long total = 0;
		for (int r = 0; r < ns; ++r)
		{
			const int v = ord[r];
			int mn = r, mx = r;
			for (int t = off[v]; t < off[v + 1]; ++t)
			{
				const int u = adj[t];
				if (mark[u] != lab) continue;
				mn = std::min(mn, lev[u]);
				mx = std::max(mx, lev[u]);
			}
			up[mn + 1] += wt[v];
			up[r + 1] -= wt[v];
			lo[r + 1] += wt[v];
			lo[mx + 1] -= wt[v];
			total += wt[v];
		}
		long long below = 0, su = 0, sl = 0;
		for (int c = 1; c < ns; ++c)
		{
			below += wt[ord[c - 1]];
			su += up[c];
			sl += lo[c];
			for (int k = 0; k < 2; ++k)
			{
				const long long sep = k ? su : sl;
				const long long a = k ? below : below - sep, b = total - a - sep;
				if (a <= 0 || b <= 0) continue;
				// the separator's front is eliminated in sep^3 operations; an unbalanced cut
				// leaves a larger half to dissect
				const double big = (double)std::max(a, b) / (double)(a + b); // 0.5 .. 1
				if (big > MAX_HALF) continue;
				const double cost = (double)sep * (1.0 + BALANCE * (big - 0.5)) * (axis == 3 ? BFS_COST : 1.0);
				if (cost < best.cost) best = {cost, axis, c, k != 0};
			}
		}
	}

	// nested dissection of a part; returns the roots of its subtrees
	std::vector<int> build(Part P)
	{
		std::vector<int> roots;
		const std::vector<int> &S = P.ord[3];
		if (S.empty()) return roots;
		const int first = xyz.empty() ? 3 : 0; // the first order that the part has
		const int lab = ++label;
		for (int v : S) mark[v] = lab;
		std::vector<int> order, ls;
		bfs(S[0], lab, order, ls);
		if (order.size() < S.size())
		{
			// disconnected: every component is its own subtree
			std::vector<Part> parts;
			for (int v : S)
				if (mark[v] == lab)
				{
					bfs(v, lab, order, ls);
					for (int u : order)
					{
						mark[u] = -1;
						lev[u] = (int)parts.size();
					}
					parts.emplace_back();
				}
			for (int d = first; d < 4; ++d)
				for (int v : P.ord[d]) parts[lev[v]].ord[d].push_back(v);
			P = Part();
			for (auto &c : parts)
			{
				std::vector<int> r = build(std::move(c));
				roots.insert(roots.end(), r.begin(), r.end());
			}
			return roots;
		}
		long long w = 0;
		for (int v : S) w += wt[v];
		if (w <= LEAF_DOFS)
		{
			roots.push_back(make_node(S, {}));
			return roots;
		}
		Cut best;
		std::vector<int> level_order;
		for (int d = first; d < 3; ++d) try_order(P.ord[d], d, lab, best);
		// the breadth-first order from a pseudo-peripheral vertex, restarting from a
		// minimum-degree vertex of the last level while the eccentricity grows
		int h = (int)ls.size() - 1;
		for (int it = 0; it < 4; ++it)
		{
			int bv = -1, bd = 1 << 30;
			for (int q = ls[h - 1]; q < ls[h]; ++q)
			{
				const int d = degree_in(order[q], lab);
				if (d < bd) bd = d, bv = order[q];
			}
			std::vector<int> o2, l2;
			bfs(bv, lab, o2, l2);
			const int h2 = (int)l2.size() - 1;
			if (h2 <= h) break;
			h = h2;
			order.swap(o2);
			ls.swap(l2);
		}
		level_order = order;
		try_order(level_order, 3, lab, best);
		if (best.axis < 0)
		{
			roots.push_back(make_node(S, {}));
			return roots;
		}
		// sides: 0 below the cut, 1 above it, 2 separator
		const std::vector<int> &ord = best.axis == 3 ? level_order : P.ord[best.axis];
		for (int q = 0; q < (int)ord.size(); ++q) lev[ord[q]] = q;
		std::vector<int> Sep;
		std::vector<char> side(ord.size());
		for (int q = 0; q < (int)ord.size(); ++q)
		{
			const int v = ord[q];
			char sd = q >= best.at;
			if ((q >= best.at) == best.upper)
				for (int t = off[v]; t < off[v + 1]; ++t)
				{
					const int u = adj[t];
					if (mark[u] == lab && (lev[u] >= best.at) != best.upper)
					{
						sd = 2;
						break;
					}
				}
			side[q] = sd;
			if (sd == 2) Sep.push_back(v);
		}
		Part A, B;
		for (int d = first; d < 4; ++d)
			for (int v : P.ord[d])
			{
				const char sd = side[lev[v]];
				if (sd == 0) A.ord[d].push_back(v);
				else if (sd == 1) B.ord[d].push_back(v);
			}
		P = Part();
		std::vector<int> ch = build(std::move(A));
		std::vector<int> cb = build(std::move(B));
		ch.insert(ch.end(), cb.begin(), cb.end());
		roots.push_back(make_node(std::move(Sep), std::move(ch)));
		return roots;
	}
};

template <class T>
static cudaError_t upload(T **d, const std::vector<T> &h)
{
	*d = nullptr;
	const size_t bytes = sizeof(T) * std::max<size_t>(h.size(), 1);
	cudaError_t e = cudaMalloc(reinterpret_cast<void **>(d), bytes);
	if (e != cudaSuccess) return e;
	if (!h.empty()) e = cudaMemcpy(*d, h.data(), sizeof(T) * h.size(), cudaMemcpyHostToDevice);
	return e;
}

} // namespace

void direct_destroy(DirectFactor *f)
{
	if (!f) return;
	void *ptrs[] = {f->d_fr,       f->d_lvl_list, f->d_child, f->d_relpos, f->d_rows, f->d_perm, f->d_amap_src,
					f->d_amap_dst, f->d_front,    f->d_work,  f->d_vec,    f->d_io,   f->d_err};
	for (void *p : ptrs)
		if (p) cudaFree(p); // a host-only analysis never touches the runtime
	delete f;
}

int direct_n(const DirectFactor *f) { return f ? f->n : 0; }
long long direct_nnz(const DirectFactor *f) { return f ? f->nnz : 0; }
long long direct_front_bytes(const DirectFactor *f) { return f ? f->front_doubles * 8 : 0; }
int direct_fronts(const DirectFactor *f) { return f ? f->ns : 0; }
bool direct_factorized(const DirectFactor *f) { return f && f->factorized; }
double *direct_io(DirectFactor *f) { return f ? f->d_io : nullptr; }

// Host analysis of a pattern (full symmetric CSC, sorted rows, n > 0 columns;
// node_pos: a position of every column, 3 n doubles, or NULL, used for the ordering only):
// ordering, fronts and every index map, each checked against the front it
// addresses before anything reaches the device.  0 ok, else a PFG error code
// with msg; *out owns the host arrays (and the maps until direct_upload).
int direct_symbolic(int n, const int *outer, const int *inner, const double *node_pos, DirectFactor **out, std::string &msg)
{
	*out = nullptr;
	auto *f = new DirectFactor();
	f->n = n;
	f->nnz = n > 0 ? outer[n] : 0;
	// 1. groups of consecutive columns with identical patterns
	std::vector<int> gof(n), gfirst;
	for (int j = 0; j < n; ++j)
	{
		bool same = false;
		if (j > 0)
		{
			const int a0 = outer[j - 1], a1 = outer[j], b0 = outer[j], b1 = outer[j + 1];
			same = (a1 - a0) == (b1 - b0) && std::equal(inner + a0, inner + a1, inner + b0);
		}
		if (same) gof[j] = gof[j - 1];
		else
		{
			gof[j] = (int)gfirst.size();
			gfirst.push_back(j);
		}
	}
	const int ng = (int)gfirst.size();
	gfirst.push_back(n);
	NdBuilder nd;
	nd.nv = ng;
	nd.off.assign(ng + 1, 0);
	nd.wt.assign(ng, 0);
	for (int g = 0; g < ng; ++g)
	{
		nd.wt[g] = gfirst[g + 1] - gfirst[g];
		const int j = gfirst[g];
		int last = -1;
		for (int t = outer[j]; t < outer[j + 1]; ++t)
		{
			const int h = gof[inner[t]];
			if (h != g && h != last) nd.adj.push_back(h);
			last = h;
		}
		nd.off[g + 1] = (int)nd.adj.size();
	}
	nd.mark.assign(ng, 0);
	nd.vis.assign(ng, 0);
	nd.lev.assign(ng, 0);
	NdBuilder::Part all;
	all.ord[3].resize(ng);
	std::iota(all.ord[3].begin(), all.ord[3].end(), 0);
	if (node_pos)
	{
		nd.xyz.resize(3 * (size_t)ng);
		for (int g = 0; g < ng; ++g)
			for (int d = 0; d < 3; ++d)
			{
				const double x = node_pos[3 * (size_t)gfirst[g] + d];
				nd.xyz[3 * (size_t)g + d] = std::isfinite(x) ? x : 0.0;
			}
		for (int d = 0; d < 3; ++d)
		{
			all.ord[d] = all.ord[3];
			const double *x = nd.xyz.data() + d;
			std::stable_sort(all.ord[d].begin(), all.ord[d].end(), [&](int a, int b) { return x[3 * (size_t)a] < x[3 * (size_t)b]; });
		}
	}
	nd.build(std::move(all));
	const int ns = (int)nd.cols.size();
	f->ns = ns;
	// 2. permutation: columns in node (postorder) order
	std::vector<int> parent(ns, -1), col0(ns), kc(ns);
	for (int s = 0; s < ns; ++s)
		for (int c : nd.children[s]) parent[c] = s;
	f->perm.resize(n);
	std::vector<int> iperm(n);
	int pos = 0;
	for (int s = 0; s < ns; ++s)
	{
		col0[s] = pos;
		for (int g : nd.cols[s])
			for (int j = gfirst[g]; j < gfirst[g + 1]; ++j)
			{
				f->perm[pos] = j;
				iperm[j] = pos++;
			}
		kc[s] = pos - col0[s];
	}
	if (pos != n)
	{
		msg = "direct solver analysis lost columns";
		direct_destroy(f);
		return PFG_ERR_STATE;
	}
	// 3. row structures below each front's columns
	std::vector<std::vector<int>> rows(ns);
	for (int s = 0; s < ns; ++s)
	{
		const int last = col0[s] + kc[s] - 1;
		std::vector<int> R;
		for (int q = col0[s]; q <= last; ++q)
		{
			const int j = f->perm[q];
			if (j > 0 && gof[j] == gof[j - 1]) continue; // the group's columns have the same rows
			for (int t = outer[j]; t < outer[j + 1]; ++t)
			{
				const int p = iperm[inner[t]];
				if (p > last) R.push_back(p);
			}
		}
		for (int c : nd.children[s])
			for (int p : rows[c])
				if (p > last) R.push_back(p);
		std::sort(R.begin(), R.end());
		R.erase(std::unique(R.begin(), R.end()), R.end());
		rows[s] = std::move(R);
	}
	// 4. heights and levels
	std::vector<int> height(ns, 0);
	int maxh = 0;
	for (int s = 0; s < ns; ++s)
	{
		for (int c : nd.children[s]) height[s] = std::max(height[s], height[c] + 1);
		maxh = std::max(maxh, height[s]);
	}
	const int nl = ns > 0 ? maxh + 1 : 0;
	f->lvl_start.assign(nl + 1, 0);
	for (int s = 0; s < ns; ++s) f->lvl_start[height[s] + 1]++;
	for (int h = 0; h < nl; ++h) f->lvl_start[h + 1] += f->lvl_start[h];
	f->lvl_list.resize(ns);
	{
		std::vector<int> fill(f->lvl_start.begin(), f->lvl_start.end() - 1);
		for (int s = 0; s < ns; ++s) f->lvl_list[fill[height[s]]++] = s;
	}
	// 5. fronts (allocated level by level), maps
	f->fr.resize(ns);
	std::vector<int> child_list, relpos, rowsflat;
	f->lvl_fbeg.assign(nl + 1, 0);
	f->lvl_abeg.assign(nl + 1, 0);
	f->lvl_maxchild.assign(nl, 0);
	f->lvl_maxrc.assign(nl, 0);
	long long fo = 0, wo = 0;
	std::vector<int> amap_src;
	std::vector<long long> amap_dst;
	// local index of a permuted position in the front at hand, where[p] valid if of[p] is that front
	std::vector<int> where(n, 0), of(n, -1);
	auto local = [&](int s, int p) -> int { return of[p] == s ? where[p] : -1; };
	bool broken = false;
	for (int s = 0; s < ns; ++s)
	{
		DevFront &d = f->fr[s];
		d.col0 = col0[s];
		d.k = kc[s];
		d.m = kc[s] + (int)rows[s].size();
		d.child0 = (int)child_list.size();
		d.nchild = (int)nd.children[s].size();
		d.pad = 0;
		for (int c : nd.children[s]) child_list.push_back(c);
		d.ioff = (long long)rowsflat.size();
		rowsflat.insert(rowsflat.end(), rows[s].begin(), rows[s].end());
		d.woff = wo;
		wo += d.m;
	}
	{
		long long ro = 0;
		for (int s = 0; s < ns; ++s)
		{
			f->fr[s].roff = ro;
			if (parent[s] >= 0) ro += (long long)rows[s].size();
			else broken |= !rows[s].empty();
		}
		relpos.resize((size_t)ro);
	}
	for (int h = 0; h < nl; ++h)
	{
		f->lvl_fbeg[h] = fo;
		f->lvl_abeg[h] = (long long)amap_src.size();
		for (int t = f->lvl_start[h]; t < f->lvl_start[h + 1]; ++t)
		{
			const int s = f->lvl_list[t];
			DevFront &d = f->fr[s];
			d.foff = fo;
			fo += (long long)d.m * (d.m + 1) / 2;
			f->lvl_maxchild[h] = std::max(f->lvl_maxchild[h], d.nchild);
			for (int q = 0; q < d.m; ++q)
			{
				const int p = q < d.k ? d.col0 + q : rows[s][q - d.k];
				where[p] = q;
				of[p] = s;
			}
			for (int c : nd.children[s])
			{
				f->lvl_maxrc[h] = std::max(f->lvl_maxrc[h], f->fr[c].m - f->fr[c].k);
				int prev = -1;
				for (size_t q = 0; q < rows[c].size(); ++q)
				{
					const int l = local(s, rows[c][q]);
					broken |= l <= prev; // present in the parent, increasing
					relpos[f->fr[c].roff + q] = l;
					prev = l;
				}
			}
			for (int q = d.col0; q < d.col0 + d.k; ++q)
			{
				const int j = f->perm[q], cl = q - d.col0;
				for (int t2 = outer[j]; t2 < outer[j + 1]; ++t2)
				{
					const int p = iperm[inner[t2]];
					if (p < q) continue; // the upper entry of the pair
					const int lr = local(s, p);
					broken |= lr < cl || lr >= d.m; // lower triangle of this front
					amap_src.push_back(t2);
					amap_dst.push_back(d.foff + pk(d.m, cl) + lr);
				}
			}
		}
	}
	f->lvl_fbeg[nl] = fo;
	f->lvl_abeg[nl] = (long long)amap_src.size();
	f->front_doubles = fo;
	f->work_doubles = wo;
	f->amap_n = (long long)amap_src.size();
	// 6. panel launches of the factorisation and the solve
	for (int h = 0; h < nl; ++h)
	{
		int maxk = 0;
		for (int t = f->lvl_start[h]; t < f->lvl_start[h + 1]; ++t) maxk = std::max(maxk, f->fr[f->lvl_list[t]].k);
		f->lvl_maxk.push_back(maxk);
		for (int j0 = 0; j0 < maxk; j0 += NBF)
		{
			// rows of 64 below the panel; of a pair's first panel: rows of 64 of its update
			// of the second panel (0 when no front has one), tiles of the rank-128 update
			long long rows = 0, upd = 0, tiles = 0;
			for (int t = f->lvl_start[h]; t < f->lvl_start[h + 1]; ++t)
			{
				const DevFront &d = f->fr[f->lvl_list[t]];
				if (d.k <= j0) continue;
				const int nb = std::min(NBF, d.k - j0), nb2 = std::min(2 * NBF, d.k - j0);
				rows = std::max(rows, ((long long)d.m - j0 - nb + ROWS_TILE - 1) / ROWS_TILE);
				if (d.k > j0 + NBF) upd = std::max(upd, ((long long)d.m - j0 - NBF + ROWS_TILE - 1) / ROWS_TILE);
				const long long n64 = (d.m - j0 - nb2 + 63) / 64, hh = n64 / 2;
				tiles = std::max(tiles, n64 % 2 ? (hh + 1) * (hh + 1) : hh * (hh + 1));
			}
			if (tiles > 0x3fffffffLL)
			{
				msg = "direct solver front too large";
				direct_destroy(f);
				return PFG_ERR_UNSUPPORTED;
			}
			f->panels.push_back({h, j0, (int)rows, (int)upd, (int)tiles});
		}
	}
	for (int h = 0; h < nl; ++h)
		if (f->lvl_start[h + 1] - f->lvl_start[h] > 65535)
		{
			msg = "direct solver: more than 65535 fronts of one height";
			direct_destroy(f);
			return PFG_ERR_UNSUPPORTED;
		}
	for (int s2 = 0; s2 < ns && !broken; ++s2)
	{
		const DevFront &d = f->fr[s2];
		broken |= d.k < 1 || d.m < d.k || d.foff < 0 || d.foff + (long long)d.m * (d.m + 1) / 2 > fo;
		const int last = d.col0 + d.k - 1;
		for (int q = 0; q < d.m - d.k && !broken; ++q)
		{
			const int p = rowsflat[d.ioff + q];
			broken |= p <= last || p >= n || (q > 0 && p <= rowsflat[d.ioff + q - 1]);
		}
	}
	if (broken)
	{
		msg = "direct solver analysis produced an inconsistent front structure";
		direct_destroy(f);
		return PFG_ERR_STATE;
	}
	f->h_child = std::move(child_list);
	f->h_relpos = std::move(relpos);
	f->h_rows = std::move(rowsflat);
	f->h_amap_src = std::move(amap_src);
	f->h_amap_dst = std::move(amap_dst);
	*out = f;
	return PFG_OK;
}

// the analysed maps to the device (the host copies are released); 0 ok, else a
// PFG error code with msg (f is left for direct_destroy)
int direct_upload(DirectFactor *f, std::string &msg)
{
	const int n = f->n;
	const long long fo = f->front_doubles, wo = f->work_doubles;
	// the fronts must fit beside what is already allocated
	size_t fre = 0, tot = 0;
	cudaError_t e = cudaMemGetInfo(&fre, &tot);
	if (e != cudaSuccess)
	{
		msg = cudaGetErrorString(e);
		return PFG_ERR_CUDA;
	}
	const double need = 8.0 * (double)fo + 8.0 * (double)wo + 12.0 * (double)f->amap_n + 24.0 * n;
	if (need > 0.85 * (double)fre)
	{
		msg = "direct solver needs " + std::to_string((long long)(need / 1e6)) + " MB of device memory for its fronts, " +
			  std::to_string((long long)(fre / 1000000)) + " MB free";
		return PFG_ERR_OOM;
	}
	if ((e = upload(&f->d_fr, f->fr)) != cudaSuccess || (e = upload(&f->d_lvl_list, f->lvl_list)) != cudaSuccess ||
		(e = upload(&f->d_child, f->h_child)) != cudaSuccess || (e = upload(&f->d_relpos, f->h_relpos)) != cudaSuccess ||
		(e = upload(&f->d_rows, f->h_rows)) != cudaSuccess || (e = upload(&f->d_perm, f->perm)) != cudaSuccess ||
		(e = upload(&f->d_amap_src, f->h_amap_src)) != cudaSuccess ||
		(e = upload(&f->d_amap_dst, f->h_amap_dst)) != cudaSuccess ||
		(e = cudaMalloc(&f->d_front, 8 * std::max<long long>(fo, 1))) != cudaSuccess ||
		(e = cudaMalloc(&f->d_work, 8 * std::max<long long>(wo, 1))) != cudaSuccess ||
		(e = cudaMalloc(&f->d_vec, 16 * (size_t)std::max(n, 1))) != cudaSuccess ||
		(e = cudaMalloc(&f->d_io, 8 * (size_t)std::max(n, 1))) != cudaSuccess ||
		(e = cudaMalloc(&f->d_err, sizeof(int))) != cudaSuccess)
	{
		msg = cudaGetErrorString(e);
		return e == cudaErrorMemoryAllocation ? PFG_ERR_OOM : PFG_ERR_CUDA;
	}
	f->h_child = {};
	f->h_relpos = {};
	f->h_rows = {};
	f->h_amap_src = {};
	f->h_amap_dst = {};
	return PFG_OK;
}

void direct_stats(const DirectFactor *f, long long *st)
{
	// [n, fronts, levels, front doubles, nnz of L (columns of the fronts), largest
	// front, flops of the factorisation: column j of a front of order m updates the
	// (m-j-1)(m-j)/2 entries of its trailing lower triangle, one multiply-add each]
	long long nnzl = 0, mx = 0;
	double fl = 0.0;
	auto s2 = [](double t) { return t * (t + 1.0) * (2.0 * t + 1.0) / 6.0; }; // sum of squares 1..t
	auto s1 = [](double t) { return t * (t + 1.0) / 2.0; };
	for (const DevFront &d : f->fr)
	{
		nnzl += (long long)d.k * (d.k + 1) / 2 + (long long)d.k * (d.m - d.k);
		mx = std::max<long long>(mx, d.m);
		// sum over t = m-k .. m-1 of t (t + 1)
		const double hi = d.m - 1.0, lo = d.m - d.k - 1.0;
		fl += (s2(hi) - s2(lo)) + (s1(hi) - s1(lo));
	}
	st[6] = (long long)fl;
	st[0] = f->n;
	st[1] = f->ns;
	st[2] = (long long)f->lvl_start.size() - 1;
	st[3] = f->front_doubles;
	st[4] = nnzl;
	st[5] = mx;
}

// ------------------------------------------------------------------ kernels

namespace
{

__global__ void k_dir_assemble(long long n, const int *__restrict__ src, const long long *__restrict__ dst,
							   const double *__restrict__ vals, double *__restrict__ F)
{
	const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
	if (t < n) F[dst[t]] = vals[src[t]];
}

// child ci of every front of the level: F_s[relpos a, relpos b] += U_c[a, b] (a >= b);
// warp w of CTA x takes column b = 8 x + w of the child's update
__global__ void __launch_bounds__(256) k_dir_extend_add(const DevFront *__restrict__ fr, const int *__restrict__ list,
														const int *__restrict__ child, const int *__restrict__ relpos,
														double *__restrict__ F, int ci)
{
	const DevFront f = fr[list[blockIdx.y]];
	if (ci >= f.nchild) return;
	const DevFront c = fr[child[f.child0 + ci]];
	const int rc = c.m - c.k;
	const int b = blockIdx.x * 8 + (threadIdx.x >> 5), lane = threadIdx.x & 31;
	if (b >= rc) return;
	const int *rp = relpos + c.roff;
	const double *U = F + c.foff + pk(c.m, c.k + b) + c.k; // U[a] = entry (k + a, k + b), a >= b
	double *P = F + f.foff + pk(f.m, rp[b]);
	for (int a = b + lane; a < rc; a += 32) P[rp[a]] += U[a];
}

__device__ __forceinline__ void cp_async8(double *dst, const double *src, bool ok)
{
	const unsigned d = (unsigned)__cvta_generic_to_shared(dst);
	const int bytes = ok ? 8 : 0; // 0: the 8 bytes are zero-filled and src is not read
	asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;" ::"r"(d), "l"(src), "r"(bytes) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }

// c (16 x 8) += a (16 x 4) b (4 x 8) on the FP64 tensor pipe: lane t holds a[t / 4 (+ 8)][t % 4],
// b[t % 4][t / 4] and c[t / 4 (+ 8)][2 (t % 4) + {0, 1}]
__device__ __forceinline__ void dmma(double (&c0)[2], double (&c1)[2], double a0, double a1, double b)
{
	asm("mma.sync.aligned.m16n8k4.row.col.f64.f64.f64.f64 {%0,%1,%2,%3},{%4,%5},{%6},{%0,%1,%2,%3};"
		: "+d"(c0[0]), "+d"(c0[1]), "+d"(c1[0]), "+d"(c1[1])
		: "d"(a0), "d"(a1), "d"(b));
}

// the same with k = 8: a0..a3 are a[t / 4 (+ 8 for odd)][t % 4 (+ 4 from a2 on)], b0, b1 are b[t % 4 (+ 4)][t / 4]
__device__ __forceinline__ void dmma_k8(double (&c0)[2], double (&c1)[2], const double (&a)[4], double b0, double b1)
{
	asm("mma.sync.aligned.m16n8k8.row.col.f64.f64.f64.f64 {%0,%1,%2,%3},{%4,%5,%6,%7},{%8,%9},{%0,%1,%2,%3};"
		: "+d"(c0[0]), "+d"(c0[1]), "+d"(c1[0]), "+d"(c1[1])
		: "d"(a[0]), "d"(a[1]), "d"(a[2]), "d"(a[3]), "d"(b0), "d"(b1));
}
// an 8 x 8 tile, c += a (8 x 4) b (4 x 8)
__device__ __forceinline__ void dmma_8x8(double (&c)[2], double a, double b)
{
	asm("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0,%1},{%2},{%3},{%0,%1};" : "+d"(c[0]), "+d"(c[1]) : "d"(a), "d"(b));
}

// 1 / d of a positive finite d: rcp_nr where its flush-to-zero range is safe, else the division
__device__ __forceinline__ double pivot_rcp(double d)
{
	if (!(d > 1e-290 && d < 1e290)) return 1.0 / d;
	return rcp_nr(d);
}

// The factorisation runs in panels of 64 columns, two at a time:
//   k_dir_diag: Cholesky of the 64 x 64 diagonal block;
//   k_dir_solve_rows: the rows below, X L_d^T = B;
//   k_dir_rows: the first panel's update of the second panel's columns;
//   (the first two kernels for the second panel;)
//   k_dir_update: the rank-128 update of the trailing lower triangle, so the
//     trailing matrix is read and written once per 128 columns.
//
// The diagonal of L is stored as its reciprocal, which is all that its readers need.
// Triangles are solved by substitution, not multiplied by their inverse: the inverse's error
// is that of the block's condition (a 24-dof Gaussian Gram matrix: normwise backward error
// 1e-12 against 2e-16; P2 with lambda / mu 1e8: 8e-16 against 1e-16).
//
// k_dir_diag, one CTA per front, the block in shared memory.  One warp factorises eight
// columns (two rows per lane, pivots and multipliers by shuffle), then all warps apply
// them to the rest in 8 x 8 tiles on the FP64 tensor pipe.  Bound by the 64 dependent
// pivot steps.  One barrier and one rank-1 update of all entries per column took 28 us a
// block at P2 24^3 (two one-warp 32-column blocks with a substitution each: 60 us); this
// takes 16.
constexpr int DIAG_LD = NBF + 4; // 4 mod 16: a fragment's rows fall on distinct banks
constexpr int DIAG_SLD = 12;     // the same for the eight scaled panel columns
constexpr size_t DIAG_SMEM = (NBF * DIAG_LD + NBF * DIAG_SLD + NBF) * sizeof(double);
__global__ void __launch_bounds__(256) k_dir_diag(const DevFront *__restrict__ fr, const int *__restrict__ list,
												  double *__restrict__ F, int j0, int *__restrict__ err)
{
	constexpr unsigned FULL = 0xffffffffu;
	const DevFront f = fr[list[blockIdx.x]];
	if (j0 >= f.k) return;
	const int nb = min(NBF, f.k - j0), tid = threadIdx.x, r = tid % NBF, g = tid / NBF;
	const int lane = tid & 31, warp = tid >> 5, fk = lane & 3, fr_ = lane >> 2;
	double *Fb = F + f.foff + pk(f.m, j0) + j0; // entry (j0 + i, j0 + l) at l (m - j0) - l (l + 1) / 2 + i
	const int ld = f.m - j0;
	extern __shared__ __align__(16) double dsm[];
	double(*M)[DIAG_LD] = reinterpret_cast<double(*)[DIAG_LD]>(dsm);                  // the block, by rows
	double(*S)[DIAG_SLD] = reinterpret_cast<double(*)[DIAG_SLD]>(dsm + NBF * DIAG_LD); // panel columns over their pivots
	double *rs = dsm + NBF * DIAG_LD + NBF * DIAG_SLD;                                 // pivots, then 1 / l_cc
#pragma unroll
	for (int i = 0; i < 16; ++i)
	{
		const int l = 4 * i + g;
		// rows past the block's end continue it as the identity
		M[r][l] = r < nb && l <= r ? Fb[l * ld - l * (l + 1) / 2 + r] : (r == l ? 1.0 : 0.0);
	}
	__syncthreads();
#pragma unroll 1
	for (int cb = 0; cb < 8; ++cb)
	{
		const int c0 = 8 * cb;
		if (warp == 0)
		{
			double p[2][8], s[2][8];
#pragma unroll
			for (int q = 0; q < 8; ++q)
			{
				p[0][q] = M[lane][c0 + q];
				p[1][q] = M[lane + 32][c0 + q];
			}
			bool bad = false;
			const bool up = c0 >= 32; // the panel's diagonal rows sit in the upper half of the lanes' rows
#pragma unroll
			for (int q = 0; q < 8; ++q)
			{
				const double x = up ? p[1][q] : p[0][q];
				double d = __shfl_sync(FULL, x, (c0 + q) & 31);
				if (!(d > 0.0) || !(d <= 1.7976931348623157e308))
				{
					bad = true;
					d = 1.0;
				}
				if (lane == 0) rs[c0 + q] = d;
				const double rd = pivot_rcp(d);
				s[0][q] = p[0][q] * rd;
				s[1][q] = p[1][q] * rd;
#pragma unroll
				for (int l = q + 1; l < 8; ++l)
				{
					const double y = __shfl_sync(FULL, x, (c0 + l) & 31);
					p[0][l] = fma(-s[0][q], y, p[0][l]);
					p[1][l] = fma(-s[1][q], y, p[1][l]);
				}
			}
#pragma unroll
			for (int q = 0; q < 8; ++q)
			{
				M[lane][c0 + q] = p[0][q];
				M[lane + 32][c0 + q] = p[1][q];
				S[lane][q] = s[0][q];
				S[lane + 32][q] = s[1][q];
			}
			if (bad && lane == 0) atomicExch(err, 1);
		}
		__syncthreads();
		// M -= S (panel)^T over the 8 x 8 tiles (i, j), cb < j <= i < 8
		const int nt = 7 - cb;
		for (int x = warp; x < nt * (nt + 1) / 2; x += 8)
		{
			int i = 0, j = x;
			while (j > i) j -= ++i;
			i = 8 * (cb + 1 + i);
			j = 8 * (cb + 1 + j);
			double2 *C = reinterpret_cast<double2 *>(&M[i + fr_][j + 2 * fk]);
			const double2 v = *C;
			double c[2] = {v.x, v.y};
			dmma_8x8(c, -S[i + fr_][fk], M[j + fr_][c0 + fk]);
			dmma_8x8(c, -S[i + fr_][4 + fk], M[j + fr_][c0 + 4 + fk]);
			*C = make_double2(c[0], c[1]);
		}
		__syncthreads();
	}
	if (tid < NBF) rs[tid] = 1.0 / sqrt(rs[tid]);
	__syncthreads();
#pragma unroll 4
	for (int i = 0; i < 16; ++i)
	{
		const int l = 4 * i + g;
		if (r < nb && l <= r) Fb[l * ld - l * (l + 1) / 2 + r] = r == l ? rs[l] : M[r][l] * rs[l];
	}
}

// X L_d^T = B in place for 64 rows below the panel per CTA, L_d the panel's triangle.  A warp
// takes 16 rows through the eight 8-column blocks: its values of the block go to shared
// memory, a lane per row substitutes the eight columns (scaled by reciprocals of the
// diagonal), and the solved columns update the later blocks, held as accumulator fragments,
// on the FP64 tensor pipe.  Bound by that chain of eight steps: 18 us a panel on average at
// P2 24^3, 16 for the product with the block's inverse that this replaced (and 21 us then for
// its diagonal block).
constexpr int ROWS_LD = NBF + 4; // 4 mod 16: the four k rows of a fragment fall on distinct banks
constexpr size_t ROWS_SMEM = 2 * NBF * ROWS_LD * sizeof(double);
__global__ void __launch_bounds__(128, 3) k_dir_solve_rows(const DevFront *__restrict__ fr, const int *__restrict__ list,
														   double *__restrict__ F, int j0)
{
	const DevFront f = fr[list[blockIdx.y]];
	if (f.k <= j0) return;
	const int nb = min(NBF, f.k - j0), o = j0 + nb, i0 = blockIdx.x * ROWS_TILE, t = f.m - o;
	if (i0 >= t) return;
	double *P = F + f.foff + pk(f.m, j0) + o; // column l of the panel from row o on: P + l ld - l (l + 1) / 2
	const int ld = f.m - j0;
	extern __shared__ __align__(16) double dsm[];
	double(*A)[ROWS_LD] = reinterpret_cast<double(*)[ROWS_LD]>(dsm);                 // [column][row] of B, then of X
	double(*D)[ROWS_LD] = reinterpret_cast<double(*)[ROWS_LD]>(dsm + NBF * ROWS_LD); // [column][row] of L_d, zeros past the panel
	const int tid = threadIdx.x, r = tid % NBF, l1 = tid / NBF;
	const bool ra = i0 + r < t;
	{
		int off = l1 * ld - l1; // l1 is 0 or 1
		int step = 2 * ld - 2 * l1 - 3;
#pragma unroll 8
		for (int q = 0; q < NBF / 2; ++q)
		{
			const int l = l1 + 2 * q;
			const bool oa = l < nb && ra, ob = l < nb && r >= l && r < nb;
			cp_async8(&A[l][r], P + (oa ? off + i0 + r : 0), oa);
			cp_async8(&D[l][r], P + (ob ? off + r - nb : 0), ob);
			off += step;
			step -= 4;
		}
	}
	cp_async_commit();
	cp_async_wait<0>();
	__syncthreads();
	const int lane = tid & 31, wr = (tid >> 5) * 16, fk = lane & 3, fr_ = lane >> 2, row = wr + (lane & 15);
	double acc[8][2][2];
#pragma unroll
	for (int j = 0; j < 8; ++j)
#pragma unroll
		for (int h = 0; h < 2; ++h)
#pragma unroll
			for (int e = 0; e < 2; ++e) acc[j][h][e] = A[8 * j + 2 * fk + e][wr + fr_ + 8 * h];
	__syncwarp();
#pragma unroll
	for (int j = 0; j < 8; ++j)
	{
		if (j > 0)
		{
#pragma unroll
			for (int h = 0; h < 2; ++h)
#pragma unroll
				for (int e = 0; e < 2; ++e) A[8 * j + 2 * fk + e][wr + fr_ + 8 * h] = acc[j][h][e];
			__syncwarp();
		}
		double x[8];
#pragma unroll
		for (int c = 0; c < 8; ++c) x[c] = A[8 * j + c][row];
#pragma unroll
		for (int c = 0; c < 8; ++c)
		{
			x[c] *= D[8 * j + c][8 * j + c];
#pragma unroll
			for (int l = c + 1; l < 8; ++l) x[l] = fma(-D[8 * j + c][8 * j + l], x[c], x[l]);
		}
		__syncwarp();
		if (lane < 16)
#pragma unroll
			for (int c = 0; c < 8; ++c) A[8 * j + c][row] = x[c];
		__syncwarp();
		if (j == 7) break;
		const double a[4] = {-A[8 * j + fk][wr + fr_], -A[8 * j + fk][wr + fr_ + 8], -A[8 * j + 4 + fk][wr + fr_],
							 -A[8 * j + 4 + fk][wr + fr_ + 8]};
#pragma unroll
		for (int n = j + 1; n < 8; ++n)
			dmma_k8(acc[n][0], acc[n][1], a, D[8 * j + fk][8 * n + fr_], D[8 * j + 4 + fk][8 * n + fr_]);
	}
	__syncthreads();
	if (ra)
	{
		int off = l1 * ld - l1 + i0 + r, step = 2 * ld - 2 * l1 - 3;
#pragma unroll 8
		for (int l = l1; l < NBF; l += 2)
		{
			if (l < nb) P[off] = A[l][r];
			off += step;
			step -= 4;
		}
	}
}

// The first panel's update of the second panel's columns, C -= P Q^T with Q the rows of P that
// belong to those columns (rows and columns from j0 + 64 on), 64 rows per CTA on the FP64
// tensor pipe, K = 64 staged at once.
// Bound by latency: one wave of CTAs that load, multiply and store once.  A thread-per-row
// update took 22 us for 32 columns at P2 24^3; this takes 8 us for 64 on the last front
// (7,056 rows).
__global__ void __launch_bounds__(128, 3) k_dir_rows(const DevFront *__restrict__ fr, const int *__restrict__ list,
													 double *__restrict__ F, int j0)
{
	const DevFront f = fr[list[blockIdx.y]];
	if (f.k <= j0 + NBF) return;
	const int o = j0 + NBF, i0 = blockIdx.x * ROWS_TILE, t = f.m - o;
	if (i0 >= t) return;
	// column l of the panel from row o on: P + l ld - l (l + 1) / 2
	const double *P = F + f.foff + pk(f.m, j0) + o;
	const int ld = f.m - j0;
	const int nc = min(NBF, f.k - o); // columns of the result
	extern __shared__ __align__(16) double dsm[];
	double(*A)[ROWS_LD] = reinterpret_cast<double(*)[ROWS_LD]>(dsm);
	double(*B)[ROWS_LD] = reinterpret_cast<double(*)[ROWS_LD]>(dsm + NBF * ROWS_LD);
	const int tid = threadIdx.x, r = tid % NBF, l1 = tid / NBF;
	{
		int off = l1 * ld - l1; // l1 is 0 or 1
		int step = 2 * ld - 2 * l1 - 3;
		const bool ra = i0 + r < t;
#pragma unroll 8
		for (int q = 0; q < NBF / 2; ++q)
		{
			const int l = l1 + 2 * q;
			cp_async8(&A[l][r], P + (ra ? off + i0 + r : 0), ra);
			cp_async8(&B[l][r], P + (r < nc ? off + r : 0), r < nc);
			off += step;
			step -= 4;
		}
	}
	cp_async_commit();
	const int lane = tid & 31, warp = tid >> 5, wr = (warp & 1) * 32, wc = (warp >> 1) * 32;
	const int fk = lane & 3, fr_ = lane >> 2;
	double *C = F + f.foff + pk(f.m, o) + o + i0; // columns o .. of the front
	double acc[4][4][2];
#pragma unroll
	for (int q = 0; q < 4; ++q)
#pragma unroll
		for (int e = 0; e < 2; ++e)
		{
			const int c = wc + 8 * q + 2 * fk + e;
			const double *src = C + (c * t - c * (c + 1) / 2);
#pragma unroll
			for (int p = 0; p < 4; ++p)
			{
				const int i = wr + 8 * p + fr_;
				acc[p][q][e] = c < nc && i0 + i < t && i0 + i >= c ? -src[i] : 0.0;
			}
		}
	cp_async_wait<0>();
	__syncthreads();
#pragma unroll 4
	for (int k = 0; k < NBF; k += 4)
	{
		double a[4], b[4];
#pragma unroll
		for (int q = 0; q < 4; ++q)
		{
			a[q] = A[k + fk][wr + 8 * q + fr_];
			b[q] = B[k + fk][wc + 8 * q + fr_];
		}
#pragma unroll
		for (int p = 0; p < 4; p += 2)
#pragma unroll
			for (int q = 0; q < 4; ++q) dmma(acc[p][q], acc[p + 1][q], a[p], a[p + 1], b[q]);
	}
#pragma unroll
	for (int q = 0; q < 4; ++q)
#pragma unroll
		for (int e = 0; e < 2; ++e)
		{
			const int c = wc + 8 * q + 2 * fk + e;
			double *dst = C + (c * t - c * (c + 1) / 2);
#pragma unroll
			for (int p = 0; p < 4; ++p)
			{
				const int i = wr + 8 * p + fr_;
				if (c < nc && i0 + i < t && i0 + i >= c) dst[i] = -acc[p][q][e];
			}
		}
}

// Trailing lower triangle C -= P P^T, P the rows below of up to 128 panel columns from
// j0.  128 x 64 tiles, four warps of 64 x 32 on the FP64 tensor pipe; the accumulators
// start from -C, so its loads overlap the first panel chunks, which arrive through a
// four-deep cp.async ring of 8 columns (8-byte copies: packed columns have no 16-byte
// alignment) addressed by running 32-bit offsets.
// Bound by the FP64 pipe: 29 of 37 TFLOP/s on fronts of order 10,512 (P2 24^3), where
// 64 x 64 tiles of 4 x 4 multiply-adds per thread reached 9.  Two CTAs per SM instead of
// three: +6%; 16 columns per ring stage: +1%; m16n8k4 steps: +3% of the factorisation.
constexpr int UT_M = 128, UT_N = 64, UT_K = 8, UT_ST = 4;
constexpr int UT_LA = UT_M + 4, UT_LB = UT_N + 4; // 4 mod 16, as above
static_assert(UT_K == 8, "one m16n8k8 step per ring stage");
constexpr size_t UPDATE_SMEM = (size_t)UT_ST * UT_K * (UT_LA + UT_LB) * sizeof(double);
__global__ void __launch_bounds__(128, 3) k_dir_update(const DevFront *__restrict__ fr, const int *__restrict__ list,
													   double *__restrict__ F, int j0)
{
	const DevFront f = fr[list[blockIdx.y]];
	if (f.k <= j0) return;
	const int K = min(2 * NBF, f.k - j0);
	const int o = j0 + K, t = f.m - o; // rows and columns o .. m-1, counted from 0 below
	int c0, r0;
	{
		// column block q from the last has ceil((q + 1) / 2) tiles of 128 rows from its
		// diagonal on; h (h + 1) tiles lie before q = 2 h, (h + 1)^2 before q = 2 h + 1
		const int n64 = (t + UT_N - 1) / UT_N, x = blockIdx.x;
		int h = (int)((sqrtf(4.f * (float)x + 1.f) - 1.f) * 0.5f);
		while ((long long)h * (h + 1) > x) --h;
		while ((long long)(h + 1) * (h + 2) <= x) ++h;
		const int odd = (long long)(h + 1) * (h + 1) <= x;
		const int q = 2 * h + odd, i = x - (odd ? (h + 1) * (h + 1) : h * (h + 1));
		if (q >= n64) return;
		c0 = (n64 - 1 - q) * UT_N;
		r0 = c0 + i * UT_M;
		if (r0 >= t) return;
	}
	extern __shared__ __align__(16) double dsm[];
	const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
	const int wr = (warp & 1) * 64, wc = (warp >> 1) * 32, fk = lane & 3, fr_ = lane >> 2;
	const int nch = (K + UT_K - 1) / UT_K;
	// staging: this thread copies row tid of A, and row tid % 64 of B in the columns of
	// parity tid / 64; the offset of the next column, and its distance to the one after
	const double *P = F + f.foff + pk(f.m, j0) + o;
	const int ld = f.m - j0, l1 = tid / UT_N;
	const bool oka = r0 + tid < t, okb = c0 + tid % UT_N < t;
	int offa = r0 + tid, stepa = ld - 1;
	int offb = c0 + tid % UT_N + l1 * ld - l1, stepb = 2 * ld - 2 * l1 - 3;
	double *sA = dsm + tid, *sB = dsm + UT_ST * UT_K * UT_LA + l1 * UT_LB + tid % UT_N;
	const auto stage = [&](int ch) {
		const int s = (ch % UT_ST) * UT_K, left = K - ch * UT_K;
#pragma unroll
		for (int q = 0; q < UT_K; ++q)
		{
			const bool ok = oka && q < left;
			cp_async8(sA + (s + q) * UT_LA, P + (ok ? offa : 0), ok);
			offa += stepa;
			--stepa;
		}
#pragma unroll
		for (int q = 0; q < UT_K; q += 2)
		{
			const bool ok = okb && q + l1 < left;
			cp_async8(sB + (s + q) * UT_LB, P + (ok ? offb : 0), ok);
			offb += stepb;
			stepb -= 4;
		}
	};
#pragma unroll
	for (int ch = 0; ch < UT_ST - 1; ++ch)
	{
		if (ch < nch) stage(ch);
		cp_async_commit();
	}
	double *C = F + f.foff + o + r0 + wr + fr_;
	double acc[8][4][2];
#pragma unroll
	for (int q = 0; q < 4; ++q)
#pragma unroll
		for (int e = 0; e < 2; ++e)
		{
			const int c = c0 + wc + 8 * q + 2 * fk + e, i0 = r0 + wr + fr_;
			const double *src = C + pk(f.m, o + min(c, t - 1));
#pragma unroll
			for (int p = 0; p < 8; ++p) acc[p][q][e] = i0 + 8 * p < t && i0 + 8 * p >= c ? -src[8 * p] : 0.0;
		}
	const double *fA = dsm + fk * UT_LA + wr + fr_, *fB = dsm + UT_ST * UT_K * UT_LA + fk * UT_LB + wc + fr_;
#pragma unroll 1
	for (int ch = 0; ch < nch; ++ch)
	{
		cp_async_wait<UT_ST - 2>();
		__syncthreads();
		if (ch + UT_ST - 1 < nch) stage(ch + UT_ST - 1);
		cp_async_commit();
		const double *cA = fA + (ch % UT_ST) * UT_K * UT_LA, *cB = fB + (ch % UT_ST) * UT_K * UT_LB;
		double b[4][2];
#pragma unroll
		for (int q = 0; q < 4; ++q)
		{
			b[q][0] = cB[8 * q];
			b[q][1] = cB[4 * UT_LB + 8 * q];
		}
#pragma unroll
		for (int p = 0; p < 8; p += 2)
		{
			const double a[4] = {cA[8 * p], cA[8 * p + 8], cA[4 * UT_LA + 8 * p], cA[4 * UT_LA + 8 * p + 8]};
#pragma unroll
			for (int q = 0; q < 4; ++q) dmma_k8(acc[p][q], acc[p + 1][q], a, b[q][0], b[q][1]);
		}
	}
#pragma unroll
	for (int q = 0; q < 4; ++q)
#pragma unroll
		for (int e = 0; e < 2; ++e)
		{
			const int c = c0 + wc + 8 * q + 2 * fk + e, i0 = r0 + wr + fr_;
			double *dst = C + pk(f.m, o + min(c, t - 1));
#pragma unroll
			for (int p = 0; p < 8; ++p)
				if (i0 + 8 * p < t && i0 + 8 * p >= c) dst[8 * p] = -acc[p][q][e];
		}
}

__global__ void k_dir_permute_in(int n, const int *__restrict__ perm, const double *__restrict__ b, double *__restrict__ bp)
{
	const int q = blockIdx.x * blockDim.x + threadIdx.x;
	if (q < n) bp[q] = b[perm[q]];
}

__global__ void k_dir_permute_out(int n, const int *__restrict__ perm, const double *__restrict__ xp, double *__restrict__ x)
{
	const int q = blockIdx.x * blockDim.x + threadIdx.x;
	if (q < n) x[perm[q]] = xp[q];
}

// Forward substitution, level by level from the leaves, in the factorisation's
// 64-column panels.  k_fwd_init: w = [b_cols; 0] plus the children's update vectors
// (one CTA per front, children in order); k_fwd_step, one launch per panel: every CTA
// solves the panel's right-hand side with the diagonal block (y, written to Y once) and
// updates its own tiles of 64 rows below.  The loads of its first 64 x 64 block of L are issued
// before y is known.  9 to 11 us a panel at P2 24^3; with a CTA per tile of rows, each
// with its own solve of the block, 13.  Two launches per 32-column panel with a substitution
// in one warp, column by column from memory, took 28.
//
// solve_block: one warp, the triangle L in shared memory (D[column][row], zeros past the
// panel), lane i with entries i and i + 32 of w.  Eight entries at a time reach all
// lanes by shuffle, every lane substitutes them (a chain of 16 operations), then takes them
// out of its own two rows.  BACK: L^T, the last eight first.  The solution goes to x[64].
constexpr int FWD_CTAS = 148 * 3;
constexpr int SUB_LD = NBF + 1; // odd: a row across the columns falls on distinct banks too
template <bool BACK>
__device__ __forceinline__ void solve_block(const double (&D)[NBF][SUB_LD], double w0, double w1, double *x)
{
	const int lane = threadIdx.x & 31;
#pragma unroll
	for (int q = 0; q < 8; ++q)
	{
		const int c0 = 8 * (BACK ? 7 - q : q);
		double v[8];
#pragma unroll
		for (int i = 0; i < 8; ++i) v[i] = __shfl_sync(0xffffffffu, c0 < 32 ? w0 : w1, (c0 + i) & 31);
#pragma unroll
		for (int j = 0; j < 8; ++j)
		{
			const int i = BACK ? 7 - j : j;
			v[i] *= D[c0 + i][c0 + i];
#pragma unroll
			for (int l = 0; l < 8; ++l)
				if (BACK ? l < i : l > i) v[l] = fma(BACK ? -D[c0 + l][c0 + i] : -D[c0 + i][c0 + l], v[i], v[l]);
		}
		if (lane == 0)
#pragma unroll
			for (int i = 0; i < 8; ++i) x[c0 + i] = v[i];
		// rows (BACK: columns) already solved take part with entries that nobody reads again
		double s0[2] = {}, s1[2] = {};
#pragma unroll
		for (int i = 0; i < 8; ++i)
		{
			s0[i & 1] = fma(BACK ? D[lane][c0 + i] : D[c0 + i][lane], v[i], s0[i & 1]);
			s1[i & 1] = fma(BACK ? D[lane + 32][c0 + i] : D[c0 + i][lane + 32], v[i], s1[i & 1]);
		}
		w0 -= s0[0] + s0[1];
		w1 -= s1[0] + s1[1];
	}
}
__global__ void __launch_bounds__(256) k_fwd_init(const DevFront *__restrict__ fr, const int *__restrict__ list,
												  const int *__restrict__ child, const int *__restrict__ relpos,
												  const double *__restrict__ bp, double *__restrict__ W)
{
	const DevFront f = fr[list[blockIdx.x]];
	double *w = W + f.woff;
	for (int i = threadIdx.x; i < f.m; i += 256) w[i] = i < f.k ? bp[f.col0 + i] : 0.0;
	__syncthreads();
	for (int ci = 0; ci < f.nchild; ++ci)
	{
		const DevFront c = fr[child[f.child0 + ci]];
		const int rc = c.m - c.k;
		const int *rp = relpos + c.roff;
		const double *wc = W + c.woff + c.k;
		for (int i = threadIdx.x; i < rc; i += 256) w[rp[i]] += wc[i];
		__syncthreads();
	}
}

__global__ void __launch_bounds__(256, 3) k_fwd_step(const DevFront *__restrict__ fr, const int *__restrict__ list,
												  const double *__restrict__ F, double *__restrict__ W,
												  double *__restrict__ Y, int j0)
{
	const DevFront f = fr[list[blockIdx.y]];
	if (j0 >= f.k) return;
	const int nb = min(NBF, f.k - j0), i0 = j0 + nb + blockIdx.x * ROWS_TILE;
	if (blockIdx.x && i0 >= f.m) return;
	const int r = threadIdx.x % NBF, g = threadIdx.x / NBF; // a row, columns 16 g .. 16 g + 15
	double *w = W + f.woff;
	const double *L = F + f.foff;
	__shared__ double D[NBF][SUB_LD], y[NBF], part[4][NBF];
	const bool row = i0 + r < f.m;
	double b[16];
#pragma unroll
	for (int q = 0; q < 16; ++q)
	{
		const int c = 16 * g + q;
		const double *Lc = L + pk(f.m, j0 + min(c, nb - 1));
		D[c][r] = c < nb && r >= c && r < nb ? Lc[j0 + r] : 0.0;
		b[q] = c < nb && row ? Lc[i0 + r] : 0.0;
	}
	const int lane = threadIdx.x;
	const double w0 = lane < 32 && lane < nb ? w[j0 + lane] : 0.0, w1 = lane < 32 && lane + 32 < nb ? w[j0 + lane + 32] : 0.0;
	__syncthreads();
	if (threadIdx.x < 32) solve_block<false>(D, w0, w1, y);
	__syncthreads();
	if (blockIdx.x == 0 && g == 0 && r < nb) Y[f.col0 + j0 + r] = y[r];
	for (int x0 = i0; x0 < f.m; x0 += gridDim.x * ROWS_TILE)
	{
		const bool on = x0 + r < f.m;
		if (x0 != i0)
#pragma unroll
			for (int q = 0; q < 16; ++q)
				b[q] = on && 16 * g + q < nb ? L[pk(f.m, j0 + 16 * g + q) + x0 + r] : 0.0;
		double s = 0.0;
#pragma unroll
		for (int q = 0; q < 16; ++q) s = fma(b[q], y[16 * g + q], s);
		part[g][r] = s;
		__syncthreads();
		if (g == 0 && on) w[x0 + r] -= (part[0][r] + part[1][r]) + (part[2][r] + part[3][r]);
		__syncthreads();
	}
}

__device__ __forceinline__ double warp_sum_d(double v)
{
#pragma unroll
	for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
	return v;
}

// Backward substitution, level by level from the root.  k_bwd_gather: w2 = the rows'
// solution (ancestors, already solved); k_bwd_l21: w1 = y - L21^T w2 (a warp per
// column); k_bwd_step, one launch per panel from the last: every CTA solves the panel's w1
// with the transposed diagonal block (x, written to X once) and
// subtracts the panel's rows times x from its own 64 earlier columns, a warp per
// column, the loads issued before x is known.
__global__ void __launch_bounds__(256) k_bwd_gather(const DevFront *__restrict__ fr, const int *__restrict__ list,
													const int *__restrict__ rows, const double *__restrict__ X,
													double *__restrict__ W)
{
	const DevFront f = fr[list[blockIdx.x]];
	double *w = W + f.woff;
	const int r = f.m - f.k;
	for (int i = threadIdx.x; i < r; i += 256) w[f.k + i] = X[rows[f.ioff + i]];
}

__global__ void __launch_bounds__(256) k_bwd_l21(const DevFront *__restrict__ fr, const int *__restrict__ list,
												 const double *__restrict__ F, const double *__restrict__ Y,
												 double *__restrict__ W)
{
	const DevFront f = fr[list[blockIdx.y]];
	const int j = blockIdx.x * 8 + (threadIdx.x >> 5), lane = threadIdx.x & 31;
	if (j >= f.k) return;
	double *w = W + f.woff;
	const int r = f.m - f.k;
	const double *Lj = F + f.foff + pk(f.m, j) + f.k;
	double s = 0.0;
#pragma unroll 4
	for (int i = lane; i < r; i += 32) s = fma(Lj[i], w[f.k + i], s);
	s = warp_sum_d(s);
	if (lane == 0) w[j] = Y[f.col0 + j] - s;
}

__global__ void __launch_bounds__(256) k_bwd_step(const DevFront *__restrict__ fr, const int *__restrict__ list,
												  const double *__restrict__ F, double *__restrict__ W,
												  double *__restrict__ X, int j0)
{
	const DevFront f = fr[list[blockIdx.y]];
	if (j0 >= f.k) return;
	const int nb = min(NBF, f.k - j0), lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
	const int c0 = blockIdx.x * NBF + warp * 8; // this warp's eight earlier columns
	if (blockIdx.x && blockIdx.x * NBF >= j0) return;
	double *w = W + f.woff;
	const double *L = F + f.foff;
	__shared__ double D[NBF][SUB_LD], x[NBF];
	const bool lo = lane < nb, hi = lane + 32 < nb;
	double b[8][2];
#pragma unroll
	for (int q = 0; q < 8; ++q)
	{
		const int l = warp * 8 + q; // column of the diagonal block
		const double *Lv = L + pk(f.m, j0 + min(l, nb - 1)) + j0;
		D[l][lane] = l < nb && lo && lane >= l ? Lv[lane] : 0.0;
		D[l][lane + 32] = l < nb && hi && lane + 32 >= l ? Lv[lane + 32] : 0.0;
		const bool on = c0 + q < j0;
		const double *Lc = L + pk(f.m, on ? c0 + q : 0) + j0;
		b[q][0] = on && lo ? Lc[lane] : 0.0;
		b[q][1] = on && hi ? Lc[lane + 32] : 0.0;
	}
	const double w0 = lo ? w[j0 + lane] : 0.0, w1 = hi ? w[j0 + lane + 32] : 0.0;
	__syncthreads();
	if (warp == 0) solve_block<true>(D, w0, w1, x);
	__syncthreads();
	const double x0 = x[lane], x1 = x[lane + 32];
	if (blockIdx.x == 0 && warp == 0)
	{
		if (lo) X[f.col0 + j0 + lane] = x0;
		if (hi) X[f.col0 + j0 + lane + 32] = x1;
	}
#pragma unroll
	for (int q = 0; q < 8; ++q)
	{
		const double s = warp_sum_d(fma(b[q][0], x0, b[q][1] * x1));
		if (lane == 0 && c0 + q < j0) w[c0 + q] -= s;
	}
}

} // namespace

// values (device, the analysed pattern's nnz) -> factor; 0 ok, 1 not positive
// definite, else a CUDA error through *ce
int direct_factorize(DirectFactor *f, const double *vals, cudaStream_t s, cudaError_t *ce)
{
	*ce = cudaSuccess;
	f->factorized = false;
	const int nl = (int)f->lvl_start.size() - 1;
	if ((*ce = cudaMemsetAsync(f->d_err, 0, sizeof(int), s)) != cudaSuccess) return 2;
	const auto smem = [&](const void *k, size_t bytes) {
		return (*ce = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes)) == cudaSuccess;
	};
	if (!smem((const void *)k_dir_diag, DIAG_SMEM) || !smem((const void *)k_dir_solve_rows, ROWS_SMEM) ||
		!smem((const void *)k_dir_rows, ROWS_SMEM) || !smem((const void *)k_dir_update, UPDATE_SMEM))
		return 2;
	size_t pi = 0;
	for (int h = 0; h < nl; ++h)
	{
		const int nf = f->lvl_start[h + 1] - f->lvl_start[h];
		const int *list = f->d_lvl_list + f->lvl_start[h];
		const long long fb = f->lvl_fbeg[h], fe = f->lvl_fbeg[h + 1];
		if ((*ce = cudaMemsetAsync(f->d_front + fb, 0, 8 * (size_t)(fe - fb), s)) != cudaSuccess) return 2;
		const long long ab = f->lvl_abeg[h], na = f->lvl_abeg[h + 1] - ab;
		if (na > 0)
			k_dir_assemble<<<(unsigned)((na + 255) / 256), 256, 0, s>>>(na, f->d_amap_src + ab, f->d_amap_dst + ab, vals,
																		 f->d_front);
		for (int ci = 0; ci < f->lvl_maxchild[h]; ++ci)
			if (f->lvl_maxrc[h] > 0)
				k_dir_extend_add<<<dim3((f->lvl_maxrc[h] + 7) / 8, nf), 256, 0, s>>>(f->d_fr, list, f->d_child,
																					 f->d_relpos, f->d_front, ci);
		for (; pi < f->panels.size() && f->panels[pi].lvl == h; ++pi)
		{
			const Panel &p = f->panels[pi];
			const bool second = (p.j0 / NBF) & 1;
			k_dir_diag<<<nf, 256, DIAG_SMEM, s>>>(f->d_fr, list, f->d_front, p.j0, f->d_err);
			if (p.rows_grid > 0) k_dir_solve_rows<<<dim3(p.rows_grid, nf), 128, ROWS_SMEM, s>>>(f->d_fr, list, f->d_front, p.j0);
			if (!second && p.upd_grid > 0)
				k_dir_rows<<<dim3(p.upd_grid, nf), 128, ROWS_SMEM, s>>>(f->d_fr, list, f->d_front, p.j0);
			// the pair's trailing update, after its last panel on this level
			const Panel &p0 = second ? f->panels[pi - 1] : p;
			if ((second || p.upd_grid == 0) && p0.tiles_grid > 0)
				k_dir_update<<<dim3(p0.tiles_grid, nf), 128, UPDATE_SMEM, s>>>(f->d_fr, list, f->d_front, p0.j0);
		}
		if ((*ce = cudaGetLastError()) != cudaSuccess) return 2;
	}
	int bad = 0;
	if ((*ce = cudaMemcpyAsync(&bad, f->d_err, sizeof(int), cudaMemcpyDeviceToHost, s)) != cudaSuccess) return 2;
	if ((*ce = cudaStreamSynchronize(s)) != cudaSuccess) return 2;
	if (bad) return 1;
	f->factorized = true;
	return 0;
}

// x = A^-1 b for device vectors b, x of n entries (x may alias b)
cudaError_t direct_solve(DirectFactor *f, const double *b, double *x, cudaStream_t s)
{
	const int n = f->n;
	if (n == 0) return cudaSuccess;
	double *bp = f->d_vec, *xp = f->d_vec + n; // bp: permuted right-hand side, then y
	const int nl = (int)f->lvl_start.size() - 1;
	k_dir_permute_in<<<(n + 255) / 256, 256, 0, s>>>(n, f->d_perm, b, bp);
	size_t pi = 0;
	for (int h = 0; h < nl; ++h)
	{
		const int nf = f->lvl_start[h + 1] - f->lvl_start[h];
		const int *list = f->d_lvl_list + f->lvl_start[h];
		k_fwd_init<<<nf, 256, 0, s>>>(f->d_fr, list, f->d_child, f->d_relpos, bp, f->d_work);
		for (; pi < f->panels.size() && f->panels[pi].lvl == h; ++pi)
		{
			// every CTA solves the block again: no more of them than the chip holds at once
			const int gx = std::max(1, std::min(f->panels[pi].rows_grid, (FWD_CTAS + nf - 1) / nf));
			k_fwd_step<<<dim3(gx, nf), 256, 0, s>>>(f->d_fr, list, f->d_front, f->d_work, bp, f->panels[pi].j0);
		}
	}
	for (int h = nl - 1; h >= 0; --h)
	{
		const int nf = f->lvl_start[h + 1] - f->lvl_start[h];
		const int *list = f->d_lvl_list + f->lvl_start[h];
		k_bwd_gather<<<nf, 256, 0, s>>>(f->d_fr, list, f->d_rows, xp, f->d_work);
		if (f->lvl_maxk[h] > 0)
			k_bwd_l21<<<dim3((f->lvl_maxk[h] + 7) / 8, nf), 256, 0, s>>>(f->d_fr, list, f->d_front, bp, f->d_work);
		for (; pi > 0 && f->panels[pi - 1].lvl == h; --pi) // this level's panels, last first
		{
			const int j0 = f->panels[pi - 1].j0;
			k_bwd_step<<<dim3(std::max((j0 + NBF - 1) / NBF, 1), nf), 256, 0, s>>>(f->d_fr, list, f->d_front, f->d_work, xp, j0);
		}
	}
	k_dir_permute_out<<<(n + 255) / 256, 256, 0, s>>>(n, f->d_perm, xp, x);
	return cudaGetLastError();
}

} // namespace pfg
