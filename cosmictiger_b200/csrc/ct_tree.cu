// Tree construction on the device, level by level (compiled with -fmad=false so that every
// float/double expression is evaluated exactly as written, matching the reference's C++).
//
// Reference: tree_create (src/tree.cpp:273-601) builds the tree recursively on the host,
// splitting each node at the midpoint of its box's longest dimension with the in-place
// two-pointer partition particles_sort (src/particles.cpp:979-1018).  Here one cooperative launch
// splits all nodes of one depth together, level after level:
//   1. classify: leaf or split, split dimension and midpoint (tree.cpp:314-348);
//   2. number the children in node order;
//   3. partition every split node's range with the exact permutation of the two-pointer
//      loop: with m = #(x < xmid), the k-th element >= xmid in [b, b+m) (counted from the left)
//      swaps with the k-th element < xmid in [b+m, e) (counted from the right);
//   4. create the children.
// The upsweep then runs deepest level first: leaf tight boxes, centres, radii and P2M
// (tree.cpp:498-571), interior unions, the two centre/radius candidates and M2M in double
// (tree.cpp:355-497).  Particles are reordered by moving x, y, z and an index; velocities
// and rungs are gathered through the index at the end (same final arrays as swapping all
// fields in the reference's loop).
#include <cstddef>

#include "ct_internal.cuh"
#include "ct_ops.cuh"

namespace ct {
namespace {

// ---------------------------------------------------------------- the levels
// One cooperative launch builds every level: a resident grid whose blocks meet at grid barriers
// between the phases of a level.  What bounded the build before was the level's structure, not its
// data: twelve launches, two scans and a host round trip a level (16^3 particles: 0.87 ms for 11
// levels and 64 KB of positions; 10^6 clustered particles: 2.7 ms for 28 levels).  A level whose
// split nodes all hold at most WARP_NODE particles takes two barriers, others five.
constexpr int LTPB = 512;             // threads of a level block
constexpr int LWARPS = LTPB / 32;
constexpr int TILE_ROWS = 8;
constexpr int TILE = LTPB * TILE_ROWS;  // particles of a tile
constexpr int WARP_NODE = 1024;       // nodes up to this size are partitioned by one warp: its lanes
                                      // hold the 32 ballots of the node's particles
constexpr int NODE_SPLIT = 2, NODE_TILES = 4;  // NodeW.flags while a level is built

// A node partitioned in tiles by the whole grid.
struct TileNode {
	int32_t node;   // index of the node
	int32_t t0;     // its first tile
	int32_t nt;     // its tiles
	int32_t m;      // particles below the midpoint
	int32_t nswap;  // swaps
};

struct LevelCtl {
	unsigned int arrived;  // barrier arrivals of this launch
	int error;             // a barrier gave up
	int status;            // 0 done, 1 the node arrays are full before `level`
	int level;
	int64_t lb, le;        // nodes of `level`
	int64_t need;          // nodes the arrays must hold
	int64_t start[MAX_DEPTH + 2];
};

struct LevelArgs {
	NodeW* nodes;
	double* gbox;
	uint64_t* key;
	int32_t* depth;
	int32_t* parent;
	uint32_t* x[3];
	int32_t* idx;   // particle index being permuted
	int32_t* posL;  // partition scratch [n]
	int32_t* posR;
	TileNode* tnode;
	int32_t* tile_of;  // tile -> entry of tnode
	int32_t* tile_lt;  // tile -> particles below the midpoint
	int4* blk;         // per block: split nodes, tile nodes, tiles of its share of a level
	LevelCtl* ctl;
	int* flags;
	const int64_t* off;
	int64_t pb, n, node_cap;
	int nroot, bucket, resume;
	double theta, hsoft;
};

// All blocks of the (cooperative) grid meet; false when one gave up waiting.  The counter only
// grows, `round` is the calling block's number of barriers so far.
__device__ __forceinline__ bool grid_meet(LevelCtl* ctl, unsigned int& round) {
	__syncthreads();
	int bad = 0;
	round++;
	if (threadIdx.x == 0) {
		__threadfence();
		const unsigned int target = round * gridDim.x;
		if (atomicAdd(&ctl->arrived, 1u) + 1u != target) {
			const volatile unsigned int* arrived = &ctl->arrived;
			const volatile int* error = &ctl->error;
			unsigned long long t0, t;
			asm volatile("mov.u64 %0, %globaltimer;" : "=l"(t0));
			while ((int) (*arrived - target) < 0 && !bad) {
				asm volatile("mov.u64 %0, %globaltimer;" : "=l"(t));
				bad = *error != 0 || t - t0 > 30000000000ull;  // 30 s: another kernel may hold the SMs for a while
			}
			if (bad) {
				atomicExch(&ctl->error, 1);
			}
		}
		__threadfence();
	}
	return !__syncthreads_or(bad);
}

// Longest side of a node's box and its midpoint (tree.cpp:336-348).
__device__ __forceinline__ int split_dim(const double* gb, double& xm) {
	int xdim = 0;
	double max_span = -1.0;
	for (int dim = 0; dim < 3; dim++) {
		const double span = gb[3 + dim] - gb[dim];
		if (span > max_span) {
			max_span = span;
			xdim = dim;
		}
	}
	xm = 0.5 * (gb[3 + xdim] + gb[xdim]);
	return xdim;
}

// The two children of node ni, split at particle `mid`, by the lanes of a warp.
__device__ __forceinline__ void make_children(const LevelArgs& a, int64_t ni, const NodeW& nd, int mid, int xd, double xm, int level, int lane) {
	const int64_t l = nd.child;
	if (lane < 2) {
		NodeW c;
		c.x = c.y = c.z = 0;
		c.radius = 0.f;
		c.child = -1;
		c.flags = 1;
		c.pbeg = lane == 0 ? nd.pbeg : mid;
		c.pend = lane == 0 ? mid : nd.pend;
		a.nodes[l + lane] = c;
		a.key[l + lane] = (a.key[ni] << 1) + lane;
		a.depth[l + lane] = level + 1;
		a.parent[l + lane] = (int32_t) ni;
	}
	if (lane < 12) {
		const int side = lane / 6, d = lane % 6;
		a.gbox[6 * (l + side) + d] = d == (side == 0 ? 3 + xd : xd) ? xm : a.gbox[6 * ni + d];
	}
}

__device__ __forceinline__ void swap_particles(const LevelArgs& a, int p, int q) {
#pragma unroll
	for (int d = 0; d < 3; d++) {
		const uint32_t t = a.x[d][p];
		a.x[d][p] = a.x[d][q];
		a.x[d][q] = t;
	}
	const int32_t t = a.idx[p];
	a.idx[p] = a.idx[q];
	a.idx[q] = t;
}

// The partition of a node of at most WARP_NODE particles by one warp: lane c keeps the ballot of
// particles 32 c .. 32 c + 31.  With m of them below the midpoint, the k-th particle at or above it
// in the first m (from the left) changes places with the k-th below it in the rest (from the
// right), which is the reference's two-pointer loop.  pos: WARP_NODE offsets in shared memory.
__device__ __forceinline__ int warp_partition(const LevelArgs& a, const NodeW& nd, const uint32_t* xd, uint32_t xm, uint16_t* pos, int lane) {
	const int n = nd.pend - nd.pbeg;
	const uint32_t* xp = xd + nd.pbeg;
	unsigned mine = 0;
	for (int c0 = 0; c0 * 32 < n; c0 += 8) {
		uint32_t v[8];
#pragma unroll
		for (int j = 0; j < 8; j++) {
			const int p = 32 * (c0 + j) + lane;
			v[j] = p < n ? xp[p] : 0xffffffffu;
		}
#pragma unroll
		for (int j = 0; j < 8; j++) {
			const unsigned lt = __ballot_sync(0xffffffffu, 32 * (c0 + j) + lane < n && v[j] < xm);
			mine = lane == c0 + j ? lt : mine;
		}
	}
	int m = __popc(mine);
	for (int o = 16; o; o >>= 1) {
		m += __shfl_xor_sync(0xffffffffu, m, o);
	}
	// this lane's 32 particles: those before the split point that are not below, and below after it
	const int first = 32 * lane;
	const unsigned valid = first >= n ? 0u : (n - first >= 32 ? 0xffffffffu : (1u << (n - first)) - 1u);
	const unsigned before = first >= m ? 0u : (m - first >= 32 ? 0xffffffffu : (1u << (m - first)) - 1u);
	unsigned L = before & ~mine & valid, R = mine & ~before;
	int cl = __popc(L), cr = __popc(R);
	int il = cl, ir = cr;
	for (int o = 1; o < 32; o <<= 1) {
		const int tl = __shfl_up_sync(0xffffffffu, il, o), tr = __shfl_up_sync(0xffffffffu, ir, o);
		il += lane >= o ? tl : 0;
		ir += lane >= o ? tr : 0;
	}
	const int ns = __shfl_sync(0xffffffffu, il, 31);  // as many on the right
	if (ns > 0) {
		uint16_t* pl = pos;
		uint16_t* pr = pos + WARP_NODE / 2;
		int k = il - cl;
		while (L) {
			pl[k++] = (uint16_t) (first + __ffs(L) - 1);
			L &= L - 1;
		}
		k = ns - 1 - (ir - cr);
		while (R) {
			pr[k--] = (uint16_t) (first + __ffs(R) - 1);
			R &= R - 1;
		}
		__syncwarp();
		for (int q = lane; q < ns; q += 32) {
			swap_particles(a, nd.pbeg + pl[q], nd.pbeg + pr[q]);
		}
		__syncwarp();
	}
	return m;
}

__global__ void __launch_bounds__(LTPB, 2) k_tree_levels(const LevelArgs a) {
	__shared__ uint16_t s_pos[LWARPS][WARP_NODE];
	__shared__ int s_cnt[TILE_ROWS * LWARPS];
	__shared__ int s_scan[3][LWARPS];
	__shared__ int s_sum[2][LWARPS];
	__shared__ int s_next;
	const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
	const unsigned lt_lane = (1u << lane) - 1u;
	LevelCtl* ctl = a.ctl;
	unsigned int round = 0;
	int level = 0;
	int64_t lb = 0, le = a.nroot;
	if (a.resume) {
		level = ctl->level;
		lb = ctl->lb;
		le = ctl->le;
	} else {
		const int64_t gt = blockIdx.x * (int64_t) LTPB + tid, gs = gridDim.x * (int64_t) LTPB;
		for (int64_t i = gt; i < a.n; i += gs) {
			a.idx[i] = (int32_t) i;
		}
		// one root per box: node s covers the unit box and particles [off[s], off[s+1]), except that
		// a single box starts at the active range
		for (int64_t s = gt; s < a.nroot; s += gs) {
			NodeW r;
			r.x = r.y = r.z = 0;
			r.radius = 0.f;
			r.pbeg = a.nroot == 1 ? (int32_t) a.pb : (int32_t) a.off[s];
			r.pend = a.nroot == 1 ? (int32_t) a.n : (int32_t) a.off[s + 1];
			r.child = -1;
			r.flags = 1;
			a.nodes[s] = r;
			for (int d = 0; d < 3; d++) {
				a.gbox[6 * s + d] = 0.0;
				a.gbox[6 * s + 3 + d] = 1.0;
			}
			a.key[s] = 1;
			a.depth[s] = 0;
			a.parent[s] = -1;
		}
		if (!grid_meet(ctl, round)) {
			return;
		}
	}
	for (;; level++) {
		const int64_t nl = le - lb;
		const int64_t share = (nl + gridDim.x - 1) / gridDim.x;  // consecutive nodes of a block
		const int64_t cb = lb + min(nl, share * blockIdx.x), ce = lb + min(nl, share * (blockIdx.x + 1));
		// ---- leaf or split (tree.cpp:314-348), counted per block
		int nsplit = 0, ntn = 0, ntile = 0;
		for (int64_t ni = cb + tid; ni < ce; ni += LTPB) {
			const int2 pr = *reinterpret_cast<const int2*>(&a.nodes[ni].pbeg);
			const int nparts = pr.y - pr.x;
			const double* gb = a.gbox + 6 * ni;
			float box_r = 0.0f;
			for (int dim = 0; dim < 3; dim++) {
				const double h = 0.5 * (gb[3 + dim] - gb[dim]);
				box_r += h * h;
			}
			box_r = sqrtf(box_r);
			const bool ewald_satisfied = (box_r < 0.25 * (a.theta / (1.0 + a.theta)) && box_r < 0.125 - 0.25 * a.hsoft);
			bool split = nparts > a.bucket || (!ewald_satisfied && nparts > 0);
			if (split && level >= MAX_DEPTH - 1) {
				atomicOr(a.flags + 2, 1);
				split = false;
			}
			const bool tiles = split && nparts > WARP_NODE;
			a.nodes[ni].flags = split ? (tiles ? NODE_SPLIT | NODE_TILES : NODE_SPLIT) : 1;
			nsplit += split;
			ntn += tiles;
			ntile += tiles ? (nparts + TILE - 1) / TILE : 0;
		}
		for (int o = 16; o; o >>= 1) {
			nsplit += __shfl_xor_sync(0xffffffffu, nsplit, o);
			ntn += __shfl_xor_sync(0xffffffffu, ntn, o);
			ntile += __shfl_xor_sync(0xffffffffu, ntile, o);
		}
		if (lane == 0) {
			s_scan[0][w] = nsplit;
			s_scan[1][w] = ntn;
			s_scan[2][w] = ntile;
		}
		__syncthreads();
		if (tid == 0) {
			int4 t = make_int4(0, 0, 0, 0);
			for (int i = 0; i < LWARPS; i++) {
				t.x += s_scan[0][i];
				t.y += s_scan[1][i];
				t.z += s_scan[2][i];
			}
			a.blk[blockIdx.x] = t;
		}
		if (!grid_meet(ctl, round)) {
			return;
		}
		// ---- totals of the level and of the blocks before this one (a warp: at most a few hundred)
		int base[3] = { 0, 0, 0 }, tot[3] = { 0, 0, 0 };
		for (int i = lane; i < (int) gridDim.x; i += 32) {
			const int4 t = __ldcg(a.blk + i);
			const bool prev = i < (int) blockIdx.x;
			tot[0] += t.x;
			tot[1] += t.y;
			tot[2] += t.z;
			base[0] += prev ? t.x : 0;
			base[1] += prev ? t.y : 0;
			base[2] += prev ? t.z : 0;
		}
		for (int o = 16; o; o >>= 1) {
			for (int q = 0; q < 3; q++) {
				tot[q] += __shfl_xor_sync(0xffffffffu, tot[q], o);
				base[q] += __shfl_xor_sync(0xffffffffu, base[q], o);
			}
		}
		const int64_t next_le = le + 2 * (int64_t) tot[0];
		if (next_le > a.node_cap) {
			// every block sees the same totals: all stop here, before the level changes anything
			if (blockIdx.x == 0 && tid == 0) {
				ctl->status = 1;
				ctl->level = level;
				ctl->lb = lb;
				ctl->le = le;
				ctl->need = next_le;
			}
			return;
		}
		if (blockIdx.x == 0 && tid == 0) {
			ctl->start[level] = lb;
			ctl->start[level + 1] = le;
			ctl->level = level;
		}
		// ---- children's indices in node order, tile nodes listed
		for (int64_t n0 = cb; n0 < ce; n0 += LTPB) {
			const int64_t ni = n0 + tid;
			const int f = ni < ce ? a.nodes[ni].flags : 1;
			const int sp = (f & NODE_SPLIT) != 0, tn = (f & NODE_TILES) != 0;
			int nt = 0;
			if (tn) {
				const int2 pr = *reinterpret_cast<const int2*>(&a.nodes[ni].pbeg);
				nt = (pr.y - pr.x + TILE - 1) / TILE;
			}
			int inc = nt;
			for (int o = 1; o < 32; o <<= 1) {
				const int t = __shfl_up_sync(0xffffffffu, inc, o);
				inc += lane >= o ? t : 0;
			}
			const unsigned ms = __ballot_sync(0xffffffffu, sp), mt = __ballot_sync(0xffffffffu, tn);
			__syncthreads();
			if (lane == 31) {
				s_scan[0][w] = __popc(ms);
				s_scan[1][w] = __popc(mt);
				s_scan[2][w] = inc;
			}
			__syncthreads();
			int e0 = base[0], e1 = base[1], e2 = base[2];
			for (int i = 0; i < LWARPS; i++) {
				const int q0 = s_scan[0][i], q1 = s_scan[1][i], q2 = s_scan[2][i];
				e0 += i < w ? q0 : 0;
				e1 += i < w ? q1 : 0;
				e2 += i < w ? q2 : 0;
				base[0] += q0;
				base[1] += q1;
				base[2] += q2;
			}
			if (sp) {
				a.nodes[ni].child = (int32_t) (le + 2 * (int64_t) (e0 + __popc(ms & lt_lane)));
				a.nodes[ni].flags = 0;
			}
			if (tn) {
				TileNode t;
				t.node = (int32_t) ni;
				t.t0 = e2 + inc - nt;
				t.nt = nt;
				t.m = t.nswap = 0;
				a.tnode[e1 + __popc(mt & lt_lane)] = t;
				for (int q = 0; q < nt; q++) {
					a.tile_of[t.t0 + q] = e1 + __popc(mt & lt_lane);
				}
			}
		}
		// ---- nodes of at most WARP_NODE particles: a warp each, taken from the block's share
		if (tid == 0) {
			s_next = 0;
		}
		__syncthreads();
		for (;;) {
			int k = 0;
			if (lane == 0) {
				k = atomicAdd(&s_next, 1);
			}
			const int64_t ni = cb + __shfl_sync(0xffffffffu, k, 0);
			if (ni >= ce) {
				break;
			}
			const NodeW nd = a.nodes[ni];
			if (nd.child < 0 || nd.pend - nd.pbeg > WARP_NODE) {
				continue;
			}
			double xm;
			const int xd = split_dim(a.gbox + 6 * ni, xm);
			const int m = warp_partition(a, nd, xd == 0 ? a.x[0] : xd == 1 ? a.x[1] : a.x[2], fixed_from_double(xm), s_pos[w], lane);
			make_children(a, ni, nd, nd.pbeg + m, xd, xm, level, lane);
		}
		if (tot[2] > 0) {
			if (!grid_meet(ctl, round)) {
				return;
			}
			// ---- larger nodes, tile by tile: particles below the midpoint
			for (int t = blockIdx.x; t < tot[2]; t += gridDim.x) {
				const TileNode tn = a.tnode[a.tile_of[t]];
				const int2 pr = *reinterpret_cast<const int2*>(&a.nodes[tn.node].pbeg);
				double xm;
				const int xd = split_dim(a.gbox + 6 * (int64_t) tn.node, xm);
				const uint32_t* x = xd == 0 ? a.x[0] : xd == 1 ? a.x[1] : a.x[2];
				const uint32_t xf = fixed_from_double(xm);
				const int p0 = pr.x + (t - tn.t0) * TILE + tid;
				int c = 0;
#pragma unroll
				for (int j = 0; j < TILE_ROWS; j++) {
					const int p = p0 + j * LTPB;
					c += p < pr.y && x[min(p, pr.y - 1)] < xf;
				}
				c = __reduce_add_sync(0xffffffffu, c);
				if (lane == 0) {
					s_sum[0][w] = c;
				}
				__syncthreads();
				if (tid == 0) {
					int s = 0;
					for (int i = 0; i < LWARPS; i++) {
						s += s_sum[0][i];
					}
					a.tile_lt[t] = s;
				}
				__syncthreads();
			}
			if (!grid_meet(ctl, round)) {
				return;
			}
			// positions of the particles on the wrong side of the split point: before it ranked from the
			// node's left, after it from the node's right.  Earlier tiles hold only particles before a
			// particle on the left, later ones only particles after one on the right, so the counts
			// below the midpoint of whole tiles give both ranks.
			for (int t = blockIdx.x; t < tot[2]; t += gridDim.x) {
				const int ti = a.tile_of[t];
				const TileNode tn = a.tnode[ti];
				const int2 pr = *reinterpret_cast<const int2*>(&a.nodes[tn.node].pbeg);
				double xm;
				const int xd = split_dim(a.gbox + 6 * (int64_t) tn.node, xm);
				const uint32_t* x = xd == 0 ? a.x[0] : xd == 1 ? a.x[1] : a.x[2];
				const uint32_t xf = fixed_from_double(xm);
				const int tb = pr.x + (t - tn.t0) * TILE, te = min(tb + TILE, pr.y);
				unsigned below = 0;  // bit j: row j's particle of this thread
#pragma unroll
				for (int j = 0; j < TILE_ROWS; j++) {
					const int p = tb + j * LTPB + tid;
					below |= (unsigned) (p < te && x[min(p, te - 1)] < xf) << j;
				}
				int all = 0, prev = 0;
				for (int q = tid; q < tn.nt; q += LTPB) {
					const int c = __ldcg(a.tile_lt + tn.t0 + q);
					all += c;
					prev += q < t - tn.t0 ? c : 0;
				}
				all = __reduce_add_sync(0xffffffffu, all);
				prev = __reduce_add_sync(0xffffffffu, prev);
				if (lane == 0) {
					s_sum[0][w] = all;
					s_sum[1][w] = prev;
				}
				__syncthreads();
				int m = 0, lt_prev = 0;
				for (int i = 0; i < LWARPS; i++) {
					m += s_sum[0][i];
					lt_prev += s_sum[1][i];
				}
				const int sp = pr.x + m;
				unsigned wrong = 0;
				int right = 0;  // wrong ones after the split point
#pragma unroll
				for (int j = 0; j < TILE_ROWS; j++) {
					const int p = tb + j * LTPB + tid;
					const bool lt = below >> j & 1u;
					const bool bad = p < te && (p < sp ? !lt : lt);
					const unsigned mk = __ballot_sync(0xffffffffu, bad);
					wrong |= (unsigned) bad << j;
					right += bad && p >= sp;
					if (lane == 0) {
						s_cnt[j * LWARPS + w] = __popc(mk);
					}
				}
				__syncthreads();
				// prefix of the rows' warps in particle order, by every warp for itself
				int mybase[TILE_ROWS], run = 0;
				{
					constexpr int PER = TILE_ROWS * LWARPS / 32;
					int c[PER], s = 0;
					for (int i = 0; i < PER; i++) {
						c[i] = s_cnt[lane * PER + i];
						s += c[i];
					}
					int inc = s;
					for (int o = 1; o < 32; o <<= 1) {
						const int v = __shfl_up_sync(0xffffffffu, inc, o);
						inc += lane >= o ? v : 0;
					}
					run = __shfl_sync(0xffffffffu, inc, 31);
					int ex[PER];
					int e = inc - s;
					for (int i = 0; i < PER; i++) {
						ex[i] = e;
						e += c[i];
					}
#pragma unroll
					for (int j = 0; j < TILE_ROWS; j++) {
						const int q = j * LWARPS + w;
						int v = 0;
						for (int i = 0; i < PER; i++) {
							const int u = __shfl_sync(0xffffffffu, ex[i], q / PER);
							v = q % PER == i ? u : v;
						}
						mybase[j] = v;
					}
				}
				right = __reduce_add_sync(0xffffffffu, right);
				__syncthreads();
				if (lane == 0) {
					s_sum[0][w] = right;
				}
				__syncthreads();
				int nright = 0;
				for (int i = 0; i < LWARPS; i++) {
					nright += s_sum[0][i];
				}
				const int lt_tile = __ldcg(a.tile_lt + t);
				const int after = m - lt_prev - lt_tile;  // below the midpoint in later tiles
				const int leftbase = (tb - pr.x) - lt_prev;
#pragma unroll
				for (int j = 0; j < TILE_ROWS; j++) {
					const bool bad = wrong >> j & 1u;
					const unsigned mk = __ballot_sync(0xffffffffu, bad);
					if (bad) {
						const int p = tb + j * LTPB + tid;
						const int e = mybase[j] + __popc(mk & lt_lane);
						if (p < sp) {
							a.posL[pr.x + leftbase + e] = p;
						} else {
							a.posR[pr.x + after + (run - e - 1)] = p;
						}
					}
				}
				if (tid == 0) {
					if (t == tn.t0) {
						a.tnode[ti].m = m;
					}
					// the tile that holds the split point (or the last one, when nothing lies after it)
					if ((tb <= sp && sp < te) || (sp == pr.y && te == pr.y)) {
						a.tnode[ti].nswap = after + nright;
					}
				}
				__syncthreads();
			}
			if (!grid_meet(ctl, round)) {
				return;
			}
			for (int t = blockIdx.x; t < tot[2]; t += gridDim.x) {
				const TileNode* tp = a.tnode + a.tile_of[t];
				const int node = tp->node, t0 = tp->t0;
				const int m = __ldcg(&tp->m), ns = __ldcg(&tp->nswap);
				const int pbeg = a.nodes[node].pbeg;
				for (int k = (t - t0) * TILE + tid; k < min(ns, (t - t0 + 1) * TILE); k += LTPB) {
					swap_particles(a, __ldcg(a.posL + pbeg + k), __ldcg(a.posR + pbeg + k));
				}
				if (t == t0 && w == 0) {
					double xm;
					const int xd = split_dim(a.gbox + 6 * (int64_t) node, xm);
					make_children(a, node, a.nodes[node], pbeg + m, xd, xm, level, lane);
				}
			}
		}
		if (tot[0] == 0) {
			break;
		}
		lb = le;
		le = next_le;
		if (!grid_meet(ctl, round)) {
			return;
		}
	}
	if (blockIdx.x == 0 && tid == 0) {
		ctl->status = 0;
	}
}

__global__ void k_gather_particles(int64_t b, int64_t n, const int32_t* idx, const float* v0, const float* v1, const float* v2, const int8_t* r,
		float* o0, float* o1, float* o2, int8_t* orr) {
	for (int64_t i = b + blockIdx.x * (int64_t) blockDim.x + threadIdx.x; i < n; i += (int64_t) gridDim.x * blockDim.x) {
		const int j = idx[i];
		o0[i] = v0[j];
		o1[i] = v1[j];
		o2[i] = v2[j];
		orr[i] = r[j];
	}
}

// ---------------------------------------------------------------- upsweep
template<class T>
__device__ __forceinline__ T warp_max(T v) {
	for (int o = 16; o; o >>= 1) {
		v = max(v, __shfl_xor_sync(0xffffffffu, v, o));
	}
	return v;
}
template<class T>
__device__ __forceinline__ T warp_min(T v) {
	for (int o = 16; o; o >>= 1) {
		v = min(v, __shfl_xor_sync(0xffffffffu, v, o));
	}
	return v;
}
template<class T>
__device__ __forceinline__ T warp_sum(T v) {
	for (int o = 16; o; o >>= 1) {
		v += __shfl_xor_sync(0xffffffffu, v, o);
	}
	return v;
}

constexpr int UTPB = 128;

// A warp per node (tree.cpp:351-571): tight box, expansion centre and radius, multipole (P2M of
// the particles for a leaf, M2M of the two children in double for an interior node).
template<class Ops>
__global__ void __launch_bounds__(UTPB) k_upsweep(int64_t lb, int64_t le, NodeW* nodes, int32_t* nbox, float* multi, double* tbox, const double* gbox,
		const uint32_t* x0, const uint32_t* x1, const uint32_t* x2, int bucket) {
	constexpr int NM = Ops::NMULT;
	const uint32_t* xs[3] = { x0, x1, x2 };
	const int lane = threadIdx.x & 31;
	const int64_t gw = (blockIdx.x * (int64_t) blockDim.x + threadIdx.x) >> 5;
	const int64_t nw = ((int64_t) gridDim.x * blockDim.x) >> 5;
	for (int64_t ni = lb + gw; ni < le; ni += nw) {
		const NodeW nd = nodes[ni];
		const int nparts = nd.pend - nd.pbeg;
		const double* gb = gbox + 6 * ni;
		if (nd.child < 0) {
			// ---- leaf (tree.cpp:498-571)
			double mn[3], mx[3];
			for (int d = 0; d < 3; d++) {
				mn[d] = gb[3 + d];
				mx[d] = gb[d];
			}
			for (int p = nd.pbeg + lane; p < nd.pend; p += 32) {
				for (int d = 0; d < 3; d++) {
					const double xx = fixed_to_double(xs[d][p]);
					mx[d] = fmax(mx[d], xx);
					mn[d] = fmin(mn[d], xx);
				}
			}
			for (int d = 0; d < 3; d++) {
				mn[d] = warp_min(mn[d]);
				mx[d] = warp_max(mx[d]);
			}
			double Xc[3];
			for (int d = 0; d < 3; d++) {
				Xc[d] = (mx[d] + mn[d]) * 0.5;
			}
			double r = 0.0;
			for (int p = nd.pbeg + lane; p < nd.pend; p += 32) {
				double this_radius = 0.0;
				for (int d = 0; d < 3; d++) {
					const double dx = fixed_to_double(xs[d][p]) - Xc[d];
					this_radius += dx * dx;
				}
				r = fmax(r, this_radius);
			}
			r = warp_max(r);
			// P2M about fixed32(Xc), summed in double
			uint32_t Y[3];
			for (int d = 0; d < 3; d++) {
				Y[d] = fixed_from_double(Xc[d]);
			}
			double M[NM];
			for (int k = 0; k < NM; k++) {
				M[k] = 0.0;
			}
			for (int p = nd.pbeg + lane; p < nd.pend; p += 32) {
				float m[NM];
				Ops::p2m(m, fixed_dist(x0[p], Y[0]), fixed_dist(x1[p], Y[1]), fixed_dist(x2[p], Y[2]));
				for (int k = 0; k < NM; k++) {
					M[k] += (double) m[k];
				}
			}
			for (int k = 0; k < NM; k++) {
				M[k] = warp_sum(M[k]);
			}
			if (lane == 0) {
				NodeW o = nd;
				o.x = Y[0];
				o.y = Y[1];
				o.z = Y[2];
				o.radius = (float) sqrt(r);
				nodes[ni] = o;
				for (int d = 0; d < 3; d++) {
					tbox[6 * ni + d] = mn[d];
					tbox[6 * ni + 3 + d] = mx[d];
					nbox[6 * ni + d] = range_fixed_from_double(mn[d]);
					nbox[6 * ni + 3 + d] = range_fixed_from_double(mx[d]);
				}
			}
#pragma unroll
			for (int k = 0; k < NM; k++) {
				if (lane == (k & 31)) {
					multi[NMULT_STRIDE * ni + k] = (float) M[k];
				}
			}
		} else {
			// ---- interior node (tree.cpp:351-497)
			const int64_t L = nd.child, R = nd.child + 1;
			const NodeW nl = nodes[L], nr = nodes[R];
			const float ml0 = multi[NMULT_STRIDE * L], mr0 = multi[NMULT_STRIDE * R];
			double bb[3], be[3];
			for (int d = 0; d < 3; d++) {
				const double lb_ = tbox[6 * L + d], le_ = tbox[6 * L + 3 + d];
				const double rb_ = tbox[6 * R + d], re_ = tbox[6 * R + 3 + d];
				if (ml0 != 0.0f && mr0 != 0.0f) {
					bb[d] = fmin(lb_, rb_);
					be[d] = fmax(le_, re_);
				} else if (ml0 != 0.0f) {
					bb[d] = lb_;
					be[d] = le_;
				} else {
					bb[d] = rb_;
					be[d] = re_;
				}
			}
			int xdim = 0;
			{
				double max_span = -1.0;
				for (int d = 0; d < 3; d++) {
					const double span = gb[3 + d] - gb[d];
					if (span > max_span) {
						max_span = span;
						xdim = d;
					}
				}
			}
			const bool tried1 = nparts <= 64 * bucket && (be[xdim] - bb[xdim] <= 0.5);
			double Xc1[3];
			float r2max = 0.0f;
			if (tried1) {
				uint32_t xc[3];
				for (int d = 0; d < 3; d++) {
					Xc1[d] = 0.5 * (bb[d] + be[d]);
					xc[d] = fixed_from_double(Xc1[d]);
				}
				for (int p = nd.pbeg + lane; p < nd.pend; p += 32) {
					const float dx = fixed_dist(x0[p], xc[0]);
					const float dy = fixed_dist(x1[p], xc[1]);
					const float dz = fixed_dist(x2[p], xc[2]);
					const float r2 = dx * dx + dy * dy + dz * dz;
					r2max = fmaxf(r2max, r2);
				}
				r2max = warp_max(r2max);
			}
			double sX[3];
			{
				const double Xl[3] = { fixed_to_double(nl.x), fixed_to_double(nl.y), fixed_to_double(nl.z) };
				const double Xr[3] = { fixed_to_double(nr.x), fixed_to_double(nr.y), fixed_to_double(nr.z) };
				const double radius1 = tried1 ? (double) sqrtf(r2max) : 0.0;
				double N[3];
				double norminv = 0.0;
				for (int d = 0; d < 3; d++) {
					N[d] = Xl[d] - Xr[d];
					norminv += N[d] * N[d];
				}
				norminv = 1.0 / sqrt(norminv);
				for (int d = 0; d < 3; d++) {
					N[d] *= norminv;
					N[d] = fabs(N[d]);
				}
				double r = 0.0, Xc2[3];
				const double Rl = nl.radius, Rr = nr.radius;
				if (mr0 != 0.0f) {
					if (ml0 != 0.0f) {
						for (int d = 0; d < 3; d++) {
							const double a = Xl[d] + N[d] * Rl, b = Xr[d] + N[d] * Rr;
							const double xmax = (a < b) ? b : a;  // std::max
							const double c = Xl[d] - N[d] * Rl, e = Xr[d] - N[d] * Rr;
							const double xmin = (e < c) ? e : c;  // std::min
							Xc2[d] = (xmax + xmin) * 0.5;
							const double t = (xmax - xmin) * 0.5;
							r += t * t;
						}
					} else {
						for (int d = 0; d < 3; d++) {
							Xc2[d] = Xr[d];
						}
						r = Rr * Rr;
					}
				} else {
					for (int d = 0; d < 3; d++) {
						Xc2[d] = Xl[d];
					}
					r = Rl * Rl;
				}
				const double radius2 = sqrt(r);
				double Xc[3];
				float radius;
				if (tried1 && radius1 < radius2) {
					for (int d = 0; d < 3; d++) {
						Xc[d] = Xc1[d];
					}
					radius = (float) radius1;
				} else {
					for (int d = 0; d < 3; d++) {
						Xc[d] = Xc2[d];
					}
					radius = (float) radius2;
				}
				r = 0.0;
				for (int d = 0; d < 3; d++) {
					const double span = be[d] - bb[d];
					r += (span * 0.5) * (span * 0.5);
				}
				r = sqrt(r);
				if (r < radius) {
					radius = (float) r;
					for (int d = 0; d < 3; d++) {
						Xc[d] = (bb[d] + be[d]) * 0.5;
					}
				}
				for (int d = 0; d < 3; d++) {
					sX[d] = Xc[d];
				}
				NodeW o = nd;
				o.x = fixed_from_double(Xc[0]);
				o.y = fixed_from_double(Xc[1]);
				o.z = fixed_from_double(Xc[2]);
				o.radius = radius;
				if (lane == 0) {
					nodes[ni] = o;
					for (int d = 0; d < 3; d++) {
						tbox[6 * ni + d] = bb[d];
						tbox[6 * ni + 3 + d] = be[d];
						nbox[6 * ni + d] = range_fixed_from_double(bb[d]);
						nbox[6 * ni + 3 + d] = range_fixed_from_double(be[d]);
					}
				}
			}
			// M2M of both children in double (tree.cpp:481-494): lane 0 the left, lane 1 the right,
			// then left + right
			double Mo[NM];
			for (int k = 0; k < NM; k++) {
				Mo[k] = 0.0;
			}
			if (lane < 2) {
				const int64_t c = lane == 0 ? L : R;
				const NodeW cn = lane == 0 ? nl : nr;
				double Ma[NM];
				for (int k = 0; k < NM; k++) {
					Ma[k] = (double) multi[NMULT_STRIDE * c + k];
				}
				Ops::m2m(Mo, Ma, fixed_to_double(cn.x) - sX[0], fixed_to_double(cn.y) - sX[1], fixed_to_double(cn.z) - sX[2]);
			}
			for (int k = 0; k < NM; k++) {
				const double right = __shfl_down_sync(0xffffffffu, Mo[k], 1);
				if (lane == 0) {
					multi[NMULT_STRIDE * ni + k] = (float) (Mo[k] + right);
				}
			}
		}
	}
}

template<class T>
ct_status grow(Ctx* c, T** p, int64_t old_n, int64_t new_n, int per, const char* what) {
	T* q = nullptr;
	CT_TRY(dalloc(c, (void**) &q, sizeof(T) * per * new_n, what));
	if (*p) {
		CT_CUDA(c, cudaMemcpyAsync(q, *p, sizeof(T) * per * old_n, cudaMemcpyDeviceToDevice, c->stream));
		CT_CUDA(c, cudaStreamSynchronize(c->stream));
		dfree(c, *p, sizeof(T) * per * old_n);
	}
	*p = q;
	return CT_OK;
}

ct_status ensure_nodes(Ctx* c, Box* b, int64_t need) {
	if (need <= b->node_cap) {
		return CT_OK;
	}
	int64_t cap = std::max<int64_t>(need, b->node_cap * 3 / 2);
	cap = std::max<int64_t>(cap, 1024);
	const int64_t old = b->node_cap;
	CT_TRY(grow(c, &b->nodes, old, cap, 1, "tree nodes"));
	CT_TRY(grow(c, &b->nbox, old, cap, 6, "node boxes"));
	CT_TRY(grow(c, &b->multi, old, cap, NMULT_STRIDE, "multipoles"));
	CT_TRY(grow(c, &b->key, old, cap, 1, "node keys"));
	CT_TRY(grow(c, &b->depth, old, cap, 1, "node depth"));
	CT_TRY(grow(c, &b->parent, old, cap, 1, "node parent"));
	CT_TRY(grow(c, &b->gbox, old, cap, 6, "node geometric box"));
	CT_TRY(grow(c, &b->tbox, old, cap, 6, "node tight box"));
	b->node_cap = cap;
	return CT_OK;
}

int grid_for(Ctx* c, int64_t work, int tpb, int per_sm = 8) {
	const int64_t g = (work + tpb - 1) / tpb;
	return (int) std::max<int64_t>(1, std::min<int64_t>(g, (int64_t) c->nsm * per_sm));
}

template<class Ops>
ct_status tree_build_t(Ctx* c, Box* b, const ct_tree_params* p) {
	cudaStream_t st = c->stream;
	const int64_t n = b->n;
	const int64_t pb = b->rung_begin;
	const int64_t np = n - pb;
	b->tree_valid = false;
	if (np > INT32_MAX / 2) {
		return fail(c, CT_ERR_ARG, "box too large for 32-bit particle indices");
	}
	// node capacity: the reference's arena, max(8 N / bucket, 2^21) (tree.cpp:247) is an
	// upper estimate; start smaller and grow per level as needed.
	CT_TRY(ensure_nodes(c, b, std::max<int64_t>(4 * np / std::max(p->bucket, 1) + 4096, 8192)));
	ct_status s1 = CT_OK;
	const int nroot = b->nsub;
	CT_TRY(ensure_nodes(c, b, nroot + 1));
	// one block an SM (two boxes built by two contexts fit side by side), fewer for a few particles
	const int nblk = (int) std::max<int64_t>(1, std::min<int64_t>(c->nsm, std::max<int64_t>(np / 64, nroot)));
	LevelArgs la;
	la.idx = (int32_t*) scratch(c, 0, sizeof(int32_t) * n, &s1);
	la.posL = (int32_t*) scratch(c, 1, sizeof(int32_t) * n, &s1);
	la.posR = (int32_t*) scratch(c, 2, sizeof(int32_t) * n, &s1);
	// nodes in tiles hold more than WARP_NODE particles each
	const int64_t max_tn = np / WARP_NODE + 1, max_tiles = np / TILE + max_tn + 1;
	la.tnode = (TileNode*) scratch(c, 3, sizeof(TileNode) * max_tn, &s1);
	la.tile_of = (int32_t*) scratch(c, 4, sizeof(int32_t) * max_tiles, &s1);
	la.tile_lt = (int32_t*) scratch(c, 5, sizeof(int32_t) * max_tiles, &s1);
	la.blk = (int4*) scratch(c, 6, sizeof(int4) * c->nsm, &s1);
	la.ctl = (LevelCtl*) scratch(c, 7, sizeof(LevelCtl), &s1);
	CT_TRY(s1);
	for (int d = 0; d < 3; d++) {
		la.x[d] = b->x[d];
	}
	la.flags = c->d_flags;
	la.off = b->d_sub_off;
	la.pb = pb;
	la.n = n;
	la.nroot = nroot;
	la.bucket = p->bucket;
	la.theta = p->theta;
	la.hsoft = p->hsoft;
	CT_CUDA(c, cudaMemsetAsync(c->d_flags, 0, 4 * sizeof(int), st));
	int32_t* h_tot = (int32_t*) c->pinned;
	LevelCtl* hc = (LevelCtl*) ((char*) c->pinned + 64);
	for (la.resume = 0;; la.resume = 1) {
		la.nodes = b->nodes;
		la.gbox = b->gbox;
		la.key = b->key;
		la.depth = b->depth;
		la.parent = b->parent;
		la.node_cap = b->node_cap;
		// (a resumed build keeps the level it stopped before)
		CT_CUDA(c, cudaMemsetAsync(la.ctl, 0, offsetof(LevelCtl, level), st));
		c->launches++;
		void* args[] = { (void*) &la };
		CT_CUDA(c, cudaLaunchCooperativeKernel((const void*) k_tree_levels, dim3(nblk), dim3(LTPB), args, 0, st));
		CT_CUDA(c, cudaMemcpyAsync(hc, la.ctl, sizeof(LevelCtl), cudaMemcpyDeviceToHost, st));
		CT_CUDA(c, cudaStreamSynchronize(st));
		if (hc->error) {
			return fail(c, CT_ERR_CUDA, "tree build: the blocks of the cooperative grid did not meet");
		}
		if (hc->status == 0) {
			break;
		}
		// the levels so far stay; the level that did not fit starts again with room for its children
		CT_TRY(ensure_nodes(c, b, hc->need));
	}
	std::vector<int64_t> levels(hc->start, hc->start + hc->level + 2);
	b->level_start = levels;  // level k = [levels[k], levels[k+1])
	b->nnodes = levels.back();
	const int32_t* perm = la.idx;
	// apply the permutation to velocities and rungs
	{
		ct_status s2 = CT_OK;
		float* t0 = (float*) scratch(c, 17, sizeof(float) * n, &s2);
		float* t1 = (float*) scratch(c, 18, sizeof(float) * n, &s2);
		float* t2 = (float*) scratch(c, 19, sizeof(float) * n, &s2);
		int8_t* tr = (int8_t*) scratch(c, 20, n + 16, &s2);
		CT_TRY(s2);
		CT_CUDA(c, cudaMemcpyAsync(t0 + pb, b->v[0] + pb, sizeof(float) * np, cudaMemcpyDeviceToDevice, st));
		CT_CUDA(c, cudaMemcpyAsync(t1 + pb, b->v[1] + pb, sizeof(float) * np, cudaMemcpyDeviceToDevice, st));
		CT_CUDA(c, cudaMemcpyAsync(t2 + pb, b->v[2] + pb, sizeof(float) * np, cudaMemcpyDeviceToDevice, st));
		CT_CUDA(c, cudaMemcpyAsync(tr + pb, b->rung + pb, np, cudaMemcpyDeviceToDevice, st));
		if (np > 0) {
			c->launches++;
			k_gather_particles<<<grid_for(c, np, 256), 256, 0, st>>>(pb, n, perm, t0, t1, t2, tr, b->v[0], b->v[1], b->v[2], b->rung);
		}
	}
	// upsweep, deepest level first
	for (int k = (int) levels.size() - 2; k >= 0; k--) {
		const int64_t a = levels[k], e = levels[k + 1];
		if (e > a) {
			c->launches++;
			k_upsweep<Ops><<<(int) std::min<int64_t>((e - a + UTPB / 32 - 1) / (UTPB / 32), (int64_t) c->nsm * 16), UTPB, 0, st>>>(a, e, b->nodes, b->nbox,
					b->multi, b->tbox, b->gbox,
					b->x[0], b->x[1], b->x[2], p->bucket);
		}
	}
	CT_CUDA(c, cudaGetLastError());
	CT_CUDA(c, cudaMemcpyAsync(h_tot, c->d_flags, 4 * sizeof(int), cudaMemcpyDeviceToHost, st));
	CT_CUDA(c, cudaStreamSynchronize(st));
	if (h_tot[2]) {
		return fail(c, CT_ERR_CAPACITY, "tree depth exceeded the maximum of 128 (coincident particles?)");
	}
	b->tparams = *p;
	b->tree_valid = true;
	return CT_OK;
}

}  // namespace

ct_status tree_build(Ctx* c, Box* b, const ct_tree_params* p) {
	if (c->order == 5) {
		return tree_build_t<Ops5>(c, b, p);
	}
	return tree_build_t<Ops7>(c, b, p);
}

}  // namespace ct
