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
#include "ct_partition.cuh"

namespace ct {
namespace {

// ---------------------------------------------------------------- the levels
// One cooperative launch builds every level: a resident grid whose blocks meet at grid barriers
// (1.2 us from the last arrival) between the phases of a level.  The launch is cooperative, for
// which CUDA guarantees that all blocks of the grid are resident together: a barrier waits for blocks
// that run, never for one without room, and that holds for each grid by itself, however many contexts
// build at a time and at whatever priority.  A barrier that has waited 30 s all the same ends the launch
// with an error.  What bounded the build before was the
// level's structure, not its data: twelve launches, two scans and a host round trip a level (16^3
// particles: 0.87 ms for 11 levels and 64 KB of positions; 10^6 clustered particles: 2.7 ms for 28
// levels).  By the number of nodes on the level:
//   few (at most 4 a block): a block partitions the nodes of its own share, by a warp up to WARP_FEW
//   particles and by the whole block up to BLOCK_LINE, which is quickest for one node.  A child is
//   counted by the block that makes it, so that the level takes one barrier.
//   many: a warp partitions up to WARP_FEW particles (WARP_MANY where there are two nodes a warp), and
//   warps take nodes from all shares, since the shares' work is uneven in a clustered box; the level
//   ends with two barriers (numbering, partition).
// Larger nodes go tile by tile over the whole grid: four barriers for a level with any (numbering,
// ballots, positions, swaps).  A level whose nodes were not counted as they were made (the first, and
// each behind a level of many nodes or of tiles) counts them itself, one barrier more.
constexpr int LTPB = 512;             // threads of a level block
constexpr int LWARPS = LTPB / 32;
constexpr int SUB = 1024;             // particles whose ballots a warp's lanes hold, one each
constexpr int BLOCK_SUB = 256;        // particles a warp takes of a node partitioned by its block
constexpr int BLOCK_LINE = BLOCK_SUB * LWARPS;
constexpr int WARP_FEW = SUB, WARP_MANY = 4 * SUB;
constexpr int NODE_SPLIT = 2;         // NodeW.flags besides bit 0 (leaf)
constexpr int TAKE = 4;               // nodes a warp takes at a time

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
	unsigned int take[2];  // nodes taken of an even and an odd level
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
	uint32_t* tile_mask;  // the tile nodes' ballots, 32 words a SUB (see mask_row)
	int4* blk;         // two levels' worth, per block: split nodes, tile nodes, tiles of a range of
	                   // consecutive nodes, and the range's first node
	LevelCtl* ctl;
	int* flags;
	const int64_t* off;
	int64_t pb, n, node_cap;
	int nroot, bucket, resume;
	int sub;        // particles a warp takes of a tile: SUB, or BLOCK_SUB while tiles of 16 SUB would
	                // leave blocks without one
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

// Row of the ballots of SUB s of tile node ti, which starts at particle pbeg: the tile nodes come in
// particle order, so rows counted by particles, one spare a node, do not meet.
__device__ __forceinline__ int64_t mask_row(const LevelArgs& a, int pbeg, int ti, int s) {
	return ((int64_t) pbeg - a.pb) / a.sub + ti + s;
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

// Leaf or split (tree.cpp:314-348): the flags of a node of box gb with nparts particles.
__device__ __forceinline__ int classify(const LevelArgs& a, const double* gb, int nparts, int level) {
	float box_r = 0.0f;
#pragma unroll
	for (int dim = 0; dim < 3; dim++) {
		const double h = 0.5 * (gb[3 + dim] - gb[dim]);
		box_r += h * h;
	}
	box_r = sqrtf(box_r);
	const bool ewald_satisfied = (box_r < 0.25 * (a.theta / (1.0 + a.theta)) && box_r < 0.125 - 0.25 * a.hsoft);
	if (!(nparts > a.bucket || (!ewald_satisfied && nparts > 0))) {
		return 1;
	}
	if (level >= MAX_DEPTH - 1) {
		atomicOr(a.flags + 2, 1);
		return 1;
	}
	return NODE_SPLIT;
}
// A level of many nodes, and the size above which its nodes go tile by tile.
__device__ __forceinline__ bool many_nodes(int64_t nl) {
	return nl > 4 * (int64_t) gridDim.x;
}
// (on a level of many nodes a warp takes the larger ones too once there are two nodes a warp)
__device__ __forceinline__ int warp_line_of(int64_t nl) {
	return nl > 2 * LWARPS * (int64_t) gridDim.x ? WARP_MANY : WARP_FEW;
}
__device__ __forceinline__ int tile_line(int64_t nl) {
	return many_nodes(nl) ? warp_line_of(nl) : BLOCK_LINE;
}
// What a node adds to its range's counts: split nodes, tile nodes, tiles.
__device__ __forceinline__ int3 counted(const LevelArgs& a, int flags, int nparts, int line) {
	const bool sp = flags & NODE_SPLIT, t = sp && nparts > line;
	const int tile = a.sub * LWARPS;
	return make_int3(sp, t, t ? (nparts + tile - 1) / tile : 0);
}

// The two children of node ni, split at particle `mid`, by the lanes of a warp; their counts (with the
// next level's tile line) are added to sum (shared memory).
__device__ __forceinline__ void make_children(const LevelArgs& a, int64_t ni, const NodeW& nd, int mid, int xd, double xm, int level, int lane, int line,
		int* sum) {
	const int64_t l = nd.child;
	double gb[6];
#pragma unroll
	for (int d = 0; d < 6; d++) {
		gb[d] = a.gbox[6 * ni + d];
	}
	const int side = lane & 1;
#pragma unroll
	for (int d = 0; d < 3; d++) {
		gb[3 + d] = side == 0 && d == xd ? xm : gb[3 + d];
		gb[d] = side == 1 && d == xd ? xm : gb[d];
	}
	if (lane < 2) {
		NodeW c;
		c.x = c.y = c.z = 0;
		c.radius = 0.f;
		c.child = -1;
		c.pbeg = lane == 0 ? nd.pbeg : mid;
		c.pend = lane == 0 ? mid : nd.pend;
		c.flags = classify(a, gb, c.pend - c.pbeg, level + 1);
		a.nodes[l + lane] = c;
		a.key[l + lane] = (a.key[ni] << 1) + lane;
		a.depth[l + lane] = level + 1;
		a.parent[l + lane] = (int32_t) ni;
#pragma unroll
		for (int d = 0; d < 6; d++) {
			a.gbox[6 * (l + lane) + d] = gb[d];
		}
		const int3 k = counted(a, c.flags, c.pend - c.pbeg, line);
		if (k.x) {
			atomicAdd(sum, k.x);
		}
		if (k.y) {
			atomicAdd(sum + 1, k.y);
			atomicAdd(sum + 2, k.z);
		}
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

// Ballots of up to SUB particles from xp on: lane c's has bit j set when particle 32 c + j lies below
// the midpoint.
__device__ __forceinline__ unsigned sub_below(const uint32_t* xp, int n, uint32_t xm, int lane) {
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
	return mine;
}
// The partition of a node of at most WARP_MANY particles by one warp.  With m particles below the
// midpoint, the k-th particle at or above it in the first m (from the left) changes places with the
// k-th below it in the rest (from the right), which is the reference's two-pointer loop.  pos: SUB
// offsets in shared memory; longer swaps go through the global scratch.
__device__ __forceinline__ int warp_partition(const LevelArgs& a, const NodeW& nd, const uint32_t* xd, uint32_t xm, uint16_t* pos, int lane) {
	constexpr int NS = WARP_MANY / SUB;
	const int n = nd.pend - nd.pbeg;
	unsigned mine[NS];
	int m = 0;
#pragma unroll
	for (int q = 0; q < NS; q++) {
		mine[q] = SUB * q < n ? sub_below(xd + nd.pbeg + SUB * q, min(SUB, n - SUB * q), xm, lane) : 0u;
		m += __popc(mine[q]);
	}
	m = __reduce_add_sync(0xffffffffu, m);
	int ns = 0;
#pragma unroll
	for (int q = 0; q < NS; q++) {
		ns += __popc(mine[q] & ~first_bits(m - SUB * q, 32 * lane));
	}
	ns = __reduce_add_sync(0xffffffffu, ns);
	if (ns == 0) {
		return m;
	}
	const bool few = ns <= SUB / 2;
	uint16_t* pl = pos;
	uint16_t* pr = pos + SUB / 2;
	int lt = 0;  // below the midpoint in earlier SUBs
#pragma unroll
	for (int q = 0; q < NS; q++) {
		if (SUB * q < n) {
			const int here = __reduce_add_sync(0xffffffffu, __popc(mine[q]));
			const int l0 = SUB * q - lt, r0 = m - lt - here;
			sub_wrong(mine[q], min(SUB, n - SUB * q), max(0, min(SUB, m - SUB * q)), lane,
					[&](int k, int o) {
						if (few) {
							pl[l0 + k] = (uint16_t) (SUB * q + o);
						} else {
							a.posL[nd.pbeg + l0 + k] = SUB * q + o;
						}
					},
					[&](int k, int o) {
						if (few) {
							pr[r0 + k] = (uint16_t) (SUB * q + o);
						} else {
							a.posR[nd.pbeg + r0 + k] = SUB * q + o;
						}
					});
			lt += here;
		}
	}
	__syncwarp();
	for (int q = lane; q < ns; q += 32) {
		swap_particles(a, nd.pbeg + (few ? pl[q] : a.posL[nd.pbeg + q]), nd.pbeg + (few ? pr[q] : a.posR[nd.pbeg + q]));
	}
	__syncwarp();
	return m;
}

// Shared memory of a level block.
struct LevelShared {
	uint16_t pos[LWARPS][SUB];
	int scan[3][LWARPS];
	int sum[LWARPS];
	int totals[7][LWARPS];
	unsigned mask[LWARPS];
	int tot[3];
	int next, ns;
};

// Block sums of three values (all threads get them).
__device__ __forceinline__ int3 block_total3(int x, int y, int z, int (*s)[LWARPS], int lane, int w) {
	x = __reduce_add_sync(0xffffffffu, x);
	y = __reduce_add_sync(0xffffffffu, y);
	z = __reduce_add_sync(0xffffffffu, z);
	__syncthreads();
	if (lane == 0) {
		s[0][w] = x;
		s[1][w] = y;
		s[2][w] = z;
	}
	__syncthreads();
	int3 t = make_int3(0, 0, 0);
#pragma unroll
	for (int i = 0; i < LWARPS; i++) {
		t.x += s[0][i];
		t.y += s[1][i];
		t.z += s[2][i];
	}
	return t;
}

// Positions of a tile's particles on the wrong side of the split point, by the block: warp w has the
// ballots of its w-th sub particles, with lt_prev particles of the node below the midpoint in earlier tiles.  Before the
// split point they are ranked from the node's left, after it from its right.  The warp that holds the
// split point puts the node's number of swaps in *ns.
__device__ __forceinline__ void tile_positions(const LevelArgs& a, LevelShared& sh, unsigned mine, int pbeg, int pend, int tb, int sub, int m, int lt_prev, int* ns, int lane,
		int w) {
	const int here = __reduce_add_sync(0xffffffffu, __popc(mine));
	__syncthreads();
	if (lane == 0) {
		sh.sum[w] = here;
	}
	__syncthreads();
	int lt = lt_prev;
	for (int i = 0; i < w; i++) {
		lt += sh.sum[i];
	}
	const int sb = tb + sub * w, n = min(sub, pend - sb);
	if (n > 0) {
		const int sp = pbeg + m, before = max(0, min(n, sp - sb));
		const int l0 = pbeg + (sb - pbeg) - lt, after = m - lt - here, r0 = pbeg + after;
		sub_wrong(mine, n, before, lane, [&](int k, int o) { a.posL[l0 + k] = sb + o; }, [&](int k, int o) { a.posR[r0 + k] = sb + o; });
		// (the last warp, when nothing lies after the split point)
		if ((sb <= sp && sp < sb + n) || (sp == pend && sb + n == pend)) {
			const int right = __reduce_add_sync(0xffffffffu, __popc(mine & ~first_bits(before, 32 * lane)));
			if (lane == 0) {
				*ns = after + right;
			}
		}
	}
}

__global__ void __launch_bounds__(LTPB, 2) k_tree_levels(const LevelArgs a) {
	__shared__ LevelShared sh;
	const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
	const unsigned lt_lane = (1u << lane) - 1u;
	const int nblk = gridDim.x;
	LevelCtl* ctl = a.ctl;
	unsigned int round = 0;
	int level = 0;
	int64_t lb = 0, le = a.nroot;
	if (a.resume) {
		level = ctl->level;
		lb = ctl->lb;
		le = ctl->le;
	} else {
		const int64_t gt = blockIdx.x * (int64_t) LTPB + tid, gs = nblk * (int64_t) LTPB;
		for (int64_t i = gt; i < a.n; i += gs) {
			a.idx[i] = (int32_t) i;
		}
		// one root per box: node s covers the unit box and particles [off[s], off[s+1]), except that
		// a single box starts at the active range
		for (int64_t s = gt; s < a.nroot; s += gs) {
			const double gb[6] = { 0.0, 0.0, 0.0, 1.0, 1.0, 1.0 };
			NodeW r;
			r.x = r.y = r.z = 0;
			r.radius = 0.f;
			r.pbeg = a.nroot == 1 ? (int32_t) a.pb : (int32_t) a.off[s];
			r.pend = a.nroot == 1 ? (int32_t) a.n : (int32_t) a.off[s + 1];
			r.child = -1;
			r.flags = classify(a, gb, r.pend - r.pbeg, 0);
			a.nodes[s] = r;
			for (int d = 0; d < 6; d++) {
				a.gbox[6 * s + d] = gb[d];
			}
			a.key[s] = 1;
			a.depth[s] = 0;
			a.parent[s] = -1;
		}
		if (!grid_meet(ctl, round)) {
			return;
		}
	}
	bool counts = false;  // the blocks' counts of this level's nodes are there
	for (;; level++) {
		const int64_t nl = le - lb;
		const int64_t share = (nl + nblk - 1) / nblk;  // consecutive nodes of a block
		const int64_t cb = lb + min(nl, share * blockIdx.x), ce = lb + min(nl, share * (blockIdx.x + 1));
		const bool many = many_nodes(nl);
		const int line = tile_line(nl), warp_line = warp_line_of(nl);
		int4* blk = a.blk + (level & 1) * nblk;
		int4* blk_next = a.blk + ((level + 1) & 1) * nblk;
		if (!counts) {
			int k0 = 0, k1 = 0, k2 = 0;
			for (int64_t ni = cb + tid; ni < ce; ni += LTPB) {
				const NodeW nd = a.nodes[ni];
				const int3 k = counted(a, nd.flags, nd.pend - nd.pbeg, line);
				k0 += k.x;
				k1 += k.y;
				k2 += k.z;
			}
			const int3 t = block_total3(k0, k1, k2, sh.scan, lane, w);
			if (tid == 0) {
				blk[blockIdx.x] = make_int4(t.x, t.y, t.z, (int) cb);
			}
			if (!grid_meet(ctl, round)) {
				return;
			}
		}
		// ---- totals of the level and of the nodes before this block's share: the ranges before it,
		// and the part of the range the share begins in (nblk is at most the block's threads)
		int base[3] = { 0, 0, 0 }, tot[3] = { 0, 0, 0 };
		int part = 0x7fffffff;  // first node of the range that holds cb
		{
			int4 t = make_int4(0, 0, 0, 0x7fffffff);
			int end = 0x7fffffff;
			if (tid < nblk) {
				t = __ldcg(blk + tid);
				end = tid + 1 < nblk ? __ldcg(&blk[tid + 1].w) : (int) le;
			}
			const bool prev = end <= (int) cb;
			int v[7] = { t.x, t.y, t.z, prev ? t.x : 0, prev ? t.y : 0, prev ? t.z : 0, t.w < (int) cb && end > (int) cb ? t.w : 0x7fffffff };
			const int nw = (nblk + 31) / 32;
			if (w < nw) {
#pragma unroll
				for (int q = 0; q < 7; q++) {
					v[q] = q < 6 ? __reduce_add_sync(0xffffffffu, v[q]) : __reduce_min_sync(0xffffffffu, v[q]);
				}
			}
			__syncthreads();
			if (lane == 0 && w < nw) {
#pragma unroll
				for (int q = 0; q < 7; q++) {
					sh.totals[q][w] = v[q];
				}
			}
			__syncthreads();
			for (int i = 0; i < nw; i++) {
#pragma unroll
				for (int q = 0; q < 3; q++) {
					tot[q] += sh.totals[q][i];
					base[q] += sh.totals[3 + q][i];
				}
				part = min(part, sh.totals[6][i]);
			}
		}
		if (part < (int) cb) {
			int k0 = 0, k1 = 0, k2 = 0;
			for (int ni = part + tid; ni < (int) cb; ni += LTPB) {
				const NodeW nd = a.nodes[ni];
				const int3 k = counted(a, nd.flags, nd.pend - nd.pbeg, line);
				k0 += k.x;
				k1 += k.y;
				k2 += k.z;
			}
			const int3 t = block_total3(k0, k1, k2, sh.scan, lane, w);
			base[0] += t.x;
			base[1] += t.y;
			base[2] += t.z;
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
			ctl->take[(level + 1) & 1] = 0;  // (the last level's takers are done)
		}
		if (tot[0] == 0) {
			break;
		}
		const int first_child = (int) le + 2 * base[0];
		const int next_line = tile_line(2 * (int64_t) tot[0]);
		__syncthreads();
		if (tid < 3) {
			sh.tot[tid] = 0;
		}
		// one node by this warp
		auto by_warp = [&](int64_t ni) {
			const NodeW nd = a.nodes[ni];
			if (nd.child < 0 || nd.pend - nd.pbeg > warp_line) {
				return;
			}
			double xm;
			const int xd = split_dim(a.gbox + 6 * ni, xm);
			const int m = warp_partition(a, nd, xd == 0 ? a.x[0] : xd == 1 ? a.x[1] : a.x[2], fixed_from_double(xm), sh.pos[w], lane);
			make_children(a, ni, nd, nd.pbeg + m, xd, xm, level, lane, next_line, sh.tot);
		};
		// ---- LTPB nodes at a time: children numbered in node order, then (few nodes) the partitions
		for (int64_t n0 = cb; n0 < ce; n0 += LTPB) {
			const int64_t ni = n0 + tid;
			int f = 1, nparts = 0;
			if (ni < ce) {
				const NodeW nd = a.nodes[ni];
				f = nd.flags;
				nparts = nd.pend - nd.pbeg;
			}
			const int3 k = counted(a, f, nparts, line);
			const int inc = lane_scan(k.z, lane);
			const unsigned ms = __ballot_sync(0xffffffffu, k.x), mt = __ballot_sync(0xffffffffu, k.y);
			const unsigned mb = __ballot_sync(0xffffffffu, k.x && !k.y && nparts > warp_line);
			__syncthreads();
			if (lane == 31) {
				sh.scan[0][w] = __popc(ms);
				sh.scan[1][w] = __popc(mt);
				sh.scan[2][w] = inc;
				sh.mask[w] = mb;
			}
			if (tid == 0) {
				sh.next = 0;
			}
			__syncthreads();
			int e0 = base[0], e1 = base[1], e2 = base[2];
			for (int i = 0; i < LWARPS; i++) {
				const int q0 = sh.scan[0][i], q1 = sh.scan[1][i], q2 = sh.scan[2][i];
				e0 += i < w ? q0 : 0;
				e1 += i < w ? q1 : 0;
				e2 += i < w ? q2 : 0;
				base[0] += q0;
				base[1] += q1;
				base[2] += q2;
			}
			if (k.x) {
				// (the flags stay: another block may still be counting up to its share)
				a.nodes[ni].child = (int32_t) (le + 2 * (int64_t) (e0 + __popc(ms & lt_lane)));
			}
			if (k.y) {
				TileNode t;
				t.node = (int32_t) ni;
				t.t0 = e2 + inc - k.z;
				t.nt = k.z;
				t.m = t.nswap = 0;
				a.tnode[e1 + __popc(mt & lt_lane)] = t;
			}
			for (unsigned q = mt; q; q &= q - 1) {
				const int src = __ffs(q) - 1;
				const int t0 = __shfl_sync(0xffffffffu, e2 + inc - k.z, src), nt = __shfl_sync(0xffffffffu, k.z, src);
				for (int i = lane; i < nt; i += 32) {
					a.tile_of[t0 + i] = e1 + __popc(mt & ((1u << src) - 1u));
				}
			}
			if (many) {
				continue;
			}
			__syncthreads();
			// nodes of at most BLOCK_LINE particles, one after the other by the block
			for (int i = 0; i < LWARPS; i++) {
				for (unsigned q = sh.mask[i]; q; q &= q - 1) {
					const int64_t bi = n0 + 32 * i + __ffs(q) - 1;
					const NodeW nd = a.nodes[bi];
					double xm;
					const int xd = split_dim(a.gbox + 6 * bi, xm);
					const uint32_t* x = xd == 0 ? a.x[0] : xd == 1 ? a.x[1] : a.x[2];
					const int sb = nd.pbeg + BLOCK_SUB * w;
					const unsigned mine = sb < nd.pend ? sub_below(x + sb, min(BLOCK_SUB, nd.pend - sb), fixed_from_double(xm), lane) : 0u;
					const int m = block_total3(__popc(mine), 0, 0, sh.scan, lane, w).x;
					tile_positions(a, sh, mine, nd.pbeg, nd.pend, nd.pbeg, BLOCK_SUB, m, 0, &sh.ns, lane, w);
					__syncthreads();
					const int ns = sh.ns;
					for (int p = tid; p < ns; p += LTPB) {
						swap_particles(a, a.posL[nd.pbeg + p], a.posR[nd.pbeg + p]);
					}
					if (w == 0) {
						make_children(a, bi, nd, nd.pbeg + m, xd, xm, level, lane, next_line, sh.tot);
					}
				}
			}
			// the others: a warp each, taken from the block's
			const int have = (int) min((int64_t) LTPB, ce - n0);
			for (;;) {
				int j = 0;
				if (lane == 0) {
					j = atomicAdd(&sh.next, 1);
				}
				j = __shfl_sync(0xffffffffu, j, 0);
				if (j >= have) {
					break;
				}
				by_warp(n0 + j);
			}
		}
		counts = !many && tot[2] == 0;
		if (counts) {
			// the children this block made are consecutive: their counts are the next level's
			__syncthreads();
			if (tid == 0) {
				blk_next[blockIdx.x] = make_int4(sh.tot[0], sh.tot[1], sh.tot[2], first_child);
			}
		} else {
			if (!grid_meet(ctl, round)) {
				return;
			}
			// ---- larger nodes, tile by tile: ballots and counts of the particles below the midpoint
			for (int t = blockIdx.x; t < tot[2]; t += nblk) {
				const int ti = a.tile_of[t];
				const TileNode tn = a.tnode[ti];
				const int2 pr = *reinterpret_cast<const int2*>(&a.nodes[tn.node].pbeg);
				double xm;
				const int xd = split_dim(a.gbox + 6 * (int64_t) tn.node, xm);
				const uint32_t* x = xd == 0 ? a.x[0] : xd == 1 ? a.x[1] : a.x[2];
				const int sb = pr.x + ((t - tn.t0) * LWARPS + w) * a.sub;
				const unsigned mine = sb < pr.y ? sub_below(x + sb, min(a.sub, pr.y - sb), fixed_from_double(xm), lane) : 0u;
				if (sb < pr.y) {
					a.tile_mask[32 * mask_row(a, pr.x, ti, (t - tn.t0) * LWARPS + w) + lane] = mine;
				}
				const int c = block_total3(__popc(mine), 0, 0, sh.scan, lane, w).x;
				if (tid == 0) {
					a.tile_lt[t] = c;
				}
			}
			if (many) {
				for (;;) {
					unsigned int j = 0;
					if (lane == 0) {
						j = atomicAdd(&ctl->take[level & 1], (unsigned int) TAKE);
					}
					j = __shfl_sync(0xffffffffu, j, 0);
					if ((int64_t) j >= nl) {
						break;
					}
					for (int64_t q = j; q < min(nl, (int64_t) j + TAKE); q++) {
						by_warp(lb + q);
					}
				}
			}
			if (tot[2] > 0) {
				if (!grid_meet(ctl, round)) {
					return;
				}
				// positions of the particles on the wrong side of the split point.  Earlier tiles hold only
				// particles before a particle on the left, later ones only particles after one on the right,
				// so the counts below the midpoint of whole tiles give both ranks.
				for (int t = blockIdx.x; t < tot[2]; t += nblk) {
					const int ti = a.tile_of[t];
					const TileNode tn = a.tnode[ti];
					const int2 pr = *reinterpret_cast<const int2*>(&a.nodes[tn.node].pbeg);
					const int sub = (t - tn.t0) * LWARPS + w;
					const unsigned mine = pr.x + a.sub * sub < pr.y ? __ldcg(a.tile_mask + 32 * mask_row(a, pr.x, ti, sub) + lane) : 0u;
					int all = 0, prev = 0;
					for (int q = tid; q < tn.nt; q += LTPB) {
						const int c = __ldcg(a.tile_lt + tn.t0 + q);
						all += c;
						prev += q < t - tn.t0 ? c : 0;
					}
					const int3 s = block_total3(all, prev, 0, sh.scan, lane, w);
					tile_positions(a, sh, mine, pr.x, pr.y, pr.x + (t - tn.t0) * LWARPS * a.sub, a.sub, s.x, s.y, &a.tnode[ti].nswap, lane, w);
					if (tid == 0 && t == tn.t0) {
						a.tnode[ti].m = s.x;
					}
				}
				if (!grid_meet(ctl, round)) {
					return;
				}
				for (int t = blockIdx.x; t < tot[2]; t += nblk) {
					const TileNode* tp = a.tnode + a.tile_of[t];
					const int node = tp->node, t0 = tp->t0;
					const int m = __ldcg(&tp->m), ns = __ldcg(&tp->nswap);
					const int pbeg = a.nodes[node].pbeg, tile = a.sub * LWARPS;
					for (int k = (t - t0) * tile + tid; k < min(ns, (t - t0 + 1) * tile); k += LTPB) {
						swap_particles(a, __ldcg(a.posL + pbeg + k), __ldcg(a.posR + pbeg + k));
					}
					if (t == t0 && w == 0) {
						double xm;
						const int xd = split_dim(a.gbox + 6 * (int64_t) node, xm);
						make_children(a, node, a.nodes[node], pbeg + m, xd, xm, level, lane, next_line, sh.tot);
					}
				}
			}
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

// The velocities and rungs of the active particles set aside for the gather: one launch, where four copies
// took 2-3 us each on a small box (16^3 step 2 to 3% shorter with the gather launched behind it).
__global__ void k_stage_particles(int64_t b, int64_t n, const float* v0, const float* v1, const float* v2, const int8_t* r, float* o0, float* o1, float* o2,
		int8_t* orr) {
	for (int64_t i = b + blockIdx.x * (int64_t) blockDim.x + threadIdx.x; i < n; i += (int64_t) gridDim.x * blockDim.x) {
		const float a0 = v0[i], a1 = v1[i], a2 = v2[i];
		const int8_t ar = r[i];
		o0[i] = a0;
		o1[i] = a1;
		o2[i] = a2;
		orr[i] = ar;
	}
}

__global__ void k_gather_particles(int64_t b, int64_t n, const int32_t* idx, const float* v0, const float* v1, const float* v2, const int8_t* r,
		float* o0, float* o1, float* o2, int8_t* orr) {
	front_done();
	for (int64_t i = b + blockIdx.x * (int64_t) blockDim.x + threadIdx.x; i < n; i += (int64_t) gridDim.x * blockDim.x) {
		const int j = idx[i];
		o0[i] = v0[j];
		o1[i] = v1[j];
		o2[i] = v2[j];
		orr[i] = r[j];
	}
}

// One of the fields alone, its values set aside in src.
template<class T>
__global__ void k_gather_field(int64_t b, int64_t n, const int32_t* idx, const T* src, T* out) {
	for (int64_t i = b + blockIdx.x * (int64_t) blockDim.x + threadIdx.x; i < n; i += (int64_t) gridDim.x * blockDim.x) {
		out[i] = src[idx[i]];
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
constexpr int UTPB = 128;

// Sums of N doubles per lane over the warp: afterwards lane l has the sums of entries k with
// k % 32 == l in out[k / 32].  Halves of the entries change places at each step, so that the warp
// moves N values instead of 5 N; the pairs added are those of a butterfly over lane distances
// 16, 8, 4, 2, 1.
template<int N, int O>
struct WarpScatterSum {
	static constexpr int HALF = (N + 1) / 2;
	static __device__ __forceinline__ void run(double* v, int lane) {
		const bool hi = lane & O;
		double w[HALF];
#pragma unroll
		for (int i = 0; i < HALF; i++) {
			const double up = HALF + i < N ? v[HALF + i] : 0.0;
			w[i] = (hi ? up : v[i]) + __shfl_xor_sync(0xffffffffu, hi ? v[i] : up, O);
		}
#pragma unroll
		for (int i = 0; i < HALF; i++) {
			v[i] = w[i];
		}
		if constexpr (O > 1) {
			WarpScatterSum<HALF, O / 2>::run(v, lane);
		}
	}
	// entry that slot `i` of a lane holds after the steps from distance O down
	static __device__ __forceinline__ int entry(int i, int lane) {
		int k = i;
		if constexpr (O > 1) {
			k = WarpScatterSum<HALF, O / 2>::entry(i, lane);
		}
		return k >= HALF || k < 0 ? -1 : ((lane & O) ? (HALF + k < N ? HALF + k : -1) : k);
	}
	static constexpr int slots() {
		if constexpr (O > 1) {
			return WarpScatterSum<HALF, O / 2>::slots();
		} else {
			return HALF;
		}
	}
};

// All leaves of the tree, a warp each (tree.cpp:498-571): tight box, centre, radius and the
// particles' multipole, summed in double.  The leaves need nothing of one another, so they run in one
// launch and not level by level; the warp's 37 sums are scattered over its lanes instead of made by
// every lane (370 shuffles before).
template<class Ops>
__global__ void __launch_bounds__(UTPB) k_leaf_moments(int64_t nn, NodeW* nodes, int32_t* nbox, float* multi, double* tbox, const double* gbox, const uint32_t* x0,
		const uint32_t* x1, const uint32_t* x2) {
	front_done();
	constexpr int NM = Ops::NMULT;
	using Sum = WarpScatterSum<NM, 16>;
	const uint32_t* xs[3] = { x0, x1, x2 };
	const int lane = threadIdx.x & 31;
	const int64_t gw = (blockIdx.x * (int64_t) blockDim.x + threadIdx.x) >> 5;
	const int64_t nw = ((int64_t) gridDim.x * blockDim.x) >> 5;
	for (int64_t ni = gw; ni < nn; ni += nw) {
		const NodeW nd = nodes[ni];
		if (nd.child >= 0) {
			continue;
		}
		const double* gb = gbox + 6 * ni;
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
#pragma unroll
		for (int k = 0; k < NM; k++) {
			M[k] = 0.0;
		}
		for (int p = nd.pbeg + lane; p < nd.pend; p += 32) {
			float m[NM];
			Ops::p2m(m, fixed_dist(x0[p], Y[0]), fixed_dist(x1[p], Y[1]), fixed_dist(x2[p], Y[2]));
#pragma unroll
			for (int k = 0; k < NM; k++) {
				M[k] += (double) m[k];
			}
		}
		Sum::run(M, lane);
		if (lane == 0) {
			NodeW o = nd;
			o.x = Y[0];
			o.y = Y[1];
			o.z = Y[2];
			o.radius = (float) sqrt(r);
			nodes[ni] = o;
		}
		if (lane < 3) {
			const double lo = lane == 0 ? mn[0] : lane == 1 ? mn[1] : mn[2], hi = lane == 0 ? mx[0] : lane == 1 ? mx[1] : mx[2];
			tbox[6 * ni + lane] = lo;
			tbox[6 * ni + 3 + lane] = hi;
			nbox[6 * ni + lane] = range_fixed_from_double(lo);
			nbox[6 * ni + 3 + lane] = range_fixed_from_double(hi);
		}
#pragma unroll
		for (int i = 0; i < Sum::slots(); i++) {
			const int k = Sum::entry(i, lane);
			if (k >= 0) {
				multi[NMULT_STRIDE * ni + k] = (float) M[i];
			}
		}
	}
}

// Component k of a stored multipole of orders < Q belongs to part 0..3 by the parities of its exponents:
// the projection of a shifted multipole onto its traceless part mixes components of equal parities only,
// so that a warp evaluating one part needs a quarter of the operator.
template<int Q>
__host__ __device__ constexpr int m2m_part(int k) {
	if (k == Q * Q) {
		return 3;  // (0, 0, 2)
	}
	const int c = k >= Q * (Q + 1) / 2;
	int r = c ? k - Q * (Q + 1) / 2 : k, s = 0;
	while (r >= s + 1) {
		r -= s + 1;
		s++;
	}
	const int a = (s - r) & 1, b = r & 1;  // (l, m, n) = (s - r, r, c)
	return a == b && b == c ? 3 : a + b + c == 1 ? (a ? 0 : b ? 1 : 2) : (!a ? 0 : !b ? 1 : 2);
}
// One part of the shift of a child's multipole to the centre of its parent: lanes 2 i and 2 i + 1 take
// the left and right child of a node, and the left one's stores the sum.
template<class Ops, int PART>
__device__ __forceinline__ void m2m_store(float* out, const float* Ma_, double x, double y, double z, bool on, bool left) {
	constexpr int NM = Ops::NMULT, Q = Ops::ORDER - 1;
	// the operator's other outputs are never formed (the compiler drops what nothing reads)
	double Mo[NM];
#pragma unroll
	for (int k = 0; k < NM; k++) {
		Mo[k] = 0.0;
	}
	if (on) {
		double Ma[NM];
#pragma unroll
		for (int k = 0; k < NM; k++) {
			Ma[k] = (double) Ma_[k];
		}
		Ops::m2m(Mo, Ma, x, y, z);
	}
	static_for<0, NM>([&](auto c) {
		constexpr int k = decltype(c)::value;
		if constexpr (m2m_part<Q>(k) == PART) {
			const double right = __shfl_down_sync(0xffffffffu, Mo[k], 1);
			if (on && left) {
				out[k] = (float) (Mo[k] + right);
			}
		}
	});
}

constexpr int UPS_TPB = 256;
constexpr int UPS_NODES = 32;    // nodes of a block, at most
constexpr int UPS_ALONE = 256;   // particles that one warp goes through by itself

// The interior nodes of one level (tree.cpp:351-497): union of the children's tight boxes, expansion
// centre and radius, M2M of the two children in double.  A block takes `group` nodes: a thread each
// for the boxes and centres, a warp each for the pass over the particles (or all eight, where a node
// has more than UPS_ALONE), and for the shifts 32 lanes for 16 nodes' 32 children, in four warps of a
// part of the components each.  With a warp a node, two of whose lanes shifted, levels of many nodes
// were bound by the issue of double operations (430 us at 33,000 nodes) and a large node's pass by 256
// dependent reads.  All levels, order 7: 256^3 particles 2,275 us -> 1,580; 64 boxes of 64^3 930 -> 610; a
// 64^3 box's upper rungs 575 -> 230; 16^3 81 -> 77 (5 to 8 us a level: one chain of reads, roots and the shift).
// Two blocks an SM bound it to 128 registers, at which order 7 spills 52 bytes; one block without spills
// took 0.85 ms more of the build of 256^3 particles.
template<class Ops>
__global__ void __launch_bounds__(UPS_TPB, 2) k_upsweep(int64_t lb, int64_t le, int group, NodeW* nodes, int32_t* nbox, float* multi, double* tbox, const double* gbox,
		const uint32_t* x0, const uint32_t* x1, const uint32_t* x2, int bucket) {
	__shared__ uint32_t s_xc[UPS_NODES][3];
	__shared__ int s_beg[UPS_NODES], s_end[UPS_NODES];  // particles to go through
	__shared__ unsigned int s_r2[UPS_NODES];            // largest squared distance (a positive float orders like its bits)
	__shared__ int s_child[UPS_NODES];
	__shared__ double s_X[UPS_NODES][3];
	front_done();
	const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
	const int64_t ngroups = (le - lb + group - 1) / group;
	for (int64_t gi = blockIdx.x; gi < ngroups; gi += gridDim.x) {
		const int64_t first = lb + gi * group;
		const int cnt = (int) (le - first < group ? le - first : group);
		const int64_t ni = first + threadIdx.x;  // the node of threads 0 .. cnt - 1
		const bool own = (int) threadIdx.x < cnt;
		NodeW nd, nl, nr;
		float ml0 = 0.f, mr0 = 0.f;
		double bb[3], be[3], Xc1[3];
		bool inner = false, tried1 = false;
		__syncthreads();
		if (own) {
			nd = nodes[ni];
			inner = nd.child >= 0;
			if (inner) {
				const int64_t L = nd.child, R = nd.child + 1;
				nl = nodes[L];
				nr = nodes[R];
				ml0 = multi[NMULT_STRIDE * L];
				mr0 = multi[NMULT_STRIDE * R];
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
				const double* gb = gbox + 6 * ni;
				double max_span = -1.0, extent = 0.0;
				for (int d = 0; d < 3; d++) {
					const double span = gb[3 + d] - gb[d];
					if (span > max_span) {
						max_span = span;
						extent = be[d] - bb[d];
					}
				}
				tried1 = nd.pend - nd.pbeg <= 64 * bucket && extent <= 0.5;
				for (int d = 0; d < 3; d++) {
					Xc1[d] = 0.5 * (bb[d] + be[d]);
					s_xc[threadIdx.x][d] = fixed_from_double(Xc1[d]);
				}
			}
			s_child[threadIdx.x] = inner ? nd.child : -1;
			s_beg[threadIdx.x] = tried1 ? nd.pbeg : 0;
			s_end[threadIdx.x] = tried1 ? nd.pend : 0;
			s_r2[threadIdx.x] = 0u;
		}
		__syncthreads();
		for (int i = 0; i < cnt; i++) {
			const int pb = s_beg[i], pe = s_end[i];
			const bool alone = pe - pb <= UPS_ALONE;
			if (pe == pb || (alone && (i & 7) != w)) {
				continue;
			}
			const uint32_t cx = s_xc[i][0], cy = s_xc[i][1], cz = s_xc[i][2];
			float r2max = 0.0f;
#pragma unroll 4
			for (int p = pb + (alone ? lane : (int) threadIdx.x); p < pe; p += alone ? 32 : UPS_TPB) {
				const float dx = fixed_dist(x0[p], cx);
				const float dy = fixed_dist(x1[p], cy);
				const float dz = fixed_dist(x2[p], cz);
				const float r2 = dx * dx + dy * dy + dz * dz;
				r2max = fmaxf(r2max, r2);
			}
			r2max = warp_max(r2max);
			if (lane == 0) {
				atomicMax(s_r2 + i, __float_as_uint(r2max));
			}
		}
		__syncthreads();
		if (inner) {
			const double Xl[3] = { fixed_to_double(nl.x), fixed_to_double(nl.y), fixed_to_double(nl.z) };
			const double Xr[3] = { fixed_to_double(nr.x), fixed_to_double(nr.y), fixed_to_double(nr.z) };
			const double radius1 = tried1 ? (double) sqrtf(__uint_as_float(s_r2[threadIdx.x])) : 0.0;
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
			const bool use1 = tried1 && radius1 < radius2;
			double Xc[3];
			float radius = (float) (use1 ? radius1 : radius2);
			for (int d = 0; d < 3; d++) {
				Xc[d] = use1 ? Xc1[d] : Xc2[d];
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
			NodeW o = nd;
			o.x = fixed_from_double(Xc[0]);
			o.y = fixed_from_double(Xc[1]);
			o.z = fixed_from_double(Xc[2]);
			o.radius = radius;
			nodes[ni] = o;
			for (int d = 0; d < 3; d++) {
				s_X[threadIdx.x][d] = Xc[d];
				tbox[6 * ni + d] = bb[d];
				tbox[6 * ni + 3 + d] = be[d];
				nbox[6 * ni + d] = range_fixed_from_double(bb[d]);
				nbox[6 * ni + 3 + d] = range_fixed_from_double(be[d]);
			}
		}
		__syncthreads();
		// M2M of both children in double (tree.cpp:481-494), left + right
		const int i = 16 * (w >> 2) + (lane >> 1);
		if (16 * (w >> 2) < cnt) {
			const int child = i < cnt ? s_child[i] : -1;
			const bool on = child >= 0, left = !(lane & 1);
			const int64_t c = on ? child + (lane & 1) : 0;
			double x = 0.0, y = 0.0, z = 0.0;
			if (on) {
				const NodeW cn = nodes[c];
				x = fixed_to_double(cn.x) - s_X[i][0];
				y = fixed_to_double(cn.y) - s_X[i][1];
				z = fixed_to_double(cn.z) - s_X[i][2];
			}
			const float* Ma = multi + NMULT_STRIDE * c;
			float* out = multi + NMULT_STRIDE * (first + i);
			switch (w & 3) {
			case 0:
				m2m_store<Ops, 0>(out, Ma, x, y, z, on, left);
				break;
			case 1:
				m2m_store<Ops, 1>(out, Ma, x, y, z, on, left);
				break;
			case 2:
				m2m_store<Ops, 2>(out, Ma, x, y, z, on, left);
				break;
			default:
				m2m_store<Ops, 3>(out, Ma, x, y, z, on, left);
			}
		}
	}
}

// The node arrays in the order of Box::node_have, with their elements a node.
template<class F>
ct_status each_node_array(Box* b, F f) {
	CT_TRY(f(&b->nodes, b->node_have[0], 1, "tree nodes"));
	CT_TRY(f(&b->nbox, b->node_have[1], 6, "node boxes"));
	CT_TRY(f(&b->multi, b->node_have[2], NMULT_STRIDE, "multipoles"));
	CT_TRY(f(&b->key, b->node_have[3], 1, "node keys"));
	CT_TRY(f(&b->depth, b->node_have[4], 1, "node depth"));
	CT_TRY(f(&b->parent, b->node_have[5], 1, "node parent"));
	CT_TRY(f(&b->gbox, b->node_have[6], 6, "node geometric box"));
	return f(&b->tbox, b->node_have[7], 6, "node tight box");
}

template<class T>
ct_status grow(Ctx* c, T** p, int64_t& have, int64_t need, int per, const char* what) {
	if (need <= have) {
		return CT_OK;
	}
	T* q = nullptr;
	CT_TRY(dalloc(c, (void**) &q, sizeof(T) * per * need, what));
	if (*p) {
		CT_CUDA(c, cudaMemcpyAsync(q, *p, sizeof(T) * per * have, cudaMemcpyDeviceToDevice, c->stream));
		CT_CUDA(c, cudaStreamSynchronize(c->stream));
		dfree(c, *p, sizeof(T) * per * have);
	}
	*p = q;
	have = need;
	return CT_OK;
}

ct_status ensure_nodes(Ctx* c, Box* b, int64_t need) {
	if (need <= b->node_cap) {
		return CT_OK;
	}
	int64_t cap = std::max<int64_t>(need, b->node_cap * 3 / 2);
	cap = std::max<int64_t>(cap, 1024);
	CT_TRY(each_node_array(b, [&](auto** p, int64_t& have, int per, const char* what) { return grow(c, p, have, cap, per, what); }));
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
	const int64_t pb = b->tree_begin();
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
	// one block an SM (half of what fits, so that two contexts build side by side), fewer for a few particles
	const int nblk = (int) std::max<int64_t>(1, std::min<int64_t>(c->nsm, std::max<int64_t>(np / 64, nroot)));
	LevelArgs la;
	la.idx = (int32_t*) scratch(c, 0, sizeof(int32_t) * n, &s1);
	la.posL = (int32_t*) scratch(c, 1, sizeof(int32_t) * n, &s1);
	la.posR = (int32_t*) scratch(c, 2, sizeof(int32_t) * n, &s1);
	la.sub = np > 2 * (int64_t) c->nsm * SUB * LWARPS ? SUB : BLOCK_SUB;
	// nodes in tiles hold more than WARP_FEW particles each
	const int64_t max_tn = np / WARP_FEW + 1, max_tiles = np / (la.sub * LWARPS) + max_tn + 1;
	la.tnode = (TileNode*) scratch(c, 3, sizeof(TileNode) * max_tn, &s1);
	la.tile_of = (int32_t*) scratch(c, 4, sizeof(int32_t) * max_tiles, &s1);
	la.tile_lt = (int32_t*) scratch(c, 5, sizeof(int32_t) * max_tiles, &s1);
	la.tile_mask = (uint32_t*) scratch(c, 8, sizeof(uint32_t) * 32 * (np / la.sub + max_tn + 2), &s1);
	la.blk = (int4*) scratch(c, 6, sizeof(int4) * 2 * nblk, &s1);
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
	// A build that ends before its gather (node arrays or the gather's scratch out of memory, a barrier that
	// gave up) has moved positions, and idx with them: a launch ends between phases, and a particle changes
	// place together with its index.  Velocities and rungs follow before the error returns, field by field
	// through the partition scratch, which takes no memory.
	auto stopped = [&](ct_status why) {
		for (int d = 0; d < 4 && np > 0; d++) {
			void* field = d < 3 ? (void*) (b->v[d] + pb) : (void*) (b->rung + pb);
			const size_t size = d < 3 ? sizeof(float) : sizeof(int8_t);
			CT_CUDA(c, cudaMemcpyAsync((char*) la.posL + size * pb, field, size * np, cudaMemcpyDeviceToDevice, st));
			c->launches++;
			if (d < 3) {
				k_gather_field<<<grid_for(c, np, 256), 256, 0, st>>>(pb, n, la.idx, (const float*) la.posL, b->v[d]);
			} else {
				k_gather_field<<<grid_for(c, np, 256), 256, 0, st>>>(pb, n, la.idx, (const int8_t*) la.posL, b->rung);
			}
			CT_CUDA(c, cudaGetLastError());
		}
		return why;
	};
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
			return stopped(fail(c, CT_ERR_CUDA, "tree build: the blocks of the cooperative grid did not meet"));
		}
		if (hc->status == 0) {
			break;
		}
		// the levels so far stay; the level that did not fit starts again with room for its children
		const ct_status room = ensure_nodes(c, b, hc->need);
		if (room != CT_OK) {
			return stopped(room);
		}
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
		if (s2 != CT_OK) {
			return stopped(s2);
		}
		if (np > 0) {
			c->launches += 2;
			k_stage_particles<<<grid_for(c, np, 256), 256, 0, st>>>(pb, n, b->v[0], b->v[1], b->v[2], b->rung, t0, t1, t2, tr);
			CT_CUDA(c, launch_behind(k_gather_particles, grid_for(c, np, 256), 256, st, pb, n, perm, t0, t1, t2, tr, b->v[0], b->v[1], b->v[2], b->rung));
		}
	}
	// upsweep: the leaves at once, then the interior nodes, deepest level first
	c->launches++;
	CT_CUDA(c, launch_behind(k_leaf_moments<Ops>, grid_for(c, 32 * b->nnodes, UTPB, 16), UTPB, st, b->nnodes, b->nodes, b->nbox, b->multi, b->tbox, b->gbox,
			b->x[0], b->x[1], b->x[2]));
	for (int k = (int) levels.size() - 2; k >= 0; k--) {
		const int64_t a = levels[k], e = levels[k + 1];
		if (k + 1 == (int) levels.size() - 1) {
			continue;  // the deepest level is all leaves
		}
		c->launches++;
		// as many nodes a block as leave four blocks an SM (two are resident): a level of few nodes is a
		// block each, so that the passes over the particles run side by side
		const int group = (int) std::max<int64_t>(1, std::min<int64_t>(UPS_NODES, (e - a) / (4 * c->nsm)));
		CT_CUDA(c, launch_behind(k_upsweep<Ops>, (int) std::min<int64_t>((e - a + group - 1) / group, (int64_t) c->nsm * 64), UPS_TPB, st, a, e, group, b->nodes,
				b->nbox, b->multi, b->tbox, b->gbox, b->x[0], b->x[1], b->x[2], p->bucket));
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

void nodes_release(Ctx* c, Box* b) {
	each_node_array(b, [&](auto** p, int64_t& have, int per, const char*) {
		dfree(c, *p, sizeof(**p) * per * have);
		*p = nullptr;
		have = 0;
		return (ct_status) CT_OK;
	});
	b->node_cap = 0;
}

ct_status tree_build(Ctx* c, Box* b, const ct_tree_params* p) {
	if (c->order == 5) {
		return tree_build_t<Ops5>(c, b, p);
	}
	return tree_build_t<Ops7>(c, b, p);
}

}  // namespace ct
