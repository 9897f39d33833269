// The volume gather as a masked matrix product on the tensor cores.
//
// A node's correction is linear in the records of the clusters that hold it:
// sum_j M_j (p - c_j) = (sum_j M_j) (p - o) - sum_j M_j (c_j - o).  Nodes that are close
// along the curve share most of their clusters, so 128 rows and the union of their clusters
// (about 850 at 64 members: every record is used ten times) form a tile:
//   sums[q][row] = sum_col value[q][col] * mask[col][row]
// with ten values per column (M, M (c - o), 1) and a 0/1 mask kept as bits.  A record is
// loaded once per tile instead of once per use (the list form is bound by the L1 wavefronts
// and the latency of 65 random 36-byte records per node), and the mask takes a third of the
// bytes of the index lists.
//
// The product runs on integers and is exact: relative to a point in the middle of the tile
// and to the largest value of its kind in the tile, a value is rounded once to 23 bits and
// cut into bytes, each a row of its own, whose sums mma.sync m16n8k32 (u8) accumulates in 32
// bits.  A value is off by at most 2^-23 of the largest of its kind, and so is a mean; the move
// of a point at most the tile's size E from o by 2^-23 w (3 M E + V) at most, with the largest M
// and M (c - o) and the inverse mass w.  Where w M E or w V is above 2^-6 of the largest
// coordinate R, and where records are not finite, the tile is done from the lists: elsewhere the
// error is at most 2^-27 R, an eighth of the rounding of a coordinate of that size (and some
// tenth of that, being a mean of 65 roundings).  One cluster far from its volume thus does not
// coarsen its neighbours.  In use w M E and w V are 2^-16 to 2^-8 of R; no more than two tiles in
// 10,000 is above 2^-6 in scenes of 2,000 to 1,000,000 Gaussians pulled, pressed and in
// contact.  The mask is the B operand straight from registers: a lane's 32-bit word holds its bits of two
// 16 x 32 blocks, one shift and one AND give a register of four 0/1 bytes.  (tcgen05 would
// need the mask expanded to bytes in shared memory, 128 per column and tile: more
// shared-memory traffic than the product itself has here.)
//
// Measured (B200, per launch, list form -> this): 1,000,000 Gaussians 286 -> 182 us, 200,000
// 72 -> 48, 20,000 20 -> 13; 250,000 with 128-member clusters 140 -> 71.
#pragma once
#include "kernels.cuh"

namespace xpbd {
namespace dev {

constexpr int kVtRows = 128;         // rows of a tile: eight groups of 16, a warp each
constexpr int kVtCols = 4096;        // columns at most
constexpr int kVtThreads = 256;
constexpr int kVtGroups = 8;
constexpr int kVtSlab = 1024;        // columns staged at a time: four per thread
constexpr int kVtStride = 136;       // row stride of the sums (8 mod 32: no bank conflicts)
constexpr int kVtMinComponent = 64;  // smaller graph components keep the list form
// Entries per row from which a tile pays.  Measured (us per launch, tile and list form): 10 a
// row 10.7 and 9.2 at 20,000 Gaussians, 36 and 26 at 250,000; 17 a row 14.5 / 12.0, 46 / 37;
// 25 a row 10.9 / 12.7, 43 / 44; 33 a row 12.8 / 16.9, 54 / 58; 65 a row 12.8 / 19.2, 56 / 82;
// 129 a row 16.9 / 25.5, 71 / 133.
constexpr int kVtMinEntries = 24;
constexpr float kVtStretch = 4.0f;   // a tile this much larger than at rest is done from the lists
constexpr float kVtMove = 0.015625f; // records above this part of the coordinates are, too (2^-6)
constexpr int kVtChunk = 2 * 512 + 64;   // bytes of a 32-column chunk: two m16 fragments, and a bank shift
constexpr int kVtSlabBytes = kVtChunk * (kVtSlab / 32);
constexpr int kVtWindow = 32;            // blocks of a group whose masks are held in shared memory
constexpr int kVtMaskBytes = kVtGroups * (kVtWindow / 2) * 128;
// shared memory: the slab (then the sums), the masks, each row's position, reverse-list bounds
// and rest length
constexpr int kVtRowsAt = kVtSlabBytes + kVtMaskBytes;
constexpr int kVtSmem = kVtRowsAt + kVtRows * (16 + 12);
static_assert(kVtSlabBytes >= 10 * kVtStride * 4, "the sums reuse the slab");


// One tile.  Its data in the word pool: the columns' rows (padded with -1 to a multiple of
// 32), the groups' blocks' column chunks (padded), then 32 mask words per pair of blocks of a
// group (a group of an odd number has a pair with an empty half).
struct VolTile {
	int row0, nrows;                 // its rows: rows[row0 ...]
	int cols;                        // columns
	int words;                       // first word in the pool
	unsigned short e[kVtGroups];     // end of each group's blocks
	unsigned short first[kVtGroups]; // each group's first pair of blocks
	float extent;                    // largest coordinate of its columns about its middle, at rest
	int masks;                       // pairs of blocks
	int mid[3];                      // three of its rows, spread along it
	int pad;
};
__host__ __device__ constexpr int vt_pad(int v) { return (v + 31) & ~31; }

// a point in the middle of the tile: per axis the median of three of its rows, so that one
// Gaussian gone astray does not move it; the origin where that is not finite
__device__ __forceinline__ float3 vt_middle(float4 a, float4 b, float4 c)
{
	auto med = [](float u, float v, float w) { return fmaxf(fminf(u, v), fminf(fmaxf(u, v), w)); };
	const float3 o = make_float3(med(a.x, b.x, c.x), med(a.y, b.y, c.y), med(a.z, b.z, c.z));
	return fin3(o) ? o : make_float3(0.0f, 0.0f, 0.0f);
}

// ---------------------------------------------------------------------------
// upload: the tile's column union and masks, one block per tile
// ---------------------------------------------------------------------------
constexpr int kVtHash = 8192;
constexpr int kVtBuildSmem = (kVtCols + kVtGroups * (kVtCols / 32) * 16) * 4;

// rank / row_of: position of a row along the curve and back (null: the same).  cols = 0 marks a
// tile whose rows keep the list form: more columns than kVtCols, a list with a repeated or
// invalid entry, or masks that take more words than the lists.
__global__ void __launch_bounds__(kVtThreads) k_tile_build(int n, VolTile* __restrict__ tiles,
	const int* __restrict__ rows, const int* __restrict__ off, const int* __restrict__ idx,
	const int* __restrict__ rank, const int* __restrict__ row_of, const float4* __restrict__ rest,
	unsigned int* __restrict__ pool, unsigned int pool_cap, unsigned int* __restrict__ bump)
{
	extern __shared__ int vt_sm[];
	int* cols = vt_sm;                                             // kVtCols
	int* hash = vt_sm + kVtCols;                                   // kVtHash, then the masks
	unsigned int* mask = reinterpret_cast<unsigned int*>(hash);    // [group][chunk][lane], 16 bits each
	__shared__ int s_count, s_bad, s_members, s_fill, s_groups[kVtGroups + 1], s_pairs[kVtGroups + 1];
	__shared__ unsigned int s_base;
	__shared__ unsigned int s_extent;
	__shared__ unsigned char s_flags[kVtGroups][kVtCols / 32];
	const int tx = threadIdx.x, lane = tx & 31, w = tx >> 5;
	const VolTile T = tiles[blockIdx.x];
	if (tx == 0) { s_count = 0; s_bad = 0; s_members = 0; s_fill = 0; s_extent = 0u; }
	for (int t = tx; t < kVtHash; t += kVtThreads) hash[t] = -1;
	__syncthreads();
	auto put = [&](int key) {
		unsigned int h = ((unsigned int)key * 2654435761u) >> 19;   // 13 bits
		for (int probe = 0; probe < kVtHash; ++probe, h = (h + 1) & (kVtHash - 1)) {
			const int old = atomicCAS(&hash[h], -1, key);
			if (old == key) return;
			if (old == -1) {
				if (atomicAdd(&s_count, 1) >= kVtCols) atomicExch(&s_bad, 1);
				return;
			}
			if (*(volatile int*)&s_bad) return;
		}
	};
	int members = 0;
	for (int r = w; r < T.nrows; r += kVtThreads / 32) {
		const int row = rows[T.row0 + r];
		const int e0 = off[row], e1 = off[row + 1];
		for (int e = e0 + lane; e < e1; e += 32) {
			const int j = idx[e];
			if (j < 0 || j >= n) { atomicExch(&s_bad, 1); continue; }
			put(rank ? rank[j] : j);
			++members;
		}
	}
	atomicAdd(&s_members, members);
	__syncthreads();
	const int U = s_count;
	if (s_bad || U == 0) {
		if (tx == 0) tiles[blockIdx.x].cols = 0;
		return;
	}
	for (int t = tx; t < kVtHash; t += kVtThreads)
		if (hash[t] >= 0) cols[atomicAdd(&s_fill, 1)] = hash[t];
	int P = 32;
	while (P < U) P <<= 1;
	__syncthreads();
	for (int t = U + tx; t < P; t += kVtThreads) cols[t] = 0x7fffffff;
	const int chunks = (U + 31) / 32;
	for (int t = tx; t < kVtGroups * chunks * 16; t += kVtThreads) mask[t] = 0u;
	__syncthreads();
	for (int k = 2; k <= P; k <<= 1)
		for (int j = k >> 1; j > 0; j >>= 1) {
			for (int t = tx; t < P; t += kVtThreads) {
				const int o = t ^ j;
				if (o > t) {
					const int a = cols[t], b = cols[o];
					if ((a > b) == ((t & k) == 0)) { cols[t] = b; cols[o] = a; }
				}
			}
			__syncthreads();
		}
	// column p, row slot r: block p / 32 of group r / 16; lane (r & 7, (p & 15) / 4), bit
	// ((r / 8) & 1, (p / 16) & 1) of nibble p & 3
	auto set = [&](int r, int key) {
		int lo = 0, hi = U - 1;
		while (lo < hi) {
			const int m = (lo + hi) >> 1;
			if (cols[m] < key) lo = m + 1;
			else hi = m;
		}
		const int l = (r & 7) * 4 + ((lo & 15) >> 2);
		const int bit = ((r >> 3) & 1) * 2 + ((lo >> 4) & 1) + 4 * (lo & 3) + 16 * (l & 1);
		const unsigned int old = atomicOr(&mask[((r >> 4) * chunks + (lo >> 5)) * 16 + (l >> 1)], 1u << bit);
		if (old & (1u << bit)) atomicExch(&s_bad, 1);
	};
	for (int r = w; r < T.nrows; r += kVtThreads / 32) {
		const int row = rows[T.row0 + r];
		const int e0 = off[row], e1 = off[row + 1];
		for (int e = e0 + lane; e < e1; e += 32) {
			const int j = idx[e];
			set(r, rank ? rank[j] : j);
		}
	}
	__syncthreads();
	for (int t = w; t < kVtGroups * chunks; t += kVtThreads / 32) {
		const bool any = __any_sync(0xffffffffu, mask[t * 16 + (lane & 15)] != 0u);
		if (lane == 0) s_flags[t / chunks][t % chunks] = any ? 1 : 0;
	}
	{
		const float3 o = vt_middle(rest[T.mid[0]], rest[T.mid[1]], rest[T.mid[2]]);
		float m = 0.0f;
		for (int t = tx; t < U; t += kVtThreads) {
			const float4 p = rest[row_of ? row_of[cols[t]] : cols[t]];
			m = fmaxf(m, fmaxf(fabsf(p.x - o.x), fmaxf(fabsf(p.y - o.y), fabsf(p.z - o.z))));
		}
		atomicMax(&s_extent, __float_as_uint(m));
	}
	__syncthreads();
	{
		int cnt = 0;
		for (int b = 0; b < chunks; b += 32)
			cnt += __popc(__ballot_sync(0xffffffffu, b + lane < chunks && s_flags[w][b + lane] != 0));
		if (lane == 0) { s_groups[w + 1] = cnt; s_pairs[w + 1] = (cnt + 1) / 2; }
	}
	__syncthreads();
	if (tx == 0) {
		s_groups[0] = s_pairs[0] = 0;
		for (int g = 0; g < kVtGroups; ++g) { s_groups[g + 1] += s_groups[g]; s_pairs[g + 1] += s_pairs[g]; }
		const int words = vt_pad(U) + vt_pad(s_groups[kVtGroups]) + 32 * s_pairs[kVtGroups];
		if (!s_bad && words <= s_members) {
			s_base = atomicAdd(bump, (unsigned int)words);
			if ((unsigned long long)s_base + words > pool_cap) s_bad = 1;
		}
		else
			s_bad = 1;
		VolTile out = T;
		out.cols = s_bad ? 0 : U;
		out.words = s_bad ? 0 : (int)s_base;
		out.extent = __uint_as_float(s_extent);
		out.masks = s_pairs[kVtGroups];
		for (int g = 0; g < kVtGroups; ++g) {
			out.e[g] = (unsigned short)s_groups[g + 1];
			out.first[g] = (unsigned short)s_pairs[g];
		}
		tiles[blockIdx.x] = out;
	}
	__syncthreads();
	if (s_bad) return;
	unsigned int* dst = pool + s_base;
	const int E = s_groups[kVtGroups];
	for (int t = tx; t < vt_pad(U); t += kVtThreads)
		dst[t] = (unsigned int)(t < U ? (row_of ? row_of[cols[t]] : cols[t]) : -1);
	unsigned int* ent = dst + vt_pad(U);
	unsigned int* out = ent + vt_pad(E) + 32 * s_pairs[w];
	for (int t = E + tx; t < vt_pad(E); t += kVtThreads) ent[t] = 0xffffffffu;
	// group w: its chunks in order; two blocks' bits per mask word, a nibble each of every byte
	int at = s_groups[w], half = 0;
	unsigned int word = 0u;
	for (int b = 0; b < chunks; b += 32) {
		const bool f = b + lane < chunks && s_flags[w][b + lane] != 0;
		const unsigned int bal = __ballot_sync(0xffffffffu, f);
		if (f) ent[at + __popc(bal & ((1u << lane) - 1u))] = (unsigned int)(b + lane);
		at += __popc(bal);
		for (unsigned int todo = bal; todo; todo &= todo - 1) {
			const int p = b + __ffs(todo) - 1;
			const unsigned int v = mask[(w * chunks + p) * 16 + (lane >> 1)] >> (16 * (lane & 1));
			const unsigned int spread = (v & 15u) | ((v & 0xf0u) << 4) | ((v & 0xf00u) << 8) | ((v & 0xf000u) << 12);
			word |= spread << (4 * half);
			if (half) {
				out[lane] = word;
				out += 32;
				word = 0u;
			}
			half ^= 1;
		}
	}
	if (half) out[lane] = word;
}

// tiles of one engine into another's arrays (serving arena): the row bases and the columns'
// rows shifted; one block per tile
__global__ void __launch_bounds__(kBlock) k_tile_copy(const VolTile* __restrict__ src, VolTile* __restrict__ dst,
	const unsigned int* __restrict__ words, unsigned int* __restrict__ pool, int row_at, int word_from, int word_at,
	int shift)
{
	VolTile T = src[blockIdx.x];
	const int count = vt_pad(T.cols) + vt_pad(T.e[kVtGroups - 1]) + 32 * T.masks;
	const unsigned int* s = words + (T.words - word_from);
	unsigned int* d = pool + (T.words - word_from) + word_at;
	for (int t = threadIdx.x; t < count; t += blockDim.x) {
		const unsigned int v = s[t];
		d[t] = t < T.cols ? v + (unsigned int)shift : v;
	}
	if (threadIdx.x == 0) {
		T.row0 += row_at;
		for (int k = 0; k < 3; ++k) T.mid[k] += shift;
		T.words += word_at - word_from;
		dst[blockIdx.x] = T;
	}
}

// ---------------------------------------------------------------------------
// the masked product
// ---------------------------------------------------------------------------
__device__ __forceinline__ void vt_mma(int (&c)[4], uint4 a, unsigned int b0, unsigned int b1)
{
	asm("mma.sync.aligned.m16n8k32.row.col.s32.u8.u8.s32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, "
		"{%0, %1, %2, %3};" : "+r"(c[0]), "+r"(c[1]), "+r"(c[2]), "+r"(c[3])
		: "r"(a.x), "r"(a.y), "r"(a.z), "r"(a.w), "r"(b0), "r"(b1));
}

constexpr float kVtTop = 4194303.0f;       // 2^22 - 1: the largest value of a kind
constexpr float kVtMagic = 12582912.0f;    // 1.5 x 2^23: v + kVtMagic rounds v to an integer, whose
                                           // 2^22 + v are the low three bytes of the sum

// four columns' integers v + kVtMagic, byte by byte: the low, middle and high bytes of each
struct VtWords { unsigned int high, mid, low; };
__device__ __forceinline__ VtWords vt_bytes4(float v0, float v1, float v2, float v3)
{
	const unsigned int a = __float_as_uint(v0), b = __float_as_uint(v1), c = __float_as_uint(v2), d = __float_as_uint(v3);
	const unsigned int ab = __byte_perm(a, b, 0x5140), cd = __byte_perm(c, d, 0x5140);   // a0 b0 a1 b1
	VtWords w;
	w.low = __byte_perm(ab, cd, 0x5410);
	w.mid = __byte_perm(ab, cd, 0x7632);
	w.high = __byte_perm(__byte_perm(a, b, 0x0062), __byte_perm(c, d, 0x0062), 0x5410);
	return w;
}
// where thread `quad`'s four columns go in the A-fragment order of m16n8k32.  The 32 rows of the
// two fragments come in pairs (r, r + 8) that lie side by side in a lane's registers; pair k,
// rows 16 (k / 8) + k % 8 and 8 more, is 8 bytes at vt_pair(k) from there
__device__ __forceinline__ unsigned char* vt_place(unsigned char* slab, int quad)
{
	return slab + (quad >> 3) * kVtChunk + (quad & 3) * 16 + ((quad >> 2) & 1) * 8;
}
__host__ __device__ constexpr int vt_pair(int k) { return 512 * (k / 8) + 64 * (k % 8); }
__device__ __forceinline__ void vt_put(unsigned char* at, int k, unsigned int first, unsigned int second)
{
	*reinterpret_cast<uint2*>(at + vt_pair(k)) = make_uint2(first, second);
}

__device__ __forceinline__ unsigned int vt_abs_bits(float v) { return __float_as_uint(v) & 0x7fffffffu; }

__device__ __forceinline__ void vt_copy16(void* to, const void* from)
{
	asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" :: "r"((unsigned int)__cvta_generic_to_shared(to)), "l"(from)
		: "memory");
}
__device__ __forceinline__ void vt_copy4(void* to, const void* from)
{
	asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" :: "r"((unsigned int)__cvta_generic_to_shared(to)), "l"(from)
		: "memory");
}
__device__ __forceinline__ void vt_copies_done() { asm volatile("cp.async.wait_all;" ::: "memory"); }

// The blocks of this warp's group.  Their masks come to shared memory a window of 32 blocks
// at a time (cp.async, sent off before the records are loaded: fetched where they are used,
// four blocks ahead, their latency was two thirds of a tile's time).
struct VtBlocks {
	const unsigned int* mask;        // the group's pairs of blocks
	const unsigned int* chunks;
	unsigned int* window;            // shared: this warp's kVtWindow / 2 x 32 words
	int count, at;                   // blocks, and how many are done
	unsigned int chunk;              // lane k: column chunk of block k of the window
	__device__ __forceinline__ VtBlocks(const VolTile* __restrict__ tile, const unsigned int* __restrict__ ent,
		unsigned char* __restrict__ masks)
	{
		const int g = threadIdx.x >> 5;
		const int e0 = g ? __ldg(&tile->e[g - 1]) : 0;
		count = __ldg(&tile->e[g]) - e0;
		chunks = ent + e0;
		mask = ent + vt_pad(__ldg(&tile->e[kVtGroups - 1])) + 32 * __ldg(&tile->first[g]);
		window = reinterpret_cast<unsigned int*>(masks) + g * (kVtWindow / 2) * 32;
		at = 0;
		fetch();
	}
	// the window that starts with block `at`
	__device__ __forceinline__ void fetch()
	{
		const int lane = threadIdx.x & 31;
		const int words = 32 * min((count - at + 1) / 2, kVtWindow / 2);
		const unsigned int* src = mask + 16 * at;
		for (int t = 4 * lane; t < words; t += 128) vt_copy16(window + t, src + t);
		chunk = at + lane < count ? __ldg(chunks + at + lane) : 0x7fffffffu;
	}
	__device__ __forceinline__ void arrive() const
	{
		vt_copies_done();
		__syncwarp();
	}
};

// acc += values x masks for the blocks whose columns lie in the slab [c0, c0 + kVtSlab)
__device__ __forceinline__ void vt_product(VtBlocks& B, const unsigned char* __restrict__ slab, int c0,
	int (&acc)[2][2][4])
{
	const int lane = threadIdx.x & 31;
	const unsigned int k0 = c0 / 32, k1 = k0 + kVtSlab / 32;
	while (B.at < B.count) {
		// the blocks of the window that lie in the slab
		const int i0 = B.at & (kVtWindow - 1);
		const int i1 = __popc(__ballot_sync(0xffffffffu, B.chunk < k1));
		struct Block { uint4 a0, a1; unsigned int w; };
		auto get = [&](int i) {
			Block b;
			const unsigned char* p = slab + (__shfl_sync(0xffffffffu, B.chunk, i) - k0) * kVtChunk + lane * 16;
			b.w = B.window[(i >> 1) * 32 + lane] >> (4 * (i & 1));
			b.a0 = *reinterpret_cast<const uint4*>(p);
			b.a1 = *reinterpret_cast<const uint4*>(p + 512);
			return b;
		};
		if (i0 < i1) {
			Block b = get(i0);
			for (int i = i0; i < i1; ++i) {   // the next block's fragments load while this one's multiply
				const Block next = get(min(i + 1, i1 - 1));
				const unsigned int b00 = b.w & 0x01010101u, b01 = (b.w >> 1) & 0x01010101u,
					b10 = (b.w >> 2) & 0x01010101u, b11 = (b.w >> 3) & 0x01010101u;
				vt_mma(acc[0][0], b.a0, b00, b01);
				vt_mma(acc[0][1], b.a0, b10, b11);
				vt_mma(acc[1][0], b.a1, b00, b01);
				vt_mma(acc[1][1], b.a1, b10, b11);
				b = next;
			}
		}
		B.at += i1 - i0;
		if (i1 < kVtWindow) break;
		__syncwarp();
		B.fetch();
		B.arrive();
	}
}

__device__ __forceinline__ void vt_clear(int (&acc)[2][2][4])
{
#pragma unroll
	for (int t = 0; t < 2; ++t)
#pragma unroll
		for (int k = 0; k < 8; ++k) acc[t][k >> 2][k & 3] = 0;
}

// The sums over the slab as floats: [value][row slot], the count in row 9.  A lane holds the
// high and middle bytes' sums of value q = lane / 4 for four row slots (first fragment) and its
// low bytes' (second); lanes 0-15 also hold value 8's bytes and the count.  bounds: the rows'
// reverse-list bounds, whose difference is the number of columns added to each row.
__device__ __forceinline__ void vt_sums(unsigned char* __restrict__ slab, const int (&acc)[2][2][4],
	const int* __restrict__ bounds, float um, float uv)
{
	const int lane = threadIdx.x & 31, q = lane >> 2, slot = (threadIdx.x >> 5) * 16 + 2 * (lane & 3);
	__syncthreads();   // the slab's last readers are done
	float* red = reinterpret_cast<float*>(slab);
	const float unit = q < 6 ? um : uv;
#pragma unroll
	for (int s = 0; s < 2; ++s) {
		const int r = slot + 8 * s;
#pragma unroll
		for (int e = 0; e < 2; ++e) {
			const int count = bounds[2 * (r + e) + 1] - bounds[2 * (r + e)];
			const int high = acc[0][s][e] - 64 * count;   // each column's 2^22 taken out
			red[q * kVtStride + r + e] = fmaf((float)high, 65536.0f, (float)(256 * acc[0][s][2 + e] + acc[1][s][e])) * unit;
			// value 8: high in lanes 0-3, middle in 4-7, low in 8-11; the count in 12-15
			const int t = acc[1][s][2 + e];
			const int mid = __shfl_down_sync(0xffffffffu, t, 4), low = __shfl_down_sync(0xffffffffu, t, 8);
			if (q == 0) red[8 * kVtStride + r + e] = fmaf((float)(t - 64 * count), 65536.0f, (float)(256 * mid + low)) * uv;
			if (q == 3) red[9 * kVtStride + r + e] = (float)t;
		}
	}
	__syncthreads();
}

// The gather of one tile by one block: sums of the records' M (xx yy zz xy xz yz), M (c - o)
// and 1 from the product, then the mean, clamp and under-relaxation per node as in the list
// form (gather_group_lane), one thread per row.  An absent record gives zeros.  slab is free
// again after the block's next barrier.
template <bool CHAIN>
__device__ __forceinline__ void tile_gather(unsigned char* __restrict__ slab, unsigned int (&part)[2][kVtThreads / 32],
	int n, const StepParams* __restrict__ P, const float4* __restrict__ pin, float4* __restrict__ pout,
	const VolTile* __restrict__ tile, const int* __restrict__ rows, const unsigned int* __restrict__ pool,
	const int* __restrict__ roff, const int* __restrict__ ridx, const float4* __restrict__ rec,
	const float* __restrict__ recz, const float* __restrict__ rest_len)
{
	const int tx = threadIdx.x;
	const int row0 = __ldg(&tile->row0), nrows = __ldg(&tile->nrows), cols = __ldg(&tile->cols);
	const float ims = P->inv_mass_scale, under_relax = P->under_relax;
	bool lists;
	{
		const unsigned int* words = pool + __ldg(&tile->words);
		// the four columns of this thread in the slab from column c0
		auto columns = [&](int c0) {
			const int c = c0 + 4 * tx;
			return c < vt_pad(cols) ? __ldg(reinterpret_cast<const int4*>(words + c)) : make_int4(-1, -1, -1, -1);
		};
		// The loads that depend on nothing but the tile go out together: the columns, the
		// mask blocks, this thread's row
		int c0 = (cols - 1) / kVtSlab * kVtSlab;
		int4 j = columns(c0);
		VtBlocks B(tile, words + vt_pad(cols), slab + kVtSlabBytes);
		float4* row_pos = reinterpret_cast<float4*>(slab + kVtRowsAt);
		int* row_bounds = reinterpret_cast<int*>(row_pos + kVtRows);
		float* row_len = reinterpret_cast<float*>(row_bounds + 2 * kVtRows);
		const int row = tx < nrows ? __ldg(rows + row0 + tx) : -1;
		if (row >= 0) {   // the row's own data, for the end
			vt_copy4(row_bounds + 2 * tx, roff + row);
			vt_copy4(row_bounds + 2 * tx + 1, roff + row + 1);
			vt_copy4(row_len + tx, rest_len + row);
		}
		else if (tx < kVtRows) row_bounds[2 * tx] = row_bounds[2 * tx + 1] = 0;
		const int i0 = __ldg(&tile->mid[0]), i1 = __ldg(&tile->mid[1]), i2 = __ldg(&tile->mid[2]);
		if (CHAIN) chain_wait();   // up to here what the upload wrote
		const float4 m0 = ldv<false>(pin, i0), m1 = ldv<false>(pin, i1), m2 = ldv<false>(pin, i2);
		float v[4][9];
		unsigned int valid;
		const float3 o = vt_middle(m0, m1, m2);
		auto load = [&]() {
			const int jj[4] = { j.x, j.y, j.z, j.w };
			float4 a[4], b[4];
			float z[4];
#pragma unroll
			for (int k = 0; k < 4; ++k) {
				a[k] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
				b[k] = make_float4(0.0f, 0.0f, CUDART_NAN_F, 0.0f);
				z[k] = 0.0f;
				if (jj[k] >= 0) { ld_rec<false>(rec, jj[k], a[k], b[k]); z[k] = ldv<false>(recz, jj[k]); }
			}
			valid = 0u;
#pragma unroll
			for (int k = 0; k < 4; ++k) {
				const bool ok = isfinite(b[k].z);
				if (ok) valid |= 1u << (8 * k);
				const float x = ok ? b[k].z - o.x : 0.0f, y = ok ? b[k].w - o.y : 0.0f, w = ok ? z[k] - o.z : 0.0f;
				v[k][0] = ok ? a[k].x : 0.0f; v[k][1] = ok ? a[k].y : 0.0f; v[k][2] = ok ? a[k].z : 0.0f;
				v[k][3] = ok ? a[k].w : 0.0f; v[k][4] = ok ? b[k].x : 0.0f; v[k][5] = ok ? b[k].y : 0.0f;
				v[k][6] = v[k][0] * x + v[k][3] * y + v[k][4] * w;
				v[k][7] = v[k][3] * x + v[k][1] * y + v[k][5] * w;
				v[k][8] = v[k][4] * x + v[k][5] * y + v[k][2] * w;
			}
		};
		unsigned int am = 0u, av = 0u;
		for (;;) {   // ends with the first slab's records in v
			if (c0 + 4 * (tx & ~31) < cols) {
				load();
#pragma unroll
				for (int k = 0; k < 4; ++k) {
#pragma unroll
					for (int q = 0; q < 6; ++q) am = max(am, vt_abs_bits(v[k][q]));
#pragma unroll
					for (int q = 6; q < 9; ++q) av = max(av, vt_abs_bits(v[k][q]));
				}
			}
			if (c0 == 0) break;
			c0 -= kVtSlab;
			j = columns(c0);
		}
		if (row >= 0) vt_copy16(row_pos + tx, pin + row);
		am = __reduce_max_sync(0xffffffffu, am);
		av = __reduce_max_sync(0xffffffffu, av);
		if ((tx & 31) == 0) { part[0][tx >> 5] = am; part[1][tx >> 5] = av; }
		__syncthreads();
#pragma unroll
		for (int k = 0; k < kVtThreads / 32; ++k) { am = max(am, part[0][k]); av = max(av, part[1][k]); }
		const float top_m = __uint_as_float(am), top_v = __uint_as_float(av);
		// records too large for 23 bits to be as good as the lists' floats (see the top), or that
		// would move a point by several times its distance, and values that are not finite, are
		// left to the lists
		const float extent = __ldg(&tile->extent);
		const float limit = kVtMove * (extent + fmaxf(fabsf(o.x), fmaxf(fabsf(o.y), fabsf(o.z))));
		lists = !(top_m <= 4.0f) || !(top_v <= 16.0f * kVtStretch * extent) || !(ims * top_m * extent <= limit) ||
			!(ims * top_v <= limit);
		if (lists) B.arrive();   // no copy is left in flight
		else {
			const float sm = kVtTop / fmaxf(top_m, 1e-30f), sv = kVtTop / fmaxf(top_v, 1e-30f);
			unsigned char* at = vt_place(slab, tx);
			auto put = [&]() {
				if (c0 + 4 * (tx & ~31) < cols) {
					const VtWords e = vt_bytes4(fmaf(v[0][8], sv, kVtMagic), fmaf(v[1][8], sv, kVtMagic),
						fmaf(v[2][8], sv, kVtMagic), fmaf(v[3][8], sv, kVtMagic));
					const unsigned int tail[8] = { e.high, e.mid, e.low, valid, 0u, 0u, 0u, 0u };
#pragma unroll
					for (int q = 0; q < 8; ++q) {
						const float s = q < 6 ? sm : sv;
						const VtWords w = vt_bytes4(fmaf(v[0][q], s, kVtMagic), fmaf(v[1][q], s, kVtMagic),
							fmaf(v[2][q], s, kVtMagic), fmaf(v[3][q], s, kVtMagic));
						vt_put(at, q, w.high, w.mid);
						vt_put(at, 8 + q, w.low, tail[q]);
					}
				}
				__syncthreads();
			};
			put();
			int acc[2][2][4];
			vt_clear(acc);
			B.arrive();
			vt_product(B, slab, 0, acc);
			for (c0 = kVtSlab; c0 < cols; c0 += kVtSlab) {
				j = columns(c0);
				if (c0 + 4 * (tx & ~31) < cols) load();
				__syncthreads();   // the slab's last readers are done
				put();
				vt_product(B, slab, c0, acc);
			}
			vt_sums(slab, acc, row_bounds, 1.0f / sm, 1.0f / sv);
			if (CHAIN) chain_next();
			if (row < 0) return;
			const float4 p4 = row_pos[tx];
			const float* sum = reinterpret_cast<const float*>(slab) + tx;
			float s[9];
#pragma unroll
			for (int q = 0; q < 9; ++q) s[q] = sum[q * kVtStride];
			const float wi = p4.w * ims, rc = sum[9 * kVtStride];
			if (!(wi > 0.0f) || !(rc > 0.0f)) { pout[row] = p4; return; }
			const float dx = p4.x - o.x, dy = p4.y - o.y, dz = p4.z - o.z;
			const float inv_rec = wi / rc;
			const float3 avg = make_float3((s[0] * dx + s[3] * dy + s[4] * dz - s[6]) * inv_rec,
				(s[3] * dx + s[1] * dy + s[5] * dz - s[7]) * inv_rec, (s[4] * dx + s[5] * dy + s[2] * dz - s[8]) * inv_rec);
			if (!fin3(avg)) { pout[row] = p4; return; }
			const float3 r = gather_finish(f3(p4), avg, row_len[tx], under_relax);
			pout[row] = make_float4(r.x, r.y, r.z, p4.w);
		}
	}
	if (lists)
		for (int t = tx; t < 4 * kVtRows; t += kVtThreads) {
			const int row = (t >> 2) < nrows ? __ldg(rows + row0 + (t >> 2)) : n;
			gather_group_lane<4>((long long)row * 4 + (t & 3), n, P, pin, pout, roff, ridx, rec, recz, rest_len);
		}
}

// three blocks per SM (80 registers, a few spilled): two without spills are as fast at 1M and
// four (64 registers) slower, 206 against 182 us
__global__ void __launch_bounds__(kVtThreads, 3) k_tile_gather(int n, const StepParams* __restrict__ P,
	const float4* __restrict__ pin, float4* __restrict__ pout, const VolTile* __restrict__ tiles,
	const int* __restrict__ rows, const unsigned int* __restrict__ pool, const int* __restrict__ roff,
	const int* __restrict__ ridx, const float4* __restrict__ rec, const float* __restrict__ recz,
	const float* __restrict__ rest_len)
{
	extern __shared__ __align__(16) unsigned char slab[];   // kVtSmem
	__shared__ unsigned int part[2][kVtThreads / 32];
	tile_gather<true>(slab, part, n, P, pin, pout, tiles + blockIdx.x, rows, pool, roff, ridx, rec, recz, rest_len);
}

}  // namespace dev
}  // namespace xpbd
