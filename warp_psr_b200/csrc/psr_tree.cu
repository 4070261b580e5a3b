// A4: sparse tree completion (warp-psr tree.py:152-201).  Integer only; keys must match
// the reference bit for bit.  Brood keys are sorted in a compact form: at level d every
// candidate brood coordinate lies in [-2^d, 2^d), so (c + 2^d) packs into d+1 bits per
// axis with the same lexicographic order as the reference's 20-bit signed tree keys.
#include "psr_internal.cuh"

namespace psr {

__device__ __forceinline__ uint64_t pack_brood(const int c[3], int d) {
  int n = 1 << d, D = d + 1;
  return (uint64_t(c[0] + n) << (2 * D)) | (uint64_t(c[1] + n) << D) | uint64_t(c[2] + n);
}
__device__ __forceinline__ void unpack_brood(uint64_t k, int d, int c[3]) {
  int n = 1 << d, D = d + 1;
  uint64_t mask = (uint64_t(1) << D) - 1;
  c[0] = int((k >> (2 * D)) & mask) - n;
  c[1] = int((k >> D) & mask) - n;
  c[2] = int(k & mask) - n;
}

// tree.py:41-50 — broods of this level's normal records with nonzero coefficients.
template <class T>
__global__ void seed_kernel(const int64_t* nkeys, const T* nvals, int64_t count, int d, uint64_t* out) {
  int64_t i = blockIdx.x * int64_t(blockDim.x) + threadIdx.x;
  if (i >= count) return;
  const T* v = nvals + 4 * i;
  T l2 = v[0] * v[0] + v[1] * v[1] + v[2] * v[2] + v[3] * v[3];
  uint64_t key = uint64_t(1) << (3 * (d + 1));
  if (double(l2) > 0.0) {
    int c[3];
    key_coords(nkeys[i], c);
    int p[3] = {c[0] >> 1, c[1] >> 1, c[2] >> 1};
    key = pack_brood(p, d);
  }
  out[i] = key;
}

// tree.py:30-34 — the full-depth coarse region, starting at -1.
__global__ void coarse_kernel(int d, int count, uint64_t* out) {
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= count * count * count) return;
  int c[3] = {i / (count * count) - 1, (i / count) % count - 1, i % count - 1};
  out[i] = pack_brood(c, d);
}

// tree.py:52-64 — (2r+1)^3 broods around the parent of every source node.
__global__ void support_kernel(const int64_t* src, int64_t count, int radius, int d, uint64_t* out) {
  int64_t i = blockIdx.x * int64_t(blockDim.x) + threadIdx.x;
  if (i >= count) return;
  int w = 2 * radius + 1;
  int c[3];
  tree_coords(src[i], c);
  int p[3] = {c[0] >> 1, c[1] >> 1, c[2] >> 1};
  int n = 1 << d;
  uint64_t sentinel = uint64_t(1) << (3 * (d + 1));
  for (int j = 0; j < w * w * w; ++j) {
    int q[3] = {p[0] + j / (w * w) - radius, p[1] + (j / w) % w - radius, p[2] + j % w - radius};
    bool ok = dmin(q[0], dmin(q[1], q[2])) >= -n && dmax(q[0], dmax(q[1], q[2])) < n;
    out[i * w * w * w + j] = ok ? pack_brood(q, d) : sentinel;
  }
}

template <class K>
__global__ void unique_heads_kernel(const K* keys, int64_t n, uint64_t sentinel, int32_t* heads) {
  int64_t i = blockIdx.x * int64_t(blockDim.x) + threadIdx.x;
  if (i >= n) return;
  heads[i] = uint64_t(keys[i]) < sentinel && (i == 0 || keys[i] != keys[i - 1]);
}

template <class K>
__global__ void compact_kernel(const K* keys, const int32_t* heads, const int32_t* prefix, int64_t n,
                               uint64_t* out) {
  int64_t i = blockIdx.x * int64_t(blockDim.x) + threadIdx.x;
  if (i < n && heads[i]) out[prefix[i] - 1] = uint64_t(keys[i]);
}

// 64-bit keys below 2^32 narrowed to 32 bits for the sort.
__global__ void narrow_keys_kernel(const uint64_t* keys, int64_t n, uint32_t* out) {
  int64_t i = blockIdx.x * int64_t(blockDim.x) + threadIdx.x;
  if (i < n) out[i] = uint32_t(keys[i]);
}

__device__ __forceinline__ int64_t lower_bound_u64(const uint64_t* a, int64_t n, uint64_t key) {
  int64_t lo = 0, hi = n;
  while (lo < hi) {
    int64_t mid = (lo + hi) / 2;
    if (a[mid] < key)
      lo = mid + 1;
    else
      hi = mid;
  }
  return lo;
}

// tree.py:78-97 — eight children per sorted unique brood, written directly in sorted order.
__global__ void expand_kernel(const uint64_t* broods, int64_t n, int d, int64_t* children, int32_t* basis_mark) {
  int64_t i = blockIdx.x * int64_t(blockDim.x) + threadIdx.x;
  if (i >= n) return;
  int D = d + 1;
  uint64_t key = broods[i];
  uint64_t x = (key >> (2 * D)) << (2 * D);
  uint64_t xy = (key >> D) << D;
  int64_t x0 = lower_bound_u64(broods, n, x), x1 = lower_bound_u64(broods, n, x + (uint64_t(1) << (2 * D)));
  int64_t xy0 = lower_bound_u64(broods, n, xy), xy1 = lower_bound_u64(broods, n, xy + (uint64_t(1) << D));
  int c[3];
  unpack_brood(key, d, c);
  int res = 1 << d;
  for (int k = 0; k < 8; ++k) {
    int ox = (k >> 2) & 1, oy = (k >> 1) & 1, oz = k & 1;
    int64_t dest = 8 * x0 + 4 * ox * (x1 - x0) + 4 * (xy0 - x0) + 2 * oy * (xy1 - xy0) + 2 * (i - xy0) + oz;
    int q[3] = {2 * c[0] + ox, 2 * c[1] + oy, 2 * c[2] + oz};
    children[dest] = tree_key(q[0], q[1], q[2]);
    basis_mark[dest] = dmin(q[0], dmin(q[1], q[2])) >= 0 && dmax(q[0], dmax(q[1], q[2])) <= res;
  }
}

__global__ void basis_fill_kernel(const int64_t* children, const int32_t* mark, const int32_t* prefix, int64_t n,
                                  int d, int64_t* out) {
  int64_t i = blockIdx.x * int64_t(blockDim.x) + threadIdx.x;
  if (i >= n || !mark[i]) return;
  int c[3];
  tree_coords(children[i], c);
  out[prefix[i] - 1] = basis_key(d, c[0], c[1], c[2]);
}

__global__ void parent_tree_keys_kernel(const int64_t* src, int64_t n, uint64_t* out) {
  int64_t i = blockIdx.x * int64_t(blockDim.x) + threadIdx.x;
  if (i >= n) return;
  int c[3];
  tree_coords(src[i], c);
  out[i] = uint64_t(tree_key(c[0] >> 1, c[1] >> 1, c[2] >> 1));
}

__global__ void u64_to_i64_kernel(const uint64_t* in, int64_t n, int64_t* out) {
  int64_t i = blockIdx.x * int64_t(blockDim.x) + threadIdx.x;
  if (i < n) out[i] = int64_t(in[i]);
}

__global__ void broods_to_tree_keys_kernel(const uint64_t* in, int64_t n, int d, int64_t* out) {
  int64_t i = blockIdx.x * int64_t(blockDim.x) + threadIdx.x;
  if (i >= n) return;
  int c[3];
  unpack_brood(in[i], d, c);
  out[i] = tree_key(c[0], c[1], c[2]);
}

// Sort + unique of n keys below `sentinel`; returns the count and the unique keys.
static int64_t sort_unique(DBuf<uint64_t>& keys, int64_t n, int end_bit, uint64_t sentinel, DBuf<uint64_t>& out,
                           cudaStream_t s) {
  if (n == 0) {
    out.alloc(0, s);
    return 0;
  }
  // Keys of at most 32 bits (depth <= 9 here) are sorted as 32-bit keys: half the data
  // through every pass for one narrowing copy.  Same order, same unique keys.
  DBuf<int32_t> heads(n, s), prefix(n, s);
  int64_t u = 0;
  auto run = [&](auto key_tag, const decltype(key_tag)* in) {
    using K = decltype(key_tag);
    DBuf<K> sorted(n, s);
    size_t temp = 0;
    PSR_CUDA(cub::DeviceRadixSort::SortKeys(nullptr, temp, in, sorted.p, n, 0, end_bit, s));
    {
      DBuf<char> t(int64_t(temp), s);
      PSR_CUDA(cub::DeviceRadixSort::SortKeys(t.p, temp, in, sorted.p, n, 0, end_bit, s));
    }
    unique_heads_kernel<K><<<blocks_for(n), kThreads, 0, s>>>(sorted.p, n, sentinel, heads.p);
    PSR_LAUNCH_CHECK();
    inclusive_sum(heads.p, prefix.p, n, s);
    u = read_scalar(prefix.p + n - 1, s);
    out.alloc(u, s);
    compact_kernel<K><<<blocks_for(n), kThreads, 0, s>>>(sorted.p, heads.p, prefix.p, n, out.p);
    PSR_LAUNCH_CHECK();
  };
  if (end_bit <= 32) {
    DBuf<uint32_t> narrow(n, s);
    narrow_keys_kernel<<<blocks_for(n), kThreads, 0, s>>>(keys.p, n, narrow.p);
    PSR_LAUNCH_CHECK();
    run(uint32_t(), narrow.p);
  } else {
    run(uint64_t(), keys.p);
  }
  return u;
}

// ------------------------------------------------------------------ the tree on bitmaps
// A brood of level d is a node of level d - 1: its coordinates lie in [-2, 2^(d-1) + 1] (the
// dilation by one of the halved coordinates of the finer level's broods, which lie in
// [-2, 2^d + 1], stays there).  One bit per node of that grid, rows along z padded to whole words,
// and a count per word: 5.7 MB through depth 9, 42 MB through depth 10, 321 MB through depth 11,
// for the levels down to the finest one with records (finer levels have no broods).  A set is then
// united by OR-ing words and comes out sorted and unique, so a level needs no sort of its 27
// candidates per request, and no count of one level is needed on the host to build the next: the
// whole tree waits for the host once instead of twice per level.  A call with 2,011 points at
// depth 5: 3.59 -> 2.84 ms, 200,000 at depth 8 10.2 -> 8.7, 800,000 at depth 9 24.9 -> 22.5.
// The tree stage against the sorts (records with the finest ones at the tree's depth, then 5 points
// in a few coarse records): depth 8 217 and 1,661 us (730,000 records), 82 and 336; depth 10 878 and
// 5,462 (8.6 million), 350 and 1,401 (135 records), 82 and 338; depth 11 2,354 and 8,415 (2.6
// million), 1,500 and 1,600 (135 records), 84 and 343 (1,460 with the empty levels' bitmaps).
// Past depth 11 the bitmaps outgrow the sorts (2.5 GB at depth 12) and build_tree sorts.
constexpr int kBitmapDepth = 11;
constexpr int kBitmapLow = -2;

__host__ __device__ constexpr int brood_side(int d) { return d == 0 ? 4 : (1 << (d - 1)) + 4; }
__host__ __device__ constexpr int brood_row(int d) { return (brood_side(d) + 31) / 32; }  // words per z-row
__host__ __device__ constexpr int64_t brood_words(int d) {
  return int64_t(brood_side(d)) * brood_side(d) * brood_row(d);
}

struct BroodLevels {
  int64_t base[kBitmapDepth + 2];  // first word of each level; one past the last level's words
  int depth;
  __device__ __forceinline__ int level_of(int64_t word) const {
    int d = 0;
    while (d < depth && word >= base[d + 1]) ++d;
    return d;
  }
};

// Seeds of every level (seed_kernel's), one thread per normal record.
template <class T>
__global__ void seed_bits_kernel(const int64_t* nkeys, const T* nvals, int64_t count, BroodLevels L, uint32_t* bits) {
  const int64_t i = blockIdx.x * int64_t(blockDim.x) + threadIdx.x;
  if (i >= count) return;
  const T* v = nvals + 4 * i;
  const T l2 = v[0] * v[0] + v[1] * v[1] + v[2] * v[2] + v[3] * v[3];
  if (!(double(l2) > 0.0)) return;
  int c[3];
  key_coords(nkeys[i], c);
  const int d = int(nkeys[i] >> 48), side = brood_side(d), row = brood_row(d);
  const int z = (c[2] >> 1) - kBitmapLow;
  const int64_t r = int64_t((c[0] >> 1) - kBitmapLow) * side + (c[1] >> 1) - kBitmapLow;
  uint32_t* word = bits + L.base[d] + r * row + z / 32;
  const uint32_t bit = 1u << (z % 32);
  if (!(*reinterpret_cast<volatile uint32_t*>(word) & bit)) atomicOr(word, bit);
}

// The coarse region of the levels through `full` (coarse_kernel's), one thread per word.
__global__ void coarse_bits_kernel(BroodLevels L, int full, uint32_t* bits) {
  const int64_t w = blockIdx.x * int64_t(blockDim.x) + threadIdx.x;
  if (w >= L.base[full + 1]) return;
  const int d = L.level_of(w), side = brood_side(d), row = brood_row(d);
  const int last = (d == 0 ? 2 : (1 << (d - 1)) + 2) - 2 - kBitmapLow;  // coordinates -1 .. last
  const int64_t r = w - L.base[d];
  const int x = int(r / row / side), y = int(r / row % side), z0 = int(r % row) * 32, first = -1 - kBitmapLow;
  if (x < first || x > last || y < first || y > last) return;
  const int lo = max(first - z0, 0), hi = min(last - z0, 31);
  if (lo <= hi) bits[w] = (0xffffffffu << lo) & (0xffffffffu >> (31 - hi));
}

// support_kernel on bitmaps: the broods of level d within `radius` (0 or 1) of the parents of the
// nodes in `src`, a bitmap of level d + 1's broods; one thread per source word.  The 32 nodes of a
// word have 16 parents along z: a mask of up to 18 bits that goes to the rows around.
__global__ void parent_bits_kernel(const uint32_t* __restrict__ src, int d, int radius, uint32_t* dst) {
  const int64_t w = blockIdx.x * int64_t(blockDim.x) + threadIdx.x;
  if (w >= brood_words(d + 1)) return;
  uint32_t t = src[w];
  if (!t) return;
  const int ss = brood_side(d + 1), sr = brood_row(d + 1), side = brood_side(d), row = brood_row(d), n = 1 << d;
  const int x = (int(w / sr / ss) + kBitmapLow) >> 1, y = (int(w / sr % ss) + kBitmapLow) >> 1, k = int(w % sr);
  t = (t | t >> 1) & 0x55555555u;
  t = (t | t >> 1) & 0x33333333u;
  t = (t | t >> 2) & 0x0f0f0f0fu;
  t = (t | t >> 4) & 0x00ff00ffu;
  t = (t | t >> 8) & 0x0000ffffu;
  // bit j of the mask: brood coordinate kBitmapLow + 16 k + j (the word's first parent, minus one)
  const uint64_t mask = uint64_t(radius ? t | t << 1 | t << 2 : t << 1) << (16 * (k & 1));
  uint32_t lo = uint32_t(mask), hi = uint32_t(mask >> 32);
  if (d < 2) lo &= ((1u << (n - kBitmapLow)) - 1u) & ~((1u << (-kBitmapLow - n)) - 1u);  // [-2^d, 2^d) as support_kernel
  for (int dx = -radius; dx <= radius; ++dx)
    for (int dy = -radius; dy <= radius; ++dy) {
      const int qx = x + dx, qy = y + dy;
      if (min(qx, qy) < -n || max(qx, qy) >= n) continue;
      uint32_t* out = dst + (int64_t(qx - kBitmapLow) * side + qy - kBitmapLow) * row + k / 2;
      if (lo && (*reinterpret_cast<volatile uint32_t*>(out) & lo) != lo) atomicOr(out, lo);
      if (hi && k / 2 + 1 < row && (*reinterpret_cast<volatile uint32_t*>(out + 1) & hi) != hi) atomicOr(out + 1, hi);
    }
}

// Children of a brood coordinate inside [0, 2^d], per axis.
__device__ __forceinline__ int valid_children(int c, int d) {
  return (2 * c >= 0 && 2 * c <= (1 << d)) + (2 * c + 1 >= 0 && 2 * c + 1 <= (1 << d));
}

// Broods of every word, and the basis nodes (children inside the grid) of every level.
__global__ void __launch_bounds__(kThreads) brood_count_kernel(const uint32_t* __restrict__ bits, BroodLevels L,
                                                               int64_t words, int32_t* counts, int* basis) {
  __shared__ int s_basis[kBitmapDepth + 1];
  if (threadIdx.x <= kBitmapDepth) s_basis[threadIdx.x] = 0;
  __syncthreads();
  const int64_t w = blockIdx.x * int64_t(blockDim.x) + threadIdx.x;
  if (w < words) {
    uint32_t t = bits[w];
    counts[w] = __popc(t);
    if (t) {
      const int d = L.level_of(w), side = brood_side(d), row = brood_row(d);
      const int64_t r = w - L.base[d];
      const int vx = valid_children(int(r / row / side) + kBitmapLow, d);
      const int vy = valid_children(int(r / row % side) + kBitmapLow, d);
      int vz = 0;
      for (; t && vx * vy; t &= t - 1) vz += valid_children(int(r % row) * 32 + __ffs(t) - 1 + kBitmapLow, d);
      if (vx * vy * vz) atomicAdd(&s_basis[d], vx * vy * vz);
    }
  }
  __syncthreads();
  if (threadIdx.x <= L.depth && s_basis[threadIdx.x]) atomicAdd(basis + threadIdx.x, s_basis[threadIdx.x]);
}

// Broods through the end of each level, beside the basis counts, for one read-back.
__global__ void brood_totals_kernel(const int32_t* prefix, BroodLevels L, int* totals) {
  if (threadIdx.x <= L.depth) totals[threadIdx.x] = prefix[L.base[threadIdx.x + 1] - 1];
}

__global__ void brood_emit_kernel(const uint32_t* __restrict__ bits, const int32_t* __restrict__ prefix,
                                  BroodLevels L, int64_t words, int4* broods) {
  const int64_t w = blockIdx.x * int64_t(blockDim.x) + threadIdx.x;
  if (w >= words) return;
  uint32_t t = bits[w];
  if (!t) return;
  const int d = L.level_of(w), side = brood_side(d), row = brood_row(d);
  const int64_t r = w - L.base[d];
  int64_t out = prefix[w] - __popc(t);
  for (; t; t &= t - 1)
    broods[out++] = make_int4(int(r / row / side), int(r / row % side), int(r % row) * 32 + __ffs(t) - 1, d);
}

struct TreeOut {
  int64_t* support[kBitmapDepth + 1];
  int64_t* basis[kBitmapDepth + 1];
  int64_t brood0[kBitmapDepth + 1];  // broods and basis nodes of the levels below
  int64_t basis0[kBitmapDepth + 1];
};

// expand_kernel for the broods of every level: a brood's children in sorted order, from the
// ranks of its x-slab's and its (x, y) row's first broods.
__global__ void brood_expand_kernel(const int4* __restrict__ broods, int64_t n, const int32_t* __restrict__ prefix,
                                    BroodLevels L, TreeOut out, int32_t* mark) {
  const int64_t i = blockIdx.x * int64_t(blockDim.x) + threadIdx.x;
  if (i >= n) return;
  const int4 b = broods[i];
  const int d = b.w, side = brood_side(d), row = brood_row(d), res = 1 << d;
  const int64_t first = out.brood0[d];
  auto rank = [&](int64_t r) {  // broods of the level before z-row r
    const int64_t w = L.base[d] + r * row;
    return (w > 0 ? int64_t(prefix[w - 1]) : 0) - first;
  };
  const int64_t slab = int64_t(b.x) * side;
  const int64_t x0 = rank(slab), x1 = rank(slab + side), xy0 = rank(slab + b.y), xy1 = rank(slab + b.y + 1);
  for (int k = 0; k < 8; ++k) {
    const int ox = (k >> 2) & 1, oy = (k >> 1) & 1, oz = k & 1;
    const int64_t dest =
        8 * x0 + 4 * ox * (x1 - x0) + 4 * (xy0 - x0) + 2 * oy * (xy1 - xy0) + 2 * (i - first - xy0) + oz;
    const int q[3] = {2 * (b.x + kBitmapLow) + ox, 2 * (b.y + kBitmapLow) + oy, 2 * (b.z + kBitmapLow) + oz};
    out.support[d][dest] = tree_key(q[0], q[1], q[2]);
    mark[8 * first + dest] = dmin(q[0], dmin(q[1], q[2])) >= 0 && dmax(q[0], dmax(q[1], q[2])) <= res;
  }
}

__global__ void brood_basis_kernel(const int32_t* __restrict__ mark, const int32_t* __restrict__ prefix, int64_t n,
                                   int depth, TreeOut out) {
  const int64_t i = blockIdx.x * int64_t(blockDim.x) + threadIdx.x;
  if (i >= n || !mark[i]) return;
  int d = 0;
  while (d < depth && i >= 8 * out.brood0[d + 1]) ++d;
  int c[3];
  tree_coords(out.support[d][i - 8 * out.brood0[d]], c);
  out.basis[d][prefix[i] - 1 - out.basis0[d]] = basis_key(d, c[0], c[1], c[2]);
}

template <class T>
static TreeData build_tree_bitmap(const NormalData<T>& N, int depth, int full_depth, int base_depth, cudaStream_t s) {
  TreeData tree;
  tree.support.resize(depth + 1);
  tree.basis.resize(depth + 1);
  tree.support_count.assign(depth + 1, 0);
  tree.basis_count.assign(depth + 1, 0);
  int top = full_depth;  // the finest level with broods
  for (int d = full_depth + 1; d <= depth; ++d)
    if (N.offsets[d + 1] > N.offsets[d]) top = d;
  BroodLevels L{};
  L.depth = top;
  for (int d = 0; d <= top; ++d) L.base[d + 1] = L.base[d] + brood_words(d);
  for (int d = top + 1; d <= kBitmapDepth; ++d) L.base[d + 1] = L.base[d];
  const int64_t words = L.base[top + 1];
  DBuf<uint32_t> bits(words, s);
  bits.zero();
  coarse_bits_kernel<<<blocks_for(L.base[full_depth + 1]), kThreads, 0, s>>>(L, full_depth, bits.p);
  PSR_LAUNCH_CHECK();
  if (N.count) {
    seed_bits_kernel<T><<<blocks_for(N.count), kThreads, 0, s>>>(N.keys.p, N.values.p, N.count, L, bits.p);
    PSR_LAUNCH_CHECK();
  }
  // tree.py:171-182: above the base depth the requests of a level are the finer level's broods
  // (their parents are among the dilated ones); from the base depth down they are the halved
  // requests of the level before, and the finer broods only add their parents.
  DBuf<uint32_t> requests;
  int requests_depth = -1;  // the level whose brood grid `requests` is on; -1: none
  for (int d = top - 1; d >= 0; --d) {
    const uint32_t* finer = bits.p + L.base[d + 1];
    const unsigned blocks = blocks_for(brood_words(d + 1));
    if (d > base_depth) {
      parent_bits_kernel<<<blocks, kThreads, 0, s>>>(finer, d, 1, bits.p + L.base[d]);
      PSR_LAUNCH_CHECK();
      continue;
    }
    parent_bits_kernel<<<blocks, kThreads, 0, s>>>(finer, d, 0, bits.p + L.base[d]);
    PSR_LAUNCH_CHECK();
    // level d + 1's requests: level d + 2's broods (none past the finest level), or the last halving
    const bool first = d == base_depth;
    if (first ? d + 2 > top : requests_depth < 0) continue;
    DBuf<uint32_t> halved(brood_words(d + 1), s);
    halved.zero();
    parent_bits_kernel<<<blocks_for(brood_words(d + 2)), kThreads, 0, s>>>(first ? bits.p + L.base[d + 2] : requests.p,
                                                                            d + 1, 0, halved.p);
    PSR_LAUNCH_CHECK();
    parent_bits_kernel<<<blocks, kThreads, 0, s>>>(halved.p, d, 1, bits.p + L.base[d]);
    PSR_LAUNCH_CHECK();
    requests = std::move(halved);
    requests_depth = d + 1;
  }
  DBuf<int32_t> prefix(words, s);  // broods of every word, summed in place
  DBuf<int> totals(2 * (top + 1), s);  // broods through each level, basis nodes of each level
  totals.zero();
  brood_count_kernel<<<blocks_for(words), kThreads, 0, s>>>(bits.p, L, words, prefix.p, totals.p + top + 1);
  PSR_LAUNCH_CHECK();
  inclusive_sum(prefix.p, prefix.p, words, s);
  brood_totals_kernel<<<1, 32, 0, s>>>(prefix.p, L, totals.p);
  PSR_LAUNCH_CHECK();
  const std::vector<int> total = read_vector(totals.p, 2 * (top + 1), s);
  TreeOut out{};
  int64_t broods = 0, basis = 0;
  for (int d = 0; d <= top; ++d) {
    out.brood0[d] = broods;
    out.basis0[d] = basis;
    tree.support_count[d] = 8 * (total[d] - broods);
    tree.basis_count[d] = total[top + 1 + d];
    tree.support[d].alloc(tree.support_count[d], s);
    tree.basis[d].alloc(tree.basis_count[d], s);
    out.support[d] = tree.support[d].p;
    out.basis[d] = tree.basis[d].p;
    broods = total[d];
    basis += tree.basis_count[d];
  }
  if (!broods) return tree;
  DBuf<int4> list(broods, s);
  brood_emit_kernel<<<blocks_for(words), kThreads, 0, s>>>(bits.p, prefix.p, L, words, list.p);
  PSR_LAUNCH_CHECK();
  DBuf<int32_t> mark(8 * broods, s), rank(8 * broods, s);
  brood_expand_kernel<<<blocks_for(broods), kThreads, 0, s>>>(list.p, broods, prefix.p, L, out, mark.p);
  PSR_LAUNCH_CHECK();
  inclusive_sum(mark.p, rank.p, 8 * broods, s);
  brood_basis_kernel<<<blocks_for(8 * broods), kThreads, 0, s>>>(mark.p, rank.p, 8 * broods, top, out);
  PSR_LAUNCH_CHECK();
  return tree;
}

template <class T>
TreeData build_tree(const NormalData<T>& N, int depth, int full_depth, int base_depth, cudaStream_t s) {
  // PSR_TREE=sort takes the sorts at any depth (test override: the path of deeper trees on
  // small cases).
  const char* mode = std::getenv("PSR_TREE");
  if (depth <= kBitmapDepth && !(mode && mode[0] == 's'))
    return build_tree_bitmap<T>(N, depth, full_depth, base_depth, s);
  TreeData tree;
  tree.support.resize(depth + 1);
  tree.basis.resize(depth + 1);
  tree.support_count.assign(depth + 1, 0);
  tree.basis_count.assign(depth + 1, 0);
  DBuf<int64_t> broods;  // tree keys of the previous (finer) level's broods = this level's refined nodes
  int64_t nbroods = 0;
  DBuf<int64_t> requests;
  int64_t nrequests = 0;
  bool have_requests = false;
  for (int d = depth; d >= 0; --d) {
    // tree.py:171-182
    const int64_t* parents = broods.p;
    int64_t nparents = nbroods;
    DBuf<int64_t> req_storage;
    const int64_t* req = nullptr;
    if (d > base_depth || !have_requests) {
      req = parents;
      nrequests = nparents;
      have_requests = true;
    } else {
      DBuf<uint64_t> pk(nrequests, s), upk;
      if (nrequests) {
        parent_tree_keys_kernel<<<blocks_for(nrequests), kThreads, 0, s>>>(requests.p, nrequests, pk.p);
        PSR_LAUNCH_CHECK();
      }
      int64_t u = sort_unique(pk, nrequests, 62, ~uint64_t(0), upk, s);
      req_storage.alloc(u, s);
      if (u) {
        u64_to_i64_kernel<<<blocks_for(u), kThreads, 0, s>>>(upk.p, u, req_storage.p);
        PSR_LAUNCH_CHECK();
      }
      nrequests = u;
      req = req_storage.p;
    }
    int64_t nseed = N.offsets[d + 1] - N.offsets[d];
    int cc = d <= full_depth ? (d == 0 ? 2 : (1 << (d - 1)) + 2) : 0;
    int64_t nc = int64_t(cc) * cc * cc;
    int64_t total = nseed + nc + 27 * nrequests + nparents;
    DBuf<uint64_t> cand(total, s);
    int64_t off = 0;
    if (nseed) {
      seed_kernel<T><<<blocks_for(nseed), kThreads, 0, s>>>(N.keys.p + N.offsets[d], N.values.p + 4 * N.offsets[d],
                                                            nseed, d, cand.p);
      PSR_LAUNCH_CHECK();
    }
    off += nseed;
    if (nc) {
      coarse_kernel<<<blocks_for(nc), kThreads, 0, s>>>(d, cc, cand.p + off);
      PSR_LAUNCH_CHECK();
    }
    off += nc;
    if (nrequests) {
      support_kernel<<<blocks_for(nrequests), kThreads, 0, s>>>(req, nrequests, 1, d, cand.p + off);
      PSR_LAUNCH_CHECK();
    }
    off += 27 * nrequests;
    if (nparents) {
      support_kernel<<<blocks_for(nparents), kThreads, 0, s>>>(parents, nparents, 0, d, cand.p + off);
      PSR_LAUNCH_CHECK();
    }
    // Keep the refined-node requests alive for the next (coarser) level.
    DBuf<int64_t> next_requests;
    if (d <= base_depth || true) {
      next_requests.alloc(nrequests, s);
      if (nrequests)
        PSR_CUDA(cudaMemcpyAsync(next_requests.p, req, nrequests * sizeof(int64_t), cudaMemcpyDeviceToDevice, s));
    }
    uint64_t sentinel = uint64_t(1) << (3 * (d + 1));
    DBuf<uint64_t> ub;
    int64_t u = sort_unique(cand, total, 3 * (d + 1) + 1, sentinel, ub, s);
    // tree.py:196-199: expand into sorted children, compact the basis.
    int64_t nch = 8 * u;
    tree.support[d].alloc(nch, s);
    tree.support_count[d] = nch;
    DBuf<int32_t> mark(nch, s), prefix(nch, s);
    if (u) {
      expand_kernel<<<blocks_for(u), kThreads, 0, s>>>(ub.p, u, d, tree.support[d].p, mark.p);
      PSR_LAUNCH_CHECK();
      inclusive_sum(mark.p, prefix.p, nch, s);
      int64_t nb = read_scalar(prefix.p + nch - 1, s);
      tree.basis[d].alloc(nb, s);
      tree.basis_count[d] = nb;
      basis_fill_kernel<<<blocks_for(nch), kThreads, 0, s>>>(tree.support[d].p, mark.p, prefix.p, nch, d,
                                                             tree.basis[d].p);
      PSR_LAUNCH_CHECK();
    }
    DBuf<int64_t> nb_keys(u, s);
    if (u) {
      broods_to_tree_keys_kernel<<<blocks_for(u), kThreads, 0, s>>>(ub.p, u, d, nb_keys.p);
      PSR_LAUNCH_CHECK();
    }
    requests = std::move(next_requests);
    broods = std::move(nb_keys);
    nbroods = u;
  }
  return tree;
}

template TreeData build_tree<float>(const NormalData<float>&, int, int, int, cudaStream_t);
template TreeData build_tree<double>(const NormalData<double>&, int, int, int, cudaStream_t);

}  // namespace psr
