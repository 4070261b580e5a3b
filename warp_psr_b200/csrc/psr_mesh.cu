// Sparse marching cubes over a regular grid of field values: the consumer of the field that
// warp-psr ships as extract_isosurface / extract_mesh (meshing.py:150-346).
//
// Grid: nx x ny x nz nodes spanning [lower, upper] in model space, node (i, j, k) at
// min(max(lower + step * (i, j, k), lower), upper), step = (upper - lower) / (n - 1) per axis;
// node index (i * ny + j) * nz + k, cell index (i * (ny - 1) + j) * (nz - 1) + k.  Values are
// centred (field - isovalue); a corner is inside when its value is >= 0 and a cell crosses
// the surface when its corners are neither all inside nor all outside (meshing.py:45-60).
//
// Steps (each a kernel or a library scan/sort, all on the caller's stream):
//  1. mark: one bit per crossing cell, from node values of an x-slab (the grid is classified
//     slab by slab so no full-grid value array is needed);
//  2. cells: popcount + scan of the mask words, then the crossing cells' indices in order;
//  3. triangulate: the eight corner values of each crossing cell -> triangles from the case
//     table; a vertex per crossing grid edge, shared by the triangles of every cell around it
//     (sort + unique of the 64-bit edge ids), placed at pa + t (pb - pa), t = fa / (fa - fb),
//     on the edge's lower (a) and upper (b) node.
//
// Case table.  Built at compile time from the cube's faces instead of a stored list: on each
// face, walking its corners counter-clockwise as seen from outside, every maximal run of
// inside corners gives one contour segment from the edge entering the run to the edge leaving
// it (a face whose inside corners are diagonal gets two segments: the inside corners are kept
// apart).  The segment of a face depends only on that face's four corner signs, so the two
// cells sharing a face cut it identically and the mesh has no cracks.  Segments chain into
// closed loops (an edge left on one face is entered on the other face holding it); each loop
// is a fan of triangles, oriented with their normals pointing from the inside (>= iso)
// toward the outside -- outward for the reconstructed indicator, which is larger inside.
#include "../../include/psr_b200.h"
#include "psr_internal.cuh"

#include <cmath>
#include <cstring>
#include <memory>
#include <string>

namespace psr {
namespace mc {

// Corner c of a cell at offset (x, y, z) (meshing.py:31-35 order: 000,100,110,010,001,...).
constexpr int kCorner[8][3] = {{0, 0, 0}, {1, 0, 0}, {1, 1, 0}, {0, 1, 0}, {0, 0, 1}, {1, 0, 1}, {1, 1, 1}, {0, 1, 1}};
// Edge e joins corners kEdge[e][0] (lower node along the edge's axis) and kEdge[e][1].
constexpr int kEdge[12][2] = {{0, 1}, {3, 2}, {0, 3}, {1, 2}, {4, 5}, {7, 6}, {4, 7}, {5, 6},
                              {0, 4}, {1, 5}, {3, 7}, {2, 6}};
// Faces, corners counter-clockwise as seen from outside the cell.
constexpr int kFace[6][4] = {{0, 3, 2, 1}, {4, 5, 6, 7}, {0, 1, 5, 4}, {3, 7, 6, 2}, {0, 4, 7, 3}, {1, 2, 6, 5}};
constexpr int kMaxTriangles = 8;

struct Tables {
  int8_t tri[256][3 * kMaxTriangles];  // edges of each triangle
  uint8_t count[256];                  // triangles per case
  int max_count;
  int8_t corner[8][3];                 // kCorner and kEdge for device code
  int8_t edge[12][2];
};

constexpr int edge_of(int a, int b) {
  for (int e = 0; e < 12; ++e)
    if ((kEdge[e][0] == a && kEdge[e][1] == b) || (kEdge[e][0] == b && kEdge[e][1] == a)) return e;
  return -1;
}

// Loops of one case as edge sequences; returns the loop count.
constexpr int case_loops(int code, int loops[6][13], int lengths[6]) {
  int entry[24] = {}, exit_[24] = {}, ns = 0;
  for (int f = 0; f < 6; ++f)
    for (int i = 0; i < 4; ++i) {
      const int c = kFace[f][i], prev = kFace[f][(i + 3) % 4];
      if (!((code >> c) & 1) || ((code >> prev) & 1)) continue;  // not the first corner of an inside run
      int j = i;
      while ((code >> kFace[f][(j + 1) % 4]) & 1) j = (j + 1) % 4;
      entry[ns] = edge_of(prev, c);
      exit_[ns] = edge_of(kFace[f][j], kFace[f][(j + 1) % 4]);
      ++ns;
    }
  bool used[24] = {};
  int nl = 0;
  for (int s = 0; s < ns; ++s) {
    if (used[s]) continue;
    int len = 0, cur = s;
    loops[nl][len++] = entry[s];
    while (true) {
      used[cur] = true;
      const int e = exit_[cur];
      if (e == loops[nl][0]) break;
      loops[nl][len++] = e;
      int next = -1;
      for (int t = 0; t < ns; ++t)
        if (!used[t] && entry[t] == e) next = t;
      if (next < 0) break;  // unreachable: every exit edge is some face's entry edge
      cur = next;
    }
    lengths[nl++] = len;
  }
  return nl;
}

constexpr double edge_mid(int e, int axis) {
  return 0.5 * (kCorner[kEdge[e][0]][axis] + kCorner[kEdge[e][1]][axis]);
}

constexpr Tables build_tables() {
  Tables t = {};
  for (int c = 0; c < 8; ++c)
    for (int a = 0; a < 3; ++a) t.corner[c][a] = int8_t(kCorner[c][a]);
  for (int e = 0; e < 12; ++e)
    for (int k = 0; k < 2; ++k) t.edge[e][k] = int8_t(kEdge[e][k]);
  // Orientation: the fan of case 1 (corner 0 inside) must face away from corner 0.
  bool flip = false;
  {
    int loops[6][13] = {}, lengths[6] = {};
    case_loops(1, loops, lengths);
    double a[3] = {}, b[3] = {}, c[3] = {};
    for (int k = 0; k < 3; ++k) {
      a[k] = edge_mid(loops[0][0], k);
      b[k] = edge_mid(loops[0][1], k);
      c[k] = edge_mid(loops[0][2], k);
    }
    const double u[3] = {b[0] - a[0], b[1] - a[1], b[2] - a[2]}, v[3] = {c[0] - a[0], c[1] - a[1], c[2] - a[2]};
    const double n[3] = {u[1] * v[2] - u[2] * v[1], u[2] * v[0] - u[0] * v[2], u[0] * v[1] - u[1] * v[0]};
    flip = n[0] + n[1] + n[2] < 0.0;  // away from corner 0 = toward +x+y+z
  }
  t.max_count = 0;
  for (int code = 0; code < 256; ++code) {
    for (int i = 0; i < 3 * kMaxTriangles; ++i) t.tri[code][i] = -1;
    int loops[6][13] = {}, lengths[6] = {};
    const int nl = case_loops(code, loops, lengths);
    int n = 0;
    for (int l = 0; l < nl; ++l)
      for (int k = 1; k + 1 < lengths[l]; ++k) {
        if (n < kMaxTriangles) {
          t.tri[code][3 * n] = int8_t(loops[l][0]);
          t.tri[code][3 * n + 1] = int8_t(loops[l][flip ? k + 1 : k]);
          t.tri[code][3 * n + 2] = int8_t(loops[l][flip ? k : k + 1]);
        }
        ++n;
      }
    t.count[code] = uint8_t(n);
    if (n > t.max_count) t.max_count = n;
  }
  return t;
}

constexpr Tables kTables = build_tables();
static_assert(kTables.max_count <= kMaxTriangles, "a case has more triangles than the table holds");
static_assert(kTables.count[0] == 0 && kTables.count[255] == 0 && kTables.count[1] == 1, "case table");
__constant__ Tables c_tables = kTables;

struct Grid {
  int64_t nx, ny, nz;
  double lower[3], upper[3], step[3];
};

// Model-space position of node (i, j, k) in the field's precision (meshing.py:38-42,88-94).
template <class T>
__device__ __forceinline__ void node_point(const Grid& g, int64_t i, int64_t j, int64_t k, T p[3]) {
  const int64_t c[3] = {i, j, k};
  for (int a = 0; a < 3; ++a) {
    const T lo = T(g.lower[a]), hi = T(g.upper[a]);
    const T v = lo + T(g.step[a]) * T(c[a]);
    p[a] = v < lo ? lo : (v > hi ? hi : v);
  }
}

__device__ __forceinline__ void cell_coords(const Grid& g, int64_t cell, int64_t c[3]) {
  c[2] = cell % (g.nz - 1);
  c[1] = (cell / (g.nz - 1)) % (g.ny - 1);
  c[0] = cell / ((g.nz - 1) * (g.ny - 1));
}

// Nodes of x-planes [start, start + width] (slab) or the eight corners of each listed cell:
// their model positions (for a caller's field callback).
template <class T>
__global__ void points_kernel(Grid g, const int64_t* cells, int64_t start, int64_t count, T* points) {
  const int64_t i = blockIdx.x * int64_t(blockDim.x) + threadIdx.x;
  if (i >= count) return;
  int64_t c[3];
  if (cells) {
    cell_coords(g, cells[i / 8], c);
    for (int a = 0; a < 3; ++a) c[a] += c_tables.corner[i % 8][a];
  } else {
    c[0] = start + i / (g.ny * g.nz);
    c[1] = (i / g.nz) % g.ny;
    c[2] = i % g.nz;
  }
  node_point(g, c[0], c[1], c[2], points + 3 * i);
}

// The same points evaluated on the library's own field, centred: value - iso (meshing.py:114-118).
template <class T>
__global__ void field_values_kernel(psr_field_handle h, Grid g, const int64_t* cells, int64_t start, int64_t count,
                                    T iso, T* values) {
  const int64_t i = blockIdx.x * int64_t(blockDim.x) + threadIdx.x;
  if (i >= count) return;
  int64_t c[3];
  if (cells) {
    cell_coords(g, cells[i / 8], c);
    for (int a = 0; a < 3; ++a) c[a] += c_tables.corner[i % 8][a];
  } else {
    c[0] = start + i / (g.ny * g.nz);
    c[1] = (i / g.nz) % g.ny;
    c[2] = i % g.nz;
  }
  T p[3];
  node_point(g, c[0], c[1], c[2], p);
  values[i] = psr_field::evaluate<T>(h, p[0], p[1], p[2]).value - iso;
}

// The same values for the nodes of x-planes [start, start + planes), one block per brick of at
// most kBrickNodes neighbouring nodes.  Neighbouring nodes read the same few basis functions, and
// a hash probe of a function costs a chain of dependent instructions and a scattered load: the
// block looks every function of the brick's cells up once per level into shared memory (about
// one probe per node where the nodes are as far apart as the finest cells) and the nodes take
// their leaf and their three levels of corners from there, with evaluate_cube's arithmetic in its
// order.  Bound by instruction issue.  A torus at depth 8 on a 301 x 257 x 129 grid, all slabs:
// 1,937 us with a thread's own ~33 probes per node, 952 us so.  A block whose cells exceed
// `cap` functions (rounding of the host's count) evaluates its nodes the direct way.
constexpr int kBrickNodes = 1024, kBrickThreads = 256, kBrickPer = kBrickNodes / kBrickThreads;
constexpr int kMaxLevels = 16;

struct Brick {
  int bx, by, bz;        // nodes of one brick
  int64_t ny_b, nz_b;    // bricks along y and z
  int64_t planes;
};

template <class T>
__device__ __forceinline__ int cell_of(T p, int n) {  // evaluate_cube's left-owned cell
  return min(max(int(ceil(psr_field::mul(p, T(n)))) - 1, 0), n - 1);
}

template <class T>
__global__ void __launch_bounds__(kBrickThreads) brick_values_kernel(psr_field_handle h, Grid g, Brick b, int64_t start,
                                                                     T iso, int cap, T* values) {
  extern __shared__ __align__(16) unsigned char brick_smem[];
  T* s_coef = reinterpret_cast<T*>(brick_smem);
  T* s_cum = s_coef + cap;
  uint8_t* s_has = reinterpret_cast<uint8_t*>(s_cum + cap);
  __shared__ T s_lim[kBrickThreads / 32][6];
  __shared__ int s_lo[kMaxLevels][3], s_dim[kMaxLevels][3], s_off[kMaxLevels + 1];
  const psr_field::View<T> f = psr_field::view<T>(h);
  const int64_t bz0 = (blockIdx.x % b.nz_b) * b.bz, by0 = (blockIdx.x / b.nz_b % b.ny_b) * b.by,
                bx0 = (blockIdx.x / b.nz_b / b.ny_b) * b.bx;
  T L[9], tr[3];
  for (int a = 0; a < 9; ++a) L[a] = T(h.linear[a]);
  for (int a = 0; a < 3; ++a) tr[a] = T(h.translation[a]);
  T p[kBrickPer][3], lim[6];
  int64_t out[kBrickPer];  // the node's place in `values`, -1 past the brick or the grid
  bool in[kBrickPer];
  for (int a = 0; a < 3; ++a) {
    lim[a] = T(INFINITY);
    lim[3 + a] = T(-INFINITY);
  }
#pragma unroll
  for (int u = 0; u < kBrickPer; ++u) {
    const int e = int(threadIdx.x) + u * kBrickThreads;
    const int64_t k = bz0 + e % b.bz, j = by0 + e / b.bz % b.by, i = bx0 + e / b.bz / b.by;
    out[u] = -1;
    in[u] = false;
    if (e >= b.bx * b.by * b.bz || k >= g.nz || j >= g.ny || i >= b.planes) continue;
    out[u] = (i * g.ny + j) * g.nz + k;
    T q[3];
    node_point(g, start + i, j, k, q);
    psr_field::to_cube(L, tr, q, p[u]);
    in[u] = psr_field::inside(p[u]);
    if (!in[u]) continue;
    for (int a = 0; a < 3; ++a) {
      lim[a] = dmin(lim[a], p[u][a]);
      lim[3 + a] = dmax(lim[3 + a], p[u][a]);
    }
  }
  for (int a = 0; a < 6; ++a)
    for (int o = 16; o > 0; o >>= 1) {
      const T v = __shfl_xor_sync(0xffffffffu, lim[a], o);
      lim[a] = a < 3 ? dmin(lim[a], v) : dmax(lim[a], v);
    }
  if ((threadIdx.x & 31) == 0)
    for (int a = 0; a < 6; ++a) s_lim[threadIdx.x >> 5][a] = lim[a];
  __syncthreads();
  for (int a = 0; a < 6; ++a)
    for (int w = 0; w < kBrickThreads / 32; ++w) lim[a] = a < 3 ? dmin(lim[a], s_lim[w][a]) : dmax(lim[a], s_lim[w][a]);
  const bool any = lim[0] <= lim[3];
  if (any && threadIdx.x <= unsigned(f.depth))
    for (int a = 0; a < 3; ++a) {
      const int n = 1 << threadIdx.x, lo = cell_of(lim[a], n);
      s_lo[threadIdx.x][a] = lo;
      s_dim[threadIdx.x][a] = cell_of(lim[3 + a], n) - lo + 2;  // both corners of every cell
    }
  __syncthreads();
  if (threadIdx.x == 0) {  // deepest level first: it holds most of the functions
    int64_t total = 0;
    for (int d = f.depth; any && d >= 0; --d) {
      s_off[d] = int(total);
      total += int64_t(s_dim[d][0]) * s_dim[d][1] * s_dim[d][2];
      if (total > cap) break;
    }
    s_off[kMaxLevels] = total > cap ? -1 : int(total);
  }
  __syncthreads();
  const int total = s_off[kMaxLevels];
  const bool cached = total >= 0;
  constexpr int kAhead = 4;  // probes in flight per thread: a probe waits for L2
  for (int e0 = threadIdx.x; e0 < total; e0 += kAhead * kBrickThreads) {
    int64_t key[kAhead];
    uint64_t slot[kAhead];
    longlong2 probe[kAhead];
#pragma unroll
    for (int u = 0; u < kAhead; ++u) {
      const int e = e0 + u * kBrickThreads;
      key[u] = -1;
      if (e >= total) continue;
      int d = f.depth;
      while (d > 0 && e >= s_off[d - 1]) --d;
      const unsigned r = unsigned(e - s_off[d]), dz = unsigned(s_dim[d][2]), dy = unsigned(s_dim[d][1]);
      const unsigned row = r / dz, x = row / dy;
      key[u] = psr_field::basis_key(d, s_lo[d][0] + int(x), s_lo[d][1] + int(row - x * dy),
                                    s_lo[d][2] + int(r - row * dz));
      slot[u] = psr_field::hash_mix(uint64_t(key[u])) & f.mask;
      probe[u] = __ldg(f.slots + slot[u]);
    }
#pragma unroll
    for (int u = 0; u < kAhead; ++u) {
      if (key[u] < 0) continue;
      while (probe[u].x != key[u] && probe[u].x != -1) {
        slot[u] = (slot[u] + 1) & f.mask;
        probe[u] = __ldg(f.slots + slot[u]);
      }
      const int e = e0 + u * kBrickThreads;
      const bool have = probe[u].x == key[u];
      s_has[e] = have;
      if (have) {
        s_coef[e] = __ldg(f.coefficients + probe[u].y);
        s_cum[e] = __ldg(f.cumulative + probe[u].y);
      }
    }
  }
  __syncthreads();
  // one level's value at p from the brick's functions (psr_field::add_level's r[0])
  auto level_value = [&](const T* coeff, const T q[3], int d) {
    const int n = 1 << d;
    T fr[3];
    int base[3], rel[3];
    for (int a = 0; a < 3; ++a) {
      const T t = psr_field::mul(q[a], T(n));
      const int cell = min(max(int(ceil(t)) - 1, 0), n - 1);
      base[a] = int(floor(t)) - cell;  // 0, or 1 on the cell's upper face
      fr[a] = psr_field::sub(t, T(int(floor(t))));
      rel[a] = cell - s_lo[d][a];
    }
    const int dz = s_dim[d][2], dy = s_dim[d][1];
    const int e0 = s_off[d] + (rel[0] * dy + rel[1]) * dz + rel[2];
    T r = T(0);
#pragma unroll
    for (int corner = 0; corner < 8; ++corner) {
      const int o[3] = {corner / 4, (corner / 2) % 2, corner % 2};
      if (min(o[0] - base[0], min(o[1] - base[1], o[2] - base[2])) < 0) continue;
      const int e = e0 + (o[0] * dy + o[1]) * dz + o[2];
      if (!s_has[e]) continue;
      T hh[3];
      for (int a = 0; a < 3; ++a) hh[a] = o[a] > base[a] ? fr[a] : psr_field::sub(T(1), fr[a]);
      r = psr_field::add(r, psr_field::mul(psr_field::mul(psr_field::mul(coeff[e], hh[0]), hh[1]), hh[2]));
    }
    return r;
  };
#pragma unroll
  for (int u = 0; u < kBrickPer; ++u) {
    if (out[u] < 0) continue;
    T v = T(NAN);
    if (in[u] && cached) {
      int leaf = 0;
      for (int d = f.depth; d >= 0; --d) {
        const int n = 1 << d;
        const int e = s_off[d] + ((cell_of(p[u][0], n) - s_lo[d][0]) * s_dim[d][1] + cell_of(p[u][1], n) - s_lo[d][1]) *
                                     s_dim[d][2] + cell_of(p[u][2], n) - s_lo[d][2];
        if (s_has[e]) {
          leaf = d;
          break;
        }
      }
      for (int a = 0; a < 3; ++a) {  // points on the cube's faces move inside, within their cells
        if (p[u][a] == T(0))
          p[u][a] = T(1e-6);
        else if (p[u][a] == T(1))
          p[u][a] = T(1.0 - 1e-6);
      }
      v = level_value(s_coef, p[u], leaf);
      if (leaf > 0) v = psr_field::add(v, level_value(s_cum, p[u], leaf - 1));
      if (leaf < f.depth) v = psr_field::add(v, level_value(s_coef, p[u], leaf + 1));
    } else if (in[u]) {
      T r[4];
      psr_field::evaluate_cube(f, p[u], r);
      v = r[0];
    }
    values[out[u]] = v - iso;
  }
}

// Crossing cells of the slab [start, start + width) from its nodes' values (meshing.py:45-60).
template <class T>
__global__ void mark_kernel(const T* values, Grid g, int64_t start, int64_t width, uint32_t* mask, int* status) {
  const int64_t i = blockIdx.x * int64_t(blockDim.x) + threadIdx.x;
  const int64_t ny = g.ny, nz = g.nz;
  if (i >= width * (ny - 1) * (nz - 1)) return;
  const int64_t x = i / ((ny - 1) * (nz - 1)), y = (i / (nz - 1)) % (ny - 1), z = i % (nz - 1);
  // every corner's offset from the cell's first node is a constant choice of strides, so the eight
  // loads go out together (19 slabs of a 301 x 257 x 129 grid: 159 -> 100 us)
  const T* node = values + (x * ny + y) * nz + z;
  int code = 0;
  bool finite = true;
#pragma unroll
  for (int c = 0; c < 8; ++c) {
    const T v = node[((c + 1) >> 1 & 1 ? ny * nz : 0) + (c >> 1 & 1 ? nz : 0) + (c >> 2)];  // kCorner[c]
    finite = finite && isfinite(v);
    if (v >= T(0)) code |= 1 << c;
  }
  if (!finite) atomicOr(status, 1);
  if (code != 0 && code != 255) {
    const int64_t index = ((start + x) * (ny - 1) + y) * (nz - 1) + z;
    atomicOr(mask + index / 32, 1u << (index % 32));
  }
}

__global__ void popc_kernel(const uint32_t* mask, int64_t words, int64_t* counts) {
  const int64_t i = blockIdx.x * int64_t(blockDim.x) + threadIdx.x;
  if (i < words) counts[i] = __popc(mask[i]);
}

// Crossing cell indices in ascending order (inclusive word offsets).
__global__ void emit_cells_kernel(const uint32_t* mask, const int64_t* inclusive, int64_t words, int64_t* cells) {
  const int64_t i = blockIdx.x * int64_t(blockDim.x) + threadIdx.x;
  if (i >= words) return;
  uint32_t bits = mask[i];
  int64_t out = inclusive[i] - __popc(bits);
  while (bits) {
    const int b = __ffs(bits) - 1;
    cells[out++] = i * 32 + b;
    bits &= bits - 1;
  }
}

template <class T>
__device__ __forceinline__ int cube_code(const T* v) {
  int code = 0;
  for (int c = 0; c < 8; ++c)
    if (v[c] >= T(0)) code |= 1 << c;
  return code;
}

template <class T>
__global__ void triangle_count_kernel(const T* corner_values, int64_t count, int64_t* triangles) {
  const int64_t i = blockIdx.x * int64_t(blockDim.x) + threadIdx.x;
  if (i < count) triangles[i] = c_tables.count[cube_code(corner_values + 8 * i)];
}

// Triangle corners of every crossing cell: the global id of the crossing edge, (node index of
// its lower node) * 3 + axis, and the flat corner-value indices of the edge's two nodes.
template <class T>
__global__ void triangle_emit_kernel(Grid g, const int64_t* cells, const T* corner_values, int64_t count,
                                     const int64_t* first, int64_t* edge_ids, int64_t* record_ids, int64_t* ends) {
  const int64_t i = blockIdx.x * int64_t(blockDim.x) + threadIdx.x;
  if (i >= count) return;
  const int code = cube_code(corner_values + 8 * i);
  int64_t c[3];
  cell_coords(g, cells[i], c);
  const int n = c_tables.count[code];
  for (int k = 0; k < 3 * n; ++k) {
    const int e = c_tables.tri[code][k];
    const int a = c_tables.edge[e][0], b = c_tables.edge[e][1];
    int axis = 0;
    while (c_tables.corner[a][axis] == c_tables.corner[b][axis]) ++axis;
    const int64_t node = ((c[0] + c_tables.corner[a][0]) * g.ny + c[1] + c_tables.corner[a][1]) * g.nz + c[2] + c_tables.corner[a][2];
    const int64_t r = 3 * first[i] + k;
    edge_ids[r] = node * 3 + axis;
    record_ids[r] = r;
    ends[2 * r] = 8 * i + a;
    ends[2 * r + 1] = 8 * i + b;
  }
}

// Sorted triangle corners -> vertex number of each (0-based, by first occurrence in edge order).
__global__ void vertex_flags_kernel(const int64_t* sorted_edges, int64_t n, int64_t* flags) {
  const int64_t i = blockIdx.x * int64_t(blockDim.x) + threadIdx.x;
  if (i < n) flags[i] = (i == 0 || sorted_edges[i] != sorted_edges[i - 1]) ? 1 : 0;
}

// One vertex per crossing edge at pa + t (pb - pa), t = fa / (fa - fb); triangle indices.
template <class T>
__global__ void vertex_kernel(Grid g, const int64_t* sorted_edges, const int64_t* sorted_records, const int64_t* number,
                              int64_t n, const int64_t* ends, const T* corner_values, T* vertices, int64_t* vertex_edges,
                              int64_t* vertex_ends, int32_t* indices) {
  const int64_t i = blockIdx.x * int64_t(blockDim.x) + threadIdx.x;
  if (i >= n) return;
  const int64_t v = number[i] - 1;
  const int64_t r = sorted_records[i];
  indices[r] = int32_t(v);
  if (i != 0 && sorted_edges[i] == sorted_edges[i - 1]) return;
  const int64_t edge = sorted_edges[i], node = edge / 3;
  const int axis = int(edge % 3);
  int64_t c[3] = {node / (g.ny * g.nz), (node / g.nz) % g.ny, node % g.nz};
  T pa[3], pb[3];
  node_point(g, c[0], c[1], c[2], pa);
  c[axis] += 1;
  node_point(g, c[0], c[1], c[2], pb);
  const T fa = corner_values[ends[2 * r]], fb = corner_values[ends[2 * r + 1]];
  const T t = fa / (fa - fb);
  for (int a = 0; a < 3; ++a) vertices[3 * v + a] = pa[a] + t * (pb[a] - pa[a]);
  vertex_edges[v] = edge;
  vertex_ends[2 * v] = ends[2 * r];
  vertex_ends[2 * v + 1] = ends[2 * r + 1];
}

}  // namespace mc
}  // namespace psr

// ------------------------------------------------------------------ C ABI
struct psr_mesh {
  int32_t dtype = PSR_FLOAT32;
  int64_t vertices = 0, triangles = 0, cells = 0;
  psr::DBuf<int64_t> cell_ids;     // crossing cells (ascending), psr_extract_mesh only
  psr::DBuf<char> positions;       // vertices x 3 (dtype)
  psr::DBuf<int32_t> indices;      // triangles x 3
  psr::DBuf<int64_t> edges;        // vertices: crossing grid edge of each vertex
  psr::DBuf<int64_t> ends;         // vertices x 2: corner values (flat cell*8 + corner) at its two nodes
};

namespace {
using namespace psr;

mc::Grid make_grid(const int64_t shape[3], const double lower[3], const double upper[3]) {
  if (!shape || !lower || !upper) throw Error(PSR_EINVAL, "shape, lower and upper are required");
  mc::Grid g{};
  g.nx = shape[0];
  g.ny = shape[1];
  g.nz = shape[2];
  for (int a = 0; a < 3; ++a) {
    if (shape[a] < 2) throw Error(PSR_EINVAL, "resolution must be an integer or three integers >= 2");
    if (!std::isfinite(lower[a]) || !std::isfinite(upper[a]) || !(lower[a] < upper[a]))
      throw Error(PSR_EINVAL, "bounds must be finite with lower < upper on every axis");
    g.lower[a] = lower[a];
    g.upper[a] = upper[a];
  }
  // float32 spacing of the grid, as the reference computes it (meshing.py:145-147); float64
  // fields use the same spacing rounded to float64 from it
  for (int a = 0; a < 3; ++a) {
    const float step = (float(upper[a]) - float(lower[a])) / float(shape[a] - 1);
    if (!std::isfinite(step) || !(step > 0.f)) throw Error(PSR_EINVAL, "bounds/spacing must be representable in float32");
    g.step[a] = double(step);
    g.lower[a] = double(float(lower[a]));
    g.upper[a] = double(float(upper[a]));
  }
  if ((g.nx - 1) * (g.ny - 1) * (g.nz - 1) > int64_t(2147483647))
    throw Error(PSR_EINVAL, "extraction cell count exceeds int32 indexing");
  if (g.nx * g.ny * g.nz > int64_t(2147483647)) throw Error(PSR_EINVAL, "grid node count exceeds int32 sampling indices");
  return g;
}

int mesh_fail(const std::exception& e, int code) {
  set_last_error(e.what());
  return code;
}

template <class T>
psr_mesh* triangulate(const mc::Grid& g, const int64_t* cells, const T* cv, int64_t count, cudaStream_t s) {
  auto M = std::make_unique<psr_mesh>();
  M->dtype = sizeof(T) == 8 ? PSR_FLOAT64 : PSR_FLOAT32;
  if (count <= 0) return M.release();
  DBuf<int64_t> tc(count, s), first(count, s);
  mc::triangle_count_kernel<T><<<blocks_for(count), kThreads, 0, s>>>(cv, count, tc.p);
  PSR_LAUNCH_CHECK();
  exclusive_sum(tc.p, first.p, count, s);
  const int64_t tris = read_scalar(first.p + count - 1, s) + read_scalar(tc.p + count - 1, s);
  if (3 * tris > int64_t(2147483647)) throw Error(PSR_EINVAL, "triangle count exceeds int32 indexing");
  M->triangles = tris;
  if (!tris) return M.release();
  const int64_t n = 3 * tris;
  DBuf<int64_t> eid(n, s), rid(n, s), ends(2 * n, s), seid(n, s), srid(n, s), number(n, s);
  mc::triangle_emit_kernel<T><<<blocks_for(count), kThreads, 0, s>>>(g, cells, cv, count, first.p, eid.p, rid.p,
                                                                      ends.p);
  PSR_LAUNCH_CHECK();
  sort_pairs(eid.p, seid.p, rid.p, srid.p, n, bits_for(uint64_t(3 * g.nx * g.ny * g.nz)), s);
  mc::vertex_flags_kernel<<<blocks_for(n), kThreads, 0, s>>>(seid.p, n, number.p);
  PSR_LAUNCH_CHECK();
  inclusive_sum(number.p, number.p, n, s);
  const int64_t nv = read_scalar(number.p + n - 1, s);
  M->vertices = nv;
  M->positions.alloc(3 * nv * int64_t(sizeof(T)), s);
  M->indices.alloc(n, s);
  M->edges.alloc(nv, s);
  M->ends.alloc(2 * nv, s);
  mc::vertex_kernel<T><<<blocks_for(n), kThreads, 0, s>>>(g, seid.p, srid.p, number.p, n, ends.p, cv,
                                                          reinterpret_cast<T*>(M->positions.p), M->edges.p, M->ends.p,
                                                          M->indices.p);
  PSR_LAUNCH_CHECK();
  return M.release();
}

template <class T>
void slab_values(const psr_field_handle& h, const mc::Grid& g, int64_t start, int64_t width, double iso, T* values,
                 cudaStream_t s) {
  const int64_t planes = width + 1, count = planes * g.ny * g.nz;
  // Bricks of about 8 x 8 x 16 nodes, evenly split along each axis.  The functions of a brick's
  // cells, at most: its extent in cells per level, rounded up, and two corners.  The brick kernel
  // is taken while there are at most three per node (grids up to about as coarse as the finest
  // cells).  Extractions with bricks against evaluating every node by itself, five fields at
  // depths 6 to 8, float32 and float64: 0.69 to 0.77 of the time at 0.7 to 2.1 functions per node
  // and a million nodes, 0.76 to 0.99 up to three, 0.84 to 1.00 at three to four, 1.00 beyond 4.4
  // (there float64 bricks of depth 8 no longer fit either).  A depth-8 torus at 1.4 and 2.3 (301
  // and 220 nodes along x): 2,679 -> 1,931 and 1,547 -> 1,161 us.
  auto even = [](int64_t n, int64_t most) { return int((n + (n + most - 1) / most - 1) / ((n + most - 1) / most)); };
  mc::Brick b{even(planes, 8), even(g.ny, 8), even(g.nz, 16), 0, 0, planes};
  b.ny_b = (g.ny + b.by - 1) / b.by;
  b.nz_b = (g.nz + b.bz - 1) / b.bz;
  const int64_t bricks = (planes + b.bx - 1) / b.bx * b.ny_b * b.nz_b;
  const double extent[3] = {g.step[0] * (b.bx - 1), g.step[1] * (b.by - 1), g.step[2] * (b.bz - 1)};
  double functions = 0;
  for (int d = 0; d <= h.depth; ++d) {
    double level = 1;
    for (int r = 0; r < 3; ++r) {
      double e = 0;
      for (int c = 0; c < 3; ++c) e += std::fabs(h.linear[3 * r + c]) * extent[c];
      level *= std::min(std::floor(e * double(1 << d) + 1e-3) + 3, double(1 << d) + 1);
    }
    functions += level;
  }
  const double bytes = functions * (2 * sizeof(T) + 1);
  if (h.depth < mc::kMaxLevels && h.cumulative && h.hash_slots && functions <= 3.0 * b.bx * b.by * b.bz &&
      bytes <= 47 * 1024) {
    int cap = int(functions);
    // PSR_MESH_BRICK_CAP lowers the functions a brick may hold (test override: bricks past the
    // capacity, which the host's count leaves to rounding, and which evaluate node by node).
    if (const char* env = std::getenv("PSR_MESH_BRICK_CAP")) cap = std::min(cap, std::max(std::atoi(env), 0));
    mc::brick_values_kernel<T><<<unsigned(bricks), mc::kBrickThreads, size_t(bytes), s>>>(h, g, b, start, T(iso), cap,
                                                                                          values);
  } else {
    mc::field_values_kernel<T><<<blocks_for(count, 128), 128, 0, s>>>(h, g, nullptr, start, count, T(iso), values);
  }
  PSR_LAUNCH_CHECK();
}

template <class T>
psr_mesh* extract(const psr_field_handle& h, const mc::Grid& g, double iso, int64_t slab, cudaStream_t s,
                  int64_t* retained) {
  const int64_t cells_total = (g.nx - 1) * (g.ny - 1) * (g.nz - 1);
  const int64_t words = (cells_total + 31) / 32;
  DBuf<uint32_t> mask(words, s);
  mask.zero();
  DBuf<int> status(1, s);
  status.zero();
  DBuf<T> values((std::min(slab, g.nx - 1) + 1) * g.ny * g.nz, s);
  for (int64_t start = 0; start < g.nx - 1; start += slab) {
    const int64_t width = std::min(slab, g.nx - 1 - start);
    slab_values<T>(h, g, start, width, iso, values.p, s);
    mc::mark_kernel<T><<<blocks_for(width * (g.ny - 1) * (g.nz - 1)), kThreads, 0, s>>>(values.p, g, start, width,
                                                                                        mask.p, status.p);
    PSR_LAUNCH_CHECK();
  }
  values.release();
  DBuf<int64_t> counts(words, s);
  mc::popc_kernel<<<blocks_for(words), kThreads, 0, s>>>(mask.p, words, counts.p);
  PSR_LAUNCH_CHECK();
  inclusive_sum(counts.p, counts.p, words, s);
  const int64_t count = read_scalar(counts.p + words - 1, s);
  if (read_scalar(status.p, s)) throw Error(PSR_EDATA, "field returned nonfinite values inside extraction bounds");
  *retained = count;
  DBuf<int64_t> cells(count, s);
  DBuf<T> cv(8 * count, s);
  if (count) {
    mc::emit_cells_kernel<<<blocks_for(words), kThreads, 0, s>>>(mask.p, counts.p, words, cells.p);
    PSR_LAUNCH_CHECK();
    mc::field_values_kernel<T><<<blocks_for(8 * count, 128), 128, 0, s>>>(h, g, cells.p, 0, 8 * count, T(iso), cv.p);
    PSR_LAUNCH_CHECK();
  }
  psr_mesh* M = triangulate<T>(g, cells.p, cv.p, count, s);
  M->cells = count;
  M->cell_ids = std::move(cells);
  return M;
}
}  // namespace

extern "C" {

int psr_mc_points(int32_t dtype, const int64_t shape[3], const double lower[3], const double upper[3],
                  const int64_t* cells, int64_t start, int64_t count, void* points, void* stream) {
  try {
    const mc::Grid g = make_grid(shape, lower, upper);
    if (count < 0 || (count > 0 && !points)) throw Error(PSR_EINVAL, "points are required");
    if (count == 0) return PSR_OK;
    cudaStream_t s = (cudaStream_t)stream;
    if (dtype == PSR_FLOAT64)
      mc::points_kernel<double><<<blocks_for(count), kThreads, 0, s>>>(g, cells, start, count, (double*)points);
    else if (dtype == PSR_FLOAT32)
      mc::points_kernel<float><<<blocks_for(count), kThreads, 0, s>>>(g, cells, start, count, (float*)points);
    else
      throw Error(PSR_EINVAL, "dtype must be float32 or float64");
    PSR_LAUNCH_CHECK();
    return PSR_OK;
  } catch (const Error& e) {
    return mesh_fail(e, e.code);
  } catch (const std::exception& e) {
    return mesh_fail(e, PSR_ECUDA);
  }
}

int psr_mc_mark(int32_t dtype, const void* values, const int64_t shape[3], int64_t start, int64_t width,
                uint32_t* mask, int32_t* status, void* stream) {
  try {
    if (!values || !shape || !mask || !status) throw Error(PSR_EINVAL, "values, shape, mask and status are required");
    mc::Grid g{};
    g.nx = shape[0];
    g.ny = shape[1];
    g.nz = shape[2];
    if (g.nx < 2 || g.ny < 2 || g.nz < 2 || start < 0 || width < 1 || start + width > g.nx - 1)
      throw Error(PSR_EINVAL, "slab outside the grid");
    cudaStream_t s = (cudaStream_t)stream;
    const int64_t cells = width * (g.ny - 1) * (g.nz - 1);
    if (dtype == PSR_FLOAT64)
      mc::mark_kernel<double><<<blocks_for(cells), kThreads, 0, s>>>((const double*)values, g, start, width, mask,
                                                                     status);
    else if (dtype == PSR_FLOAT32)
      mc::mark_kernel<float><<<blocks_for(cells), kThreads, 0, s>>>((const float*)values, g, start, width, mask,
                                                                    status);
    else
      throw Error(PSR_EINVAL, "dtype must be float32 or float64");
    PSR_LAUNCH_CHECK();
    return PSR_OK;
  } catch (const Error& e) {
    return mesh_fail(e, e.code);
  } catch (const std::exception& e) {
    return mesh_fail(e, PSR_ECUDA);
  }
}

int psr_mc_cells(const uint32_t* mask, int64_t words, int64_t* cells, int64_t capacity, int64_t* count, void* stream) {
  try {
    if (!mask || !count || words < 0) throw Error(PSR_EINVAL, "mask and count are required");
    cudaStream_t s = (cudaStream_t)stream;
    *count = 0;
    if (!words) return PSR_OK;
    DBuf<int64_t> counts(words, s);
    mc::popc_kernel<<<blocks_for(words), kThreads, 0, s>>>(mask, words, counts.p);
    PSR_LAUNCH_CHECK();
    inclusive_sum(counts.p, counts.p, words, s);
    *count = read_scalar(counts.p + words - 1, s);
    if (cells && *count) {
      if (capacity < *count) throw Error(PSR_EINVAL, "cells capacity is smaller than the crossing cell count");
      mc::emit_cells_kernel<<<blocks_for(words), kThreads, 0, s>>>(mask, counts.p, words, cells);
      PSR_LAUNCH_CHECK();
    }
    return PSR_OK;
  } catch (const Error& e) {
    return mesh_fail(e, e.code);
  } catch (const std::exception& e) {
    return mesh_fail(e, PSR_ECUDA);
  }
}

int psr_mc_triangulate(int32_t dtype, const int64_t shape[3], const double lower[3], const double upper[3],
                       const int64_t* cells, const void* corner_values, int64_t count, psr_mesh** out, void* stream) {
  try {
    if (!out) throw Error(PSR_EINVAL, "out must not be NULL");
    *out = nullptr;
    const mc::Grid g = make_grid(shape, lower, upper);
    if (count < 0 || (count > 0 && (!cells || !corner_values))) throw Error(PSR_EINVAL, "cells and values are required");
    cudaStream_t s = (cudaStream_t)stream;
    if (dtype == PSR_FLOAT64)
      *out = triangulate<double>(g, cells, (const double*)corner_values, count, s);
    else if (dtype == PSR_FLOAT32)
      *out = triangulate<float>(g, cells, (const float*)corner_values, count, s);
    else
      throw Error(PSR_EINVAL, "dtype must be float32 or float64");
    return PSR_OK;
  } catch (const Error& e) {
    return mesh_fail(e, e.code);
  } catch (const std::exception& e) {
    return mesh_fail(e, PSR_ECUDA);
  }
}

int psr_extract_mesh(const psr_result* result, const int64_t shape[3], const double lower[3], const double upper[3],
                     double iso, int64_t slab, int64_t* retained, psr_mesh** out, void* stream) {
  try {
    if (!result || !out || !retained) throw Error(PSR_EINVAL, "result, retained and out are required");
    *out = nullptr;
    if (!std::isfinite(iso)) throw Error(PSR_EINVAL, "iso_value must be finite");
    if (slab < 1) throw Error(PSR_EINVAL, "slab_size must be a positive integer");
    const mc::Grid g = make_grid(shape, lower, upper);
    psr_field_handle h;
    int rc = psr_device_field(result, &h);
    if (rc) return rc;
    cudaStream_t s = (cudaStream_t)stream;
    if (h.dtype == PSR_FLOAT64)
      *out = extract<double>(h, g, iso, slab, s, retained);
    else
      *out = extract<float>(h, g, iso, slab, s, retained);
    return PSR_OK;
  } catch (const Error& e) {
    return mesh_fail(e, e.code);
  } catch (const std::exception& e) {
    return mesh_fail(e, PSR_ECUDA);
  }
}

int psr_mesh_info(const psr_mesh* mesh, int32_t* dtype, int64_t* vertices, int64_t* triangles, int64_t* cells) {
  if (!mesh || !dtype || !vertices || !triangles || !cells) {
    set_last_error("NULL argument");
    return PSR_EINVAL;
  }
  *dtype = mesh->dtype;
  *vertices = mesh->vertices;
  *triangles = mesh->triangles;
  *cells = mesh->cell_ids.p ? mesh->cells : 0;
  return PSR_OK;
}

int psr_mesh_arrays(const psr_mesh* mesh, const void** vertices, const int32_t** indices, const int64_t** edges,
                    const int64_t** ends, const int64_t** cells) {
  if (!mesh || !vertices || !indices || !edges || !ends || !cells) {
    set_last_error("NULL argument");
    return PSR_EINVAL;
  }
  *vertices = mesh->positions.p;
  *indices = mesh->indices.p;
  *edges = mesh->edges.p;
  *ends = mesh->ends.p;
  *cells = mesh->cell_ids.p;
  return PSR_OK;
}

int psr_mesh_free(psr_mesh* mesh) {
  if (!mesh) return PSR_OK;
  cudaDeviceSynchronize();
  delete mesh;
  return PSR_OK;
}

}  // extern "C"
