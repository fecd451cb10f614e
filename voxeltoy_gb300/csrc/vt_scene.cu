// vt_scene.cu — kernels that build the device-resident scene and environment:
//   occupancy bit-bricks, emissive-voxel pruning flags and discovery, the
//   environment map's FP16 texels and importance-sampling CDFs (FP64 prefix
//   sums), and the triangle/voxel-overlap voxelizer.
#include <cuda_fp16.h>
#include <algorithm>
#include "vt_kernels.h"
#include "vt_builtins.h"

namespace vt {

// ------------------------------------------------------------- bit-bricks
// One thread per brick of the padded brick grid (one border brick on every
// side), in the array's order.
// Voxels outside the volume read as occupied, so the DDA stops on the first
// voxel beyond the volume without a separate bounds test.
//
// With `max_entry`, the largest palette entry of the volume is atomically
// max-ed into *max_entry (the host checks it against the palette size).
// Bound by the read of the volume; border bricks are written without a look
// at their voxels, and the indices (below 2^32 bricks) take two high
// multiplies.  Call with allocation and wait, us: 256^3, 1024^3 and 1048574x1x1
// with 64-bit divisions and every voxel of the border looked at 41, 699 and
// 184; without, a warp to a row and eight rows a block, whose reads lie further
// apart and which leaves a volume along x to a few warps, 27, 840 and 15294;
// now 20, 386 and 36 (a volume just uploaded is read in one round trip to
// memory: 64^3 scenes build 8 us faster than with the loads in turns).
constexpr int kBrickThreads = 256;
__global__ void __launch_bounds__(kBrickThreads) k_build_bricks(const uint8_t* __restrict__ grid, int32_t rx,
                                                                int32_t ry, int32_t rz,
                                                                unsigned long long* __restrict__ bricks, int32_t bx,
                                                                int32_t by, int32_t bz, uint64_t m_px, uint64_t m_pxy,
                                                                const BrickShape sh, unsigned long long* max_entry) {
  const uint32_t px = bx + 2, pxy = px * (uint32_t)(by + 2);
  const uint32_t b = blockIdx.x * kBrickThreads + threadIdx.x;
  unsigned top = 0;
  const int iz = (int)udiv(b, m_pxy);
  if (iz < bz + 2) {
    const uint32_t r = b - (uint32_t)iz * pxy;
    const int iy = (int)udiv(r, m_px), ix = (int)(r - (uint32_t)iy * px);
    unsigned long long w = 0ull;
    const int ex = 1 << sh.sx, ey = 1 << sh.sy, ez = 1 << sh.sz;
    const int x0 = (ix - 1) * ex, y0 = (iy - 1) * ey, z0 = (iz - 1) * ez;
    if (ix == 0 || iy == 0 || iz == 0 || ix > bx || iy > by || iz > bz) {
      w = ~0ull;   // border
    } else if (sh.sx == 2 && sh.sy == 2 && (rx & 3) == 0) {
      // 4x4x4 bricks: rows of four voxels as one aligned 32-bit word where
      // rows start on 4-byte boundaries; the sixteen loads are issued before
      // any is used
      uint32_t v4[16];
#pragma unroll
      for (int k = 0; k < 16; ++k) {
        const int y = y0 + (k & 3), z = z0 + (k >> 2);
        v4[k] = y < ry && z < rz
                    ? *reinterpret_cast<const uint32_t*>(grid + (size_t)x0 + (size_t)rx * ((size_t)y + (size_t)ry * (size_t)z))
                    : ~0u;
      }
      unsigned tops = 0u;   // byte-wise maximum of the word rows
#pragma unroll
      for (int k = 0; k < 16; ++k) {
        const bool in = y0 + (k & 3) < ry && z0 + (k >> 2) < rz;
        tops = __vmaxu4(tops, in ? v4[k] : 0u);
        uint32_t m = __vcmpne4(v4[k], 0u) & 0x01010101u;   // bit 0 of each non-zero byte
        m = (m | (m >> 7) | (m >> 14) | (m >> 21)) & 0xfu;
        w |= (unsigned long long)m << (4 * k);             // rows outside the volume read as set
      }
      for (int k = 0; k < 32; k += 8) top = max(top, (tops >> k) & 0xffu);
    } else {
      for (int k = 0; k < 64; ++k) {
        const int x = x0 + (k & (ex - 1)), y = y0 + ((k >> sh.sx) & (ey - 1)), z = z0 + (k >> (sh.sx + sh.sy));
        const bool outside = x >= rx || y >= ry || z >= rz;
        const unsigned v = outside ? 0u : grid[(size_t)x + (size_t)rx * ((size_t)y + (size_t)ry * (size_t)z)];
        top = v > top ? v : top;
        if (outside || v != 0) w |= 1ull << k;
      }
    }
    bricks[b] = w;
  }
  if (!max_entry) return;
  // one atomic a block, and only where it would raise the maximum
  __shared__ unsigned s_top[kBrickThreads / 32];
  top = __reduce_max_sync(0xffffffffu, top);
  if ((threadIdx.x & 31) == 0) s_top[threadIdx.x >> 5] = top;
  __syncthreads();
  if (threadIdx.x != 0) return;
  for (unsigned t : s_top) top = max(top, t);
  if (top > *(volatile unsigned long long*)max_entry) atomicMax(max_entry, (unsigned long long)top);
}

// ------------------------------------------------------------- free cubes
// Per 4x4x4 brick and octant, the side in bricks of an empty cube of bricks
// that starts with the brick and extends towards the octant: 1, 2, 3, 4, 6, 8,
// 12 or 16, the largest of these that is empty.  The DDA crosses such a cube
// in one leap (dda_leap).
//
// A bitmap per side over the padded brick rows, 32 bricks a word, bit set:
// the cube of that side from the brick towards +x, +y, +z is empty (bricks
// beyond the padded array count as occupied).  The cube towards another
// octant is the same cube seen from its other end, so eight bitmaps serve the
// eight octants.  Three passes of word operations and one that turns bits
// into bytes: 1024^3 (17 M bricks) takes about as long as reading the bricks
// and writing the bytes.
constexpr int kCubeSides = 8;
__device__ constexpr int kCubeSide[kCubeSides] = {1, 2, 3, 4, 6, 8, 12, 16};   // free_cube_side of 1 .. 8
static int64_t cube_words(int32_t bx) { return ((int64_t)bx + 2 + 31) / 32; }
size_t free_cube_scratch_bytes(int32_t bx, int32_t by, int32_t bz) {
  return sizeof(uint32_t) * (kCubeSides * (size_t)(cube_words(bx) * (by + 2) * (bz + 2)) + 32);
}

// Side 1, one warp per word: bit i set if brick 32 w + i of the row is empty.
// (A bitmap has fewer than 2^31 words: 32-bit indices and divisions.)  Bound by
// the read of the bricks, so a warp has four words' reads under way (one: 41 us
// for 1024^3, four: 27).
__global__ void __launch_bounds__(256) k_cubes_1(const unsigned long long* __restrict__ bricks, int32_t px, uint32_t n,
                                                 uint32_t words, uint32_t* __restrict__ e1) {
  const int lane = threadIdx.x & 31;
  const uint32_t warps = gridDim.x * (blockDim.x >> 5);
  for (uint32_t i0 = 4 * (blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5)); i0 < n; i0 += 4 * warps) {
    unsigned long long v[4];
#pragma unroll
    for (uint32_t k = 0; k < 4; ++k) {
      const uint32_t r = (i0 + k) / words;
      const int x = (int)(i0 + k - r * words) * 32 + lane;
      v[k] = i0 + k < n && x < px ? bricks[(int64_t)r * px + x] : ~0ull;
    }
#pragma unroll
    for (uint32_t k = 0; k < 4; ++k) {
      const uint32_t w = __ballot_sync(0xffffffffu, v[k] == 0ull);
      if (lane == 0 && i0 + k < n) e1[i0 + k] = w;
    }
  }
}

// 64 bricks of row (y, z) from word w on; none beyond the array.
__device__ __forceinline__ unsigned long long cube_bits(const uint32_t* __restrict__ e, int w, int y, int z, int32_t words,
                                                        int32_t py, int32_t pz) {
  if (y >= py || z >= pz) return 0ull;
  const uint32_t* r = e + ((int64_t)z * py + y) * words + w;
  return (unsigned long long)r[0] | (w + 1 < words ? (unsigned long long)r[1] << 32 : 0ull);
}

// Sides 2, 3 and 4 from side 1, and behind the bitmaps the number of bricks
// that start a cube of side 4 (in 32 parts); sides 6, 8, 12 and 16 from sides 3 and 4.
// A thread takes a word of kRun slices in turn: the bits of four rows of
// a slice make its squares, the squares of up to four slices the cubes, so a
// word costs four rows and not sixteen.  The counts go out once a warp.
// 1024^3: 51 -> 14 us at eight slices; bitmaps of less than 2^18 words, which
// would leave most of the chip idle then, take two (256^3: 11 us at eight, 5.7 at two).
template <int kRun>
__global__ void __launch_bounds__(128) k_cubes_small(uint32_t* __restrict__ e, int32_t words, int32_t py, int32_t pz) {
  const int64_t n = (int64_t)words * py * pz;
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x, slice = (uint32_t)words * py;
  const uint32_t run = i / slice, at = i - run * slice;   // the word of every slice of the run
  const int y = (int)(at / (uint32_t)words), w = (int)(at - (uint32_t)y * words);
  const int z0 = (int)(run * kRun);   // past the last slice: nothing to do
  uint32_t s2 = 0u, s3[2] = {0u, 0u}, s4[3] = {0u, 0u, 0u}, open = 0u;   // squares of the slices before, latest first
#pragma unroll
  for (int k = 0; k < kRun + 3; ++k) {
    uint32_t q2 = ~0u, q3 = ~0u, q4 = ~0u;
#pragma unroll
    for (int dy = 0; dy < 4; ++dy) {
      const unsigned long long r = cube_bits(e, w, y + dy, z0 + k, words, py, pz);
      const unsigned long long x2 = r & (r >> 1);
      if (dy < 2) q2 &= (uint32_t)x2;
      if (dy < 3) q3 &= (uint32_t)(x2 & (r >> 2));
      q4 &= (uint32_t)(x2 & (x2 >> 2));
    }
    // cubes that end with this slice
    if (k >= 1 && k <= kRun && z0 + k - 1 < pz) e[n + (int64_t)(z0 + k - 1) * slice + at] = q2 & s2;
    if (k >= 2 && k <= kRun + 1 && z0 + k - 2 < pz)
      e[2 * n + (int64_t)(z0 + k - 2) * slice + at] = q3 & s3[0] & s3[1];
    if (k >= 3 && z0 + k - 3 < pz) {
      const uint32_t c4 = q4 & s4[0] & s4[1] & s4[2];
      e[3 * n + (int64_t)(z0 + k - 3) * slice + at] = c4;
      open += (uint32_t)__popc(c4);
    }
    s2 = q2;
    s3[1] = s3[0]; s3[0] = q3;
    s4[2] = s4[1]; s4[1] = s4[0]; s4[0] = q4;
  }
  open = __reduce_add_sync(0xffffffffu, open);
  if ((threadIdx.x & 31) == 0 && open) atomicAdd(&e[kCubeSides * n + ((i >> 5) & 31)], open);
}
__global__ void k_cubes_large(uint32_t* __restrict__ e, int32_t words, int32_t py, int32_t pz) {
  const int64_t n = (int64_t)words * py * pz;
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const uint32_t row = i / (uint32_t)words;
  const int w = (int)(i - row * words), z = (int)(row / (uint32_t)py), y = (int)(row - (uint32_t)z * py);
  uint32_t c6 = ~0u, c8 = ~0u, c12 = ~0u, c16 = ~0u;
  for (int dz = 0; dz < 2; ++dz)
    for (int dy = 0; dy < 2; ++dy) {
      const unsigned long long r = cube_bits(e + 2 * n, w, y + 3 * dy, z + 3 * dz, words, py, pz);
      c6 &= (uint32_t)(r & (r >> 3));
    }
  for (int dz = 0; dz < 4; ++dz)
    for (int dy = 0; dy < 4; ++dy) {
      const unsigned long long r = cube_bits(e + 3 * n, w, y + 4 * dy, z + 4 * dz, words, py, pz);
      const unsigned long long x8 = r & (r >> 4);
      if (dz < 2 && dy < 2) c8 &= (uint32_t)x8;
      if (dz < 3 && dy < 3) c12 &= (uint32_t)(x8 & (r >> 8));
      c16 &= (uint32_t)(x8 & (x8 >> 8));
    }
  e[4 * n + i] = c6;
  e[5 * n + i] = c8;
  e[6 * n + i] = c12;
  e[7 * n + i] = c16;
}

// A warp takes four words at a time: lane 8 i + o reads octant o of word i,
// eight bitmaps, and spreads the levels of its 32 bricks to a byte each, four
// bricks a 32-bit word; through shared memory lane 8 i + g then gets those of
// all octants for bricks 4 g .. 4 g + 3 of word i, and turns the 4 x 8 bytes
// into a word per brick.  What bounds it is issue.  1024^3: 70 us; with a warp
// per word, four lanes reading each octant and the bytes changing places one
// by one, 158.  A warp takes kCubeRun words in a row, since a sector holds
// eight words of a bitmap.
constexpr int kCubeWarps = 4;
constexpr uint32_t kCubeRun = 8;
constexpr int kCubePitch = 72;   // 32-bit words between the four words' bytes: 64 and a shift of the banks
__global__ void __launch_bounds__(32 * kCubeWarps) k_cubes_bytes(const uint32_t* __restrict__ e, int32_t words,
                                                                 int32_t px, int32_t py, int32_t pz,
                                                                 unsigned long long* __restrict__ runs) {
  __shared__ __align__(16) uint32_t s[kCubeWarps][4 * kCubePitch];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int o = lane & 7;
  const uint32_t n = (uint32_t)words * py * pz;
  const uint32_t first = (blockIdx.x * kCubeWarps + warp) * kCubeRun, last = min(n, first + kCubeRun);
  if (first >= n) return;   // the whole warp
  const uint32_t down = ((o & 2) ? 0u : (uint32_t)words) + ((o & 4) ? 0u : (uint32_t)words * py);
  uint32_t i = first + (lane >> 3);
  const uint32_t row = i / (uint32_t)words;
  int w = (int)(i - row * words), z = (int)(row / (uint32_t)py), y = (int)(row - (uint32_t)z * py);
  uint32_t* const mine = &s[warp][(lane >> 3) * kCubePitch];
  for (uint32_t i0 = first; i0 < last; i0 += 4, i += 4) {   // the same turns for every lane
    if (i < last) {
      // the cube's lowest row lies (side - 1) rows and slices down where the
      // octant's y, z point down: in the array if side - 1 is at most `low`
      const int low = min((o & 2) ? kMaxFreeCube : y, (o & 4) ? kMaxFreeCube : z);
      uint32_t c[kCubeSides];
#pragma unroll
      for (int k = 0; k < kCubeSides; ++k) {   // every read is issued before any is used
        const int off = kCubeSide[k] - 1;
        const uint32_t* r = e + (size_t)k * n + (i - (uint32_t)off * down);
        const bool in = off <= low;
        const uint32_t cur = in ? r[0] : 0u, prev = in && !(o & 1) && w > 0 ? r[-1] : 0u;
        c[k] = (o & 1) ? cur : __funnelshift_l(prev, cur, off);   // and from its lowest brick
      }
      // levels passed, 0 to 8, in four bit planes: each level implies the ones before it
      const uint32_t b0 = (c[0] & ~c[1]) | (c[2] & ~c[3]) | (c[4] & ~c[5]) | (c[6] & ~c[7]);
      const uint32_t b1 = (c[1] & ~c[3]) | (c[5] & ~c[7]);
      const uint32_t b2 = c[3] & ~c[7], b3 = c[7];
#pragma unroll
      for (int g = 0; g < 8; ++g) {   // a byte per brick: bit j of a nibble to bit 8 j
        uint32_t v = (((b0 >> (4 * g)) & 15u) * 0x00204081u) & 0x01010101u;
        v |= (((b1 >> (4 * g)) & 15u) * 0x00408102u) & 0x02020202u;
        v |= (((b2 >> (4 * g)) & 15u) * 0x00810204u) & 0x04040404u;
        v |= (((b3 >> (4 * g)) & 15u) * 0x01020408u) & 0x08080808u;
        mine[8 * g + o] = v;
      }
    }
    __syncwarp();
    if (i < last) {
      const int g = o;
      const uint4 a = *(const uint4*)&mine[8 * g], b = *(const uint4*)&mine[8 * g + 4];
      // bricks 0, 1 and (h) 2, 3 of octant pairs, then the pairs of each brick
      const uint32_t a01 = __byte_perm(a.x, a.y, 0x5140), a23 = __byte_perm(a.z, a.w, 0x5140);
      const uint32_t a01h = __byte_perm(a.x, a.y, 0x7362), a23h = __byte_perm(a.z, a.w, 0x7362);
      const uint32_t b01 = __byte_perm(b.x, b.y, 0x5140), b23 = __byte_perm(b.z, b.w, 0x5140);
      const uint32_t b01h = __byte_perm(b.x, b.y, 0x7362), b23h = __byte_perm(b.z, b.w, 0x7362);
      const int x = 32 * w + 4 * g;
      unsigned long long* at = runs + ((int64_t)z * py + y) * px + x;
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const uint32_t pick = (j & 1) ? 0x7632u : 0x5410u;
        const uint32_t lo = j < 2 ? __byte_perm(a01, a23, pick) : __byte_perm(a01h, a23h, pick);
        const uint32_t hi = j < 2 ? __byte_perm(b01, b23, pick) : __byte_perm(b01h, b23h, pick);
        if (x + j < px) at[j] = ((unsigned long long)hi << 32) | lo;
      }
    }
    __syncwarp();
    for (w += 4; w >= words; w -= words)
      if (++y == py) { y = 0; ++z; }
  }
}

cudaError_t launch_free_cubes_open(const unsigned long long* bricks, int32_t bx, int32_t by, int32_t bz, void* scratch,
                                   uint32_t** open, int sm_count, cudaStream_t st) {
  const int32_t words = (int32_t)cube_words(bx), py = by + 2, pz = bz + 2;
  const int64_t n = (int64_t)words * py * pz;
  uint32_t* e = (uint32_t*)scratch;
  *open = e + kCubeSides * n;
  const cudaError_t m = cudaMemsetAsync(*open, 0, 32 * sizeof(uint32_t), st);
  if (m != cudaSuccess) return m;
  k_cubes_1<<<(unsigned)std::min<int64_t>((n + 31) / 32, (int64_t)sm_count * 64), 256, 0, st>>>(bricks, bx + 2,
                                                                                             (uint32_t)n, words, e);
  const int run = n < (1 << 18) ? 2 : 8;
  const unsigned blocks = (unsigned)(((int64_t)words * py * ((pz + run - 1) / run) + 127) / 128);
  if (run == 2) k_cubes_small<2><<<blocks, 128, 0, st>>>(e, words, py, pz);
  else k_cubes_small<8><<<blocks, 128, 0, st>>>(e, words, py, pz);
  return cudaGetLastError();
}

cudaError_t launch_free_cubes(int32_t bx, int32_t by, int32_t bz, void* scratch, unsigned long long* runs,
                              cudaStream_t st) {
  const int32_t words = (int32_t)cube_words(bx), py = by + 2, pz = bz + 2;
  const int64_t n = (int64_t)words * py * pz, per_block = kCubeWarps * kCubeRun;
  uint32_t* e = (uint32_t*)scratch;
  k_cubes_large<<<(unsigned)((n + 127) / 128), 128, 0, st>>>(e, words, py, pz);
  k_cubes_bytes<<<(unsigned)((n + per_block - 1) / per_block), 32 * kCubeWarps, 0, st>>>(e, words, bx + 2, py, pz, runs);
  return cudaGetLastError();
}

// Free cubes around a brick that became occupied: a cube that holds it ends
// before it.  One thread per brick within reach; a brick that became empty
// leaves them as they are, still lower bounds.
constexpr int kReach = 2 * kMaxFreeCube - 1;
constexpr int kReachBricks = kReach * kReach * kReach;
__device__ __forceinline__ void cubes_edit(int i, unsigned long long* runs, int32_t px, int32_t py, int32_t pz, int32_t x,
                                           int32_t y, int32_t z) {
  const int ox = i % kReach - (kMaxFreeCube - 1), oy = (i / kReach) % kReach - (kMaxFreeCube - 1),
            oz = i / (kReach * kReach) - (kMaxFreeCube - 1);
  const int vx = x - ox, vy = y - oy, vz = z - oz;   // the edited brick lies (ox, oy, oz) from this one
  if (vx < 0 || vy < 0 || vz < 0 || vx >= px || vy >= py || vz >= pz) return;
  const uint32_t d = (uint32_t)max(abs(ox), max(abs(oy), abs(oz)));
  unsigned long long* at = runs + ((int64_t)vx + (int64_t)px * ((int64_t)vy + (int64_t)py * vz));
  unsigned long long w = *at;
  for (int o = 0; o < 8; ++o) {
    const bool towards = ((o & 1) ? ox >= 0 : ox <= 0) && ((o & 2) ? oy >= 0 : oy <= 0) && ((o & 4) ? oz >= 0 : oz <= 0);
    uint32_t level = (uint32_t)(w >> (8 * o)) & 0xffu;
    if (!towards || free_cube_side(level) <= d) continue;
    while (free_cube_side(level) > d) --level;
    w = (w & ~(0xffull << (8 * o))) | ((unsigned long long)level << (8 * o));
  }
  *at = w;
}

// One voxel edit: its grid entry and its bit in the padded brick grid, and with
// `runs` the free cubes around its brick, in the same launch (a second one made
// an edit of a scene with free cubes 10.5 -> 12.3 us).
__global__ void k_set_voxel(uint8_t* grid, unsigned long long* bricks, int32_t rx, int32_t ry, int32_t bx, int32_t by,
                            int32_t bz, const BrickShape sh, int32_t x, int32_t y, int32_t z, uint8_t entry,
                            unsigned long long* runs) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i == 0) {
    grid[(size_t)x + (size_t)rx * ((size_t)y + (size_t)ry * (size_t)z)] = entry;
    const int64_t b = brick_index_of(sh, bx, by, x, y, z);
    const unsigned long long bit = 1ull << brick_bit_of(sh, x, y, z);
    if (entry) atomicOr(&bricks[b], bit);
    else atomicAnd(&bricks[b], ~bit);
  }
  if (runs && i < kReachBricks)   // 4x4x4 bricks
    cubes_edit(i, runs, bx + 2, by + 2, bz + 2, (x >> 2) + 1, (y >> 2) + 1, (z >> 2) + 1);
}

cudaError_t launch_set_voxel(uint8_t* grid, unsigned long long* bricks, int32_t rx, int32_t ry, int32_t bx, int32_t by,
                             int32_t bz, const BrickShape& sh, int32_t x, int32_t y, int32_t z, uint8_t entry,
                             unsigned long long* runs, cudaStream_t st) {
  if (!entry) runs = nullptr;
  const int threads = runs ? 128 : 32, blocks = runs ? (kReachBricks + threads - 1) / threads : 1;
  k_set_voxel<<<blocks, threads, 0, st>>>(grid, bricks, rx, ry, bx, by, bz, sh, x, y, z, entry, runs);
  return cudaGetLastError();
}

cudaError_t launch_build_bricks(const uint8_t* grid, int32_t rx, int32_t ry, int32_t rz,
                                unsigned long long* bricks, int32_t bx, int32_t by, int32_t bz, const BrickShape& sh,
                                unsigned long long* max_entry, cudaStream_t st) {
  const uint32_t px = bx + 2, pxy = px * (uint32_t)(by + 2);
  const int64_t n = (int64_t)pxy * (bz + 2);
  k_build_bricks<<<(unsigned)((n + kBrickThreads - 1) / kBrickThreads), kBrickThreads, 0, st>>>(
      grid, rx, ry, rz, bricks, bx, by, bz, udiv_magic(px), udiv_magic(pxy), sh, max_entry);
  return cudaGetLastError();
}

// --------------------------------------------------------- emissive voxels
// Whether voxel v has an empty or out-of-range 6-neighbour (anyVisibleFace,
// src/renderer/import.cpp:133-178).
__device__ __forceinline__ bool visible_face(const uint8_t* __restrict__ grid, const EmissiveVolume& V, int64_t v) {
  const uint32_t i = (uint32_t)v;   // fewer than 2^31 voxels
  const uint32_t z = udiv(i, V.m_xy), r = i - z * (uint32_t)(V.rx * V.ry);
  const uint32_t y = udiv(r, V.m_x), x = r - y * (uint32_t)V.rx;
  if (x == 0 || y == 0 || z == 0 || x == (uint32_t)V.rx - 1u || y == (uint32_t)V.ry - 1u || z == (uint32_t)V.rz - 1u)
    return true;
  const size_t sy = (size_t)V.rx, sz = (size_t)V.rx * V.ry;
  const uint8_t* g = grid + v;
  return g[1] == 0 || *(g - 1) == 0 || g[sy] == 0 || *(g - sy) == 0 || g[sz] == 0 || *(g - sz) == 0;
}

// keep[i] = 1 if listed emissive voxel i has a visible face.
__global__ void k_emissive_flags(const uint8_t* __restrict__ grid, const EmissiveVolume V,
                                 const int32_t* __restrict__ emissive, int64_t n, uint8_t* __restrict__ keep) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) keep[i] = visible_face(grid, V, emissive[i]) ? 1 : 0;
}

cudaError_t launch_emissive_flags(const uint8_t* grid, const EmissiveVolume& V, const int32_t* emissive, int64_t n,
                                  uint8_t* keep, cudaStream_t st) {
  if (n <= 0) return cudaSuccess;
  k_emissive_flags<<<(unsigned)((n + 255) / 256), 256, 0, st>>>(grid, V, emissive, n, keep);
  return cudaGetLastError();
}

// Emissive list of a volume (the voxels whose palette entry emits,
// emissive_entry[g] != 0), pruned on request to those with a visible face, in
// the order that the reference's sequential removal leaves: the full list is
// in voxel order, and each removed element is replaced by the last one still
// in it (import.cpp:180-203).  With K elements kept, that is: a kept element
// whose place in the full list is below K stays there, and the kept ones from
// K on, last first, fill the removed places below K in increasing order.
//
// The volume is cut into chunks of kEmChunk voxels.  k_emissive_count counts
// each chunk's emissive and kept voxels, one block turns the counts into
// offsets, and k_emissive_write visits the chunks again and writes every kept
// element below K to its place, ~r to the r-th removed place below K, and the
// kept ones from K on to the mover list by their rank from the end;
// k_emissive_fill puts mover r in the place that holds ~r.  16
// voxels per thread and load, one block-wide prefix a chunk: reading the
// volume a byte per thread in rows with a prefix each took 56 us of a 256^3
// volume (now 18), and the pruning on the host, with its copies both ways, 0.4
// ms of its 0.64 ms load (now 0.22).
constexpr int kEmThreads = 256;
constexpr int64_t kEmChunk = (int64_t)kEmThreads * 16;

// Exclusive prefix of `v` over the block (kThreads threads); *total gets the sum.
template <class V, int kThreads = kEmThreads>
__device__ __forceinline__ V block_prefix(V v, V* warp_sums, V* total) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  V x = v;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const V y = __shfl_up_sync(0xffffffffu, x, o);
    if (lane >= o) x += y;
  }
  if (lane == 31) warp_sums[warp] = x;
  __syncthreads();
  V before = 0, all = 0;
  for (int w = 0; w < kThreads / 32; ++w) {
    before += w < warp ? warp_sums[w] : (V)0;
    all += warp_sums[w];
  }
  __syncthreads();   // warp_sums is reused by the next call
  *total = all;
  return before + x - v;
}

// The 16 voxels of this thread in its chunk: bit i of *em set if voxel
// base + i emits, of *keep if it is also listed after pruning.
__device__ __forceinline__ void emissive_bits(const uint8_t* __restrict__ grid, const EmissiveVolume& V, int64_t base,
                                              const uint8_t* s_em, uint32_t* em, uint32_t* keep) {
  uint32_t e = 0u, k = 0u;
  if (base + 16 <= V.n) {   // base is a multiple of 16, the grid starts on a 16-byte boundary
    const uint4 q = *(const uint4*)(grid + base);
    const uint32_t w[4] = {q.x, q.y, q.z, q.w};
    if (q.x | q.y | q.z | q.w) {
#pragma unroll
      for (int i = 0; i < 16; ++i) e |= (uint32_t)s_em[(w[i >> 2] >> (8 * (i & 3))) & 0xffu] << i;
    }
  } else {
    for (int i = 0; i < 16 && base + i < V.n; ++i) e |= (uint32_t)s_em[grid[base + i]] << i;
  }
  for (uint32_t left = e; left; left &= left - 1u) {
    const int i = __ffs(left) - 1;
    if (!V.prune || visible_face(grid, V, base + i)) k |= 1u << i;
  }
  *em = e;
  *keep = k;
}

__device__ __forceinline__ void emissive_table(const uint8_t* emissive_entry, uint8_t* s_em) {
  for (int i = threadIdx.x; i < 256; i += blockDim.x) s_em[i] = emissive_entry[i] ? 1 : 0;
  __syncthreads();
}

// counts[chunk]: emissive voxels in the low, kept ones in the high 32 bits.
__global__ void __launch_bounds__(kEmThreads) k_emissive_count(const uint8_t* __restrict__ grid, const EmissiveVolume V,
                                                               const uint8_t* __restrict__ emissive_entry,
                                                               unsigned long long* __restrict__ counts) {
  __shared__ uint8_t s_em[256];
  __shared__ uint32_t s_warp[kEmThreads / 32];
  emissive_table(emissive_entry, s_em);
  uint32_t em, keep;
  emissive_bits(grid, V, (int64_t)blockIdx.x * kEmChunk + 16 * threadIdx.x, s_em, &em, &keep);
  uint32_t total;   // a chunk holds at most 4096 of either
  block_prefix((uint32_t)__popc(em) | ((uint32_t)__popc(keep) << 16), s_warp, &total);
  if (threadIdx.x == 0) counts[blockIdx.x] = (unsigned long long)(total & 0xffffu) | ((unsigned long long)(total >> 16) << 32);
}

// In place: counts[0..n) -> exclusive offsets of both counts, counts[n] = the
// totals.  One block of kScanThreads threads, each over a contiguous run.
constexpr int kScanThreads = 1024;
__global__ void __launch_bounds__(kScanThreads) k_emissive_offsets(unsigned long long* counts, int64_t n) {
  __shared__ unsigned long long s_warp[kScanThreads / 32];
  const int64_t per = (n + kScanThreads - 1) / kScanThreads;
  const int64_t b = (int64_t)threadIdx.x * per, e = b + per < n ? b + per : n;
  unsigned long long sum = 0;
  for (int64_t i = b; i < e; ++i) sum += counts[i];   // either half stays below 2^31
  unsigned long long total;
  unsigned long long run = block_prefix<unsigned long long, kScanThreads>(sum, s_warp, &total);
  for (int64_t i = b; i < e; ++i) {
    const unsigned long long c = counts[i];
    counts[i] = run;
    run += c;
  }
  if (threadIdx.x == 0) counts[n] = total;
}

__global__ void __launch_bounds__(kEmThreads) k_emissive_write(const uint8_t* __restrict__ grid, const EmissiveVolume V,
                                                               const uint8_t* __restrict__ emissive_entry,
                                                               const unsigned long long* __restrict__ counts,
                                                               int64_t chunks, int32_t* __restrict__ out,
                                                               int32_t* __restrict__ movers) {
  __shared__ uint8_t s_em[256];
  __shared__ uint32_t s_warp[kEmThreads / 32];
  const unsigned long long first = counts[blockIdx.x], next = counts[blockIdx.x + 1];
  if ((uint32_t)first == (uint32_t)next) return;   // nothing emits in this chunk
  emissive_table(emissive_entry, s_em);
  const int64_t base = (int64_t)blockIdx.x * kEmChunk + 16 * threadIdx.x;
  uint32_t em, keep;
  emissive_bits(grid, V, base, s_em, &em, &keep);
  uint32_t total;
  const uint32_t pre = block_prefix((uint32_t)__popc(em) | ((uint32_t)__popc(keep) << 16), s_warp, &total);
  const uint32_t K = (uint32_t)(counts[chunks] >> 32);
  uint32_t pos = (uint32_t)first + (pre & 0xffffu), kept = (uint32_t)(first >> 32) + (pre >> 16);
  for (uint32_t left = em; left; left &= left - 1u) {
    const int i = __ffs(left) - 1;
    if ((keep >> i) & 1u) {
      if (pos < K) out[pos] = (int32_t)(base + i);
      else movers[K - 1u - kept] = (int32_t)(base + i);   // its rank from the end of the kept ones
      ++kept;
    } else if (pos < K) {
      out[pos] = (int32_t)~(pos - kept);
    }
    ++pos;
  }
}

__global__ void k_emissive_fill(const int32_t* __restrict__ movers, int64_t listed, int32_t* __restrict__ out) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= listed) return;
  const int32_t v = out[i];
  if (v < 0) out[i] = movers[~v];
}

int64_t emissive_chunks(int64_t n_voxels) { return (n_voxels + kEmChunk - 1) / kEmChunk; }

cudaError_t launch_emissive_count(const uint8_t* grid, const EmissiveVolume& V, const uint8_t* emissive_entry,
                                  unsigned long long* counts, cudaStream_t st) {
  const int64_t chunks = emissive_chunks(V.n);
  if (chunks <= 0) return cudaSuccess;
  k_emissive_count<<<(unsigned)chunks, kEmThreads, 0, st>>>(grid, V, emissive_entry, counts);
  k_emissive_offsets<<<1, kScanThreads, 0, st>>>(counts, chunks);
  return cudaGetLastError();
}

cudaError_t launch_emissive_write(const uint8_t* grid, const EmissiveVolume& V, const uint8_t* emissive_entry,
                                  const unsigned long long* counts, int32_t* out, int64_t listed, int32_t* movers,
                                  cudaStream_t st) {
  const int64_t chunks = emissive_chunks(V.n);
  if (chunks <= 0 || listed <= 0) return cudaSuccess;
  k_emissive_write<<<(unsigned)chunks, kEmThreads, 0, st>>>(grid, V, emissive_entry, counts, chunks, out, movers);
  if (movers) k_emissive_fill<<<(unsigned)((listed + 255) / 256), 256, 0, st>>>(movers, listed, out);
  return cudaGetLastError();
}

// ------------------------------------------------------------ environment
// Three-tap Gaussian (sigma = 0.75 px) normalised to sum 1:
//   w_side = e / (1 + 2e), w_mid = 1 / (1 + 2e), e = exp(-1 / (2 * 0.75^2)).
#define VT_BLUR_SIDE 0.225610111284051620f
#define VT_BLUR_MID 0.548779777431896800f

// FP16 texels (A = 1) and the luminance of the quantised RGB
// (generateImageFunction's channel_sum, src/renderer/image.cpp:326-335).
// `bad` receives the smallest index of a texel with a non-finite channel.
__global__ void k_env_texels(const float* __restrict__ rgb, int64_t n, uint2* __restrict__ texels,
                             float* __restrict__ lum, uint32_t* bad) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  if (!(isfinite(rgb[3 * i]) && isfinite(rgb[3 * i + 1]) && isfinite(rgb[3 * i + 2]))) atomicMin(bad, (uint32_t)i);
  const uint16_t r = vtb::f2h(vtb::clamp_half(rgb[3 * i])), g = vtb::f2h(vtb::clamp_half(rgb[3 * i + 1])),
                 b = vtb::f2h(vtb::clamp_half(rgb[3 * i + 2]));
  texels[i] = make_uint2((uint32_t)r | ((uint32_t)g << 16), (uint32_t)b | (0x3c00u << 16));
  const float fr = vtb::h2f(r), fg = vtb::h2f(g), fb = vtb::h2f(b);
  lum[i] = (fr * 0.2126f + fg * 0.7152f) + fb * 0.0722f;
}

// The sampled function of one texel: 3x3 separable blur of the luminance,
// clamp to edge (image.cpp:337-342), then the max(0, .) and the sin(theta)
// weight of calculateImageIntegral (image.cpp:361-374).
__device__ __forceinline__ float blur_row(const float* __restrict__ lum, int32_t w, int x, int y) {
  const float* r = lum + (int64_t)y * w;
  const int xm = x > 0 ? x - 1 : 0, xp = x < w - 1 ? x + 1 : w - 1;
  return (VT_BLUR_SIDE * r[xm] + VT_BLUR_MID * r[x]) + VT_BLUR_SIDE * r[xp];
}
__device__ __forceinline__ float env_function(const float* __restrict__ lum, int32_t w, int32_t h, int x, int y,
                                              float sin_theta) {
  const int ym = y > 0 ? y - 1 : 0, yp = y < h - 1 ? y + 1 : h - 1;
  const float v = (VT_BLUR_SIDE * blur_row(lum, w, x, ym) + VT_BLUR_MID * blur_row(lum, w, x, y)) +
                  VT_BLUR_SIDE * blur_row(lum, w, x, yp);
  return vtb::gmax(0.0f, v) * sin_theta;
}

// Prefix sums in FP64 with a fixed association order, so that the CPU
// restatement reproduces them exactly: consecutive chunks of 32 inputs are
// summed left to right, chunk offsets are accumulated left to right, and
// element prefix = chunk offset + in-chunk prefix.  A block of kCdfThreads
// threads takes kCdfTile inputs at a time: loaded coalesced into shared
// memory (one double of padding per chunk), summed by a thread per chunk, the
// offsets chained by thread 0 from one tile to the next.  What bounds it is
// the length of the two chains, 32 additions and one per chunk; reading and
// writing the chunks in global memory instead, a warp per row, cost a memory
// round trip per addition (1024x512: 58 us for the rows, 19 for the marginal,
// now 25 and 8.5, the 13 us of two blur passes folded in).
constexpr int kCdfThreads = 128;
constexpr int kCdfTile = 32 * kCdfThreads;
__device__ __forceinline__ int cdf_at(int i) { return i + (i >> 5); }

// Prefixes of in(0 .. n) in s (element i after input i, at cdf_at(i)), or past
// the first tile in `pre` (element i after input i) as well; returns the total.
template <class In>
__device__ double block_chunked_prefix(const In& in, int n, double* s, double* s_off, double* __restrict__ pre) {
  double carry = 0.0;   // offset of the tile's first chunk
  const int tid = threadIdx.x;
  for (int base = 0; base < n; base += kCdfTile) {
    const int m = min(kCdfTile, n - base), chunks = (m + 31) / 32;
    for (int i = threadIdx.x; i < m; i += kCdfThreads) s[cdf_at(i)] = (double)in(base + i);
    __syncthreads();
    if (tid < chunks) {
      const int c0 = tid * 32, c1 = min(m, c0 + 32);
      double* const sc = s + cdf_at(c0);   // a chunk lies contiguous
      double acc = 0.0;
      int i = 0;
      for (; c0 + i + 8 <= c1; i += 8) {   // eight reads in flight ahead of the additions
        double v[8];
#pragma unroll
        for (int k = 0; k < 8; ++k) v[k] = sc[i + k];
#pragma unroll
        for (int k = 0; k < 8; ++k) {
          acc = acc + v[k];
          sc[i + k] = acc;
        }
      }
      for (; c0 + i < c1; ++i) {
        acc = acc + sc[i];
        sc[i] = acc;
      }
      s_off[tid] = acc;
    }
    __syncthreads();
    if (tid < 32) {   // chunk totals -> offsets, 32 at a time from a warp's registers
      double o = carry;
      for (int c0 = 0; c0 < chunks; c0 += 32) {
        const int c = c0 + tid;
        const double t = c < chunks ? s_off[c] : 0.0;
        double mine = 0.0;
        for (int k = 0; k < 32 && c0 + k < chunks; ++k) {
          const double tk = __shfl_sync(0xffffffffu, t, k);
          if (tid == k) mine = o;
          o = base + c0 + k == 0 ? tk : o + tk;
        }
        if (c < chunks) s_off[c] = mine;
      }
      if (tid == 0) s_off[kCdfThreads] = o;
    }
    __syncthreads();
    carry = s_off[kCdfThreads];
    const bool whole = n <= kCdfTile;
    for (int i = threadIdx.x; i < m; i += kCdfThreads) {
      const int c = i >> 5;
      const double v = s[cdf_at(i)], p = base + c == 0 ? v : s_off[c] + v;
      if (whole) s[cdf_at(i)] = p;
      else pre[base + i] = p;
    }
    __syncthreads();
  }
  return carry;
}

// (float)(a / b) for 0 <= a <= b, b normal: a product with the reciprocal is
// within two units of the double quotient, so both round to the same float
// unless the product lies that close to the middle of two floats or below
// the normal floats; those few divide.
__device__ __forceinline__ float quotient(double a, double b, double rcp) {
  const double q = a * rcp;
  const uint32_t low = (uint32_t)__double_as_longlong(q) & 0x1fffffffu;   // bits below a float's
  if (q >= 1.2e-38 && low - 0x0ffffff8u > 16u) return (float)q;
  return (float)(a / b);
}

// One block per row (image.cpp:212-247): the row of the sampled function
// (kEnv: from the luminance; otherwise given), its FP64 prefixes, normalised
// conditional CDF (uniform if the row is black), row integral = row sum / width.
template <bool kEnv>
__global__ void __launch_bounds__(kCdfThreads) k_cdf_rows(const float* __restrict__ f, int32_t w, int32_t h,
                                                          const float* __restrict__ sin_theta,
                                                          double* __restrict__ pre_all, float* __restrict__ cdf_u,
                                                          double* __restrict__ row_int) {
  __shared__ double s[kCdfTile + kCdfThreads];
  __shared__ double s_off[kCdfThreads + 1];
  const int row = blockIdx.x;
  double* pre = pre_all + (int64_t)row * (w + 1);
  double total;
  if constexpr (kEnv) {
    const float st = sin_theta[row];
    total = block_chunked_prefix([&](int x) { return env_function(f, w, h, x, row, st); }, w, s, s_off, pre);
  } else {
    total = block_chunked_prefix([&](int x) { return f[(int64_t)row * w + x]; }, w, s, s_off, pre);
  }
  float* out = cdf_u + (int64_t)row * (w + 1);
  if (threadIdx.x == 0) {   // one thread's divisions: FP64 is scarce
    s_off[0] = 1.0 / total;
    row_int[row] = total / (double)w;
  }
  __syncthreads();
  const double rcp = s_off[0];
  const bool whole = w <= kCdfTile;
  for (int x = threadIdx.x; x <= w; x += kCdfThreads) {
    if (total > 0.0) out[x] = x == 0 ? 0.0f : quotient(whole ? s[cdf_at(x - 1)] : pre[x - 1], total, rcp);
    else out[x] = (float)x / (float)w;
  }
}

// Marginal CDF over the row integrals (image.cpp:251-280) and the radiance
// integral 2 pi^2 * mean(f) (image.cpp:381-386).  One block.
__global__ void __launch_bounds__(kCdfThreads) k_cdf_marginal(const double* __restrict__ row_int, int32_t h,
                                                              double* __restrict__ pre, float* __restrict__ cdf_v,
                                                              float* integral) {
  __shared__ double s[kCdfTile + kCdfThreads];
  __shared__ double s_off[kCdfThreads + 1];
  const double total = block_chunked_prefix([&](int y) { return row_int[y]; }, h, s, s_off, pre);
  if (threadIdx.x == 0) s_off[0] = 1.0 / total;
  __syncthreads();
  const double rcp = s_off[0];
  const bool whole = h <= kCdfTile;
  for (int y = threadIdx.x; y <= h; y += kCdfThreads) {
    if (total > 0.0) cdf_v[y] = y == 0 ? 0.0f : quotient(whole ? s[cdf_at(y - 1)] : pre[y - 1], total, rcp);
    else cdf_v[y] = (float)y / (float)h;
  }
  if (threadIdx.x == 0 && integral) {
    *integral = (float)((total / (double)h) * (2.0 * 3.14159265358979323846 * 3.14159265358979323846));
  }
}

template <bool kEnv>
static cudaError_t cdf(const float* f, int32_t w, int32_t h, const EnvScratch& S, float* cdf_u, float* cdf_v,
                       float* integral, cudaStream_t st) {
  k_cdf_rows<kEnv><<<h, kCdfThreads, 0, st>>>(f, w, h, S.sin_theta, S.row_pre, cdf_u, S.row_int);
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return e;
  k_cdf_marginal<<<1, kCdfThreads, 0, st>>>(S.row_int, h, S.marg_pre, cdf_v, integral);
  return cudaGetLastError();
}

cudaError_t launch_cdf(const float* func, int32_t w, int32_t h, const EnvScratch& S, float* cdf_u,
                       float* cdf_v, float* integral, cudaStream_t st) {
  return cdf<false>(func, w, h, S, cdf_u, cdf_v, integral, st);
}

// The CDF image of a shrunk environment (image.cpp:308-320): each output
// texel is the area-weighted average of the FP16 texels its footprint
// covers (double sums, rows then columns in index order), then its Rec.709
// luminance.  A box filter standing in for OpenImageIO's resize.
__global__ void k_env_shrink_lum(const uint2* __restrict__ texels, int32_t w, int32_t h, int32_t ow, int32_t oh,
                                 float* __restrict__ lum) {
  const int64_t o = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (o >= (int64_t)ow * oh) return;
  const int ox = (int)(o % ow), oy = (int)(o / ow);
  const double sx = (double)w / (double)ow, sy = (double)h / (double)oh;
  const double y0 = (double)oy * sy, y1 = (double)(oy + 1) * sy;
  const double x0 = (double)ox * sx, x1 = (double)(ox + 1) * sx;
  double acc0 = 0.0, acc1 = 0.0, acc2 = 0.0;
  for (int j = (int)floor(y0); j < (int)ceil(y1) && j < h; ++j) {
    const double wy = fmin(y1, (double)(j + 1)) - fmax(y0, (double)j);
    for (int i = (int)floor(x0); i < (int)ceil(x1) && i < w; ++i) {
      const double wx = fmin(x1, (double)(i + 1)) - fmax(x0, (double)i);
      const double wgt = wx * wy;
      const uint2 q = texels[(int64_t)j * w + i];
      acc0 = acc0 + wgt * (double)vtb::h2f((uint16_t)(q.x & 0xffffu));
      acc1 = acc1 + wgt * (double)vtb::h2f((uint16_t)(q.x >> 16));
      acc2 = acc2 + wgt * (double)vtb::h2f((uint16_t)(q.y & 0xffffu));
    }
  }
  const double area = sx * sy;
  const float fr = (float)(acc0 / area), fg = (float)(acc1 / area), fb = (float)(acc2 / area);
  lum[o] = (fr * 0.2126f + fg * 0.7152f) + fb * 0.0722f;
}

cudaError_t launch_env_build(const float* rgb, int32_t w, int32_t h, int32_t cw, int32_t ch, const EnvScratch& S,
                             uint2* texels, float* cdf_u, float* cdf_v, float* integral, uint32_t* bad,
                             cudaStream_t st) {
  const int64_t n = (int64_t)w * h;
  k_env_texels<<<(unsigned)((n + 255) / 256), 256, 0, st>>>(rgb, n, texels, S.lum, bad);
  const int64_t m = (int64_t)cw * ch;
  if (cw != w || ch != h)
    k_env_shrink_lum<<<(unsigned)((m + 255) / 256), 256, 0, st>>>(texels, w, h, cw, ch, S.lum);
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return e;
  return cdf<true>(S.lum, cw, ch, S, cdf_u, cdf_v, integral, st);
}

// --------------------------------------------------------------- voxelizer
// Rauwendaal & Bailey, "Hybrid Computational Voxelization Using the Graphics
// Pipeline" (JCGT 2013) as implemented by src/shaders/shared/voxelize.gs:55-251
// and src/voxelize/cpuVoxelizer.cpp:42-235: project on the dominant axis,
// test the XY edge functions per column, derive the Z range from the plane,
// test the YZ and ZX edge functions per voxel.  mode 0 = THIN (6-separating,
// figure 18), 1 = FAT (conservative, figure 17).  The scan range of a
// triangle is its bounding box in the swizzled frame, clamped to the grid's
// extent along the swizzled axes; with ref_bounds, against the unswizzled
// resolution as voxelize.gs:247-248 does (the same on cubic grids; on others
// voxels near the far faces of the shorter axes are lost).  FAT without
// ref_bounds marks exactly the voxels that a separating-axis test marks,
// up to float rounding where a voxel only touches the triangle.
struct TriSetup {
  float d_xy[3], d_yz[3], d_zx[3];
  float n_xy[3][2], n_yz[3][2], n_zx[3][2];
  float nproj[3];
  float dmin, dmax, nz_inv;
  int perm;           // 0: swizzled yzx, 1: zxy, 2: identity
  int lo[3], hi[3];   // voxel index range in swizzled space
  bool valid;
};

__device__ __forceinline__ int sat_int(float f) {
  // float -> int with NaN and out-of-range values mapped into +-1e9
  if (f >= -1.0e9f && f <= 1.0e9f) return (int)f;
  return f > 0.0f ? 1000000000 : -1000000000;
}

__device__ __forceinline__ void edge_normal(float ea, float eb, bool pos, float* nrm) {
  // pos ? vec2(-eb, ea) : vec2(eb, -ea) for an edge (ea, eb)
  if (pos) { nrm[0] = -eb; nrm[1] = ea; } else { nrm[0] = eb; nrm[1] = -ea; }
}

__device__ __forceinline__ float edge_d(const float* nrm, float pa, float pb, int mode) {
  if (mode == 0) {
    // dot(n, .5 - v) + 0.5 * max(|n.x|, |n.y|)   (voxelize.gs:140-150)
    return (nrm[0] * (0.5f - pa) + nrm[1] * (0.5f - pb)) + 0.5f * vtb::gmax(fabsf(nrm[0]), fabsf(nrm[1]));
  }
  // -dot(n, v) + max(0, n.x) + max(0, n.y)      (voxelize.gs:152-162)
  return (-(nrm[0] * pa + nrm[1] * pb) + vtb::gmax(0.0f, nrm[0])) + vtb::gmax(0.0f, nrm[1]);
}

__device__ bool tri_setup(const float* V, int64_t nv, const uint32_t* I, int64_t t, int32_t rx, int32_t ry,
                          int32_t rz, int mode, bool ref_bounds, TriSetup& S) {
  float v[3][3];
  for (int k = 0; k < 3; ++k) {
    const uint32_t vi = I[3 * t + k];
    if ((int64_t)vi >= nv) return false;   // recorded by k_mesh_scan; the call fails
    v[k][0] = V[3 * (int64_t)vi]; v[k][1] = V[3 * (int64_t)vi + 1]; v[k][2] = V[3 * (int64_t)vi + 2];
  }
  // n = cross(v1 - v0, v2 - v1)   (voxelize.gs:62)
  const float a0 = v[1][0] - v[0][0], a1 = v[1][1] - v[0][1], a2 = v[1][2] - v[0][2];
  const float b0 = v[2][0] - v[1][0], b1 = v[2][1] - v[1][1], b2 = v[2][2] - v[1][2];
  float n[3] = {a1 * b2 - b1 * a2, a2 * b0 - b2 * a0, a0 * b1 - b0 * a1};
  const float ax = fabsf(n[0]), ay = fabsf(n[1]), az = fabsf(n[2]);
  int perm;
  if (ax >= ay && ax >= az) perm = 0;        // look down X: xyz <- yzx
  else if (ay >= ax && ay >= az) perm = 1;   // look down Y: xyz <- zxy
  else perm = 2;
  if (perm != 2) {
    const int i0 = perm == 0 ? 1 : 2, i1 = perm == 0 ? 2 : 0, i2 = perm == 0 ? 0 : 1;
    for (int k = 0; k < 3; ++k) {
      const float p0 = v[k][i0], p1 = v[k][i1], p2 = v[k][i2];
      v[k][0] = p0; v[k][1] = p1; v[k][2] = p2;
    }
    const float m0 = n[i0], m1 = n[i1], m2 = n[i2];
    n[0] = m0; n[1] = m1; n[2] = m2;
  }
  S.perm = perm;
  // grid extent along the swizzled axes: yzx -> (ry, rz, rx), zxy -> (rz, rx, ry)
  int res[3] = {rx, ry, rz};
  if (!ref_bounds && perm == 0) { res[0] = ry; res[1] = rz; res[2] = rx; }
  if (!ref_bounds && perm == 1) { res[0] = rz; res[1] = rx; res[2] = ry; }
  // ivec3(clamp(floor(min), 0, res)), ivec3(clamp(ceil(max), 0, res))
  // (voxelize.gs:247-248); a FAT scan also takes the voxels that only touch
  // the triangle at an integer bound, ceil(min) - 1 and floor(max) + 1, which
  // that range skips (a triangle lying in an integer plane would mark nothing).
  const bool touch = !ref_bounds && mode == 1;
  for (int c = 0; c < 3; ++c) {
    const float mn = vtb::gmin(vtb::gmin(v[0][c], v[1][c]), v[2][c]);
    const float mx = vtb::gmax(vtb::gmax(v[0][c], v[1][c]), v[2][c]);
    const int l = touch ? sat_int(ceilf(mn)) - 1 : sat_int(floorf(mn));
    const int u = touch ? sat_int(floorf(mx)) + 1 : sat_int(ceilf(mx));
    S.lo[c] = min(max(l, 0), res[c]);
    S.hi[c] = min(max(u, 0), res[c]);
  }
  float e[3][3];
  for (int c = 0; c < 3; ++c) {
    e[0][c] = v[1][c] - v[0][c];
    e[1][c] = v[2][c] - v[1][c];
    e[2][c] = v[0][c] - v[2][c];
  }
  for (int k = 0; k < 3; ++k) {
    edge_normal(e[k][0], e[k][1], n[2] >= 0.0f, S.n_xy[k]);   // (x, y)
    edge_normal(e[k][1], e[k][2], n[0] >= 0.0f, S.n_yz[k]);   // (y, z)
    edge_normal(e[k][2], e[k][0], n[1] >= 0.0f, S.n_zx[k]);   // (z, x)
    S.d_xy[k] = edge_d(S.n_xy[k], v[k][0], v[k][1], mode);
    S.d_yz[k] = edge_d(S.n_yz[k], v[k][1], v[k][2], mode);
    S.d_zx[k] = edge_d(S.n_zx[k], v[k][2], v[k][0], mode);
  }
  const bool neg = n[2] < 0.0f;
  S.nproj[0] = neg ? -n[0] : n[0]; S.nproj[1] = neg ? -n[1] : n[1]; S.nproj[2] = neg ? -n[2] : n[2];
  const float dtri = (S.nproj[0] * v[0][0] + S.nproj[1] * v[0][1]) + S.nproj[2] * v[0][2];
  if (mode == 0) {
    S.dmin = dtri - (S.nproj[0] * 0.5f + S.nproj[1] * 0.5f);  // voxelize.gs:169
    S.dmax = S.dmin;
  } else {
    S.dmin = (dtri - vtb::gmax(S.nproj[0], 0.0f)) - vtb::gmax(S.nproj[1], 0.0f);   // :171
    S.dmax = (dtri - vtb::gmin(S.nproj[0], 0.0f)) - vtb::gmin(S.nproj[1], 0.0f);   // :172
  }
  S.valid = S.nproj[2] != 0.0f;   // zero-area triangles cover nothing
  S.nz_inv = 1.0f / S.nproj[2];
  return S.valid;
}

// Where a voxelized voxel is recorded: its grid byte and, when the scene's
// bricks are being built alongside, its bit of the padded brick grid.
struct VoxOut {
  uint8_t* grid;
  uint8_t value;
  unsigned long long* bricks;   // nullable
  int32_t bx, by;               // bricks per row / column inside the border
  BrickShape sh;
};

// Brick bits a thread has set, gathered while they fall in one brick and
// OR'ed into the brick grid with one atomic when the brick changes.
struct BrickAcc {
  int64_t b = -1;
  unsigned long long bits = 0ull;
  __device__ __forceinline__ void add(const VoxOut& O, int64_t nb, unsigned long long bit) {
    if (nb != b) {
      flush(O);
      b = nb;
    }
    bits |= bit;
  }
  __device__ __forceinline__ void flush(const VoxOut& O) {
    if (bits) atomicOr(&O.bricks[b], bits);
    bits = 0ull;
  }
};

__device__ __forceinline__ void tri_column(const TriSetup& S, int px, int py, int mode, int32_t rx, int32_t ry,
                                           int32_t rz, const VoxOut& O, BrickAcc& acc) {
  bool xy = true;
  for (int k = 0; k < 3; ++k) {
    const float dd = S.d_xy[k] + (S.n_xy[k][0] * (float)px + S.n_xy[k][1] * (float)py);
    xy = xy && (dd >= 0.0f);
  }
  if (!xy) return;
  const float dnp = S.nproj[0] * (float)px + S.nproj[1] * (float)py;
  const float zmin_i = (-dnp + S.dmin) * S.nz_inv;
  const float zmax_i = (-dnp + S.dmax) * S.nz_inv;
  const float zmin_f = floorf(zmin_i), zmax_c = ceilf(zmax_i);
  int zmin = sat_int(zmin_f) - (zmin_f == zmin_i ? 1 : 0);
  int zmax = sat_int(zmax_c) + (zmax_c == zmax_i ? 1 : 0);
  zmin = max(S.lo[2], zmin);
  zmax = min(S.hi[2], zmax);
  for (int pz = zmin; pz < zmax; ++pz) {
    bool ok = true;
    for (int k = 0; k < 3; ++k) {
      const float dyz = S.d_yz[k] + (S.n_yz[k][0] * (float)py + S.n_yz[k][1] * (float)pz);
      const float dzx = S.d_zx[k] + (S.n_zx[k][0] * (float)pz + S.n_zx[k][1] * (float)px);
      ok = ok && (dyz >= 0.0f) && (dzx >= 0.0f);
    }
    if (!ok) continue;
    // unswizzle (voxelize.gs:40-48): yzx -> (z, x, y), zxy -> (y, z, x)
    int ox, oy, oz;
    if (S.perm == 0) { ox = pz; oy = px; oz = py; }
    else if (S.perm == 1) { ox = py; oy = pz; oz = px; }
    else { ox = px; oy = py; oz = pz; }
    // imageStore outside the image has no effect
    if (ox < 0 || oy < 0 || oz < 0 || ox >= rx || oy >= ry || oz >= rz) continue;
    O.grid[(size_t)ox + (size_t)rx * ((size_t)oy + (size_t)ry * (size_t)oz)] = O.value;
    if (O.bricks) acc.add(O, brick_index_of(O.sh, O.bx, O.by, ox, oy, oz), 1ull << brick_bit_of(O.sh, ox, oy, oz));
  }
  (void)mode;
}

constexpr int kLargeColumns = 64;

// One thread per triangle for triangles whose XY footprint is small; larger
// ones are appended to a list for the block-per-triangle kernel.
__global__ void k_vox_small(const float* __restrict__ V, int64_t nv, const uint32_t* __restrict__ I,
                            int64_t n_tris, int32_t rx, int32_t ry, int32_t rz, int mode, bool ref_bounds,
                            const VoxOut O, int64_t* large, unsigned long long* n_large) {
  const int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= n_tris) return;
  TriSetup S;
  if (!tri_setup(V, nv, I, t, rx, ry, rz, mode, ref_bounds, S)) return;
  const int64_t cols = (int64_t)(S.hi[0] - S.lo[0]) * (int64_t)(S.hi[1] - S.lo[1]);
  if (cols > kLargeColumns) {
    const unsigned long long slot = atomicAdd(n_large, 1ull);
    large[slot] = t;
    return;
  }
  BrickAcc acc;
  for (int px = S.lo[0]; px < S.hi[0]; ++px)
    for (int py = S.lo[1]; py < S.hi[1]; ++py) tri_column(S, px, py, mode, rx, ry, rz, O, acc);
  if (O.bricks) acc.flush(O);
}

__global__ void k_vox_large(const float* __restrict__ V, int64_t nv, const uint32_t* __restrict__ I,
                            const int64_t* large, const unsigned long long* n_large, int32_t rx, int32_t ry,
                            int32_t rz, int mode, bool ref_bounds, const VoxOut O) {
  __shared__ TriSetup S;
  const unsigned long long n = *n_large;
  for (unsigned long long k = blockIdx.x; k < n; k += gridDim.x) {
    __syncthreads();
    if (threadIdx.x == 0) tri_setup(V, nv, I, large[k], rx, ry, rz, mode, ref_bounds, S);   // listed: valid
    __syncthreads();
    const int wx = S.hi[0] - S.lo[0], wy = S.hi[1] - S.lo[1];
    const int64_t cols = (int64_t)wx * wy;
    BrickAcc acc;
    for (int64_t c = threadIdx.x; c < cols; c += blockDim.x) {
      const int px = S.lo[0] + (int)(c / wy), py = S.lo[1] + (int)(c % wy);
      tri_column(S, px, py, mode, rx, ry, rz, O, acc);
    }
    if (O.bricks) acc.flush(O);
  }
}

// Scratch of a voxelization: the large-triangle list, then 256 bytes for its
// length, then 256 bytes for the MeshPrep record.
static size_t large_list_bytes(int64_t n_tris) {
  return (sizeof(int64_t) * (size_t)std::max<int64_t>(n_tris, 1) + 255) / 256 * 256;
}
size_t voxelize_scratch_bytes(int64_t n_tris) { return large_list_bytes(n_tris) + 512; }
MeshPrep* voxelize_prep_record(void* scratch, int64_t n_tris) {
  return (MeshPrep*)((char*)scratch + large_list_bytes(n_tris) + 256);
}

// Order-preserving 32-bit keys of floats (not NaN): unsigned comparison of
// keys is float comparison, with -0 below +0.
__device__ __forceinline__ uint32_t fkey(float f) {
  const uint32_t b = __float_as_uint(f);
  return (b & 0x80000000u) ? ~b : (b | 0x80000000u);
}
__device__ __forceinline__ float fkey_value(uint32_t k) {
  return __uint_as_float((k & 0x80000000u) ? (k & 0x7fffffffu) : ~k);
}

// Triangle indices at or past the vertex count (the largest one is kept),
// and with `bounds` the vertices' bounding box (NaN coordinates ignored, as
// the left-to-right min / max of import.cpp:49-52 ignores them).
__global__ void __launch_bounds__(256) k_mesh_scan(const float* __restrict__ V, int64_t nv,
                                                   const uint32_t* __restrict__ I, int64_t n_idx, bool bounds,
                                                   MeshPrep* P) {
  uint32_t lo[3] = {0xffffffffu, 0xffffffffu, 0xffffffffu}, hi[3] = {0u, 0u, 0u};
  unsigned long long bad = 0ull;
  const int64_t stride = (int64_t)gridDim.x * blockDim.x;
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n_idx; i += stride) {
    const uint32_t vi = I[i];
    if ((int64_t)vi >= nv) bad = max(bad, (1ull << 32) | vi);
  }
  if (bounds)
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < nv; i += stride)
      for (int c = 0; c < 3; ++c) {
        const float f = V[3 * i + c];
        if (f == f) {
          lo[c] = min(lo[c], fkey(f));
          hi[c] = max(hi[c], fkey(f));
        }
      }
  // warp, then block (256 threads), then one atomic per value and block
  for (int o = 16; o > 0; o >>= 1) {
    bad = max(bad, __shfl_xor_sync(0xffffffffu, bad, o));
    for (int c = 0; c < 3; ++c) {
      lo[c] = min(lo[c], __shfl_xor_sync(0xffffffffu, lo[c], o));
      hi[c] = max(hi[c], __shfl_xor_sync(0xffffffffu, hi[c], o));
    }
  }
  __shared__ unsigned long long s_bad[8];
  __shared__ uint32_t s_lo[3][8], s_hi[3][8];
  const int warp = threadIdx.x >> 5;
  if ((threadIdx.x & 31) == 0) {
    s_bad[warp] = bad;
    for (int c = 0; c < 3; ++c) { s_lo[c][warp] = lo[c]; s_hi[c][warp] = hi[c]; }
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    for (int w = 1; w < (int)(blockDim.x >> 5); ++w) {
      bad = max(bad, s_bad[w]);
      for (int c = 0; c < 3; ++c) { lo[c] = min(lo[c], s_lo[c][w]); hi[c] = max(hi[c], s_hi[c][w]); }
    }
    if (bad) atomicMax(&P->bad, bad);
    if (bounds)
      for (int c = 0; c < 3; ++c) {
        if (lo[c] != 0xffffffffu) atomicMin(&P->kmin[c], lo[c]);
        if (hi[c] != 0u) atomicMax(&P->kmax[c], hi[c]);
      }
  }
}

// computeMeshTransform (import.cpp:46-64) from the scanned bounds, in the
// host's float and double arithmetic, then the vertex shader's
// modelTransform * v * voxelResolution (voxelize.vs:20-27) on every vertex in
// place.  One block; every thread computes the same matrix.
__global__ void k_mesh_fit(float* __restrict__ V, int64_t nv, int32_t rx, int32_t ry, int32_t rz,
                           const MeshPrep* P) {
  float bmin[3], bmax[3];
  for (int c = 0; c < 3; ++c) {   // an axis whose coordinates are all NaN keeps +inf / -inf, as on the host
    bmin[c] = P->kmin[c] == 0xffffffffu ? INFINITY : fkey_value(P->kmin[c]);
    bmax[c] = P->kmax[c] == 0u ? -INFINITY : fkey_value(P->kmax[c]);
  }
  const float res[3] = {(float)rx, (float)ry, (float)rz};
  float size[3], margin[3];
  for (int c = 0; c < 3; ++c) { size[c] = bmax[c] - bmin[c]; margin[c] = 1.0f / res[c]; }
  int major = 0;
  if (size[1] > size[major]) major = 1;
  if (size[2] > size[major]) major = 2;
  const float sc = (float)((1.0f - 2.0 * (double)margin[major]) / (double)size[major]);
  float M[12];
  for (int r = 0; r < 3; ++r) {
    const float t = -bmin[r] + margin[r] / sc;
    M[4 * r] = r == 0 ? sc : 0.0f;
    M[4 * r + 1] = r == 1 ? sc : 0.0f;
    M[4 * r + 2] = r == 2 ? sc : 0.0f;
    M[4 * r + 3] = t * sc;
  }
  const int64_t stride = (int64_t)gridDim.x * blockDim.x;
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < nv; i += stride) {
    const float x = V[3 * i], y = V[3 * i + 1], z = V[3 * i + 2];
    for (int r = 0; r < 3; ++r) {
      const float p = ((M[4 * r] * x + M[4 * r + 1] * y) + M[4 * r + 2] * z) + M[4 * r + 3] * 1.0f;
      V[3 * i + r] = p * res[r];
    }
  }
}

cudaError_t launch_mesh_prep(float* V, int64_t nv, const uint32_t* I, int64_t n_tris, bool fit, int32_t rx,
                             int32_t ry, int32_t rz, MeshPrep* P, int sm_count, cudaStream_t st) {
  MeshPrep init;
  for (int c = 0; c < 3; ++c) { init.kmin[c] = 0xffffffffu; init.kmax[c] = 0u; }
  init.bad = 0ull;
  // pageable source: read when the copy returns
  cudaError_t e = cudaMemcpyAsync(P, &init, sizeof(init), cudaMemcpyHostToDevice, st);
  if (e != cudaSuccess) return e;
  const int64_t work = std::max<int64_t>(3 * n_tris, fit ? nv : 0);
  if (work <= 0) return cudaSuccess;
  const int blocks = (int)std::min<int64_t>((work + 255) / 256, (int64_t)sm_count * 8);
  k_mesh_scan<<<blocks, 256, 0, st>>>(V, nv, I, 3 * n_tris, fit, P);   // 256 threads: eight warps
  if (fit && nv > 0) {
    // the matrix needs the whole scan: a second launch, each block rebuilds it
    const int fb = (int)std::min<int64_t>((nv + 255) / 256, (int64_t)sm_count * 8);
    k_mesh_fit<<<fb, 256, 0, st>>>(V, nv, rx, ry, rz, P);
  }
  return cudaGetLastError();
}

cudaError_t launch_voxelize(const float* verts_voxel_space, int64_t n_vertices, const uint32_t* indices,
                            int64_t n_tris, int32_t rx, int32_t ry, int32_t rz, int32_t mode, bool reference_bounds,
                            uint8_t* grid, uint8_t value, unsigned long long* bricks, int32_t bx, int32_t by,
                            const BrickShape& sh, void* scratch, int large_blocks, cudaStream_t st) {
  if (n_tris <= 0) return cudaSuccess;
  int64_t* large = (int64_t*)scratch;
  unsigned long long* n_large = (unsigned long long*)((char*)scratch + large_list_bytes(n_tris));
  cudaError_t e = cudaMemsetAsync(n_large, 0, sizeof(unsigned long long), st);
  if (e != cudaSuccess) return e;
  VoxOut O;
  O.grid = grid;
  O.value = value;
  O.bricks = bricks ? bricks : nullptr;
  O.bx = bx;
  O.by = by;
  O.sh = sh;
  k_vox_small<<<(unsigned)((n_tris + 127) / 128), 128, 0, st>>>(verts_voxel_space, n_vertices, indices, n_tris, rx,
                                                                ry, rz, mode, reference_bounds, O, large, n_large);
  k_vox_large<<<std::max(1, large_blocks), 256, 0, st>>>(verts_voxel_space, n_vertices, indices, large, n_large, rx,
                                                         ry, rz, mode, reference_bounds, O);
  return cudaGetLastError();
}

// Word of brick (ix, iy, iz) of the padded grid of an empty volume: all bits
// of a border brick, and of an interior brick the bits of voxels at or
// beyond (rx, ry, rz); zero for every other brick.
__device__ __forceinline__ unsigned long long empty_brick_word(int ix, int iy, int iz, int32_t px, int32_t py,
                                                               int32_t pz, int32_t rx, int32_t ry, int32_t rz,
                                                               const BrickShape& sh) {
  if (ix == 0 || iy == 0 || iz == 0 || ix == px - 1 || iy == py - 1 || iz == pz - 1) return ~0ull;   // border
  const int ex = 1 << sh.sx, ey = 1 << sh.sy, ez = 1 << sh.sz;
  const int x0 = (ix - 1) * ex, y0 = (iy - 1) * ey, z0 = (iz - 1) * ez;
  unsigned long long w = 0ull;
  if (x0 < 0 || y0 < 0 || z0 < 0 || x0 + ex > rx || y0 + ey > ry || z0 + ez > rz) {
    for (int k = 0; k < 64; ++k) {
      const int x = x0 + (k & (ex - 1)), y = y0 + ((k >> sh.sx) & (ey - 1)), z = z0 + (k >> (sh.sx + sh.sy));
      if (x < 0 || y < 0 || z < 0 || x >= rx || y >= ry || z >= rz) w |= 1ull << k;
    }
  }
  return w;
}

// The bricks of an empty volume that are not zero, over a zeroed array: the
// border and the last interior brick along each axis (the only interior
// bricks that can reach past the volume).  One warp per row of the padded
// grid: rows in the y or z shell are written whole, the others at their
// three x-shell bricks (0, px - 2, px - 1).
__global__ void k_bricks_shell(unsigned long long* __restrict__ bricks, int32_t rx, int32_t ry, int32_t rz,
                               int32_t bx, int32_t by, int32_t bz, const BrickShape sh) {
  const int px = bx + 2, py = by + 2, pz = bz + 2;
  const int lane = threadIdx.x & 31;
  const int64_t rows = (int64_t)py * pz;
  const int64_t warps = (int64_t)gridDim.x * (blockDim.x >> 5);
  for (int64_t r = (int64_t)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5); r < rows; r += warps) {
    const int iz = (int)(r / py), iy = (int)(r - (int64_t)iz * py);
    unsigned long long* row = bricks + r * px;
    if (iy == 0 || iy >= py - 2 || iz == 0 || iz >= pz - 2) {
      for (int ix = lane; ix < px; ix += 32) row[ix] = empty_brick_word(ix, iy, iz, px, py, pz, rx, ry, rz, sh);
    } else if (lane < 3) {
      const int ix = lane == 0 ? 0 : px - 3 + lane;
      row[ix] = empty_brick_word(ix, iy, iz, px, py, pz, rx, ry, rz, sh);
    }
  }
}

cudaError_t launch_bricks_init(unsigned long long* bricks, int32_t rx, int32_t ry, int32_t rz, int32_t bx,
                               int32_t by, int32_t bz, const BrickShape& sh, cudaStream_t st) {
  // a linear zero fill runs at copy bandwidth; the shell is a few rows' worth
  const int64_t px = bx + 2, py = by + 2, pz = bz + 2;
  cudaError_t e = cudaMemsetAsync(bricks, 0, sizeof(unsigned long long) * (size_t)(px * py * pz), st);
  if (e != cudaSuccess) return e;
  const int64_t blocks = std::min<int64_t>((py * pz + 7) / 8, 8192);
  k_bricks_shell<<<(unsigned)blocks, 256, 0, st>>>(bricks, rx, ry, rz, bx, by, bz, sh);
  return cudaGetLastError();
}

}  // namespace vt
