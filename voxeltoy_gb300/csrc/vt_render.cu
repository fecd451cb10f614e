// vt_render.cu — path-tracing kernels.
//
//   k_plain       one thread per pixel, `passes` samples per launch; the
//                 reference's one-pass-per-draw structure (renderer.cpp:584-611)
//   wavefront     many jobs and passes per launch, in rounds of two kernels:
//                 k_wf_shade (one thread per path slot: segment results ->
//                 shading -> new segments appended to a queue by warp
//                 ballot, new items started as paths finish) and k_wf_trace
//                 (DDA of every queued segment with per-warp refill from the
//                 queue); per-sample outputs land in a sample buffer that
//                 k_wf_accumulate reduces in sample order.
//   k_paths       one thread per sample (launches of few samples)
//   k_paths_block wavefronts inside blocks, one kernel per launch (launches of
//                 up to a few million samples)
//   k_diag        per-sample output and first-hit record (parity tests)
//   k_trace_rays  DDA of caller-supplied rays (parity tests)
//   k_pick        focal-distance pick of one pixel (focalDistance.vs:45-81)
//   k_resolve     average = sum / n (+ tonemap / flip) for readback
#include "vt_kernels.h"
#include "vt_shade.cuh"

namespace vt {

template <bool kCount>
__device__ __forceinline__ void flush_counters(Cnt<kCount>& cnt, unsigned long long* out) {
  if (!kCount || out == nullptr) return;
#pragma unroll
  for (int i = 0; i < C_NUM; ++i) {
    unsigned long long v = cnt.c[i];
    for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
    if ((threadIdx.x & 31) == 0 && v) atomicAdd(&out[i], v);
  }
}

// Samples a warp of the thread-per-sample kernels takes, 8, 16 or 32: the
// fewest that leave about one wave of warps (16 an SM are resident).  A warp
// runs the union of its lanes' paths, so a launch that leaves warps free
// spreads its samples over more of them, down to 8 (160x120 samples of 64^3
// spheres 142 us at 32 a warp, 125 at 16, 118 at 8; 240x180 143, 129, 132;
// 256x192 of 128^3 noise 218, 232, 319).
int samples_per_warp(int64_t n, int sm_count) {
  int per = 8;
  while (per < 32 && (n + per - 1) / per > 18 * (int64_t)sm_count) per *= 2;
  return per;
}

// ------------------------------------------------------------------ plain
template <bool kCount>
__global__ void __launch_bounds__(128) k_plain(const Frame F, const JobDev J, int sample_base, int passes,
                                               int per_warp, unsigned long long* counters) {
  Cnt<kCount> cnt;
#pragma unroll
  for (int i = 0; i < C_NUM; ++i) cnt.c[i] = 0;
  const int lane = threadIdx.x & 31;
  const int idx = (int)(blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5)) * per_warp + lane;
  const int n = F.width * F.height;
  if (lane < per_warp && idx < n) {
    const int px = idx % F.width, py = idx / F.width;
    float4 sum = J.sum[idx], comp = J.comp[idx];
    for (int k = 0; k < passes; ++k) {
      const float4 v = trace_sample(F, J, px, py, sample_base + k, cnt, (HitRecord*)nullptr);
      kahan_add(sum, comp, v);
    }
    J.sum[idx] = sum;
    J.comp[idx] = comp;
  }
  flush_counters(cnt, counters);
}

// The edit-mode integrator by itself: a warp takes a tile of 8 x per_warp / 8
// pixels.  What bounds it is the latency of the longest rays' dependent brick
// reads, and the instructions between them.  Without the path tracer's code it
// fits in half of k_plain's 128 registers, so that a 512^2 image's warps run in
// two turns instead of four, and the rays of a tile end closer together than
// those of a row.  Eight resident blocks, without spills; at twelve, with 64
// bytes of them, more warps run at once and every image is slower: a 1.3
// M-triangle mesh into 1024^3 and its first 512^2 image 1017 us against 982, 8
// passes of 512^2 of 128^3 noise 355 against 315 (541 in k_plain), a 160x120
// view inside a 48^3 room 36.1 us against 31.8 (34.5).
template <bool kCount>
__global__ void __launch_bounds__(128, 8) k_edit(const Frame F, const JobDev J, int sample_base, int passes,
                                                  int per_warp, int tiles_x, unsigned long long* counters) {
  Cnt<kCount> cnt;
#pragma unroll
  for (int i = 0; i < C_NUM; ++i) cnt.c[i] = 0;
  const int lane = threadIdx.x & 31;
  const int tile = (int)(blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5));
  const int ty = tile / tiles_x;
  const int px = 8 * (tile - ty * tiles_x) + (lane & 7), py = (per_warp >> 3) * ty + (lane >> 3);
  if (lane < per_warp && px < F.width && py < F.height) {
    const int idx = py * F.width + px;
    for (int k = 0; k < passes; ++k) {
      const float4 v = edit_sample(F, J, px, py, sample_base + k, cnt, (HitRecord*)nullptr);
      float4 sum = J.sum[idx], comp = J.comp[idx];   // not held across the walks
      kahan_add(sum, comp, v);
      J.sum[idx] = sum;
      J.comp[idx] = comp;
    }
  }
  flush_counters(cnt, counters);
}

cudaError_t launch_plain(const Frame& F, const JobDev& J, int sample_base, int passes, int sm_count,
                         unsigned long long* counters, cudaStream_t st) {
  const int n = F.width * F.height;
  const int threads = 128;
  const int per_warp = samples_per_warp(n, sm_count);
  if (F.integrator == 1) {
    const int tiles_x = (F.width + 7) / 8, tiles_y = (F.height + per_warp / 8 - 1) / (per_warp / 8);
    const unsigned blocks = (unsigned)(((int64_t)tiles_x * tiles_y + threads / 32 - 1) / (threads / 32));
    if (counters) k_edit<true><<<blocks, threads, 0, st>>>(F, J, sample_base, passes, per_warp, tiles_x, counters);
    else k_edit<false><<<blocks, threads, 0, st>>>(F, J, sample_base, passes, per_warp, tiles_x, nullptr);
    return cudaGetLastError();
  }
  const int warps = (n + per_warp - 1) / per_warp, blocks = (warps + threads / 32 - 1) / (threads / 32);
  if (counters) k_plain<true><<<blocks, threads, 0, st>>>(F, J, sample_base, passes, per_warp, counters);
  else k_plain<false><<<blocks, threads, 0, st>>>(F, J, sample_base, passes, per_warp, nullptr);
  return cudaGetLastError();
}

// ------------------------------------------------------------------- diag
__global__ void k_diag(const Frame F, const JobDev J, int sample, float4* out, HitRecord* hits,
                       unsigned long long* counters) {
  Cnt<true> cnt;
#pragma unroll
  for (int i = 0; i < C_NUM; ++i) cnt.c[i] = 0;
  const int idx = blockIdx.x * blockDim.x + threadIdx.x;
  const int n = F.width * F.height;
  if (idx < n) {
    const int px = idx % F.width, py = idx / F.width;
    HitRecord h;
    const float4 v = F.integrator == 1 ? edit_sample(F, J, px, py, sample, cnt, &h)
                                       : trace_sample(F, J, px, py, sample, cnt, &h);
    out[idx] = v;
    if (hits) hits[idx] = h;
  }
  flush_counters(cnt, counters);
}

cudaError_t launch_diag(const Frame& F, const JobDev& J, int sample, float4* out, HitRecord* hits,
                        unsigned long long* counters, cudaStream_t st) {
  const int n = F.width * F.height;
  k_diag<<<(n + 127) / 128, 128, 0, st>>>(F, J, sample, out, hits, counters);
  return cudaGetLastError();
}

// -------------------------------------------------------------- wavefront
// Slot flags.
enum : uint32_t {
  SL_BOUNCES = 0xffu,
  SL_PRIMARY = 1u << 8,
  SL_HAS_CONT = 1u << 9,
  SL_EXT = 1u << 10,      // an extension segment was traced for this slot
  SL_SHADOW = 1u << 11,   // a shadow segment was traced for this slot
  SL_ACTIVE = 1u << 12,   // a path (0: an empty position of the stream)
  // bits 14..16: non-finite throughput components of the pending light sample
  // bits 17..31: job of the path
};
constexpr int kSlotJobShift = 17;
static_assert(kWfMaxJobs == (1 << (32 - kSlotJobShift)), "job bits of the slot flags");

__device__ __forceinline__ v3 xyz4(float4 v) { return mk3(v.x, v.y, v.z); }
__device__ __forceinline__ float4 pack4(v3 a, float w) { return make_float4(a.x, a.y, a.z, w); }

// Job and grid records: from the global tables, or (WfJobTable) from the
// kernel's parameter block.
struct WfNoTable {
  int unused;
};
template <class Par>
__device__ __forceinline__ const JobEntry& job_entry(const Par& P, const WfNoTable&, uint32_t j) {
  return P.jobs[j];
}
template <class Par>
__device__ __forceinline__ const JobEntry& job_entry(const Par&, const WfJobTable& T, uint32_t j) {
  return T.e[j];
}
template <class Par>
__device__ __forceinline__ const Grid& grid_entry(const Par& P, const WfNoTable&, uint32_t j) {
  return P.grids[j];
}
template <class Par>
__device__ __forceinline__ const Grid& grid_entry(const Par&, const WfJobTable& T, uint32_t j) {
  return T.g[j];
}
template <class Par>
__device__ __forceinline__ const JobEntry& job_entry(const Par&, const WfOneJob& T, uint32_t) { return T.e; }
template <class Par>
__device__ __forceinline__ const Grid& grid_entry(const Par&, const WfOneJob& T, uint32_t) { return T.g; }

// Job of a global item index (binary search over tile_begin).
template <class Par>
__device__ __forceinline__ int job_of(const Par&, const WfOneJob&, unsigned long long) { return 0; }
template <class Par, class Tab>
__device__ __forceinline__ int job_of(const Par& P, const Tab& T, unsigned long long item) {
  int lo = 0, hi = P.n_jobs - 1;
  while (lo < hi) {
    const int mid = (lo + hi + 1) >> 1;
    if ((unsigned long long)job_entry(P, T, (uint32_t)mid).tile_begin <= item) lo = mid; else hi = mid - 1;
  }
  return lo;
}

// Path state (WfState): a0 = (ro, -), a1 = (rd, item), a3 = (L, rng),
// a4 = (T, bsdf_pdf), a5 = (nee_P, light) for paths with a shadow segment;
// the job, bounces and flag bits live in `flags`, and pixel and sample
// follow from the item.
// k_wf_shade reads what ending a segment needs (a1, a3, a4, a5 for a shadow
// result, a0 for a hit it keeps) and copies kept hits into hit records;
// k_wf_hit reads only the hit records.
__device__ __forceinline__ void load_flags(uint32_t fl, Path& p) {
  p.bounces = (int)(fl & SL_BOUNCES);
  p.primary = (fl & SL_PRIMARY) ? 1 : 0;
  p.has_cont = (fl & SL_HAS_CONT) ? 1 : 0;
  p.nee_nf = (int)((fl >> 14) & 7u);
}

__device__ __forceinline__ void load_for_shade(const WfState& st, int i, uint32_t fl, Path& p, uint32_t& item,
                                               float& rng_word) {
  const float4 a1 = st.a1[i], a3 = st.a3[i], a4 = st.a4[i];
  p.rd = xyz4(a1);
  item = __float_as_uint(a1.w);
  p.L = xyz4(a3);
  rng_word = a3.w;
  p.T = xyz4(a4); p.bsdf_pdf = a4.w;
  if (fl & SL_SHADOW) {
    const float4 a5 = st.a5[i];
    p.nee_P = xyz4(a5); p.light = __float_as_int(a5.w);
  }
  load_flags(fl, p);
}

__device__ __forceinline__ void rng_from_item(const JobEntry& E, uint32_t item, uint32_t rng, Path& p) {
  // item - tile_begin = pass * n_pixels + pixel (< 2^32 items per launch)
  const uint32_t r = item - (uint32_t)E.tile_begin;
  const uint32_t np = (uint32_t)E.n_pixels;   // = width * height
  const uint32_t pass = udiv(r, E.F.m_pixels);
  p.rng.pixel = r - pass * np;
  p.rng.sample = (uint32_t)E.sample_base + pass;
  if (E.F.rng_mode == 1) { p.rng.ox = (int32_t)(rng & 0xffffu); p.rng.oy = (int32_t)(rng >> 16); p.rng.call = 0; }
  else { p.rng.call = rng; p.rng.ox = p.rng.oy = 0; }
}

// The state the next round's shading reads (the shadow direction is only
// needed for the segment record written beside it, so it is not stored).
__device__ __forceinline__ void store_path(const WfState& st, int i, const Frame& F, const Path& p, uint32_t item,
                                           bool shadow) {
  const uint32_t rng = (F.rng_mode == 1) ? ((uint32_t)p.rng.ox | ((uint32_t)p.rng.oy << 16)) : p.rng.call;
  st.a0[i] = pack4(p.ro, 0.0f);
  st.a1[i] = pack4(p.rd, __uint_as_float(item));
  st.a3[i] = pack4(p.L, __uint_as_float(rng));
  st.a4[i] = pack4(p.T, p.bsdf_pdf);
  if (shadow) st.a5[i] = pack4(p.nee_P, __int_as_float(p.light));
}

// Block-wide reservation on N counters with one atomic per counter and
// block instead of per warp: `n[i]` is this thread's count for counter i;
// returns in base[i] the first entry of the thread's warp (the offsets of
// the thread within its warp come from ballots).  Every thread of the block
// must call it (three barriers).
constexpr int kWfWarps = 4;   // warps per shade / hit / regen block (128 threads)
template <int N>
__device__ __forceinline__ void block_reserve(uint32_t* const (&ctr)[N], const uint32_t (&n)[N], uint32_t (&base)[N]) {
  __shared__ uint32_t s_n[N][kWfWarps];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
#pragma unroll
  for (int i = 0; i < N; ++i) {
    uint32_t v = n[i];
    for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
    if (lane == 0) s_n[i][warp] = v;
  }
  __syncthreads();
  if (threadIdx.x < N) {
    const int i = threadIdx.x;
    uint32_t t = 0, pre[kWfWarps];
#pragma unroll
    for (int w = 0; w < kWfWarps; ++w) { pre[w] = t; t += s_n[i][w]; }
    const uint32_t b0 = t ? atomicAdd(ctr[i], t) : 0u;
#pragma unroll
    for (int w = 0; w < kWfWarps; ++w) s_n[i][w] = b0 + pre[w];
  }
  __syncthreads();
#pragma unroll
  for (int i = 0; i < N; ++i) base[i] = s_n[i][warp];
  __syncthreads();   // the next call may overwrite s_n
}

// Write this warp's next segments (queue entries from `base`) as 32-byte ray
// records {vo.xyz, inc.x} {inc.yz, slot << 1 | kind, job}: the origin in
// voxel space and the reciprocal direction as seg_rec gives them to the DDA
// set-up, computed here in coherent warps rather than by the DDA kernel's
// lanes as they start segments at different times.  The warp's extension
// records first, then its shadow records.  emit: 1 extension (from
// `ext_o`), 2 shadow.
__device__ __forceinline__ void write_segments(const WfParams& P, int par, uint32_t base, uint32_t emit, int slot,
                                               uint32_t job, v3 ext_o, const Path& p, const Frame& F) {
  const unsigned FULL = 0xffffffffu;
  const unsigned lt = (1u << (threadIdx.x & 31)) - 1u;
  const uint32_t n1 = (emit & 1u) ? 1u : 0u, n2 = (emit & 2u) ? 1u : 0u;
  const unsigned b1 = __ballot_sync(FULL, n1), b2 = __ballot_sync(FULL, n2);
  float4* q = P.queue[par];
  if (n1) {
    const size_t at = 2 * (size_t)(base + __popc(b1 & lt));
    const SegRec sr = seg_rec(F, ext_o, p.rd);
    q[at] = make_float4(sr.vo.x, sr.vo.y, sr.vo.z, sr.inc.x);
    q[at + 1] = make_float4(sr.inc.y, sr.inc.z, __uint_as_float((uint32_t)slot << 1), __uint_as_float(job));
  }
  if (n2) {
    const size_t at = 2 * (size_t)(base + __popc(b1) + __popc(b2 & lt));
    const SegRec sr = seg_rec(F, p.ro, p.sd);
    q[at] = make_float4(sr.vo.x, sr.vo.y, sr.vo.z, sr.inc.x);
    q[at + 1] = make_float4(sr.inc.y, sr.inc.z, __uint_as_float(((uint32_t)slot << 1) | 1u), __uint_as_float(job));
  }
}

__device__ __forceinline__ uint32_t slot_flags(const Path& p, uint32_t emit, uint32_t job) {
  return SL_ACTIVE | (uint32_t)(p.bounces & 0xff) | (p.primary ? SL_PRIMARY : 0u) | (p.has_cont ? SL_HAS_CONT : 0u) |
         ((emit & 1u) ? SL_EXT : 0u) | ((emit & 2u) ? SL_SHADOW : 0u) | ((uint32_t)(p.nee_nf & 7) << 14) |
         (job << kSlotJobShift);
}

// A round has four kernels over the stream x[par] (n paths, written by the
// previous round) and builds the stream x[par ^ 1]:
//   k_wf_shade  every position: shadow results (NEE added if visible),
//               extension results (miss -> environment, bounce limit,
//               selection), finished paths -> sample buffer; surviving hits
//               -> hit records, Lambert hits from the front of the list, the
//               others from its back, so that k_wf_hit's warps mostly run one
//               BSDF
//   k_wf_hit    the hit records: vertex shading, light and BSDF samples;
//               writes its paths to positions [0, hits) of the next stream
//               and their next segments to the queue; reserves the first
//               items of the new paths
//   k_wf_regen  new paths in positions [hits, capacity) of the next stream,
//               primary segments to the queue after the hit kernel's
//   k_wf_trace  the queue: DDA of every segment, ends stored by position
// Every state access is to consecutive positions.  k_wf_hit keeps eight
// resident blocks per SM (64 registers): the extra warps hide more of the
// load latency than the few spills cost; the lighter k_wf_shade and (with one
// job) k_wf_regen fit twelve.
template <bool kCount, class Tab>
__global__ void __launch_bounds__(128, 12) k_wf_shade(const WfParams P, const __grid_constant__ Tab T, int par) {
  const unsigned FULL = 0xffffffffu;
  const int lane = threadIdx.x & 31;
  const unsigned lt = (1u << lane) - 1u;
  if (blockIdx.x == 0 && threadIdx.x == 0)    // items taken before this round, for k_wf_regen
    *(unsigned long long*)&P.ctl[ctl_index(par, CTL_ITEM_SNAP)] = *(volatile unsigned long long*)P.next_item;
  const uint32_t n = *(volatile uint32_t*)&P.ctl[ctl_index(par ^ 1, CTL_NEXT_N)];
  if (blockIdx.x * blockDim.x >= n) return;   // the whole block lies beyond the stream
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  const WfState& src = P.x[par];
  Cnt<kCount> cnt;
#pragma unroll
  for (int k = 0; k < C_NUM; ++k) cnt.c[k] = 0;
  const uint32_t fl = (uint32_t)i < n ? src.flags[i] : 0u;
  bool hit = false;
  int cls = 0;
  Path p;
  uint32_t item = 0;
  float rng_word = 0.0f;
  SegEnd e;
  e.x = e.y = e.z = e.state = 0;
  if (fl & SL_ACTIVE) {
    cnt.add(C_POSITIONS, 1);
    const uint32_t job = fl >> kSlotJobShift;
    const JobEntry& E = job_entry(P, T, job);
    // every load of the position is issued before any of them is used (the
    // origin is read for every extension, whether or not it hits)
    const unsigned long long hs = (fl & SL_SHADOW) ? P.hits[(size_t)P.n_slots + i] : 0ull;
    const unsigned long long he = (fl & SL_EXT) ? P.hits[i] : 0ull;
    const float4 a0v = (fl & SL_EXT) ? src.a0[i] : make_float4(0.f, 0.f, 0.f, 0.f);
    load_for_shade(src, i, fl, p, item, rng_word);
    if (fl & SL_SHADOW) shadow_end(E.F, p, unpack_end(hs));
    if (fl & SL_EXT) {
      e = unpack_end(he);
      hit = ext_resolve(E.F, E.J, p, e, cnt);
      if (hit) cls = hit_class(E.F, E.J, e);
    }
    if (hit) p.ro = xyz4(a0v);
    else if (chk(item < P.n_items, CHK_SAMPLE)) P.sbuf[item] = path_output(E.F, p);
  }
  uint32_t* const ctr[2] = {&P.ctl[ctl_index(par, CTL_HITS_LAMBERT)], &P.ctl[ctl_index(par, CTL_HITS_OTHER)]};
  const uint32_t cnt_l = (hit && cls == 0) ? 1u : 0u, cnt_o = (hit && cls != 0) ? 1u : 0u;
  const uint32_t nn[2] = {cnt_l, cnt_o};
  uint32_t base[2];
  block_reserve<2>(ctr, nn, base);
  const unsigned bl = __ballot_sync(FULL, cnt_l), bo = __ballot_sync(FULL, cnt_o);
  if (hit) {
    const uint32_t j = cnt_l ? base[0] + __popc(bl & lt) : (uint32_t)P.n_slots - 1u - (base[1] + __popc(bo & lt));
    P.hr.h0[j] = pack4(p.ro, __uint_as_float(item));
    P.hr.h1[j] = pack4(p.rd, __uint_as_float(slot_flags(p, 1u, fl >> kSlotJobShift)));
    P.hr.h2[j] = pack4(p.L, rng_word);
    P.hr.h3[j] = pack4(p.T, p.bsdf_pdf);
    P.hr.h4[j] = pack_end(e.x, e.y, e.z, e.state);
  }
  flush_counters(cnt, P.counters);
}

// The hit records of this round: list entry v (Lambert entries [0, nl), then
// the others, stored from the back) becomes position v of the next stream.
// A block-uniform grid-stride loop.
template <bool kCount, class Tab>
__global__ void __launch_bounds__(128, 8) k_wf_hit(const WfParams P, const __grid_constant__ Tab T, int par) {
  const uint32_t nl = *(volatile uint32_t*)&P.ctl[ctl_index(par, CTL_HITS_LAMBERT)];
  const uint32_t no = *(volatile uint32_t*)&P.ctl[ctl_index(par, CTL_HITS_OTHER)];
  const uint32_t n_hits = nl + no;
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    // items [taken, taken + m) go to k_wf_regen's m positions, position k
    // taking item taken + k first; its lanes claim further items only after
    const unsigned long long taken = *(volatile unsigned long long*)&P.ctl[ctl_index(par, CTL_ITEM_SNAP)];
    const unsigned long long left = P.n_items > taken ? P.n_items - taken : 0ull;
    const uint32_t m = (uint32_t)min((unsigned long long)((uint32_t)P.n_slots - n_hits), left);
    if (m) atomicAdd(P.next_item, (unsigned long long)m);
  }
  const WfState& dst = P.x[par ^ 1];
  Cnt<kCount> cnt;
#pragma unroll
  for (int k = 0; k < C_NUM; ++k) cnt.c[k] = 0;
  const uint32_t stride = gridDim.x * blockDim.x;
  for (uint32_t b0 = blockIdx.x * blockDim.x; b0 < n_hits; b0 += stride) {   // block-uniform
    const uint32_t v = b0 + threadIdx.x;
    const bool mine = v < n_hits;
    Path p;
    uint32_t job = 0, item = 0;
    uint32_t emit = 0;
    if (mine) {
      const uint32_t j = v < nl ? v : (uint32_t)P.n_slots - 1u - (v - nl);
      const float4 h0 = P.hr.h0[j], h1 = P.hr.h1[j], h2 = P.hr.h2[j], h3 = P.hr.h3[j];
      const unsigned long long h4 = P.hr.h4[j];
      const uint32_t fl = __float_as_uint(h1.w);
      job = fl >> kSlotJobShift;
      const JobEntry& E = job_entry(P, T, job);
      p.ro = xyz4(h0);
      item = __float_as_uint(h0.w);
      p.rd = xyz4(h1);
      p.L = xyz4(h2);
      p.T = xyz4(h3); p.bsdf_pdf = h3.w;
      load_flags(fl, p);
      rng_from_item(E, item, __float_as_uint(h2.w), p);
      const SegEnd e = unpack_end(h4);
      ext_hit(E.F, E.J, p, e, cnt);
      emit = 2u | (p.has_cont ? 1u : 0u);
    }
    uint32_t* const ctr[1] = {&P.ctl[ctl_index(par, CTL_QCOUNT)]};
    const uint32_t nn[1] = {(emit & 1u) + (emit >> 1)};
    uint32_t base[1];
    block_reserve<1>(ctr, nn, base);
    write_segments(P, par, base[0], emit, (int)v, job, p.ro, p, job_entry(P, T, job).F);
    if (mine) {
      store_path(dst, (int)v, job_entry(P, T, job).F, p, item, (emit & 2u) != 0);
      dst.flags[v] = slot_flags(p, emit, job);
    }
  }
  flush_counters(cnt, P.counters);
}

// New paths at positions [hits, hits + m) of the next stream, m = the free
// capacity or the items left, whichever is smaller.  Position k starts with
// item taken + k (reserved by k_wf_hit); a lane whose path misses its job's
// volume (finished at once) claims further items with one atomic per warp,
// until a path enters the volume or the items run out (the position stays
// empty).  The primary segment starts at the volume entry point; position
// k's queue record is entry QCOUNT + k of the round's queue (the hit
// kernel's records come first), a record without a segment for an empty
// position, so that the kernel needs no block-wide reservation.
// Resident blocks the new-path kernel is compiled for: twelve with one job
// (40 registers, no spill), eight with a job table (whose records need more).
template <class Tab> struct RegenBlocks { static constexpr int value = 8; };
template <> struct RegenBlocks<WfOneJob> { static constexpr int value = 12; };

template <bool kCount, class Tab>
__global__ void __launch_bounds__(128, RegenBlocks<Tab>::value) k_wf_regen(const WfParams P, const __grid_constant__ Tab T, int par) {
  const unsigned FULL = 0xffffffffu;
  const int lane = threadIdx.x & 31;
  const unsigned lt = (1u << lane) - 1u;
  const uint32_t n_hits = *(volatile uint32_t*)&P.ctl[ctl_index(par, CTL_HITS_LAMBERT)] +
                          *(volatile uint32_t*)&P.ctl[ctl_index(par, CTL_HITS_OTHER)];
  const unsigned long long taken = *(volatile unsigned long long*)&P.ctl[ctl_index(par, CTL_ITEM_SNAP)];
  const unsigned long long left = P.n_items > taken ? P.n_items - taken : 0ull;
  const uint32_t m = (uint32_t)min((unsigned long long)((uint32_t)P.n_slots - n_hits), left);
  const uint32_t qbase = *(volatile uint32_t*)&P.ctl[ctl_index(par, CTL_QCOUNT)];
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    P.ctl[ctl_index(par, CTL_NEXT_N)] = n_hits + m;
    P.ctl[ctl_index(par, CTL_REGEN_N)] = m;
  }
  // the next round's counters: this round's shading, which read the stream
  // length among them, is done
  if (blockIdx.x == 0 && threadIdx.x < CTL_PER_PARITY) P.ctl[ctl_index(par ^ 1, (int)threadIdx.x)] = 0u;
  const WfState& dst = P.x[par ^ 1];
  float4* const q = P.queue[par];
  Cnt<kCount> cnt;
#pragma unroll
  for (int k = 0; k < C_NUM; ++k) cnt.c[k] = 0;
  const uint32_t stride = gridDim.x * blockDim.x;
  for (uint32_t b0 = blockIdx.x * blockDim.x; b0 < m; b0 += stride) {   // block-uniform
    const uint32_t k = b0 + threadIdx.x;
    const bool mine = k < m;
    const uint32_t pos = n_hits + k;
    unsigned long long my = taken + k;
    bool need_new = mine, active = false;
    Path p;
    uint32_t job = 0, item = 0;
    float t_enter = 0.0f;
    for (;;) {
      if (need_new) {
        if (my >= P.n_items) {
          need_new = false;   // no items left: the position stays empty
        } else {
          item = (uint32_t)my;
          job = (uint32_t)job_of(P, T, my);
          const JobEntry& E = job_entry(P, T, job);
          const uint32_t r = (uint32_t)(my - (unsigned long long)E.tile_begin);   // < 2^32 items per launch
          const uint32_t np = (uint32_t)E.n_pixels;   // = width * height
          const uint32_t pass = udiv(r, E.F.m_pixels);
          const uint32_t pixel = r - pass * np;
          const uint32_t w = (uint32_t)E.F.width;
          const int py = (int)udiv(pixel, E.F.m_width), px = (int)(pixel - (uint32_t)py * w);
          if (path_start(E.F, E.J, p, px, py, E.sample_base + (int)pass, cnt, t_enter)) {
            active = true;
            need_new = false;
          } else {
            if (chk(item < P.n_items, CHK_SAMPLE))
              P.sbuf[item] = path_output(E.F, p);   // missed the volume: finished, take another item
          }
        }
      }
      const unsigned want = __ballot_sync(FULL, need_new);
      if (!want) break;
      const int leader = __ffs(want) - 1;
      unsigned long long base = 0;
      if (lane == leader) base = atomicAdd(P.next_item, (unsigned long long)__popc(want));
      base = __shfl_sync(FULL, base, leader);
      my = base + __popc(want & lt);
    }
    if (mine) {
      const size_t at = 2 * (size_t)(qbase + k);
      if (active) {
        const v3 o = p.ro + t_enter * p.rd;   // the primary segment starts at the volume entry point
        const SegRec sr = seg_rec(job_entry(P, T, job).F, o, p.rd);
        q[at] = make_float4(sr.vo.x, sr.vo.y, sr.vo.z, sr.inc.x);
        q[at + 1] = make_float4(sr.inc.y, sr.inc.z, __uint_as_float((uint32_t)pos << 1), __uint_as_float(job));
        store_path(dst, (int)pos, job_entry(P, T, job).F, p, item, false);   // a primary path has no shadow segment
        dst.flags[pos] = slot_flags(p, 1u, job);
      } else {
        q[at + 1] = make_float4(0.0f, 0.0f, __uint_as_float(kNoSegment), 0.0f);
        dst.flags[pos] = 0u;
      }
    }
  }
  flush_counters(cnt, P.counters);
}

// Before a warp's step loop: segments that stand in a large enough free cube
// cross it in one leap (dda_leap, some 110 instructions for the warp, however
// few of its lanes take it, against 33 a step).  Asking for 4, 8 or 12 such
// lanes first measured slower: a 1024^3 shell 10.5, 11.2, 11.3 ms against 9.3,
// 256^3 noise 1-2%.
// A second leap where the first one ends in another cube: shell 8.8 ms, noise
// 118.8 against 114.2 ms.
__device__ __forceinline__ void leap(const Grid& g, Dda& s) {
  if (!g.runs) return;
  const int room = dda_room(g, s);
  if (room >= 2) dda_leap(s, room);
}

// The grid record of a lane's current segment: a register copy, or with one
// job the record in the parameter block itself (constant operands).
template <class Tab>
struct GridHold {
  Grid g;
  template <class Par>
  __device__ __forceinline__ void set(const Par& P, const Tab& T, uint32_t job) { g = grid_entry(P, T, job); }
  __device__ __forceinline__ const Grid& get(const Tab&) const { return g; }
};
template <>
struct GridHold<WfOneJob> {
  template <class Par>
  __device__ __forceinline__ void set(const Par&, const WfOneJob&, uint32_t) {}
  __device__ __forceinline__ const Grid& get(const WfOneJob& T) const { return T.g; }
};

// One round of tracing: every queued segment runs its DDA to the end.  Each
// warp takes chunks of queue records with one atomic and hands them to its
// lanes; every kTraceSteps steps (with kVote also as soon as fewer than
// P.refill_min lanes step) the lanes whose segments ended take the next ones.
// What bounds it is issue: 33 or so warp instructions a step, and per refill
// the record read and the segment set-up at the efficiency of the lanes that
// need one.  So the refill is short: no second record is kept loaded per lane
// (eight registers; the warps that then fit hide the read instead), the chunk
// hand-out is straight-line, and an end inside the volume is packed without
// clamps.  A chunk is P.trace_chunk records, but no more than leaves every
// warp four turns, down to 32: with 128 always, a queue of half a million
// records kept two thirds of the warps busy.  Measured with the prefetched
// records and fixed chunks before -> now (2 lanes, 8M slots): 1024^2 x 256 spp
// of 256^3 noise 134 -> 123 ms, 1024^2 x 16 spp of a 1024^3 shell 23.7 -> 19.9
// ms, 256^2 x 16 spp of 64^3 spheres 0.86 -> 0.72 ms, 512^2 x 1 spp 1.13 ->
// 0.94 ms.
// Resident blocks the trace kernel is compiled for: eight with one job (its
// grid record is constant; 32 registers, no spill; six blocks measure 126 and
// 20.6 ms on the two large frames), five with a job table, whose per-lane grid
// record would otherwise spill.
template <class Tab> struct TraceBlocks { static constexpr int value = 5; };
template <> struct TraceBlocks<WfOneJob> { static constexpr int value = 8; };

template <bool kCount, int kTraceSteps, bool kVote, bool k444, class Tab>
__global__ void __launch_bounds__(256, TraceBlocks<Tab>::value) k_wf_trace(const WfParams P, const __grid_constant__ Tab T, int par) {
  static_assert(kTraceSteps % 4 == 0, "the 4x4x4 loop steps four at a time");
  const unsigned FULL = 0xffffffffu;
  const int lane = threadIdx.x & 31;
  const unsigned lt = (1u << lane) - 1u;
  const uint32_t n = *(volatile uint32_t*)&P.ctl[ctl_index(par, CTL_QCOUNT)] +
                     *(volatile uint32_t*)&P.ctl[ctl_index(par, CTL_REGEN_N)];   // hit, then new-path records
  if (n == 0) return;
  const float4* q = P.queue[par];
  Cnt<kCount> cnt;
#pragma unroll
  for (int i = 0; i < C_NUM; ++i) cnt.c[i] = 0;
  const uint32_t chunk = min(P.trace_chunk, max(32u, n / (gridDim.x * 32u) & ~31u));   // eight warps a block
  uint32_t pool = 0, pool_end = 0;   // the rest of this warp's chunk of queue records
  bool have = false, more = true;    // more: the queue may hold another chunk
  GridHold<Tab> gh;
  Dda s;
  uint32_t tag = 0;   // position << 1 | kind of the current segment
  for (;;) {
    const unsigned need = __ballot_sync(FULL, !have);
    if (need) {   // idle lanes take the next records
      const uint32_t avail = pool_end - pool, want = __popc(need), r = __popc(need & lt);
      uint32_t rec = r < avail ? pool + r : n;
      pool += min(want, avail);
      if (want > avail && more) {
        uint32_t c = 0;
        if (lane == 0) c = atomicAdd(&P.ctl[ctl_index(par, CTL_QHEAD)], chunk);
        c = __shfl_sync(FULL, c, 0);
        more = c < n;
        if (more) {
          if (r >= avail) rec = c + (r - avail);   // within the chunk: it holds 32 records or more
          pool_end = min(c + chunk, n);
          pool = min(c + (want - avail), pool_end);
        }
      }
      if (!have && rec < n) {
        const float4 na = __ldg(&q[2 * (size_t)rec]), nb = __ldg(&q[2 * (size_t)rec + 1]);
        tag = __float_as_uint(nb.z);
        if (tag != kNoSegment) {
          gh.set(P, T, __float_as_uint(nb.w));
          dda_begin_rec(gh.get(T), s, mk3(na.x, na.y, na.z), mk3(na.w, nb.x, nb.y));
          if (!kCount && k444 && s.state == DDA_RUNNING) dda_end_stuck(gh.get(T), s);
          if (s.state == DDA_RUNNING) have = true;
          else P.hits[(size_t)(tag & 1u) * P.n_slots + (tag >> 1)] = pack_end(s.x, s.y, s.z, s.state);
        }
      }
      if (!__any_sync(FULL, have) && !more && pool >= pool_end) break;
    }
    if (have) {
      if constexpr (!kCount && k444) leap(gh.get(T), s);
      if constexpr (!kCount && k444) dda_steps_444<kVote>(gh.get(T), s, kTraceSteps, P.refill_min);
      else dda_steps<kCount, kVote, k444>(gh.get(T), s, kTraceSteps, cnt, P.refill_min);
      if (s.state != DDA_RUNNING) {
        P.hits[(size_t)(tag & 1u) * P.n_slots + (tag >> 1)] = pack_end_inside(s.x, s.y, s.z, s.state);
        have = false;
      }
    }
  }
  flush_counters(cnt, P.counters);
}

// One round of tracing, pooled form: each warp keeps up to kPoolSegs
// segments set up and ready to step in shared memory.  The segment set-up
// (dda_begin: nudge, divisions, floor, bounds test) runs for a warp's worth
// of queue records at once, every lane busy; a lane whose segment ended takes
// a ready one after each batch of kTraceSteps steps, so lanes rarely wait
// for a set-up.  Same segments, same ends, same bits as k_wf_trace.
constexpr int kPoolSegs = 64;
constexpr int kTraceWarps = 8;   // 256-thread blocks

__device__ __forceinline__ int32_t pack_signs(const Dda& t) {
  return (t.sx + 1) | ((t.sy + 1) << 2) | ((t.sz + 1) << 4);
}

template <bool kCount, int kTraceSteps, bool k444, class Tab>
__global__ void __launch_bounds__(256, 4) k_wf_trace_pool(const WfParams P, const __grid_constant__ Tab T, int par) {
  static_assert(kTraceSteps % 4 == 0, "the 4x4x4 loop steps four at a time");
  __shared__ int32_t s_i[4][kTraceWarps][kPoolSegs];    // x, y, z, packed signs
  __shared__ float s_f[6][kTraceWarps][kPoolSegs];      // dx, dy, dz, ax, ay, az
  __shared__ uint32_t s_u[2][kTraceWarps][kPoolSegs];   // position << 1 | kind, job
  const unsigned FULL = 0xffffffffu;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const unsigned lt = (1u << lane) - 1u;
  const uint32_t n = *(volatile uint32_t*)&P.ctl[ctl_index(par, CTL_QCOUNT)] +
                     *(volatile uint32_t*)&P.ctl[ctl_index(par, CTL_REGEN_N)];   // hit, then new-path records
  if (n == 0) return;
  const float4* q = P.queue[par];
  Cnt<kCount> cnt;
#pragma unroll
  for (int i = 0; i < C_NUM; ++i) cnt.c[i] = 0;
  uint32_t chunk = 0, chunk_end = 0;
  bool exhausted = false, active = false;
  int count = 0;   // ready segments in this warp's pool (the same in every lane)
  GridHold<Tab> gh;
  Dda s;
  uint32_t tag = 0;
  for (;;) {
    // set up new segments, a warp's worth at a time, while the pool has room
    while (count <= kPoolSegs - 32 && !exhausted) {
      if (chunk >= chunk_end) {
        uint32_t c = 0;
        if (lane == 0) c = atomicAdd(&P.ctl[ctl_index(par, CTL_QHEAD)], P.trace_chunk);
        c = __shfl_sync(FULL, c, 0);
        if (c >= n) { exhausted = true; break; }
        chunk = c;
        chunk_end = min(c + P.trace_chunk, n);
      }
      const uint32_t rec = chunk + (uint32_t)lane;
      chunk = min(chunk + 32u, chunk_end);
      bool run = false;
      Dda t;
      uint32_t ttag = 0, tjob = 0;
      if (rec < chunk_end && __float_as_uint(__ldg(&q[2 * (size_t)rec + 1]).z) != kNoSegment) {
        const float4 a = __ldg(&q[2 * (size_t)rec]), b = __ldg(&q[2 * (size_t)rec + 1]);
        ttag = __float_as_uint(b.z);
        tjob = __float_as_uint(b.w);
        GridHold<Tab> tg;
        tg.set(P, T, tjob);
        dda_begin_rec(tg.get(T), t, mk3(a.x, a.y, a.z), mk3(a.w, b.x, b.y));
        if (!kCount && k444 && t.state == DDA_RUNNING) dda_end_stuck(tg.get(T), t);
        run = t.state == DDA_RUNNING;
        if (!run) P.hits[(size_t)(ttag & 1u) * P.n_slots + (ttag >> 1)] = pack_end(t.x, t.y, t.z, t.state);
      }
      const unsigned rm = __ballot_sync(FULL, run);
      if (run) {
        const int at = count + __popc(rm & lt);
        s_i[0][warp][at] = t.x; s_i[1][warp][at] = t.y; s_i[2][warp][at] = t.z; s_i[3][warp][at] = pack_signs(t);
        s_f[0][warp][at] = t.dx; s_f[1][warp][at] = t.dy; s_f[2][warp][at] = t.dz;
        s_f[3][warp][at] = t.ax; s_f[4][warp][at] = t.ay; s_f[5][warp][at] = t.az;
        s_u[0][warp][at] = ttag; s_u[1][warp][at] = tjob;
      }
      count += __popc(rm);
    }
    __syncwarp();
    // lanes without a segment take ready ones, from the top of the pool
    const unsigned need = __ballot_sync(FULL, !active);
    const int take = min(__popc(need), count);
    if (!active) {
      const int r = __popc(need & lt);
      if (r < take) {
        const int at = count - 1 - r;
        s.x = s_i[0][warp][at]; s.y = s_i[1][warp][at]; s.z = s_i[2][warp][at];
        const int32_t sg = s_i[3][warp][at];
        s.sx = (sg & 3) - 1; s.sy = ((sg >> 2) & 3) - 1; s.sz = ((sg >> 4) & 3) - 1;
        s.dx = s_f[0][warp][at]; s.dy = s_f[1][warp][at]; s.dz = s_f[2][warp][at];
        s.ax = s_f[3][warp][at]; s.ay = s_f[4][warp][at]; s.az = s_f[5][warp][at];
        s.steps = 0; s.cb = -1; s.bits = 0ull; s.state = DDA_RUNNING;
        tag = s_u[0][warp][at];
        gh.set(P, T, s_u[1][warp][at]);
        active = true;
      }
    }
    count -= take;
    __syncwarp();
    if (!__any_sync(FULL, active)) break;   // pool empty and queue exhausted
    if (active) {
      if constexpr (!kCount && k444) dda_steps_444<false>(gh.get(T), s, kTraceSteps, 0);
      else dda_steps<kCount, false, k444>(gh.get(T), s, kTraceSteps, cnt, 0);
      if (s.state != DDA_RUNNING) {
        P.hits[(size_t)(tag & 1u) * P.n_slots + (tag >> 1)] = pack_end(s.x, s.y, s.z, s.state);
        active = false;
      }
    }
  }
  flush_counters(cnt, P.counters);
}

// ------------------------------------------------------- block wavefront
// The wavefront's round in one block: each block holds `slots` paths (their
// state in a region of its own, L2-resident; lists of slots and of segments in
// shared memory) and takes them through rounds of the same four parts, with
// block barriers where the wavefront starts a kernel, drawing new samples from
// one counter until none is left.  Blocks never wait for one another, so a
// launch is one kernel.
//
// A wavefront launch costs some 0.25 ms more than its paths (0.5 ms with eight
// bounces): four kernels a round and lane, most of them a few microseconds.
// Here a round costs its block three barriers.  Per sample the block form is
// the slower one: all four parts run at the registers of the largest (64, 1024
// threads an SM, with spills of 256 bytes a thread for one job and 480 to 588
// for a table of jobs), and a block of a thousand paths ends every DDA part
// waiting for its longest segments.  Measured (us, thread per sample / block /
// wavefront; the line to the wavefront is drawn in vt_api.cu, with more):
//   19 k samples of 64^3 spheres          118 /  170 /    -
//   262 k of 128^3 noise, 8 bounces       610 /  462 /  761
//   1.05 M of 64^3 spheres                805 /  560 /  625
//   2.1 M of a 203x117x89 noise volume   1477 /  694 /  896
//   3.1 M of 128^3 noise                    - / 2248 / 1876
// 512 slots against 1024: 545 and 568 us at 1.05 M samples, 748 and 676 at
// 2.1 M: about a third of a block's samples in flight is best.
// State fields of a path slot.
enum {
  BF_RO = 0,       // ro.xyz, -
  BF_RD = 1,       // rd.xyz, item
  BF_L = 2,        // L.xyz, rng word
  BF_T = 3,        // T.xyz, bsdf_pdf
  BF_NEE = 4,      // nee_P.xyz, light
  BF_EXT = 5,      // extension segment: vo.xyz, inc.x; next field: inc.yz, end (8 bytes)
  BF_SHADOW = 7,   // shadow segment, the same
};
enum { BC_LAMBERT = 0, BC_OTHER = 1, BC_FREE = 2, BC_QUEUE = 3, BC_HEAD = 4, BC_NUM = 5 };

// Entry of this lane in a shared list after `ctr` for the lanes with `want`:
// one shared atomic per warp.  All lanes of the warp must call it.
__device__ __forceinline__ uint32_t warp_push(uint32_t* ctr, bool want, int lane, unsigned lt) {
  const unsigned m = __ballot_sync(0xffffffffu, want);
  uint32_t base = 0;
  if (lane == 0 && m) base = atomicAdd(ctr, (uint32_t)__popc(m));
  base = __shfl_sync(0xffffffffu, base, 0);
  return base + __popc(m & lt);
}

template <bool k444, class Tab>
__global__ void __launch_bounds__(kBlockThreads, kBlocksPerSm) k_paths_block(const BlockParams P,
                                                                            const __grid_constant__ Tab T) {
  __shared__ uint32_t s_flags[kBlockSlots];
  __shared__ uint16_t s_queue[2 * kBlockSlots];
  __shared__ uint16_t s_hits[kBlockSlots];
  __shared__ uint16_t s_free[kBlockSlots];
  __shared__ uint32_t s_n[2][BC_NUM];
  const unsigned FULL = 0xffffffffu;
  const int lane = threadIdx.x & 31;
  const unsigned lt = (1u << lane) - 1u;
  const int warp_first = threadIdx.x & ~31;
  const int S = P.slots;
  float4* const st = P.state + (size_t)blockIdx.x * kBlockFields * S;
  Cnt<false> cnt;
  for (int i = threadIdx.x; i < S; i += kBlockThreads) s_flags[i] = 0u;
  if (threadIdx.x < 2 * BC_NUM) s_n[threadIdx.x / BC_NUM][threadIdx.x % BC_NUM] = 0u;
  __syncthreads();
  for (int round = 0;; ++round) {
    if (round >= P.max_rounds) {
      if (threadIdx.x == 0) *P.error = 1;
      break;
    }
    uint32_t* const ctr = s_n[round & 1];
    // ---- segment ends: finished paths out, kept hits and free slots listed
    for (int b0 = warp_first; b0 < S; b0 += kBlockThreads) {
      const int i = b0 + lane;
      const bool mine = i < S;
      const uint32_t fl = mine ? s_flags[i] : 0u;
      bool hit = false;
      int cls = 0;
      if (fl & SL_ACTIVE) {
        const JobEntry& E = job_entry(P, T, fl >> kSlotJobShift);
        Path p;
        // every load of the slot is issued before any of them is used
        const float4 a1 = st[BF_RD * S + i], a3 = st[BF_L * S + i], a4 = st[BF_T * S + i];
        float4 a5 = make_float4(0.f, 0.f, 0.f, 0.f);
        unsigned long long hs = 0ull, he = 0ull;
        if (fl & SL_SHADOW) {
          a5 = st[BF_NEE * S + i];
          hs = ((const unsigned long long*)&st[(BF_SHADOW + 1) * S + i])[1];
        }
        if (fl & SL_EXT) he = ((const unsigned long long*)&st[(BF_EXT + 1) * S + i])[1];
        p.rd = xyz4(a1);
        const uint32_t item = __float_as_uint(a1.w);
        p.L = xyz4(a3);
        p.T = xyz4(a4); p.bsdf_pdf = a4.w;
        p.nee_P = xyz4(a5); p.light = __float_as_int(a5.w);
        load_flags(fl, p);
        if (fl & SL_SHADOW) shadow_end(E.F, p, unpack_end(hs));
        if (fl & SL_EXT) {
          const SegEnd e = unpack_end(he);
          hit = ext_resolve(E.F, E.J, p, e, cnt);
          if (hit) cls = hit_class(E.F, E.J, e);
        }
        if (hit) {
          if (fl & SL_SHADOW) st[BF_L * S + i] = pack4(p.L, a3.w);
          s_flags[i] = slot_flags(p, 1u, fl >> kSlotJobShift);
        } else {
          if (chk(item < P.n_items, CHK_SAMPLE)) P.sbuf[item] = path_output(E.F, p);
          s_flags[i] = 0u;
        }
      }
      const uint32_t jl = warp_push(&ctr[BC_LAMBERT], hit && cls == 0, lane, lt);
      const uint32_t jo = warp_push(&ctr[BC_OTHER], hit && cls != 0, lane, lt);
      const uint32_t jf = warp_push(&ctr[BC_FREE], mine && !hit, lane, lt);
      if (hit) s_hits[cls == 0 ? jl : (uint32_t)S - 1u - jo] = (uint16_t)i;
      else if (mine) s_free[jf] = (uint16_t)i;
    }
    if (threadIdx.x < BC_NUM) s_n[(round & 1) ^ 1][threadIdx.x] = 0u;   // the next round's counters
    __syncthreads();
    // ---- vertices of the kept hits, Lambert first
    const uint32_t nl = ctr[BC_LAMBERT], n_hits = nl + ctr[BC_OTHER], n_free = ctr[BC_FREE];
    for (uint32_t v0 = warp_first; v0 < n_hits; v0 += kBlockThreads) {
      const uint32_t v = v0 + lane;
      const bool mine = v < n_hits;
      uint32_t emit = 0u, i = 0u;
      if (mine) {
        i = s_hits[v < nl ? v : (uint32_t)S - 1u - (v - nl)];
        const uint32_t fl = s_flags[i];
        const float4 h0 = st[BF_RO * S + i], h1 = st[BF_RD * S + i], h2 = st[BF_L * S + i], h3 = st[BF_T * S + i];
        const unsigned long long he = ((const unsigned long long*)&st[(BF_EXT + 1) * S + i])[1];
        const uint32_t job = fl >> kSlotJobShift;
        const JobEntry& E = job_entry(P, T, job);
        Path p;
        p.ro = xyz4(h0);
        p.rd = xyz4(h1);
        const uint32_t item = __float_as_uint(h1.w);
        p.L = xyz4(h2);
        p.T = xyz4(h3); p.bsdf_pdf = h3.w;
        load_flags(fl, p);
        rng_from_item(E, item, __float_as_uint(h2.w), p);
        ext_hit(E.F, E.J, p, unpack_end(he), cnt);
        emit = 2u | (p.has_cont ? 1u : 0u);
        const uint32_t rng = (E.F.rng_mode == 1) ? ((uint32_t)p.rng.ox | ((uint32_t)p.rng.oy << 16)) : p.rng.call;
        st[BF_RO * S + i] = pack4(p.ro, 0.0f);
        st[BF_RD * S + i] = pack4(p.rd, __uint_as_float(item));
        st[BF_L * S + i] = pack4(p.L, __uint_as_float(rng));
        st[BF_T * S + i] = pack4(p.T, p.bsdf_pdf);
        st[BF_NEE * S + i] = pack4(p.nee_P, __int_as_float(p.light));
        if (emit & 1u) {
          const SegRec sr = seg_rec(E.F, p.ro, p.rd);
          st[BF_EXT * S + i] = make_float4(sr.vo.x, sr.vo.y, sr.vo.z, sr.inc.x);
          *(float2*)&st[(BF_EXT + 1) * S + i] = make_float2(sr.inc.y, sr.inc.z);
        }
        const SegRec sr = seg_rec(E.F, p.ro, p.sd);
        st[BF_SHADOW * S + i] = make_float4(sr.vo.x, sr.vo.y, sr.vo.z, sr.inc.x);
        *(float2*)&st[(BF_SHADOW + 1) * S + i] = make_float2(sr.inc.y, sr.inc.z);
        s_flags[i] = slot_flags(p, emit, job);
      }
      const uint32_t q1 = warp_push(&ctr[BC_QUEUE], (emit & 1u) != 0u, lane, lt);
      if (emit & 1u) s_queue[q1] = (uint16_t)(i << 1);
      const uint32_t q2 = warp_push(&ctr[BC_QUEUE], (emit & 2u) != 0u, lane, lt);
      if (emit & 2u) s_queue[q2] = (uint16_t)((i << 1) | 1u);
    }
    // ---- new paths in the free slots
    for (uint32_t k0 = warp_first; k0 < n_free; k0 += kBlockThreads) {
      const bool left = lane == 0 && *(volatile unsigned long long*)P.next_item < P.n_items;
      if (!__any_sync(FULL, left)) break;
      const uint32_t k = k0 + lane;
      const bool mine = k < n_free;
      bool need_new = mine, active = false;
      Path p;
      uint32_t job = 0, item = 0;
      float t_enter = 0.0f;
      for (;;) {
        const unsigned want = __ballot_sync(FULL, need_new);
        if (!want) break;
        unsigned long long my = 0;
        if (lane == 0) my = atomicAdd(P.next_item, (unsigned long long)__popc(want));
        my = __shfl_sync(FULL, my, 0) + __popc(want & lt);
        if (!need_new) continue;
        if (my >= P.n_items) {
          need_new = false;   // no items left
        } else {
          item = (uint32_t)my;
          job = (uint32_t)job_of(P, T, my);
          const JobEntry& E = job_entry(P, T, job);
          const uint32_t r = (uint32_t)(my - (unsigned long long)E.tile_begin);   // < 2^32 items per launch
          const uint32_t pass = udiv(r, E.F.m_pixels);
          const uint32_t pixel = r - pass * (uint32_t)E.n_pixels;
          const uint32_t py = udiv(pixel, E.F.m_width), px = pixel - py * (uint32_t)E.F.width;
          if (path_start(E.F, E.J, p, (int)px, (int)py, E.sample_base + (int)pass, cnt, t_enter)) {
            active = true;
            need_new = false;
          } else if (chk(item < P.n_items, CHK_SAMPLE)) {
            P.sbuf[item] = path_output(E.F, p);   // missed the volume: finished, take another item
          }
        }
      }
      const uint32_t q1 = warp_push(&ctr[BC_QUEUE], active, lane, lt);
      if (active) {
        const uint32_t i = s_free[k];
        const Frame& F = job_entry(P, T, job).F;
        const uint32_t rng = (F.rng_mode == 1) ? ((uint32_t)p.rng.ox | ((uint32_t)p.rng.oy << 16)) : p.rng.call;
        const v3 o = p.ro + t_enter * p.rd;   // the primary segment starts at the volume entry point
        const SegRec sr = seg_rec(F, o, p.rd);
        st[BF_RO * S + i] = pack4(p.ro, 0.0f);
        st[BF_RD * S + i] = pack4(p.rd, __uint_as_float(item));
        st[BF_L * S + i] = pack4(p.L, __uint_as_float(rng));
        st[BF_T * S + i] = pack4(p.T, p.bsdf_pdf);
        st[BF_EXT * S + i] = make_float4(sr.vo.x, sr.vo.y, sr.vo.z, sr.inc.x);
        *(float2*)&st[(BF_EXT + 1) * S + i] = make_float2(sr.inc.y, sr.inc.z);
        s_flags[i] = slot_flags(p, 1u, job);
        s_queue[q1] = (uint16_t)(i << 1);
      }
    }
    __syncthreads();
    // ---- DDA of every listed segment
    const uint32_t n = ctr[BC_QUEUE];
    if (n == 0u) break;   // no path is left, and no item was
    {
      bool have = false, more = true;
      GridHold<Tab> gh;
      Dda s;
      uint32_t tag = 0u;
      for (;;) {
        const unsigned need = __ballot_sync(FULL, !have);
        if (need && more) {
          const uint32_t want = __popc(need);
          uint32_t c = 0;
          if (lane == 0) c = atomicAdd(&ctr[BC_HEAD], want);
          c = __shfl_sync(FULL, c, 0);
          more = c + want < n;
          const uint32_t rec = c + __popc(need & lt);
          if (!have && rec < n) {
            tag = s_queue[rec];
            const float4* at = st + (BF_EXT + 2 * (tag & 1u)) * S + (tag >> 1);
            const float4 na = at[0];
            const float2 nb = *(const float2*)&at[S];
            gh.set(P, T, s_flags[tag >> 1] >> kSlotJobShift);
            dda_begin_rec(gh.get(T), s, mk3(na.x, na.y, na.z), mk3(na.w, nb.x, nb.y));
            if (k444 && s.state == DDA_RUNNING) dda_end_stuck(gh.get(T), s);
            if (s.state == DDA_RUNNING) have = true;
            else ((unsigned long long*)&st[(BF_EXT + 1 + 2 * (tag & 1u)) * S + (tag >> 1)])[1] =
                     pack_end(s.x, s.y, s.z, s.state);
          }
        }
        if (!more && !__any_sync(FULL, have)) break;
        if (have) {
          if constexpr (k444) leap(gh.get(T), s);
          if constexpr (k444) dda_steps_444<false>(gh.get(T), s, P.trace_steps, 0);
          else dda_steps<false, false, false>(gh.get(T), s, P.trace_steps, cnt, 0);
          if (s.state != DDA_RUNNING) {
            ((unsigned long long*)&st[(BF_EXT + 1 + 2 * (tag & 1u)) * S + (tag >> 1)])[1] =
                pack_end_inside(s.x, s.y, s.z, s.state);
            have = false;
          }
        }
      }
    }
    __syncthreads();
  }
}

template <class Tab>
static void paths_block(const BlockParams& P, const Tab& T, int blocks, cudaStream_t st) {
  if (P.bricks_444) k_paths_block<true><<<blocks, kBlockThreads, 0, st>>>(P, T);
  else k_paths_block<false><<<blocks, kBlockThreads, 0, st>>>(P, T);
}
static WfOneJob one_job(const WfJobTable& T);
cudaError_t launch_paths_block(const BlockParams& P, int blocks, cudaStream_t st, const WfJobTable* T) {
  if (T && P.n_jobs == 1) paths_block(P, one_job(*T), blocks, st);
  else if (T && P.n_jobs <= kWfParamJobs) paths_block(P, *T, blocks, st);
  else paths_block(P, WfNoTable{0}, blocks, st);
  return cudaGetLastError();
}

// Launches of few samples, where only the longest path's time counts: one
// thread carries a whole sample from the camera to its output.
template <class Tab>
__global__ void __launch_bounds__(128) k_paths(const WfParams P, const __grid_constant__ Tab T, int per_warp) {
  const int lane = threadIdx.x & 31;
  const unsigned long long i =
      (unsigned long long)(blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5)) * per_warp + lane;
  if (lane >= per_warp || i >= P.n_items) return;
  const JobEntry& E = job_entry(P, T, (uint32_t)job_of(P, T, i));
  const uint32_t r = (uint32_t)(i - (unsigned long long)E.tile_begin);
  const uint32_t pass = udiv(r, E.F.m_pixels);
  const uint32_t pixel = r - pass * (uint32_t)E.n_pixels;
  const uint32_t py = udiv(pixel, E.F.m_width), px = pixel - py * (uint32_t)E.F.width;
  Cnt<false> cnt;
  P.sbuf[i] = trace_sample(E.F, E.J, (int)px, (int)py, E.sample_base + (int)pass, cnt, (HitRecord*)nullptr);
}

// Ordered reduction of the per-sample outputs into each pixel's Kahan sums:
// sample order within a pixel is the same as one sample per launch.
__global__ void k_wf_accumulate(const JobEntry* jobs, const float4* sbuf) {
  const JobEntry& E = jobs[blockIdx.y];
  const long long px = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (px >= E.n_pixels || E.passes <= 0) return;
  float4 sum = E.J.sum[px], comp = E.J.comp[px];
  for (int k = 0; k < E.passes; ++k) kahan_add(sum, comp, sbuf[E.tile_begin + (long long)k * E.n_pixels + px]);
  E.J.sum[px] = sum;
  E.J.comp[px] = comp;
}

template <class Tab>
static void wf_shade(const WfParams& P, const Tab& T, int par, int persist_blocks, bool count, cudaStream_t st) {
  const int blocks = (P.n_slots + 127) / 128;
  if (count) {
    k_wf_shade<true, Tab><<<blocks, 128, 0, st>>>(P, T, par);
    k_wf_hit<true, Tab><<<persist_blocks, 128, 0, st>>>(P, T, par);
    k_wf_regen<true, Tab><<<persist_blocks / 8 * RegenBlocks<Tab>::value, 128, 0, st>>>(P, T, par);
  } else {
    k_wf_shade<false, Tab><<<blocks, 128, 0, st>>>(P, T, par);
    k_wf_hit<false, Tab><<<persist_blocks, 128, 0, st>>>(P, T, par);
    k_wf_regen<false, Tab><<<persist_blocks / 8 * RegenBlocks<Tab>::value, 128, 0, st>>>(P, T, par);
  }
}

static WfOneJob one_job(const WfJobTable& T) {
  WfOneJob o;
  o.e = T.e[0];
  o.g = T.g[0];
  return o;
}

cudaError_t launch_wf_shade(const WfParams& P, int par, int persist_blocks, bool count, cudaStream_t st,
                            const WfJobTable* T) {
  if (T && P.n_jobs == 1) wf_shade(P, one_job(*T), par, persist_blocks, count, st);
  else if (T && P.n_jobs <= kWfParamJobs) wf_shade(P, *T, par, persist_blocks, count, st);
  else wf_shade(P, WfNoTable{0}, par, persist_blocks, count, st);
  return cudaGetLastError();
}

cudaError_t launch_paths(const WfParams& P, int sm_count, cudaStream_t st, const WfJobTable* T) {
  const int per_warp = samples_per_warp((int64_t)P.n_items, sm_count);
  const unsigned blocks = (unsigned)((P.n_items + 4 * per_warp - 1) / (4 * per_warp));   // four warps
  if (T && P.n_jobs == 1) k_paths<<<blocks, 128, 0, st>>>(P, one_job(*T), per_warp);
  else if (T && P.n_jobs <= kWfParamJobs) k_paths<<<blocks, 128, 0, st>>>(P, *T, per_warp);
  else k_paths<<<blocks, 128, 0, st>>>(P, WfNoTable{0}, per_warp);
  return cudaGetLastError();
}

template <bool kVote, bool k444, class Tab>
static void wf_trace_steps(const WfParams& P, const Tab& T, int par, int blocks, int steps, cudaStream_t st) {
  if (steps <= 8) k_wf_trace<false, 8, kVote, k444, Tab><<<blocks, 256, 0, st>>>(P, T, par);
  else if (steps <= 16) k_wf_trace<false, 16, kVote, k444, Tab><<<blocks, 256, 0, st>>>(P, T, par);
  else k_wf_trace<false, 32, kVote, k444, Tab><<<blocks, 256, 0, st>>>(P, T, par);
}

template <bool k444, class Tab>
static void wf_trace_shape(const WfParams& P, const Tab& T, int par, int blocks, int steps, bool count,
                           cudaStream_t st) {
  if (P.trace_form == 1) {   // pooled set-up
    if (count) k_wf_trace_pool<true, 8, k444, Tab><<<blocks, 256, 0, st>>>(P, T, par);
    else if (steps <= 4) k_wf_trace_pool<false, 4, k444, Tab><<<blocks, 256, 0, st>>>(P, T, par);
    else if (steps <= 8) k_wf_trace_pool<false, 8, k444, Tab><<<blocks, 256, 0, st>>>(P, T, par);
    else k_wf_trace_pool<false, 16, k444, Tab><<<blocks, 256, 0, st>>>(P, T, par);
    return;
  }
  if (count) k_wf_trace<true, 16, false, k444, Tab><<<blocks, 256, 0, st>>>(P, T, par);
  else if (P.refill_min > 0) wf_trace_steps<true, k444>(P, T, par, blocks, steps, st);
  else wf_trace_steps<false, k444>(P, T, par, blocks, steps, st);
}

template <class Tab>
static void wf_trace(const WfParams& P, const Tab& T, int par, int blocks, int steps, bool count, cudaStream_t st) {
  if (P.bricks_444) wf_trace_shape<true>(P, T, par, blocks, steps, count, st);
  else wf_trace_shape<false>(P, T, par, blocks, steps, count, st);
}

cudaError_t launch_wf_trace(const WfParams& P, int par, int blocks, int steps, bool count, cudaStream_t st,
                            const WfJobTable* T) {
  if (T && P.n_jobs == 1) wf_trace(P, one_job(*T), par, blocks, steps, count, st);
  else if (T && P.n_jobs <= kWfParamJobs) wf_trace(P, *T, par, blocks, steps, count, st);
  else wf_trace(P, WfNoTable{0}, par, blocks, steps, count, st);
  return cudaGetLastError();
}

cudaError_t launch_wf_accumulate(const JobEntry* jobs, int n_jobs, long long max_pixels, const float4* sbuf,
                                 cudaStream_t st) {
  if (n_jobs <= 0 || max_pixels <= 0) return cudaSuccess;
  dim3 grid((unsigned)((max_pixels + 255) / 256), (unsigned)n_jobs);
  k_wf_accumulate<<<grid, 256, 0, st>>>(jobs, sbuf);
  return cudaGetLastError();
}

void wf_carve(void* mem, size_t S, WfParams& P) {
  float4* f = (float4*)mem;
  for (int s = 0; s < 2; ++s) {
    WfState& x = P.x[s];
    x.a0 = f; x.a1 = f + S; x.a3 = f + 2 * S; x.a4 = f + 3 * S; x.a5 = f + 4 * S;
    f += 5 * S;
  }
  P.hr.h0 = f; P.hr.h1 = f + S; P.hr.h2 = f + 2 * S; P.hr.h3 = f + 3 * S;
  f += 4 * S;
  P.queue[0] = f;
  P.queue[1] = f + 4 * S;
  f += 8 * S;
  unsigned long long* h = (unsigned long long*)f;
  P.hits = h;
  P.hr.h4 = h + 2 * S;
  uint32_t* u = (uint32_t*)(h + 3 * S);
  P.x[0].flags = u;
  P.x[1].flags = u + S;
}

int wf_trace_blocks_per_sm() {
  int n = 0;
  cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, k_wf_trace<false, 8, false, true, WfOneJob>, 256, 0);
  return n;
}

// ------------------------------------------------------------- trace rays
// out[4*i] = voxel x, y, z, flags (hit << 8 | ground << 9 | normal code).
__global__ void k_trace_rays(const Frame F, const JobDev J, const float* origins, const float* dirs,
                             int64_t n, int32_t* out) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  Cnt<false> cnt;
  const v3 o = mk3(origins[3 * i], origins[3 * i + 1], origins[3 * i + 2]);
  const v3 d = mk3(dirs[3 * i], dirs[3 * i + 1], dirs[3 * i + 2]);
  Dda s;
  const Grid g = grid_of(F, J);
  dda_begin(g, s, o, d);
  if (s.state == DDA_RUNNING) {   // the loops that count steps
    if (bricks_444(g)) dda_steps<false, false, true>(g, s, 0x7fffffff, cnt, 0);
    else dda_steps<false, false, false>(g, s, 0x7fffffff, cnt, 0);
  }
  const bool h = dda_hit(F, s);
  int flags = (h ? 1 : 0) << 8 | ((h && s.state != DDA_HIT) ? 1 : 0) << 9 | (s.steps << 10);
  if (h) {
    const Basis b = voxel_basis(F, s.x, s.y, s.z, o, d);
    flags |= ((int)b.normal.x + 1) | (((int)b.normal.y + 1) << 2) | (((int)b.normal.z + 1) << 4);
  }
  out[4 * i] = s.x; out[4 * i + 1] = s.y; out[4 * i + 2] = s.z; out[4 * i + 3] = flags;
}

cudaError_t launch_trace_rays(const Frame& F, const JobDev& J, const float* origins, const float* dirs,
                              int64_t n, int32_t* out, cudaStream_t st) {
  if (n <= 0) return cudaSuccess;
  k_trace_rays<<<(unsigned)((n + 127) / 128), 128, 0, st>>>(F, J, origins, dirs, n, out);
  return cudaGetLastError();
}

// ------------------------------------------------------------------- pick
// focalDistance.vs:45-81: generateRay with rngOffset (0,0) and no pixel
// jitter consumption difference (the pinhole draws its jitter from the
// sequence start), AABB clip, traverse, exact voxel distance.
__global__ void k_pick(const Frame F, const JobDev J, float x, float y, float* out_dist, int32_t* out_voxel) {
  if (threadIdx.x != 0 || blockIdx.x != 0) return;
  Cnt<false> cnt;
  Rng rng;
  rng.pixel = 0; rng.sample = 0; rng.call = 0; rng.ox = 0; rng.oy = 0;
  v3 o, d;
  generate_ray(F, J, mk3(x, y, 0.0f), rng, o, d);
  *out_dist = kInfinity;
  out_voxel[0] = out_voxel[1] = out_voxel[2] = -1;
  const float t = ray_aabb(o, d, ld3(F.bmin), ld3(F.bmax));
  if (t < 0.0f) return;
  Dda s;
  const Grid g = grid_of(F, J);
  dda_begin(g, s, o + t * d, d);
  dda_finish(g, s, cnt);
  if (!dda_hit(F, s)) return;
  const v3 vs = ld3(F.vsize);
  const v3 vmin = mk3((float)s.x, (float)s.y, (float)s.z) * vs + ld3(F.bmin);
  *out_dist = ray_aabb(o, d, vmin, vmin + vs);
  out_voxel[0] = s.x; out_voxel[1] = s.y; out_voxel[2] = s.z;
}

// selectVoxel.vs:35-69: generateRay at window depth frag_z (the shader
// passes cameraNear), AABB clip, traverse, and the basis normal of the hit
// (voxelSpaceToWorldSpace).  Nothing hit: out[3] = 0.
__global__ void k_select(const Frame F, const JobDev J, float x, float y, float frag_z, int32_t* out) {
  if (threadIdx.x != 0 || blockIdx.x != 0) return;
  Cnt<false> cnt;
  Rng rng;
  rng.pixel = 0; rng.sample = 0; rng.call = 0; rng.ox = 0; rng.oy = 0;
  v3 o, d;
  generate_ray(F, J, mk3(x, y, frag_z), rng, o, d);
  out[0] = out[1] = out[2] = -1;
  out[3] = 0;
  float* nrm = (float*)(out + 4);
  nrm[0] = nrm[1] = nrm[2] = 0.0f;
  const float t = ray_aabb(o, d, ld3(F.bmin), ld3(F.bmax));
  if (t < 0.0f) return;
  Dda s;
  const Grid g = grid_of(F, J);
  dda_begin(g, s, o + t * d, d);
  dda_finish(g, s, cnt);
  if (!dda_hit(F, s)) return;
  const Basis b = voxel_basis(F, s.x, s.y, s.z, o, d);
  out[0] = s.x; out[1] = s.y; out[2] = s.z; out[3] = 1;
  nrm[0] = b.normal.x; nrm[1] = b.normal.y; nrm[2] = b.normal.z;
}

cudaError_t launch_select(const Frame& F, const JobDev& J, float x, float y, float frag_z, int32_t* out,
                          cudaStream_t st) {
  k_select<<<1, 32, 0, st>>>(F, J, x, y, frag_z, out);
  return cudaGetLastError();
}

cudaError_t launch_pick(const Frame& F, const JobDev& J, float x, float y, float* out_dist,
                        int32_t* out_voxel, cudaStream_t st) {
  k_pick<<<1, 32, 0, st>>>(F, J, x, y, out_dist, out_voxel);
  return cudaGetLastError();
}

// ---------------------------------------------------------------- resolve
__global__ void k_resolve(const float4* sum, int32_t w, int32_t h, int32_t samples, float exposure,
                          float inv_gamma, uint32_t flags, float4* out) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= (int64_t)w * h) return;
  const int x = (int)(i % w), y = (int)(i / w);
  float4 v = sum[i];
  const float n = samples > 0 ? (float)samples : 1.0f;
  v.x = v.x / n; v.y = v.y / n; v.z = v.z / n; v.w = v.w / n;
  if (flags & 2u) {
    v.x = vtb::vpow(v.x * exposure, inv_gamma);
    v.y = vtb::vpow(v.y * exposure, inv_gamma);
    v.z = vtb::vpow(v.z * exposure, inv_gamma);
  }
  const int oy = (flags & 1u) ? (h - 1 - y) : y;
  out[(int64_t)oy * w + x] = v;
}

cudaError_t launch_resolve(const float4* sum, int32_t w, int32_t h, int32_t samples, float exposure,
                           float inv_gamma, uint32_t flags, float4* out, cudaStream_t st) {
  const int64_t n = (int64_t)w * h;
  if (n <= 0) return cudaSuccess;
  k_resolve<<<(unsigned)((n + 255) / 256), 256, 0, st>>>(sum, w, h, samples, exposure, inv_gamma, flags, out);
  return cudaGetLastError();
}

// --------------------------------------------------------------- builtins
__global__ void k_builtins(int32_t fn, const float* a, const float* b, float* out, int64_t n) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const float x = a[i];
  float r;
  switch (fn) {
    case 0: r = vtb::vsin(x); break;
    case 1: r = vtb::vcos(x); break;
    case 2: r = vtb::vpow(x, b[i]); break;
    case 3: r = vtb::vacos(x); break;
    case 4: r = vtb::vatan2(x, b[i]); break;
    case 5: r = vtb::vlog2(x); break;
    case 6: r = vtb::vexp2(x); break;
    case 7: r = vtb::h2f(vtb::f2h(x)); break;
    default: r = 0.0f; break;
  }
  out[i] = r;
}

cudaError_t launch_builtins(int32_t fn, const float* a, const float* b, float* out, int64_t n,
                            cudaStream_t st) {
  if (n <= 0) return cudaSuccess;
  k_builtins<<<(unsigned)((n + 255) / 256), 256, 0, st>>>(fn, a, b, out, n);
  return cudaGetLastError();
}

// ------------------------------------------------------ L2 read bandwidth
// `reps` sweeps of an L2-resident buffer in one launch, loads bypassing L1
// (ld.global.cg), four independent 16-byte loads in flight per thread; the
// XOR of everything read is stored per thread so that no load is dropped.
// Each sweep starts one grid-width further on, so a thread does not read
// the same lines in consecutive sweeps.
__global__ void __launch_bounds__(512) k_l2_read(const uint4* __restrict__ buf, uint32_t n, int32_t reps,
                                                 uint4* __restrict__ out) {
  const uint32_t T = gridDim.x * blockDim.x;
  const uint32_t t = blockIdx.x * blockDim.x + threadIdx.x;
  uint4 acc = make_uint4(0u, 0u, 0u, 0u);
  for (int32_t r = 0; r < reps; ++r) {
    const uint32_t base = (uint32_t)(((uint64_t)r * T + t) % n);
    uint32_t i = 0;
    for (; i + 3 * T < n; i += 4 * T) {
      uint4 v[4];
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        uint32_t j = base + i + (uint32_t)k * T;
        if (j >= n) j -= n;
        v[k] = __ldcg(&buf[j]);
      }
#pragma unroll
      for (int k = 0; k < 4; ++k) { acc.x ^= v[k].x; acc.y ^= v[k].y; acc.z ^= v[k].z; acc.w ^= v[k].w; }
    }
    for (; i < n; i += T) {
      uint32_t j = base + i;
      if (j >= n) j -= n;
      const uint4 v = __ldcg(&buf[j]);
      acc.x ^= v.x; acc.y ^= v.y; acc.z ^= v.z; acc.w ^= v.w;
    }
  }
  out[t] = acc;
}

cudaError_t launch_l2_read(const uint4* buf, uint32_t n, int32_t reps, uint4* out, int blocks, cudaStream_t st) {
  if (n == 0 || reps <= 0 || blocks <= 0) return cudaSuccess;
  k_l2_read<<<blocks, 512, 0, st>>>(buf, n, reps, out);
  return cudaGetLastError();
}

}  // namespace vt

namespace vt {
// The check word of the bounds-checked build (0 and enabled = false in a
// release build); reset clears it after reading.
cudaError_t read_check_word(uint32_t* word, bool* enabled, bool reset) {
#ifdef VT_CHECKED
  *enabled = true;
  cudaError_t e = cudaMemcpyFromSymbol(word, g_check_word, sizeof(uint32_t));
  if (e == cudaSuccess && reset) {
    const uint32_t zero = 0;
    e = cudaMemcpyToSymbol(g_check_word, &zero, sizeof(uint32_t));
  }
  return e;
#else
  *enabled = false;
  *word = 0;
  (void)reset;
  return cudaSuccess;
#endif
}
}  // namespace vt
