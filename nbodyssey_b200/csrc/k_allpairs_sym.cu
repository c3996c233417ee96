// All-pairs softened gravity (src/forces.cu:17-60) with each unordered pair
// evaluated once, for n from kSymMin on.
//
// The tiled kernel (k_allpairs.cu) spends 12 packed FP32 operations and two
// MUFU rsqrt per two interactions and runs its FMA pipe at about 81 %; only
// fewer operations make it faster.  Here a pair (i, j) is evaluated once and
// added to both particles: 17 packed operations per four interactions instead
// of 24, and half the rsqrt.
//
// Work item (I, c): the targets of tile I against the sources of chunk c (not
// before the tile).  A CTA of four warps takes the tile in sub-tiles of 256:
// every warp holds the same 256 targets in registers (8 a lane), and a quarter
// of the chunk each.  64 sources at a time sit two per lane, packed, with
// their own sums and move around the warp's ring by shuffles, so after 32
// steps every source has met all 256 targets and is back in its lane with its
// whole sum: no atomics and no reduction across lanes.  14 shuffles a step
// against 136 packed operations keep the FMA pipe the limit.  (Targets packed
// in pairs and one source per lane need fewer shuffles but a register copy of
// every source coordinate: 21.7 ms against 20.2 at n = 262,144.)  Where all
// masses of a round are the same, the source's factor equals the target's, so
// one is computed: 15 operations, the same bits.  The targets' sums are added
// over the four warps at the end of a sub-tile.  Chunks inside the tile itself
// are taken in both orders (targets' sums only).
//
// Two CTAs per SM: three (168 registers instead of 208) leave the compiler too
// few registers to overlap the eight targets' chains (21.2 ms against 20.2).
//
// The sums go to a table of partials: row I holds tile I's contribution to
// every later target, row c (a second table) chunk c's contribution to the
// targets of the tiles before it.  k_ap_sym_reduce adds a target's partials in
// a fixed order -- tiles before its own, then the chunks from its own tile on
// -- and applies the closing kick, so results repeat bit for bit.  A table that
// would be larger than the scratch at hand is used for a few rows of tiles at
// a time, or for a few chunks of one row, the running sums kept in `acc`; the
// order, and so every bit, is the same.
#include <algorithm>
#include <vector>

#include "f32x2.cuh"
#include "nb_internal.cuh"

namespace nb {

constexpr int kSymSub = 256;           // targets in registers
constexpr int kSymK = kSymSub / 32;    // targets per lane
constexpr int kSymRound = 64;          // sources around the ring, two per lane
constexpr int kSymWarps = 4;
constexpr int kSymThreads = 32 * kSymWarps;

// Tile and chunk by n: a function of n alone, so that the order of the sums
// is too.  The smallest items fill 148 SMs x 2 CTAs evenly (n = 12,000: 1,128
// items of 256 x 256 take 57.5 us a step, 576 of 512 x 256 58.7, 300 of 512 x
// 512 75); from there the tile grows with n, the chunk half a tile, so that
// the table stays below 1 GiB (at n = 262,144, chunks of a whole tile would take
// 0.5 instead of 0.8 GB and 18.4 ms instead of 17.8; 4,096-tiles at 140,000 lose 8 %
// to the last wave of items).
SymGeom allpairs_sym_geometry(int n) {
  SymGeom g;
  g.tile = n <= 16384 ? 256 : n <= 24576 ? 512 : n <= 65536 ? 1024 : n <= 163840 ? 2048 : 4096;
  g.chunk = std::max(256, g.tile / 2);   // at most kSymChunkMax
  g.tiles = (n + g.tile - 1) / g.tile;
  g.chunks = (n + g.chunk - 1) / g.chunk;
  return g;
}

bool allpairs_sym(int n) { return n >= kSymMin && n <= kSymMax; }

// Table float4 of one row of tiles: its row over all targets, and the chunks'
// rows over its own targets.
size_t allpairs_sym_row_f4(int n) {
  const SymGeom g = allpairs_sym_geometry(n);
  return (size_t)n + (size_t)g.chunks * g.tile;
}

size_t allpairs_sym_least_f4(int n) {
  const SymGeom g = allpairs_sym_geometry(n);
  return (size_t)g.chunk + g.tile;
}

// A lane's targets (negated positions and masses, each in both halves of a
// packed register) and their sums over even and odd sources.
struct SymTargets {
  f2 x[kSymK], y[kSymK], z[kSymK], m[kSymK];
  f2 ax[kSymK], ay[kSymK], az[kSymK];
};
// Two sources and their sums.
struct SymSources {
  f2 x, y, z, m;
  f2 bx, by, bz;
};

enum { kSymOwn, kSymEqual, kSymAny };

__device__ __forceinline__ f2 ring(f2 v) {
  return __shfl_sync(0xffffffffu, v, (int)threadIdx.x + 1);   // lane + 1, modulo the warp
}

// 32 steps: the sources go once around the ring.  kSymOwn adds to the targets
// only; kSymEqual needs one mass for all targets and sources.
template <int MODE>
__device__ __forceinline__ void sym_round(SymTargets& t, SymSources& s, f2 e2) {
#pragma unroll 1
  for (int step = 0; step < 32; ++step) {
#pragma unroll
    for (int k = 0; k < kSymK; ++k) {
      const f2 dx = add2(s.x, t.x[k]), dy = add2(s.y, t.y[k]), dz = add2(s.z, t.z[k]);
      const f2 r2 = fma2(dx, dx, fma2(dy, dy, fma2(dz, dz, e2)));
      float q0, q1;
      up2(r2, q0, q1);
      const f2 inv = pk2(mufu_rsqrt(q0), mufu_rsqrt(q1));
      const f2 i2 = mul2(inv, inv);
      const f2 f = mul2(mul2(inv, s.m), i2);
      t.ax[k] = fma2(dx, f, t.ax[k]);
      t.ay[k] = fma2(dy, f, t.ay[k]);
      t.az[k] = fma2(dz, f, t.az[k]);
      if (MODE != kSymOwn) {
        const f2 g = MODE == kSymEqual ? f : mul2(mul2(inv, t.m[k]), i2);
        s.bx = fma2(dx, g, s.bx);
        s.by = fma2(dy, g, s.by);
        s.bz = fma2(dz, g, s.bz);
      }
    }
    s.x = ring(s.x);
    s.y = ring(s.y);
    s.z = ring(s.z);
    if (MODE != kSymEqual) s.m = ring(s.m);
    if (MODE != kSymOwn) {
      s.bx = ring(s.bx);
      s.by = ring(s.by);
      s.bz = ring(s.bz);
    }
  }
}

// Work item (I, c); every thread of the CTA calls it.
__device__ __forceinline__ void sym_item(const SymArgs& a, int I, int c) {
  extern __shared__ float s_sym[];
  float* s_red = s_sym;                                  // [warps][3][kSymSub]
  float* s_j = s_sym + kSymWarps * 3 * kSymSub;          // [3][chunk]
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const bool own = c < (I + 1) * (a.tile / a.chunk);   // the chunk lies in the tile
  const int quarter = a.chunk / kSymWarps;
  const int jw = c * a.chunk + w * quarter;   // this warp's sources
  const f2 e2 = pk2(a.eps2, a.eps2);

  for (int sub = 0; sub < a.tile; sub += kSymSub) {
    const int i0 = I * a.tile + sub;
    if (i0 >= a.n) break;   // the same for the whole CTA
    SymTargets t;
    const float mass = a.pos[i0].w;
    bool equal = true;
#pragma unroll
    for (int k = 0; k < kSymK; ++k) {
      const int i = i0 + 32 * k + lane;
      const float4 p = a.pos[min(i, a.n - 1)];
      const float m = i < a.n ? p.w : 0.f;
      t.x[k] = pk2(-p.x, -p.x);
      t.y[k] = pk2(-p.y, -p.y);
      t.z[k] = pk2(-p.z, -p.z);
      t.m[k] = pk2(m, m);
      t.ax[k] = t.ay[k] = t.az[k] = 0ull;
      equal = equal && m == mass;
    }
    const bool last_sub = i0 + kSymSub >= min(a.n, (I + 1) * a.tile);
    for (int r = 0; r < quarter; r += kSymRound) {
      const int j = jw + r + lane;
      if (jw + r >= a.n) break;   // the same for the whole warp
      float4 p = a.pos[min(j, a.n - 1)], q = a.pos[min(j + 32, a.n - 1)];
      if (j >= a.n) p.w = 0.f;
      if (j + 32 >= a.n) q.w = 0.f;
      SymSources s;
      s.x = pk2(p.x, q.x);
      s.y = pk2(p.y, q.y);
      s.z = pk2(p.z, q.z);
      s.m = pk2(p.w, q.w);
      s.bx = s.by = s.bz = 0ull;
      if (own) {
        sym_round<kSymOwn>(t, s, e2);
        continue;
      }
      if (__all_sync(0xffffffffu, equal && p.w == mass && q.w == mass))
        sym_round<kSymEqual>(t, s, e2);
      else
        sym_round<kSymAny>(t, s, e2);
      // back in their lane; d points from the target to the source, which is
      // pulled by -d
      float bx[2], by[2], bz[2];
      up2(s.bx, bx[0], bx[1]);
      up2(s.by, by[0], by[1]);
      up2(s.bz, bz[0], bz[1]);
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        float* o = &s_j[w * quarter + r + 32 * h + lane];   // this lane's alone
        float3 b = make_float3(-bx[h], -by[h], -bz[h]);
        if (sub > 0) {
          b.x += o[0];
          b.y += o[a.chunk];
          b.z += o[2 * a.chunk];
        }
        if (!last_sub) {
          o[0] = b.x;
          o[a.chunk] = b.y;
          o[2 * a.chunk] = b.z;
        } else if (j + 32 * h < a.n) {
          a.row[(size_t)(I - a.ta) * a.n + j + 32 * h] = make_float4(b.x, b.y, b.z, 0.f);
        }
      }
    }
    __syncthreads();   // the previous sub-tile's sums have been read
#pragma unroll
    for (int k = 0; k < kSymK; ++k) {
      float* o = &s_red[w * 3 * kSymSub + 32 * k + lane];
      float u, v;
      up2(t.ax[k], u, v); o[0] = u + v;
      up2(t.ay[k], u, v); o[kSymSub] = u + v;
      up2(t.az[k], u, v); o[2 * kSymSub] = u + v;
    }
    __syncthreads();
    float4* col = a.col + (size_t)c * ((a.tb - a.ta) * a.tile) + (I - a.ta) * a.tile + sub;
    for (int k = threadIdx.x; k < kSymSub && i0 + k < a.n; k += kSymThreads) {
      float3 f = make_float3(0.f, 0.f, 0.f);
#pragma unroll
      for (int v = 0; v < kSymWarps; ++v) {
        const float* o = &s_red[v * 3 * kSymSub + k];
        f.x += o[0];
        f.y += o[kSymSub];
        f.z += o[2 * kSymSub];
      }
      col[k] = make_float4(f.x, f.y, f.z, 0.f);
    }
  }
}

// One simulation: rows of tiles are folded in pairs (first with last), whose
// chunk counts add up to the same number, so the grid is a rectangle.
__global__ void __launch_bounds__(kSymThreads, 2) k_ap_sym(SymArgs a) {
  const int per = a.tile / a.chunk;
  int I = a.ta + blockIdx.y, x = blockIdx.x + max(0, a.ca - I * per);
  const int last = a.tb - 1 - blockIdx.y;
  if (x >= a.cb - I * per) {
    x -= a.cb - I * per;
    if (last <= I) return;   // the middle row of an odd count
    I = last;
    if (x >= a.cb - I * per) return;
  }
  sym_item(a, I, I * per + x);
}

// Many simulations' items, (simulation entry, I, c), one per CTA.
__global__ void __launch_bounds__(kSymThreads, 2) k_ap_sym_batch(
    const SymArgs* __restrict__ args, int nargs, const int4* __restrict__ items,
    unsigned* err) {
  const int4 it = items[blockIdx.x];
  bool ok = it.x >= 0 && it.x < nargs;
  SymArgs a{};
  if (ok) {
    a = args[it.x];
    ok = it.y >= a.ta && it.y < a.tb && it.z >= max(it.y * (a.tile / a.chunk), a.ca) &&
         it.z < a.cb;
  }
  if (!ok) {   // a stale or corrupt item: skipped, reported
    if (threadIdx.x == 0) raise_err(err, NB_DEVERR_QUEUE);
    return;
  }
  sym_item(a, it.y, it.z);
}

// Adds target t's partials of tiles [ta, tb) and chunks [ca, cb); the pass that
// holds its own tile's last chunk ends its sum.
__device__ __forceinline__ void sym_reduce(const SymArgs& a, int block, bool kick) {
  const int t = a.ta * a.tile + block * kSymThreads + threadIdx.x;
  if (t >= a.n) return;
  const int T = t / a.tile;
  float3 s = make_float3(0.f, 0.f, 0.f);
  if (a.ta > 0 || a.ca > 0) {
    const float4 r = a.acc[t];
    s = make_float3(r.x, r.y, r.z);
  }
  // cnt partials `stride` apart, kAhead loads in flight, added in order
  auto add = [&](const float4* p, size_t stride, int cnt) {
    constexpr int kAhead = 16;
    for (int r = 0; r < cnt; r += kAhead) {
      float4 v[kAhead];
#pragma unroll
      for (int q = 0; q < kAhead; ++q)
        v[q] = r + q < cnt ? __ldcs(p + (r + q) * stride) : make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
      for (int q = 0; q < kAhead; ++q) {
        if (r + q < cnt) {
          s.x += v[q].x; s.y += v[q].y; s.z += v[q].z;
        }
      }
    }
  };
  // the pass holds this target's rows when it holds its chunk
  const bool rows = t >= a.ca * a.chunk && t < a.cb * a.chunk;
  add(a.row + t, a.n, rows ? min(T, a.tb) - a.ta : 0);
  if (T >= a.tb) {
    a.acc[t] = make_float4(s.x, s.y, s.z, 0.f);
    return;
  }
  const size_t width = (size_t)(a.tb - a.ta) * a.tile;
  const int c0 = max(T * (a.tile / a.chunk), a.ca);
  add(a.col + c0 * width + (t - a.ta * a.tile), width, a.cb - c0);
  if (a.cb < a.chunks) {
    a.acc[t] = make_float4(s.x, s.y, s.z, 0.f);
    return;
  }
  const float4 acc = make_float4(a.G * s.x, a.G * s.y, a.G * s.z, 0.f);
  a.acc[t] = acc;
  if (kick && a.vel) {
    float4 v = a.vel[t];
    v.x = __fmaf_rn(a.half_dt, acc.x, v.x);
    v.y = __fmaf_rn(a.half_dt, acc.y, v.y);
    v.z = __fmaf_rn(a.half_dt, acc.z, v.z);
    a.vel[t] = v;
  }
}

__global__ void __launch_bounds__(kSymThreads) k_ap_sym_reduce(SymArgs a) {
  sym_reduce(a, blockIdx.x, true);
}

__global__ void __launch_bounds__(kSymThreads) k_ap_sym_reduce_batch(
    const SymArgs* __restrict__ args, int nargs, const int2* __restrict__ blocks, int kick,
    unsigned* err) {
  const int2 it = blocks[blockIdx.x];
  if (it.x < 0 || it.x >= nargs || it.y < 0) {
    if (threadIdx.x == 0) raise_err(err, NB_DEVERR_QUEUE);
    return;
  }
  const SymArgs a = args[it.x];
  sym_reduce(a, it.y, kick != 0);
}

// Dynamic shared memory of an item: below the 48 KB that every launch may ask
// for, so no launch raises the kernels' limit -- it belongs to the function, and
// a smaller call of another thread would lower it between a raise and its launch.
constexpr int kSymChunkMax = 2048;
static constexpr int sym_smem(int chunk) {
  return (kSymWarps * 3 * kSymSub + 3 * chunk) * (int)sizeof(float);
}
static_assert(sym_smem(kSymChunkMax) <= 48 * 1024, "no opt-in shared memory");

// Fields that depend on n alone.
static SymArgs sym_args(int n) {
  const SymGeom g = allpairs_sym_geometry(n);
  SymArgs a{};
  a.n = n;
  a.tile = g.tile;
  a.chunk = g.chunk;
  a.tiles = g.tiles;
  a.chunks = g.chunks;
  return a;
}

// Calls fn for each pass over a table of scratch_f4 float4: as many rows of
// tiles as it holds, all their chunks, or, when it does not hold one row, as
// many chunks of one.
template <typename F>
static int sym_passes(SymArgs a, size_t scratch_f4, F fn) {
  const size_t rows = scratch_f4 / allpairs_sym_row_f4(a.n);
  if (rows > 0) {
    a.ca = 0;
    a.cb = a.chunks;
    for (a.ta = 0; a.ta < a.tiles; a.ta = a.tb) {
      a.tb = (int)std::min<size_t>(a.tiles, a.ta + rows);
      NB_TRY(fn(a));
    }
    return NB_OK;
  }
  const int span = (int)(scratch_f4 / allpairs_sym_least_f4(a.n));
  if (span < 1) return set_error(NB_ERR_NOMEM, "all-pairs scratch too small");
  for (a.ta = 0; a.ta < a.tiles; ++a.ta) {
    a.tb = a.ta + 1;
    for (a.ca = a.ta * (a.tile / a.chunk); a.ca < a.chunks; a.ca = a.cb) {
      a.cb = std::min(a.chunks, a.ca + span);
      NB_TRY(fn(a));
    }
  }
  return NB_OK;
}

// The pass's table in `scratch`: row [tb - ta][n], col [chunks][(tb - ta) tile].
// A pass over some chunks of one row holds their part of both; the kernels index
// from where chunk 0 would lie.
static void sym_place(SymArgs& a, float4* scratch) {
  const size_t cnt = a.tb - a.ta;
  const bool all = a.ca == 0 && a.cb == a.chunks;
  const size_t row_f4 = all ? cnt * a.n : (size_t)(a.cb - a.ca) * a.chunk;
  a.row = scratch - (size_t)a.ca * a.chunk;
  a.col = scratch + row_f4 - (size_t)a.ca * cnt * a.tile;
}

int launch_allpairs_sym(int n, const float4* pos, float4* acc, float4* vel, float eps2,
                        float G, float half_dt, float4* scratch, size_t scratch_f4,
                        cudaStream_t st) {
  SymArgs base = sym_args(n);
  base.pos = pos;
  base.acc = acc;
  base.vel = vel;
  base.eps2 = eps2;
  base.G = G;
  base.half_dt = half_dt;
  const int smem = sym_smem(base.chunk);
  const int per = base.tile / base.chunk;
  return sym_passes(base, scratch_f4, [&](SymArgs a) {
    sym_place(a, scratch);
    const int cnt = a.tb - a.ta;
    // chunks of the first and the last row of a folded pair together
    int wide = a.cb - std::max(a.ca, a.ta * per);
    if (cnt > 1) wide += a.chunks - (a.tb - 1) * per;
    k_ap_sym<<<dim3(wide, (cnt + 1) / 2), kSymThreads, smem, st>>>(a);
    NB_CUDA(cudaGetLastError());
    const int left = n - a.ta * a.tile;
    k_ap_sym_reduce<<<(left + kSymThreads - 1) / kSymThreads, kSymThreads, 0, st>>>(a);
    NB_CUDA(cudaGetLastError());
    return NB_OK;
  });
}

// A simulation of a batch takes its passes over the `region_f4` float4 that it
// has at `region` of the pool; the batch's launches of pass k hold pass k of
// every simulation.
void SymPlan::clear() {
  args.clear();
  sim.clear();
  region.clear();
  pass.clear();
  items.clear();
  blocks.clear();
  passes.clear();
}

void SymPlan::add(int s, const SimDesc& d, size_t at, size_t region_f4) {
  SymArgs base = sym_args(d.n);
  base.eps2 = d.eps2;
  base.G = d.G;
  base.half_dt = d.half_dt;
  int k = 0;
  sym_passes(base, region_f4, [&](const SymArgs& a) {   // the caller has checked the least
    args.push_back(a);
    sim.push_back(s);
    region.push_back(at);
    pass.push_back(k++);
    return NB_OK;
  });
}

// Items and reduction blocks, pass by pass; larger chunks first.
void SymPlan::finish() {
  const int last = pass.empty() ? -1 : *std::max_element(pass.begin(), pass.end());
  std::vector<int> order;
  for (int i = 0; i < (int)args.size(); ++i) order.push_back(i);
  std::stable_sort(order.begin(), order.end(),
                   [&](int x, int y) { return args[x].tile > args[y].tile; });
  for (int k = 0; k <= last; ++k) {
    Pass p{(int)items.size(), 0, (int)blocks.size(), 0, 0};
    for (int i : order) {
      if (pass[i] != k) continue;
      const SymArgs& a = args[i];
      const int per = a.tile / a.chunk;
      for (int I = a.ta; I < a.tb; ++I)
        for (int c = std::max(I * per, a.ca); c < a.cb; ++c)
          items.push_back(make_int4(i, I, c, 0));
      const int left = a.n - a.ta * a.tile;
      for (int b = 0; b < (left + kSymThreads - 1) / kSymThreads; ++b)
        blocks.push_back(make_int2(i, b));
      p.chunk = std::max(p.chunk, a.chunk);
    }
    p.items = (int)items.size() - p.first_item;
    p.blocks = (int)blocks.size() - p.first_block;
    passes.push_back(p);
  }
}

size_t SymPlan::bytes() const {
  return args.size() * sizeof(SymArgs) + items.size() * sizeof(int4) +
         blocks.size() * sizeof(int2);
}

int SymPlan::bind(const SimDesc* sims, const EnsArgs& e, float4* pool, cudaStream_t st) {
  for (size_t i = 0; i < args.size(); ++i) {
    const SimDesc& d = sims[sim[i]];
    SymArgs& a = args[i];
    a.pos = e.pos + d.base;
    a.acc = e.acc + d.base;
    a.vel = d.active == 1 ? e.vel + d.base : nullptr;
    sym_place(a, pool + region[i]);
  }
  if (args.empty()) return NB_OK;
  // items first: 16-byte entries at the start of the allocation
  unsigned char* p = d_table;
  NB_CUDA(cudaMemcpyAsync(p, items.data(), items.size() * sizeof(int4),
                          cudaMemcpyHostToDevice, st));
  p += items.size() * sizeof(int4);
  NB_CUDA(cudaMemcpyAsync(p, args.data(), args.size() * sizeof(SymArgs),
                          cudaMemcpyHostToDevice, st));
  p += args.size() * sizeof(SymArgs);
  NB_CUDA(cudaMemcpyAsync(p, blocks.data(), blocks.size() * sizeof(int2),
                          cudaMemcpyHostToDevice, st));
  return NB_OK;
}

int SymPlan::launch(const EnsArgs& e, cudaStream_t st) const {
  if (args.empty()) return NB_OK;
  const int4* d_items = reinterpret_cast<const int4*>(d_table);
  const SymArgs* d_args = reinterpret_cast<const SymArgs*>(d_items + items.size());
  const int2* d_blocks = reinterpret_cast<const int2*>(d_args + args.size());
  const int nargs = (int)args.size();
  for (const Pass& p : passes) {
    k_ap_sym_batch<<<p.items, kSymThreads, sym_smem(p.chunk), st>>>(
        d_args, nargs, d_items + p.first_item, e.err);
    NB_CUDA(cudaGetLastError());
    k_ap_sym_reduce_batch<<<p.blocks, kSymThreads, 0, st>>>(
        d_args, nargs, d_blocks + p.first_block, e.kick_after ? 1 : 0, e.err);
    NB_CUDA(cudaGetLastError());
  }
  return NB_OK;
}

int warm_allpairs_sym_kernels() {
  return warm_fns(k_ap_sym, k_ap_sym_reduce, k_ap_sym_batch, k_ap_sym_reduce_batch);
}

}  // namespace nb
