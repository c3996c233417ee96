// All-pairs softened gravity (src/forces.cu:17-60) for n below kSymMin: a warp
// per few targets, its lanes over the sources.
//
// Bound: latency.  A thousand particles are a million pairs, a microsecond of
// the device's FP32 rate, so what counts is that one launch reads the particles
// as they are (no packing pass, no split of the sources to sum up afterwards)
// and that every SM has work.  A warp holds K targets, packed in pairs and the
// same in every lane; lane l takes sources l, l + 32, ..., two batches of loads
// in flight, and the lanes' sums are added by shuffles at the end (kick
// included).  A target's sum depends on n alone, not on K or on the other
// targets, so a simulation gets the same bits alone and in a batch.
#include "f32x2.cuh"
#include "nb_internal.cuh"

namespace nb {

constexpr int kSmallWarps = 4;
constexpr int kSmallBatch = 4;   // sources a lane loads together

// Targets [t0, t0 + K) of one simulation; all 32 lanes of a warp call it.
template <int K>
__device__ __forceinline__ void small_targets(const APArgs& a, int t0, bool kick) {
  static_assert(K % 2 == 0, "targets are packed in pairs");
  constexpr int P = K / 2;
  const int lane = threadIdx.x & 31;
  if (t0 >= a.n) return;   // the whole warp
  f2 nx[P], ny[P], nz[P], ax[P], ay[P], az[P];
#pragma unroll
  for (int p = 0; p < P; ++p) {
    const float4 u = a.pos[min(t0 + 2 * p, a.n - 1)], v = a.pos[min(t0 + 2 * p + 1, a.n - 1)];
    nx[p] = pk2(-u.x, -v.x);
    ny[p] = pk2(-u.y, -v.y);
    nz[p] = pk2(-u.z, -v.z);
    ax[p] = ay[p] = az[p] = 0ull;
  }
  const f2 e2 = pk2(a.eps2, a.eps2);
  // a source past the end: the last particle without mass
  auto load = [&](float4* s, int j0) {
#pragma unroll
    for (int q = 0; q < kSmallBatch; ++q) {
      const int j = j0 + 32 * q + lane;
      s[q] = a.pos[min(j, a.n - 1)];
      if (j >= a.n) s[q].w = 0.f;
    }
  };
  float4 cur[kSmallBatch], next[kSmallBatch];
  load(cur, 0);
  for (int j0 = 0; j0 < a.n; j0 += 32 * kSmallBatch) {
    load(next, j0 + 32 * kSmallBatch);
#pragma unroll
    for (int q = 0; q < kSmallBatch; ++q) {
      const f2 x = pk2(cur[q].x, cur[q].x), y = pk2(cur[q].y, cur[q].y),
               z = pk2(cur[q].z, cur[q].z), m = pk2(cur[q].w, cur[q].w);
#pragma unroll
      for (int p = 0; p < P; ++p) {
        const f2 dx = add2(x, nx[p]), dy = add2(y, ny[p]), dz = add2(z, nz[p]);
        const f2 r2 = fma2(dx, dx, fma2(dy, dy, fma2(dz, dz, e2)));
        float r0, r1;
        up2(r2, r0, r1);
        const f2 inv = pk2(mufu_rsqrt(r0), mufu_rsqrt(r1));
        const f2 f = mul2(mul2(inv, m), mul2(inv, inv));
        ax[p] = fma2(dx, f, ax[p]);
        ay[p] = fma2(dy, f, ay[p]);
        az[p] = fma2(dz, f, az[p]);
      }
    }
#pragma unroll
    for (int q = 0; q < kSmallBatch; ++q) cur[q] = next[q];
  }
  // sums over the lanes: the same in every lane; lane k keeps target t0 + k's
  float3 mine = make_float3(0.f, 0.f, 0.f);
#pragma unroll
  for (int p = 0; p < P; ++p) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      ax[p] = add2(ax[p], __shfl_xor_sync(0xffffffffu, ax[p], o));
      ay[p] = add2(ay[p], __shfl_xor_sync(0xffffffffu, ay[p], o));
      az[p] = add2(az[p], __shfl_xor_sync(0xffffffffu, az[p], o));
    }
    float3 u, v;
    up2(ax[p], u.x, v.x);
    up2(ay[p], u.y, v.y);
    up2(az[p], u.z, v.z);
    if (lane == 2 * p) mine = u;
    if (lane == 2 * p + 1) mine = v;
  }
  const int t = t0 + lane;
  if (lane >= K || t >= a.n) return;
  const float4 acc = make_float4(a.G * mine.x, a.G * mine.y, a.G * mine.z, 0.f);
  a.acc[t] = acc;
  if (kick && a.vel) {
    float4 v = a.vel[t];
    v.x = __fmaf_rn(a.half_dt, acc.x, v.x);
    v.y = __fmaf_rn(a.half_dt, acc.y, v.y);
    v.z = __fmaf_rn(a.half_dt, acc.z, v.z);
    a.vel[t] = v;
  }
}

template <int K>
__global__ void __launch_bounds__(32 * kSmallWarps) k_ap_small(APArgs a) {
  small_targets<K>(a, (blockIdx.x * kSmallWarps + (threadIdx.x >> 5)) * K, true);
}

// Many simulations: (entry, first target) per CTA of kSmallWarps x 8 targets
// (with warps to spare, more targets share each source's load and copies).
// 500 simulations of 1,000 particles take 264 us a step, 276 through a work queue
// of tiles; 64 of them 45 against 59.
__global__ void __launch_bounds__(32 * kSmallWarps) k_ap_small_batch(
    const APArgs* __restrict__ args, int nargs, const int2* __restrict__ items, int kick,
    unsigned* err) {
  const int2 it = items[blockIdx.x];
  if (it.x < 0 || it.x >= nargs || it.y < 0) {   // a stale or corrupt item: skipped, reported
    if (threadIdx.x == 0) raise_err(err, NB_DEVERR_QUEUE);
    return;
  }
  const APArgs a = args[it.x];
  small_targets<8>(a, it.y + 8 * (int)(threadIdx.x >> 5), kick != 0);
}

// Two targets per warp up to as many warps as the device has schedulers (4 per
// SM), four above.  A step takes 8.2 us at n = 1,000 and 10.3 at 2,048, 20.5 at both
// with the packed, source-split tiles of k_allpairs.cu; eight targets per warp
// 12.3 at 2,048, too few warps.
int launch_allpairs_small(const APArgs& a, cudaStream_t st) {
  const int K = a.n <= 8 * device_sm_count() ? 2 : 4;
  const int blocks = (a.n + K * kSmallWarps - 1) / (K * kSmallWarps);
  if (K == 2) k_ap_small<2><<<blocks, 32 * kSmallWarps, 0, st>>>(a);
  else k_ap_small<4><<<blocks, 32 * kSmallWarps, 0, st>>>(a);
  NB_CUDA(cudaGetLastError());
  return NB_OK;
}

int small_batch_targets() { return 8 * kSmallWarps; }

int launch_allpairs_small_batch(const APArgs* args, int nargs, const int2* items, int nitems,
                                bool kick, unsigned* err, cudaStream_t st) {
  k_ap_small_batch<<<nitems, 32 * kSmallWarps, 0, st>>>(args, nargs, items, kick ? 1 : 0, err);
  NB_CUDA(cudaGetLastError());
  return NB_OK;
}

int warm_allpairs_small_kernels() {
  return warm_fns(k_ap_small<2>, k_ap_small<4>, k_ap_small_batch);
}

}  // namespace nb
