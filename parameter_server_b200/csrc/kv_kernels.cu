// Key-range sharded key→value vector on peer memory: the device form of KVVector
// (src/parameter/kv_vector.h) and of the push / pull message pair of SharedParameter
// (src/parameter/shared_parameter.h:14-26, 90-149).
//
// Every rank (server) holds the sorted keys of its key range and k fp32 values per key in
// peer-addressable buffers.  A worker resolves its keys once — owner by key range, slot by binary
// search in the owner's key array, read over NVLink — which is the steady state of the
// reference's key cache (src/system/remote_node.cc:96-184): afterwards pushes and pulls carry
// values only.
//   pull  out[i, :]            = vals[owner_i][slot_i, :]      plain peer loads (16-byte vectors when k % 4 == 0)
//   push  vals[owner_i][slot_i, :] += in[i, :]                 red.add (v4 / v2 / scalar) on peer memory:
//                                                              the sum over workers happens at the owner
// Unknown keys resolve to slot -1: pulls return zeros for them and pushes skip them.
#include "psb_common.cuh"

namespace psb {

struct KvPeers {
  const uint64_t* keys[PSB_MAX_RANKS];   // sorted unique keys of every shard
  float* vals[PSB_MAX_RANKS];            // [nkeys, k]
  int64_t nkeys[PSB_MAX_RANKS];
  KeySeps seps;
  int k;
  int pad;
};

// first index in keys[0, n) whose key is >= `key` (n: none).  All 32 lanes call it: a step splits the range
// into 33 parts, so 2^21 keys take 5 dependent loads where a bisection takes 21.
__device__ __forceinline__ int64_t warp_lower_bound(const uint64_t* keys, int64_t n, uint64_t key, int lane) {
  int64_t lo = 0, hi = n;             // the answer is in [lo, hi]
  while (lo < hi) {
    const int64_t len = hi - lo;
    const int64_t at = len <= 32 ? lo + lane : lo + (len * (lane + 1)) / 33;
    const unsigned below = __ballot_sync(0xffffffffu, at < hi && ld_relaxed_sys_u64(keys + at) < key);
    const int c = __popc(below);      // the first c probes are below the key
    if (len <= 32) return lo + c;
    const int64_t nlo = c > 0 ? lo + (len * c) / 33 + 1 : lo;
    const int64_t nhi = c < 32 ? lo + (len * (c + 1)) / 33 : hi;
    lo = nlo; hi = nhi;
  }
  return lo;
}

// Places of the keys of a list.  Key lists are usually ordered, so the keys of one tile of the list fall into a
// narrow run of the owner's keys: two warps find the run of the tile's first and last key, the block copies it into
// shared memory and every key is looked for there.  A tile over several owners, or a long run, is bisected in the
// owners' memory between those bounds, a tile that is not ordered without them.
// Bound by the dependent loads of a search, not by bytes.  Ordered queries among twice as many keys, one bisection
// per key -> this: 3 x 10^6 queries 101 -> 63 us, 10^6 42 -> 32 us, 3 x 10^5 29 -> 22 us.
constexpr int kResolveThreads = 256, kResolveStage = 3072;   // 24 KB: eight blocks per SM

template <int kPer>     // queries per thread
__global__ void __launch_bounds__(kResolveThreads)
k_kv_resolve(KvPeers P, const uint64_t* __restrict__ q, size_t n, int32_t* __restrict__ owner, int32_t* __restrict__ slot) {
  __shared__ uint64_t s_keys[kResolveStage];
  __shared__ int64_t s_run[2];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  constexpr int kResolveTile = kPer * kResolveThreads;
  const size_t tiles = (n + kResolveTile - 1) / kResolveTile;
  for (size_t t = blockIdx.x; t < tiles; t += gridDim.x) {
    const size_t first = t * kResolveTile, end = first + kResolveTile < n ? first + kResolveTile : n;
    uint64_t key[kPer];
    bool ascending = true;
#pragma unroll
    for (int r = 0; r < kPer; ++r) {
      const size_t i = first + (size_t)r * kResolveThreads + threadIdx.x;
      key[r] = i < end ? q[i] : 0ull;
      if (i < end && i > first) ascending = ascending && q[i - 1] <= key[r];
    }
    const bool ordered = __syncthreads_and(ascending);     // (and the previous tile's shared memory has been read)
    const uint64_t mn = ordered ? q[first] : 0ull, mx = ordered ? q[end - 1] : ~0ull - 1ull;
    const int o0 = route_owner(P.seps, mn), o1 = route_owner(P.seps, mx);
    if (ordered) {
      if (warp < 2) {
        const int64_t at = warp_lower_bound(P.keys[warp == 0 ? o0 : o1], P.nkeys[warp == 0 ? o0 : o1], warp == 0 ? mn : mx, lane);
        if (lane == 0) s_run[warp] = at;
      }
    } else if (threadIdx.x == 0) {
      s_run[0] = 0;
      s_run[1] = P.nkeys[o1];
    }
    __syncthreads();
    const int64_t r0 = s_run[0], last = P.nkeys[o1];
    const int64_t r1 = s_run[1] < last ? s_run[1] + 1 : last;      // one past the largest key's place
    const bool staged = ordered && o0 == o1 && r1 - r0 <= kResolveStage;
    if (staged) {
      for (int64_t i = r0 + threadIdx.x; i < r1; i += kResolveThreads) s_keys[i - r0] = ld_relaxed_sys_u64(P.keys[o0] + i);
      __syncthreads();
    }
#pragma unroll
    for (int r = 0; r < kPer; ++r) {
      const size_t i = t * kResolveTile + (size_t)r * kResolveThreads + threadIdx.x;
      if (i >= n) continue;
      if (staged) {
        int lo = 0, hi = (int)(r1 - r0);
        while (lo < hi) {
          const int mid = (lo + hi) >> 1;
          if (s_keys[mid] < key[r]) lo = mid + 1; else hi = mid;
        }
        owner[i] = o0;
        slot[i] = (lo < (int)(r1 - r0) && s_keys[lo] == key[r]) ? (int32_t)(r0 + lo) : -1;
      } else {
        const int o = o0 == o1 ? o0 : route_owner(P.seps, key[r]);
        const uint64_t* k = P.keys[o];
        int64_t lo = o == o0 ? r0 : 0, hi = o == o1 ? r1 : P.nkeys[o];
        while (lo < hi) {
          const int64_t mid = (lo + hi) >> 1;
          if (ld_relaxed_sys_u64(k + mid) < key[r]) lo = mid + 1; else hi = mid;
        }
        owner[i] = o;
        slot[i] = (lo < P.nkeys[o] && ld_relaxed_sys_u64(k + lo) == key[r]) ? (int32_t)lo : -1;
      }
    }
  }
}

// one thread per (row, 4-float chunk) when k % 4 == 0, otherwise one thread per element
__global__ void k_kv_pull(KvPeers P, const int32_t* __restrict__ owner, const int32_t* __restrict__ slot, size_t n, float* __restrict__ out) {
  const int k = P.k;
  if ((k & 3) == 0) {
    const int chunks = k >> 2;
    const size_t total = n * (size_t)chunks;
    for (size_t t = (size_t)blockIdx.x * blockDim.x + threadIdx.x; t < total; t += (size_t)gridDim.x * blockDim.x) {
      const size_t i = t / chunks;
      const int c = (int)(t % chunks);
      const int32_t s = slot[i];
      float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
      if (s >= 0) {
        const float4* src = reinterpret_cast<const float4*>(P.vals[owner[i]] + (size_t)s * k) + c;
        asm volatile("ld.relaxed.sys.global.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "l"(src) : "memory");
      }
      reinterpret_cast<float4*>(out + i * (size_t)k)[c] = v;
    }
  } else {
    const size_t total = n * (size_t)k;
    for (size_t t = (size_t)blockIdx.x * blockDim.x + threadIdx.x; t < total; t += (size_t)gridDim.x * blockDim.x) {
      const size_t i = t / k;
      const int c = (int)(t % k);
      const int32_t s = slot[i];
      out[t] = s >= 0 ? ld_relaxed_sys_f32(P.vals[owner[i]] + (size_t)s * k + c) : 0.f;
    }
  }
}

__global__ void k_kv_push(KvPeers P, const int32_t* __restrict__ owner, const int32_t* __restrict__ slot, size_t n, const float* __restrict__ in) {
  const int k = P.k;
  if ((k & 3) == 0) {
    const int chunks = k >> 2;
    const size_t total = n * (size_t)chunks;
    for (size_t t = (size_t)blockIdx.x * blockDim.x + threadIdx.x; t < total; t += (size_t)gridDim.x * blockDim.x) {
      const size_t i = t / chunks;
      const int c = (int)(t % chunks);
      const int32_t s = slot[i];
      if (s < 0) continue;
      const float4 v = reinterpret_cast<const float4*>(in + i * (size_t)k)[c];
      float* dst = P.vals[owner[i]] + (size_t)s * k + 4 * c;
      asm volatile("red.relaxed.sys.global.add.v4.f32 [%0], {%1, %2, %3, %4};" ::"l"(dst), "f"(v.x), "f"(v.y), "f"(v.z), "f"(v.w) : "memory");
    }
  } else {
    const size_t total = n * (size_t)k;
    for (size_t t = (size_t)blockIdx.x * blockDim.x + threadIdx.x; t < total; t += (size_t)gridDim.x * blockDim.x) {
      const size_t i = t / k;
      const int32_t s = slot[i];
      if (s >= 0) red_add_sys_f32(P.vals[owner[i]] + (size_t)s * k + (t % k), in[t]);
    }
  }
  __threadfence_system();
}

// baseline helpers: gather / scatter-add on local memory only (used with all_to_all exchanges)
__global__ void k_rows_gather(const float* __restrict__ vals, const int32_t* __restrict__ slot, size_t n, int k, float* __restrict__ out) {
  const size_t total = n * (size_t)k;
  for (size_t t = (size_t)blockIdx.x * blockDim.x + threadIdx.x; t < total; t += (size_t)gridDim.x * blockDim.x) {
    const int32_t s = slot[t / k];
    out[t] = s >= 0 ? vals[(size_t)s * k + (t % k)] : 0.f;
  }
}
__global__ void k_rows_scatter_add(float* __restrict__ vals, const int32_t* __restrict__ slot, size_t n, int k, const float* __restrict__ in) {
  const size_t total = n * (size_t)k;
  for (size_t t = (size_t)blockIdx.x * blockDim.x + threadIdx.x; t < total; t += (size_t)gridDim.x * blockDim.x) {
    const int32_t s = slot[t / k];
    if (s >= 0) atomicAdd(&vals[(size_t)s * k + (t % k)], in[t]);
  }
}

}  // namespace psb

using namespace psb;

namespace {
inline int kgrid(size_t n) { size_t b = (n + 255) / 256; if (b < 1) b = 1; if (b > 148 * 16) b = 148 * 16; return (int)b; }
}

extern "C" {

int psb_kv_resolve(const KvPeers* P, const uint64_t* q, size_t n, int32_t* owner, int32_t* slot, cudaStream_t s) {
  // longer tiles search for fewer runs, as long as every SM still has two of them
  if (n >= 4 * kResolveThreads * 296) k_kv_resolve<4><<<kgrid((n + 3) / 4), kResolveThreads, 0, s>>>(*P, q, n, owner, slot);
  else if (n >= 2 * kResolveThreads * 296) k_kv_resolve<2><<<kgrid((n + 1) / 2), kResolveThreads, 0, s>>>(*P, q, n, owner, slot);
  else k_kv_resolve<1><<<kgrid(n), kResolveThreads, 0, s>>>(*P, q, n, owner, slot);
  return (int)cudaGetLastError();
}
int psb_kv_pull(const KvPeers* P, const int32_t* owner, const int32_t* slot, size_t n, float* out, cudaStream_t s) {
  k_kv_pull<<<kgrid(n * (size_t)((P->k & 3) ? P->k : P->k / 4)), 256, 0, s>>>(*P, owner, slot, n, out);
  return (int)cudaGetLastError();
}
int psb_kv_push(const KvPeers* P, const int32_t* owner, const int32_t* slot, size_t n, const float* in, cudaStream_t s) {
  k_kv_push<<<kgrid(n * (size_t)((P->k & 3) ? P->k : P->k / 4)), 256, 0, s>>>(*P, owner, slot, n, in);
  return (int)cudaGetLastError();
}
int psb_rows_gather(const float* vals, const int32_t* slot, size_t n, int k, float* out, cudaStream_t s) {
  k_rows_gather<<<kgrid(n * (size_t)k), 256, 0, s>>>(vals, slot, n, k, out);
  return (int)cudaGetLastError();
}
int psb_rows_scatter_add(float* vals, const int32_t* slot, size_t n, int k, const float* in, cudaStream_t s) {
  k_rows_scatter_add<<<kgrid(n * (size_t)k), 256, 0, s>>>(vals, slot, n, k, in);
  return (int)cudaGetLastError();
}

}  // extern "C"
