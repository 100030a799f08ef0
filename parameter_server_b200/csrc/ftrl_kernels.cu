// Online FTRL-proximal on key-range sharded device hash tables: the fused
// communication+compute kernels of the product path, plus the same phases as
// stand-alone kernels for the unfused NCCL baseline.
//
// One rank = one GPU = worker r (streams minibatches) + server r (owns the keys
// of [sep[r], sep[r+1]) in an open-addressing table {key -> w, z, pos, neg}).
// A training step is one cooperative kernel, or two for a large minibatch:
//
//   pull : de-duplicate the minibatch's keys into a per-minibatch table that is laid
//          out by owner; every owner then reads "its" region of every worker's table
//          with coalesced peer loads over NVLink, looks the keys up in its own shard
//          (creating missing ones), remembers the shard slot of every request and
//          stores the weights straight into the worker's weight array with coalesced
//          peer stores.
//   rows : row by row X·w, the logistic loss, the coefficient −y/(1+e^{y·Xw}) and at
//          once the row's part of Xᵀ·coef and of the pos/neg row counts per unique
//          key, into the worker's accumulator array.
//   push : every owner reads its region of every worker's accumulators with coalesced
//          peer loads and applies the FTRL update to the slots it remembered, worker
//          by worker.
//
// No key is hashed twice on the owner, no record is packed, routed or copied into an
// inbox: the per-minibatch table IS the message, and what crosses NVLink are whole
// 1024-slot chunks (8 bytes of key out, 4 bytes of weight back, 4 or 16 bytes of
// gradient out per slot).
//
// The arithmetic is the reference's server rule FTRLModel::setValue
// (src/linear_method/ftrl_model.h:81-112), the worker gradient of LogitLoss
// (src/linear_method/loss.h:73-88) and FTRL::countKeys
// (src/linear_method/ftrl.cc:154-174); the message flow replaces
// SharedParameter::push/pull (src/parameter/shared_parameter.h:14-26,90-149) and
// KVVector::getValue (src/parameter/kv_vector.h:215-227).
// The schedule is bulk-synchronous (one legal serialisation of the reference's
// eventual-consistency execution): pull(e) sees every update of step e-1.
#include <cstddef>
#include <cstdlib>

#include "psb_common.cuh"

namespace psb {

struct ShardState {  // per-key state as the update rule sees it
  float w;
  float z;
  uint32_t pos;  // rule 0: #positive rows seen; rule 1: bit pattern of Σg² (float)
  uint32_t neg;
};

// One slot of an owner's table: 32 bytes = one DRAM sector.  Key and weight sit in
// the same 16 bytes, so a lookup is ONE 16-byte load per probe; an update is a
// read-modify-write of the same sector.
struct __align__(32) ShardSlot {
  uint64_t key;      // offset 0: kEmptyKey when free
  float w;           // offset 8
  float z;           // offset 12
  uint32_t pos;      // offset 16
  uint32_t neg;      // offset 20
  uint64_t reserved; // offset 24
};
static_assert(sizeof(ShardSlot) == 32 && offsetof(ShardSlot, w) == 8 && offsetof(ShardSlot, pos) == 16, "ShardSlot layout");

struct FtrlHyper {
  float alpha, beta, l1, l2;
  int rule;  // 0 = count-based ‖g‖ estimate (reference), 1 = Σ g² (McMahan et al.)
  int pad;
  // Tail-feature filter (src/linear_method/ftrl.cc:99-106, src/parameter/frequency_filter.h:28-43):
  // the owner adds every pushed key's row count to its count-min sketch and updates (and creates)
  // a key only once the estimate exceeds tail_freq, so rare keys never enter the model.  The
  // reference filters on the pull path; here the counts travel with the push anyway, the sketch
  // is local to the owner, and a key without a table entry pulls as 0 — the same model, no extra
  // message.  Off when tail_freq == 0 or cm == nullptr.
  uint32_t* cm;
  uint32_t cm_width;
  int cm_k;
  uint32_t tail_freq;
  uint32_t pad2;
};

// The per-minibatch table of every rank is cut into one region of R = 2^region_log2 slots per
// owner: a key of owner o lives in region o at the top region_log2 bits of its hash (linear
// probing confined to an aligned chunk of kChunkSlots slots).  The shard tables index with the
// top bits of the same hash, so chunk c of region o on EVERY worker covers the same contiguous
// range of owner o's shard table: an owner block that takes chunk c walks all workers' requests
// for one narrow range of its table, and the same key sent by two workers is always in the
// same chunk (worker-by-worker order needs block-level barriers only).
constexpr int kChunkSlots = 1024;
constexpr uint32_t kBadSlot = 0xFFFFFFFFu;   // request slot is empty
constexpr uint32_t kAbsent = 0xFFFFFFFEu;    // key has no entry in the shard (and none was made)

struct FtrlPeers {
  KeySeps seps;
  int rank;
  int max_probe;
  uint64_t tab_mask;                       // shard capacity − 1
  ShardSlot* tab;                          // this rank's shard (only its owner touches it)
  uint64_t* lt_keys[PSB_MAX_RANKS];        // rank r: per-minibatch key table [world << region_log2]
  float* lt_w[PSB_MAX_RANKS];              // rank r: pulled weight per slot (written by the owners)
  void* lt_acc[PSB_MAX_RANKS];             // rank r: gradient accumulators, two buffers of float or float4 per slot
  uint64_t* ready[PSB_MAX_RANKS];          // rank o: [sender] pull sequence whose table is complete
  uint64_t* replied[PSB_MAX_RANKS];        // rank s: [owner]  pull sequence whose weights are written
  uint64_t* grads[PSB_MAX_RANKS];          // rank o: [sender] push sequence whose accumulators are complete
  uint32_t* in_slot;                       // owner: [sender << region_log2 | index] shard slot of the request
  uint64_t* in_keys;                       // owner: copy of the requested keys (tail filter only, else nullptr)
  uint64_t timeout_ns;
  uint32_t tab_shift;                      // 64 − log2(shard capacity): slot = mix64(key) >> tab_shift
  uint32_t region_log2;
};

struct Minibatch {
  const void* offsets;     // rows+1, int64 (or int32 when off32)
  const void* keys;        // nnz keys: uint64, or uint32 feature ids (key_mode 1, 2)
  const float* vals;       // nnz values or nullptr (binary features)
  const float* y;          // rows, ±1
  int64_t nnz;
  int rows;
  uint16_t off32;          // offsets are int32
  uint16_t key_mode;       // 0: uint64 keys; 1: uint32 ids, key = id; 2: uint32 ids, key = mix64(id)
};

__device__ __forceinline__ int64_t mb_offset(const Minibatch& M, int64_t r) {
  return M.off32 ? (int64_t) reinterpret_cast<const int32_t*>(M.offsets)[r] : reinterpret_cast<const int64_t*>(M.offsets)[r];
}

struct __align__(16) AccSlot {  // accumulator of one per-minibatch slot when row counts are tracked
  float g;    // gradient
  float pos;  // #positive rows containing the key (exact in fp32: a minibatch has < 2^24 rows)
  float neg;  // #negative rows containing the key
  float pad;
};

// One 16-byte vector reduction per non-zero instead of separate atomics on g and counts.
__device__ __forceinline__ void red_add_acc(AccSlot* p, float g, float pos, float neg) {
  asm volatile("red.global.add.v4.f32 [%0], {%1, %2, %3, %4};" ::"l"(p), "f"(g), "f"(pos), "f"(neg), "f"(0.f) : "memory");
}

struct LocalScratch {
  uint64_t* lt_keys;   // this rank's per-minibatch table (all kEmptyKey between steps)
  float* lt_w;         // pulled weight per slot
  void* lt_acc;        // accumulators: [2][slots] float (soa) or AccSlot
  uint64_t lt_slots;   // world << region_log2
  uint32_t* slot_of;   // nnz: local slot of each non-zero
  float* coef;         // rows: −y/(1+e^{y·Xw})
  float* xw;           // rows: X·w (predictions)
  uint32_t* send_cnt;  // [PSB_MAX_RANKS] scratch of the unfused baseline
  uint32_t* recv_cnt;  // [PSB_MAX_RANKS] scratch of the unfused baseline
  double* stats;       // [0] Σloss [1] rows [2] ‖w‖₁ [3] ‖w‖₂² [4] nnz(w) [5] unique keys [6] table entries
  uint32_t* status;    // StatusCode etc.
  uint64_t* trace;     // optional [16]: globaltimer at phase boundaries of the last step (see kTrace*)
  // soa != 0: no pos/neg row counts are tracked, an accumulator is one float (the random
  // accesses of the gradient scatter then stay inside L2: a quarter of the footprint).
  uint32_t soa;
  uint32_t parity;     // which of the two accumulator buffers this step uses
  uint32_t* region;    // state of the table's size, see below
  int64_t two_launch_nnz;  // non-zeros from which on a step takes two launches (0: kTwoLaunchNnz)
};

// How much of the per-minibatch table a step uses.  The table is allocated for the largest minibatch the job may
// send, but every slot of it is walked four times a step (owner lookup, owner update, key reset, accumulator
// reset) and its keys and accumulators are probed at random, so a step works in the first 2^r slots only: r from
// the minibatch's non-zeros (first_region_log2), twice the slots as often as its keys do not fit (phase_localize).
// One GPU only: with several, chunk c of every worker's table must cover the same key range.
// B200, 10,000 rows (0.34 M keys) with the tail filter in 2^22 / 2^20 slots: step 264 / 167 us before the other changes;
// 100,000 rows (2.4 M keys) in 2^24 / 2^22: 825 / 699 us.
enum RegionWord : int {
  kRegionNow = 0,       // log2 slots of the last pull; the push of the same step works in it too
  kRegionFloor = 1,     // log2 slots that some minibatch of this engine needed: no step starts with fewer
  kRegionMisfit = 2,    // log2 slots in which a pull's keys did not fit last
};

template <bool kCounts>
__device__ __forceinline__ size_t acc_bytes() { return kCounts ? sizeof(AccSlot) : sizeof(float); }

// Streams (keys, slot map) are read or written once per phase; they carry an evict-first L2 policy so
// that the hash tables stay resident (gradient phase 200 -> 181 us with 16-byte accumulators, measured).
#define PSB_STREAM_POLICY(pol) const uint64_t pol = l2_evict_first_policy()
#define PSB_LD_U64(p, pol) ld_stream_u64((p), (pol))
#define PSB_LD_U32(p, pol) ld_stream_u32((p), (pol))
#define PSB_LD_F32(p, pol) ld_stream_f32((p), (pol))
#define PSB_ST_U32(p, v, pol) st_stream_u32((p), (v), (pol))

// trace slots: 0 start, 1 localized, 2 all owners replied, 3 rows done (a step: gradients too),
//              4 flags sent and tables cleared, 5 applied; of two launches 6 the start of the second
#define PSB_TRACE(L, gtid, i) do { if ((L).trace != nullptr && (gtid) == 0) (L).trace[i] = globaltimer_ns(); } while (0)

// Both tables index with the TOP bits of the same 64-bit hash (see FtrlPeers).
__device__ __forceinline__ uint64_t shard_hash(uint64_t key, uint32_t shift) { return mix64(key) >> shift; }

__device__ __forceinline__ uint64_t mb_key(const Minibatch& M, int64_t i, uint64_t pol) {
  if (M.key_mode == 0) return PSB_LD_U64(reinterpret_cast<const uint64_t*>(M.keys) + i, pol);
  const uint64_t id = PSB_LD_U32(reinterpret_cast<const uint32_t*>(M.keys) + i, pol);
  return M.key_mode == 2 ? mix64(id) : id;
}

// ------------------------------------------------------------------ phases
// A non-zero's reference to its key: the slot, and the entry of the gradient cache that the key may use.  The entry
// comes from the key's home in the WHOLE table, so which keys share an entry (and with it how their sums round) does
// not depend on the slots that a step works in.  With more slots than kRefBits can tell, or several GPUs, the
// reference is the slot alone and the entry is made from it.
constexpr int kHotLog2 = 10;
constexpr int kHotEntries = 1 << kHotLog2;
constexpr uint32_t kRefBits = 32 - kHotLog2;
__device__ __forceinline__ uint32_t hot_entry(uint32_t slot) { return (slot * 2654435761u) >> (32 - kHotLog2); }  // top bits
struct Refs {
  bool packed;
  __device__ __forceinline__ Refs(const FtrlPeers& P, uint32_t rlog2) : packed(P.seps.world == 1 && rlog2 <= kRefBits) {}
  __device__ __forceinline__ uint32_t make(uint32_t slot, uint32_t entry) const {
    if (!packed || slot == kBadSlot) return slot;
    const uint32_t ref = entry << kRefBits | slot;
    return ref == kBadSlot ? ref - (1u << kRefBits) : ref;
  }
  __device__ __forceinline__ uint32_t slot(uint32_t ref) const { return packed ? ref & ((1u << kRefBits) - 1u) : ref; }
  __device__ __forceinline__ uint32_t entry(uint32_t ref) const { return packed ? ref >> kRefBits : hot_entry(ref); }
};

// Home slot of `key` in a per-minibatch table (region of its owner, top bits of its hash inside) in the low half, its
// cache entry in the high half.  A region has at least 4 slots.
__device__ __forceinline__ uint64_t local_home(const FtrlPeers& P, uint64_t key, uint32_t rlog2) {
  const uint64_t o = P.seps.world > 1 ? (uint64_t)route_owner(P.seps, key) : 0ull, x = mix64(key);
  return (o << rlog2) | (x >> (64 - rlog2)) | (uint64_t)hot_entry((uint32_t)(x >> (64 - P.region_log2))) << 32;
}

// De-duplication of the minibatch's keys is bound by memory latency, not by bandwidth: every key
// costs a streamed load of the key and then a dependent random read of the table.  The loop is
// therefore software-pipelined: while a key is resolved, the table read of the thread's next key and the load of the
// key after that are already in flight (the asm loads are issued in program
// order, their results are used one and two iterations later).  A table read that is stale by the
// time it is used only sends the key through the compare-and-swap path, which re-reads.
__device__ __forceinline__ uint64_t ld_table_u64(const uint64_t* p) {
  uint64_t v; asm volatile("ld.global.u64 %0, [%1];" : "=l"(v) : "l"(p)); return v;
}

// Slot of `key` in a per-minibatch table, entered when it is new; `cur` is what its home slot h held when it was read
// (nothing is removed while keys are entered, so a stale value is an empty slot at worst, and the compare-and-swap
// tells).  ~0 when the probe limit is hit.  (Looking at the home slot again cost an L2 request per new or displaced
// key: 9.6 M non-zeros of 2.4 M keys in 2^23 slots 133 -> 110 us.)
__device__ __forceinline__ uint64_t place_key(uint64_t* keys, uint64_t cmask, uint64_t h, uint64_t key, int max_probe, uint64_t cur,
                                              uint32_t* fresh) {
  const uint64_t base = h & ~cmask;
  for (int i = 1;; ++i) {
    if (cur == key) return h;
    if (cur == kEmptyKey) {
      cur = atomicCAS(reinterpret_cast<unsigned long long*>(keys + h), (unsigned long long)kEmptyKey, (unsigned long long)key);
      if (cur == kEmptyKey) { ++*fresh; return h; }
      if (cur == key) return h;
    }
    if (i >= max_probe) return ~0ull;
    h = base | ((h + 1) & cmask);
    cur = keys[h];
  }
}

// Returns the number of keys this thread entered.  With fewer than 2^P.region_log2 slots a key that finds no
// place within kFullChain slots leaves the size in the misfit word instead of an error, and its block gives up: the
// caller starts over with more slots.  So long a chain comes up when about 0.7 of a large table is taken, and from
// there on a new key walks dozens of slots, one dependent read each.  B200, 9.6 M non-zeros, sum of squares, in 2^22 /
// 2^23 / 2^24 slots: 2.9 M keys (0.69 of the smallest) 611 / 553 / 697 us a step, 3.2 M 680 / 575 / 707, 3.5 M 806 / 594 / 728.
// The step that finds out takes 0.3 to 1 ms more, once for an engine.
constexpr int kFullChain = 256;
__device__ __forceinline__ uint32_t phase_localize(const FtrlPeers& P, const Minibatch& M, const LocalScratch& L,
                                                   size_t gtid, size_t gsz, uint32_t rlog2) {
  PSB_STREAM_POLICY(pol);
  const int64_t step = (int64_t)gsz;
  const uint64_t region = 1ull << rlog2;
  const uint64_t cmask = (region < (uint64_t)kChunkSlots ? region : (uint64_t)kChunkSlots) - 1;
  const Refs refs(P, rlog2);
  const int max_probe = rlog2 < P.region_log2 && kFullChain < P.max_probe ? kFullChain : P.max_probe;
  __shared__ int s_full;
  if (threadIdx.x == 0) s_full = 0;
  __syncthreads();
  uint32_t fresh = 0;
  int64_t i = (int64_t)gtid;
  if (i >= M.nnz) return 0u;
  uint64_t key0 = mb_key(M, i, pol);
  uint64_t key1 = i + step < M.nnz ? mb_key(M, i + step, pol) : kEmptyKey;
  uint64_t h0 = local_home(P, key0, rlog2);
  uint64_t cur0 = ld_table_u64(L.lt_keys + (uint32_t)h0);
  for (; i < M.nnz; i += step) {
    uint64_t key2 = kEmptyKey, h1 = 0, cur1 = 0;
    if (i + 2 * step < M.nnz) key2 = mb_key(M, i + 2 * step, pol);
    if (i + step < M.nnz) {
      h1 = local_home(P, key1, rlog2);
      cur1 = ld_table_u64(L.lt_keys + (uint32_t)h1);
    }
    const uint64_t at = place_key(L.lt_keys, cmask, (uint32_t)h0, key0, max_probe, cur0, &fresh);
    if (*(volatile int*)&s_full) break;
    if (at == ~0ull) {
      if (rlog2 < P.region_log2) { L.region[kRegionMisfit] = rlog2; s_full = 1; break; }
      set_status(L.status, kLocalTableFull, 0, 0);
    }
    PSB_ST_U32(L.slot_of + i, refs.make((uint32_t)at, (uint32_t)(h0 >> 32)), pol);      // (uint32_t)~0 is kBadSlot
    key0 = key1; h0 = h1; cur0 = cur1; key1 = key2;
  }
  return fresh;
}
// Adds a block's values to stats[at], ..., stats[at + kN - 1] with one fp64 atomic each; every thread of the block calls
// it.  (One per warp, thousands of warps wait in line at one address: 20 us of a 600 us step at each use.)
template <int kN>
__device__ __forceinline__ void block_add(double* stats, const int (&at)[kN], const double (&v)[kN]) {
  __shared__ double sh[8][kN];     // blocks of 256 threads
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  __syncthreads();
#pragma unroll
  for (int k = 0; k < kN; ++k) {
    const double s = warp_sum_d(v[k]);
    if (lane == 0) sh[warp][k] = s;
  }
  __syncthreads();
#pragma unroll
  for (int k = 0; k < kN; ++k) {
    if (threadIdx.x != k) continue;
    double s = 0.0;
    for (int w = 0; w < (int)(blockDim.x >> 5); ++w) s += sh[w][k];
    if (s != 0.0) atomicAdd(stats + at[k], s);
  }
}
__device__ __forceinline__ void block_add1(double* stats, int at, double v) {
  const int a[1] = {at};
  const double x[1] = {v};
  block_add<1>(stats, a, x);
}

// ---- shard table probes (owner side, this GPU's own memory)
// weight of `key` and its slot; kAbsent when the key has no entry
__device__ __forceinline__ uint32_t shard_find(const ShardSlot* tab, uint64_t mask, uint32_t shift, uint64_t key,
                                               int max_probe, float* w) {
  uint64_t slot = shard_hash(key, shift) & mask;
  for (int i = 0; i < max_probe; ++i) {
    uint64_t k, wz;
    asm volatile("ld.global.v2.u64 {%0, %1}, [%2];" : "=l"(k), "=l"(wz) : "l"(tab + slot) : "memory");
    if (k == key) { *w = __uint_as_float((uint32_t)wz); return (uint32_t)slot; }
    if (k == kEmptyKey) break;
    slot = (slot + 1) & mask;
  }
  *w = 0.f;
  return kAbsent;
}

// slot of `key`, created when missing (w = z = n = 0: the same model as "absent"); kAbsent when the
// probe limit is reached
__device__ __forceinline__ uint32_t shard_find_or_insert(ShardSlot* tab, uint64_t mask, uint32_t shift, uint64_t key,
                                                         int max_probe, float* w, int* inserted) {
  uint64_t slot = shard_hash(key, shift) & mask;
  for (int i = 0; i < max_probe; ++i) {
    uint64_t k, wz;
    asm volatile("ld.global.v2.u64 {%0, %1}, [%2];" : "=l"(k), "=l"(wz) : "l"(tab + slot) : "memory");
    if (k == key) { *w = __uint_as_float((uint32_t)wz); return (uint32_t)slot; }
    if (k == kEmptyKey) {
      const unsigned long long prev = atomicCAS(reinterpret_cast<unsigned long long*>(&tab[slot].key),
                                                (unsigned long long)kEmptyKey, (unsigned long long)key);
      if (prev == kEmptyKey) { *w = 0.f; ++*inserted; return (uint32_t)slot; }
      if (prev == key) { *w = tab[slot].w; return (uint32_t)slot; }
    }
    slot = (slot + 1) & mask;
  }
  *w = 0.f;
  return kAbsent;
}

// One thread of a block waits (bounded) until flag's epoch reaches `want`; the block learns the outcome.
__device__ __forceinline__ bool block_wait_flag(const uint64_t* flag, uint32_t want, uint64_t timeout_ns, int* sh_ok) {
  __syncthreads();
  if (threadIdx.x == 0) {
    bool ok;
    wait_epoch_ge(flag, want, timeout_ns, &ok);
    *sh_ok = ok ? 1 : 0;
  }
  __syncthreads();
  return *sh_ok != 0;
}

constexpr int kLookupItems = kChunkSlots / 256;   // slots per thread and chunk (blocks of 256 threads)

// Owner side of the pull.  A task is (sender s, chunk c of this owner's region in s's table).
// Tasks are numbered sender-major starting with this rank itself, so the blocks that serve
// different senders wait for different flags and a slow sender holds up only its own blocks.
// `insert`: create missing keys (training); off for predictions and under the tail filter.
// kAhead: home slots of the shard that are on their way before the first is looked at.
template <int kAhead>
__device__ __forceinline__ void phase_lookup(const FtrlPeers& P, const LocalScratch& L, uint32_t seq, bool insert,
                                             uint32_t rlog2, int* sh_ok) {
  const int world = P.seps.world;
  const uint64_t region = 1ull << rlog2;
  const uint32_t chunk = region < (uint64_t)kChunkSlots ? (uint32_t)region : (uint32_t)kChunkSlots;
  const uint32_t chunks = (uint32_t)(region / chunk);
  const uint32_t tasks = chunks * (uint32_t)world;
  int dins = 0;
  int have = -1;   // sender whose flag this block has seen
  bool have_ok = false;
  for (uint32_t t = blockIdx.x; t < tasks; t += gridDim.x) {
    const int s = (P.rank + (int)(t / chunks)) % world;
    const uint32_t c = t % chunks;
    if (s != have) {
      have_ok = s == P.rank ? true : block_wait_flag(P.ready[P.rank] + s, seq, P.timeout_ns, sh_ok);
      have = s;
      if (!have_ok && threadIdx.x == 0) set_status(L.status, kWaitTimeout, (uint32_t)s, 1);
    }
    const size_t in0 = ((size_t)s << rlog2) + (size_t)c * chunk;          // owner-side index
    const size_t lt0 = ((size_t)P.rank << rlog2) + (size_t)c * chunk;     // index in the sender's table
    const bool peer = s != P.rank;
    const uint64_t* rk = P.lt_keys[s] + lt0;
    float* rw = P.lt_w[s] + lt0;
    uint64_t key[kLookupItems];
#pragma unroll
    for (int k = 0; k < kLookupItems; ++k) {
      const uint32_t i = (uint32_t)k * 256u + threadIdx.x;
      key[k] = kEmptyKey;
      if (i < chunk && have_ok) key[k] = peer ? ld_relaxed_sys_u64(rk + i) : __ldcg(rk + i);
    }
#pragma unroll
    for (int k = 0; k < kLookupItems; k += kAhead) {
      uint64_t hk[kAhead], hw[kAhead];
#pragma unroll
      for (int j = 0; j < kAhead; ++j) {
        hk[j] = kEmptyKey; hw[j] = 0ull;
        if (kAhead > 1 && key[k + j] != kEmptyKey)
          asm volatile("ld.global.v2.u64 {%0, %1}, [%2];" : "=l"(hk[j]), "=l"(hw[j])
                       : "l"(P.tab + (shard_hash(key[k + j], P.tab_shift) & P.tab_mask)) : "memory");
      }
#pragma unroll
      for (int j = 0; j < kAhead; ++j) {
        const uint32_t i = (uint32_t)(k + j) * 256u + threadIdx.x;
        uint32_t slot = kBadSlot;
        float w = 0.f;
        if (key[k + j] != kEmptyKey) {
          if (kAhead > 1 && hk[j] == key[k + j]) {
            slot = (uint32_t)(shard_hash(key[k + j], P.tab_shift) & P.tab_mask);
            w = __uint_as_float((uint32_t)hw[j]);
          } else if (insert) {
            slot = shard_find_or_insert(P.tab, P.tab_mask, P.tab_shift, key[k + j], P.max_probe, &w, &dins);
            if (slot == kAbsent) set_status(L.status, kShardTableFull, 0, 0);
          } else {
            slot = kAhead > 1 && hk[j] == kEmptyKey ? kAbsent : shard_find(P.tab, P.tab_mask, P.tab_shift, key[k + j], P.max_probe, &w);
          }
        }
        // Lanes leave the probes above at different times.  Without the meeting point a warp stores in pieces, and parts
        // of sectors are slow: 9.6 M distinct keys in 2^24 slots, lookup 312 -> 217 us.
        __syncwarp();
        if (i >= chunk) continue;
        P.in_slot[in0 + i] = slot;
        if (P.in_keys != nullptr) P.in_keys[in0 + i] = key[k + j];
        if (have_ok) {
          if (peer) st_relaxed_sys_f32(rw + i, w); else rw[i] = w;
        }
      }
    }
  }
  if (insert) block_add1(L.stats, 6, (double)dins);
}

// Rows are walked a warp at a time; a lane first issues the loads of up to kRowBatch of its
// non-zeros, then consumes them, so that several slot-map loads are in flight per lane.
constexpr int kRowBatch = 4;

__device__ __forceinline__ void phase_spmv_loss(const Minibatch& M, const LocalScratch& L, const Refs refs, size_t gwarp,
                                                size_t nwarps, int lane, bool count) {
  double loss = 0.0;
  PSB_STREAM_POLICY(pol);
  for (int64_t row = (int64_t)gwarp; row < M.rows; row += (int64_t)nwarps) {
    const int64_t b = mb_offset(M, row), e = mb_offset(M, row + 1);
    float s = 0.f;
    for (int64_t i0 = b + lane; i0 < e; i0 += 32 * kRowBatch) {
      uint32_t sl[kRowBatch];
      float x[kRowBatch];
#pragma unroll
      for (int k = 0; k < kRowBatch; ++k) {
        const int64_t i = i0 + 32 * k;
        sl[k] = i < e ? PSB_LD_U32(L.slot_of + i, pol) : kBadSlot;
        x[k] = (M.vals != nullptr && i < e) ? PSB_LD_F32(M.vals + i, pol) : 1.f;
      }
#pragma unroll
      for (int k = 0; k < kRowBatch; ++k) {
        if (sl[k] != kBadSlot) s += x[k] * __ldcg(L.lt_w + refs.slot(sl[k]));   // written by other GPUs: not through L1
      }
    }
    s = warp_sum(s);
    if (lane == 0) {
      const float y = M.y[row];
      const float m = y * s;
      loss += (double)log1pexp(-m);
      L.coef[row] = -y / (1.f + __expf(m));
      L.xw[row] = s;
    }
  }
  if (count) block_add1(L.stats, 0, loss);      // (lane 0 has the row's loss, the others zero)
}

// Block-local cache of gradient accumulators for frequently hit slots.  Under Zipf
// popularity a few keys receive a large share of all non-zeros; accumulating them in
// shared memory and flushing once per block removes the same-address serialisation of
// global atomics.  Entries are claimed first come, first served; a slot that finds its
// cache line taken by another slot falls back to the global atomic.
struct HotCache {
  uint32_t slot[kHotEntries];
  float g[kHotEntries];
  uint32_t pos[kHotEntries], neg[kHotEntries];   // native 32-bit shared-memory atomics; a block sees fewer than 2^31 non-zeros
};

// Adds gradients (and row counts) to the accumulators of this step through the block's cache.
template <bool kCounts>
struct HotScatter {
  HotCache* hc;
  float* accf;
  AccSlot* accv;
  __device__ __forceinline__ HotScatter(const LocalScratch& L, HotCache* h) : hc(h) {
    accf = reinterpret_cast<float*>(L.lt_acc) + (size_t)L.parity * L.lt_slots;
    accv = reinterpret_cast<AccSlot*>(L.lt_acc) + (size_t)L.parity * L.lt_slots;
    for (int i = threadIdx.x; i < kHotEntries; i += blockDim.x) {
      hc->slot[i] = kBadSlot;
      hc->g[i] = 0.f;
      if (kCounts) hc->pos[i] = hc->neg[i] = 0u;
    }
    __syncthreads();
  }
  __device__ __forceinline__ void add(uint32_t sl, uint32_t h, float gv, bool is_pos) {
    uint32_t cur = hc->slot[h];
    if (cur == kBadSlot) {
      const uint32_t prev = atomicCAS(&hc->slot[h], kBadSlot, sl);
      cur = prev == kBadSlot ? sl : prev;
    }
    if (cur == sl) {
      atomicAdd(&hc->g[h], gv);
      if (kCounts) atomicAdd(is_pos ? &hc->pos[h] : &hc->neg[h], 1u);
    } else if (kCounts) {
      red_add_acc(accv + sl, gv, is_pos ? 1.f : 0.f, is_pos ? 0.f : 1.f);
    } else {
      atomicAdd(accf + sl, gv);
    }
  }
  __device__ __forceinline__ void flush() {
    __syncthreads();
    for (int i = threadIdx.x; i < kHotEntries; i += blockDim.x) {
      const uint32_t sl = hc->slot[i];
      if (sl == kBadSlot) continue;
      if (kCounts) {
        red_add_acc(accv + sl, hc->g[i], (float)hc->pos[i], (float)hc->neg[i]);
      } else {
        atomicAdd(accf + sl, hc->g[i]);
      }
    }
  }
};

// gradient alone, from stored coefficients (the unfused baseline)
template <bool kCounts>
__device__ __forceinline__ void phase_grad(const Minibatch& M, const LocalScratch& L, const Refs refs, size_t gwarp,
                                           size_t nwarps, int lane, HotCache* hc) {
  HotScatter<kCounts> scatter(L, hc);
  PSB_STREAM_POLICY(pol);
  for (int64_t row = (int64_t)gwarp; row < M.rows; row += (int64_t)nwarps) {
    const int64_t b = mb_offset(M, row), e = mb_offset(M, row + 1);
    const float c = L.coef[row];
    const bool is_pos = M.y[row] > 0.f;
    for (int64_t i0 = b + lane; i0 < e; i0 += 32 * kRowBatch) {
      uint32_t sls[kRowBatch];
      float x[kRowBatch];
#pragma unroll
      for (int k = 0; k < kRowBatch; ++k) {
        const int64_t i = i0 + 32 * k;
        sls[k] = i < e ? PSB_LD_U32(L.slot_of + i, pol) : kBadSlot;
        x[k] = (M.vals != nullptr && i < e) ? PSB_LD_F32(M.vals + i, pol) : 1.f;
      }
#pragma unroll
      for (int k = 0; k < kRowBatch; ++k)
        if (sls[k] != kBadSlot) scatter.add(refs.slot(sls[k]), refs.entry(sls[k]), c * x[k], is_pos);
    }
  }
  scatter.flush();
}

// A training step's rows, forward and backward in one walk: a warp multiplies a row with the pulled weights, has
// the row's coefficient in registers and scatters the row's gradient at once.  The slots of a row's first
// 32·kRowBatch non-zeros are read once and kept; the coefficient needs no array and the two halves no barrier.
// B200, 100,000 rows: 239 us where X·w and gradient took 42 + 289 (16-byte accumulators, 2^22 slots against 2^24),
// 187 us against 38 + 145 (4-byte).  Bound by the L2: a random weight sector and an atomic per non-zero.
template <bool kCounts>
__device__ __forceinline__ void phase_rows(const Minibatch& M, const LocalScratch& L, const Refs refs, size_t gwarp, size_t nwarps, int lane, HotCache* hc) {
  HotScatter<kCounts> scatter(L, hc);
  double loss = 0.0;
  PSB_STREAM_POLICY(pol);
  for (int64_t row = (int64_t)gwarp; row < M.rows; row += (int64_t)nwarps) {
    const int64_t b = mb_offset(M, row), e = mb_offset(M, row + 1);
    const float y = M.y[row];
    uint32_t sl[kRowBatch];
    float x[kRowBatch], s = 0.f;
    for (int64_t i0 = b + lane, first = 1; first || i0 < e; i0 += 32 * kRowBatch, first = 0) {
      uint32_t t[kRowBatch];
      float v[kRowBatch];
#pragma unroll
      for (int k = 0; k < kRowBatch; ++k) {
        const int64_t i = i0 + 32 * k;
        t[k] = i < e ? PSB_LD_U32(L.slot_of + i, pol) : kBadSlot;
        v[k] = (M.vals != nullptr && i < e) ? PSB_LD_F32(M.vals + i, pol) : 1.f;
      }
#pragma unroll
      for (int k = 0; k < kRowBatch; ++k) {
        if (t[k] != kBadSlot) s += v[k] * __ldcg(L.lt_w + refs.slot(t[k]));   // written by other GPUs: not through L1
        if (first) { sl[k] = t[k]; x[k] = v[k]; }
      }
    }
    s = warp_sum(s);
    const float m = y * s;
    const float c = -y / (1.f + __expf(m));
    if (lane == 0) {
      loss += (double)log1pexp(-m);
      L.xw[row] = s;
    }
    const bool is_pos = y > 0.f;
#pragma unroll
    for (int k = 0; k < kRowBatch; ++k)
      if (sl[k] != kBadSlot) scatter.add(refs.slot(sl[k]), refs.entry(sl[k]), c * x[k], is_pos);
    for (int64_t i = b + lane + 32 * kRowBatch; i < e; i += 32) {
      const uint32_t t = PSB_LD_U32(L.slot_of + i, pol);
      const float v = M.vals != nullptr ? PSB_LD_F32(M.vals + i, pol) : 1.f;
      if (t != kBadSlot) scatter.add(refs.slot(t), refs.entry(t), c * v, is_pos);
    }
  }
  block_add1(L.stats, 0, loss);      // (lane 0 has the row's loss, the others zero)
  scatter.flush();
}

// Between the gradient phase and the owners' update a worker empties its key table for the next
// minibatch (every owner has finished reading it: the worker saw all `replied` flags before its
// SpMV) and zeroes the accumulator buffer of the NEXT step (the owners read that one during the
// previous step's update, which they finished before they replied to this step's pull).
__device__ __forceinline__ void clear_keys(uint64_t* keys, size_t slots, size_t gtid, size_t gsz) {
  uint4* k = reinterpret_cast<uint4*>(keys);
  const uint4 empty = make_uint4(0xFFFFFFFFu, 0xFFFFFFFFu, 0xFFFFFFFFu, 0xFFFFFFFFu);
  for (size_t i = gtid; i < slots / 2; i += gsz) k[i] = empty;
  if (slots & 1) { if (gtid == 0) keys[slots - 1] = kEmptyKey; }
}
// With one GPU nobody else reads the accumulators: the update zeroes each where it reads it and there is one buffer.
template <bool kCounts>
__device__ __forceinline__ void phase_reset_tables(const FtrlPeers& P, const LocalScratch& L, uint32_t rlog2, size_t gtid, size_t gsz) {
  clear_keys(L.lt_keys, (size_t)P.seps.world << rlog2, gtid, gsz);
  if (P.seps.world == 1) return;
  const size_t bytes = L.lt_slots * acc_bytes<kCounts>();
  char* next = reinterpret_cast<char*>(L.lt_acc) + (size_t)(L.parity ^ 1u) * bytes;
  uint4* a = reinterpret_cast<uint4*>(next);
  const uint4 zero = make_uint4(0u, 0u, 0u, 0u);
  for (size_t i = gtid; i < bytes / 16; i += gsz) a[i] = zero;
  for (size_t i = (bytes / 16) * 16 + gtid; i < bytes; i += gsz) next[i] = 0;
}

__device__ __forceinline__ float ftrl_sqrt_n(float pos, float neg) {
  const float all = pos + neg;
  return all == 0.f ? 0.f : sqrtf(pos * neg / all);
}

// The reference's per-key server update (src/linear_method/ftrl_model.h:88-110).
__device__ __forceinline__ void ftrl_update(ShardState& e, float g, uint32_t dpos, uint32_t dneg,
                                            const FtrlHyper& h, float& dn1, float& dn2, int& dnnz) {
  float sqrt_n, sqrt_n_new;
  if (h.rule == 0) {
    sqrt_n = ftrl_sqrt_n((float)e.pos, (float)e.neg);
    e.pos += dpos;
    e.neg += dneg;
    sqrt_n_new = ftrl_sqrt_n((float)e.pos, (float)e.neg);
  } else {
    float n = __uint_as_float(e.pos);
    sqrt_n = sqrtf(n);
    n += g * g;
    sqrt_n_new = sqrtf(n);
    e.pos = __float_as_uint(n);
    e.neg += dpos + dneg;
  }
  const float sigma = (sqrt_n_new - sqrt_n) / h.alpha;
  e.z += g - sigma * e.w;
  const float l2 = h.l2 + (h.beta + sqrt_n_new) / h.alpha;
  const float w_old = e.w;
  const float az = fabsf(e.z) - h.l1;
  const float w = az > 0.f ? -copysignf(az, e.z) / l2 : 0.f;
  e.w = w;
  dn1 += fabsf(w) - fabsf(w_old);
  dn2 += w * w - w_old * w_old;
  dnnz += (w != 0.f && w_old == 0.f) - (w == 0.f && w_old != 0.f);
}

__device__ __forceinline__ bool tail_filter_on(const FtrlHyper& h) { return h.tail_freq != 0u && h.cm != nullptr; }

struct ApplyAcc {  // per-thread deltas of the model statistics, flushed once per kernel
  float dn1 = 0.f, dn2 = 0.f;
  int dnnz = 0, dins = 0;
};

__device__ __forceinline__ void apply_flush(ApplyAcc& a, double* stats) {
  const int at[4] = {2, 3, 4, 6};
  const double v[4] = {(double)a.dn1, (double)a.dn2, (double)a.dnnz, (double)a.dins};
  block_add<4>(stats, at, v);
  a = ApplyAcc();
}

// A slot is read and written as the 32-byte sector it is: one 256-bit access each way.  (Two 8-byte stores into a
// sector cost the L2 twice the operations, and what a partial write evicts has to be merged in memory.)
struct SlotWords { uint64_t key, wz, pn, reserved; };
__device__ __forceinline__ SlotWords load_slot(const ShardSlot* p) {
  SlotWords v;
  asm volatile("ld.global.v4.u64 {%0, %1, %2, %3}, [%4];" : "=l"(v.key), "=l"(v.wz), "=l"(v.pn), "=l"(v.reserved) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ void store_slot(ShardSlot* p, const SlotWords& v) {
  asm volatile("st.global.v4.u64 [%0], {%1, %2, %3, %4};" ::"l"(p), "l"(v.key), "l"(v.wz), "l"(v.pn), "l"(v.reserved) : "memory");
}
// The key of a slot is written once, before any update of it, so storing it again changes nothing.  A caller that may
// have entered the key just now stores the key it has: a 32-byte load need not see this thread's own 8-byte
// compare-and-swap, since the memory model orders accesses of the same size only.
__device__ __forceinline__ void apply_slot(ShardSlot* tab, uint32_t slot, SlotWords v, float g, uint32_t dpos, uint32_t dneg,
                                           const FtrlHyper& h, ApplyAcc& acc) {
  ShardState e{__uint_as_float((uint32_t)v.wz), __uint_as_float((uint32_t)(v.wz >> 32)), (uint32_t)v.pn, (uint32_t)(v.pn >> 32)};
  ftrl_update(e, g, dpos, dneg, h, acc.dn1, acc.dn2, acc.dnnz);
  v.wz = (uint64_t)__float_as_uint(e.z) << 32 | __float_as_uint(e.w);
  v.pn = (uint64_t)e.neg << 32 | e.pos;
  store_slot(tab + slot, v);
}

// gradient (and row counts) of request `i` of a chunk, from the sender's accumulators
template <bool kCounts>
__device__ __forceinline__ void load_acc(const void* base, size_t i, bool peer, float* g, uint32_t* dpos, uint32_t* dneg) {
  if (kCounts) {
    const AccSlot* p = reinterpret_cast<const AccSlot*>(base) + i;
    float4 v;
    if (peer)
      asm volatile("ld.relaxed.sys.global.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "l"(p) : "memory");
    else
      v = __ldcg(reinterpret_cast<const float4*>(p));
    *g = v.x; *dpos = (uint32_t)v.y; *dneg = (uint32_t)v.z;
  } else {
    const float* p = reinterpret_cast<const float*>(base) + i;
    *g = peer ? ld_relaxed_sys_f32(p) : __ldcg(p);
    *dpos = 0u; *dneg = 0u;
  }
}

template <bool kCounts>
__device__ __forceinline__ void zero_acc(void* base, size_t i) {
  if (kCounts) reinterpret_cast<float4*>(base)[i] = make_float4(0.f, 0.f, 0.f, 0.f);
  else reinterpret_cast<float*>(base)[i] = 0.f;
}

// Lanes hold consecutive slots: does this lane's 32-byte sector of accumulators hold a used one?  Used sectors are
// zeroed whole.  All 32 lanes call it.  (A partial write of a sector is much slower: 10 k rows in 2^22 slots, update
// phase 433 us with the used 16 bytes alone, 169 us with all slots.)
template <bool kCounts>
__device__ __forceinline__ bool sector_used(bool used) {
  const unsigned m = __ballot_sync(0xffffffffu, used);
  return kCounts ? (m >> (threadIdx.x & 30) & 3u) != 0u : (m >> (threadIdx.x & 24) & 255u) != 0u;
}

// Owner side of the push: chunk c of every sender, sender by sender in rank order (the reference
// applies each worker's push separately; the order only matters per key, and a key is in the
// same chunk on every sender).  The shard slots were resolved by the pull of the same step.
template <bool kCounts>
__device__ __forceinline__ void phase_apply_chunks(const FtrlPeers& P, const LocalScratch& L, const FtrlHyper& H,
                                                   uint32_t seq, uint32_t rlog2, ApplyAcc& acc, int* sh_ok) {
  const int world = P.seps.world;
  const uint64_t region = 1ull << rlog2;
  const uint32_t chunk = region < (uint64_t)kChunkSlots ? (uint32_t)region : (uint32_t)kChunkSlots;
  const uint32_t chunks = (uint32_t)(region / chunk);
  const size_t abytes = L.lt_slots * acc_bytes<kCounts>();
  uint32_t arrived = 0, failed = 0;   // bit s: this block has seen sender s's flag / its wait ran out
  for (uint32_t c = blockIdx.x; c < chunks; c += gridDim.x) {
    for (int s = 0; s < world; ++s) {
      if (!((arrived | failed) >> s & 1u)) {
        const bool ok = s == P.rank ? true : block_wait_flag(P.grads[P.rank] + s, seq, P.timeout_ns, sh_ok);
        if (ok) arrived |= 1u << s; else failed |= 1u << s;
        if (!ok && threadIdx.x == 0) set_status(L.status, kWaitTimeout, (uint32_t)s, 2);
      }
      if (failed >> s & 1u) continue;   // a sender that never arrived is skipped
      const size_t in0 = ((size_t)s << rlog2) + (size_t)c * chunk;
      const size_t lt0 = ((size_t)P.rank << rlog2) + (size_t)c * chunk;
      const bool peer = s != P.rank;
      char* abase = reinterpret_cast<char*>(P.lt_acc[s]) + (size_t)L.parity * abytes;
      uint32_t slot[kLookupItems];
#pragma unroll
      for (int k = 0; k < kLookupItems; ++k) {
        const uint32_t i = (uint32_t)k * 256u + threadIdx.x;
        slot[k] = i < chunk ? __ldcg(P.in_slot + in0 + i) : kBadSlot;
      }
      // two slots at a time: the random reads of both sectors are in flight before the first is written (a sender's
      // keys are distinct, so are their slots)
#pragma unroll
      for (int k = 0; k < kLookupItems; k += 2) {
        float g[2]; uint32_t dpos[2], dneg[2];
        SlotWords e[2];
        const auto zero = [&](int j) {
          const uint32_t i = (uint32_t)(k + j) * 256u + threadIdx.x;
          if (world == 1 && sector_used<kCounts>(slot[k + j] != kBadSlot) && i < chunk) zero_acc<kCounts>(abase, lt0 + i);
        };
#pragma unroll
        for (int j = 0; j < 2; ++j) {
          const uint32_t i = (uint32_t)(k + j) * 256u + threadIdx.x;
          if (slot[k + j] < kAbsent) {
            e[j] = load_slot(P.tab + slot[k + j]);
            load_acc<kCounts>(abase, lt0 + i, peer, &g[j], &dpos[j], &dneg[j]);
          }
          if (kCounts) zero(j);
        }
#pragma unroll
        for (int j = 0; j < 2; ++j)
          if (slot[k + j] < kAbsent) apply_slot(P.tab, slot[k + j], e[j], g[j], dpos[j], dneg[j], H, acc);
        // one-float accumulators: zeroed between the loads above and the updates, the warp's next reads waited for the
        // stores (2.4 M keys in 2^24 slots: step 712 -> 639 us; with counts 784 us here, 780 there)
        if (!kCounts) { zero(0); zero(1); }
      }
      __syncthreads();
    }
  }
}

// Tail-filter form of the owner's update: a sender's counts must all be in the sketch before any
// of its keys is queried, so every sender is bracketed by grid-wide barriers; keys that pass the
// filter and have no entry yet get one here (the pull did not create them).
__device__ __forceinline__ void phase_apply_filtered(cg::grid_group& grid, const FtrlPeers& P, const LocalScratch& L,
                                                     const FtrlHyper& H, uint32_t seq, uint32_t rlog2, ApplyAcc& acc,
                                                     int* sh_ok) {
  const int world = P.seps.world;
  const uint64_t region = 1ull << rlog2;
  const size_t abytes = L.lt_slots * sizeof(AccSlot);
  const size_t gtid = (size_t)blockIdx.x * blockDim.x + threadIdx.x, gsz = (size_t)gridDim.x * blockDim.x;
  for (int s = 0; s < world; ++s) {
    const bool ok = s == P.rank ? true : block_wait_flag(P.grads[P.rank] + s, seq, P.timeout_ns, sh_ok);
    if (!ok && threadIdx.x == 0) set_status(L.status, kWaitTimeout, (uint32_t)s, 2);
    const size_t in0 = (size_t)s << rlog2, lt0 = (size_t)P.rank << rlog2;
    const bool peer = s != P.rank;
    char* abase = reinterpret_cast<char*>(P.lt_acc[s]) + (size_t)L.parity * abytes;
    for (size_t i = gtid; ok && i < region; i += gsz) {
      const uint64_t key = P.in_keys[in0 + i];
      if (key == kEmptyKey) continue;
      float g; uint32_t dpos, dneg;
      load_acc<true>(abase, lt0 + i, peer, &g, &dpos, &dneg);
      cm_insert(H.cm, H.cm_width, H.cm_k, key, dpos + dneg);
    }
    grid.sync();
    const int lane = threadIdx.x & 31;
    for (size_t i0 = gtid - lane; ok && i0 < region; i0 += gsz) {    // whole warps: a region may be shorter than one
      const size_t i = i0 + lane;
      const uint64_t key = i < region ? P.in_keys[in0 + i] : kEmptyKey;
      float g = 0.f; uint32_t dpos = 0u, dneg = 0u;
      if (key != kEmptyKey) load_acc<true>(abase, lt0 + i, peer, &g, &dpos, &dneg);
      if (world == 1 && sector_used<true>(key != kEmptyKey) && i < region) zero_acc<true>(abase, lt0 + i);
      __syncwarp();
      if (key == kEmptyKey) continue;
      if (cm_query(H.cm, H.cm_width, H.cm_k, key, 0xFFFFFFFFu) <= H.tail_freq) continue;
      uint32_t slot = __ldcg(P.in_slot + in0 + i);
      if (slot >= kAbsent) {
        float w;
        slot = shard_find_or_insert(P.tab, P.tab_mask, P.tab_shift, key, P.max_probe, &w, &acc.dins);
        if (slot == kAbsent) { set_status(L.status, kShardTableFull, 0, 0); continue; }
      }
      SlotWords v = load_slot(P.tab + slot);
      v.key = key;
      apply_slot(P.tab, slot, v, g, dpos, dneg, H, acc);
    }
    grid.sync();
  }
}

// ------------------------------------------------------------ fused kernels
constexpr uint32_t kPullInsert = 1u;   // flags: create missing keys in the shard
constexpr uint32_t kPullPredict = 2u;  // ftrl_pull_kernel: a prediction

// De-duplication and lookup: the table is complete, every owner has been told, this rank's owner side has served
// every worker, and every owner has served this one.  Returns the log2 slots worked in.
template <int kAhead>
__device__ __forceinline__ uint32_t pull_weights(cg::grid_group& grid, const FtrlPeers& P, const Minibatch& M, const LocalScratch& L,
                                                 uint32_t seq, uint32_t flags, uint32_t try_log2, size_t gtid, size_t gsz, int* sh_ok) {
  const int world = P.seps.world;
  uint32_t rlog2 = world > 1 ? P.region_log2 : min(P.region_log2, max(try_log2, __ldcg(L.region + kRegionFloor)));
  uint32_t fresh;
  for (;;) {
    fresh = phase_localize(P, M, L, gtid, gsz, rlog2);
    if (world > 1) __threadfence_system();   // the table must be visible to its owners before the flag is
    grid.sync();
    // uniform: the word is written before the barrier above or, with another value, after the one below
    if (rlog2 >= P.region_log2 || __ldcg(L.region + kRegionMisfit) != rlog2) break;
    clear_keys(L.lt_keys, (size_t)1 << rlog2, gtid, gsz);
    ++rlog2;
    grid.sync();
    if (gtid == 0) L.region[kRegionFloor] = rlog2;    // a size that did not fit is never tried again
  }
  if (!(flags & kPullPredict)) block_add1(L.stats, 5, (double)fresh);
  if (gtid == 0) L.region[kRegionNow] = rlog2;
  PSB_TRACE(L, gtid, 1);
  // this worker's table is complete: tell every owner, then serve the other workers' tables
  if (blockIdx.x == 0 && threadIdx.x < world && world > 1) {
    __threadfence_system();
    st_release_sys_u64(P.ready[threadIdx.x] + P.rank, (uint64_t)seq << 32);
  }
  phase_lookup<kAhead>(P, L, seq, (flags & kPullInsert) != 0u, rlog2, sh_ok);
  if (world > 1) __threadfence_system();   // the weights must be visible to their workers before the flag is
  grid.sync();
  if (blockIdx.x == 0 && threadIdx.x < world && world > 1)
    st_release_sys_u64(P.replied[threadIdx.x] + P.rank, (uint64_t)seq << 32);
  // every owner must have answered before the rows are multiplied
  if (world > 1) {
    __syncthreads();
    if (threadIdx.x < world && threadIdx.x != P.rank) {
      bool ok;
      wait_epoch_ge(P.replied[P.rank] + threadIdx.x, seq, P.timeout_ns, &ok);
      if (!ok) set_status(L.status, kWaitTimeout, threadIdx.x, 3);
    }
    __syncthreads();
  }
  PSB_TRACE(L, gtid, 2);
  return rlog2;
}

// The pull on its own: of a large training step, and of a prediction, which also multiplies the rows, empties the
// key table again (every owner has replied, nobody reads it any more) and leaves the statistics alone: one launch
// where saving and restoring them and emptying the table took four more.  8 blocks of 256 threads per SM (32
// registers per thread, 24 bytes spilled): its phases are bound by memory latency.  9.6 M non-zeros of 2.4 M keys take
// the same time with 6 blocks and no spills, and with the prediction compiled apart.
constexpr int kPullBlocksPerSM = 8;
__global__ void __launch_bounds__(256, kPullBlocksPerSM)
ftrl_pull_kernel(FtrlPeers P, Minibatch M, LocalScratch L, uint32_t seq, uint32_t flags, uint32_t try_log2) {
  cg::grid_group grid = cg::this_grid();
  const size_t gtid = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  const size_t gsz = (size_t)gridDim.x * blockDim.x;
  __shared__ int sh_ok;
  const bool predict = (flags & kPullPredict) != 0u;
  if (gtid == 0 && !predict) L.stats[1] += (double)M.rows;
  PSB_TRACE(L, gtid, 0);
  const uint32_t rlog2 = pull_weights<1>(grid, P, M, L, seq, flags, try_log2, gtid, gsz, &sh_ok);
  if (predict) {
    clear_keys(L.lt_keys, (size_t)P.seps.world << rlog2, gtid, gsz);
    phase_spmv_loss(M, L, Refs(P, rlog2), gtid >> 5, gsz >> 5, threadIdx.x & 31, false);
    PSB_TRACE(L, gtid, 3);
  }
}

// A training step, whole (kPull) or after ftrl_pull_kernel: rows and push.  Rows and push alone: 100,000 rows with
// 3 / 4 / 5 / 6 blocks per SM take 657 / 639 / 656 / 676 us a step (count rule), 690 / 580 / 590 / 600 (sum of squares);
// from 5 on registers spill (at 4, 16 bytes of the sum of squares), with 3 too few random accesses are in flight.  Whole, 4 and
// 5 measure the same; 5 spills 36 to 68 bytes.
constexpr int kStepBlocksPerSM = 5, kPushBlocksPerSM = 4;
// Slots from which on the rows are walked twice, weights first, gradients then, when the table is larger than the
// non-zeros alone ask for, that is when almost every slot is used: weights (64 MB) and accumulators fit the L2 one after
// the other, not together.  9.6 M non-zeros in 2^24 slots, one walk / two: 9.6 M keys 1174 / 1136 us a step (sum of
// squares) and 1444 / 1396 (count), 8.2 M 1065 / 1043 and 1305 / 1291, 6.7 M 944 / 945; 2.4 M 639 / 698.
constexpr uint32_t kTwoWalksLog2 = 24;
template <bool kCounts, bool kPull>
__global__ void __launch_bounds__(256, kPull ? kStepBlocksPerSM : kPushBlocksPerSM)
ftrl_step_kernel(FtrlPeers P, Minibatch M, LocalScratch L, FtrlHyper H, uint32_t pull_seq, uint32_t push_seq, uint32_t flags,
                 uint32_t try_log2) {
  cg::grid_group grid = cg::this_grid();
  const size_t gtid = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  const size_t gsz = (size_t)gridDim.x * blockDim.x;
  const int lane = threadIdx.x & 31;
  const int world = P.seps.world;
  __shared__ HotCache hot;
  __shared__ int sh_ok;

  uint32_t rlog2;
  if (kPull) {
    if (gtid == 0) L.stats[1] += (double)M.rows;
    PSB_TRACE(L, gtid, 0);
    rlog2 = pull_weights<2>(grid, P, M, L, pull_seq, flags, try_log2, gtid, gsz, &sh_ok);
  } else {
    rlog2 = __ldcg(L.region + kRegionNow);
    PSB_TRACE(L, gtid, 6);
  }
  if (!kPull && world == 1 && rlog2 >= kTwoWalksLog2 && rlog2 > try_log2) {
    phase_spmv_loss(M, L, Refs(P, rlog2), gtid >> 5, gsz >> 5, lane, true);
    grid.sync();
    phase_grad<kCounts>(M, L, Refs(P, rlog2), gtid >> 5, gsz >> 5, lane, &hot);
  } else {
    phase_rows<kCounts>(M, L, Refs(P, rlog2), gtid >> 5, gsz >> 5, lane, &hot);
  }
  if (world > 1) __threadfence_system();   // the accumulators must be visible to their owners before the flag is
  grid.sync();
  PSB_TRACE(L, gtid, 3);
  if (blockIdx.x == 0 && threadIdx.x < world && world > 1)
    st_release_sys_u64(P.grads[threadIdx.x] + P.rank, (uint64_t)push_seq << 32);
  phase_reset_tables<kCounts>(P, L, rlog2, gtid, gsz);
  PSB_TRACE(L, gtid, 4);
  {
    ApplyAcc acc;
    if (kCounts && tail_filter_on(H)) {
      phase_apply_filtered(grid, P, L, H, push_seq, rlog2, acc, &sh_ok);
    } else {
      phase_apply_chunks<kCounts>(P, L, H, push_seq, rlog2, acc, &sh_ok);
    }
    apply_flush(acc, L.stats);
  }
  PSB_TRACE(L, gtid, 5);
}

// ------------------------------------------------- stand-alone phase kernels
// (the unfused baseline: same arithmetic, records packed by owner and exchanged with all_to_all)
__global__ void k_localize(FtrlPeers P, Minibatch M, LocalScratch L) {
  const uint32_t fresh = phase_localize(P, M, L, (size_t)blockIdx.x * blockDim.x + threadIdx.x, (size_t)gridDim.x * blockDim.x, P.region_log2);
  block_add1(L.stats, 5, (double)fresh);
}
__global__ void k_spmv_loss(FtrlPeers P, Minibatch M, LocalScratch L) {
  const size_t gtid = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (gtid == 0) L.stats[1] += (double)M.rows;
  phase_spmv_loss(M, L, Refs(P, P.region_log2), gtid >> 5, ((size_t)gridDim.x * blockDim.x) >> 5, threadIdx.x & 31, true);
}
__global__ void k_grad(FtrlPeers P, Minibatch M, LocalScratch L) {
  const size_t gtid = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  __shared__ HotCache hot;
  phase_grad<true>(M, L, Refs(P, P.region_log2), gtid >> 5, ((size_t)gridDim.x * blockDim.x) >> 5, threadIdx.x & 31, &hot);
}
// count unique keys per owner (pass 1 of packing for all_to_all_v)
__global__ void k_count_owner(KeySeps seps, LocalScratch L, uint32_t* counts) {
  const size_t gsz = (size_t)gridDim.x * blockDim.x;
  uint32_t c[PSB_MAX_RANKS] = {0};
  for (uint64_t s = (size_t)blockIdx.x * blockDim.x + threadIdx.x; s < L.lt_slots; s += gsz) {
    const uint64_t key = L.lt_keys[s];
    if (key != kEmptyKey) {
      const int o = route_owner(seps, key);
#pragma unroll
      for (int t = 0; t < PSB_MAX_RANKS; ++t) c[t] += (o == t);
    }
  }
#pragma unroll
  for (int t = 0; t < PSB_MAX_RANKS; ++t) {
    const uint32_t v = __reduce_add_sync(0xffffffffu, c[t]);
    if ((threadIdx.x & 31) == 0 && v) atomicAdd(counts + t, v);
  }
}
// pass 2: write (key, slot) grouped by owner; cursors[] start at the segment bases
__global__ void k_pack_keys(KeySeps seps, LocalScratch L, uint32_t* cursors, uint64_t* out_keys,
                            uint32_t* out_slot) {
  const size_t gsz = (size_t)gridDim.x * blockDim.x;
  for (uint64_t s = (size_t)blockIdx.x * blockDim.x + threadIdx.x; s < L.lt_slots; s += gsz) {
    const uint64_t key = L.lt_keys[s];
    if (key != kEmptyKey) {
      const int o = route_owner(seps, key);
      const unsigned m = __match_any_sync(__activemask(), o);
      const int leader = __ffs(m) - 1, lane = threadIdx.x & 31;
      uint32_t base = 0;
      if (lane == leader) base = atomicAdd(cursors + o, (uint32_t)__popc(m));
      base = __shfl_sync(m, base, leader);
      const uint32_t at = base + __popc(m & ((1u << lane) - 1u));
      out_keys[at] = key;
      out_slot[at] = (uint32_t)s;
    }
  }
}
// owner side of an unfused pull: w for each requested key (0 when absent)
__global__ void k_lookup(const ShardSlot* tab, uint64_t mask, uint32_t shift, int max_probe,
                         const uint64_t* keys, uint32_t n, float* out_w) {
  for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x) {
    float w;
    shard_find(tab, mask, shift, keys[i], max_probe, &w);
    out_w[i] = w;
  }
}
__global__ void k_scatter_w(const uint32_t* slots, const float* w, uint32_t n, LocalScratch L) {
  AccSlot* acc = reinterpret_cast<AccSlot*>(L.lt_acc) + (size_t)L.parity * L.lt_slots;
  for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x) {
    const uint32_t s = slots[i];
    L.lt_w[s] = w[i];
    AccSlot z;
    z.g = 0.f; z.pos = 0.f; z.neg = 0.f; z.pad = 0.f;
    acc[s] = z;
  }
}
__global__ void k_pack_push(const uint32_t* slots, uint32_t n, LocalScratch L, float* out_g, uint64_t* out_cnt) {
  const AccSlot* acc = reinterpret_cast<const AccSlot*>(L.lt_acc) + (size_t)L.parity * L.lt_slots;
  for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x) {
    const uint32_t s = slots[i];
    out_g[i] = acc[s].g;
    out_cnt[i] = ((uint64_t)(uint32_t)acc[s].pos << 32) | (uint64_t)(uint32_t)acc[s].neg;
    L.lt_keys[s] = kEmptyKey;
  }
}
__global__ void k_sketch_insert(const uint64_t* rk, const uint64_t* rc, uint32_t n, FtrlHyper h) {
  for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x) {
    const uint64_t key = __ldcg(rk + i);
    if (key == kEmptyKey) continue;
    const uint64_t c = __ldcg(rc + i);
    cm_insert(h.cm, h.cm_width, h.cm_k, key, (uint32_t)(c >> 32) + (uint32_t)c);
  }
}
// one flat record list of one sender: find or create every key, apply the update
__global__ void k_apply(ShardSlot* tab, uint64_t mask, uint32_t shift, int max_probe, const uint64_t* rk,
                        const float* rg, const uint64_t* rc, uint32_t n, FtrlHyper h, double* stats,
                        uint32_t* status) {
  ApplyAcc acc;
  const bool filter = tail_filter_on(h);
  for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x) {
    const uint64_t key = __ldcg(rk + i);
    if (key == kEmptyKey) continue;
    if (filter && cm_query(h.cm, h.cm_width, h.cm_k, key, 0xFFFFFFFFu) <= h.tail_freq) continue;
    float w;
    const uint32_t slot = shard_find_or_insert(tab, mask, shift, key, max_probe, &w, &acc.dins);
    if (slot == kAbsent) { set_status(status, kShardTableFull, 0, 0); continue; }
    const uint64_t c = __ldcg(rc + i);
    SlotWords v = load_slot(tab + slot);
    v.key = key;
    apply_slot(tab, slot, v, __ldcg(rg + i), (uint32_t)(c >> 32), (uint32_t)c, h, acc);
  }
  apply_flush(acc, stats);
}
__global__ void k_clear_local(LocalScratch L) {
  clear_keys(L.lt_keys, L.lt_slots, (size_t)blockIdx.x * blockDim.x + threadIdx.x,
             (size_t)gridDim.x * blockDim.x);
}
// dump the non-zero weights of a shard: out_keys/out_w sized by capacity, *count receives the number
__global__ void k_dump_nonzero(const ShardSlot* tab, uint64_t mask, uint64_t* out_keys,
                               float* out_w, unsigned long long* count) {
  for (uint64_t s = (size_t)blockIdx.x * blockDim.x + threadIdx.x; s <= mask; s += (size_t)gridDim.x * blockDim.x) {
    const uint64_t k = tab[s].key;
    if (k != kEmptyKey && tab[s].w != 0.f) {
      const unsigned long long at = atomicAdd(count, 1ull);
      out_keys[at] = k;
      out_w[at] = tab[s].w;
    }
  }
}
// Move every entry of a shard into a larger table (same hash, more top bits): the table grows
// like the reference's unordered_map (src/linear_method/ftrl_model.h:57) instead of filling up.
__global__ void k_rehash(const ShardSlot* from, uint64_t from_mask, ShardSlot* to, uint64_t to_mask, uint32_t to_shift,
                         int max_probe, uint32_t* status) {
  for (uint64_t s = (size_t)blockIdx.x * blockDim.x + threadIdx.x; s <= from_mask; s += (size_t)gridDim.x * blockDim.x) {
    const ShardSlot e = from[s];
    if (e.key == kEmptyKey) continue;
    float w;
    int ins = 0;
    const uint32_t slot = shard_find_or_insert(to, to_mask, to_shift, e.key, max_probe, &w, &ins);
    if (slot == kAbsent) { set_status(status, kShardTableFull, 0, 1); continue; }
    *reinterpret_cast<float2*>(&to[slot].w) = make_float2(e.w, e.z);
    *reinterpret_cast<uint2*>(&to[slot].pos) = make_uint2(e.pos, e.neg);
  }
}

}  // namespace psb

// ------------------------------------------------------------------ C ABI
using namespace psb;

namespace {
int g_coop_blocks_pull[16] = {0}, g_coop_blocks_step[4][16] = {{0}};

template <typename K>
int coop_grid(K kernel, int* cache) {
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev < 0 || dev >= 16) dev = 0;
  if (cache[dev] == 0) {
    int per_sm = 0, sms = 0;
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, 256, 0);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    if (per_sm > 8) per_sm = 8;
    cache[dev] = per_sm * sms;
  }
  return cache[dev];
}
inline int flat_grid(size_t n, int cap = 148 * 8) {
  size_t b = (n + 255) / 256;
  if (b < 1) b = 1;
  if (b > (size_t)cap) b = cap;
  return (int)b;
}
}  // namespace

extern "C" {

// log2 of the slots a minibatch starts with: three quarters of its non-zeros (a click stream has 0.25 to 0.5 distinct
// keys per non-zero), but up to 2^17 slots, where walking the table costs next to nothing, four times the non-zeros.
static uint32_t first_region_log2(int64_t nnz) {
  const uint64_t n = nnz > 0 ? (uint64_t)nnz : 1ull;
  const uint64_t small = n * 4 < 131072ull ? n * 4 : 131072ull;
  const uint64_t want = n / 4 * 3 > small ? n / 4 * 3 : small;
  uint32_t l = 2;
  while ((1ull << l) < want) ++l;
  // one more bit than a packed reference holds: three eighths will do
  if (l == kRefBits + 1 && (1ull << kRefBits) >= n / 8 * 3) l = kRefBits;
  return l;
}

// Blocks of a launch: every grid-wide barrier costs more with more blocks, so a small minibatch gets one thread for
// every two of its non-zeros and of the slots it works in (and at least a block per SM).
static int step_grid(const FtrlPeers& P, const Minibatch& M, int full, uint32_t try_log2) {
  if (P.seps.world > 1) return full;
  const uint64_t slots = 1ull << (try_log2 < P.region_log2 ? try_log2 : P.region_log2);
  const uint64_t n = (uint64_t)(M.nnz > 0 ? M.nnz : 0) > slots ? (uint64_t)M.nnz : slots;
  const uint64_t want = (n + 511) / 512;
  return want >= (uint64_t)full ? full : want < 148 ? (full < 148 ? full : 148) : (int)want;
}

static int launch_pull(const FtrlPeers* P, const Minibatch* M, const LocalScratch* L, uint32_t seq, uint32_t flags, cudaStream_t stream) {
  uint32_t try_log2 = first_region_log2(M->nnz);
  const int full = coop_grid(ftrl_pull_kernel, g_coop_blocks_pull);
  if (full <= 0) return (int)cudaErrorLaunchFailure;
  const int grid = step_grid(*P, *M, full, try_log2);
  FtrlPeers p = *P; Minibatch m = *M; LocalScratch l = *L;
  void* args[] = {&p, &m, &l, &seq, &flags, &try_log2};
  return (int)cudaLaunchCooperativeKernel((void*)ftrl_pull_kernel, dim3(grid), dim3(256), args, 0, stream);
}

// A prediction: X·w with the weights as they are; no key is created, no statistic changes.
int psb_ftrl_pull_spmv(const FtrlPeers* P, const Minibatch* M, const LocalScratch* L, uint32_t seq, cudaStream_t stream) {
  if (L->lt_w == nullptr || L->lt_acc == nullptr || P->in_slot == nullptr || L->region == nullptr) return (int)cudaErrorInvalidValue;
  return launch_pull(P, M, L, seq, kPullPredict, stream);
}

// Non-zeros from which on a step takes two launches: the pull gains more from its own 8 blocks per SM than the second
// launch costs.  B200, step in one / two launches (count rule, 6 blocks per SM in the second): 48 k non-zeros 44 / 48 us,
// 1 M 185 / 190, 2.9 M 325 / 315, 5.3 M 432 / 419, 9.6 M 738 / 670.
constexpr int64_t kTwoLaunchNnz = 1500000;

// One training step: pull, rows, push (sequence numbers of the pull's and the push's flags).  flags bit 0: create
// missing keys in the shard.  launches: the kernels launched are added.
int psb_ftrl_step(const FtrlPeers* P, const Minibatch* M, const LocalScratch* L, const FtrlHyper* H, uint32_t pull_seq,
                  uint32_t push_seq, uint32_t flags, int* launches, cudaStream_t stream) {
  const bool soa = L->soa != 0;
  const bool filter = H->tail_freq != 0u && H->cm != nullptr;
  if (L->lt_w == nullptr || L->lt_acc == nullptr || P->in_slot == nullptr || L->region == nullptr) return (int)cudaErrorInvalidValue;
  // the count-based rule and the tail filter need the pos/neg counts that the one-float accumulators do not carry
  if (soa && (H->rule == 0 || filter)) return (int)cudaErrorInvalidValue;
  if (filter && P->in_keys == nullptr) return (int)cudaErrorInvalidValue;
  const bool two = M->nnz >= (L->two_launch_nnz > 0 ? L->two_launch_nnz : kTwoLaunchNnz);
  if (two) {
    const int e = launch_pull(P, M, L, pull_seq, flags & kPullInsert, stream);
    if (e != 0) return e;
    ++*launches;
  }
  const void* kernels[4] = {(const void*)ftrl_step_kernel<false, false>, (const void*)ftrl_step_kernel<true, false>,
                            (const void*)ftrl_step_kernel<false, true>, (const void*)ftrl_step_kernel<true, true>};
  const int which = (soa ? 0 : 1) + (two ? 0 : 2);
  const int full = coop_grid(kernels[which], g_coop_blocks_step[which]);
  if (full <= 0) return (int)cudaErrorLaunchFailure;
  uint32_t try_log2 = first_region_log2(M->nnz);
  const int grid = step_grid(*P, *M, full, try_log2);
  FtrlPeers p = *P; Minibatch m = *M; LocalScratch l = *L; FtrlHyper h = *H;
  void* args[] = {&p, &m, &l, &h, &pull_seq, &push_seq, &flags, &try_log2};
  ++*launches;
  return (int)cudaLaunchCooperativeKernel(kernels[which], dim3(grid), dim3(256), args, 0, stream);
}

int psb_ftrl_localize(const FtrlPeers* P, const Minibatch* M, const LocalScratch* L, cudaStream_t s) {
  k_localize<<<flat_grid(M->nnz), 256, 0, s>>>(*P, *M, *L);
  return (int)cudaGetLastError();
}
int psb_ftrl_spmv_loss(const FtrlPeers* P, const Minibatch* M, const LocalScratch* L, cudaStream_t s) {
  k_spmv_loss<<<flat_grid((size_t)M->rows * 32), 256, 0, s>>>(*P, *M, *L);
  return (int)cudaGetLastError();
}
int psb_ftrl_grad(const FtrlPeers* P, const Minibatch* M, const LocalScratch* L, cudaStream_t s) {
  k_grad<<<flat_grid((size_t)M->rows * 32), 256, 0, s>>>(*P, *M, *L);
  return (int)cudaGetLastError();
}
int psb_ftrl_count_owner(const KeySeps* seps, const LocalScratch* L, uint32_t* counts, cudaStream_t s) {
  k_count_owner<<<flat_grid(L->lt_slots), 256, 0, s>>>(*seps, *L, counts);
  return (int)cudaGetLastError();
}
int psb_ftrl_pack_keys(const KeySeps* seps, const LocalScratch* L, uint32_t* cursors, uint64_t* out_keys,
                       uint32_t* out_slot, cudaStream_t s) {
  k_pack_keys<<<flat_grid(L->lt_slots), 256, 0, s>>>(*seps, *L, cursors, out_keys, out_slot);
  return (int)cudaGetLastError();
}
int psb_ftrl_lookup(const void* tab, uint64_t mask, uint32_t shift, int max_probe, const uint64_t* keys,
                    uint32_t n, float* out_w, cudaStream_t s) {
  k_lookup<<<flat_grid(n), 256, 0, s>>>((const ShardSlot*)tab, mask, shift, max_probe, keys, n, out_w);
  return (int)cudaGetLastError();
}
int psb_ftrl_scatter_w(const uint32_t* slots, const float* w, uint32_t n, const LocalScratch* L, cudaStream_t s) {
  k_scatter_w<<<flat_grid(n), 256, 0, s>>>(slots, w, n, *L);
  return (int)cudaGetLastError();
}
int psb_ftrl_pack_push(const uint32_t* slots, uint32_t n, const LocalScratch* L, float* out_g, uint64_t* out_cnt,
                       cudaStream_t s) {
  k_pack_push<<<flat_grid(n), 256, 0, s>>>(slots, n, *L, out_g, out_cnt);
  return (int)cudaGetLastError();
}
int psb_ftrl_apply(void* tab, uint64_t mask, uint32_t shift, int max_probe, const uint64_t* rk, const float* rg,
                   const uint64_t* rc, uint32_t n, const FtrlHyper* h, double* stats, uint32_t* status,
                   cudaStream_t s) {
  if (h->tail_freq != 0u && h->cm != nullptr) k_sketch_insert<<<flat_grid(n), 256, 0, s>>>(rk, rc, n, *h);
  k_apply<<<flat_grid(n), 256, 0, s>>>((ShardSlot*)tab, mask, shift, max_probe, rk, rg, rc, n, *h, stats, status);
  return (int)cudaGetLastError();
}
int psb_ftrl_clear_local(const LocalScratch* L, cudaStream_t s) {
  k_clear_local<<<flat_grid(L->lt_slots), 256, 0, s>>>(*L);
  return (int)cudaGetLastError();
}
int psb_ftrl_dump_nonzero(const void* tab, uint64_t mask, uint64_t* out_keys, float* out_w,
                          unsigned long long* count, cudaStream_t s) {
  k_dump_nonzero<<<flat_grid(mask + 1), 256, 0, s>>>((const ShardSlot*)tab, mask, out_keys, out_w, count);
  return (int)cudaGetLastError();
}
int psb_ftrl_rehash(const void* from, uint64_t from_mask, void* to, uint64_t to_mask, uint32_t to_shift, int max_probe,
                    uint32_t* status, cudaStream_t s) {
  k_rehash<<<flat_grid(from_mask + 1), 256, 0, s>>>((const ShardSlot*)from, from_mask, (ShardSlot*)to, to_mask, to_shift,
                                                     max_probe, status);
  return (int)cudaGetLastError();
}

}  // extern "C"
