// Fused sparse pull and push: the per-batch id dedup / virtual-index assignment, the
// all-to-all exchange with the owning GPUs over NVLink peer memory, the owner-side hash
// probe (insert on miss) and the optimizer update each run as ONE persistent cooperative
// kernel per direction.  Peer traffic is plain ld/st to symmetric-heap addresses with
// release/acquire flags at system scope; no collective library is involved.  On one GPU there is nothing to push to
// anybody: the row updates are an ordinary kernel there (sparse_push_local_kernel).
//
// What these kernels replace in the reference:
//   pull : SparsePullVarInfo dedup + per-shard RPC fan-out + SparseTable::Pull + scatter back
//          (core/kernels/sparse_table_ops.cc:113-270, core/ps/table/sparse_table.cc:52-66)
//   push : SparsePushVarInfo show/click counting + per-shard RPC + SparseTable::Push + Value::Apply
//          (core/kernels/sparse_table_ops.cc:274-373, core/ps/table/sparse_table.cc:68-83,
//           core/ps/optimizer/{ada_grad,adam,ftrl}_kernel.cc)
//
// Semantics that differ on purpose: the step is synchronous, and gradients of one sign
// arriving from several GPUs (or several columns) are summed and applied once.
//
// Counters that every thread would otherwise hit (per-owner unique counts, the row slab
// bump pointer, the owner-unique index) are advanced once per warp: lanes that need a slot
// are found with a ballot, one lane adds the population count and the others take their
// rank inside the ballot.
#include "sparse_table.cuh"
#include "dense_step.cuh"

namespace tn {

namespace {

constexpr int kThreads = 1024;
constexpr int kRiderUnroll = 2;      // 16-byte reductions in flight per thread of the CTAs that carry the dense step
enum SigKind { kSigPullReq = 0, kSigPullDone = 1, kSigPushReq = 2, kSigPushDone = 3 };
__device__ __forceinline__ unsigned long long* sig_word(unsigned long long* base, int kind, int src) {
  return base + kind * kMaxWorld + src;
}

__device__ __forceinline__ unsigned group_mask(int G) {
  if (G >= 32) return 0xffffffffu;
  unsigned lane = threadIdx.x & 31;
  return ((1u << G) - 1u) << (lane & ~(unsigned)(G - 1));
}
__device__ __forceinline__ unsigned lanemask_lt() {
  unsigned m;
  asm("mov.u32 %0, %%lanemask_lt;" : "=r"(m));
  return m;
}

// Number of ids of this batch: the launch's count, or less when the buffer of a captured step is not full.
__device__ __forceinline__ int batch_ids(const PullArgs& a) {
  return a.n_dev != nullptr ? min(a.n_ids, max(__ldg(a.n_dev), 0)) : a.n_ids;
}

// Warp-aggregated "counter += 1 for every lane in `mask`"; returns this lane's old value.
// Must be called by all 32 lanes; lanes outside `mask` get an unspecified value.
__device__ __forceinline__ int warp_alloc(int* counter, unsigned mask) {
  if (mask == 0) return 0;
  const unsigned lane = threadIdx.x & 31;
  const int leader = __ffs(mask) - 1;
  int base = 0;
  if ((int)lane == leader) base = atomicAdd(counter, __popc(mask));
  base = __shfl_sync(0xffffffffu, base, leader);
  return base + __popc(mask & lanemask_lt());
}

// One GPU: word of `bar` that is set when an error has been met by the time a batch's signs are looked up.  All CTAs of the
// kernels behind go by this word: the status word may change while they run, by their own insertions or those of another
// table in the same launch, and CTAs that start later would do otherwise than those that went before.
constexpr int kLocalSkip = 5;

// ---- dedup of a batch ------------------------------------------------------------------------------------------
// A warp takes `per` x 32 ids at a time (a lane: ids base + lane, base + 32 + lane, ...).  What a batch costs here is the
// latency of the dedup table, which is why a lane has several probes in flight, and the counter that hands out
// positions, which all warps add to: one probe in flight and one atomic per 32 ids took 115 us for 2.1 M ids, four and
// one per 128 ids take 77 us (adding up a whole block's winners first: 101 us, its barriers cost more than the atomics).
// Batches that give a lane only one id keep one.
constexpr int kDedupIds = 4;
__device__ __forceinline__ int dedup_ids_per_lane(int n_ids, int nth) {
  const int per = (n_ids + nth - 1) / nth;
  return per < 1 ? 1 : (per > kDedupIds ? kDedupIds : per);
}

// First occurrence of a sign allocates a position in its owner's segment.  The slot of the dedup table that holds an
// id's sign is left in inverse[] as -2 - slot (negative: "no row" to every reader until dedup_resolve has run), so
// that the second pass is one load per id instead of another probe: 65 -> 31 us for 2.1 M ids.
// kLocal (one GPU): whoever allocates a position also looks the sign up in the table `t` and leaves its row in
// req_row[position]; positions of signs that have no row yet are listed in req_ou[0 .. *ocount).  The table is only read.
// A warp waits for the longest of its chains of dependent accesses, so a lane with one id saves what it can of them: it
// goes to the dedup table with a compare-and-swap at once (in a large batch the later occurrences of a hot sign had better
// find it without queueing an atomic on the same word) and asks for the sign's home slot in the table meanwhile: 10 K ids
// 16.7 -> 13.0 us, but 2.1 M ids, four to a lane, 126 -> 149 us.
template <bool kLocal>
__device__ __forceinline__ void dedup_assign(const PullArgs& a, const TableView& t, int n_ids, int tid, int nth) {
  const SparseCommView& c = a.c;
  const int lane = threadIdx.x & 31, W = kLocal ? 1 : c.world, capo = c.capo;
  const int per = dedup_ids_per_lane(n_ids, nth);
  const bool early = kLocal && per == 1;
  for (long long base = (long long)(tid - lane) * per; base < n_ids; base += (long long)nth * per) {
    unsigned long long key[kDedupIds], old[kDedupIds];
    unsigned hw[kDedupIds];
    unsigned lead = 0, win = 0;              // bit k: this lane probes for / allocates its k-th id
    int from[kDedupIds];
    unsigned long long tkey[kDedupIds];      // kLocal: the table slot a new sign has got to, and its row
    int trow[kDedupIds];
#pragma unroll
    for (int k = 0; k < kDedupIds; ++k) {
      const long long i = base + 32 * k + lane;
      key[k] = (k < per && i < n_ids) ? canon_key((unsigned long long)a.ids[i]) : kEmptyKey;
    }
#pragma unroll
    for (int k = 0; k < kDedupIds; ++k) {
      if (k >= per) continue;
      // lanes of the warp that carry the same sign elect one representative: a hot sign costs one probe per warp
      from[k] = __ffs(__match_any_sync(0xffffffffu, key[k])) - 1;
      hw[k] = (unsigned)mix64(key[k] ^ 0x2545F4914F6CDD1Dull) & c.dd_mask;
      if (key[k] != kEmptyKey && lane == from[k]) {
        lead |= 1u << k;
        old[k] = early ? atomicCAS(&c.dd_keys[hw[k]], kEmptyKey, key[k]) : __ldcg(&c.dd_keys[hw[k]]);
        if (early) {
          const unsigned h = table_home(t, key[k]);
          tkey[k] = __ldcg(&t.keys[h]);
          trow[k] = __ldcg(&t.slots[h]);
        }
      }
    }
    if (early && (lead & 1u) && old[0] == kEmptyKey) { win = 1u; old[0] = key[0]; }
    // Rounds: all of the lane's ids that are still on their way take a step side by side.  One that stands before an empty
    // slot takes it with a compare-and-swap, one that has met another sign moves on to the next slot.
    unsigned todo = lead;
    for (unsigned probes = 0; todo != 0; ++probes) {
      unsigned tried = 0;
#pragma unroll
      for (int k = 0; k < kDedupIds; ++k) {
        if (!((todo >> k) & 1u) || old[k] != kEmptyKey) continue;
        old[k] = atomicCAS(&c.dd_keys[hw[k]], kEmptyKey, key[k]);
        tried |= 1u << k;
      }
#pragma unroll
      for (int k = 0; k < kDedupIds; ++k) {
        if (!((todo >> k) & 1u)) continue;
        if (((tried >> k) & 1u) && old[k] == kEmptyKey) { win |= 1u << k; todo &= ~(1u << k); continue; }
        if (old[k] == key[k]) { todo &= ~(1u << k); continue; }
        hw[k] = (hw[k] + 1) & c.dd_mask;
        old[k] = __ldcg(&c.dd_keys[hw[k]]);
      }
      if (todo != 0 && probes > c.dd_mask) {
        set_status(c.status, kDedupOverflow, 1, 0);
        if (kLocal) c.bar[kLocalSkip] = 1;
#pragma unroll
        for (int k = 0; k < kDedupIds; ++k) if ((todo >> k) & 1u) hw[k] = 0xffffffffu;
        break;
      }
    }
    __syncwarp();
    if (kLocal && !early) {                  // the home slots of the new signs, while their positions are handed out
#pragma unroll
      for (int k = 0; k < kDedupIds; ++k) {
        if (!((win >> k) & 1u)) continue;
        const unsigned h = table_home(t, key[k]);
        tkey[k] = __ldcg(&t.keys[h]);
        trow[k] = __ldcg(&t.slots[h]);
      }
    }
    int pos0 = 0;                            // one owner: positions of all the warp's winners in one go
    if (W == 1) {
      int total = 0;
#pragma unroll
      for (int k = 0; k < kDedupIds; ++k) total += k < per ? __popc(__ballot_sync(0xffffffffu, (win >> k) & 1u)) : 0;
      if (total > 0) {
        if (lane == 0) pos0 = atomicAdd(&c.cnt[0], total);
        pos0 = __shfl_sync(0xffffffffu, pos0, 0);
      }
    }
    if (kLocal) {                            // walk on from home slots that hold another sign, in rounds as well
      unsigned walk = win;
      for (unsigned probes = 1; walk != 0 && probes <= t.cap_mask; ++probes) {
#pragma unroll
        for (int k = 0; k < kDedupIds; ++k) {
          if (!((walk >> k) & 1u)) continue;
          if (tkey[k] == key[k] || tkey[k] == kEmptyKey) { walk &= ~(1u << k); continue; }
          const unsigned h = (table_home(t, key[k]) + probes) & t.cap_mask;
          tkey[k] = __ldcg(&t.keys[h]);
          trow[k] = __ldcg(&t.slots[h]);
        }
      }
    }
#pragma unroll
    for (int k = 0; k < kDedupIds; ++k) {
      if (k >= per) continue;
      const bool winner = (win >> k) & 1u;
      int owner = 0, pos = 0;
      if (W == 1) {
        const unsigned m = __ballot_sync(0xffffffffu, winner);
        pos = pos0 + __popc(m & lanemask_lt());
        pos0 += __popc(m);
      } else {
        owner = winner ? owner_of(key[k], W) : -1;
        const unsigned peers = __match_any_sync(0xffffffffu, owner);
        if (winner) {
          const int leader = __ffs(peers) - 1;
          int b = 0;
          if (lane == leader) b = atomicAdd(&c.cnt[owner], __popc(peers));
          b = __shfl_sync(peers, b, leader);
          pos = b + __popc(peers & lanemask_lt());
        }
      }
      bool missing = false;
      if (winner) {
        if (pos >= capo) {
          set_status(c.status, kOwnerSegOverflow, 1, owner);
          if (kLocal) c.bar[kLocalSkip] = 1;
          c.dd_vals[hw[k]] = -1;
        } else {
          c.stage_ids[owner * capo + pos] = key[k];
          c.dd_vals[hw[k]] = owner * capo + pos;
          if (kLocal) {
            missing = tkey[k] != key[k] && !a.lookup_only;
            c.req_row[pos] = tkey[k] == key[k] && trow[k] >= 0 ? trow[k] : kReqNone;
          }
        }
      }
      if (kLocal) {
        const unsigned mm = __ballot_sync(0xffffffffu, missing);
        const int at = warp_alloc(c.ocount, mm);
        if (missing) c.req_ou[at] = pos;
      }
      __syncwarp();
      const unsigned slot = __shfl_sync(0xffffffffu, hw[k], from[k]);
      const long long i = base + 32 * k + lane;
      if (i < n_ids) a.inverse[i] = slot == 0xffffffffu ? -1 : -2 - (int)slot;
    }
  }
}

// inverse[i]: dedup slot -> position of the sign; with `count`, the batch's show / click counts of every sign.
__device__ __forceinline__ void dedup_resolve(const PullArgs& a, int n_ids, int tid, int nth, bool count) {
  const SparseCommView& c = a.c;
  const int lane = threadIdx.x & 31;
  const int per = dedup_ids_per_lane(n_ids, nth);
  for (long long base = (long long)(tid - lane) * per; base < n_ids; base += (long long)nth * per) {
    int v[kDedupIds];
#pragma unroll
    for (int k = 0; k < kDedupIds; ++k) {
      const long long i = base + 32 * k + lane;
      v[k] = (k < per && i < n_ids) ? a.inverse[i] : -1;
    }
#pragma unroll
    for (int k = 0; k < kDedupIds; ++k) v[k] = v[k] < -1 ? __ldcg(&c.dd_vals[-2 - v[k]]) : -1;
#pragma unroll
    for (int k = 0; k < kDedupIds; ++k) {
      if (k >= per) continue;
      const long long i = base + 32 * k + lane;
      if (i < n_ids) a.inverse[i] = v[k];
      if (!count) continue;
      const unsigned same = __match_any_sync(0xffffffffu, v[k] >= 0 ? v[k] : -2 - lane);
      if (v[k] < 0) continue;
      float* rec = c.cnts + 2 * (size_t)v[k];                       // compact (show, click) pair: stays in L2
      if (lane == __ffs(same) - 1) atomicAdd(rec, (float)__popc(same));      // show: one add per warp and sign
      if (a.labels != nullptr) {
        const float y = a.label_mod > 0 ? a.labels[i % a.label_mod] : a.labels[i];
        if (y != 0.f) atomicAdd(rec + 1, y);
      }
    }
  }
}

// Show / click counts of a batch whose inverse map is complete.
__device__ __forceinline__ void count_shows(const PullArgs& a, int n_ids, int tid, int nth) {
  const int lane = threadIdx.x & 31;
  for (int base = tid - lane; base < n_ids; base += nth) {
    const int i = base + lane;
    const int v = i < n_ids ? a.inverse[i] : -1;
    const unsigned same = __match_any_sync(0xffffffffu, v >= 0 ? v : -2 - lane);
    if (v < 0) continue;
    float* rec = a.c.cnts + 2 * (size_t)v;
    if (lane == __ffs(same) - 1) atomicAdd(rec, (float)__popc(same));
    if (a.labels != nullptr) {
      const float y = a.label_mod > 0 ? a.labels[i % a.label_mod] : a.labels[i];
      if (y != 0.f) atomicAdd(rec + 1, y);
    }
  }
}

// Default value of stored-row element `e` (e < stride) for a brand-new row.
__device__ __forceinline__ float new_row_elem(const SparseOptParams& o, unsigned long long key, int e, int dim) {
  if (e < dim) return o.zero_init ? 0.f : init_weight(o.seed, key, e, dim, o.initial_scale);
  if (o.kind == kAdaGrad && e == dim) return o.initial_g2sum;
  return 0.f;  // slots, show, click; int fields are bit-zero
}

// A group's lanes ask L2 for the 128-byte lines of a row the group will touch in its next loop iteration,
// so the HBM latency of iteration k+1 overlaps the arithmetic and stores of iteration k.
__device__ __forceinline__ void prefetch_row_l2(const float* row, int n_floats, int lane, int G) {
  for (int l = lane; l * 32 < n_floats; l += G) asm volatile("prefetch.global.L2 [%0];" ::"l"(row + 32 * l));
}

__device__ __forceinline__ void prof_mark(const SparseCommView& c, int slot) {
  if (c.prof != nullptr && blockIdx.x == 0 && threadIdx.x == 0) c.prof[slot] = globaltimer_ns();
}

// One requested row, handled by a group of G lanes: initialise a brand-new row (owner) or recompute its initial
// value (other requesters of the same step), or read the stored row; write the pulled row (w[dim], the two CVM
// columns when enabled, zero padding) to `dst`, which is either the requester's matrix itself or a shared-memory
// tile that is written out afterwards.  `rr` is the resolved request word of the probe.
__device__ __forceinline__ void pull_return_row(const PullArgs& a, const TableView& t, int rr, unsigned long long key,
                                                float* dst, int gl, int G) {
  const SparseCommView& c = a.c;
  const SparseOptParams& o = a.opt;
  const int dim = t.dim, stride = t.stride;
  const int uchunks = c.ustride >> 2, rchunks = stride >> 2;
  if (rr == kReqNone) {
    for (int ch = gl; ch < uchunks; ch += G) *reinterpret_cast<float4*>(dst + 4 * ch) = make_float4(0.f, 0.f, 0.f, 0.f);
    return;
  }
  const int r = rr & kReqRowMask;
  float* row = t.rows + (size_t)r * stride;
  if (rr & (kReqNewOwner | kReqNewCopy)) {
    const bool write_row = (rr & kReqNewOwner) != 0;
    const int nch = write_row ? max(rchunks, uchunks) : uchunks;
    for (int ch = gl; ch < nch; ch += G) {
      float4 v;
      v.x = new_row_elem(o, key, 4 * ch + 0, dim);
      v.y = new_row_elem(o, key, 4 * ch + 1, dim);
      v.z = new_row_elem(o, key, 4 * ch + 2, dim);
      v.w = new_row_elem(o, key, 4 * ch + 3, dim);
      if (write_row && ch < rchunks) *reinterpret_cast<float4*>(row + 4 * ch) = v;
      if (ch < uchunks) {
        // pulled row = w[dim] (+ two zero CVM columns for a new row), zero padding
        float4 u;
        u.x = 4 * ch + 0 < dim ? v.x : 0.f;
        u.y = 4 * ch + 1 < dim ? v.y : 0.f;
        u.z = 4 * ch + 2 < dim ? v.z : 0.f;
        u.w = 4 * ch + 3 < dim ? v.w : 0.f;
        *reinterpret_cast<float4*>(dst + 4 * ch) = u;
      }
    }
    return;
  }
  float show = 0.f, click = 0.f;
  if (t.use_cvm && o.kind == kAdaGrad) { show = row[dim + 1]; click = row[dim + 2]; }
  // up to four 16-byte loads in flight per lane (G >= ceil(uchunks / 4)), then the stores
  float4 buf[4];
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    const int ch = gl + k * G;
    if (ch < uchunks) buf[k] = *reinterpret_cast<const float4*>(row + 4 * ch);   // stride >= ustride by layout
  }
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    const int ch = gl + k * G;
    if (ch >= uchunks) continue;
    float4 v = buf[k];
    if (4 * ch + 4 > dim) {
      float e[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
      for (int kk = 0; kk < 4; ++kk) {
        int idx = 4 * ch + kk;
        if (idx >= dim) {
          float x = 0.f;
          if (t.use_cvm && o.kind == kAdaGrad) {
            if (idx == dim) x = show;
            else if (idx == dim + 1) x = logf(click + 1.f) - logf(show + 1.f);
          }
          e[kk] = x;
        }
      }
      v = make_float4(e[0], e[1], e[2], e[3]);
    }
    *reinterpret_cast<float4*>(dst + 4 * ch) = v;
  }
}

}  // namespace

// =======================================================================================
// sparse_pull_fused
// =======================================================================================
// kTiled: the staged row return (PullArgs::tile_rows > 0); one instantiation per form keeps the other form's code and
// registers out of the loop.
template <bool kTiled>
__global__ void __launch_bounds__(kThreads, 1) sparse_pull_fused_kernel(const __grid_constant__ PullArgs a) {
  const SparseCommView& c = a.c;
  // The table's arrays are read through a descriptor in device memory when the caller has one: the shard can then
  // grow (new key array, longer row slab) between two launches of an already captured CUDA graph.
  __shared__ TableView s_tbl;
  if (threadIdx.x == 0) s_tbl = a.tbl_dev != nullptr ? *a.tbl_dev : a.tbl;
  __syncthreads();
  const TableView& t = s_tbl;
  GridSync gs;
  gs.init(c.bar, c.status, c.wait_ns);
  __shared__ unsigned long long s_flag;
  __shared__ int s_n[kMaxWorld];
  __shared__ int s_pre[kMaxWorld + 1];

  const int tid = blockIdx.x * blockDim.x + threadIdx.x;
  const int nth = gridDim.x * blockDim.x;
  const int lane = threadIdx.x & 31;
  const int W = c.world, R = c.rank, capo = c.capo;
  const int n_ids = batch_ids(a);
  const unsigned long long epoch = __ldcg(c.epoch) + 1ull;
  const int dim = t.dim;
  const bool need_ou = a.training && W > 1;

  const bool front_done = a.front_done != 0;     // dedup, id dispatch and inverse map already ran (pull_front_*)
  if (tid == 0 && !front_done) *c.ocount = 0;    // (with the front ahead, the push of the previous step re-armed it)
  prof_mark(c, 0);

  if (front_done) {
    // show / click counts of the batch into the gradient records (the front runs while the previous step's records
    // are still in use, so it leaves them alone)
    if (a.training) count_shows(a, n_ids, tid, nth);
    prof_mark(c, 1);
    prof_mark(c, 2);
  } else {
  // ---- phase A: dedup; first occurrence of a sign allocates a slot in its owner's segment --------
  dedup_assign<false>(a, t, n_ids, tid, nth);
  if (!gs.sync(1, false)) goto done;
  prof_mark(c, 1);

  // ---- phase A2: ship id segments to the owners (first, so that the link latency and the owners' wait overlap
  // the rest of this phase), then inverse map and show/click counts ---------------------------------------
  if (W > 1) {
    // coalesced 16-byte peer stores of each owner's id segment
    for (int p = 0; p < W; ++p) {
      if (p == R) continue;
      int n = __ldcg(&c.cnt[p]);
      if (n > capo) n = capo;
      const ulonglong2* src = reinterpret_cast<const ulonglong2*>(c.stage_ids + (size_t)p * capo);
      ulonglong2* dst = reinterpret_cast<ulonglong2*>(c.inbox_ids[p] + (size_t)R * capo);
      int n2 = (n + 1) >> 1;
      for (int j = tid; j < n2; j += nth) dst[j] = __ldcg(&src[j]);
    }
    // no grid barrier: the CTA that finishes shipping last tells the owners their segments are complete, while
    // the others already probe the local segment (which only needs phase A, and that is behind barrier 1)
    if (last_cta_arrives(&c.bar[2], true) && threadIdx.x < W && threadIdx.x != R) {
      int p = threadIdx.x;
      int n = min(__ldcg(&c.cnt[p]), capo);
      st_release_sys_u64(sig_word(c.sig[p], kSigPullReq, R), (epoch << 32) | (unsigned long long)n);
    }
  }
  dedup_resolve(a, n_ids, tid, nth, a.training != 0);
  gs.arrive();       // this CTA no longer reads the dedup scratch; phase C waits for all of them before clearing it
  prof_mark(c, 2);
  }

  // ---- phase B: as owner, probe / insert every requested sign and return its row ----------------------
  // A warp takes 32 requests at a time: every lane probes (or inserts) one sign, then the warp's lane groups
  // return the 32 rows.  No grid barrier separates probing from the row return, so the row stores of one warp
  // cross NVLink while other warps still wait on their probes.  Two passes: this GPU's own segment first
  // (nothing to wait for), then the segments of all other senders as ONE flat space of units, so that with many
  // GPUs no warp idles on a short per-sender segment.  A unit is one shared-memory tile of the staged return
  // (tile_rows consecutive requests of one sender) or, without staging, a single request.
  // s_pre[k] = units of the senders that precede the k-th sender of the pass.
  {
    const int G = a.lanes;
    const int gl = threadIdx.x % G, sub = lane / G, rpp = 32 / G;
    const int ustride = c.ustride, uchunks = ustride >> 2;
    const int TR = kTiled ? a.tile_rows : 0;
    const int urows = kTiled ? TR : 1;
    const int upw = 32 / urows;                        // units per warp step
    extern __shared__ float4 s_tiles[];
    float* tile = reinterpret_cast<float*>(s_tiles) + (size_t)(threadIdx.x >> 5) * TR * ustride;
    const int n_warps = nth >> 5;
    for (int part = 0; part < (W > 1 ? 2 : 1); ++part) {
      __syncthreads();
      if (part == 0 && threadIdx.x == 0) {
        const int v = min(__ldcg(&c.cnt[R]), capo);
        s_n[R] = v;
        if (blockIdx.x == 0) c.req_n[R] = v;
        s_pre[0] = 0;
        s_pre[1] = (v + urows - 1) / urows;
        s_flag = (unsigned long long)s_pre[1];
      }
      if (part == 1 && threadIdx.x < 32) {
        // one lane per sender: the W-1 flags are polled side by side, the counts they carry are turned into the
        // flat unit space with a warp scan
        const int k = threadIdx.x;
        const int sk = (R + 1 + k) % W;
        unsigned long long f = 0;
        bool ok = true;
        if (k + 1 < W) ok = wait_flag_ge(sig_word(c.sig[R], kSigPullReq, sk), epoch, &f, c.wait_ns, c.status, 3, sk);
        const bool all_ok = __all_sync(0xffffffffu, ok);
        const int n_k = (k + 1 < W && all_ok) ? (int)(f & 0xffffffffull) : 0;
        int incl = (n_k + urows - 1) / urows;
#pragma unroll
        for (int o = 1; o < kMaxWorld; o <<= 1) {
          const int up = __shfl_up_sync(0xffffffffu, incl, o);
          if (k >= o) incl += up;
        }
        if (k + 1 < W) {
          s_n[sk] = n_k;
          if (blockIdx.x == 0) c.req_n[sk] = n_k;
          s_pre[k + 1] = incl;
        }
        if (k == 0) s_pre[0] = 0;
        const int total = __shfl_sync(0xffffffffu, incl, W - 2);
        if (k == 0) s_flag = all_ok ? (unsigned long long)total : ~0ull;
      }
      __syncthreads();
      if (s_flag == ~0ull) { gs.failed = true; break; }
      const int n_units = (int)(s_flag & 0xffffffffull);
      const int first = part == 0 ? R : R + 1;
      // units per warp step: all 32 lanes probe when there is enough work for every warp, fewer when a small batch
      // would otherwise leave most warps idle while a few return 32 rows one after the other
      int su = min(upw, (n_units + n_warps - 1) / n_warps);
      if (!kTiled) su = min(32, (su + rpp - 1) / rpp * rpp);
      if (su < 1) su = 1;
      for (int wu = (tid >> 5) * su; wu < n_units; wu += n_warps * su) {
        // -- probe: one request per lane
        const int lu = lane / urows;
        const int u = wu + lu;
        int s = R, j = 0;
        bool valid = false;
        if (lu < su && u < n_units) {
          int k = 0;
          while (u >= s_pre[k + 1]) ++k;
          s = (first + k) % W;
          j = (u - s_pre[k]) * urows + lane % urows;
          valid = j < s_n[s];
        }
        const unsigned long long* src = (s == R) ? c.stage_ids + (size_t)R * capo : c.inbox_ids[R] + (size_t)s * capo;
        int rr = kReqNone, ou = -1;
        bool is_new = false, need_claim = false;
        unsigned hnew = 0;
        int r_exist = -1;
        unsigned long long tag_seen = 0, key = 0;
        if (valid) {
          key = __ldcg(&src[j]);
          unsigned h = table_home(t, key);
          bool placed = false;
          for (unsigned probes = 0; probes <= t.cap_mask; ++probes) {
            // the row index is fetched beside the key: two misses in a multi-gigabyte table overlap instead of adding up
            unsigned long long k = __ldcg(&t.keys[h]);
            const int r = ld_volatile_s32(&t.slots[h]);
            if (k == kEmptyKey) {
              if (a.lookup_only) { placed = true; break; }        // read-only table (serving): an unknown sign pulls zeros
              k = atomicCAS(&t.keys[h], kEmptyKey, key);
              if (k == kEmptyKey) { is_new = true; hnew = h; placed = true; break; }
            }
            if (k == key) {
              if (r == -1) {          // no row published (when we looked): resolved below, after this warp's own inserts
                rr = kReqPending;
                ou = (int)h;
              } else if (r >= 0) {
                rr = r;
                if (W > 1) {
                  const unsigned long long tg = *((volatile unsigned long long*)&t.row_tag[r]);
                  if ((tg >> 32) == epoch) {
                    if (tg & kTagNew) rr = r | kReqNewCopy;
                    if (need_ou) ou = (int)(tg & 0x7fffffffull);
                  } else if (need_ou) {
                    need_claim = true; r_exist = r; tag_seen = tg;
                  }
                }
              }
              placed = true;
              break;
            }
            h = (h + 1) & t.cap_mask;
          }
          if (!placed) set_status(c.status, kTableFull, 3, s);
        }
        __syncwarp();
        const unsigned nm = __ballot_sync(0xffffffffu, is_new);
        const unsigned cm = __ballot_sync(0xffffffffu, need_claim);
        const int r_new = warp_alloc(t.n_rows, nm);
        int my_ou = -1;
        if (need_ou) my_ou = warp_alloc(c.ocount, nm | cm);
        if (is_new) {
          if (r_new >= t.row_cap) {
            atomicSub(t.n_rows, 1);
            set_status(c.status, kTableFull, 3, s);
            *((volatile int*)&t.slots[hnew]) = -3;
            if (need_ou) c.ou_row[my_ou] = -1;
          } else {
            t.row_keys[r_new] = key;
            unsigned long long tag = (epoch << 32) | kTagNew;
            if (need_ou) { c.ou_row[my_ou] = r_new; tag |= (unsigned long long)my_ou; ou = my_ou; }
            t.row_tag[r_new] = tag;
            __threadfence();
            *((volatile int*)&t.slots[hnew]) = r_new;
            rr = r_new | kReqNewOwner;
          }
        } else if (need_claim) {
          const unsigned long long old = atomicCAS(&t.row_tag[r_exist], tag_seen, (epoch << 32) | (unsigned long long)my_ou);
          if (old == tag_seen) {
            c.ou_row[my_ou] = r_exist;
            ou = my_ou;
          } else {                     // another sender claimed the row first: my index stays a hole
            c.ou_row[my_ou] = -1;
            ou = (int)(old & 0x7fffffffull);
          }
        }
        __syncwarp();
        if (rr == kReqPending) {
          // Another thread won the insert of this sign in this very step and publishes the row index a few
          // instructions after its CAS (a lane of this warp has done so above); wait for it, with a limit.
          const int h = ou;
          int r = ld_volatile_s32(&t.slots[h]);
          const unsigned long long t0 = globaltimer_ns();
          while (r == -1) {
            if (globaltimer_ns() - t0 > c.wait_ns) { set_status(c.status, kGridBarrierTimeout, 4, s); break; }
            r = ld_volatile_s32(&t.slots[h]);
          }
          __threadfence();
          rr = kReqNone;
          ou = -1;
          if (r >= 0) {
            const unsigned long long tg = *((volatile unsigned long long*)&t.row_tag[r]);
            const bool fresh = (tg >> 32) == epoch && (tg & kTagNew);
            rr = fresh ? (r | kReqNewCopy) : r;
            if (need_ou) ou = (int)(tg & 0x7fffffffull);
          }
        }
        if (valid) {
          const int q = s * capo + j;
          c.req_row[q] = rr;
          c.req_ou[q] = ou;
        }
        __syncwarp();
        // -- return: groups of G lanes take the warp's rows in turn
        const unsigned vmask = __ballot_sync(0xffffffffu, valid);
        if (kTiled) {
          // Staged return: the warp gathers the rows of a tile into shared memory and then writes the tile out as
          // one contiguous run of full 128-byte lines (16 bytes per lane, 512 per instruction).  Row-by-row stores
          // of short rows (80 bytes for dim 16 + linear) reach a peer as partial lines and lose about a third of
          // the NVLink write rate; the local case gains too.
          for (int ti = 0; ti < su; ++ti) {
            const unsigned tmask = (vmask >> (ti * TR)) & (TR >= 32 ? 0xffffffffu : ((1u << TR) - 1u));
            if (tmask == 0) continue;
            const int nrows = __popc(tmask);            // the valid requests of a tile are its first ones
            const int s_t = __shfl_sync(0xffffffffu, s, ti * TR), j0 = __shfl_sync(0xffffffffu, j, ti * TR);
            for (int p0 = 0; p0 < TR; p0 += rpp) {
              const int jr = p0 + sub;
              const int from = (ti * TR + jr) & 31;
              const int rr_s = __shfl_sync(0xffffffffu, rr, from);
              const unsigned long long key_s = __shfl_sync(0xffffffffu, key, from);
              if (jr < nrows) pull_return_row(a, t, rr_s, key_s, tile + (size_t)jr * ustride, gl, G);
            }
            __syncwarp();
            float4* d4 = reinterpret_cast<float4*>(c.U[s_t] + ((size_t)R * capo + j0) * ustride);
            const float4* t4 = reinterpret_cast<const float4*>(tile);
            const int n4 = nrows * uchunks;
            for (int i = lane; i < n4; i += 32) d4[i] = t4[i];
            __syncwarp();
          }
        } else {
          for (int p0 = 0; p0 < su; p0 += rpp) {
            const int from = p0 + sub;
            const int rr_s = __shfl_sync(0xffffffffu, rr, from);
            const unsigned long long key_s = __shfl_sync(0xffffffffu, key, from);
            const int s_s = __shfl_sync(0xffffffffu, s, from), j_s = __shfl_sync(0xffffffffu, j, from);
            if ((vmask >> from) & 1u)
              pull_return_row(a, t, rr_s, key_s, c.U[s_s] + ((size_t)R * capo + j_s) * ustride, gl, G);
          }
        }
      }
      if (part == 0) prof_mark(c, 3);
    }
  }
  if (gs.failed) goto done;
  if (c.prof != nullptr && threadIdx.x == 0) atomicMax(&c.prof[6], globaltimer_ns());   // slowest CTA's end of the row return
  prof_mark(c, 4);

  // ---- phase C: tell the requesters their rows have landed; clear the dedup scratch while the flags travel -----
  {
    // The CTA that returns its rows last saves the per-owner counts of this step for pooling / push and re-arms
    // them, and tells every requester that its matrix is complete; CTA 0 then keeps the kernel alive until the
    // same word has arrived from every owner.
    const bool last = last_cta_arrives(&c.bar[3], W > 1);
    if (last && threadIdx.x < W) {
      c.cnt_saved[threadIdx.x] = min(c.cnt[threadIdx.x], capo);
      c.cnt[threadIdx.x] = 0;
      if (threadIdx.x != R) st_release_sys_u64(sig_word(c.sig[threadIdx.x], kSigPullDone, R), epoch << 32);
    }
    if (!front_done) {
      if (!gs.wait(4)) goto done;      // every CTA has finished its inverse map (it arrived before phase B)
      ulonglong2* kk = reinterpret_cast<ulonglong2*>(c.dd_keys);
      const int n2 = (int)((c.dd_mask + 1u) >> 1);
      for (int i = tid; i < n2; i += nth) kk[i] = make_ulonglong2(kEmptyKey, kEmptyKey);
    }
    if (W > 1 && blockIdx.x == 0 && threadIdx.x < W && threadIdx.x != R) {
      unsigned long long v;
      wait_flag_ge(sig_word(c.sig[R], kSigPullDone, threadIdx.x), epoch, &v, c.wait_ns, c.status, 6, threadIdx.x);
    }
    __syncthreads();
  }
  if (tid == 0) *c.epoch = epoch;
  prof_mark(c, 5);

done:
  gs.leave();
}

// =======================================================================================
// pull front: phases A and A2 of the pull (without the show / click counts) as two ordinary kernels.  They need
// only the ids of a batch, so they can run on a second stream while the previous step's forward and backward
// passes run; their CTAs are small and fit beside the GEMM CTAs.  `c.bar[4]` counts the CTAs of the second kernel
// (the cooperative kernels of the same link use bar[0..3] and may run at the same time).
// =======================================================================================
constexpr int kFrontThreads = 256;

__global__ void __launch_bounds__(kFrontThreads) pull_front_dedup_kernel(const __grid_constant__ PullArgs a) {
  const SparseCommView& c = a.c;
  // one read per CTA: all its threads take the same way out (a CTA barrier follows in the shipping kernel)
  __shared__ int s_bad;
  if (threadIdx.x == 0) s_bad = ld_volatile_s32(c.status);
  __syncthreads();
  if (s_bad != 0) return;
  const int tid = blockIdx.x * blockDim.x + threadIdx.x;
  const int nth = gridDim.x * blockDim.x;
  const int n_ids = a.n_ids;
  if (c.prof != nullptr && tid == 0) c.prof[16] = globaltimer_ns();
  dedup_assign<false>(a, a.tbl, n_ids, tid, nth);
  if (c.prof != nullptr && threadIdx.x == 0) atomicMax(&c.prof[17], globaltimer_ns());      // last CTA's end
}

__global__ void __launch_bounds__(kFrontThreads) pull_front_ship_kernel(const __grid_constant__ PullArgs a) {
  const SparseCommView& c = a.c;
  // one read per CTA: all its threads take the same way out (a CTA barrier follows in the shipping kernel)
  __shared__ int s_bad;
  if (threadIdx.x == 0) s_bad = ld_volatile_s32(c.status);
  __syncthreads();
  if (s_bad != 0) return;
  const int tid = blockIdx.x * blockDim.x + threadIdx.x;
  const int nth = gridDim.x * blockDim.x;
  const int W = c.world, R = c.rank, capo = c.capo;
  const int n_ids = a.n_ids;
  const unsigned long long epoch = __ldcg(c.epoch) + 1ull;
  if (W > 1) {
    for (int p = 0; p < W; ++p) {
      if (p == R) continue;
      int n = __ldcg(&c.cnt[p]);
      if (n > capo) n = capo;
      const ulonglong2* src = reinterpret_cast<const ulonglong2*>(c.stage_ids + (size_t)p * capo);
      ulonglong2* dst = reinterpret_cast<ulonglong2*>(c.inbox_ids[p] + (size_t)R * capo);
      const int n2 = (n + 1) >> 1;
      for (int j = tid; j < n2; j += nth) dst[j] = __ldcg(&src[j]);
    }
    // the CTA that finishes shipping last tells the owners their segments are complete and re-arms the counter
    if (last_cta_arrives(&c.bar[4], true)) {
      if (threadIdx.x < W && threadIdx.x != R) {
        const int p = threadIdx.x;
        const int n = min(__ldcg(&c.cnt[p]), capo);
        st_release_sys_u64(sig_word(c.sig[p], kSigPullReq, R), (epoch << 32) | (unsigned long long)n);
      }
      if (threadIdx.x == 0) c.bar[4] = 0;
    }
  }
  dedup_resolve(a, n_ids, tid, nth, false);
  if (c.prof != nullptr && threadIdx.x == 0) atomicMax(&c.prof[18], globaltimer_ns());      // last CTA's end
}

// =======================================================================================
// One GPU: nothing is exchanged, so a pull is two ordinary kernels and leaves the rows where they are.  The first one
// deduplicates the batch and looks every distinct sign up; the second one turns dedup slots into positions, counts shows
// and clicks, gives signs that have no row yet their row and puts the scratch back.  Pooling then reads the table's rows
// through req_row (RowSource), so no row is copied into a per-batch matrix and read from there again.  As one
// cooperative kernel that writes the rows out, a pull cost a grid barrier per phase and the copy.  Bound by the latency of
// dependent accesses, for large batches by random sectors.  Pull (and pooling) before and now, us: 10 K ids 33 (2.4) and
// 8.0 + 4.7 (3.0); 64 K ids 31 (3.4) and 8.5 + 5.7 (3.7); 213 K ids 51 (9) and 24 + 6 (11); 2.1 M ids with rows of 128
// floats 420 (312) and 121 + 40 (329).
// The price is paid by signs without a row, whose key and slot sectors are asked for twice, by the lookup and by the
// insertion: 4.2 M new signs 2 280 us then and 560 + 1 840 now (Ftrl, dim 64), 1 190 and 570 + 770 (Adam, 20), 790 and 455 +
// 490 (AdaGrad, 8).  What did not help: several insertions in flight per lane (490 -> 550), the arithmetic of the initial
// values spread evenly over the lanes, rows cleared as one run before their weights are written.
// Ahead of its step (pull_local_probe_kernel, pull_local_resolve_kernel on a second stream) the table's index is only
// read; what the step itself still runs is the second kernel without its first part.
// =======================================================================================
constexpr int kLocalThreads = 256;

// Both kernels take the pulls of two tables at once (blockIdx.y): a model's pulls need only the ids of the batch, and a small
// one is all latency.  Two of 10 K ids, one after the other and together: 26 and 14 us.
// (Launches of one table carry one table's arguments: a parameter block of 3 KB costs the host more than a microsecond.)
template <int N> struct PullArgsOf { PullArgs a[N]; };
template <int N>
__global__ void __launch_bounds__(kLocalThreads, 4) pull_local_probe_kernel(const __grid_constant__ PullArgsOf<N> batch) {
  const PullArgs& a = batch.a[N == 1 ? 0 : blockIdx.y];
  const TableView t = *a.tbl_dev;         // (changes between steps only: safe to read before the kernel ahead has finished)
  pdl_sync();
  const SparseCommView& c = a.c;
  const int tid = blockIdx.x * blockDim.x + threadIdx.x, nth = gridDim.x * blockDim.x;
  const int n_ids = batch_ids(a);
  if (c.prof != nullptr && tid == 0) c.prof[a.front_done ? 16 : 0] = globaltimer_ns();
  if (ld_volatile_s32(c.status) != 0) {   // an earlier error has not been dealt with: no id has a row
    if (threadIdx.x == 0) c.bar[kLocalSkip] = 1;
    for (int i = tid; i < n_ids; i += nth) a.inverse[i] = -1;
    return;
  }
  dedup_assign<true>(a, t, n_ids, tid, nth);
  if (c.prof != nullptr && threadIdx.x == 0) atomicMax(&c.prof[a.front_done ? 17 : 1], globaltimer_ns());      // last CTA's end
}

__device__ __forceinline__ void clear_dedup_keys(const SparseCommView& c, int tid, int nth) {
  ulonglong2* kk = reinterpret_cast<ulonglong2*>(c.dd_keys);
  const int n2 = (int)((c.dd_mask + 1u) >> 1);
  for (int i = tid; i < n2; i += nth) kk[i] = make_ulonglong2(kEmptyKey, kEmptyKey);
}

// Second half of a front: positions, and the dedup keys (which only the first kernel reads) back to empty.
__global__ void __launch_bounds__(kLocalThreads) pull_local_resolve_kernel(const __grid_constant__ PullArgs a) {
  pdl_sync();
  const int tid = blockIdx.x * blockDim.x + threadIdx.x, nth = gridDim.x * blockDim.x;
  dedup_resolve(a, batch_ids(a), tid, nth, false);
  clear_dedup_keys(a.c, tid, nth);
  if (a.c.prof != nullptr && threadIdx.x == 0) atomicMax(&a.c.prof[18], globaltimer_ns());
}

// ---- One GPU, nobody asks for gradients (scoring, evaluation): the row of every id, straight from the table's index ------------
// No dedup: nothing is summed per sign, and the second occurrence of a sign finds its sectors in L2.  A chain is then home slot
// (key and row number together), with a quarter of the ids one slot more, instead of dedup slot, home slot, position, row
// number.  Signs without a row are marked and counted; two more kernels give them one (whoever places the key creates
// the row) and look them up again, and have nothing to do where there are none.
// 213 K ids, 20 M rows: 14.1 us and 2 + 1.5 for the other two, where the pull takes 22.3 + 5.9 (and the gather behind it 1 us more,
// for the positions).  Four slots of the index at a time (a sector of keys, sixteen bytes of rows): 16.7.
constexpr int kLookupMissing = 6, kLookupLeft = 7;      // words of `bar`: ids without a row; blocks that are through with them
constexpr int kNoRowYet = -2;                           // in a.inverse, until the last kernel has run

__device__ __forceinline__ void write_new_row(const PullArgs& a, const TableView& t, int r, unsigned long long key, int first, int step) {
  float* row = t.rows + (size_t)r * t.stride;
  for (int ch = first; ch < (t.stride >> 2); ch += step)
    *reinterpret_cast<float4*>(row + 4 * ch) = make_float4(new_row_elem(a.opt, key, 4 * ch, t.dim), new_row_elem(a.opt, key, 4 * ch + 1, t.dim),
                                                           new_row_elem(a.opt, key, 4 * ch + 2, t.dim), new_row_elem(a.opt, key, 4 * ch + 3, t.dim));
}
// The row of a new key that this lane may have to create, for all lanes of a warp; lanes without `want` only help.  The key is
// placed with one compare-and-swap, the rows of the warp's winners come from one addition to the row counter and are written by
// its groups of G lanes.  Returns the row, or kReqNone when somebody else is placing the key or the table is full.
__device__ __forceinline__ int insert_new(const PullArgs& a, const TableView& t, bool want, unsigned long long key) {
  const SparseCommView& c = a.c;
  const int lane = threadIdx.x & 31;
  int r = kReqNone;
  unsigned h = 0;
  bool is_new = false;
  if (want) {
    bool placed = false;
    h = table_home(t, key);
    for (unsigned probes = 0; probes <= t.cap_mask; ++probes) {
      unsigned long long k = __ldcg(&t.keys[h]);
      if (k == kEmptyKey) {
        k = atomicCAS(&t.keys[h], kEmptyKey, key);
        if (k == kEmptyKey) { is_new = placed = true; break; }
      }
      if (k == key) { r = ld_volatile_s32(&t.slots[h]); placed = true; break; }     // inserted since it was looked up
      h = (h + 1) & t.cap_mask;
    }
    if (!placed) set_status(c.status, kTableFull, 3, 0);
  }
  __syncwarp();
  const int r_new = warp_alloc(t.n_rows, __ballot_sync(0xffffffffu, is_new));
  if (is_new) {
    if (r_new >= t.row_cap) {
      atomicSub(t.n_rows, 1);
      set_status(c.status, kTableFull, 3, 0);
      t.slots[h] = -3;
      is_new = false;
    } else {
      t.row_keys[r_new] = key;
      t.slots[h] = r_new;
      r = r_new;
    }
  }
  const int G = a.lanes, gl = threadIdx.x % G, sub = lane / G, rpp = 32 / G;
  unsigned left = __ballot_sync(0xffffffffu, is_new);
  while (left != 0) {                  // the warp's groups write one new row each
    unsigned rest = left;
    for (int k = 0; k < sub; ++k) rest &= rest - 1;
    const int from = rest != 0 ? __ffs(rest) - 1 : 0;
    const int r_s = __shfl_sync(0xffffffffu, r, from);
    const unsigned long long key_s = __shfl_sync(0xffffffffu, key, from);
    if (rest != 0) write_new_row(a, t, r_s, key_s, gl, G);
    for (int k = 0; k < rpp; ++k) left &= left - 1;
  }
  return r >= 0 ? r : kReqNone;
}

template <int N>
__global__ void __launch_bounds__(kLocalThreads, 4) pull_local_finish_kernel(const __grid_constant__ PullArgsOf<N> batch) {
  const PullArgs& a = batch.a[N == 1 ? 0 : blockIdx.y];
  const TableView t = *a.tbl_dev;
  pdl_sync();
  const SparseCommView& c = a.c;
  __shared__ int s_bad, s_new;
  const int tid = blockIdx.x * blockDim.x + threadIdx.x, nth = gridDim.x * blockDim.x;
  const int lane = threadIdx.x & 31;
  if (a.front_done) { prof_mark(c, 0); prof_mark(c, 1); }
  prof_mark(c, 2);
  if (threadIdx.x == 0) {
    s_bad = (int)__ldcg(&c.bar[kLocalSkip]);
    s_new = __ldcg(c.ocount);
  }
  __syncthreads();
  const bool bad = s_bad != 0;
  const int n_new = s_new;
  if (threadIdx.x == 0) {
    // the CTA that is the last to have read the counters leaves them ready for the next pull: no tail at the end
    __threadfence();
    if (atomicAdd(&c.bar[3], 1u) == gridDim.x - 1) {
      c.cnt_saved[0] = bad ? 0 : min(__ldcg(&c.cnt[0]), c.capo);
      c.cnt[0] = 0;
      *c.ocount = 0;
      c.bar[3] = 0;
      c.bar[kLocalSkip] = 0;
      *c.epoch = __ldcg(c.epoch) + 1ull;
    }
  }
  if (!bad) {
    const int n_ids = batch_ids(a);
    if (!a.front_done) {
      dedup_resolve(a, n_ids, tid, nth, a.training != 0);
      clear_dedup_keys(c, tid, nth);
    } else if (a.training) {
      count_shows(a, n_ids, tid, nth);
    }
    // new rows, 32 to a warp: the keys are distinct and nobody else inserts, so a lane never meets its own key half done
    for (int base = tid - lane; base < n_new; base += nth) {
      const int m = base + lane, pos = m < n_new ? __ldcg(&c.req_ou[m]) : -1;
      const int r = insert_new(a, t, pos >= 0, pos >= 0 ? __ldcg(&c.stage_ids[pos]) : kEmptyKey);
      if (pos >= 0) c.req_row[pos] = r;
    }
  }
  if (c.prof != nullptr && threadIdx.x == 0) {
    const unsigned long long now = globaltimer_ns();
    atomicMax(&c.prof[3], now); atomicMax(&c.prof[4], now); atomicMax(&c.prof[5], now);
  }
}

template <int N>
__global__ void __launch_bounds__(kLocalThreads, 8) lookup_rows_kernel(const __grid_constant__ PullArgsOf<N> batch) {
  const PullArgs& a = batch.a[N == 1 ? 0 : blockIdx.y];
  const TableView t = *a.tbl_dev;         // (as in pull_local_probe_kernel)
  pdl_sync();
  const SparseCommView& c = a.c;
  const int tid = blockIdx.x * blockDim.x + threadIdx.x, nth = gridDim.x * blockDim.x, lane = threadIdx.x & 31;
  const int n_ids = batch_ids(a);
  const bool bad = ld_volatile_s32(c.status) != 0;      // an earlier error has not been dealt with: no id has a row
  for (int base = tid - lane; base < n_ids; base += nth) {
    const int i = base + lane;
    int r = kReqNone;
    bool missing = false;
    if (i < n_ids && !bad) {
      const unsigned long long key = canon_key((unsigned long long)a.ids[i]);
      unsigned h = table_home(t, key);
      for (unsigned probes = 0; probes <= t.cap_mask; ++probes) {
        const unsigned long long k = __ldcg(&t.keys[h]);
        const int row = __ldcg(&t.slots[h]);
        if (k == key) { r = row >= 0 ? row : kReqNone; break; }
        if (k == kEmptyKey) { missing = !a.lookup_only; break; }
        h = (h + 1) & t.cap_mask;
      }
    }
    const unsigned mm = __ballot_sync(0xffffffffu, missing);
    if (i < n_ids) a.inverse[i] = missing ? kNoRowYet : r;
    if (mm != 0 && lane == 0) atomicAdd(&c.bar[kLookupMissing], (unsigned)__popc(mm));
  }
}
template <int N>
__global__ void __launch_bounds__(kLocalThreads, 4) lookup_insert_kernel(const __grid_constant__ PullArgsOf<N> batch) {
  const PullArgs& a = batch.a[N == 1 ? 0 : blockIdx.y];
  const TableView t = *a.tbl_dev;
  pdl_sync();
  if (__ldcg(&a.c.bar[kLookupMissing]) == 0) return;
  const int tid = blockIdx.x * blockDim.x + threadIdx.x, nth = gridDim.x * blockDim.x, lane = threadIdx.x & 31;
  const int n_ids = batch_ids(a);
  for (int base = tid - lane; base < n_ids; base += nth) {
    const int i = base + lane;
    const bool want = i < n_ids && a.inverse[i] == kNoRowYet;
    const unsigned long long key = want ? canon_key((unsigned long long)a.ids[i]) : kEmptyKey;
    const unsigned same = __match_any_sync(0xffffffffu, key);            // (every lane of the warp takes part)
    if (__ballot_sync(0xffffffffu, want) != 0) insert_new(a, t, want && __ffs(same) - 1 == lane, key);
  }
}
// (whose rows are all there now, but for those the table had no room for)
template <int N>
__global__ void __launch_bounds__(kLocalThreads, 8) lookup_again_kernel(const __grid_constant__ PullArgsOf<N> batch) {
  const PullArgs& a = batch.a[N == 1 ? 0 : blockIdx.y];
  const TableView t = *a.tbl_dev;
  pdl_sync();
  unsigned* bar = a.c.bar;
  __shared__ int s_any;
  if (threadIdx.x == 0) s_any = (int)__ldcg(&bar[kLookupMissing]);
  __syncthreads();
  if (s_any == 0) return;
  if (threadIdx.x == 0) {              // the block that is the last to have read the count clears it
    __threadfence();
    if (atomicAdd(&bar[kLookupLeft], 1u) == gridDim.x - 1) { bar[kLookupMissing] = 0; bar[kLookupLeft] = 0; }
  }
  const int n_ids = batch_ids(a);
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n_ids; i += gridDim.x * blockDim.x) {
    if (a.inverse[i] != kNoRowYet) continue;
    const int r = table_find(t, canon_key((unsigned long long)a.ids[i]));
    a.inverse[i] = r >= 0 ? r : kReqNone;
  }
}

// The rows of the distinct signs of the last pull into the per-batch matrix, for callers that ask for it.
__global__ void __launch_bounds__(kLocalThreads) pull_local_rows_kernel(const __grid_constant__ PullArgs a) {
  pdl_sync();
  const SparseCommView& c = a.c;
  __shared__ TableView s_tbl;
  if (threadIdx.x == 0) s_tbl = *a.tbl_dev;
  __syncthreads();
  const int G = a.lanes, gl = threadIdx.x % G;
  const int n = __ldcg(&c.cnt_saved[0]);
  for (int j = (blockIdx.x * blockDim.x + threadIdx.x) / G; j < n; j += gridDim.x * blockDim.x / G)
    pull_return_row(a, s_tbl, __ldcg(&c.req_row[j]), 0ull, c.U[0] + (size_t)j * c.ustride, gl, G);
}

// =======================================================================================
// sparse_push_fused
// =======================================================================================
namespace {

// The row updates run at 1024 threads per SM with a dozen memory operations per element group; IEEE division and
// square root (software sequences of 10-20 instructions each) then cost as much issue time as the memory
// round trips.  The approximate forms are good to 2 ulp, far inside the parity tolerance with the CPU restatement.
__device__ __forceinline__ float fast_sqrt(float x) {
  float y;
  asm("sqrt.approx.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
__device__ __forceinline__ float fast_div(float a, float b) { return __fdividef(a, b); }

// The element-wise optimizers on one 16-byte chunk of a row (w, two slots) and its gradient x.
__device__ __forceinline__ void adam_chunk(const SparseOptParams& o, const float4& x, float4& w, float4& mm, float4& vv) {
  const float c1 = 1.f - o.beta1, c2 = 1.f - o.beta2;
#define TN_SADAM(cmp) \
  mm.cmp = o.beta1 * mm.cmp + c1 * x.cmp; vv.cmp = o.beta2 * vv.cmp + c2 * x.cmp * x.cmp; \
  w.cmp -= fast_div(o.lr * mm.cmp, o.eps + fast_sqrt(vv.cmp));
  TN_SADAM(x) TN_SADAM(y) TN_SADAM(z) TN_SADAM(w)
#undef TN_SADAM
}
__device__ __forceinline__ void ftrl_chunk(const SparseOptParams& o, const float4& x, float4& w, float4& zz, float4& nn) {
#define TN_SFTRL(cmp) { \
  const float g2 = x.cmp * x.cmp; \
  const float sn = fast_sqrt(nn.cmp + g2); \
  zz.cmp += x.cmp - o.lr * (sn - fast_sqrt(nn.cmp)) * w.cmp; \
  nn.cmp += g2; \
  const float shr = zz.cmp > 0.f ? zz.cmp - o.lambda1 : zz.cmp + o.lambda1; \
  w.cmp = fabsf(zz.cmp) > o.lambda1 ? -fast_div(shr, (o.ftrl_beta + sn) * o.lr + o.lambda2) : 0.f; }
  TN_SFTRL(x) TN_SFTRL(y) TN_SFTRL(z) TN_SFTRL(w)
#undef TN_SFTRL
}

// One optimizer step on one row by a group of G lanes.  `g` points at the gradient (dim floats), bshow / bclick
// are the batch's show and click counts of the sign.   Math as in the reference's Sparse*Value::Apply.
// VEC: dim is a multiple of 4, every lane works on float4 chunks.
template <bool VEC>
__device__ __forceinline__ void apply_row(const SparseOptParams& o, float* row, const float* g, float bshow, float bclick,
                                          int dim, int lane, int G, unsigned gmask) {
  if (o.kind == kAdaGrad) {
    if (VEC && (dim >> 2) <= 2 * G) {
      // Every load of the row is issued before the first use, so a row costs one memory round trip instead of
      // three (gradient -> squared norm -> accumulator -> weights): up to two float4 chunks per lane.
      const int nch = dim >> 2;
      const int c0 = lane, c1 = lane + G;
      float4 x0 = make_float4(0.f, 0.f, 0.f, 0.f), x1 = x0, w0 = x0, w1 = x0;
      if (c0 < nch) { x0 = *reinterpret_cast<const float4*>(g + 4 * c0); w0 = *reinterpret_cast<const float4*>(row + 4 * c0); }
      if (c1 < nch) { x1 = *reinterpret_cast<const float4*>(g + 4 * c1); w1 = *reinterpret_cast<const float4*>(row + 4 * c1); }
      const float g2old = row[dim];
      float ss = x0.x * x0.x + x0.y * x0.y + x0.z * x0.z + x0.w * x0.w;
      ss += x1.x * x1.x + x1.y * x1.y + x1.z * x1.z + x1.w * x1.w;
      for (int off = G >> 1; off > 0; off >>= 1) ss += __shfl_xor_sync(gmask, ss, off);
      const float g2 = g2old + ss / (float)dim;
      const float scale = fast_div(o.lr, o.eps + fast_sqrt(g2));
      if (c0 < nch) {
        w0.x -= scale * x0.x; w0.y -= scale * x0.y; w0.z -= scale * x0.z; w0.w -= scale * x0.w;
        *reinterpret_cast<float4*>(row + 4 * c0) = w0;
      }
      if (c1 < nch) {
        w1.x -= scale * x1.x; w1.y -= scale * x1.y; w1.z -= scale * x1.z; w1.w -= scale * x1.w;
        *reinterpret_cast<float4*>(row + 4 * c1) = w1;
      }
      __syncwarp(gmask);
      if (lane == 0) {
        row[dim] = g2;
        row[dim + 1] += bshow;
        row[dim + 2] += bclick;
        reinterpret_cast<int*>(row)[dim + 3] = 0;
      }
      return;
    }
    float ss = 0.f;
    if (VEC) {
      for (int ch = lane; ch < (dim >> 2); ch += G) {
        const float4 x = *reinterpret_cast<const float4*>(g + 4 * ch);
        ss += x.x * x.x + x.y * x.y + x.z * x.z + x.w * x.w;
      }
    } else {
      for (int e = lane; e < dim; e += G) { float x = g[e]; ss += x * x; }
    }
    for (int off = G >> 1; off > 0; off >>= 1) ss += __shfl_xor_sync(gmask, ss, off);
    const float g2 = row[dim] + ss / (float)dim;
    const float scale = o.lr / (o.eps + sqrtf(g2));
    if (VEC) {
      for (int ch = lane; ch < (dim >> 2); ch += G) {
        const float4 x = *reinterpret_cast<const float4*>(g + 4 * ch);
        float4 w = *reinterpret_cast<float4*>(row + 4 * ch);
        w.x -= scale * x.x; w.y -= scale * x.y; w.z -= scale * x.z; w.w -= scale * x.w;
        *reinterpret_cast<float4*>(row + 4 * ch) = w;
      }
    } else {
      for (int e = lane; e < dim; e += G) row[e] -= scale * g[e];
    }
    __syncwarp(gmask);
    if (lane == 0) {
      row[dim] = g2;
      row[dim + 1] += bshow;
      row[dim + 2] += bclick;
      reinterpret_cast<int*>(row)[dim + 3] = 0;
    }
  } else if (o.kind == kAdam) {
    float* m = row + dim;
    float* v = row + 2 * dim;
    const float c1 = 1.f - o.beta1, c2 = 1.f - o.beta2;
    if (VEC) {
      for (int ch = lane; ch < (dim >> 2); ch += G) {
        const float4 x = *reinterpret_cast<const float4*>(g + 4 * ch);
        float4 mm = *reinterpret_cast<float4*>(m + 4 * ch), vv = *reinterpret_cast<float4*>(v + 4 * ch);
        float4 w = *reinterpret_cast<float4*>(row + 4 * ch);
        adam_chunk(o, x, w, mm, vv);
        *reinterpret_cast<float4*>(m + 4 * ch) = mm;
        *reinterpret_cast<float4*>(v + 4 * ch) = vv;
        *reinterpret_cast<float4*>(row + 4 * ch) = w;
      }
    } else {
      for (int e = lane; e < dim; e += G) {
        float x = g[e];
        float mm = o.beta1 * m[e] + c1 * x;
        float vv = o.beta2 * v[e] + c2 * x * x;
        m[e] = mm; v[e] = vv;
        row[e] -= o.lr * mm / (o.eps + sqrtf(vv));
      }
    }
    if (lane == 0) reinterpret_cast<int*>(row)[3 * dim + 1] += (int)bshow;
  } else {
    float* z = row + dim;
    float* n = row + 2 * dim;
    if (VEC) {
      // all four 16-byte loads of a chunk are issued before the arithmetic; approximate sqrt / division as in the
      // other two optimizers (three square roots and a division per element otherwise dominate the update)
      for (int ch = lane; ch < (dim >> 2); ch += G) {
        const float4 x = *reinterpret_cast<const float4*>(g + 4 * ch);
        float4 zz = *reinterpret_cast<float4*>(z + 4 * ch), nn = *reinterpret_cast<float4*>(n + 4 * ch);
        float4 w = *reinterpret_cast<float4*>(row + 4 * ch);
          ftrl_chunk(o, x, w, zz, nn);
        *reinterpret_cast<float4*>(z + 4 * ch) = zz;
        *reinterpret_cast<float4*>(n + 4 * ch) = nn;
        *reinterpret_cast<float4*>(row + 4 * ch) = w;
      }
    } else {
    for (int e = lane; e < dim; e += G) {
      float x = g[e], w = row[e], nn = n[e];
      float g2 = x * x;
      float zz = z[e] + x - o.lr * (sqrtf(nn + g2) - sqrtf(nn)) * w;
      nn += g2;
      float nw = 0.f;
      if (fabsf(zz) > o.lambda1) {
        nw = -1.f / ((o.ftrl_beta + sqrtf(nn)) * o.lr + o.lambda2);
        nw *= zz > 0.f ? zz - o.lambda1 : zz + o.lambda1;
      }
      z[e] = zz; n[e] = nn; row[e] = nw;
    }
    }
    if (lane == 0) reinterpret_cast<int*>(row)[3 * dim + 1] += (int)bshow;
  }
}

}  // namespace

// One GPU: every distinct sign of the batch maps to exactly one row, so there is nothing to exchange and nothing to wait
// for: an ordinary kernel updates the rows in place.  What bounds it is random access to gradient, row and optimizer slots:
// all loads of a row, its counters included, are issued before the first use (one chunk of 16 bytes per lane: dim a
// multiple of 4, at most 128), and the grid is one wave of resident blocks.  Rows in flight against blocks per SM, and
// whether the next round's rows are asked for from L2 meanwhile, were measured: 1.1 M AdaGrad rows of 128 take 515 us
// with one row, six blocks and prefetching (two rows, four blocks: 544 without, 570 with; four rows, two blocks: 682); 2.2 M
// Ftrl rows of 64, three times the bytes and registers, 930-980 us with two rows, three blocks and none (with: 1057; one
// row, six blocks: 1253).  As a branch of the cooperative kernel, one row per group after the other: 702 and 1371 us.
template <int KIND> struct LocalPush { static constexpr int kRows = 2, kBlocks = 3; static constexpr bool kPrefetch = false; };
template <> struct LocalPush<kAdaGrad> { static constexpr int kRows = 1, kBlocks = 6; static constexpr bool kPrefetch = true; };

template <int KIND>
__global__ void __launch_bounds__(256, LocalPush<KIND>::kBlocks) sparse_push_local_kernel(const __grid_constant__ PushArgs a) {
  constexpr int R = LocalPush<KIND>::kRows;
  pdl_sync();
  const SparseCommView& c = a.c;
  const SparseOptParams& o = a.opt;
  prof_mark(c, 8);
  __shared__ TableView s_tbl;
  if (threadIdx.x == 0) s_tbl = a.tbl_dev != nullptr ? *a.tbl_dev : a.tbl;
  __syncthreads();
  const TableView& t = s_tbl;
  const int n = __ldcg(&c.cnt_saved[0]);
  const int G = a.lanes, lane = threadIdx.x % G;
  const int gid = (blockIdx.x * blockDim.x + threadIdx.x) / G, ngroups = gridDim.x * blockDim.x / G;
  const unsigned gmask = group_mask(G);
  const int dim = t.dim, stride = t.stride, gstride = c.gstride;
  const bool has = 4 * lane < dim;                  // lanes of a group beyond the row only take part in the shuffles
  const float4 zero4 = make_float4(0.f, 0.f, 0.f, 0.f);
  for (int j0 = gid; j0 < n; j0 += R * ngroups) {
    float* row[R];
    float4 x[R], w[R], s1[R], s2[R];
    float4 tail[R];                  // AdaGrad: accumulator, show, click, days without show
    int delta[R];                    // Adam, Ftrl: shows since the last save
    float2 cn[R];
#pragma unroll
    for (int q = 0; q < R; ++q) {
      const int j = j0 + q * ngroups;
      row[q] = nullptr;
      x[q] = zero4;
      if (j >= n) continue;
      const int rr = __ldcg(&c.req_row[j]);
      if (has) x[q] = ldcg_f4(c.gU + (size_t)j * gstride + 4 * lane);
      if (lane == 0) cn[q] = __ldcg(reinterpret_cast<const float2*>(c.cnts) + j);
      if (rr != kReqNone && rr != kReqPending) row[q] = t.rows + (size_t)(rr & kReqRowMask) * stride;
    }
#pragma unroll
    for (int q = 0; q < R; ++q) {
      w[q] = s1[q] = s2[q] = zero4;
      tail[q] = zero4;
      delta[q] = 0;
      if (row[q] == nullptr) continue;
      if (has) {
        w[q] = ldcg_f4(row[q] + 4 * lane);
        if (KIND != kAdaGrad) {
          s1[q] = ldcg_f4(row[q] + dim + 4 * lane);
          s2[q] = ldcg_f4(row[q] + 2 * dim + 4 * lane);
        }
      }
      if (KIND == kAdaGrad) tail[q] = ldcg_f4(row[q] + dim);
      else if (lane == 0) delta[q] = __ldcg(reinterpret_cast<const int*>(row[q]) + 3 * dim + 1);
    }
#pragma unroll
    for (int q = 0; LocalPush<KIND>::kPrefetch && q < R; ++q) {
      const int j = j0 + (R + q) * ngroups;
      if (j >= n) continue;
      const int rr = __ldcg(&c.req_row[j]);
      prefetch_row_l2(c.gU + (size_t)j * gstride, dim, lane, G);
      if (rr != kReqNone && rr != kReqPending) prefetch_row_l2(t.rows + (size_t)(rr & kReqRowMask) * stride, stride, lane, G);
    }
#pragma unroll
    for (int q = 0; q < R; ++q) {
      const int j = j0 + q * ngroups;
      if (j >= n) continue;                         // the same for all lanes of a group
      if (KIND == kAdaGrad) {
        float ss = x[q].x * x[q].x + x[q].y * x[q].y + x[q].z * x[q].z + x[q].w * x[q].w;
        for (int off = G >> 1; off > 0; off >>= 1) ss += __shfl_xor_sync(gmask, ss, off);
        tail[q].x += ss / (float)dim;
        const float scale = fast_div(o.lr, o.eps + fast_sqrt(tail[q].x));
        w[q].x -= scale * x[q].x; w[q].y -= scale * x[q].y; w[q].z -= scale * x[q].z; w[q].w -= scale * x[q].w;
      } else if (KIND == kAdam) {
        adam_chunk(o, x[q], w[q], s1[q], s2[q]);
      } else {
        ftrl_chunk(o, x[q], w[q], s1[q], s2[q]);
      }
      if (row[q] != nullptr) {
        if (has) {
          *reinterpret_cast<float4*>(row[q] + 4 * lane) = w[q];
          if (KIND != kAdaGrad) {
            *reinterpret_cast<float4*>(row[q] + dim + 4 * lane) = s1[q];
            *reinterpret_cast<float4*>(row[q] + 2 * dim + 4 * lane) = s2[q];
          }
        }
        if (lane == 0) {
          if (KIND == kAdaGrad) {
            *reinterpret_cast<float4*>(row[q] + dim) = make_float4(tail[q].x, tail[q].y + cn[q].x, tail[q].z + cn[q].y, 0.f);
          } else {
            reinterpret_cast<int*>(row[q])[3 * dim + 1] = delta[q] + (int)cn[q].x;
          }
        }
      }
      if (has) *reinterpret_cast<float4*>(c.gU + (size_t)j * gstride + 4 * lane) = zero4;
      if (lane == 0) reinterpret_cast<float2*>(c.cnts)[j] = make_float2(0.f, 0.f);
    }
  }
  prof_mark(c, 13);
}

// AdaGrad rows whose width is no multiple of four (linear weights have one column): accumulator and counters then start in
// the middle of a 16-byte piece.  A row is whole pieces all the same, so a lane takes one of them, whatever it holds, the
// accumulator is handed round the group, and the row costs one load and one store per lane.  Two rows at a time,
// 84 K rows of ten columns and of one: 24.1 us a row at a time and element by element, 16.5 now.
// (Adam and Ftrl keep three arrays of such a width, which start at three different places of their pieces: a column's three
// values then lie with different lanes.  Those rows are left to sparse_push_local_rows_kernel.)
constexpr int kOddRows = 2;
__global__ void __launch_bounds__(256, 5) sparse_push_local_odd_kernel(const __grid_constant__ PushArgs a) {
  const float* const rows = a.tbl_dev->rows;        // (changes between steps only)
  pdl_sync();
  const SparseCommView& c = a.c;
  const SparseOptParams& o = a.opt;
  prof_mark(c, 8);
  const int n = __ldcg(&c.cnt_saved[0]);
  const int G = a.lanes, lane = threadIdx.x % G;
  const int gid = (blockIdx.x * blockDim.x + threadIdx.x) / G, ngroups = gridDim.x * blockDim.x / G;
  const unsigned gmask = group_mask(G);
  const int dim = a.tbl.dim, stride = a.tbl.stride, gstride = c.gstride;
  const bool has = 4 * lane < dim + 4;
  for (int j0 = gid; j0 < n; j0 += kOddRows * ngroups) {
    float* row[kOddRows];
    float4 x[kOddRows], v[kOddRows];
    float2 cn[kOddRows];
#pragma unroll
    for (int q = 0; q < kOddRows; ++q) {
      const int j = j0 + q * ngroups;
      row[q] = nullptr;
      x[q] = v[q] = make_float4(0.f, 0.f, 0.f, 0.f);
      cn[q] = make_float2(0.f, 0.f);
      if (j >= n) continue;
      const int rr = __ldcg(&c.req_row[j]);
      if (4 * lane < dim) x[q] = ldcg_f4(c.gU + (size_t)j * gstride + 4 * lane);
      cn[q] = __ldcg(reinterpret_cast<const float2*>(c.cnts) + j);
      if (rr != kReqNone && rr != kReqPending) row[q] = const_cast<float*>(rows) + (size_t)(rr & kReqRowMask) * stride;
    }
#pragma unroll
    for (int q = 0; q < kOddRows; ++q)
      if (row[q] != nullptr && has) v[q] = ldcg_f4(row[q] + 4 * lane);
#pragma unroll
    for (int q = 0; q < kOddRows; ++q) {
      const int j = j0 + q * ngroups;
      if (j >= n) continue;                         // the same for all lanes of a group
      float g[4] = {x[q].x, x[q].y, x[q].z, x[q].w}, e[4] = {v[q].x, v[q].y, v[q].z, v[q].w};
      float ss = 0.f, acc = 0.f;
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        if (4 * lane + k < dim) ss += g[k] * g[k];
        if (k == (dim & 3)) acc = e[k];
      }
      for (int off = G >> 1; off > 0; off >>= 1) ss += __shfl_xor_sync(gmask, ss, off);
      const float g2 = __shfl_sync(gmask, acc, dim >> 2, G) + ss / (float)dim;
      const float scale = o.lr / (o.eps + sqrtf(g2));
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        const int i = 4 * lane + k;
        if (i < dim) e[k] -= scale * g[k];
        else if (i == dim) e[k] = g2;
        else if (i == dim + 1) e[k] += cn[q].x;
        else if (i == dim + 2) e[k] += cn[q].y;
        else if (i == dim + 3) e[k] = 0.f;          // days without a show, an integer
      }
      if (row[q] != nullptr && has) *reinterpret_cast<float4*>(row[q] + 4 * lane) = make_float4(e[0], e[1], e[2], e[3]);
      if (4 * lane < gstride) *reinterpret_cast<float4*>(c.gU + (size_t)j * gstride + 4 * lane) = make_float4(0.f, 0.f, 0.f, 0.f);
      if (lane == 0) reinterpret_cast<float2*>(c.cnts)[j] = make_float2(0.f, 0.f);
    }
  }
  prof_mark(c, 13);
}

// The other row widths (no multiple of 4, or above 128): one row per group at a time, the next one asked for from L2.
__global__ void __launch_bounds__(256) sparse_push_local_rows_kernel(const __grid_constant__ PushArgs a) {
  pdl_sync();
  const SparseCommView& c = a.c;
  prof_mark(c, 8);
  __shared__ TableView s_tbl;
  if (threadIdx.x == 0) s_tbl = a.tbl_dev != nullptr ? *a.tbl_dev : a.tbl;
  __syncthreads();
  const TableView& t = s_tbl;
  const int n = __ldcg(&c.cnt_saved[0]);
  const int G = a.lanes, lane = threadIdx.x % G;
  const int gid = (blockIdx.x * blockDim.x + threadIdx.x) / G, ngroups = gridDim.x * blockDim.x / G;
  const unsigned gmask = group_mask(G);
  const int dim = t.dim, gstride = c.gstride, gch = gstride >> 2;
  const bool vec = (dim & 3) == 0;
  const float4 zero4 = make_float4(0.f, 0.f, 0.f, 0.f);
  for (int j = gid; j < n; j += ngroups) {
    const int rr = __ldcg(&c.req_row[j]);
    if (j + ngroups < n) {
      const int r2 = __ldcg(&c.req_row[j + ngroups]);
      if (r2 != kReqNone && r2 != kReqPending) prefetch_row_l2(t.rows + (size_t)(r2 & kReqRowMask) * t.stride, t.stride, lane, G);
    }
    float* g = c.gU + (size_t)j * gstride;
    float* cn = c.cnts + 2 * (size_t)j;
    if (rr != kReqNone && rr != kReqPending) {
      float* row = t.rows + (size_t)(rr & kReqRowMask) * t.stride;
      const float bshow = cn[0], bclick = cn[1];
      if (vec) apply_row<true>(a.opt, row, g, bshow, bclick, dim, lane, G, gmask);
      else apply_row<false>(a.opt, row, g, bshow, bclick, dim, lane, G, gmask);
    }
    __syncwarp(gmask);
    for (int ch = lane; ch < gch; ch += G) *reinterpret_cast<float4*>(g + 4 * ch) = zero4;
    if (lane == 0) { cn[0] = 0.f; cn[1] = 0.f; }
  }
  prof_mark(c, 13);
}

// Several GPUs.
// `dense_ctas` > 0: the last `dense_ctas` CTAs of the grid run the dense step `d` of the same training step (reduce-
// scatter of the flat gradient, optimizer on the owned chunk, all-gather of the new weights) while the others push.
// Both exchanges wait on the same peers at the same point of the step, so side by side they cost one wait instead
// of two; the dense CTAs use the dense table's own barrier and flag words.
__global__ void __launch_bounds__(kThreads, 1) sparse_push_fused_kernel(const __grid_constant__ PushArgs a,
                                                                        const __grid_constant__ DenseStepArgs d,
                                                                        const int dense_ctas) {
  const int nb = (int)gridDim.x - dense_ctas;      // CTAs of the push proper
  if ((int)blockIdx.x >= nb) {
    dense::fused_step<kRiderUnroll>(d, (int)blockIdx.x - nb, dense_ctas);   // two loads in flight: fits the 64-register budget of 1024 threads
    return;
  }
  const SparseCommView& c = a.c;
  __shared__ TableView s_tbl;
  if (threadIdx.x == 0) s_tbl = a.tbl_dev != nullptr ? *a.tbl_dev : a.tbl;
  __syncthreads();
  const TableView& t = s_tbl;
  GridSync gs;
  gs.init(c.bar, c.status, c.wait_ns, (unsigned)nb);
  __shared__ unsigned long long s_flag;
  __shared__ int s_pre[kMaxWorld + 1];

  const int tid = blockIdx.x * blockDim.x + threadIdx.x;
  const int nth = nb * blockDim.x;
  const int W = c.world, R = c.rank, capo = c.capo;
  const unsigned long long epoch = __ldcg(c.epoch);
  const int dim = t.dim, gstride = c.gstride, gch = gstride >> 2;
  const int G = a.lanes;
  const int lane = threadIdx.x % G;
  const int gid = tid / G, ngroups = nth / G;
  const unsigned gmask = group_mask(G);
  const float4 zero4 = make_float4(0.f, 0.f, 0.f, 0.f);
  const bool vec = (dim & 3) == 0;

  prof_mark(c, 8);
  // ---- phase A: tell every owner that this GPU's gradient records are complete.  They are: the backward pass that
  // wrote them precedes this kernel in the stream.  The records stay where they are; each owner READS its segment of
  // every GPU's records over NVLink and sums as it reads.  (Shipping them into inboxes first cost a pass of peer
  // stores, a system-wide fence to drain it and a second pass to sum: 36 us of a 72 us push on eight GPUs.)
  if (blockIdx.x == 0 && threadIdx.x < W && threadIdx.x != R)
    st_release_sys_u64(sig_word(c.sig[threadIdx.x], kSigPushReq, R), epoch << 32);
  prof_mark(c, 9);
  prof_mark(c, 10);

  // ---- phase B: as owner, sum records of equal sign coming from different GPUs --------------------
  // own records first (nothing to wait for)
  {
    const int n_s = __ldcg(&c.req_n[R]);
    const float* src = c.gU + (size_t)R * capo * gstride;
    const int total = n_s * gch;
    for (int i = tid; i < total; i += nth) {
      const int j = i / gch, ch = i - j * gch;
      const int ou = __ldcg(&c.req_ou[R * capo + j]);
      if (ou < 0) continue;
      red_add_f32x4(c.acc + (size_t)ou * gstride + 4 * ch, ldcg_f4(src + 4 * (size_t)i));
    }
    const float2* csrc = reinterpret_cast<const float2*>(c.cnts) + (size_t)R * capo;
    for (int j = tid; j < n_s; j += nth) {
      const int ou = __ldcg(&c.req_ou[R * capo + j]);
      if (ou < 0) continue;
      const float2 sc = __ldcg(&csrc[j]);
      float* g = c.acc + (size_t)ou * gstride + dim;          // the record's show / click slots
      atomicAdd(g, sc.x);
      if (sc.y != 0.f) atomicAdd(g + 1, sc.y);
    }
  }
  prof_mark(c, 14);
  // then everybody else's, as one flat index space over the senders so that no thread idles on a short segment
  {
    __syncthreads();
    if (threadIdx.x < 32) {       // one lane per sender polls its flag; a warp scan lays the segments end to end
      const int k = threadIdx.x;
      const int sk = (R + 1 + k) % W;
      unsigned long long v;
      bool ok = true;
      if (k + 1 < W) ok = wait_flag_ge(sig_word(c.sig[R], kSigPushReq, sk), epoch, &v, c.wait_ns, c.status, 12, sk);
      const bool all_ok = __all_sync(0xffffffffu, ok);
      int incl = (k + 1 < W) ? __ldcg(&c.req_n[sk]) : 0;
#pragma unroll
      for (int o = 1; o < kMaxWorld; o <<= 1) {
        const int up = __shfl_up_sync(0xffffffffu, incl, o);
        if (k >= o) incl += up;
      }
      if (k + 1 < W) s_pre[k + 1] = incl;
      if (k == 0) { s_pre[0] = 0; s_flag = all_ok ? 0ull : ~0ull; }
    }
    __syncthreads();
    prof_mark(c, 15);
    if (s_flag == ~0ull) { gs.failed = true; }
    else {
      const int n_all = s_pre[W - 1];
      const int total = n_all * gch;
      for (int i = tid; i < total; i += nth) {
        const int jj = i / gch, ch = i - jj * gch;
        int k = 0;
        while (jj >= s_pre[k + 1]) ++k;
        const int sk = (R + 1 + k) % W, j = jj - s_pre[k];
        const int ou = __ldcg(&c.req_ou[sk * capo + j]);
        if (ou < 0) continue;
        // sender sk keeps the records it owes this GPU in segment R of its gradient matrix
        const float4 v = ldcg_f4(c.gU_peer[sk] + ((size_t)R * capo + j) * gstride + 4 * ch);
        red_add_f32x4(c.acc + (size_t)ou * gstride + 4 * ch, v);
      }
      for (int jj = tid; jj < n_all; jj += nth) {
        int k = 0;
        while (jj >= s_pre[k + 1]) ++k;
        const int sk = (R + 1 + k) % W, j = jj - s_pre[k];
        const int ou = __ldcg(&c.req_ou[sk * capo + j]);
        if (ou < 0) continue;
        const float2 sc = __ldcg(reinterpret_cast<const float2*>(c.cnts_peer[sk]) + (size_t)R * capo + j);
        float* g = c.acc + (size_t)ou * gstride + dim;
        atomicAdd(g, sc.x);
        if (sc.y != 0.f) atomicAdd(g + 1, sc.y);
      }
    }
  }
  if (gs.failed) goto done;
  prof_mark(c, 11);
  // every value read from a peer has been consumed once all CTAs are here: the senders may clear their records
  if (last_cta_arrives(&c.bar[2], false, (unsigned)nb) && threadIdx.x < W && threadIdx.x != R)
    st_release_sys_u64(sig_word(c.sig[threadIdx.x], kSigPushDone, R), epoch << 32);
  if (!gs.sync(13, false)) goto done;
  prof_mark(c, 12);

  // ---- phase C: one optimizer update per touched row ----------------------------------------------
  {
    const int n_ou = __ldcg(c.ocount);
    for (int ou = gid; ou < n_ou; ou += ngroups) {
      const int r = __ldcg(&c.ou_row[ou]);
      if (ou + ngroups < n_ou) {
        const int r2 = __ldcg(&c.ou_row[ou + ngroups]);
        if (r2 >= 0) prefetch_row_l2(t.rows + (size_t)r2 * t.stride, t.stride, lane, G);
      }
      float* g = c.acc + (size_t)ou * gstride;
      if (r >= 0) {
        float* row = t.rows + (size_t)r * t.stride;
        const float bshow = g[dim], bclick = g[dim + 1];
        if (vec) apply_row<true>(a.opt, row, g, bshow, bclick, dim, lane, G, gmask);
        else apply_row<false>(a.opt, row, g, bshow, bclick, dim, lane, G, gmask);
      }
      __syncwarp(gmask);
      for (int ch = lane; ch < gch; ch += G) *reinterpret_cast<float4*>(g + 4 * ch) = zero4;
    }
  }
  prof_mark(c, 13);
  // every CTA is past its row updates: re-arm the owner-unique counter for a pull whose front ran ahead
  if (last_cta_arrives(&c.bar[3], false, (unsigned)nb) && threadIdx.x == 0) *c.ocount = 0;

  // ---- tail: once every owner has read this GPU's records, clear them for the next backward pass (the owners' reads
  // finished while this GPU updated its rows, so the wait is short)
  {
    __syncthreads();
    if (threadIdx.x < 32) {
      const int p = threadIdx.x;
      unsigned long long v;
      bool ok = true;
      if (p < W && p != R) ok = wait_flag_ge(sig_word(c.sig[R], kSigPushDone, p), epoch, &v, c.wait_ns, c.status, 16, p);
      const bool all_ok = __all_sync(0xffffffffu, ok);
      if (threadIdx.x == 0) s_flag = all_ok ? 0ull : ~0ull;
    }
    __syncthreads();
    if (s_flag == ~0ull) { gs.failed = true; goto done; }
    for (int p = 0; p < W; ++p) {
      const int n = __ldcg(&c.cnt_saved[p]);
      float4* g4 = reinterpret_cast<float4*>(c.gU + (size_t)p * capo * gstride);
      const int total = n * gch;
      for (int i = tid; i < total; i += nth) g4[i] = zero4;
      float2* c2 = reinterpret_cast<float2*>(c.cnts) + (size_t)p * capo;
      for (int j = tid; j < n; j += nth) c2[j] = make_float2(0.f, 0.f);
    }
  }

done:
  gs.leave();
}

// =======================================================================================
// host launchers
// =======================================================================================
static int coop_grid(const void* fn, int device) {
  int per_sm = 0, sms = 0;
  cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, fn, kThreads, 0);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device);
  if (per_sm < 1) per_sm = 1;
  if (per_sm > 1) per_sm = 1;
  return per_sm * sms;
}

// A thread per id up to what the chip holds at once; kernels that also clear the dedup keys have a thread per 16 of them.
static int local_grid(const PullArgs& args, bool clears) {
  long long work = args.n_ids;
  if (clears && ((long long)args.c.dd_mask + 1) / 16 > work) work = ((long long)args.c.dd_mask + 1) / 16;
  const long long blocks = (work + kLocalThreads - 1) / kLocalThreads;
  return blocks < 1 ? 1 : (int)(blocks > 148ll * 4 ? 148ll * 4 : blocks);
}

template <int N>
static cudaError_t launch_pulls(const PullArgs* pulls, int n, cudaStream_t stream) {
  PullArgsOf<N> batch;
  int probe = 1, finish = 1;
  for (int k = 0; k < n; ++k) {
    batch.a[k] = pulls[k];
    if (pulls[k].front_done != pulls[0].front_done) return cudaErrorInvalidValue;
    probe = max(probe, local_grid(pulls[k], false));
    finish = max(finish, local_grid(pulls[k], !pulls[k].front_done));
  }
  const dim3 block(kLocalThreads);
  cudaError_t e = cudaSuccess;
  if (!pulls[0].front_done) e = launch_pdl(pull_local_probe_kernel<N>, dim3(probe, n), block, 0, stream, batch);
  return e == cudaSuccess ? launch_pdl(pull_local_finish_kernel<N>, dim3(finish, n), block, 0, stream, batch) : e;
}
// One GPU, rows left in the table (see pull_local_probe_kernel).  The `n` pulls are all behind a front or all not.
cudaError_t launch_sparse_pull_local(const PullArgs* pulls, int n, cudaStream_t stream) {
  static_assert(kMaxPullBatch == 2, "instances below");
  if (n < 1 || n > kMaxPullBatch) return cudaErrorInvalidValue;
  return n == 1 ? launch_pulls<1>(pulls, n, stream) : launch_pulls<2>(pulls, n, stream);
}

// The rows of a batch's ids (see lookup_rows_kernel).
template <int N>
static cudaError_t launch_lookups(const PullArgs* pulls, int n, cudaStream_t stream) {
  PullArgsOf<N> batch;
  int most = 1;
  for (int k = 0; k < n; ++k) { batch.a[k] = pulls[k]; most = max(most, pulls[k].n_ids); }
  const long long blocks = ((long long)most + kLocalThreads - 1) / kLocalThreads;
  const dim3 block(kLocalThreads), all((unsigned)min(blocks, 148ll * 8), n), half((unsigned)min(blocks, 148ll * 4), n);
  cudaError_t e = launch_pdl(lookup_rows_kernel<N>, all, block, 0, stream, batch);
  if (e == cudaSuccess && !pulls[0].lookup_only) {
    e = launch_pdl(lookup_insert_kernel<N>, half, block, 0, stream, batch);
    if (e == cudaSuccess) e = launch_pdl(lookup_again_kernel<N>, half, block, 0, stream, batch);
  }
  return e;
}
cudaError_t launch_sparse_lookup(const PullArgs* pulls, int n, cudaStream_t stream) {
  if (n < 1 || n > kMaxPullBatch) return cudaErrorInvalidValue;
  return n == 1 ? launch_lookups<1>(pulls, n, stream) : launch_lookups<2>(pulls, n, stream);
}

// The pulled rows also into the per-batch matrix.
cudaError_t launch_sparse_pull_local_rows(const PullArgs& args, cudaStream_t stream) {
  const long long want = ((long long)args.n_ids * args.lanes + kLocalThreads - 1) / kLocalThreads;
  return launch_pdl(pull_local_rows_kernel, dim3(want > 148 * 8 ? 148 * 8 : want < 1 ? 1 : (int)want), dim3(kLocalThreads), 0, stream, args);
}

// Fronts run beside the backward pass, whose GEMMs leave room on an SM for one block of 256 threads and have priority.  A grid
// that fills the chip keeps the GEMMs out until it has run; one that is too small outlasts the backward pass, and the step ends
// with it.  Two blocks per SM as long as a thread has at most two ids, three beyond.  Over 160 workloads (DeepFM, Wide&Deep,
// Deep&Cross, DCN-v2; 20 K to 790 K single-hot ids; towers from 64-32 to 1024-512-256) three take 0.2 % less per step than the
// pull's own grid of up to four; two take 0.1 to 0.2 % less than three up to 151 K ids, 0.6 to 1 % more beyond 300 K.  Two tables of
// 2999 x 39 ids beside 300-150-75: 147.4 us with two, 149.4 with three, 154 with four; 8192 x 26 beside 64-32: 146, 142, 141.  Blocks
// of 128 threads, of which more fit beside a GEMM, four per SM (two for the second kernel): 1.7 to 2.5 % more than four of 256 on
// the mean, and where the tower is short up to a quarter (7753 x 46 beside 128-128: 218 -> 270 us).
cudaError_t launch_sparse_pull_local_front(const PullArgs& args, cudaStream_t stream) {
  PullArgsOf<1> batch;
  batch.a[0] = args;
  const dim3 block(kLocalThreads);
  const int most = args.n_ids <= 2 * 2 * 148 * kLocalThreads ? 148 * 2 : 148 * 3;
  const cudaError_t e = launch_pdl(pull_local_probe_kernel<1>, dim3(min(local_grid(args, false), most)), block, 0, stream, batch);
  return e != cudaSuccess ? e : launch_pdl(pull_local_resolve_kernel, dim3(min(local_grid(args, true), most)), block, 0, stream, args);
}

cudaError_t launch_sparse_pull(const PullArgs& args, int work_items, cudaStream_t stream) {
  int dev = 0;
  cudaGetDevice(&dev);
  const bool tiled = args.tile_rows > 0;
  const void* fn = tiled ? (const void*)sparse_pull_fused_kernel<true> : (const void*)sparse_pull_fused_kernel<false>;
  static int grid_max[64][2] = {{0}};
  if (grid_max[dev][tiled] == 0) grid_max[dev][tiled] = coop_grid(fn, dev);
  int grid = (work_items + kThreads - 1) / kThreads;
  if (grid < 1) grid = 1;
  if (grid > grid_max[dev][tiled]) grid = grid_max[dev][tiled];
  const size_t smem = (size_t)args.tile_rows * args.c.ustride * sizeof(float) * (kThreads / 32);
  static bool attr_set[64] = {false};
  // static + dynamic shared memory beyond 48 KiB needs the opt-in; a 48 KiB tile buffer alone already crosses it
  if (smem > 32 * 1024 && !attr_set[dev]) {
    cudaError_t e = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, 200 * 1024);
    if (e != cudaSuccess) return e;
    attr_set[dev] = true;
  }
  void* params[] = {(void*)&args};
  return cudaLaunchCooperativeKernel(fn, dim3(grid), dim3(kThreads), params, smem, stream);
}

cudaError_t launch_sparse_pull_front(const PullArgs& args, cudaStream_t stream) {
  int dev = 0, sms = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  int grid = (args.n_ids + kFrontThreads - 1) / kFrontThreads;
  if (grid < 1) grid = 1;
  if (grid > 4 * sms) grid = 4 * sms;
  pull_front_dedup_kernel<<<grid, kFrontThreads, 0, stream>>>(args);
  pull_front_ship_kernel<<<grid, kFrontThreads, 0, stream>>>(args);
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return e;
  // the inverse map is complete: the dedup scratch goes back to all-empty (kEmptyKey is all ones)
  return cudaMemsetAsync(args.c.dd_keys, 0xFF, ((size_t)args.c.dd_mask + 1u) * sizeof(unsigned long long), stream);
}

static cudaError_t launch_sparse_push_local(PushArgs args, long long rows, int max_ctas, cudaStream_t stream) {
  const int dim = args.tbl.dim, kind = args.opt.kind;
  const bool chunk_per_lane = (dim & 3) == 0 && dim <= 128;
  const bool odd_pieces = kind == kAdaGrad && (dim & 3) != 0 && dim + 4 <= 128 && args.tbl_dev != nullptr;
  if (chunk_per_lane) args.lanes = lanes_for_width(dim);
  if (odd_pieces) args.lanes = lanes_for_width(dim + 4);
  void (*kernel)(PushArgs) = sparse_push_local_rows_kernel;
  int rows_per_group = 1, per_sm = 4;
  auto take = [&](void (*k)(PushArgs), int r, int blocks) { kernel = k; rows_per_group = r; per_sm = blocks; };
  if (odd_pieces) take(sparse_push_local_odd_kernel, kOddRows, 5);
  if (chunk_per_lane) {
    if (kind == kAdaGrad) take(sparse_push_local_kernel<kAdaGrad>, LocalPush<kAdaGrad>::kRows, LocalPush<kAdaGrad>::kBlocks);
    else if (kind == kAdam) take(sparse_push_local_kernel<kAdam>, LocalPush<kAdam>::kRows, LocalPush<kAdam>::kBlocks);
    else take(sparse_push_local_kernel<kFtrl>, LocalPush<kFtrl>::kRows, LocalPush<kFtrl>::kBlocks);
  }
  long long blocks = (rows * args.lanes + 256ll * rows_per_group - 1) / (256ll * rows_per_group);
  if (blocks < 1) blocks = 1;
  // Blocks that come while those of the kernel ahead drain are spread unevenly over the SMs, and these stay to the end: the rows of
  // 8192 examples of DCN-v2 (4 M ids, width 64, Ftrl) 1 240 us, and 940 when launched behind it.  A push of a few passes is over before that tells, and an early start
  // is 1 to 2 us less (sixteen steps of Wide&Deep at 1024: 1 165 -> 1 135 us).
  const bool many = blocks > 8 * 148ll * per_sm;
  if (blocks > 148ll * per_sm) blocks = 148ll * per_sm;
  if (max_ctas > 0 && blocks > (long long)max_ctas * per_sm) blocks = (long long)max_ctas * per_sm;
  if (many) {
    kernel<<<dim3((unsigned)blocks), dim3(256), 0, stream>>>(args);
    return cudaGetLastError();
  }
  return launch_pdl(kernel, dim3((unsigned)blocks), dim3(256), 0, stream, args);
}

// `max_ctas` > 0 caps the grid below the SM count, leaving whole SMs to a kernel running on another stream.
// `dense` != null (several GPUs only): the dense step rides on `dense_ctas` extra CTAs of the same cooperative grid.
cudaError_t launch_sparse_push(const PushArgs& args, int work_items, int max_ctas, const DenseStepArgs* dense, cudaStream_t stream) {
  if (args.c.world == 1 && dense == nullptr) return launch_sparse_push_local(args, work_items / args.lanes, max_ctas, stream);
  int dev = 0;
  cudaGetDevice(&dev);
  static int grid_max[64] = {0};
  if (grid_max[dev] == 0) grid_max[dev] = coop_grid((const void*)sparse_push_fused_kernel, dev);
  int grid = (work_items + kThreads - 1) / kThreads;
  if (grid < 1) grid = 1;
  int dense_ctas = 0;
  DenseStepArgs d{};
  if (dense != nullptr) {
    if (dense->world < 2 || dense->n % 4 || dense->chunk % 4) return cudaErrorInvalidValue;
    d = *dense;
    // one pass of the owned chunk: 1024 threads x kDenseUnroll 16-byte groups per CTA, at most 16 CTAs
    const long long per_cta = (long long)kThreads * kRiderUnroll * 4;
    dense_ctas = (int)((d.chunk + per_cta - 1) / per_cta);
    if (dense_ctas < 1) dense_ctas = 1;
    if (dense_ctas > 16) dense_ctas = 16;
  }
  const int room = grid_max[dev] - dense_ctas;
  if (grid > room) grid = room;
  if (max_ctas > 0 && grid > max_ctas) grid = max_ctas;
  if (grid < 1) return cudaErrorInvalidValue;
  grid += dense_ctas;
  void* params[] = {(void*)&args, (void*)&d, (void*)&dense_ctas};
  return cudaLaunchCooperativeKernel((const void*)sparse_push_fused_kernel, dim3(grid), dim3(kThreads), params, 0, stream);
}

}  // namespace tn
