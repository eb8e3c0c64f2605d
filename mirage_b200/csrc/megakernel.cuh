// The decode megakernel: one launch executes one iteration of the task graph.  Included by the files that
// instantiate it (decoder_kernels.cu, hybrid_kernel_*.cu).
//
// Replaces the reference's persistent runtime (worker/scheduler loops and queues,
// include/mirage/persistent_kernel/persistent_kernel.cuh:513-1082) and the task bodies
// it dispatches to (include/mirage/persistent_kernel/tasks/**) for the decode path.
//
// Structure of a worker CTA (one per SM, 288 threads; 384 in the general instantiations):
//   * warp 8 is the weight streamer.  It walks the worker's task list ahead of the
//     compute warps and issues cp.async.bulk copies of the weight rows every linear
//     task will need into a ring of 32 KB shared-memory stages guarded by mbarriers.
//     Weights never depend on events, so the stream keeps HBM busy across task
//     boundaries, dependency waits and attention tasks.
//   * warps 0-7 execute tasks in order: acquire-poll the task's event counters, run
//     the body, release-increment the trigger counter.
// Counters grow monotonically: a dependency is complete when
// counter >= arrivals_per_iteration * iteration.  The iteration number lives in device
// memory and is advanced by the last CTA to leave the kernel, so a captured CUDA graph
// of launches can be replayed.
//
// Every wait (event counter, mbarrier) is bounded by a wall-clock budget; on expiry the
// CTA records where it gave up, raises a global abort flag that all other waits poll,
// drains its own in-flight copies and returns.
#pragma once
#include <cuda_bf16.h>
#include <cuda_fp8.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include "device_utils.cuh"
#include "runtime_types.h"

namespace mpk {

constexpr int kFlagsOffset = 960;   // of the flags in the area of small things
constexpr int kXIssuers = 5;        // warps that issue the MMAs of a tcgen05 linear, at most
constexpr int kXBarsOffset = 1248;  // of the barriers of the tcgen05 linears' activations and borrowed slots
static_assert(kFlagsOffset + 64 + 8 * kAttnStages * 8 + 32 <= kXBarsOffset && kXBarsOffset + 33 * 8 <= kMiscBytes, "small things overlap");

struct Smem {
  uint8_t *stages;      // num_stages * stage_bytes
  uint8_t *xtile;       // x_tile_bytes (activation tile / attention scratch)
  float *partial;       // kPartialBytes (directly after xtile)
  uint64_t *full;       // [num_stages]
  uint64_t *empty;      // [num_stages]
  TaskDesc *desc;       // [2]
  float *red;           // [64]
  int *flags;           // [0] abort  [1] broadcast scratch
  uint64_t *acc_bar;    // tcgen05 path: "accumulators complete / activation tile free" barrier (count 1)
  uint32_t *tmem_holder;   // tensor-memory base address written by tcgen05.alloc
};

__device__ __forceinline__ Smem carve(uint8_t *base, const KernelParams &P) {
  Smem s;
  s.stages = base;
  s.xtile = base + (size_t)P.num_stages * P.stage_bytes;
  s.partial = reinterpret_cast<float *>(s.xtile + P.x_tile_bytes);
  uint8_t *misc = reinterpret_cast<uint8_t *>(s.partial) + kPartialBytes;
  s.full = reinterpret_cast<uint64_t *>(misc);            // 16 * 8
  s.empty = s.full + 16;                                    // 16 * 8
  s.desc = reinterpret_cast<TaskDesc *>(misc + 256);        // 2 * 224 = 448
  s.red = reinterpret_cast<float *>(misc + 704);            // 64 * 4 = 256
  s.flags = reinterpret_cast<int *>(misc + kFlagsOffset);   // 16 ints
  s.acc_bar = s.empty + 8;                                  // entries 8.. of the empty-barrier array are unused (<= 8 stages)
  s.tmem_holder = reinterpret_cast<uint32_t *>(s.empty + 9);
  return s;
}

struct LinearState {   // position of the compute warps in the weight stage ring
  int stage;
  uint32_t phase;       // parity of the next completion of its slots behind `stage`; with borrowed slots (XRing) a bit for each slot
  uint32_t acc_phase;   // parity of the next completion of the tcgen05 accumulator barrier
};

struct Ctx {
  const KernelParams &P;
  Smem s;
  unsigned long long iteration;
  uint64_t deadline_ns;   // absolute globaltimer value after which waits give up
  int worker;
  uint32_t tmem_base;     // tensor-memory address of column 0 (general instantiation, graphs with tcgen05 tasks)
};

// Barriers of the activations of tcgen05 linears, behind those of the attention rings: [0, 8) ring slot full, [8, 16) ring slot free (one arrival
// per issuing warp, at most); of the borrowed weight slots: [16, 24) full, [24, 32) free, [32] the tile area is the task's.
__device__ __forceinline__ uint64_t *x_bars(const Ctx &c) { return c.s.full + kXBarsOffset / 8; }

// Weight slots of a tcgen05 linear in graphs without other streaming tasks (KernelParams::borrow).  The tile area, which attention and other bodies need
// between linears, is mostly empty during one: the task borrows what its activations leave of it for further slots.  Boxes 0, 1, ... of a task go
// to positions 0, 1, ... of a ring of `base` slots, which are filled ahead of the task, and `extra` borrowed ones, which are filled once the task
// has begun.  What bounds the stream is the bytes in flight: a box takes some 2.3 us from its copy to the commit that frees its slot, so 148
// workers need about 100 KB each to draw 6.5 TB/s (64 tokens, gate and up rows of width 4096: 70 KB 45 us, 90 KB 34 us).
struct XRing {
  int base, size;              // slots of the ring proper, with the borrowed ones
  uint32_t stages, extra;      // shared-memory addresses
  uint64_t *full, *empty, *xbars;
  int bytes;                   // of a slot
  __device__ __forceinline__ uint32_t slot(int i) const { return i < base ? stages + (uint32_t)(i * bytes) : extra + (uint32_t)((i - base) * bytes); }
  __device__ __forceinline__ uint64_t *full_bar(int i) const { return i < base ? full + i : xbars + 16 + i - base; }
  __device__ __forceinline__ uint64_t *empty_bar(int i) const { return i < base ? empty + i : xbars + 24 + i - base; }
};
__device__ __forceinline__ XRing x_ring(const Ctx &c, const TaskDesc &d) {
  XRing r;
  r.base = c.P.num_stages;
  r.size = r.base + d.a[LX_EXTRA];
  r.bytes = c.P.stage_bytes;
  r.stages = smem_u32(c.s.stages);
  r.extra = smem_u32(c.s.xtile) + (uint32_t)d.a[LX_XBYTES];
  r.full = c.s.full; r.empty = c.s.empty; r.xbars = x_bars(c);
  return r;
}

// ---------------------------------------------------------------------------
// bounded waits
// ---------------------------------------------------------------------------
static __device__ __noinline__ void report_timeout(DeviceStatus *st, int worker, int where, int task) {
  if (atomicCAS(&st->error, 0, -4) == 0) {
    st->where = where;
    st->worker = worker;
    st->task = task;
    __threadfence();
  }
}

// Returns false when the wait was abandoned (timeout here or abort raised elsewhere).
__device__ __forceinline__ bool wait_mbar(const Ctx &c, uint64_t *bar, uint32_t parity, int task) {
  uint32_t polls = 0;
  while (!mbar_try_wait(bar, parity)) {
    if ((++polls & 0x3ff) == 0) {
      if (ld_volatile_i32(&c.P.status->error) != 0) return false;
      if (globaltimer_ns() > c.deadline_ns) {
        report_timeout(c.P.status, c.worker, 2, task);
        return false;
      }
    }
  }
  return true;
}

// The same for bodies that take no Ctx, on a shared-memory address.
static __device__ __noinline__ bool wait_bar_slow(const KernelParams &P, uint32_t bar, uint32_t parity, uint64_t deadline, int task) {
  uint32_t polls = 0;
  while (!bar_try_wait(bar, parity)) {
    if ((++polls & 0x3ff) == 0) {
      if (ld_volatile_i32(&P.status->error) != 0) return false;
      if (globaltimer_ns() > deadline) {
        report_timeout(P.status, (int)blockIdx.x, 2, task);
        return false;
      }
    }
  }
  return true;
}
__device__ __forceinline__ bool wait_bar(const KernelParams &P, uint32_t bar, uint32_t parity, uint64_t deadline, int task) {
  if (bar_try_wait(bar, parity)) return true;
  return wait_bar_slow(P, bar, parity, deadline, task);
}

__device__ __forceinline__ bool wait_counter(const Ctx &c, const unsigned long long *ctr,
                                             unsigned long long need, bool sys_scope, int where, int task) {
  uint32_t polls = 0;
  while (true) {
    unsigned long long v = sys_scope ? ld_acquire_sys(ctr) : ld_acquire_gpu(ctr);
    if (v >= need) return true;
    if ((++polls & 0xff) == 0) {
      if (ld_volatile_i32(&c.P.status->error) != 0) return false;
      if (globaltimer_ns() > c.deadline_ns) {
        report_timeout(c.P.status, c.worker, where, task);
        return false;
      }
    }
    if (c.P.poll_sleep_ns) __nanosleep(c.P.poll_sleep_ns);
  }
}

static __device__ void prefetch_attention_kv_l2(const Ctx &c, const TaskDesc *d, int lane, int task);

// ---------------------------------------------------------------------------
// weight streamer (warp 8)
// ---------------------------------------------------------------------------
// A linear task streams its weight panel [n0, n1) x K as chunks of 16 rows x KC columns (KC <= 1024):
// one cp.async.bulk per row segment, rows padded by 16 bytes in shared memory so that ldmatrix reads
// are bank-conflict free.  Order: k tile (activation tile) -> 16-row group -> k chunk.
// The same for graphs whose streaming tasks are all tcgen05 linears, with slots borrowed from the tile area (XRing).  A wait, the barrier's byte
// count and a tensor-map copy take a thread 290 cycles whatever the box (16 KB boxes: 57 bytes a cycle), so all four warps of the streaming
// warpgroup issue, one thread each; a slot belongs to one of them.
// (Inlined: a function of its own could use more registers than the streaming warp keeps.)
__device__ __forceinline__ void stream_borrowing(const Ctx &c, int t_begin, int t_end) {
  const KernelParams &P = c.P;
  const uint64_t policy = l2_policy_evict_first();
  const int mine = (threadIdx.x >> 5) & 3;
  uint32_t par = 0, used = 0, gate = 0;   // per slot of this warp: parity of its uses, used at all
  bool ok = true;
  for (int t = t_begin; t < t_end && ok; ++t) {
    const TaskDesc *d = &P.tasks[t];
    if (d->type != TASK_LINEAR) continue;
    if (d->flags & TF_STREAM_AFTER_DEP) {
      for (int i = 0; i < kMaxDeps && ok; ++i)
        if (d->dep_event[i] >= 0) ok = wait_counter(c, &P.counters[d->dep_event[i]], (unsigned long long)d->dep_need[i] * c.iteration, false, 1, t);
      fence_proxy_async_all();   // the weights were written through the generic proxy; the copies read through the async proxy
    }
    const XRing r = x_ring(c, *d);
    const uint8_t *tmap = reinterpret_cast<const uint8_t *>(P.tmaps) + (size_t)d->a[L_TMAP] * 128;
    const int RB = d->a[L_ROWS], nkb = d->a[L_KC] / kTcKBlock, kball = d->a[L_K] / kTcKBlock, tiles = (d->a[L_N1] - d->a[L_N0] + RB - 1) / RB;
    const uint32_t tx = (uint32_t)(nkb * RB * 128);
    int s = 0;
    bool open = false;
    for (int kb = 0; kb < kball && ok; kb += nkb)
      for (int tile = 0; tile < tiles && ok; ++tile) {
        if (s >= r.base && !open) {   // (every warp, so that none falls behind the gate's phases)
          ok = wait_mbar(c, r.xbars + 32, gate, t);
          gate ^= 1u;
          open = true;
        }
        if ((s & 3) == mine) {
          ok = ok && wait_mbar(c, r.empty_bar(s), ((par >> s) & 1u) ^ 1u, t);
          if (!ok) break;
          mbar_arrive_expect_tx(r.full_bar(s), tx);
          tma_load_3d_hint(r.slot(s), tmap, 0, tile * RB, kb, smem_u32(r.full_bar(s)), policy);
          mbar_arrive_n(r.empty_bar(s), 7);   // (of the eight arrivals its barrier counts; the last is the commit of the warp that reads the slot)
          used |= 1u << s;
          par ^= 1u << s;
        }
        if (++s == r.size) s = 0;
      }
  }
  // Every copy must have landed before the CTA may exit.
  for (int i = 0; i < 16; ++i) {
    if (!((used >> i) & 1u)) continue;
    uint64_t *bar = i < P.num_stages ? c.s.full + i : x_bars(c) + 16 + i - P.num_stages;
    uint32_t polls = 0;
    while (!mbar_try_wait(bar, ((par >> i) & 1u) ^ 1u) && ++polls < (1u << 24)) {}   // copies in flight always complete; the bound only guards the loop
  }
}

template <bool GENERAL, int HYB>
__device__ void streamer_loop(const Ctx &c, int t_begin, int t_end) {
  constexpr bool kMoe = HYB ? HYB == HYB_BF16 : GENERAL;   // expert projections stream one panel per active expert
  const KernelParams &P = c.P;
  const int lane = threadIdx.x & 31;
  const uint64_t policy = l2_policy_evict_first();
  const int NST = P.num_stages;
  uint32_t issued = 0;
  int s = 0;
  uint32_t ph = 0;
  int s_land = 0;          // oldest chunk that may still be in flight (pacing)
  uint32_t ph_land = 0;
  const uint32_t max_inflight = (uint32_t)P.max_inflight;
  bool ok = true;
  // The whole warp walks the task list; lane 0 owns the barrier traffic, lane r copies row r of a chunk.
  for (int t = t_begin; t < t_end && ok; ++t) {
    const TaskDesc *d = &P.tasks[t];
    if (!GENERAL && !HYB && d->type == TASK_ATTENTION && P.kv_l2_prefetch) prefetch_attention_kv_l2(c, d, lane, t);
    if (d->type != TASK_LINEAR && !(kMoe && d->type == TASK_MOE_GEMM)) continue;
    if (d->flags & TF_STREAM_AFTER_DEP) {
      if (lane == 0)
        for (int i = 0; i < kMaxDeps && ok; ++i)
          if (d->dep_event[i] >= 0)
            ok = wait_counter(c, &P.counters[d->dep_event[i]], (unsigned long long)d->dep_need[i] * c.iteration,
                              false, 1, t);
      ok = __shfl_sync(0xffffffffu, (int)ok, 0) != 0;
      if (!ok) break;
      fence_proxy_async_all();   // the weights were written through the generic proxy; the bulk copies read through the async proxy
    }
    if (GENERAL && (d->flags & TF_TC)) {
      // tcgen05 path: one tensor-map TMA per ring slot brings a box of {64 columns, RB rows, nkb k blocks} of the
      // task's own row panel (rows past the panel are filled with zeros and cost no HBM traffic) in the
      // 128-byte-swizzled layout the MMA reads.  Order: k tile -> row tile -> k blocks.
      const uint8_t *tmap = reinterpret_cast<const uint8_t *>(P.tmaps) + (size_t)d->a[L_TMAP] * 128;
      const int rows = d->a[L_N1] - d->a[L_N0], RB = d->a[L_ROWS];
      const int kbe = (!HYB && (d->flags & TF_FP8)) ? 2 * kTcKBlock : kTcKBlock;   // elements of one 128-byte k block
      const int nkb = d->a[L_KC] / kbe, kbt = d->a[L_KT] / kbe, kball = d->a[L_K] / kbe;
      const uint32_t tx = (uint32_t)(nkb * RB * 128);
      if (kMoe && d->type == TASK_MOE_GEMM) {
        // expert projections on the tensor path: the row tiles of the active experts, dealt out to the layer's tasks in turn
        const int *act = reinterpret_cast<const int *>(d->p[5]);
        const int N = d->a[L_N], per = (N + RB - 1) / RB, items = min(__ldcg(&act[d->a[M_NEXP]]), d->a[M_NEXP]) * per;
        for (int it = d->a[L_N0]; it < items && ok; it += d->a[L_N1]) {
          const int row = __ldcg(&act[it / per]) * N + it % per * RB;
          for (int kb = 0; kb < kball; kb += nkb) {
            if (lane == 0) {
              ok = wait_mbar(c, &c.s.empty[s], ph ^ 1u, t);
              if (ok) {
                mbar_arrive_expect_tx(&c.s.full[s], tx);
                tma_load_3d(c.s.stages + (size_t)s * P.stage_bytes, tmap, 0, row, kb, &c.s.full[s], policy);
              }
            }
            ok = __shfl_sync(0xffffffffu, (int)ok, 0) != 0;
            if (!ok) break;
            ++issued;
            if (++s == NST) { s = 0; ph ^= 1u; }
          }
        }
        continue;
      }
      const int tiles = (rows + RB - 1) / RB;
      for (int kb_t = 0; kb_t < kball && ok; kb_t += kbt)
        for (int tile = 0; tile < tiles && ok; ++tile)
          for (int kb = 0; kb < kbt; kb += nkb) {
            if (lane == 0) {
              ok = wait_mbar(c, &c.s.empty[s], ph ^ 1u, t);
              if (ok) {
                mbar_arrive_expect_tx(&c.s.full[s], tx);
                tma_load_3d(c.s.stages + (size_t)s * P.stage_bytes, tmap, 0, tile * RB, kb_t + kb, &c.s.full[s], policy);
              }
            }
            ok = __shfl_sync(0xffffffffu, (int)ok, 0) != 0;
            if (!ok) break;
            ++issued;
            if (++s == NST) { s = 0; ph ^= 1u; }
          }
      continue;
    }
    const uint8_t *W = reinterpret_cast<const uint8_t *>(d->p[0]);
    const int n0 = d->a[L_N0], n1 = d->a[L_N1], K = d->a[L_K], ldw = d->a[L_LDW];
    const int KT = d->a[L_KT], KC = d->a[L_KC], R = d->a[L_ROWS];
    const uint32_t esz = (GENERAL && !HYB && (d->flags & TF_FP8)) ? 1u : 2u;   // e4m3 or bf16 weights
    const uint32_t seg_bytes = (uint32_t)KC * esz;
    const uint32_t row_stride = seg_bytes + kRowPadBytes;
    // an expert task repeats the panel loop once per active expert (the list is final: the task waited for it)
    int reps = 1;
    const int *act = nullptr;
    if (kMoe && d->type == TASK_MOE_GEMM) {
      act = reinterpret_cast<const int *>(d->p[5]);
      reps = min(__ldcg(&act[d->a[M_NEXP]]), d->a[M_NEXP]);
    }
    for (int rep = 0; rep < reps && ok; ++rep) {
    const uint8_t *Wp = W;
    if (kMoe && act != nullptr) Wp = W + (size_t)__ldcg(&act[rep]) * (size_t)d->a[M_ESTRIDE] * esz;
    for (int kt = 0; kt < K && ok; kt += KT) {
      for (int r0 = n0; r0 < n1 && ok; r0 += R) {
        const int rows = min(R, n1 - r0);
        const uint8_t *src_row = Wp + ((size_t)(r0 + lane) * ldw + kt) * esz;   // valid for lane < rows
        for (int kc = 0; kc < KT; kc += KC) {
          if (lane == 0) {
            ok = wait_mbar(c, &c.s.empty[s], ph ^ 1u, t);
            // pacing: keep at most max_inflight chunks between "issued" and "landed", so that the
            // latency-critical loads and stores of the compute warps do not queue behind a full ring
            if (ok && max_inflight < (uint32_t)NST && issued >= max_inflight) {
              ok = wait_mbar(c, &c.s.full[s_land], ph_land, t);
              if (++s_land == NST) { s_land = 0; ph_land ^= 1u; }
            }
            // quiet mode: while the compute warps run a latency-bound task (attention), hold the weight
            // stream back so that their loads do not wait behind megabytes of queued weight traffic
            if (ok && P.quiet_streaming) {
              uint32_t polls = 0;
              while (*reinterpret_cast<volatile int *>(&c.s.flags[2]) != 0) {
                __nanosleep(100);
                if ((++polls & 0xff) == 0 && (ld_volatile_i32(&P.status->error) != 0 || globaltimer_ns() > c.deadline_ns)) break;
              }
            }
            if (ok) mbar_arrive_expect_tx(&c.s.full[s], (uint32_t)rows * seg_bytes);
          }
          ok = __shfl_sync(0xffffffffu, (int)ok, 0) != 0;
          if (!ok) break;
          if (lane < rows)
            bulk_g2s(c.s.stages + (size_t)s * P.stage_bytes + (size_t)lane * row_stride, src_row + (size_t)kc * esz,
                     seg_bytes, &c.s.full[s], policy);
          ++issued;
          if (++s == NST) { s = 0; ph ^= 1u; }
        }
      }
    }
    }
  }
  // Drain: every copy this warp issued must have landed before the CTA may exit.
  if (lane == 0) {
    const uint32_t pending = issued < (uint32_t)NST ? issued : (uint32_t)NST;
    for (uint32_t q = 0; q < pending; ++q) {
      if (--s < 0) { s = NST - 1; ph ^= 1u; }
      uint32_t polls = 0;
      while (!mbar_try_wait(&c.s.full[s], ph)) {
        if (++polls > (1u << 24)) break;   // copies in flight always complete; the bound only guards the loop
      }
    }
  }
  __syncwarp();
}

// ---------------------------------------------------------------------------
// TASK_LINEAR: weight-streaming skinny GEMM for up to 8 tokens on mma.sync m16n8k16
// (16 weight rows x 16 k per instruction, the tokens are the n dimension)
// ---------------------------------------------------------------------------
__device__ __forceinline__ int active_tokens(const KernelParams &P) {
  if (P.test_mode || P.meta.qo_indptr == nullptr) return P.max_num_batched_tokens;
  return __ldcg(&P.meta.qo_indptr[P.max_num_batched_requests]);
}

__device__ __forceinline__ void ldmatrix_x4(uint32_t (&r)[4], uint32_t smem_addr) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
               : "r"(smem_addr));
}
__device__ __forceinline__ void mma_bf16_16816(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
  asm volatile(
      "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
      : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}

// 16-bit sequence number of an allreduce instance: never 0 (a zeroed inbox is invalid).  Two instances carry the same
// number AND use the same inbox buffer when they are a multiple of 131070 (= lcm(65535, 2)) instances apart.  Rows
// [0, active tokens) of a buffer are rewritten by every instance that uses it, so only a token row that sat idle
// since exactly such an instance and becomes active again could show a consumer a stale word that passes the check.
// The batching task therefore clears the rows that go idle when the number of active tokens drops (run_batch; race
// free: every word of the finished iteration has been consumed, and peers push only rows below the new count), which
// leaves no stale sequence number behind.  Graphs without a batching task keep a fixed token count (test mode) or take
// it from the caller (online_notoken: a caller that shrinks and regrows the batch within 131070 / allreduces-per-
// iteration iterations of the same run is not covered).
__device__ __forceinline__ uint32_t ll_seq(unsigned long long iteration, int n_ar, int ar_idx) {
  return (uint32_t)((iteration * (unsigned long long)n_ar + (unsigned long long)ar_idx) % 65535ull) + 1u;
}

// fast silu: x * sigmoid(x) with ex2.approx based exp and approximate divide (error far below bf16 rounding)
__device__ __forceinline__ float silu_f(float x) { return __fdividef(x, 1.0f + __expf(-x)); }
// activations of hybrid graphs: float32 accuracy
__device__ __forceinline__ float silu_exact_f(float x) { return x / (1.0f + expf(-x)); }
__device__ __forceinline__ float gelu_tanh_f(float x) {
  return 0.5f * x * (1.0f + tanhf(0.7978845608028654f * (x + 0.044715f * x * x * x)));
}

// Stage the activation tile [B, KT] (bf16, rows padded by 16 bytes) for k range [k0, k0 + KT).
// `gpre` holds this thread's first two gamma vectors, loaded before the dependency wait.
// Address of 16-byte vector v (k elements 8v .. 8v + 7 of the tile) of token row b.  MODE 0 / 1: row-major rows
// padded by 16 bytes (mma.sync fragments); MODE 2 (FP8 linears): the tcgen05 operand layout -- blocks of 64 columns, each block
// [token rows][128 bytes] with the 16-byte chunks of a row XOR-swizzled by (row & 7) (128-byte swizzle, K-major).
template <int MODE>
__device__ __forceinline__ uint8_t *x_vec(uint8_t *xs, int b, int v, int xstride, int np) {
  if (MODE == 2)
    return xs + (size_t)(v >> 3) * (size_t)(np * 128) + (size_t)b * 128 + (size_t)(((v & 7) ^ (b & 7)) << 4);
  return xs + (size_t)b * xstride + (size_t)v * 16;
}

// Fused tensor-parallel allreduce, consumer side, with every rank's words of a vector requested before any of them
// is examined: a vector costs one L2 round trip (plus re-polls of the ranks that had not arrived) instead of one per
// rank.  Returns the thread's sum of squares over the vectors it wrote; `good` turns false when a wait ran out.
template <int MODE>
__device__ __forceinline__ float gather_row(const Ctx &c, const TaskDesc &d, const uint32_t *inbox, uint32_t seq, int b, int k0,
                                            int vec_per_row, int xstride, int np, bool &good) {
  const KernelParams &P = c.P;
  const int tid = threadIdx.x;
  const int K = d.a[L_K], slot = d.a[L_G_SLOT], W = P.world_size;
  const __nv_bfloat16 *res = reinterpret_cast<const __nv_bfloat16 *>(d.p[6]);
  __nv_bfloat16 *yout = reinterpret_cast<__nv_bfloat16 *>(d.p[7]);
  float ss = 0.f;
  for (int v = tid; v < vec_per_row && good; v += kConsumerThreads) {
    const uint32_t *wp = inbox + (size_t)b * K + k0 + v * 8;
    float acc[8];
#pragma unroll
    for (int e = 0; e < 8; ++e) acc[e] = 0.f;
    // four ranks per trip: their eight 16-byte loads are in flight together; the quad is re-read until all of it has
    // arrived and only then added, in rank order (every rank forms the same sum)
#pragma unroll
    for (int h = 0; h < kMaxWorld; h += 4) {
      if (h >= W) break;
      uint4 w0[4], w1[4];
      uint32_t polls = 0;
      while (true) {
        bool all = true;
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          if (h + i < W) {
            const uint32_t *q = wp + (size_t)(h + i) * slot;
            asm volatile("ld.relaxed.sys.global.v4.u32 {%0,%1,%2,%3}, [%4];"
                         : "=r"(w0[i].x), "=r"(w0[i].y), "=r"(w0[i].z), "=r"(w0[i].w) : "l"(q) : "memory");
            asm volatile("ld.relaxed.sys.global.v4.u32 {%0,%1,%2,%3}, [%4];"
                         : "=r"(w1[i].x), "=r"(w1[i].y), "=r"(w1[i].z), "=r"(w1[i].w) : "l"(q + 4) : "memory");
          }
        }
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          if (h + i < W)
            all = all && (w0[i].x >> 16) == seq && (w0[i].y >> 16) == seq && (w0[i].z >> 16) == seq && (w0[i].w >> 16) == seq &&
                  (w1[i].x >> 16) == seq && (w1[i].y >> 16) == seq && (w1[i].z >> 16) == seq && (w1[i].w >> 16) == seq;
        }
        if (all) break;
        if ((++polls & 0x3f) == 0) {
          if (ld_volatile_i32(&P.status->error) != 0) { good = false; break; }
          if (globaltimer_ns() > c.deadline_ns) {
            report_timeout(P.status, c.worker, 3, h);
            good = false;
            break;
          }
        }
      }
      if (!good) break;
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        if (h + i < W) {
          const uint32_t ww[8] = {w0[i].x, w0[i].y, w0[i].z, w0[i].w, w1[i].x, w1[i].y, w1[i].z, w1[i].w};
#pragma unroll
          for (int e = 0; e < 8; ++e) acc[e] += __uint_as_float(ww[e] << 16);
        }
      }
    }
    if (!good) break;
    if (res) {
      const uint4 rv = __ldcg(reinterpret_cast<const uint4 *>(res + (size_t)b * d.a[L_G_LDRES] + k0) + v);
      const uint32_t rw[4] = {rv.x, rv.y, rv.z, rv.w};
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        acc[2 * q] += bf16_lo(rw[q]);
        acc[2 * q + 1] += bf16_hi(rw[q]);
      }
    }
    uint32_t ow[4];
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      ow[q] = pack_bf16(acc[2 * q], acc[2 * q + 1]);
      const float a = bf16_lo(ow[q]), e = bf16_hi(ow[q]);
      ss += a * a + e * e;
    }
    const uint4 o4 = make_uint4(ow[0], ow[1], ow[2], ow[3]);
    *reinterpret_cast<uint4 *>(x_vec<MODE>(c.s.xtile, b, v, xstride, np)) = o4;
    reinterpret_cast<uint4 *>(yout + (size_t)b * d.a[L_G_LDOUT] + k0)[v] = o4;
  }
  return ss;
}

// PRO_RESNORM (hybrid graphs of a few tokens): the stream's residual sum and both norms in the consumer's prologue.  Every
// task of the layer computes the same rows and writes the same values to x_out, which is another buffer than x.
static __device__ __noinline__ void stage_resnorm(const Ctx c, const TaskDesc &d, int B) {
  constexpr int NV = 4;   // rows of at most 4096 columns, in registers
  const int tid = threadIdx.x, W = d.a[L_GROUPS], K = d.a[L_K], warp = tid >> 5;
  const bool layer_norm = (d.a[L_G_SLOT] & 4) != 0;
  const float eps = __int_as_float(d.a[L_EPS]), off = (d.a[L_G_SLOT] & 2) ? 1.0f : 0.0f, factor = __int_as_float(d.a[LR_POST]);
  const float *add = *reinterpret_cast<const float *const *>(&d.a[LR_ADD]);
  const uint64_t rowp = *reinterpret_cast<const uint64_t *>(&d.a[LR_ROW]);
  const bool has_y = d.p[6] != 0, has_post = d.p[3] != 0, moved = has_y || add != nullptr || rowp != 0, average = (d.a[L_G_SLOT] & 8) != 0;
  const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f);
  auto values = [&](uint64_t base, int j, float o) {
    const uint2 v = __ldg(reinterpret_cast<const uint2 *>(base + 2ull * j));
    return make_float4(o + bf16_lo(v.x), o + bf16_hi(v.x), o + bf16_lo(v.y), o + bf16_hi(v.y));
  };
  auto total = [&](float v, float *slots) {
    v = warp_sum(v);
    if ((tid & 31) == 0) slots[warp] = v;
    consumer_sync();
    float t = 0.f;
#pragma unroll
    for (int w = 0; w < 8; ++w) t += slots[w];
    return t;
  };
  for (int b = 0; b < B; ++b) {
    const float *x = reinterpret_cast<const float *>(d.p[1]) + (size_t)b * d.a[L_LDX];
    const float *y = reinterpret_cast<const float *>(d.p[6]) + (size_t)b * d.a[L_G_LDRES];
    float *xo = reinterpret_cast<float *>(d.p[7]) + (size_t)b * d.a[L_G_LDOUT];
    float4 xv[NV], yv[NV], wp[NV], wn[NV];
#pragma unroll
    for (int i = 0; i < NV; ++i) {
      const int j = (i * kConsumerThreads + tid) * 4;
      const bool in = j < W;
      yv[i] = in && has_y ? __ldcg(reinterpret_cast<const float4 *>(y + j)) : zero;
      xv[i] = in ? __ldcg(reinterpret_cast<const float4 *>(x + j)) : zero;
      wp[i] = in && has_post ? values(d.p[3], j, off) : make_float4(1.f, 1.f, 1.f, 1.f);
      wn[i] = !in ? zero : d.p[4] != 0 ? values(d.p[4], j, off) : make_float4(1.f, 1.f, 1.f, 1.f);
    }
    if (has_y) {
      float inv = 1.f;
      if (has_post) {
        float ss = 0.f;
#pragma unroll
        for (int i = 0; i < NV; ++i) ss += yv[i].x * yv[i].x + yv[i].y * yv[i].y + yv[i].z * yv[i].z + yv[i].w * yv[i].w;
        inv = factor / sqrtf(total(ss, c.s.red) / (float)W + eps);
      }
#pragma unroll
      for (int i = 0; i < NV; ++i) {
        xv[i].x += yv[i].x * inv * wp[i].x; xv[i].y += yv[i].y * inv * wp[i].y;
        xv[i].z += yv[i].z * inv * wp[i].z; xv[i].w += yv[i].w * inv * wp[i].w;
      }
    }
    if (average) {
      float *res = const_cast<float *>(add) + (size_t)b * W;
      const int last = d.a[L_LDR] - 1, step = d.a[LR_LDADD];
      auto weight = [&](int k) { return bf16_to_f(__ldg(reinterpret_cast<const __nv_bfloat16 *>(rowp) + k)); };
      const float wl = weight(last);
#pragma unroll
      for (int i = 0; i < NV; ++i) {
        const int j = (i * kConsumerThreads + tid) * 4;
        if (j < W) *reinterpret_cast<float4 *>(res + (size_t)last * step + j) = xv[i];
        xv[i].x *= wl; xv[i].y *= wl; xv[i].z *= wl; xv[i].w *= wl;
      }
      for (int k = 0; k < last; k += 2) {   // two results in flight
        float4 e[2][NV];
#pragma unroll
        for (int u = 0; u < 2; ++u)
#pragma unroll
          for (int i = 0; i < NV; ++i) {
            const int j = (i * kConsumerThreads + tid) * 4;
            e[u][i] = j < W && k + u < last ? __ldcg(reinterpret_cast<const float4 *>(res + (size_t)(k + u) * step + j)) : zero;
          }
#pragma unroll
        for (int u = 0; u < 2; ++u) {
          const float wk = k + u < last ? weight(k + u) : 0.f;
#pragma unroll
          for (int i = 0; i < NV; ++i) {
            xv[i].x = fmaf(wk, e[u][i].x, xv[i].x); xv[i].y = fmaf(wk, e[u][i].y, xv[i].y);
            xv[i].z = fmaf(wk, e[u][i].z, xv[i].z); xv[i].w = fmaf(wk, e[u][i].w, xv[i].w);
          }
        }
      }
    } else if (add != nullptr || rowp != 0) {
#pragma unroll
      for (int i = 0; i < NV; ++i) {
        const int j = (i * kConsumerThreads + tid) * 4;
        if (j >= W) continue;
        const float4 a = add != nullptr ? __ldcg(reinterpret_cast<const float4 *>(add + (size_t)b * d.a[LR_LDADD] + j)) : zero;
        const float4 r = rowp != 0 ? values(rowp, j, 0.f) : zero;
        xv[i].x = xv[i].x + a.x + r.x; xv[i].y = xv[i].y + a.y + r.y; xv[i].z = xv[i].z + a.z + r.z; xv[i].w = xv[i].w + a.w + r.w;
      }
    }
    if (moved && d.p[7] != 0) {
#pragma unroll
      for (int i = 0; i < NV; ++i) {
        const int j = (i * kConsumerThreads + tid) * 4;
        if (j < W) *reinterpret_cast<float4 *>(xo + j) = xv[i];
      }
    }
    if (layer_norm) {
      float s = 0.f;
#pragma unroll
      for (int i = 0; i < NV; ++i) s += xv[i].x + xv[i].y + xv[i].z + xv[i].w;
      const float mean = total(s, c.s.red + 16) / (float)W;
#pragma unroll
      for (int i = 0; i < NV; ++i)
        if ((i * kConsumerThreads + tid) * 4 < W) { xv[i].x -= mean; xv[i].y -= mean; xv[i].z -= mean; xv[i].w -= mean; }
    }
    float inv = 1.f;   // (no norm weight: the stream as it is)
    if (d.p[4] != 0) {
      float ss = 0.f;
#pragma unroll
      for (int i = 0; i < NV; ++i) ss += xv[i].x * xv[i].x + xv[i].y * xv[i].y + xv[i].z * xv[i].z + xv[i].w * xv[i].w;
      inv = 1.0f / sqrtf(total(ss, c.s.red + 8) / (float)W + eps);
    }
    uint8_t *row = c.s.xtile + (size_t)b * (K * 2 + kRowPadBytes);
#pragma unroll
    for (int i = 0; i < NV; ++i) {   // (the padding columns behind the row come out as zeros)
      const int j = (i * kConsumerThreads + tid) * 4;
      const float4 bias = d.p[5] != 0 && j < W ? values(d.p[5], j, 0.f) : zero;
      if (j < K)
        *reinterpret_cast<uint2 *>(row + 2 * j) =
            make_uint2(pack_bf16(xv[i].x * inv * wn[i].x + bias.x, xv[i].y * inv * wn[i].y + bias.y),
                       pack_bf16(xv[i].z * inv * wn[i].z + bias.z, xv[i].w * inv * wn[i].w + bias.w));
    }
    consumer_sync();   // (also: the reduction slots are used again)
  }
}

// PRO_POLY (hybrid_tasks.cuh).
static __device__ __noinline__ void stage_poly(const Ctx c, const TaskDesc &d, int B);

// Copies B rows of `vecs` 16-byte vectors into the activation tile, one warp per row, every copy in flight.  A function of its own:
// at the register cap of the linear bodies its loop would reload spilled variables for each copy.
static __device__ __noinline__ void stage_rows(uint32_t xs, const uint4 *src, int ld, int B, int vecs, int xstride) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  for (int b = warp; b < B; b += 8) {
    const uint4 *row = src + (size_t)b * ld;
    const uint32_t dst = xs + b * xstride + lane * 16;
#pragma unroll 4
    for (int v = lane; v < vecs; v += 32)
      asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst + (uint32_t)(v - lane) * 16u), "l"(row + v) : "memory");
  }
  asm volatile("cp.async.commit_group;" ::: "memory");
  asm volatile("cp.async.wait_group 0;" ::: "memory");
}

template <int MODE, bool TPX = false>
__device__ void stage_x(const Ctx &c, const TaskDesc &d, int B, int k0, int KT, const uint4 (&gpre)[2]) {
  constexpr bool WIDE = MODE != 0;
  const int np = c.P.tc_tokens;
  const int tid = threadIdx.x;
  const int K = d.a[L_K];
  const int ldx = d.a[L_LDX];
  const int pro = d.a[L_PRO];
  const int vec_per_row = KT / 8;
  const int xstride = KT * 2 + kRowPadBytes;   // bytes
  uint8_t *xs = c.s.xtile;
  // per-token, per-warp sums of squares: 8 x 8 floats, or up to 64 x 8 in the partial-sum area (idle while the
  // activation tile is staged)
  float *red = WIDE ? c.s.partial : c.s.red;
  const __nv_bfloat16 *src = reinterpret_cast<const __nv_bfloat16 *>(d.p[1]);
  if (d.a[L_GATHER] > 0) {
    // Fused tensor-parallel allreduce: every rank pushed {bf16 partial, sequence} words for this allreduce
    // instance into our inbox.  Poll until all words of a vector carry the expected sequence number, sum the
    // ranks in rank order in fp32, add the residual, round once: that is the reduced activation row.  It is
    // staged in shared memory for this task and written to its tensor (every task writes the same values).
    const KernelParams &P = c.P;
    const int ar = d.a[L_GATHER] - 1;
    const unsigned long long inst = c.iteration * (unsigned)d.a[L_NAR] + (unsigned)ar;
    const uint32_t seq = ll_seq(c.iteration, d.a[L_NAR], ar);
    const uint32_t *inbox = reinterpret_cast<const uint32_t *>(P.peer_inbox[P.rank]) + (size_t)d.p[5] +
                            (size_t)(inst & 1ull) * (size_t)d.a[L_PARSTRIDE];
    const __nv_bfloat16 *res = reinterpret_cast<const __nv_bfloat16 *>(d.p[6]);
    __nv_bfloat16 *yout = reinterpret_cast<__nv_bfloat16 *>(d.p[7]);
    const int slot = d.a[L_G_SLOT];
    const int warp = tid >> 5, lane = tid & 31;
    bool good = true;
    for (int b = 0; b < B; ++b) {
      float ss = 0.f;
      if (TPX && MODE == 0) ss = gather_row<MODE>(c, d, inbox, seq, b, k0, vec_per_row, xstride, np, good);
      for (int v = tid; !(TPX && MODE == 0) && v < vec_per_row; v += kConsumerThreads) {
        float acc[8];
#pragma unroll
        for (int e = 0; e < 8; ++e) acc[e] = 0.f;
        for (int r = 0; r < P.world_size; ++r) {
          const uint32_t *wp = inbox + (size_t)r * slot + (size_t)b * K + k0 + v * 8;
          uint4 w0, w1;
          uint32_t polls = 0;
          while (true) {
            asm volatile("ld.relaxed.sys.global.v4.u32 {%0,%1,%2,%3}, [%4];"
                         : "=r"(w0.x), "=r"(w0.y), "=r"(w0.z), "=r"(w0.w) : "l"(wp) : "memory");
            asm volatile("ld.relaxed.sys.global.v4.u32 {%0,%1,%2,%3}, [%4];"
                         : "=r"(w1.x), "=r"(w1.y), "=r"(w1.z), "=r"(w1.w) : "l"(wp + 4) : "memory");
            const bool ok8 = (w0.x >> 16) == seq && (w0.y >> 16) == seq && (w0.z >> 16) == seq && (w0.w >> 16) == seq &&
                             (w1.x >> 16) == seq && (w1.y >> 16) == seq && (w1.z >> 16) == seq && (w1.w >> 16) == seq;
            if (ok8) break;
            if ((++polls & 0xff) == 0) {
              if (ld_volatile_i32(&P.status->error) != 0) { good = false; break; }
              if (globaltimer_ns() > c.deadline_ns) {
                report_timeout(P.status, c.worker, 3, r);
                good = false;
                break;
              }
            }
          }
          if (!good) break;
          const uint32_t ww[8] = {w0.x, w0.y, w0.z, w0.w, w1.x, w1.y, w1.z, w1.w};
#pragma unroll
          for (int e = 0; e < 8; ++e) acc[e] += __uint_as_float(ww[e] << 16);
        }
        uint32_t ow[4];
        if (res) {
          const uint4 rv = __ldcg(reinterpret_cast<const uint4 *>(res + (size_t)b * d.a[L_G_LDRES] + k0) + v);
          const uint32_t rw[4] = {rv.x, rv.y, rv.z, rv.w};
#pragma unroll
          for (int q = 0; q < 4; ++q) {
            acc[2 * q] += bf16_lo(rw[q]);
            acc[2 * q + 1] += bf16_hi(rw[q]);
          }
        }
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          ow[q] = pack_bf16(acc[2 * q], acc[2 * q + 1]);
          const float a = bf16_lo(ow[q]), e = bf16_hi(ow[q]);
          ss += a * a + e * e;
        }
        const uint4 o4 = make_uint4(ow[0], ow[1], ow[2], ow[3]);
        *reinterpret_cast<uint4 *>(x_vec<MODE>(xs, b, v, xstride, np)) = o4;
        reinterpret_cast<uint4 *>(yout + (size_t)b * d.a[L_G_LDOUT] + k0)[v] = o4;
      }
      if (!WIDE || pro == PRO_RMSNORM) {   // (whole row staged: the partial-sum area is not holding sums of a previous k tile)
        ss = warp_sum(ss);
        if (lane == 0) red[b * 8 + warp] = ss;
      }
    }
    if (!good) c.s.flags[0] = 1;
    consumer_sync();
    if (pro != PRO_RMSNORM) return;
    const float eps = __int_as_float(d.a[L_EPS]);
    const __nv_bfloat16 *gam = reinterpret_cast<const __nv_bfloat16 *>(d.p[4]);
    for (int b = 0; b < B; ++b) {
      float tot = 0.f;
#pragma unroll
      for (int w = 0; w < 8; ++w) tot += red[b * 8 + w];
      const float inv = rsqrtf(tot / (float)K + eps);
      int it = 0;
      for (int v = tid; v < vec_per_row; v += kConsumerThreads, ++it) {
        uint4 *xp = reinterpret_cast<uint4 *>(x_vec<MODE>(xs, b, v, xstride, np));
        const uint4 xv = *xp;
        const uint4 gv = (it < 2) ? gpre[it] : __ldg(reinterpret_cast<const uint4 *>(gam + k0) + v);
        const uint32_t xw[4] = {xv.x, xv.y, xv.z, xv.w};
        const uint32_t gw[4] = {gv.x, gv.y, gv.z, gv.w};
        uint32_t ow[4];
#pragma unroll
        for (int q = 0; q < 4; ++q)
          ow[q] = pack_bf16(bf16_lo(xw[q]) * inv * bf16_lo(gw[q]), bf16_hi(xw[q]) * inv * bf16_hi(gw[q]));
        *xp = make_uint4(ow[0], ow[1], ow[2], ow[3]);
      }
    }
    consumer_sync();
    return;
  }
  if (pro == PRO_SILU_MUL) {
    const int groups = d.a[L_GROUPS];
    const int per = K / groups;   // activation columns per interleave group
    for (int b = 0; b < B; ++b) {
      for (int v = tid; v < vec_per_row; v += kConsumerThreads) {
        const int j = k0 + v * 8;
        const int g = j / per, off = j - g * per;
        const __nv_bfloat16 *gp = src + (size_t)b * ldx + (size_t)g * 2 * per + off;
        const uint4 gv = __ldcg(reinterpret_cast<const uint4 *>(gp));
        const uint4 uv = __ldcg(reinterpret_cast<const uint4 *>(gp + per));
        const uint32_t gw[4] = {gv.x, gv.y, gv.z, gv.w};
        const uint32_t uw[4] = {uv.x, uv.y, uv.z, uv.w};
        uint32_t ow[4];
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          const float a0 = round_bf16(silu_f(bf16_lo(gw[q])));
          const float a1 = round_bf16(silu_f(bf16_hi(gw[q])));
          ow[q] = pack_bf16(a0 * bf16_lo(uw[q]), a1 * bf16_hi(uw[q]));
        }
        *reinterpret_cast<uint4 *>(x_vec<MODE>(xs, b, v, xstride, np)) = make_uint4(ow[0], ow[1], ow[2], ow[3]);
      }
    }
    consumer_sync();
    return;
  }
  if (WIDE && (pro == PRO_PLAIN || pro == PRO_RMSNORM)) {
    // many tokens: asynchronous 16-byte copies straight into shared memory (all in flight, no registers held)
    stage_rows(smem_u32(xs), reinterpret_cast<const uint4 *>(src + k0), ldx >> 3, B, vec_per_row, xstride);
    consumer_sync();
    if (pro == PRO_PLAIN) return;
    // RMSNorm in place.  Pass 1: one warp per token sums the squares and leaves 1 / rms in shared memory.  Pass 2:
    // a thread owns vector positions v = tid, tid + 256, ... of EVERY token, so that gamma (fetched before the
    // dependency wait for the first two positions) sits in registers and no global load is left in the loop.
    const int warp = tid >> 5, lane = tid & 31;
    const float eps = __int_as_float(d.a[L_EPS]);
    const __nv_bfloat16 *gam = reinterpret_cast<const __nv_bfloat16 *>(d.p[4]);
    for (int b = warp; b < B; b += 8) {
      float ss = 0.f;
      for (int v = lane; v < vec_per_row; v += 32) {
        const uint4 xv = *reinterpret_cast<const uint4 *>(x_vec<MODE>(xs, b, v, xstride, np));
        const uint32_t w[4] = {xv.x, xv.y, xv.z, xv.w};
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          const float a = bf16_lo(w[q]), e = bf16_hi(w[q]);
          ss += a * a + e * e;
        }
      }
      ss = warp_sum(ss);
      if (lane == 0) red[b] = rsqrtf(ss / (float)K + eps);
    }
    consumer_sync();
    int it = 0;
    for (int v = tid; v < vec_per_row; v += kConsumerThreads, ++it) {
      const uint4 gv = (it < 2) ? gpre[it] : __ldg(reinterpret_cast<const uint4 *>(gam + k0) + v);
      const uint32_t gw[4] = {gv.x, gv.y, gv.z, gv.w};
      float gf[8];
#pragma unroll
      for (int q = 0; q < 4; ++q) { gf[2 * q] = bf16_lo(gw[q]); gf[2 * q + 1] = bf16_hi(gw[q]); }
#pragma unroll 4
      for (int b = 0; b < B; ++b) {
        const float inv = red[b];
        uint4 *xp = reinterpret_cast<uint4 *>(x_vec<MODE>(xs, b, v, xstride, np));
        const uint4 xv = *xp;
        const uint32_t xw[4] = {xv.x, xv.y, xv.z, xv.w};
        uint32_t ow[4];
#pragma unroll
        for (int q = 0; q < 4; ++q)
          ow[q] = pack_bf16(bf16_lo(xw[q]) * inv * gf[2 * q], bf16_hi(xw[q]) * inv * gf[2 * q + 1]);
        *xp = make_uint4(ow[0], ow[1], ow[2], ow[3]);
      }
    }
    consumer_sync();
    return;
  }
  if (pro != PRO_RMSNORM) {
    for (int b = 0; b < B; ++b)
      for (int v = tid; v < vec_per_row; v += kConsumerThreads)
        *reinterpret_cast<uint4 *>(x_vec<MODE>(xs, b, v, xstride, np)) =
            __ldcg(reinterpret_cast<const uint4 *>(src + (size_t)b * ldx + k0) + v);
    consumer_sync();
    return;
  }
  // RMSNorm over the full row (the builder guarantees KT == K for this prologue).
  const int warp = tid >> 5, lane = tid & 31;
  for (int b = 0; b < B; ++b) {
    float ss = 0.f;
    for (int v = tid; v < vec_per_row; v += kConsumerThreads) {
      const uint4 xv = __ldcg(reinterpret_cast<const uint4 *>(src + (size_t)b * ldx + k0) + v);
      *reinterpret_cast<uint4 *>(x_vec<MODE>(xs, b, v, xstride, np)) = xv;
      const uint32_t w[4] = {xv.x, xv.y, xv.z, xv.w};
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        const float a = bf16_lo(w[q]), e = bf16_hi(w[q]);
        ss += a * a + e * e;
      }
    }
    ss = warp_sum(ss);
    if (lane == 0) red[b * 8 + warp] = ss;
  }
  consumer_sync();
  const float eps = __int_as_float(d.a[L_EPS]);
  const __nv_bfloat16 *gam = reinterpret_cast<const __nv_bfloat16 *>(d.p[4]);
  for (int b = 0; b < B; ++b) {
    float tot = 0.f;
#pragma unroll
    for (int w = 0; w < 8; ++w) tot += red[b * 8 + w];
    const float inv = rsqrtf(tot / (float)K + eps);
    int it = 0;
    for (int v = tid; v < vec_per_row; v += kConsumerThreads, ++it) {
      uint4 *xp = reinterpret_cast<uint4 *>(x_vec<MODE>(xs, b, v, xstride, np));
      const uint4 xv = *xp;
      const uint4 gv = (it < 2) ? gpre[it] : __ldg(reinterpret_cast<const uint4 *>(gam + k0) + v);
      const uint32_t xw[4] = {xv.x, xv.y, xv.z, xv.w};
      const uint32_t gw[4] = {gv.x, gv.y, gv.z, gv.w};
      uint32_t ow[4];
#pragma unroll
      for (int q = 0; q < 4; ++q)
        ow[q] = pack_bf16(bf16_lo(xw[q]) * inv * bf16_lo(gw[q]), bf16_hi(xw[q]) * inv * bf16_hi(gw[q]));
      *xp = make_uint4(ow[0], ow[1], ow[2], ow[3]);
    }
  }
  consumer_sync();
}

// Sum the 8 warps' partial tiles of one 16-row group and run the epilogue for its rows.
// WIDE = false: at most 8 tokens, every warp holds the same token tile (the batch-1 hot path, all constants);
// WIDE = true: warp w holds token tile w % NT (8 tokens each) and every (8 / NT)-th k step.
template <bool WIDE, int HYB>
__device__ __forceinline__ void linear_output(const Ctx &c, const TaskDesc &d, int NT, int r0, int rows,
                                              const float *part, int item);

template <bool WIDE, int HYB>
__device__ __forceinline__ void linear_group_epilogue(const Ctx &c, const TaskDesc &d, int B, int NT, int r0, int rows,
                                                      const float *part) {
  if (!WIDE) {
    const int tid = threadIdx.x;
    if (tid < 128 && (tid >> 4) < B) linear_output<false, HYB>(c, d, 1, r0, rows, part, tid);
  } else {
    for (int item = threadIdx.x; item < B * 16; item += kConsumerThreads) linear_output<true, HYB>(c, d, NT, r0, rows, part, item);
  }
}

template <bool WIDE, int HYB>
__device__ __forceinline__ void linear_output(const Ctx &c, const TaskDesc &d, int NT, int r0, int rows,
                                              const float *part, int item) {
  const KernelParams &P = c.P;
  const int b = item >> 4, r = item & 15;
  if (r >= rows) return;
  float v = 0.f;
  if (WIDE) {
    for (int w = b >> 3; w < 8; w += NT) v += part[(w * 16 + r) * 8 + (b & 7)];
  } else {
#pragma unroll
    for (int w = 0; w < 8; ++w) v += part[(w * 16 + r) * 8 + b];
  }
  const int epi = d.a[L_EPI];
  const int col = r0 + r;
  if (epi == EPI_PUSH_LL) {
    // one 32-bit word per element: bf16 partial sum in the low half, sequence number in the high half
    const int N = d.a[L_N];
    const unsigned long long inst = c.iteration * (unsigned)d.a[L_NAR] + (unsigned)d.a[L_ARIDX];
    const size_t off = (size_t)d.p[5] + (size_t)(inst & 1ull) * (size_t)d.a[L_PARSTRIDE] +
                       (size_t)P.rank * (size_t)d.a[L_SLOT] + (size_t)b * N + col;
    const __nv_bfloat16 hv = __float2bfloat16_rn(v);
    const uint32_t word = (uint32_t)(*reinterpret_cast<const unsigned short *>(&hv)) |
                          (ll_seq(c.iteration, d.a[L_NAR], d.a[L_ARIDX]) << 16);
    for (int peer = 0; peer < P.world_size; ++peer)
      asm volatile("st.relaxed.sys.global.u32 [%0], %1;" ::"l"(reinterpret_cast<uint32_t *>(P.peer_inbox[peer]) + off),
                   "r"(word)
                   : "memory");
  } else if (epi == EPI_PUSH_F32) {
    const int N = d.a[L_N];
    const size_t parity = (size_t)((c.iteration * (unsigned)d.a[L_NAR] + (unsigned)d.a[L_ARIDX]) & 1ull);
    const size_t off = (size_t)d.p[5] + parity * (size_t)d.a[L_PARSTRIDE] + (size_t)P.rank * (size_t)d.a[L_SLOT] +
                       (size_t)b * N + col;
    for (int peer = 0; peer < P.world_size; ++peer) P.peer_inbox[peer][off] = v;
  } else if (epi == EPI_SILU_PAIR) {
    // rows come as [gate, gate, up, up]: the threads on gate rows finish the pair
    if ((r & 2) == 0) {
      float u = 0.f;
      if (WIDE) {
        for (int w = b >> 3; w < 8; w += NT) u += part[(w * 16 + r + 2) * 8 + (b & 7)];
      } else {
#pragma unroll
        for (int w = 0; w < 8; ++w) u += part[(w * 16 + r + 2) * 8 + b];
      }
      const float gv = round_bf16(v);
      const float a = round_bf16(silu_f(gv));
      __nv_bfloat16 *out = reinterpret_cast<__nv_bfloat16 *>(d.p[2]);
      out[(size_t)b * d.a[L_LDO] + ((col >> 2) << 1) + (r & 1)] = __float2bfloat16_rn(a * round_bf16(u));
    }
  } else if (HYB && epi == EPI_STORE_F32) {
    reinterpret_cast<float *>(d.p[2])[(size_t)b * d.a[L_LDO] + col] = v;
  } else if (HYB && epi == EPI_BIAS_F32) {
    const __nv_bfloat16 *bias = *reinterpret_cast<const __nv_bfloat16 *const *>(&d.a[LR_BIAS]);
    reinterpret_cast<float *>(d.p[2])[(size_t)b * d.a[L_LDO] + col] = v + bf16_to_f(__ldg(bias + col));
  } else if (HYB && epi == EPI_RELU2) {
    const float a = fmaxf(v, 0.f);
    reinterpret_cast<__nv_bfloat16 *>(d.p[2])[(size_t)b * d.a[L_LDO] + col] = __float2bfloat16_rn(a * a);
  } else if (HYB && epi == EPI_SOFTCAP) {
    const float cap = __int_as_float(d.a[L_CAP]);
    reinterpret_cast<float *>(d.p[2])[(size_t)b * d.a[L_LDO] + col] = cap * tanhf(v / cap);
  } else if (HYB && epi == EPI_SCALE_F32) {
    reinterpret_cast<float *>(d.p[2])[(size_t)b * d.a[L_LDO] + col] = __int_as_float(d.a[L_CAP]) * v;
  } else if (HYB && epi == EPI_GATE_SIGMOID) {
    const float g = __ldcg(reinterpret_cast<const float *>(d.p[3]) + (size_t)b * d.a[L_LDR] + col);
    reinterpret_cast<__nv_bfloat16 *>(d.p[2])[(size_t)b * d.a[L_LDO] + col] = __float2bfloat16_rn(v / (1.0f + expf(-g)));
  } else if (HYB && (epi == EPI_GATED_SILU || epi == EPI_GATED_GELU)) {
    if ((r & 2) == 0) {
      float u = 0.f;
      if (WIDE) {
        for (int w = b >> 3; w < 8; w += NT) u += part[(w * 16 + r + 2) * 8 + (b & 7)];
      } else {
#pragma unroll
        for (int w = 0; w < 8; ++w) u += part[(w * 16 + r + 2) * 8 + b];
      }
      const float a = epi == EPI_GATED_SILU ? silu_exact_f(v) : gelu_tanh_f(v);
      reinterpret_cast<__nv_bfloat16 *>(d.p[2])[(size_t)b * d.a[L_LDO] + ((col >> 2) << 1) + (r & 1)] = __float2bfloat16_rn(a * u);
    }
  } else {
    __nv_bfloat16 *out = reinterpret_cast<__nv_bfloat16 *>(d.p[2]);
    if (epi == EPI_RESIDUAL) {
      const __nv_bfloat16 *res = reinterpret_cast<const __nv_bfloat16 *>(d.p[3]);
      v += bf16_to_f(__ldcg(&res[(size_t)b * d.a[L_LDR] + col]));
    }
    out[(size_t)b * d.a[L_LDO] + col] = __float2bfloat16_rn(v);
  }
}

template <bool WIDE, bool TPX = false, int HYB = 0>
__device__ __forceinline__ void run_linear(const Ctx &c, const TaskDesc &d, LinearState &ls, int task,
                                           const uint4 (&gpre)[2], bool ok) {
  const KernelParams &P = c.P;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int B = ok ? min(active_tokens(P), WIDE ? kMaxLinearTokens : 8) : 0;
  const int NT = !WIDE || B <= 8 ? 1 : (B <= 16 ? 2 : (B <= 32 ? 4 : 8));   // token tiles of 8
  const int nt = WIDE ? warp % NT : 0, ks = WIDE ? warp / NT : warp, kstride = WIDE ? 8 / NT : 8;
  const int n0 = d.a[L_N0], n1 = d.a[L_N1], K = d.a[L_K];
  const int KT = d.a[L_KT], KC = d.a[L_KC], R = d.a[L_ROWS];
  const int NST = P.num_stages;
  const int steps = KC / 16;
  const uint32_t row_stride = (uint32_t)KC * 2u + kRowPadBytes;
  const uint32_t xstride = (uint32_t)KT * 2u + kRowPadBytes;
  const int g = lane >> 2, q = lane & 3;
  const bool tok_valid = nt * 8 + g < B;
  const bool multi_tile = KT < K;          // accumulate across k tiles in shared memory (task has <= 2 groups)
  // lanes 0-15 address the 16 rows of the m-tile; with 8-row chunks rows 8-15 alias rows 0-7 (their results are unused)
  const uint32_t a_lane_off = (uint32_t)(lane & (R - 1)) * row_stride + (uint32_t)(lane >> 4) * 16u;
  const uint32_t x_lane_base =
      smem_u32(c.s.xtile) + (uint32_t)(tok_valid ? nt * 8 + g : 0) * xstride + (uint32_t)q * 4u;
  const bool prof = P.profiler != nullptr && (uint64_t)(task + 1) * 8 <= P.profiler_entries;
  int group_seq = 0;
  int nchunk = 0;
  for (int kt = 0; kt < K; kt += KT) {
    if (B > 0 && !((d.flags & TF_SAME_X_AS_PREV) && !multi_tile)) {
      if (kt > 0) consumer_sync();   // everyone is done reading the previous tile
      if (HYB && !WIDE && d.a[L_PRO] == PRO_RESNORM) stage_resnorm(c, d, B);
      else if (HYB && !WIDE && d.a[L_PRO] == PRO_POLY) stage_poly(c, d, B);
      else stage_x<WIDE ? 1 : 0, TPX>(c, d, B, kt, KT, gpre);
    }
    if (tid == 0 && prof && kt == 0) P.profiler[(size_t)task * 8 + 4] = globaltimer_ns();
    int gi = 0;
    for (int r0 = n0; r0 < n1; r0 += R, ++gi) {
      float acc[4] = {0.f, 0.f, 0.f, 0.f};
      float acc2[4] = {0.f, 0.f, 0.f, 0.f};   // second accumulator chain: back-to-back mma do not serialise
      for (int kc = 0; kc < KT; kc += KC) {
        const int s = ls.stage;
        const uint32_t ph = ls.phase;
        if (++ls.stage == NST) { ls.stage = 0; ls.phase ^= 1u; }
        if (ok) ok = wait_mbar(c, &c.s.full[s], ph, task);
        if (ok && B > 0) {
          const uint32_t a_base = smem_u32(c.s.stages + (size_t)s * P.stage_bytes) + a_lane_off;
          const uint32_t x_base = x_lane_base + (uint32_t)kc * 2u;
          // this warp's k steps are warp, warp + 8, ...; fetch the fragments of four steps, then issue their mma
          const int nj = WIDE ? (steps - ks + kstride - 1) / kstride : (steps - warp + 7) >> 3;
          for (int j0 = 0; j0 < nj; j0 += 4) {
            uint32_t a[4][4], b[4][2];
#pragma unroll
            for (int u = 0; u < 4; ++u) {
              if (j0 + u < nj) {
                const uint32_t o = (uint32_t)(ks + kstride * (j0 + u)) * 32u;
                ldmatrix_x4(a[u], a_base + o);
                asm volatile("ld.shared.b32 %0, [%1];" : "=r"(b[u][0]) : "r"(x_base + o));
                asm volatile("ld.shared.b32 %0, [%1];" : "=r"(b[u][1]) : "r"(x_base + o + 16u));
              }
            }
#pragma unroll
            for (int u = 0; u < 4; ++u) {
              if (j0 + u < nj) {
                if (!tok_valid) b[u][0] = b[u][1] = 0u;   // token columns beyond the batch contribute nothing
                if (u & 1) mma_bf16_16816(acc2, a[u], b[u][0], b[u][1]);
                else mma_bf16_16816(acc, a[u], b[u][0], b[u][1]);
              }
            }
          }
        }
        __syncwarp();
        if (lane == 0) mbar_arrive(&c.s.empty[s]);
        if (tid == 0 && prof) {
          ++nchunk;
          if (nchunk == 1) P.profiler[(size_t)task * 8 + 6] = globaltimer_ns();
          if (nchunk == 6) P.profiler[(size_t)task * 8 + 7] = globaltimer_ns();
        }
      }
      if (B > 0) {
#pragma unroll
        for (int i = 0; i < 4; ++i) acc[i] += acc2[i];
        // this warp's 16 x 8 partial tile -> shared memory
        float *part = c.s.partial + (size_t)((multi_tile ? gi : group_seq) & 1) * (8 * 16 * 8);
        float *mine = part + (size_t)warp * (16 * 8);
        float2 *p0 = reinterpret_cast<float2 *>(mine + g * 8 + q * 2);
        float2 *p1 = reinterpret_cast<float2 *>(mine + (g + 8) * 8 + q * 2);
        if (multi_tile && kt > 0) {
          float2 o0 = *p0, o1 = *p1;
          *p0 = make_float2(o0.x + acc[0], o0.y + acc[1]);
          *p1 = make_float2(o1.x + acc[2], o1.y + acc[3]);
        } else {
          *p0 = make_float2(acc[0], acc[1]);
          *p1 = make_float2(acc[2], acc[3]);
        }
        if (!multi_tile) {
          consumer_sync();
          linear_group_epilogue<WIDE, HYB>(c, d, B, NT, r0, min(R, n1 - r0), part);
        }
      }
      ++group_seq;
    }
  }
  if (!ok) c.s.flags[0] = 1;
  if (tid == 0 && prof) P.profiler[(size_t)task * 8 + 5] = globaltimer_ns();
  if (B > 0 && multi_tile) {
    consumer_sync();
    int gi = 0;
    for (int r0 = n0; r0 < n1; r0 += R, ++gi)
      linear_group_epilogue<WIDE, HYB>(c, d, B, NT, r0, min(R, n1 - r0), c.s.partial + (size_t)(gi & 1) * (8 * 16 * 8));
  }
}

// ---------------------------------------------------------------------------
// Everything the epilogue of a tcgen05 linear task needs from its descriptor, read once into registers: the
// descriptor lives in shared memory behind a generic reference, and a load from it may not move across the global
// stores of the epilogue (they could alias), so reading it per element costs a chain of dependent loads every time.
struct EmitArgs {
  int epi, ldo, world;
  __nv_bfloat16 *out;
  size_t push_off;      // element offset of (token 0, column 0) of this rank's slot in an inbox buffer
  int push_n;           // row length of the pushed matrix
  uint32_t seq_hi;      // sequence number of the allreduce instance, already shifted to the high half (EPI_SOFTCAP, EPI_SCALE_F32: cap / factor bits)
};

__device__ __forceinline__ EmitArgs emit_args(const Ctx &c, const TaskDesc &d) {
  EmitArgs e;
  e.epi = d.a[L_EPI];
  e.ldo = d.a[L_LDO];
  e.world = c.P.world_size;
  e.out = reinterpret_cast<__nv_bfloat16 *>(d.p[2]);
  const unsigned long long inst = c.iteration * (unsigned)d.a[L_NAR] + (unsigned)d.a[L_ARIDX];
  e.push_off = (size_t)d.p[5] + (size_t)(inst & 1ull) * (size_t)d.a[L_PARSTRIDE] + (size_t)c.P.rank * (size_t)d.a[L_SLOT];
  e.push_n = d.a[L_N];
  e.seq_hi = e.epi == EPI_SOFTCAP || e.epi == EPI_SCALE_F32 ? (uint32_t)d.a[L_CAP] : ll_seq(c.iteration, d.a[L_NAR], d.a[L_ARIDX]) << 16;
  return e;
}

template <int HYB>
__device__ __forceinline__ void linear_emit(const Ctx &c, const EmitArgs &e, int b, int col, float v, float u, float resv) {
  if (e.epi == EPI_PUSH_LL) {
    // one 32-bit word per element: bf16 partial sum in the low half, sequence number in the high half
    const size_t off = e.push_off + (size_t)b * e.push_n + col;
    const __nv_bfloat16 hv = __float2bfloat16_rn(v);
    const uint32_t word = (uint32_t)(*reinterpret_cast<const unsigned short *>(&hv)) | e.seq_hi;
    for (int peer = 0; peer < e.world; ++peer)
      asm volatile("st.relaxed.sys.global.u32 [%0], %1;" ::"l"(reinterpret_cast<uint32_t *>(c.P.peer_inbox[peer]) + off),
                   "r"(word)
                   : "memory");
  } else if (e.epi == EPI_PUSH_F32) {
    const size_t off = e.push_off + (size_t)b * e.push_n + col;
    for (int peer = 0; peer < e.world; ++peer) c.P.peer_inbox[peer][off] = v;
  } else if (e.epi == EPI_SILU_PAIR) {
    // rows come as [gate, gate, up, up]: the threads on gate rows finish the pair (u = the value two rows on)
    if ((col & 2) == 0) {
      const float a = round_bf16(silu_f(round_bf16(v)));
      e.out[(size_t)b * e.ldo + ((col >> 2) << 1) + (col & 1)] = __float2bfloat16_rn(a * round_bf16(u));
    }
  } else if (HYB && (e.epi == EPI_STORE_F32 || e.epi == EPI_BIAS_F32)) {
    reinterpret_cast<float *>(e.out)[(size_t)b * e.ldo + col] = v + resv;   // resv: the bias, or 0
  } else if (HYB && e.epi == EPI_RELU2) {
    const float a = fmaxf(v, 0.f);
    e.out[(size_t)b * e.ldo + col] = __float2bfloat16_rn(a * a);
  } else if (HYB && e.epi == EPI_SOFTCAP) {
    const float cap = __uint_as_float(e.seq_hi);
    reinterpret_cast<float *>(e.out)[(size_t)b * e.ldo + col] = cap * tanhf(v / cap);
  } else if (HYB && e.epi == EPI_SCALE_F32) {
    reinterpret_cast<float *>(e.out)[(size_t)b * e.ldo + col] = __uint_as_float(e.seq_hi) * v;
  } else if (HYB && e.epi == EPI_GATE_SIGMOID) {
    e.out[(size_t)b * e.ldo + col] = __float2bfloat16_rn(v / (1.0f + expf(-resv)));   // resv: the gate
  } else if (HYB && (e.epi == EPI_GATED_SILU || e.epi == EPI_GATED_GELU)) {
    if ((col & 2) == 0)
      e.out[(size_t)b * e.ldo + ((col >> 2) << 1) + (col & 1)] =
          __float2bfloat16_rn((e.epi == EPI_GATED_SILU ? silu_exact_f(v) : gelu_tanh_f(v)) * u);
  } else {
    e.out[(size_t)b * e.ldo + col] = __float2bfloat16_rn(v + resv);   // resv: the residual element, or 0
  }
}

// Four rows of two tokens through the epilogue (fewer rows at the end of the panel: `cnt`); `wide`: output and operands lie on vector boundaries.
struct XsOut {
  EmitArgs e;
  const uint8_t *operand;   // residual (bf16), gate (float32) or bias (bf16, a row of it: ldr = 0)
  int ldr;
  bool wide;
};
template <int HYB>
__device__ __forceinline__ void xs_emit(const Ctx &c, const XsOut &x, int b0, int b1, int col, int cnt, const float (&v)[2][4]) {   // tokens b0 and b1 (-1: none)
  const int epi = x.e.epi;
  if (epi == EPI_SILU_PAIR || (HYB && (epi == EPI_GATED_SILU || epi == EPI_GATED_GELU))) {   // rows come as [gate, gate, up, up]
    float o[2][2];
#pragma unroll
    for (int t = 0; t < 2; ++t)
#pragma unroll
      for (int j = 0; j < 2; ++j) {
        if (!HYB || epi == EPI_SILU_PAIR) o[t][j] = round_bf16(silu_f(round_bf16(v[t][j]))) * round_bf16(v[t][j + 2]);
        else o[t][j] = (epi == EPI_GATED_SILU ? silu_exact_f(v[t][j]) : gelu_tanh_f(v[t][j])) * v[t][j + 2];
      }
#pragma unroll
    for (int t = 0; t < 2; ++t) {
      const int b = t == 0 ? b0 : b1;
      if (b < 0) return;
      __nv_bfloat16 *out = x.e.out + (size_t)b * x.e.ldo + (col >> 1);
      if (x.wide) *reinterpret_cast<uint32_t *>(out) = pack_bf16(o[t][0], o[t][1]);
      else { out[0] = __float2bfloat16_rn(o[t][0]); out[1] = __float2bfloat16_rn(o[t][1]); }
    }
    return;
  }
  if (epi == EPI_PUSH_LL || epi == EPI_PUSH_F32) {
#pragma unroll
    for (int t = 0; t < 2; ++t)
#pragma unroll
      for (int j = 0; j < 4; ++j)
        if (j < cnt && (t == 0 ? b0 : b1) >= 0) linear_emit<HYB>(c, x.e, t == 0 ? b0 : b1, col + j, v[t][j], 0.f, 0.f);
    return;
  }
  float o[2][4];
#pragma unroll
  for (int t = 0; t < 2; ++t) {
    const int b = t == 0 || b1 < 0 ? b0 : b1;
#pragma unroll
    for (int j = 0; j < 4; ++j) o[t][j] = v[t][j];
    if (epi == EPI_RESIDUAL || (HYB && epi == EPI_BIAS_F32)) {
      const __nv_bfloat16 *r = reinterpret_cast<const __nv_bfloat16 *>(x.operand) + (size_t)b * x.ldr + col;
      if (x.wide && cnt == 4) {
        const uint2 w = __ldcg(reinterpret_cast<const uint2 *>(r));
        o[t][0] += bf16_lo(w.x); o[t][1] += bf16_hi(w.x); o[t][2] += bf16_lo(w.y); o[t][3] += bf16_hi(w.y);
      } else {
#pragma unroll
        for (int j = 0; j < 4; ++j) if (j < cnt) o[t][j] += bf16_to_f(__ldcg(r + j));
      }
    }
    if (HYB && epi == EPI_GATE_SIGMOID) {
      const float *g = reinterpret_cast<const float *>(x.operand) + (size_t)b * x.ldr + col;
#pragma unroll
      for (int j = 0; j < 4; ++j) if (j < cnt) o[t][j] /= 1.0f + expf(-__ldcg(g + j));
    }
    if (HYB && epi == EPI_RELU2) {
#pragma unroll
      for (int j = 0; j < 4; ++j) o[t][j] = fmaxf(o[t][j], 0.f) * fmaxf(o[t][j], 0.f);
    }
    if (HYB && (epi == EPI_SOFTCAP || epi == EPI_SCALE_F32)) {
      const float f = __uint_as_float(x.e.seq_hi);
#pragma unroll
      for (int j = 0; j < 4; ++j) o[t][j] = epi == EPI_SCALE_F32 ? f * o[t][j] : f * tanhf(o[t][j] / f);
    }
  }
#pragma unroll
  for (int t = 0; t < 2; ++t) {
    const int b = t == 0 ? b0 : b1;
    if (b < 0) return;
    const size_t at = (size_t)b * x.e.ldo + col;
    if (HYB && (epi == EPI_STORE_F32 || epi == EPI_BIAS_F32 || epi == EPI_SOFTCAP || epi == EPI_SCALE_F32)) {
      float *out = reinterpret_cast<float *>(x.e.out) + at;
      if (x.wide && cnt == 4) {
        *reinterpret_cast<float4 *>(out) = make_float4(o[t][0], o[t][1], o[t][2], o[t][3]);
      } else {
#pragma unroll
        for (int j = 0; j < 4; ++j) if (j < cnt) out[j] = o[t][j];
      }
    } else {
      __nv_bfloat16 *out = x.e.out + at;
      if (x.wide && cnt == 4) {
        *reinterpret_cast<uint2 *>(out) = make_uint2(pack_bf16(o[t][0], o[t][1]), pack_bf16(o[t][2], o[t][3]));
      } else {
#pragma unroll
        for (int j = 0; j < 4; ++j) if (j < cnt) out[j] = __float2bfloat16_rn(o[t][j]);
      }
    }
  }
}

// Prologue PRO_RMSNORM: the whole rows as the operand tile, bf16(x / rms * gamma).  Rows and gamma are copied with everything in flight, then a
// warp sums and scales its own rows (16 tokens of 4096 columns: 6.5 us beside the weight stream).
static __device__ __noinline__ void xs_stage_norm(const uint4 *src, const uint4 *gam, uint32_t xs, uint32_t gsm, int ldv, int B, int NP, int vecs, float eps) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const bool gamma_here = vecs * 16 <= kPartialBytes;
  for (int b = warp; b < B; b += 8) {
    const uint32_t row = xs + b * 128 + (((lane & 7) ^ (b & 7)) << 4);
#pragma unroll 4
    for (int v = lane; v < vecs; v += 32)
      asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(row + (uint32_t)((v >> 3) * NP * 128)), "l"(src + (size_t)b * ldv + v) : "memory");
  }
  if (gamma_here)
    for (int v = threadIdx.x; v < vecs; v += kConsumerThreads) asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(gsm + v * 16), "l"(gam + v) : "memory");
  asm volatile("cp.async.commit_group;" ::: "memory");
  asm volatile("cp.async.wait_group 0;" ::: "memory");
  consumer_sync();
  for (int b = warp; b < B; b += 8) {
    const uint32_t row = xs + b * 128 + (((lane & 7) ^ (b & 7)) << 4);
    float ss = 0.f;
#pragma unroll 4
    for (int v = lane; v < vecs; v += 32) {
      const uint4 x = lds_u4(row + (uint32_t)((v >> 3) * NP * 128));
      const uint32_t w[4] = {x.x, x.y, x.z, x.w};
#pragma unroll
      for (int q = 0; q < 4; ++q) ss += bf16_lo(w[q]) * bf16_lo(w[q]) + bf16_hi(w[q]) * bf16_hi(w[q]);
    }
    const float inv = rsqrtf(warp_sum(ss) / (float)(vecs * 8) + eps);
#pragma unroll 4
    for (int v = lane; v < vecs; v += 32) {
      const uint32_t at = row + (uint32_t)((v >> 3) * NP * 128);
      const uint4 x = lds_u4(at), g = gamma_here ? lds_u4(gsm + v * 16) : __ldg(gam + v);
      const uint32_t xw[4] = {x.x, x.y, x.z, x.w}, gw[4] = {g.x, g.y, g.z, g.w};
      uint32_t ow[4];
#pragma unroll
      for (int q = 0; q < 4; ++q) ow[q] = pack_bf16(bf16_lo(xw[q]) * inv * bf16_lo(gw[q]), bf16_hi(xw[q]) * inv * bf16_hi(gw[q]));
      asm volatile("st.shared.v4.b32 [%0], {%1,%2,%3,%4};" ::"r"(at), "r"(ow[0]), "r"(ow[1]), "r"(ow[2]), "r"(ow[3]) : "memory");
    }
  }
  fence_proxy_async_smem();   // written with generic stores, read by the MMAs
  consumer_sync();
}

// ---------------------------------------------------------------------------
// TASK_LINEAR on the tensor path (general instantiation, graphs with more than 8 batched tokens): the weights are the M operand (swap-AB, as in
// include/mirage/persistent_kernel/tasks/blackwell/linear_sm100_mpk.cuh:31-735), 128 rows per tcgen05.mma, the batched tokens the N operand
// (16 .. 64), fp32 accumulators in tensor memory.
//
// The task is one pipeline along k.  A ring slot brings nkb k blocks of 64 columns of one row tile (RB <= 128 rows), all tiles of a k
// position in turn; the activations of that position come once, for all tiles, through a ring of their own: one box {64 columns, token rows,
// nkb blocks} of the tensor map of the layer's input, issued by warp 7 as soon as the dependency is met (PRO_RMSNORM: the whole rows are there
// from the start).  Measured: an MMA takes a thread 64 cycles to issue and a commit 200, while the tensor pipe needs 39 (16 tokens) to 49 (64
// tokens) for any M up to 128, so up to four warps issue, each its row tiles and chunks of k, those of different chunks into accumulators of their
// own (`sets`, added in order by the epilogue): results do not depend on timing.  Commits hand the slots of both rings back.
// Where a row panel per worker would be thin (a linear of few rows and long k), `splits` workers share a panel and each takes a part of k
// (LX_*): full MMAs, and each reads its part of the activations only.  Parts meet in scratch memory in fp32; the last worker to arrive adds
// them up in order.
// ---------------------------------------------------------------------------
template <int N> struct Columns { static constexpr int value = N; };

template <int HYB>
__device__ __noinline__ LinearState run_linear_tc(const Ctx c, const TaskDesc &d, LinearState ls, int task, bool ok) {
  const KernelParams &P = c.P;
  if (!ok) return ls;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const uint32_t x_par = (uint32_t)c.s.flags[3];            // parities of the next completions of the activation ring's slots
  const int B = min(active_tokens(P), kMaxLinearTokens);
  const int NP = P.tc_tokens;                               // token rows of the operand tile / columns per accumulator
  const int Nmma = min(NP, max(16, (B + 15) & ~15));        // N of the instruction
  const int n0 = d.a[L_N0], rows = d.a[L_N1] - n0, RB = d.a[L_ROWS];
  const int nkb = d.a[L_KC] / kTcKBlock, kball = d.a[L_K] / kTcKBlock;
  const int tiles = (rows + RB - 1) / RB;
  const XRing ring = x_ring(c, d);
  const bool staged = d.a[L_PRO] == PRO_RMSNORM;
  const bool prof = P.profiler != nullptr && (uint64_t)(task + 1) * 8 <= P.profiler_entries;
  uint64_t *xfull = x_bars(c), *xempty = xfull + 8;
  const uint32_t x_chunk = (uint32_t)(NP * nkb * 128);                // bytes of a ring chunk
  const int nx = d.a[LX_NX], nch = (kball + nkb - 1) / nkb;
  // where the ring stands: borrowing tasks start at its first slot (ls.phase: a bit per slot), others follow on
  const int s0 = P.borrow ? 0 : ls.stage;
  const uint32_t par0 = P.borrow ? ls.phase : (ls.phase ? 0xffffu : 0u) ^ ((1u << ls.stage) - 1u);
  if (tid == 0 && ring.size > ring.base && nch * tiles > ring.base) mbar_arrive(ring.xbars + 32);   // (the tile area is free: all threads are past their last task)
  const uint32_t xs_smem = smem_u32(c.s.xtile);
  // Issuing warps.  A warp must neither fall a lap of a ring behind nor run one ahead (a barrier's parity says no more than that), and following slots
  // that are another's costs 300 cycles each; so a slot belongs to one warp, by row tile and by chunk.  Measured (64 tokens, two row tiles, chunks of one
  // k block): a chunk takes a warp 1550 cycles, 670 of them for four MMAs and their commit, so that two warps drew 3.7 TB/s.
  const XIssuers wi = x_issuers(tiles, ring.size, staged ? 0 : nx);
  const int issuers = wi.tiles * wi.chunks, sets = min(wi.chunks, nch);
  if (staged)
    xs_stage_norm(reinterpret_cast<const uint4 *>(d.p[1]), reinterpret_cast<const uint4 *>(d.p[4]), xs_smem, smem_u32(c.s.partial), d.a[L_LDX] >> 3, B, NP,
                  d.a[L_K] / 8, __int_as_float(d.a[L_EPS]));
  if (warp < issuers) {
    const uint32_t idesc = umma_idesc(1u, 128, Nmma);
    const uint64_t desc_hi = umma_desc_k_sw128(0);   // shared-memory addresses enter as (address >> 4) in the low 14 bits
    const int first = warp / wi.tiles, tile0 = warp - first * wi.tiles;   // chunk and row tile of this warp
    int xslot = 0;
    uint32_t par = par0, xpar = x_par;
    int s = s0;
    for (int i = 0; i < nch && ok; ++i) {
      const bool mine = (i & (wi.chunks - 1)) == first;   // (a power of two)
      if (mine) {
        const int kb = i * nkb, nb = min(nkb, kball - kb);
        uint32_t xa = xs_smem >> 4;
        if (staged) {
          xa += (uint32_t)(kb * NP * 8);
        } else {
          ok = wait_mbar(c, &xfull[xslot], (xpar >> xslot) & 1u, task);
          xa += (uint32_t)xslot * (x_chunk >> 4);
        }
        if (prof && tid == 0 && i == 0) P.profiler[(size_t)task * 8 + 4] = globaltimer_ns();
        for (int tile = tile0; tile < tiles && ok; tile += wi.tiles) {
          const int sl = s + tile < ring.size ? s + tile : s + tile - ring.size;
          ok = wait_mbar(c, ring.full_bar(sl), (par >> sl) & 1u, task);
          if (!ok) break;
          if (lane == 0) {
            tc_fence_after_sync();
            const uint32_t wa = ring.slot(sl) >> 4, dt = c.tmem_base + (uint32_t)((first * tiles + tile) * NP);
            for (int j = 0; j < nb; ++j) {
              const uint64_t a0 = desc_hi | (wa + (uint32_t)(j * RB * 8)), b0 = desc_hi | (xa + (uint32_t)(j * NP * 8));
#pragma unroll
              for (int ks = 0; ks < 4; ++ks) umma_bf16(dt, a0 + ks * 2, b0 + ks * 2, idesc, i - first + j + ks > 0 ? 1u : 0u);
            }
            if (!P.borrow) mbar_arrive_n(ring.empty_bar(sl), 7);   // (the slot's barrier counts the eight warps of the other bodies)
            umma_commit(ring.empty_bar(sl));
          }
          __syncwarp();
        }
        if (!staged && lane == 0 && ok) umma_commit(&xempty[xslot]);
        __syncwarp();
      }
      // on by the chunk's boxes: a pass over the ring's end flips the parities of its slots
      par ^= ((1u << tiles) - 1u) << s;
      s += tiles;
      if (s >= ring.size) { s -= ring.size; par = (par & ((1u << ring.size) - 1u)) ^ ((1u << s) - 1u); }
      xpar ^= 1u << xslot;
      if (++xslot == nx) xslot = 0;
    }
    if (lane == 0 && ok) {
      if (warp == 0) mbar_arrive_n(c.s.acc_bar, 8 - issuers);
      umma_commit(c.s.acc_bar);
    }
    __syncwarp();
  } else if (warp == 7 && !staged) {
    if (lane == 0) {
      const uint8_t *xmap = reinterpret_cast<const uint8_t *>(P.tmaps) + (size_t)d.a[LX_TMAP] * 128;
      uint32_t xpar = x_par;
      int xslot = 0, issued = 0;
      bool good = true;
      fence_proxy_async_all();   // the activations were written through the generic proxy
      for (int i = 0; i < nch && good; ++i) {
        if (i >= nx) good = wait_mbar(c, &xempty[xslot], ((xpar >> xslot) & 1u) ^ 1u, task);
        if (!good) break;
        mbar_arrive_expect_tx(&xfull[xslot], x_chunk);
        if (wi.tiles < kXIssuers) mbar_arrive_n(&xempty[xslot], kXIssuers - wi.tiles);   // (of the arrivals its barrier counts; a warp of each row tile commits)
        tma_load_3d_shared(xs_smem + (uint32_t)xslot * x_chunk, xmap, 0, 0, i * nkb, smem_u32(&xfull[xslot]));
        xpar ^= 1u << xslot;
        if (++xslot == nx) xslot = 0;
        ++issued;
      }
      // the launch is being abandoned: what this thread issued lands before the CTA may exit
      for (int i = 0; !good && i < min(issued, nx); ++i) {
        uint32_t polls = 0;
        while (!mbar_try_wait(&xfull[i], ((xpar >> i) & 1u) ^ 1u) && ++polls < (1u << 24)) {}
      }
    }
    __syncwarp();
  }
  // what all threads know about the rings after this task
  {
    const int used = s0 + nch * tiles;
    if (P.borrow) {
      const int laps = used / ring.size, rest = used - laps * ring.size;
      ls.phase ^= ((laps & 1 ? 0xffffu : 0u) ^ ((1u << rest) - 1u)) & ((1u << ring.size) - 1u);
    } else {
      ls.phase ^= (uint32_t)(used / ring.size) & 1u;
      ls.stage = used % ring.size;
    }
  }
  if (!wait_mbar(c, c.s.acc_bar, ls.acc_phase, task)) ok = false;
  ls.acc_phase ^= 1u;
  if (!ok) c.s.flags[0] = 1;
  consumer_sync();
  if (c.s.flags[0] != 0) return ls;
  tc_fence_after_sync();
  if (tid == 0 && !staged) {
    uint32_t flips = 0;
    for (int i = 0; i < nx; ++i) flips |= (uint32_t)((nch + nx - 1 - i) / nx & 1) << i;
    c.s.flags[3] = (int)(x_par ^ flips);
  }
  if (tid == 0 && prof) P.profiler[(size_t)task * 8 + 5] = globaltimer_ns();
  if (B == 0) { tc_fence_before_sync(); return ls; }
  // Epilogue.  A warp reads its lane quadrant of half the tokens, adds the sets and leaves the sums as [token][row] in shared memory (the tile
  // area is free now), or in scratch memory where the panel is shared; then a warp takes a token at a time, four rows a lane.  Straight from
  // the accumulators to the output, a row per lane, it took 1 to 1.5 us for eight tokens of a tile: long unrolled code that leaves the
  // instruction caches at each pass, and stores of single elements (64 tokens, gate and up rows of width 4096: 25 us before, 6 now).
  const int quad = warp & 3, half = warp >> 2;
  const int nh = Nmma >> 1;   // tokens of a warp's half: a multiple of 8
  const int S = d.a[LX_SPLITS];
  float *sums = reinterpret_cast<float *>(c.s.xtile);
  const size_t part_floats = (size_t)tiles * NP * RB;
  if (S > 1) sums = P.split_scratch + d.p[6] + (size_t)d.a[LX_PART] * part_floats;
  const int fit = S > 1 ? tiles : P.x_tile_bytes / (NP * RB * 4);   // row tiles at a time
  XsOut xo{emit_args(c, d), reinterpret_cast<const uint8_t *>(d.p[3]), d.a[L_LDR], false};
  {
    const int epi = xo.e.epi;
    const bool f32 = HYB && (epi == EPI_STORE_F32 || epi == EPI_BIAS_F32 || epi == EPI_SOFTCAP || epi == EPI_SCALE_F32);
    if (HYB && epi == EPI_BIAS_F32) { xo.operand = *reinterpret_cast<const uint8_t *const *>(&d.a[LR_BIAS]); xo.ldr = 0; }
    const bool reads = epi == EPI_RESIDUAL || (HYB && epi == EPI_BIAS_F32);
    xo.wide = (n0 & 3) == 0 && (reinterpret_cast<uintptr_t>(xo.e.out) & (f32 ? 15 : 7)) == 0 && (xo.e.ldo & 3) == 0 &&
              (!reads || ((reinterpret_cast<uintptr_t>(xo.operand) & 7) == 0 && (xo.ldr & 3) == 0));
  }
  for (int tile0 = 0; tile0 < tiles; tile0 += fit) {
    const int tile1 = min(tiles, tile0 + fit);
    if (tile0 > 0) consumer_sync();
    for (int tile = tile0; quad * 32 < RB && tile < tile1; ++tile) {
      const uint32_t at = c.tmem_base + ((uint32_t)(quad * 32) << 16) + (uint32_t)(tile * NP + half * nh);
      float *dst = sums + (size_t)((tile - tile0) * NP + half * nh) * RB + quad * 32 + lane;
      const bool keep = quad * 32 + lane < RB;
      const auto add_sets = [&](auto n, int c0) {
        constexpr int kCols = decltype(n)::value;
        float v[kCols];
#pragma unroll
        for (int j = 0; j < kCols; ++j) v[j] = 0.f;
#pragma unroll 1
        for (int q = 0; q < sets; ++q) {   // (two loads at a time cost the kernel that calls this 260 bytes of spills)
          uint32_t r[kCols];
          tmem_ld(at + (uint32_t)(q * tiles * NP + c0), r);
          tmem_ld_wait();
#pragma unroll
          for (int j = 0; j < kCols; ++j) v[j] += __uint_as_float(r[j]);
        }
        if (keep)
#pragma unroll
          for (int j = 0; j < kCols; ++j) dst[(c0 + j) * RB] = v[j];
      };
      int c0 = 0;
#pragma unroll 1
      for (; c0 + 16 <= nh; c0 += 16) add_sets(Columns<16>(), c0);
      if (c0 < nh) add_sets(Columns<8>(), c0);
    }
    if (S > 1) {
      __threadfence();
      consumer_sync();
      if (tid == 0) {
        unsigned int *ticket = P.attn_tickets + d.a[LX_TICKET];
        const unsigned int old = atomicAdd(ticket, 1u);
        __threadfence();
        if (old == (unsigned)S - 1u) *ticket = 0u;   // (its next use waits for this task)
        c.s.flags[1] = old == (unsigned)S - 1u ? 1 : 0;
      }
      consumer_sync();
      if (c.s.flags[1] == 0) break;
      sums = P.split_scratch + d.p[6];
    } else {
      consumer_sync();
    }
    if (tid == 0 && prof && tile0 == 0) P.profiler[(size_t)task * 8 + 6] = globaltimer_ns();
    const int lanes = RB > 64 ? 32 : RB > 32 ? 16 : 8, sub = lane & (lanes - 1), step = 8 * (32 / lanes);
    const int r0 = sub * 4;
    for (int tile = tile0; r0 < RB && tile < tile1; ++tile) {
      const int row = tile * RB + r0, cnt = min(4, rows - row);
      if (cnt <= 0) break;
      const size_t src = (size_t)(tile - tile0) * NP * RB + r0;
#pragma unroll 1
      for (int b = warp * (32 / lanes) + lane / lanes; b < B; b += 2 * step) {   // two tokens at a time, so that their chains overlap
        float v[2][4];
        const int b1 = min(b + step, B - 1);
        if (S > 1) {
#pragma unroll
          for (int j = 0; j < 4; ++j) v[0][j] = v[1][j] = 0.f;
#pragma unroll 2
          for (int p = 0; p < S; ++p) {
            const float *at = sums + (size_t)p * part_floats + src;
            const float4 t = __ldcg(reinterpret_cast<const float4 *>(at + (size_t)b * RB)), u = __ldcg(reinterpret_cast<const float4 *>(at + (size_t)b1 * RB));
            v[0][0] += t.x; v[0][1] += t.y; v[0][2] += t.z; v[0][3] += t.w;
            v[1][0] += u.x; v[1][1] += u.y; v[1][2] += u.z; v[1][3] += u.w;
          }
        } else {
          lds_f4(xs_smem + (uint32_t)(src + (size_t)b * RB) * 4, v[0]);
          lds_f4(xs_smem + (uint32_t)(src + (size_t)b1 * RB) * 4, v[1]);
        }
        xs_emit<HYB>(c, xo, b, b + step < B ? b1 : -1, n0 + row, cnt, v);
      }
    }
    if (tid == 0 && prof && tile0 == 0) P.profiler[(size_t)task * 8 + 7] = globaltimer_ns();
  }
  tc_fence_before_sync();   // the accumulators have been read: the next task's MMAs may overwrite them after the task barrier
  return ls;
}

// ---------------------------------------------------------------------------
// FP8 TASK_LINEAR on the tensor path: tcgen05.mma kind::mxf8f6f4 with block scaling, the form the reference uses
// (include/mirage/persistent_kernel/tasks/blackwell/linear_fp8_1d2d_sm100.cuh:69-727).  Geometry as in run_linear_tc
// with one byte per element: a 128-byte k block is 128 columns = one scale group = four MMAs of K = 32.  The scale
// tensors hold four UE8M0 exponents per uint32 (four consecutive groups, 512 columns): such a word per row IS the
// tensor-memory scale column the instruction wants, the group within it is the instruction's scale id.  Per 512
// columns and row tile, 128 weight-scale words (and 128 activation-scale words per 512 columns) are staged in shared
// memory in the [32 lanes][4 words] order tcgen05.cp copies to tensor memory.  A 512-column "super group" of a tile
// belongs to one warp, which copies its scale words into its own eight tensor-memory columns and then issues the 16
// MMAs in order behind the copy; super groups rotate over the issuing warps.
// ---------------------------------------------------------------------------
static __device__ void run_linear_fp8_tc(const Ctx &c, const TaskDesc &d, LinearState &ls, int task, bool ok) {
  const KernelParams &P = c.P;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int B = ok ? min(active_tokens(P), kMaxLinearTokens) : 0;
  const int NP = P.tc_tokens;
  const int Nmma = min(NP, max(16, (B + 15) & ~15));
  const int n0 = d.a[L_N0], rows = d.a[L_N1] - n0, K = d.a[L_K], KT = d.a[L_KT], RB = d.a[L_ROWS];
  const int nkb = d.a[L_KC] / 128, kbt = KT / 128, nsg = KT / 512;
  const int tiles = (rows + RB - 1) / RB;
  const int NST = P.num_stages;
  uint8_t *xt = c.s.xtile;                                   // [kbt][NP][128 bytes], swizzled
  uint32_t *sfb = reinterpret_cast<uint32_t *>(xt + (size_t)NP * KT);              // [nsg][128 words]
  uint32_t *sfa = sfb + (size_t)nsg * 128;                   // [tiles][nsg][128 words]
  // one accumulator set per issuing warp, added in set order by the epilogue (see run_linear_tc): bit-reproducible
  const int sets = max(1, min(8, kTcAccCols / (tiles * NP)));
  tc_fence_after_sync();
  if (ok && warp < 4) {
    const uint32_t t0 = c.tmem_base + ((uint32_t)(warp * 32) << 16);
    for (int col = 0; col < sets * tiles * NP; col += 16) tmem_st_zero_x16(t0 + (uint32_t)col);
    tmem_st_wait();
  }
  tc_fence_before_sync();
  const uint64_t desc_hi = umma_desc_k_sw128(0);
  const uint32_t x_base = smem_u32(xt) >> 4;
  const uint32_t my_sfa = c.tmem_base + (uint32_t)(kTcAccCols + warp * 8), my_sfb = my_sfa + 4u;
  const uint32_t *ws = reinterpret_cast<const uint32_t *>(d.p[6]);
  const uint32_t *xs = reinterpret_cast<const uint32_t *>(d.p[7]);
  int sg_seq = 0;                                            // running count of (tile, super group) units: owner = sg_seq % 8
  for (int kt = 0; kt < K; kt += KT) {
    if (ok) {
      const bool with_x = !((d.flags & TF_SAME_X_AS_PREV) && KT == K);
      if (with_x) {
        const uint8_t *x = reinterpret_cast<const uint8_t *>(d.p[1]);
        const int ldx = d.a[L_LDX], vecs = KT / 16;
        for (int b = 0; b < B; ++b)
          for (int v = tid; v < vecs; v += kConsumerThreads)
            asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(smem_u32(x_vec<2>(xt, b, v, 0, NP))),
                         "l"(reinterpret_cast<const uint4 *>(x + (size_t)b * ldx + kt) + v)
                         : "memory");
        asm volatile("cp.async.commit_group;" ::: "memory");
        // activation scale words, token b of super group sg -> word (b % 32) * 4 + b / 32 of the group's block
        const int s0 = d.a[L_XS_S0], s1 = d.a[L_XS_S1];
        // (four loads in flight per thread before the first store: a store to shared memory through a generic
        // pointer keeps the compiler from moving the next load above it)
        for (int i0 = tid; i0 < nsg * 128; i0 += 4 * kConsumerThreads) {
          uint32_t w[4];
#pragma unroll
          for (int u = 0; u < 4; ++u) {
            const int i = i0 + u * kConsumerThreads, sg = i >> 7, b = i & 127;
            w[u] = (i < nsg * 128 && b < B) ? __ldcg(xs + (size_t)b * s0 + (size_t)(kt / 512 + sg) * s1) : 0u;
          }
#pragma unroll
          for (int u = 0; u < 4; ++u) {
            const int i = i0 + u * kConsumerThreads, sg = i >> 7, b = i & 127;
            if (i < nsg * 128) sfb[sg * 128 + (b & 31) * 4 + (b >> 5)] = w[u];
          }
        }
      }
      {
        const int s0 = d.a[L_WS_S0], s1 = d.a[L_WS_S1];
        for (int i0 = tid; i0 < tiles * nsg * 128; i0 += 4 * kConsumerThreads) {
          uint32_t w[4];
#pragma unroll
          for (int u = 0; u < 4; ++u) {
            const int i = i0 + u * kConsumerThreads, r = i & 127, uu = i >> 7, tile = uu / nsg, sg = uu - tile * nsg;
            const int row = tile * RB + r;
            w[u] = (i < tiles * nsg * 128 && r < RB && row < rows)
                       ? __ldcg(ws + (size_t)(n0 + row) * s0 + (size_t)(kt / 512 + sg) * s1) : 0u;
          }
#pragma unroll
          for (int u = 0; u < 4; ++u) {
            const int i = i0 + u * kConsumerThreads, r = i & 127, uu = i >> 7;
            if (i < tiles * nsg * 128) sfa[uu * 128 + (r & 31) * 4 + (r >> 5)] = w[u];
          }
        }
      }
      asm volatile("cp.async.wait_group 0;" ::: "memory");
      fence_proxy_async_smem();
    }
    consumer_sync();
    tc_fence_after_sync();
    for (int tile = 0; tile < tiles; ++tile) {
      const uint32_t d_tmem = c.tmem_base + (uint32_t)((warp * tiles + tile) * NP);   // (used by warps < sets only)
      for (int kb = 0; kb < kbt; kb += nkb) {
        const int s = ls.stage;
        const uint32_t ph = ls.phase;
        if (++ls.stage == NST) { ls.stage = 0; ls.phase ^= 1u; }
        if (ok) ok = wait_mbar(c, &c.s.full[s], ph, task);
        if (ok && lane == 0) {
          tc_fence_after_sync();
          const uint32_t a_base = smem_u32(c.s.stages + (size_t)s * P.stage_bytes) >> 4;
          for (int j = 0; j < nkb; ++j) {
            const int g = kb + j, sg = g >> 2;                // k block (= scale group) and its super group within the k tile
            if ((sg_seq + sg) % sets != warp) continue;
            if ((g & 3) == 0 || j == 0) {
              // (first block of the super group that this slot brings: if the group began in an earlier slot the
              // words are already in place, and copying them again behind the earlier MMAs is harmless)
              utccp_sf_128(my_sfa, smem_u32(sfa + (size_t)(tile * nsg + sg) * 128));
              utccp_sf_128(my_sfb, smem_u32(sfb + (size_t)sg * 128));
            }
            const uint32_t idesc = umma_idesc_mxf8(128, Nmma, (uint32_t)(g & 3));
#pragma unroll
            for (int ks = 0; ks < 4; ++ks)
              umma_mxf8_acc(d_tmem, desc_hi | (a_base + (uint32_t)(j * RB * 8 + ks * 2)),
                            desc_hi | (x_base + (uint32_t)(g * NP * 8 + ks * 2)), idesc, my_sfa, my_sfb);
          }
          umma_commit(&c.s.empty[s]);
        }
        __syncwarp();
      }
      sg_seq += nsg;
    }
    if (lane == 0) umma_commit(c.s.acc_bar);
    if (!wait_mbar(c, c.s.acc_bar, ls.acc_phase, task)) ok = false;
    ls.acc_phase ^= 1u;
    if (!ok) c.s.flags[0] = 1;
    consumer_sync();
    ok = ok && (c.s.flags[0] == 0);
    if (!ok) break;
  }
  if (!ok) { c.s.flags[0] = 1; return; }
  tc_fence_after_sync();
  if (B > 0) {
    const int quad = warp & 3, half = warp >> 2;
    const int nh = Nmma >> 1;
    const EmitArgs ea = emit_args(c, d);
    const __nv_bfloat16 *resp = reinterpret_cast<const __nv_bfloat16 *>(d.p[3]);
    const int ldr = d.a[L_LDR];
    for (int tile = 0; tile < tiles; ++tile) {
      if (quad * 32 >= RB) break;
      const int r_in_tile = quad * 32 + lane;
      const int row = tile * RB + r_in_tile;
      const bool row_ok = r_in_tile < RB && row < rows;
      const uint32_t taddr = c.tmem_base + ((uint32_t)(quad * 32) << 16) + (uint32_t)(tile * NP + half * nh);
      for (int c0 = 0; c0 < nh; c0 += 8) {
        uint32_t r[8];
        tmem_ld_x8(taddr + (uint32_t)c0, r);
        for (int st = 1; st < sets; ++st) {
          uint32_t r2[8];
          tmem_ld_wait();
          tmem_ld_x8(taddr + (uint32_t)(st * tiles * NP + c0), r2);
          tmem_ld_wait();
#pragma unroll
          for (int j = 0; j < 8; ++j) r[j] = __float_as_uint(__uint_as_float(r[j]) + __uint_as_float(r2[j]));
        }
        float resv[8];
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          const int b = half * nh + c0 + j;
          resv[j] = 0.f;
          if (ea.epi == EPI_RESIDUAL && row_ok && b < B) resv[j] = bf16_to_f(__ldcg(resp + (size_t)b * ldr + n0 + row));
        }
        tmem_ld_wait();
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          const int b = half * nh + c0 + j;
          if (row_ok && b < B) linear_emit<0>(c, ea, b, n0 + row, __uint_as_float(r[j]), 0.f, resv[j]);
        }
      }
    }
  }
  tc_fence_before_sync();
}

// ---------------------------------------------------------------------------
// FP8 linear: e4m3 weights and activations with one UE8M0 (power-of-two) scale per 128 columns of every
// row, on mma.sync m16n8k32.  Replaces linear_fp8_1d2d_sm100 and its residual form
// (include/mirage/persistent_kernel/tasks/blackwell/linear_fp8_1d2d_sm100.cuh).  The streaming geometry
// is that of the bf16 task with one byte per element: an e4m3 k step of 32 columns spans the same 32 bytes
// of a row as a bf16 step of 16, so the fragment addressing is identical.  Each warp takes whole 128-column
// groups: four mma into a fresh accumulator, then acc += tmp * 2^(ew + ea - 254).
// ---------------------------------------------------------------------------
__device__ __forceinline__ void mma_e4m3_16832(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
  asm volatile(
      "mma.sync.aligned.m16n8k32.row.col.f32.e4m3.e4m3.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
      : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}

// The same contraction with the e4m3 operands widened to f16 in registers (exact: every e4m3 value is an f16 value)
// and two f16 MMAs of k = 16: thread (g, q) holds bytes 4q .. 4q + 3 of a row in each e4m3 fragment register; the
// first two become the f16 fragment's columns (2q, 2q + 1), the last two its columns (2q + 8, 2q + 9), in A and B
// alike, so that both operands see the same permutation of k within the step.
__device__ __forceinline__ void cvt_e4m3x4_f16x4(uint32_t src, uint32_t &lo, uint32_t &hi) {
  asm("{\n\t.reg .b16 l, h;\n\tmov.b32 {l, h}, %2;\n\tcvt.rn.f16x2.e4m3x2 %0, l;\n\tcvt.rn.f16x2.e4m3x2 %1, h;\n\t}"
      : "=r"(lo), "=r"(hi)
      : "r"(src));
}

__device__ __forceinline__ void mma_f16_16816(float (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0,
                                              uint32_t b1) {
  asm volatile(
      "mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
      : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
      : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}

__device__ __forceinline__ void mma_e4m3_as_f16(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
  uint32_t al[4], ah[4], bl[2], bh[2];
#pragma unroll
  for (int i = 0; i < 4; ++i) cvt_e4m3x4_f16x4(a[i], al[i], ah[i]);
  cvt_e4m3x4_f16x4(b0, bl[0], bh[0]);
  cvt_e4m3x4_f16x4(b1, bl[1], bh[1]);
  mma_f16_16816(d, al[0], al[1], ah[0], ah[1], bl[0], bh[0]);   // k 0 .. 15 of the step
  mma_f16_16816(d, al[2], al[3], ah[2], ah[3], bl[1], bh[1]);   // k 16 .. 31
}

// 2^(ew - 127) * 2^(ea - 127) as a float, clamped to the normal range
__device__ __forceinline__ float ue8m0_pair_scale(uint32_t ew, uint32_t ea) {
  int e = (int)ew + (int)ea - 127;
  e = max(1, min(254, e));
  return __int_as_float(e << 23);
}

__device__ __forceinline__ uint32_t align16u(uint32_t v) { return (v + 15u) & ~15u; }

// Stage, for k range [k0, k0 + KT): the activation rows and their scale exponents (unless the previous task
// left them in place), and the scale exponents of this task's weight rows.
static __device__ void stage_fp8(const Ctx &c, const TaskDesc &d, int B, int k0, int KT, bool with_x) {
  const int tid = threadIdx.x;
  const uint32_t xstride = (uint32_t)KT + kRowPadBytes;
  const int NG = KT / 128, g0 = k0 / 128;
  uint8_t *xt = c.s.xtile;
  uint8_t *xsc = xt + align16u((uint32_t)B * xstride);
  uint8_t *wsc = xsc + align16u((uint32_t)(B * NG));
  if (with_x) {
    const uint8_t *x = reinterpret_cast<const uint8_t *>(d.p[1]);
    const int ldx = d.a[L_LDX];
    const int vecs = KT / 16;
    for (int i = tid; i < B * vecs; i += kConsumerThreads) {   // asynchronous copies, all in flight together
      const int b = i / vecs, v = i - b * vecs;
      asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(smem_u32(xt + (size_t)b * xstride + (size_t)v * 16)),
                   "l"(reinterpret_cast<const uint4 *>(x + (size_t)b * ldx + k0) + v)
                   : "memory");
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
    const uint32_t *xs = reinterpret_cast<const uint32_t *>(d.p[7]);
    const int s0 = d.a[L_XS_S0], s1 = d.a[L_XS_S1];
    for (int i = tid; i < B * NG; i += kConsumerThreads) {
      const int b = i / NG, ga = g0 + (i - b * NG);
      const uint32_t word = __ldcg(xs + (size_t)b * s0 + (size_t)(ga >> 2) * s1);
      xsc[i] = (uint8_t)((word >> ((ga & 3) * 8)) & 0xffu);
    }
  }
  {
    const uint32_t *ws = reinterpret_cast<const uint32_t *>(d.p[6]);
    const int s0 = d.a[L_WS_S0], s1 = d.a[L_WS_S1];
    const int n0 = d.a[L_N0], rows = d.a[L_N1] - n0;
    for (int i = tid; i < rows * NG; i += kConsumerThreads) {
      const int r = i / NG, ga = g0 + (i - r * NG);
      const uint32_t word = __ldcg(ws + (size_t)(n0 + r) * s0 + (size_t)(ga >> 2) * s1);
      wsc[i] = (uint8_t)((word >> ((ga & 3) * 8)) & 0xffu);
    }
  }
  asm volatile("cp.async.wait_group 0;" ::: "memory");
  consumer_sync();
}

__device__ __forceinline__ void run_linear_fp8(const Ctx &c, const TaskDesc &d, LinearState &ls, int task, bool ok) {
  const KernelParams &P = c.P;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  int stage = ls.stage;
  uint32_t phase = ls.phase;
  const int B = ok ? min(active_tokens(P), kMaxLinearTokens) : 0;
  const int NT = B <= 8 ? 1 : (B <= 16 ? 2 : (B <= 32 ? 4 : 8));
  const int nt = warp % NT, ks = warp / NT, kstride = 8 / NT;
  const int n0 = d.a[L_N0], n1 = d.a[L_N1], K = d.a[L_K];
  const int KT = d.a[L_KT], KC = d.a[L_KC], R = d.a[L_ROWS];
  const int NST = P.num_stages;
  const int ngc = KC / 128, NG = KT / 128;
  const uint32_t row_stride = (uint32_t)KC + kRowPadBytes;
  const uint32_t xstride = (uint32_t)KT + kRowPadBytes;
  const int g = lane >> 2, q = lane & 3;
  const bool tok_valid = nt * 8 + g < B;
  const bool multi_tile = KT < K;
  const uint32_t a_lane_off = (uint32_t)(lane & 15) * row_stride + (uint32_t)(lane >> 4) * 16u;
  const uint32_t x_lane_base = smem_u32(c.s.xtile) + (uint32_t)(tok_valid ? nt * 8 + g : 0) * xstride + (uint32_t)q * 4u;
  const uint8_t *xsc = c.s.xtile + align16u((uint32_t)B * xstride);
  const uint8_t *wsc = xsc + align16u((uint32_t)(B * NG));
  const uint8_t *xsc0 = xsc + (size_t)(nt * 8 + 2 * q) * NG, *xsc1 = xsc0 + NG;
  int group_seq = 0;
  for (int kt = 0; kt < K; kt += KT) {
    if (B > 0) {
      if (kt > 0) consumer_sync();
      stage_fp8(c, d, B, kt, KT, !((d.flags & TF_SAME_X_AS_PREV) && !multi_tile));
    }
    int gi = 0;
    for (int r0 = n0; r0 < n1; r0 += R, ++gi) {
      float acc[4] = {0.f, 0.f, 0.f, 0.f};
      const uint8_t *wsc0 = wsc + (size_t)(r0 - n0 + g) * NG, *wsc1 = wsc0 + 8 * NG;
      for (int kc = 0; kc < KT; kc += KC) {
        const int s = stage;
        const uint32_t ph = phase;
        if (++stage == NST) { stage = 0; phase ^= 1u; }
        if (ok) ok = wait_mbar(c, &c.s.full[s], ph, task);
        if (ok && B > 0) {
          const uint32_t a_base = smem_u32(c.s.stages + (size_t)s * P.stage_bytes) + a_lane_off;
          const uint32_t x_base = x_lane_base + (uint32_t)kc;
          for (int m = ks; m < ngc; m += kstride) {
            uint32_t a[4][4], b[4][2];
#pragma unroll
            for (int u = 0; u < 4; ++u) {
              const uint32_t o = (uint32_t)(m * 4 + u) * 32u;
              ldmatrix_x4(a[u], a_base + o);
              asm volatile("ld.shared.b32 %0, [%1];" : "=r"(b[u][0]) : "r"(x_base + o));
              asm volatile("ld.shared.b32 %0, [%1];" : "=r"(b[u][1]) : "r"(x_base + o + 16u));
            }
            float t0[4] = {0.f, 0.f, 0.f, 0.f}, t1[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
            for (int u = 0; u < 4; ++u) {
              if (!tok_valid) b[u][0] = b[u][1] = 0u;
              if (u & 1) mma_e4m3_16832(t1, a[u], b[u][0], b[u][1]);
              else mma_e4m3_16832(t0, a[u], b[u][0], b[u][1]);
            }
            const int gt = kc / 128 + m;
            const uint32_t ew0 = wsc0[gt], ew1 = wsc1[gt], ea0 = xsc0[gt], ea1 = xsc1[gt];
            acc[0] += (t0[0] + t1[0]) * ue8m0_pair_scale(ew0, ea0);
            acc[1] += (t0[1] + t1[1]) * ue8m0_pair_scale(ew0, ea1);
            acc[2] += (t0[2] + t1[2]) * ue8m0_pair_scale(ew1, ea0);
            acc[3] += (t0[3] + t1[3]) * ue8m0_pair_scale(ew1, ea1);
          }
        }
        __syncwarp();
        if (lane == 0) mbar_arrive(&c.s.empty[s]);
      }
      if (B > 0) {
        float *part = c.s.partial + (size_t)((multi_tile ? gi : group_seq) & 1) * (8 * 16 * 8);
        float *mine = part + (size_t)warp * (16 * 8);
        float2 *p0 = reinterpret_cast<float2 *>(mine + g * 8 + q * 2);
        float2 *p1 = reinterpret_cast<float2 *>(mine + (g + 8) * 8 + q * 2);
        if (multi_tile && kt > 0) {
          float2 o0 = *p0, o1 = *p1;
          *p0 = make_float2(o0.x + acc[0], o0.y + acc[1]);
          *p1 = make_float2(o1.x + acc[2], o1.y + acc[3]);
        } else {
          *p0 = make_float2(acc[0], acc[1]);
          *p1 = make_float2(acc[2], acc[3]);
        }
        if (!multi_tile) {
          consumer_sync();
          linear_group_epilogue<true, 0>(c, d, B, NT, r0, min(R, n1 - r0), part);
        }
      }
      ++group_seq;
    }
  }
  if (!ok) c.s.flags[0] = 1;
  if (B > 0 && multi_tile) {
    consumer_sync();
    int gi = 0;
    for (int r0 = n0; r0 < n1; r0 += R, ++gi)
      linear_group_epilogue<true, 0>(c, d, B, NT, r0, min(R, n1 - r0), c.s.partial + (size_t)(gi & 1) * (8 * 16 * 8));
  }
  ls.stage = stage;
  ls.phase = phase;
}

// TASK_QUANTIZE_FP8: bf16 -> e4m3 with one scale per (row, 128 columns); a warp owns a pack of four groups.
// Follows per_token_group_quantize_fp8 (include/mirage/persistent_kernel/tasks/blackwell/
// per_token_group_quantize_fp8.cuh:33-160): amax clamped at 1e-10, scale = amax / 448, for UE8M0 rounded up
// to a power of two (computed on the exponent bits, which is exact) and packed four to a uint32 word.
static __device__ void run_quantize_fp8(const Ctx &c, const TaskDesc &d) {
  const KernelParams &P = c.P;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int K = d.a[2], ldx = d.a[3], ldq = d.a[4], per_tok = d.a[6], s0 = d.a[7], s1 = d.a[8], pk = d.a[9];
  const bool ue8m0 = d.a[5] != 0;
  const int ng = K / 128;
  const int active = active_tokens(P);
  const __nv_bfloat16 *x = reinterpret_cast<const __nv_bfloat16 *>(d.p[0]);
  uint8_t *qo = reinterpret_cast<uint8_t *>(d.p[1]);
  for (int u = d.a[0] + warp; u < d.a[1]; u += kConsumerThreads / 32) {
    const int row = u / pk, j = u - row * pk;
    if (row / per_tok >= active) continue;
    uint32_t word = 0;
    for (int gi = 0; gi < 4; ++gi) {
      const int gidx = j * 4 + gi;
      if (gidx >= ng) break;
      const uint2 raw = __ldcg(reinterpret_cast<const uint2 *>(x + (size_t)row * ldx + (size_t)gidx * 128) + lane);
      float v[4];
      v[0] = __uint_as_float(raw.x << 16); v[1] = __uint_as_float(raw.x & 0xffff0000u);
      v[2] = __uint_as_float(raw.y << 16); v[3] = __uint_as_float(raw.y & 0xffff0000u);
      float amax = fmaxf(fmaxf(fabsf(v[0]), fabsf(v[1])), fmaxf(fabsf(v[2]), fabsf(v[3])));
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, o));
      amax = fmaxf(amax, 1e-10f);
      float scale = __fdiv_rn(amax, 448.0f);
      if (ue8m0) {
        const uint32_t bits = __float_as_uint(scale);
        uint32_t e = (bits >> 23) & 0xffu;
        if (bits & 0x7fffffu) ++e;                 // ceil(log2(scale)) + 127
        e = min(e, 254u);
        scale = __uint_as_float(e << 23);
        word |= e << (8 * gi);
      } else if (lane == 0) {
        reinterpret_cast<float *>(d.p[2])[(size_t)row * s0 + (size_t)gidx * s1] = scale;
      }
      float qv[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) qv[i] = fminf(fmaxf(__fdiv_rn(v[i], scale), -448.0f), 448.0f);
      const uint32_t lo = __nv_cvt_float2_to_fp8x2(make_float2(qv[0], qv[1]), __NV_SATFINITE, __NV_E4M3);
      const uint32_t hi = __nv_cvt_float2_to_fp8x2(make_float2(qv[2], qv[3]), __NV_SATFINITE, __NV_E4M3);
      *reinterpret_cast<uint32_t *>(qo + (size_t)row * ldq + (size_t)gidx * 128 + (size_t)lane * 4) = lo | (hi << 16);
    }
    if (ue8m0 && lane == 0) reinterpret_cast<uint32_t *>(d.p[2])[(size_t)row * s0 + (size_t)j * s1] = word;
  }
}

// ---------------------------------------------------------------------------
// Mixture of experts (general instantiation only)
// ---------------------------------------------------------------------------
// TASK_MOE_ROUTING: DeepSeek-V3 group-aware sigmoid routing, one warp per token
// (include/mirage/persistent_kernel/tasks/blackwell/topk_sigmoid_sm100.cuh:75-362): selection on
// sigmoid + bias, group score = sum of the group's two largest biased scores, `keep` groups survive (ties: lowest
// group), top-k experts by repeated argmax (ties: lowest expert), weights from the unbiased scores.  The list of
// active experts is written in ascending order (the reference's order depends on atomics).  The logits are
// zeroed after they are read, as the reference does for its accumulating gate projection.
static __device__ void run_moe_routing(const Ctx &c, const TaskDesc &d) {
  const KernelParams &P = c.P;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int E = d.a[0], topk = d.a[1], groups = d.a[2], keep = d.a[3];
  const float scaling = __int_as_float(d.a[4]);
  const int ldl = d.a[5], ldw = d.a[6], ldr = d.a[7];
  const bool f32_in = d.a[8] != 0;
  // expert parallelism: this rank runs experts [e_lo, e_hi) only.  Selection and normalisation are those of the whole
  // expert set (every rank computes the same routing); slots of experts of other ranks get weight 0 and stay out
  // of the active list, so the grouped projections skip them and the weighted sum ignores their rows.
  const int e_lo = d.a[9], e_hi = d.a[10];
  const int per = E / groups;
  const int B = min(active_tokens(P), ldr);
  float *wout = reinterpret_cast<float *>(d.p[2]);
  int *routing = reinterpret_cast<int *>(d.p[3]);
  int *active = reinterpret_cast<int *>(d.p[4]);
  const float *bias = reinterpret_cast<const float *>(d.p[1]);
  // shared: per warp [E] unbiased, [E] biased, [64] group scores; then [E] marks, [8] warp counts
  float *wbase = reinterpret_cast<float *>(c.s.xtile) + (size_t)warp * (2 * E + 64);
  float *sc = wbase, *bi = wbase + E, *gs = wbase + 2 * E;
  int *mark = reinterpret_cast<int *>(reinterpret_cast<float *>(c.s.xtile) + (size_t)8 * (2 * E + 64));
  int *wcount = mark + E;
  for (int i = tid; i < E * ldr; i += kConsumerThreads) routing[i] = 0;
  for (int i = tid; i < E; i += kConsumerThreads) mark[i] = 0;
  consumer_sync();
  const bool keep_logits = d.a[12] != 0;
  const bool softmax = d.a[11] != 0;   // moe_topk_softmax_routing_layer: scores = softmax over the experts, no bias, logits kept
  for (int row = warp; row < B; row += 8) {
    float row_max = -INFINITY;
    // eight logits of a lane at a time, loaded before the first is cleared: cleared one by one, the loads waited for one another
    for (int e0 = lane; e0 < E; e0 += 256) {
      float logit[8];
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        const int e = e0 + 32 * j;
        logit[j] = 0.f;
        if (e < E) logit[j] = f32_in ? __ldcg(reinterpret_cast<const float *>(d.p[0]) + (size_t)row * ldl + e)
                                     : bf16_to_f(__ldcg(reinterpret_cast<const __nv_bfloat16 *>(d.p[0]) + (size_t)row * ldl + e));
      }
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        const int e = e0 + 32 * j;
        if (e >= E) continue;
        if (!softmax && !keep_logits) {
          if (f32_in) reinterpret_cast<float *>(d.p[0])[(size_t)row * ldl + e] = 0.f;
          else reinterpret_cast<__nv_bfloat16 *>(d.p[0])[(size_t)row * ldl + e] = __float2bfloat16_rn(0.f);
        }
        if (softmax) {
          sc[e] = logit[j];
          row_max = fmaxf(row_max, logit[j]);
        } else {
          const float sig = __fdiv_rn(1.0f, 1.0f + expf(-logit[j]));
          sc[e] = sig;
          bi[e] = sig + __ldg(&bias[e]);
        }
      }
    }
    if (softmax) {
      // exp(x - max) / sum in fp32 (tasks/blackwell/topk_softmax_sm100.cuh:193-216); selection on the probabilities
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) row_max = fmaxf(row_max, __shfl_xor_sync(0xffffffffu, row_max, o));
      float row_sum = 0.f;
      for (int e = lane; e < E; e += 32) {
        const float p = expf(sc[e] - row_max);
        sc[e] = p;
        row_sum += p;
      }
      row_sum = warp_sum(row_sum);
      const float inv_sum = __fdiv_rn(1.0f, row_sum);
      for (int e = lane; e < E; e += 32) {
        const float p = sc[e] * inv_sum;
        sc[e] = p;
        bi[e] = p;
      }
    }
    __syncwarp();
    if (groups > 1) {   // (one group: nothing to choose between)
      // the two largest of a group: its lanes take every `share`-th expert (groups, a power of two up to 32, share the warp out), then meet
      const int share = groups <= 32 && (groups & (groups - 1)) == 0 && per >= 32 / groups && per > 1 ? 32 / groups : 0;
      if (share > 0) {
        const int g = lane / share, i0 = lane - g * share;
        float t1 = -INFINITY, t2 = -INFINITY;
        for (int i = i0; i < per; i += share) {
          const float v = bi[g * per + i];
          if (v > t1) { t2 = t1; t1 = v; }
          else if (v > t2) t2 = v;
        }
        for (int o = 1; o < share; o <<= 1) {
          const float u1 = __shfl_xor_sync(0xffffffffu, t1, o), u2 = __shfl_xor_sync(0xffffffffu, t2, o);
          t2 = fmaxf(fminf(t1, u1), fmaxf(t2, u2));
          t1 = fmaxf(t1, u1);
        }
        const float head = bi[g * per];   // (a group that begins with NaN is never chosen)
        if (i0 == 0) gs[g] = head == head ? t1 + fmaxf(t2, -1e30f) : head;
      }
      for (int g = lane; share == 0 && g < groups; g += 32) {
        float t1 = bi[g * per], t2 = -1e30f;
        for (int i = 1; i < per; ++i) {
          const float v = bi[g * per + i];
          if (v > t1) { t2 = t1; t1 = v; }
          else if (v > t2) t2 = v;
        }
        gs[g] = per > 1 ? t1 + t2 : t1;
      }
      __syncwarp();
      unsigned long long selected = 0ull;
      for (int k = 0; k < keep; ++k) {
        int best = 0;
        float best_s = -1e30f;
        for (int g = 0; g < groups; ++g)
          if (!((selected >> g) & 1ull) && gs[g] > best_s) { best_s = gs[g]; best = g; }
        selected |= 1ull << best;
      }
      for (int e = lane; e < E; e += 32)
        if (!((selected >> (e / per)) & 1ull)) bi[e] = -10000.f;
      __syncwarp();
    }
    float total = 0.f;
    float mine = 0.f;   // lane k < topk: slot k's weight (0: its expert belongs to another rank)
    for (int k = 0; k < topk; ++k) {
      float mv = -3.0e38f;
      int me = E;
      for (int e = lane; e < E; e += 32) {
        const float v = bi[e];
        if (v > mv) { mv = v; me = e; }
      }
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) {
        const float ov = __shfl_xor_sync(0xffffffffu, mv, o);
        const int oe = __shfl_xor_sync(0xffffffffu, me, o);
        if (ov > mv || (ov == mv && oe < me)) { mv = ov; me = oe; }
      }
      const float orig = sc[me];
      const bool local = me >= e_lo && me < e_hi;
      total += orig;
      if (lane == k && local) mine = orig;
      __syncwarp();
      if (lane == 0) {
        if (local) {
          routing[(size_t)me * ldr + row] = k + 1;
          mark[me] = 1;
        }
        bi[me] = -10000.f;
      }
      __syncwarp();
    }
    const float inv = d.a[13] ? 1.0f : __fdiv_rn(1.0f, total + 1e-20f);
    if (lane < topk) wout[(size_t)row * ldw + lane] = mine * inv * scaling;
    __syncwarp();
  }
  consumer_sync();
  // ascending list of the experts that received a token; count at index E, unused entries -1
  int base = 0;
  for (int e0 = 0; e0 < E; e0 += kConsumerThreads) {
    const int e = e0 + tid;
    const bool on = e < E && mark[e] != 0;
    const unsigned bal = __ballot_sync(0xffffffffu, on);
    if (lane == 0) wcount[warp] = __popc(bal);
    consumer_sync();
    int before = base;
    for (int w = 0; w < warp; ++w) before += wcount[w];
    if (on) active[before + __popc(bal & ((1u << lane) - 1u))] = e;
    int all = 0;
    for (int w = 0; w < 8; ++w) all += wcount[w];
    base += all;
    consumer_sync();
  }
  for (int i = base + tid; i < E; i += kConsumerThreads) active[i] = -1;
  if (tid == 0) active[E] = base;
}

// TASK_MOE_GEMM: out[b, slot, n0:n1] = x_row . W[e, n, :] for every active expert e and every token routed to it
// (moe_w13 / moe_w2, bf16 or e4m3 with float32 scales per 128 columns; the scales are floored to powers of two
// by taking their exponent bits, as fp8_group_gemm_sm100.cuh:1378 does).  The task owns the row range [n0, n1) of
// EVERY expert: all workers walk the same active list, so the load is balanced whatever the routing.  The
// streamer walks the same list (it waits for the routing first) and streams the panel of each active expert.
template <bool HYBRID>
__device__ void run_moe_gemm(const Ctx &c, const TaskDesc &d, LinearState &ls, int task, bool ok) {
  const KernelParams &P = c.P;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  int stage = ls.stage;
  uint32_t phase = ls.phase;
  const bool fp8 = !HYBRID && (d.flags & TF_FP8) != 0;
  const uint32_t esz = fp8 ? 1u : 2u;
  const int Bt = ok ? min(active_tokens(P), kMaxLinearTokens) : 0;
  const int n0 = d.a[L_N0], n1 = d.a[L_N1], K = d.a[L_K], N = d.a[L_N];
  const int KT = d.a[L_KT], KC = d.a[L_KC], R = d.a[L_ROWS];
  const int E = d.a[M_NEXP], topk = d.a[M_NTOPK], ldr = d.a[M_LDR];
  const bool per_slot = d.a[M_PER_SLOT] != 0;
  const int NST = P.num_stages;
  const uint32_t seg = (uint32_t)KC * esz, row_stride = seg + kRowPadBytes;
  const uint32_t xstride = (uint32_t)KT * esz + kRowPadBytes;
  const int NG = fp8 ? KT / 128 : 0, ngtot = K / 128;
  const int g = lane >> 2, q = lane & 3;
  const int nkt = K / KT;
  const bool multi_tile = nkt > 1;
  const int *routing = reinterpret_cast<const int *>(d.p[4]);
  const int *active = reinterpret_cast<const int *>(d.p[5]);
  // token | slot << 8 of an expert's tokens (token < 64, slot < 255): two lists, the expert being computed and the next
  unsigned short *tokmaps = reinterpret_cast<unsigned short *>(c.s.red);
  int *cnt_s = c.s.flags + 8;
  const int n_act = ok ? min(__ldcg(&active[E]), E) : 0;
  const uint32_t a_lane_off = (uint32_t)(lane & 15) * row_stride + (uint32_t)(lane >> 4) * 16u;
  const uint8_t *xg = reinterpret_cast<const uint8_t *>(d.p[1]);
  __nv_bfloat16 *out = reinterpret_cast<__nv_bfloat16 *>(d.p[2]);
  if (n_act <= 0) {
    if (!ok) c.s.flags[0] = 1;
    return;
  }
  // The loop runs over steps (expert, k tile).  A step's operands -- the gathered activation rows of the expert's
  // tokens, their float32 scales and the scales of this task's weight rows, copied raw (the power-of-two floor is
  // taken from the exponent bits where they are used) -- live in a region of the activation tile: rows, token
  // scales, weight-row scales.  While one step computes, the token list of the next expert is built and the next
  // step's operands are copied asynchronously into the free part of the tile (after the current region, or in front
  // of it), so that a step does not begin with a round trip to global memory; a step whose operands do not fit beside
  // the current ones is staged after it.
  auto region_bytes = [&](int cnt) -> uint32_t {
    const int n = max(cnt, 1);
    return align16u((uint32_t)n * xstride) + 4u * (uint32_t)((n * NG + 3) & ~3) + align16u(4u * (uint32_t)((n1 - n0) * NG));
  };
  // routing entries of one expert, held by warps 0 and 1 (token = warp * 32 + lane)
  auto load_routing = [&](int j) -> int {
    if (warp >= 2 || j >= n_act) return 0;
    const int b = warp * 32 + lane;
    return (b < Bt) ? __ldcg(&routing[(size_t)__ldcg(&active[j]) * ldr + b]) : 0;
  };
  // warps 0 and 1: the expert's tokens in token order -> list `which`, counts -> cnt_s[0..1]
  auto build_tokmap = [&](int r, int which) {
    if (warp < 2) {
      unsigned short *tm = tokmaps + which * 64;
      const int b = warp * 32 + lane;
      const unsigned bal = __ballot_sync(0xffffffffu, r != 0);
      if (lane == 0) cnt_s[warp] = __popc(bal);
      if (warp == 0 && r != 0) tm[__popc(bal & ((1u << lane) - 1u))] = (unsigned short)(b | ((r - 1) << 8));
      asm volatile("bar.sync 2, 64;");   // the second half is appended after the first: it needs that count
      if (warp == 1 && r != 0) tm[cnt_s[0] + __popc(bal & ((1u << lane) - 1u))] = (unsigned short)(b | ((r - 1) << 8));
    }
  };
  // asynchronous copies of one step's operands into the region at `off` (committed, not waited for)
  auto stage_step = [&](int e, int cnt, int which, int kt, uint32_t off) {
    const unsigned short *tm = tokmaps + which * 64;
    uint8_t *xr = c.s.xtile + off;
    float *xsc = reinterpret_cast<float *>(xr + align16u((uint32_t)max(cnt, 1) * xstride));
    float *wsc = xsc + (size_t)((max(cnt, 1) * NG + 3) & ~3);
    const int vecs = (int)((uint32_t)KT * esz / 16u);
    for (int i = tid; i < cnt * vecs; i += kConsumerThreads) {
      const int t = i / vecs, v = i - t * vecs;
      const int tmv = tm[t];
      const size_t xrow = per_slot ? (size_t)(tmv & 0xff) * topk + (tmv >> 8) : (size_t)(tmv & 0xff);
      asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(smem_u32(xr + (size_t)t * xstride + (size_t)v * 16)),
                   "l"(reinterpret_cast<const uint4 *>(xg + (xrow * d.a[L_LDX] + kt) * esz) + v)
                   : "memory");
    }
    if constexpr (!HYBRID) if (fp8) {
      const float *xs = reinterpret_cast<const float *>(d.p[7]);
      const float *ws = reinterpret_cast<const float *>(d.p[6]);
      const int g0 = kt / 128;
      if (((NG | ngtot) & 3) == 0) {
        // four scales per copy: a row's scales of this k tile are NG consecutive floats, 16-byte aligned on both sides
        const int nv = NG >> 2;
        for (int i = tid; i < cnt * nv; i += kConsumerThreads) {
          const int t = i / nv, v = i - t * nv;
          const int tmv = tm[t];
          const size_t xrow = per_slot ? (size_t)(tmv & 0xff) * topk + (tmv >> 8) : (size_t)(tmv & 0xff);
          asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(smem_u32(xsc + (size_t)t * NG + v * 4)),
                       "l"(&xs[xrow * ngtot + g0 + v * 4])
                       : "memory");
        }
        for (int i = tid; i < (n1 - n0) * nv; i += kConsumerThreads) {
          const int r = i / nv, v = i - r * nv;
          asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(smem_u32(wsc + (size_t)r * NG + v * 4)),
                       "l"(&ws[((size_t)e * N + n0 + r) * ngtot + g0 + v * 4])
                       : "memory");
        }
      } else {
        for (int i = tid; i < cnt * NG; i += kConsumerThreads) {
          const int t = i / NG, gi = i - t * NG;
          const int tmv = tm[t];
          const size_t xrow = per_slot ? (size_t)(tmv & 0xff) * topk + (tmv >> 8) : (size_t)(tmv & 0xff);
          asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(smem_u32(xsc + i)), "l"(&xs[xrow * ngtot + g0 + gi]) : "memory");
        }
        for (int i = tid; i < (n1 - n0) * NG; i += kConsumerThreads) {
          const int r = i / NG, gi = i - r * NG;
          asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(smem_u32(wsc + i)),
                       "l"(&ws[((size_t)e * N + n0 + r) * ngtot + g0 + gi])
                       : "memory");
        }
      }
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };

  // first step: token list and operands of the first expert, synchronously
  consumer_sync();
  int r_next = load_routing(0);
  build_tokmap(r_next, 0);
  r_next = load_routing(1);
  consumer_sync();
  int cnt = cnt_s[0] + cnt_s[1];
  uint32_t off = 0;
  stage_step(__ldcg(&active[0]), cnt, 0, 0, 0u);
  asm volatile("cp.async.wait_group 0;" ::: "memory");
  consumer_sync();

  for (int j = 0; j < n_act; ++j) {
    const int e = __ldcg(&active[j]);
    const int which = j & 1;
    const unsigned short *tokmap = tokmaps + which * 64;
    const int NT = cnt <= 8 ? 1 : (cnt <= 16 ? 2 : (cnt <= 32 ? 4 : 8));
    const int nt = warp % NT, ks = warp / NT, kstride = 8 / NT;
    const bool tok_valid = nt * 8 + g < cnt;
    for (int kt = 0, kti = 0; kt < K; kt += KT, ++kti) {
      // ---- the next step: token list (new expert) and operand copies ----
      const bool last_tile = kti == nkt - 1;
      const bool has_next = !(last_tile && j == n_act - 1);
      int cnt_n = cnt;
      if (has_next && last_tile) {
        build_tokmap(r_next, which ^ 1);
        r_next = load_routing(j + 2);
        consumer_sync();
        cnt_n = cnt_s[0] + cnt_s[1];
      }
      const int e_n = last_tile ? (has_next ? __ldcg(&active[j + 1]) : e) : e;
      const int which_n = last_tile ? which ^ 1 : which;
      const int kt_n = last_tile ? 0 : kt + KT;
      const uint32_t need_c = region_bytes(cnt), need_n = region_bytes(cnt_n);
      uint32_t off_n = off + need_c;
      bool ahead = has_next;
      if (off_n + need_n > (uint32_t)P.x_tile_bytes) {
        off_n = 0;
        if (need_n > off) ahead = false;
      }
      if (has_next && ahead) stage_step(e_n, cnt_n, which_n, kt_n, off_n);

      // ---- this step ----
      const uint8_t *xr = c.s.xtile + off;
      const float *xsc = reinterpret_cast<const float *>(xr + align16u((uint32_t)max(cnt, 1) * xstride));
      const float *wsc = xsc + (size_t)((max(cnt, 1) * NG + 3) & ~3);
      const float *xsc0 = xsc + (size_t)(nt * 8 + 2 * q) * NG, *xsc1 = xsc0 + NG;
      const uint32_t x_lane_base = smem_u32(xr) + (uint32_t)(tok_valid ? nt * 8 + g : 0) * xstride + (uint32_t)q * 4u;
      int gi = 0;
      for (int r0 = n0; r0 < n1; r0 += R, ++gi) {
        float acc[4] = {0.f, 0.f, 0.f, 0.f};
        const float *wsc0 = wsc + (size_t)(r0 - n0 + g) * NG, *wsc1 = wsc0 + 8 * NG;
        for (int kc = 0; kc < KT; kc += KC) {
          const int s = stage;
          const uint32_t ph = phase;
          if (++stage == NST) { stage = 0; phase ^= 1u; }
          if (ok) ok = wait_mbar(c, &c.s.full[s], ph, task);
          if (ok && cnt > 0) {
            const uint32_t a_base = smem_u32(c.s.stages + (size_t)s * P.stage_bytes) + a_lane_off;
            const uint32_t x_base = x_lane_base + (uint32_t)kc * esz;
            const int nquad = (int)(seg / 128u);          // groups of four 32-byte k steps
            for (int m = ks; m < nquad; m += kstride) {
              uint32_t a[4][4], b[4][2];
#pragma unroll
              for (int u = 0; u < 4; ++u) {
                const uint32_t o = (uint32_t)(m * 4 + u) * 32u;
                ldmatrix_x4(a[u], a_base + o);
                asm volatile("ld.shared.b32 %0, [%1];" : "=r"(b[u][0]) : "r"(x_base + o));
                asm volatile("ld.shared.b32 %0, [%1];" : "=r"(b[u][1]) : "r"(x_base + o + 16u));
                if (!tok_valid) b[u][0] = b[u][1] = 0u;
              }
              if (fp8) {
                float t0[4] = {0.f, 0.f, 0.f, 0.f}, t1[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
                for (int u = 0; u < 4; ++u) {
                  if (u & 1) mma_e4m3_as_f16(t1, a[u], b[u][0], b[u][1]);
                  else mma_e4m3_as_f16(t0, a[u], b[u][0], b[u][1]);
                }
                const int gt = kc / 128 + m;
                const uint32_t ew0 = (__float_as_uint(wsc0[gt]) >> 23) & 0xffu, ew1 = (__float_as_uint(wsc1[gt]) >> 23) & 0xffu;
                const uint32_t ea0 = (__float_as_uint(xsc0[gt]) >> 23) & 0xffu, ea1 = (__float_as_uint(xsc1[gt]) >> 23) & 0xffu;
                acc[0] += (t0[0] + t1[0]) * ue8m0_pair_scale(ew0, ea0);
                acc[1] += (t0[1] + t1[1]) * ue8m0_pair_scale(ew0, ea1);
                acc[2] += (t0[2] + t1[2]) * ue8m0_pair_scale(ew1, ea0);
                acc[3] += (t0[3] + t1[3]) * ue8m0_pair_scale(ew1, ea1);
              } else {
#pragma unroll
                for (int u = 0; u < 4; ++u) mma_bf16_16816(acc, a[u], b[u][0], b[u][1]);
              }
            }
          }
          __syncwarp();
          if (lane == 0) mbar_arrive(&c.s.empty[s]);
        }
        // partial tiles of the eight warps: two buffers, used by row groups in turn (a task with several k tiles has
        // at most two row groups, whose partials stay there across the tiles)
        float *part = c.s.partial + (size_t)(gi & 1) * (8 * 16 * 8);
        float *mine = part + (size_t)warp * (16 * 8);
        float2 *p0 = reinterpret_cast<float2 *>(mine + g * 8 + q * 2);
        float2 *p1 = reinterpret_cast<float2 *>(mine + (g + 8) * 8 + q * 2);
        if (kti > 0) {
          float2 o0 = *p0, o1 = *p1;
          *p0 = make_float2(o0.x + acc[0], o0.y + acc[1]);
          *p1 = make_float2(o1.x + acc[2], o1.y + acc[3]);
        } else {
          *p0 = make_float2(acc[0], acc[1]);
          *p1 = make_float2(acc[2], acc[3]);
        }
        // after the last k tile: sum the warps' partials and write the rows, for the two row groups held at a time
        const bool pair_done = (gi & 1) == 1 || r0 + R >= n1;
        if (last_tile && pair_done) {
          consumer_sync();
          for (int gg = gi & ~1; gg <= gi; ++gg) {
            const float *pp = c.s.partial + (size_t)(gg & 1) * (8 * 16 * 8);
            const int rbase = n0 + gg * R;
            const int rows = min(R, n1 - rbase);
            for (int item = tid; item < cnt * 16; item += kConsumerThreads) {
              const int t = item >> 4, r = item & 15;
              if (r >= rows) continue;
              float v = 0.f;
              for (int w = t >> 3; w < 8; w += NT) v += pp[(w * 16 + r) * 8 + (t & 7)];
              const int tmv = tokmap[t];
              const size_t orow = ((size_t)(tmv & 0xff) * topk + (tmv >> 8)) * d.a[L_LDO];
              if (HYBRID && d.a[L_EPI] == EPI_STORE_F32) {
                reinterpret_cast<float *>(out)[orow + rbase + r] = v;
              } else if (HYBRID && d.a[L_EPI] == EPI_RELU2) {
                const float a = fmaxf(v, 0.f);
                out[orow + rbase + r] = __float2bfloat16_rn(a * a);
              } else if (HYBRID && d.a[L_EPI] >= EPI_GATED_SILU) {   // rows [gate, gate, up, up]
                if (r & 2) continue;
                float u = 0.f;
                for (int w = t >> 3; w < 8; w += NT) u += pp[(w * 16 + r + 2) * 8 + (t & 7)];
                const float a = d.a[L_EPI] == EPI_GATED_SILU ? silu_exact_f(v) : gelu_tanh_f(v);
                out[orow + (((rbase + r) >> 2) << 1) + (r & 1)] = __float2bfloat16_rn(a * u);
              } else {
                out[orow + rbase + r] = __float2bfloat16_rn(v);
              }
            }
          }
          if (r0 + R < n1) consumer_sync();   // further row groups reuse the buffers
        }
      }
      // ---- hand over to the next step ----
      if (has_next && !ahead) {
        consumer_sync();                     // every warp is done with the current region
        stage_step(e_n, cnt_n, which_n, kt_n, 0u);
      }
      asm volatile("cp.async.wait_group 0;" ::: "memory");
      consumer_sync();
      off = off_n;
      cnt = cnt_n;
    }
  }
  if (!ok) c.s.flags[0] = 1;
  ls.stage = stage;
  ls.phase = phase;
}

// TASK_MOE_SILU_MUL: rows of [gate | up] -> bf16(silu(gate)) * up  (tasks/ampere/silu_mul.cuh:20-42 on the
// flattened [token x slot] rows, as register_moe_silu_mul_task sets it up)
// Expert projections on tcgen05 (bf16 hybrid graphs of more than 8 batched tokens).  A row tile of an active expert is a linear of
// RB <= 128 rows over the tokens routed to it: the weight tile streams through the ring as swizzled boxes, the tokens' rows are
// gathered into the operand tile (N = their number rounded up to 16), eight warps issue MMAs into accumulators of their own, and the
// epilogue scatters to (token, slot) rows.  Row tiles are dealt out to the workers in turn, whatever the routing; the next tile's
// token rows are gathered while the current one's MMAs run where both fit.
static __device__ void run_moe_gemm_tc(const Ctx &c, const TaskDesc &d, LinearState &ls, int task, bool ok) {
  const KernelParams &P = c.P;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int B = ok ? min(active_tokens(P), kMaxLinearTokens) : 0;
  const int K = d.a[L_K], RB = d.a[L_ROWS], N = d.a[L_N], E = d.a[M_NEXP], topk = d.a[M_NTOPK], ldr = d.a[M_LDR], ldx = d.a[L_LDX];
  const int nkb = d.a[L_KC] / kTcKBlock, kball = K / kTcKBlock, per = (N + RB - 1) / RB, step = d.a[L_N1], epi = d.a[L_EPI], ldo = d.a[L_LDO];
  const bool per_slot = d.a[M_PER_SLOT] != 0;
  const int NST = P.num_stages, stage_bytes = P.stage_bytes, room = P.x_tile_bytes;
  const int *routing = reinterpret_cast<const int *>(d.p[4]), *active = reinterpret_cast<const int *>(d.p[5]);
  const uint8_t *xg = reinterpret_cast<const uint8_t *>(d.p[1]);
  uint8_t *out = reinterpret_cast<uint8_t *>(d.p[2]);
  const int items = ok ? min(__ldcg(&active[E]), E) * per : 0;
  unsigned short *lists = reinterpret_cast<unsigned short *>(c.s.red);   // two lists of token | slot << 8
  int *cnt_s = c.s.flags + 8;                                            // their lengths: [list][half]
  const uint32_t x0 = smem_u32(c.s.xtile), st0 = smem_u32(c.s.stages), tmem = c.tmem_base;
  const uint64_t desc_hi = umma_desc_k_sw128(0);
  // warps 0 and 1: the expert's tokens; complete after the next barrier of the compute warps
  auto build = [&](int it, int which) {
    if (warp < 2) {
      const int b = warp * 32 + lane;
      const int r = b < B ? __ldcg(&routing[(size_t)__ldcg(&active[it / per]) * ldr + b]) : 0;
      const unsigned bal = __ballot_sync(0xffffffffu, r != 0);
      if (lane == 0) cnt_s[2 * which + warp] = __popc(bal);
      asm volatile("bar.sync 2, 64;");
      if (r != 0) lists[which * 64 + (warp ? cnt_s[2 * which] : 0) + __popc(bal & ((1u << lane) - 1u))] = (unsigned short)(b | ((r - 1) << 8));
    }
  };
  // asynchronous copies of columns [k0, k0 + kn) of the list's token rows into the operand tile at `off` (committed)
  auto gather = [&](int which, int cnt, int NP, int k0, int kn, uint32_t off) {
    const int vecs = kn >> 3;
    for (int i = tid; i < cnt * vecs; i += kConsumerThreads) {
      const int t = i / vecs, v = i - t * vecs, tm = lists[which * 64 + t];
      const size_t row = per_slot ? (size_t)(tm & 0xff) * topk + (tm >> 8) : (size_t)(tm & 0xff);
      asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(x0 + off + (uint32_t)((v >> 3) * NP * 128 + t * 128 + (((v & 7) ^ (t & 7)) << 4))),
                   "l"(xg + (row * ldx + k0) * 2 + (size_t)v * 16)
                   : "memory");
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  auto padded = [](int cnt) { return max(16, (cnt + 15) & ~15); };
  int it = d.a[L_N0], which = 0, stage = ls.stage;
  uint32_t phase = ls.phase, off = 0;
  bool staged = false;
  if (it < items) {
    build(it, 0);
    consumer_sync();
  }
  for (; it < items && ok; it += step, which ^= 1) {
    const int cnt = cnt_s[2 * which] + cnt_s[2 * which + 1], NP = padded(cnt);
    const int KT = min(K, room / (NP * 128) / nkb * nkb * kTcKBlock);
    const int row0 = it % per * RB;
    const uint32_t idesc = umma_idesc(1u, 128, NP);
    const int sets = min(8, kTcAccCols / NP);
    const bool more = it + step < items;
    tc_fence_after_sync();
    if (warp < 4) {
      for (int col = 0; col < sets * NP; col += 16) tmem_st_zero_x16(tmem + ((uint32_t)(warp * 32) << 16) + (uint32_t)col);
      tmem_st_wait();
    }
    tc_fence_before_sync();
    uint32_t off_n = 0;
    bool staged_n = false;
    for (int k0 = 0; k0 < K; k0 += KT) {
      const int kn = min(KT, K - k0);
      if (!staged || k0 > 0) gather(which, cnt, NP, k0, kn, k0 > 0 ? 0u : off);
      if (k0 == 0 && more) build(it + step, which ^ 1);
      asm volatile("cp.async.wait_group 0;" ::: "memory");
      fence_proxy_async_smem();   // the tile was written through the generic proxy; the MMA reads it through the async proxy
      consumer_sync();
      tc_fence_after_sync();
      if (k0 == 0 && more && KT == K) {
        const int cn = cnt_s[2 * (which ^ 1)] + cnt_s[2 * (which ^ 1) + 1], NPn = padded(cn);
        const uint32_t mine = (uint32_t)(NP * 2 * K), next = (uint32_t)(NPn * 2 * K);
        off_n = off + mine;
        staged_n = off_n + next <= (uint32_t)room;
        if (!staged_n && next <= off) { off_n = 0; staged_n = true; }
        if (staged_n) gather(which ^ 1, cn, NPn, 0, K, off_n);
        else off_n = 0;
      }
      const uint32_t xb = (x0 + (k0 > 0 ? 0u : off)) >> 4;
      for (int kb = 0; kb < kn / kTcKBlock; kb += nkb) {
        const int s = stage;
        const uint32_t ph = phase;
        if (++stage == NST) { stage = 0; phase ^= 1u; }
        if (ok) ok = wait_mbar(c, &c.s.full[s], ph, task);
        if (ok && lane == 0) {
          tc_fence_after_sync();
          const uint32_t a_base = (st0 + (uint32_t)(s * stage_bytes)) >> 4;
          for (int m = warp; warp < sets && m < nkb * 4; m += sets) {
            const int j = m >> 2, kk = m & 3;
            umma_bf16_acc(tmem + (uint32_t)(warp * NP), desc_hi | (a_base + (uint32_t)(j * RB * 8 + kk * 2)),
                          desc_hi | (xb + (uint32_t)((kb + j) * NP * 8 + kk * 2)), idesc);
          }
          umma_commit(&c.s.empty[s]);
        }
        __syncwarp();
      }
      // accumulators complete for these columns / operand tile free again: one arrival per warp
      if (lane == 0) umma_commit(c.s.acc_bar);
      if (!wait_mbar(c, c.s.acc_bar, ls.acc_phase, task)) ok = false;
      ls.acc_phase ^= 1u;
      if (!ok) c.s.flags[0] = 1;
      consumer_sync();
      ok = ok && (c.s.flags[0] == 0);
      if (!ok) break;
    }
    if (!ok) break;
    tc_fence_after_sync();
    const int quad = warp & 3, half = warp >> 2, nh = NP >> 1, r = quad * 32 + lane, row = row0 + r;
    if (quad * 32 < RB) {
      const bool row_ok = r < RB && row < N;
      const uint32_t taddr = tmem + ((uint32_t)(quad * 32) << 16) + (uint32_t)(half * nh);
      for (int c0 = 0; c0 < nh && half * nh + c0 < cnt; c0 += 8) {
        uint32_t v[8];
        tmem_ld_x8(taddr + (uint32_t)c0, v);
        for (int st = 1; st < sets; ++st) {   // the other issuers' accumulators, in set order
          uint32_t v2[8];
          tmem_ld_wait();
          tmem_ld_x8(taddr + (uint32_t)(st * NP + c0), v2);
          tmem_ld_wait();
#pragma unroll
          for (int j = 0; j < 8; ++j) v[j] = __float_as_uint(__uint_as_float(v[j]) + __uint_as_float(v2[j]));
        }
        tmem_ld_wait();
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          const float x = __uint_as_float(v[j]), u = __shfl_down_sync(0xffffffffu, x, 2);
          const int t = half * nh + c0 + j;
          if (!row_ok || t >= cnt) continue;
          const int tm = lists[which * 64 + t];
          const size_t orow = ((size_t)(tm & 0xff) * topk + (tm >> 8)) * ldo;
          if (epi == EPI_STORE_F32) reinterpret_cast<float *>(out)[orow + row] = x;
          else if (epi == EPI_STORE) reinterpret_cast<__nv_bfloat16 *>(out)[orow + row] = __float2bfloat16_rn(x);
          else if (epi == EPI_RELU2) reinterpret_cast<__nv_bfloat16 *>(out)[orow + row] = __float2bfloat16_rn(fmaxf(x, 0.f) * fmaxf(x, 0.f));
          else if ((row & 2) == 0)
            reinterpret_cast<__nv_bfloat16 *>(out)[orow + ((row >> 2) << 1) + (row & 1)] =
                __float2bfloat16_rn((epi == EPI_GATED_SILU ? silu_exact_f(x) : gelu_tanh_f(x)) * u);
        }
      }
    }
    tc_fence_before_sync();   // the accumulators have been read: the next item clears them after this barrier
    consumer_sync();
    staged = staged_n;
    off = off_n;
  }
  asm volatile("cp.async.wait_group 0;" ::: "memory");
  if (!ok) c.s.flags[0] = 1;
  ls.stage = stage;
  ls.phase = phase;
}

// Hybrid graphs (bf16 only): a function of its own, state of the stage ring by value, so that the linear loop's registers stay as
// they are.
template <bool GENERAL>
__device__ __noinline__ LinearState run_moe_gemm_hybrid(const Ctx c, const TaskDesc &d, LinearState ls, int task, bool ok) {
  if (GENERAL && (d.flags & TF_TC)) run_moe_gemm_tc(c, d, ls, task, ok);
  else run_moe_gemm<true>(c, d, ls, task, ok);
  return ls;
}

// Out of line: inlined beside the other bodies its loop comes out worse with 224 registers than with the 168 a function call gets
// (32 tokens, 103 experts: 2038 us inlined, 1926 us like this, 1870 to 1910 us before the register split).
static __device__ __noinline__ LinearState run_moe_gemm_decoder(const Ctx c, const TaskDesc &d, LinearState ls, int task, bool ok) {
  run_moe_gemm<false>(c, d, ls, task, ok);
  return ls;
}

static __device__ void run_moe_silu_mul(const Ctx &c, const TaskDesc &d) {
  const int I = d.a[2], ldi = d.a[3], ldo = d.a[4];
  const int r1 = min(d.a[1], active_tokens(c.P) * d.a[5]);
  const __nv_bfloat16 *in = reinterpret_cast<const __nv_bfloat16 *>(d.p[0]);
  __nv_bfloat16 *out = reinterpret_cast<__nv_bfloat16 *>(d.p[2]);
  for (int r = d.a[0]; r < r1; ++r)
    for (int j = threadIdx.x; j < I; j += kConsumerThreads) {
      const float gv = bf16_to_f(__ldcg(&in[(size_t)r * ldi + j]));
      const float uv = bf16_to_f(__ldcg(&in[(size_t)r * ldi + I + j]));
      const float a = round_bf16(gv / (1.0f + expf(-gv)));
      out[(size_t)r * ldo + j] = __float2bfloat16_rn(a * uv);
    }
}

// TASK_MOE_MUL_SUM_ADD: out[b, h] = residual[b, h] + sum_k in[b, k, h] * w[b, k]  (mul_sum_add_sm100.cuh:19-49)
static __device__ void run_moe_mul_sum_add(const Ctx &c, const TaskDesc &d) {
  const int c0 = d.a[0], c1 = d.a[1], H = d.a[2], topk = d.a[3], ldo = d.a[4], ldres = d.a[5], ldw = d.a[6];
  const int B = min(d.a[7], active_tokens(c.P));
  const __nv_bfloat16 *in = reinterpret_cast<const __nv_bfloat16 *>(d.p[0]);
  const float *w = reinterpret_cast<const float *>(d.p[1]);
  const __nv_bfloat16 *res = reinterpret_cast<const __nv_bfloat16 *>(d.p[3]);
  __nv_bfloat16 *out = reinterpret_cast<__nv_bfloat16 *>(d.p[2]);
  if (((c0 | c1 | H | ldo | ldres) & 7) == 0 && ((d.p[0] | d.p[2] | d.p[3]) & 15) == 0) {
    // Eight columns of a token a thread, the slots' rows in flight together: a task holds 64 columns of every token, and walked
    // token by token, slot by slot it took 50 us for 32 tokens x 8 slots.  The sum runs in slot order as below.
    const int nv = (c1 - c0) >> 3;
    for (int i = threadIdx.x; i < nv * B; i += kConsumerThreads) {
      const int b = i / nv, h = c0 + ((i - b * nv) << 3);
      float acc[8];
      uint4 r = make_uint4(0, 0, 0, 0);
      if (res) r = __ldcg(reinterpret_cast<const uint4 *>(res + (size_t)b * ldres + h));
      const uint32_t rw[4] = {r.x, r.y, r.z, r.w};
#pragma unroll
      for (int q = 0; q < 4; ++q) { acc[2 * q] = bf16_lo(rw[q]); acc[2 * q + 1] = bf16_hi(rw[q]); }
      for (int k0 = 0; k0 < topk; k0 += 4) {
        float wk[4];
        uint4 x[4];
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          wk[k] = k0 + k < topk ? __ldcg(&w[(size_t)b * ldw + k0 + k]) : 0.f;   // 0: the row may never have been written
          x[k] = make_uint4(0, 0, 0, 0);
          if (wk[k] != 0.f) x[k] = __ldcg(reinterpret_cast<const uint4 *>(in + ((size_t)b * topk + k0 + k) * H + h));
        }
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          if (wk[k] == 0.f) continue;
          const uint32_t xw[4] = {x[k].x, x[k].y, x[k].z, x[k].w};
#pragma unroll
          for (int q = 0; q < 4; ++q) {
            acc[2 * q] += bf16_lo(xw[q]) * wk[k];
            acc[2 * q + 1] += bf16_hi(xw[q]) * wk[k];
          }
        }
      }
      *reinterpret_cast<uint4 *>(out + (size_t)b * ldo + h) =
          make_uint4(pack_bf16(acc[0], acc[1]), pack_bf16(acc[2], acc[3]), pack_bf16(acc[4], acc[5]), pack_bf16(acc[6], acc[7]));
    }
    return;
  }
  for (int b = 0; b < B; ++b)
    for (int h = c0 + threadIdx.x; h < c1; h += kConsumerThreads) {
      float acc = res ? bf16_to_f(__ldcg(&res[(size_t)b * ldres + h])) : 0.f;
      for (int k = 0; k < topk; ++k) {
        const float wk = __ldcg(&w[(size_t)b * ldw + k]);   // 0: the slot's expert lives on another rank (row never written)
        if (wk != 0.f) acc += bf16_to_f(__ldcg(&in[((size_t)b * topk + k) * H + h])) * wk;
      }
      out[(size_t)b * ldo + h] = __float2bfloat16_rn(acc);
    }
}

// ---------------------------------------------------------------------------
// Multi-head latent attention decode (general instantiation only)
// ---------------------------------------------------------------------------
constexpr int kMlaDk = 576, kMlaDv = 512;
constexpr int kMlaRow = kMlaDk * 2 + 16;      // shared-memory row stride of q / kv rows (bytes, conflict-free ldmatrix)
constexpr int kMlaSub = 64;                   // kv rows per shared-memory tile
constexpr int kMlaSplit = 128;                // kv rows per split
constexpr int kMlaPRow = kMlaSub * 2 + 16;    // row stride of the probability tile

// TASK_MLA_APPEND: the request's new [c_latent | k_pe] rows go to their positions in the paged cache
// (step 1 of mla_kv_cache_gather_sm100.cuh:36-128; the decode tasks read the paged cache in place, so the
// reference's second step -- copying the whole sequence to a contiguous buffer -- has no counterpart).
static __device__ void run_mla_append(const Ctx &c, const TaskDesc &d) {
  const KernelParams &P = c.P;
  const int slot = d.a[0], ldc = d.a[1], ldp = d.a[2], page = d.a[3], dk = d.a[4], dv = d.a[5];
  const int q0 = __ldcg(&P.meta.qo_indptr[slot]);
  const int nq = __ldcg(&P.meta.qo_indptr[slot + 1]) - q0;
  const int kv0 = __ldcg(&P.meta.paged_kv_indptr[slot]);
  const int npages = __ldcg(&P.meta.paged_kv_indptr[slot + 1]) - kv0;
  if (nq <= 0 || npages <= 0) return;
  const int seq_len = (npages - 1) * page + __ldcg(&P.meta.paged_kv_last_page_len[slot]);
  const __nv_bfloat16 *lat = reinterpret_cast<const __nv_bfloat16 *>(d.p[0]);
  const __nv_bfloat16 *pe = reinterpret_cast<const __nv_bfloat16 *>(d.p[1]);
  __nv_bfloat16 *cache = reinterpret_cast<__nv_bfloat16 *>(d.p[2]);
  for (int tok = 0; tok < nq; ++tok) {
    const int pos = seq_len - nq + tok;
    if (pos < 0) continue;
    const int pid = __ldcg(&P.meta.paged_kv_indices[kv0 + pos / page]);
    __nv_bfloat16 *dst = cache + ((size_t)pid * page + pos % page) * dk;
    for (int v = threadIdx.x; v < dk / 8; v += kConsumerThreads) {
      const uint4 val = v < dv / 8 ? __ldcg(reinterpret_cast<const uint4 *>(lat + (size_t)(q0 + tok) * ldc) + v)
                                   : __ldcg(reinterpret_cast<const uint4 *>(pe + (size_t)(q0 + tok) * ldp) + (v - dv / 8));
      reinterpret_cast<uint4 *>(dst)[v] = val;
    }
  }
}

__device__ __forceinline__ void ldmatrix_x4_trans(uint32_t (&r)[4], uint32_t smem_addr) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
               : "r"(smem_addr));
}

// TASK_MLA_DECODE: one query token x one 128-row split of its kv range x 16 heads, on mma.sync m16n8k16
// (replaces mla_mtp_decode_sm100 and its tensor-parallel variants).  Per 64-row tile: warp w computes the scores
// of kv rows [8w, 8w + 8) for all 16 heads (36 k steps over the 576 latent + rope dims), the row maxima and sums
// go through shared memory, the probabilities are written as a bf16 tile, and warp w accumulates output columns
// [64w, 64w + 64) of P.V with V read transposed from the same kv tile.  Output: O normalised by the split's own
// sum (bf16) and the split's log-sum-exp (fp32); TASK_MLA_REDUCE merges the splits.
static __device__ void run_mla_decode(const Ctx &c, const TaskDesc &d) {
  const KernelParams &P = c.P;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = lane >> 2, q = lane & 3;
  const int t = d.a[0], split = d.a[1], head0 = d.a[2], H = d.a[3], S = d.a[4], page = d.a[5], ldq = d.a[6];
  const float scale = __int_as_float(d.a[7]);
  if (t >= active_tokens(P)) return;
  // the request that owns token t, its length and the number of kv positions the token may see
  int kv0 = 0, lim = 0;
  size_t contiguous_base = 0;
  if (page > 0) {
    // every thread tests one request slot; the owner publishes its index
    int *owner = c.s.flags + 10;
    if (tid == 0) *owner = -1;
    consumer_sync();
    for (int r = tid; r < P.max_num_batched_requests; r += kConsumerThreads) {
      const int a0 = __ldcg(&P.meta.qo_indptr[r]), a1 = __ldcg(&P.meta.qo_indptr[r + 1]);
      if (t >= a0 && t < a1) *owner = r;
    }
    consumer_sync();
    const int r = *owner;
    if (r >= 0) {
      const int q0 = __ldcg(&P.meta.qo_indptr[r]), q1 = __ldcg(&P.meta.qo_indptr[r + 1]);
      kv0 = __ldcg(&P.meta.paged_kv_indptr[r]);
      const int npages = __ldcg(&P.meta.paged_kv_indptr[r + 1]) - kv0;
      const int seq_len = (npages - 1) * page + __ldcg(&P.meta.paged_kv_last_page_len[r]);
      lim = seq_len - (q1 - q0) + (t - q0) + 1;
    }
  } else {
    const int q_len = d.a[8], kv_len = d.a[9];
    const int r = t / q_len;
    contiguous_base = (size_t)r * kv_len;
    lim = kv_len - q_len + (t - r * q_len) + 1;
  }
  const int k_begin = split * kMlaSplit, k_end = min(k_begin + kMlaSplit, lim);
  __nv_bfloat16 *po = reinterpret_cast<__nv_bfloat16 *>(d.p[2]);
  float *plse = reinterpret_cast<float *>(d.p[3]);
  if (k_begin >= k_end) {   // nothing to see in this split: the merge skips it
    if (tid < 16) plse[((size_t)t * H + head0 + tid) * S + split] = -INFINITY;
    return;
  }
  uint8_t *Qs = c.s.xtile;
  uint8_t *KVs = Qs + 16 * kMlaRow;
  uint8_t *Ps = KVs + kMlaSub * kMlaRow;
  float *mx = reinterpret_cast<float *>(Ps + 16 * kMlaPRow);   // [8 warps][16 rows]
  float *sm = mx + 8 * 16;
  const __nv_bfloat16 *cache = reinterpret_cast<const __nv_bfloat16 *>(d.p[1]);
  {
    const __nv_bfloat16 *qg = reinterpret_cast<const __nv_bfloat16 *>(d.p[0]) + (size_t)t * ldq + (size_t)head0 * kMlaDk;
    for (int i = tid; i < 16 * (kMlaDk / 8); i += kConsumerThreads) {
      const int h = i / (kMlaDk / 8), v = i - h * (kMlaDk / 8);
      *reinterpret_cast<uint4 *>(Qs + (size_t)h * kMlaRow + (size_t)v * 16) =
          __ldcg(reinterpret_cast<const uint4 *>(qg + (size_t)h * kMlaDk) + v);
    }
  }
  float o[8][4];
#pragma unroll
  for (int i = 0; i < 8; ++i) o[i][0] = o[i][1] = o[i][2] = o[i][3] = 0.f;
  float m0 = -INFINITY, m1 = -INFINITY, l0 = 0.f, l1 = 0.f;   // running max / sum of rows g and g + 8
  const uint32_t q_addr = smem_u32(Qs) + (uint32_t)(lane & 15) * kMlaRow + (uint32_t)(lane >> 4) * 16u;
  const uint32_t k_addr = smem_u32(KVs) + (uint32_t)(warp * 8 + g) * kMlaRow + (uint32_t)q * 4u;
  const uint32_t p_addr = smem_u32(Ps) + (uint32_t)(lane & 15) * kMlaPRow + (uint32_t)(lane >> 4) * 16u;
  const uint32_t v_addr = smem_u32(KVs) + (uint32_t)(((lane >> 3) & 1) * 8 + (lane & 7)) * kMlaRow +
                          (uint32_t)(warp * 64 + (lane >> 4) * 8) * 2u;
  for (int sub = k_begin; sub < k_end; sub += kMlaSub) {
    const int nrows = min(kMlaSub, k_end - sub);
    consumer_sync();   // the previous tile (and the q tile of the previous task) is no longer read
    {
      // four threads per kv row: one page-table lookup, then 18 asynchronous 16-byte copies straight into
      // shared memory (no registers held, all in flight together); rows past the end are zero-filled
      const int r = tid >> 2, part = tid & 3;
      const uint32_t dst = smem_u32(KVs + (size_t)r * kMlaRow) + (uint32_t)part * 288u;
      if (r < nrows) {
        const int pos = sub + r;
        size_t row;
        if (page > 0) {
          const int pid = __ldcg(&P.meta.paged_kv_indices[kv0 + pos / page]);
          row = (size_t)pid * page + pos % page;
        } else {
          row = contiguous_base + pos;
        }
        const uint8_t *src = reinterpret_cast<const uint8_t *>(cache + row * kMlaDk) + part * 288;
#pragma unroll
        for (int j = 0; j < 18; ++j)
          asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst + j * 16u), "l"(src + j * 16) : "memory");
      } else {
#pragma unroll
        for (int j = 0; j < 18; ++j)
          asm volatile("st.shared.v4.b32 [%0], {%1, %1, %1, %1};" ::"r"(dst + j * 16u), "r"(0u) : "memory");
      }
      asm volatile("cp.async.commit_group;" ::: "memory");
      asm volatile("cp.async.wait_group 0;" ::: "memory");
    }
    consumer_sync();
    // scores of this warp's 8 kv rows
    float sacc[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll 4
    for (int ks = 0; ks < kMlaDk / 16; ++ks) {
      uint32_t a[4], b0, b1;
      ldmatrix_x4(a, q_addr + (uint32_t)ks * 32u);
      asm volatile("ld.shared.b32 %0, [%1];" : "=r"(b0) : "r"(k_addr + (uint32_t)ks * 32u));
      asm volatile("ld.shared.b32 %0, [%1];" : "=r"(b1) : "r"(k_addr + (uint32_t)ks * 32u + 16u));
      mma_bf16_16816(sacc, a, b0, b1);
    }
    const int j0 = warp * 8 + 2 * q;
    const bool v0 = j0 < nrows, v1 = j0 + 1 < nrows;
    sacc[0] = v0 ? sacc[0] * scale : -INFINITY;
    sacc[1] = v1 ? sacc[1] * scale : -INFINITY;
    sacc[2] = v0 ? sacc[2] * scale : -INFINITY;
    sacc[3] = v1 ? sacc[3] * scale : -INFINITY;
    float r0 = fmaxf(sacc[0], sacc[1]), r1 = fmaxf(sacc[2], sacc[3]);
    r0 = fmaxf(r0, __shfl_xor_sync(0xffffffffu, r0, 1));
    r0 = fmaxf(r0, __shfl_xor_sync(0xffffffffu, r0, 2));
    r1 = fmaxf(r1, __shfl_xor_sync(0xffffffffu, r1, 1));
    r1 = fmaxf(r1, __shfl_xor_sync(0xffffffffu, r1, 2));
    if (q == 0) { mx[warp * 16 + g] = r0; mx[warp * 16 + g + 8] = r1; }
    consumer_sync();
    float n0 = m0, n1 = m1;
#pragma unroll
    for (int w = 0; w < 8; ++w) { n0 = fmaxf(n0, mx[w * 16 + g]); n1 = fmaxf(n1, mx[w * 16 + g + 8]); }
    const float p00 = __expf(sacc[0] - n0), p01 = __expf(sacc[1] - n0);   // exp(-inf) = 0 for masked rows
    const float p10 = __expf(sacc[2] - n1), p11 = __expf(sacc[3] - n1);
    float s0 = p00 + p01, s1 = p10 + p11;
    s0 += __shfl_xor_sync(0xffffffffu, s0, 1);
    s0 += __shfl_xor_sync(0xffffffffu, s0, 2);
    s1 += __shfl_xor_sync(0xffffffffu, s1, 1);
    s1 += __shfl_xor_sync(0xffffffffu, s1, 2);
    if (q == 0) { sm[warp * 16 + g] = s0; sm[warp * 16 + g + 8] = s1; }
    {
      const __nv_bfloat162 w0 = __floats2bfloat162_rn(p00, p01), w1 = __floats2bfloat162_rn(p10, p11);
      *reinterpret_cast<__nv_bfloat162 *>(Ps + (size_t)g * kMlaPRow + (size_t)j0 * 2) = w0;
      *reinterpret_cast<__nv_bfloat162 *>(Ps + (size_t)(g + 8) * kMlaPRow + (size_t)j0 * 2) = w1;
    }
    consumer_sync();
    const float al0 = __expf(m0 - n0), al1 = __expf(m1 - n1);   // 0 on the first tile (m = -inf)
    float t0 = 0.f, t1 = 0.f;
#pragma unroll
    for (int w = 0; w < 8; ++w) { t0 += sm[w * 16 + g]; t1 += sm[w * 16 + g + 8]; }
    l0 = l0 * al0 + t0;
    l1 = l1 * al1 + t1;
    m0 = n0;
    m1 = n1;
#pragma unroll
    for (int i = 0; i < 8; ++i) { o[i][0] *= al0; o[i][1] *= al0; o[i][2] *= al1; o[i][3] *= al1; }
    // O[:, 64 warp ...] += P . V
#pragma unroll
    for (int ks = 0; ks < kMlaSub / 16; ++ks) {
      uint32_t a[4];
      ldmatrix_x4(a, p_addr + (uint32_t)ks * 32u);
#pragma unroll
      for (int np = 0; np < 4; ++np) {
        uint32_t b[4];
        ldmatrix_x4_trans(b, v_addr + (uint32_t)(ks * 16) * kMlaRow + (uint32_t)np * 32u);
        mma_bf16_16816(o[2 * np], a, b[0], b[1]);
        mma_bf16_16816(o[2 * np + 1], a, b[2], b[3]);
      }
    }
  }
  const float i0 = __fdividef(1.0f, l0), i1 = __fdividef(1.0f, l1);
  const size_t row0 = ((size_t)t * H + head0 + g) * S + split, row1 = ((size_t)t * H + head0 + g + 8) * S + split;
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    const int col = warp * 64 + i * 8 + 2 * q;
    *reinterpret_cast<__nv_bfloat162 *>(po + row0 * kMlaDv + col) = __floats2bfloat162_rn(o[i][0] * i0, o[i][1] * i0);
    *reinterpret_cast<__nv_bfloat162 *>(po + row1 * kMlaDv + col) = __floats2bfloat162_rn(o[i][2] * i1, o[i][3] * i1);
  }
  if (warp == 0 && q == 0) {
    plse[row0] = m0 + __logf(l0);
    plse[row1] = m1 + __logf(l1);
  }
}

// TASK_MLA_REDUCE: out[token, head] = sum_s w_s O_s with w_s = exp(lse_s - max) / sum: one warp per (token, head) row
// (mla_reduce_sm100.cuh:28-76 / mla_mtp_reduce).
static __device__ void run_mla_reduce(const Ctx &c, const TaskDesc &d) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int H = d.a[2], S = d.a[3], ldo = d.a[4];
  const int r1 = min(d.a[1], active_tokens(c.P) * H);
  const __nv_bfloat16 *po = reinterpret_cast<const __nv_bfloat16 *>(d.p[0]);
  const float *plse = reinterpret_cast<const float *>(d.p[1]);
  __nv_bfloat16 *out = reinterpret_cast<__nv_bfloat16 *>(d.p[2]);
  for (int row = d.a[0] + warp; row < r1; row += kConsumerThreads / 32) {
    // lane s keeps the weights of splits s and s + 32 (S <= 64); the O rows of four splits are fetched together
    const float ls0 = lane < S ? __ldcg(&plse[(size_t)row * S + lane]) : -INFINITY;
    const float ls1 = lane + 32 < S ? __ldcg(&plse[(size_t)row * S + lane + 32]) : -INFINITY;
    float mxv = fmaxf(ls0, ls1);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) mxv = fmaxf(mxv, __shfl_xor_sync(0xffffffffu, mxv, o));
    const float w0 = ls0 == -INFINITY ? 0.f : __expf(ls0 - mxv), w1 = ls1 == -INFINITY ? 0.f : __expf(ls1 - mxv);
    float tot = w0 + w1;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) tot += __shfl_xor_sync(0xffffffffu, tot, o);
    float acc[16];
#pragma unroll
    for (int i = 0; i < 16; ++i) acc[i] = 0.f;
    for (int s0 = 0; s0 < S; s0 += 4) {
      float w[4];
      uint4 x0[4], x1[4];
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        const int s = s0 + u;
        w[u] = __shfl_sync(0xffffffffu, s < 32 ? w0 : w1, s & 31);
        if (s >= S) w[u] = 0.f;
        x0[u] = x1[u] = make_uint4(0, 0, 0, 0);
        if (w[u] != 0.f) {
          const uint4 *src = reinterpret_cast<const uint4 *>(po + ((size_t)row * S + s) * kMlaDv + lane * 16);
          x0[u] = __ldcg(src);
          x1[u] = __ldcg(src + 1);
        }
      }
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        const uint32_t xs[8] = {x0[u].x, x0[u].y, x0[u].z, x0[u].w, x1[u].x, x1[u].y, x1[u].z, x1[u].w};
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          acc[2 * i] += w[u] * __uint_as_float(xs[i] << 16);
          acc[2 * i + 1] += w[u] * __uint_as_float(xs[i] & 0xffff0000u);
        }
      }
    }
    const float inv = tot > 0.f ? __fdividef(1.0f, tot) : 0.f;
    const int tok = row / H, h = row - tok * H;
    __nv_bfloat16 *dst = out + (size_t)tok * ldo + (size_t)h * kMlaDv + lane * 16;
#pragma unroll
    for (int i = 0; i < 8; ++i)
      *reinterpret_cast<__nv_bfloat162 *>(dst + 2 * i) = __floats2bfloat162_rn(acc[2 * i] * inv, acc[2 * i + 1] * inv);
  }
}

// ---------------------------------------------------------------------------
// TASK_ATTENTION: paged split-KV GQA decode attention with fused QK-norm, RoPE, KV append
// ---------------------------------------------------------------------------
// One task = (request slot, kv head, kv chunk).  Work that does not depend on this layer's qkv
// projection -- the request's page table and the K/V rows already in the cache -- is fetched into
// registers BEFORE the task waits for its dependency, so that after the wait only the new token's
// q/k/v have to be loaded.  Partial results of the chunks are merged by the last chunk to finish.
struct ReqView {
  int q0, nq, kv0, seq_len;
};

constexpr int kAttnPre = 4;   // kv rows per half-warp fetched ahead of the dependency (64 rows per CTA)

struct AttnPre {
  ReqView rv;
  int start, end, new_start, n_active;
  uint4 k[kAttnPre], v[kAttnPre];
  uint2 cs0, sn0;   // rotary cos / sin of the first new position (this lane's dims)
};

__device__ __forceinline__ ReqView request_view(const KernelParams &P, const TaskDesc &d) {
  ReqView r;
  const int slot = d.a[A_SLOT];
  if (d.a[A_FLAGS] & 4) {   // contiguous cache: one token per slot, length = step + 1
    r.q0 = slot;
    r.nq = (slot < active_tokens(P)) ? 1 : 0;
    r.kv0 = 0;
    r.seq_len = P.meta.step ? __ldcg(&P.meta.step[slot]) + 1 : 1;
    return r;
  }
  r.q0 = __ldcg(&P.meta.qo_indptr[slot]);
  r.nq = __ldcg(&P.meta.qo_indptr[slot + 1]) - r.q0;
  r.kv0 = __ldcg(&P.meta.paged_kv_indptr[slot]);
  const int npages = __ldcg(&P.meta.paged_kv_indptr[slot + 1]) - r.kv0;
  r.seq_len = (npages - 1) * d.a[A_PAGE] + __ldcg(&P.meta.paged_kv_last_page_len[slot]);
  return r;
}

// element offset of (position, kv head) inside a [pages, page, Hkv, 128] cache
__device__ __forceinline__ size_t kv_offset(const KernelParams &P, const TaskDesc &d, const ReqView &rv, int pos) {
  const int page = d.a[A_PAGE];
  const int hkv = d.a[A_HKV];
  if (d.a[A_FLAGS] & 4)
    return (((size_t)d.a[A_SLOT] * d.a[A_CSEQ] + pos) * hkv + d.a[A_HEAD]) * 128;
  const int pidx = pos / page;
  const int pid = __ldcg(&P.meta.paged_kv_indices[rv.kv0 + pidx]);
  return (((size_t)pid * page + (pos - pidx * page)) * hkv + d.a[A_HEAD]) * 128;
}

// Issued by the streaming warp when it walks past an attention task, i.e. while the compute warps are
// still a few chunks away from it: pulls the cached K/V rows of the task's chunk into L2.  The batch
// description may still be the previous iteration's when this runs early in a launch; every index read
// here stays inside its buffer for any mix of old and new values, and a stale prefetch is harmless.
//
// It also leaves the request's description and the page ids of the chunk's first 64 positions in shared memory
// (`attention stash`, the unused tail of the full-barrier array) for the compute warps, which would otherwise pay
// two dependent L2 round trips for them right before their dependency wait.  The stash is published only when the
// batching event of this iteration had already fired (acquire), i.e. when what was read is final; it carries the task
// index, is written index-last and read index-first-and-last, so a reader either gets a consistent record of its own
// task or falls back to its own loads.
__device__ __forceinline__ volatile int *attention_stash(const Ctx &c) {
  return reinterpret_cast<volatile int *>(&c.s.full[8]);
}

static __device__ void prefetch_attention_kv_l2(const Ctx &c, const TaskDesc *d, int lane, int task) {
  const KernelParams &P = c.P;
  if ((d->a[A_FLAGS] & 4) || P.meta.qo_indptr == nullptr) return;
  const bool final_meta = P.meta_static || ld_acquire_gpu(&P.counters[0]) >= c.iteration;
  const int slot = d->a[A_SLOT];
  const int q0 = __ldcg(&P.meta.qo_indptr[slot]);
  const int nq = __ldcg(&P.meta.qo_indptr[slot + 1]) - q0;
  const int kv0 = __ldcg(&P.meta.paged_kv_indptr[slot]);
  const int npages = __ldcg(&P.meta.paged_kv_indptr[slot + 1]) - kv0;
  const int page = d->a[A_PAGE], hkv = d->a[A_HKV];
  if (nq <= 0 || npages <= 0 || kv0 < 0 || kv0 + npages > P.max_num_pages) return;
  const int seq_len = (npages - 1) * page + min(max(__ldcg(&P.meta.paged_kv_last_page_len[slot]), 1), page);
  const int NC = d->a[A_NCHUNK];
  int L = (seq_len + NC - 1) / NC;
  L = (L + 15) & ~15;
  const int start = d->a[A_CHUNK] * L;
  const int old_end = min(min(seq_len, start + L), seq_len - nq);
  const char *kc = reinterpret_cast<const char *>(d->p[1]);
  const char *vc = reinterpret_cast<const char *>(d->p[2]);
  if (final_meta && page >= 64 && start < seq_len) {
    const int pb = start / page;
    const int p0 = __ldcg(&P.meta.paged_kv_indices[kv0 + pb]);
    const int p1 = (pb + 1 < npages) ? __ldcg(&P.meta.paged_kv_indices[kv0 + pb + 1]) : p0;
    if (lane == 0) {
      volatile int *st = attention_stash(c);
      st[0] = -1;
      __threadfence_block();
      st[1] = q0; st[2] = nq; st[3] = kv0; st[4] = (npages - 1) * page + __ldcg(&P.meta.paged_kv_last_page_len[slot]);
      st[5] = pb; st[6] = p0; st[7] = p1;
      __threadfence_block();
      st[0] = task;
    }
  }
  for (int pos = start + lane; pos < old_end; pos += 32) {
    const int pidx = pos / page;
    const int pid = min(max(__ldcg(&P.meta.paged_kv_indices[kv0 + pidx]), 0), P.max_num_pages - 1);
    const size_t off = ((((size_t)pid * page + (pos - pidx * page)) * hkv + d->a[A_HEAD]) * 128) * 2;
    asm volatile("prefetch.global.L2 [%0];" ::"l"(kc + off));
    asm volatile("prefetch.global.L2 [%0];" ::"l"(kc + off + 128));
    asm volatile("prefetch.global.L2 [%0];" ::"l"(vc + off));
    asm volatile("prefetch.global.L2 [%0];" ::"l"(vc + off + 128));
  }
}

__device__ __forceinline__ void load_rope(const __nv_bfloat16 *cosT, const __nv_bfloat16 *sinT, int pos, int rows,
                                          int lane, uint2 &cs, uint2 &sn);

// Runs before the dependency wait (the batch description is already final).
__device__ __forceinline__ void attention_prefetch(const Ctx &c, const TaskDesc &d, AttnPre &pre, int task) {
  const KernelParams &P = c.P;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  // the streaming warp may have left this task's request description and first page ids in shared memory
  const volatile int *st = attention_stash(c);
  bool hit = st[0] == task;
  int pb = 0, p0 = 0, p1 = 0;
  if (hit) {
    pre.rv.q0 = st[1]; pre.rv.nq = st[2]; pre.rv.kv0 = st[3]; pre.rv.seq_len = st[4];
    pb = st[5]; p0 = st[6]; p1 = st[7];
    __threadfence_block();
    hit = st[0] == task;
  }
  if (!hit) pre.rv = request_view(P, d);
  const int NC = d.a[A_NCHUNK];
  int L = (pre.rv.seq_len + NC - 1) / NC;
  L = (L + 15) & ~15;
  pre.n_active = pre.rv.nq > 0 ? (pre.rv.seq_len + L - 1) / L : 0;
  pre.start = d.a[A_CHUNK] * L;
  pre.end = min(pre.rv.seq_len, pre.start + L);
  pre.new_start = pre.rv.seq_len - pre.rv.nq;
  pre.cs0 = pre.sn0 = make_uint2(0, 0);
  if (pre.rv.nq <= 0) return;
  load_rope((d.a[A_FLAGS] & 2) ? reinterpret_cast<const __nv_bfloat16 *>(d.p[5]) : nullptr,
            reinterpret_cast<const __nv_bfloat16 *>(d.p[6]), pre.new_start, d.a[A_ROPE_ROWS], lane, pre.cs0, pre.sn0);
  const __nv_bfloat16 *kc = reinterpret_cast<const __nv_bfloat16 *>(d.p[1]);
  const __nv_bfloat16 *vc = reinterpret_cast<const __nv_bfloat16 *>(d.p[2]);
  const int hw = lane >> 4, hl = lane & 15;
  const int old_end = min(pre.end, pre.new_start);
#pragma unroll
  for (int i = 0; i < kAttnPre; ++i) {
    const int pos = pre.start + warp * 2 + hw + 16 * i;
    // Rows outside the range get defined zeros: every row is read later (masked), and leaving them
    // indeterminate would let the compiler make these loads unconditional, i.e. read out of range.
    pre.k[i] = make_uint4(0, 0, 0, 0);
    pre.v[i] = make_uint4(0, 0, 0, 0);
    if (pos < old_end) {
      size_t off;
      if (hit) {   // positions start .. start + 63 lie in the page of `start` or the next one (pages hold >= 64 rows)
        const int page = d.a[A_PAGE], pidx = pos / page;
        off = (((size_t)(pidx == pb ? p0 : p1) * page + (pos - pidx * page)) * d.a[A_HKV] + d.a[A_HEAD]) * 128 + hl * 8;
      } else {
        off = kv_offset(P, d, pre.rv, pos) + hl * 8;
      }
      pre.k[i] = __ldcs(reinterpret_cast<const uint4 *>(kc + off));
      pre.v[i] = __ldcs(reinterpret_cast<const uint4 *>(vc + off));
    }
  }
}

// One warp: RMS-normalise (optional) and rotate (optional) a 128-wide head vector.
// Lane l holds elements 4l..4l+3.  Norm result is rounded to bf16 before the rotation,
// as include/mirage/persistent_kernel/tasks/blackwell/norm_sm100.cuh:96-126 does.
__device__ __forceinline__ void norm_rope_head(float (&x)[4], const __nv_bfloat16 *norm_w, float eps, bool rope,
                                               uint2 cs, uint2 sn, int lane) {
  if (norm_w) {
    float ss = x[0] * x[0] + x[1] * x[1] + x[2] * x[2] + x[3] * x[3];
    ss = warp_sum(ss);
    const float inv = rsqrtf(ss * (1.0f / 128.0f) + eps);
    const uint2 nw = __ldg(reinterpret_cast<const uint2 *>(norm_w + lane * 4));
    const float w[4] = {bf16_lo(nw.x), bf16_hi(nw.x), bf16_lo(nw.y), bf16_hi(nw.y)};
#pragma unroll
    for (int i = 0; i < 4; ++i) x[i] = round_bf16(x[i] * inv * w[i]);
  }
  if (rope) {
    const float cf[4] = {bf16_lo(cs.x), bf16_hi(cs.x), bf16_lo(cs.y), bf16_hi(cs.y)};
    const float sf[4] = {bf16_lo(sn.x), bf16_hi(sn.x), bf16_lo(sn.y), bf16_hi(sn.y)};
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const float other = __shfl_xor_sync(0xffffffffu, x[i], 16);   // element d +/- 64
      const float rot = (lane < 16) ? -other : other;
      x[i] = round_bf16(x[i] * cf[i] + rot * sf[i]);
    }
  }
}

// cos / sin of one position for this lane's four dims (zeros when the layer has no rotary embedding)
__device__ __forceinline__ void load_rope(const __nv_bfloat16 *cosT, const __nv_bfloat16 *sinT, int pos, int rows,
                                          int lane, uint2 &cs, uint2 &sn) {
  cs = sn = make_uint2(0, 0);
  if (cosT) {
    const size_t o = (size_t)min(pos, rows - 1) * 128 + lane * 4;
    cs = __ldg(reinterpret_cast<const uint2 *>(cosT + o));
    sn = __ldg(reinterpret_cast<const uint2 *>(sinT + o));
  }
}

template <int G>
struct AttnState {
  float m[G], l[G], o[G][8];
};

// one kv row (8 of its 128 dims per lane) against the G query heads of this kv head
template <int G>
__device__ __forceinline__ void attn_row(AttnState<G> &s, const float (&q)[G][8], const uint4 &kr, const uint4 &vr,
                                         unsigned hmask) {
  const float kf[8] = {bf16_lo(kr.x), bf16_hi(kr.x), bf16_lo(kr.y), bf16_hi(kr.y),
                       bf16_lo(kr.z), bf16_hi(kr.z), bf16_lo(kr.w), bf16_hi(kr.w)};
  const float vf[8] = {bf16_lo(vr.x), bf16_hi(vr.x), bf16_lo(vr.y), bf16_hi(vr.y),
                       bf16_lo(vr.z), bf16_hi(vr.z), bf16_lo(vr.w), bf16_hi(vr.w)};
#pragma unroll
  for (int g = 0; g < G; ++g) {
    float sc = 0.f;
#pragma unroll
    for (int i = 0; i < 8; ++i) sc = fmaf(q[g][i], kf[i], sc);
    sc += __shfl_xor_sync(hmask, sc, 8);
    sc += __shfl_xor_sync(hmask, sc, 4);
    sc += __shfl_xor_sync(hmask, sc, 2);
    sc += __shfl_xor_sync(hmask, sc, 1);
    const float mn = fmaxf(s.m[g], sc);
    const float corr = exp2f(s.m[g] - mn);
    const float p = exp2f(sc - mn);
    s.m[g] = mn;
    s.l[g] = s.l[g] * corr + p;
#pragma unroll
    for (int i = 0; i < 8; ++i) s.o[g][i] = fmaf(p, vf[i], s.o[g][i] * corr);
  }
}

// Up to four kv rows at once: the dot products and their shuffle reductions are independent chains, and the
// running softmax state is updated once for the whole batch.
template <int G>
__device__ __forceinline__ void attn_rows4(AttnState<G> &s, const float (&q)[G][8], const uint4 (&kr)[kAttnPre],
                                           const uint4 (&vr)[kAttnPre], int nrows, unsigned hmask) {
  float sc[kAttnPre][G];
#pragma unroll
  for (int i = 0; i < kAttnPre; ++i) {
    const float kf[8] = {bf16_lo(kr[i].x), bf16_hi(kr[i].x), bf16_lo(kr[i].y), bf16_hi(kr[i].y),
                         bf16_lo(kr[i].z), bf16_hi(kr[i].z), bf16_lo(kr[i].w), bf16_hi(kr[i].w)};
#pragma unroll
    for (int g = 0; g < G; ++g) {
      float a = 0.f;
#pragma unroll
      for (int e = 0; e < 8; ++e) a = fmaf(q[g][e], kf[e], a);
      sc[i][g] = a;
    }
  }
#pragma unroll
  for (int o = 8; o > 0; o >>= 1)
#pragma unroll
    for (int i = 0; i < kAttnPre; ++i)
#pragma unroll
      for (int g = 0; g < G; ++g) sc[i][g] += __shfl_xor_sync(hmask, sc[i][g], o);
#pragma unroll
  for (int g = 0; g < G; ++g) {
    float mn = s.m[g];
#pragma unroll
    for (int i = 0; i < kAttnPre; ++i)
      if (i < nrows) mn = fmaxf(mn, sc[i][g]);
    const float corr = exp2f(s.m[g] - mn);
    float p[kAttnPre];
    float psum = 0.f;
#pragma unroll
    for (int i = 0; i < kAttnPre; ++i) {
      p[i] = (i < nrows) ? exp2f(sc[i][g] - mn) : 0.f;
      psum += p[i];
    }
    s.m[g] = mn;
    s.l[g] = s.l[g] * corr + psum;
#pragma unroll
    for (int e = 0; e < 8; ++e) s.o[g][e] *= corr;
#pragma unroll
    for (int i = 0; i < kAttnPre; ++i) {
      const float vf[8] = {bf16_lo(vr[i].x), bf16_hi(vr[i].x), bf16_lo(vr[i].y), bf16_hi(vr[i].y),
                           bf16_lo(vr[i].z), bf16_hi(vr[i].z), bf16_lo(vr[i].w), bf16_hi(vr[i].w)};
#pragma unroll
      for (int e = 0; e < 8; ++e) s.o[g][e] = fmaf(p[i], vf[e], s.o[g][e]);
    }
  }
}

template <int GT>
__device__ __forceinline__ void attention_body(const Ctx &c, const TaskDesc &d, const AttnPre &pre, const int G,
                                               int task) {
  const KernelParams &P = c.P;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const ReqView rv = pre.rv;
  if (rv.nq <= 0) return;
  const int NC = d.a[A_NCHUNK], chunk = d.a[A_CHUNK], head = d.a[A_HEAD];
  const int hq = d.a[A_HQ];
  const int flags = d.a[A_FLAGS];
  const float eps = __int_as_float(d.a[A_EPS]);
  const __nv_bfloat16 *qkv = reinterpret_cast<const __nv_bfloat16 *>(d.p[0]);
  __nv_bfloat16 *kc = reinterpret_cast<__nv_bfloat16 *>(d.p[1]);
  __nv_bfloat16 *vc = reinterpret_cast<__nv_bfloat16 *>(d.p[2]);
  const __nv_bfloat16 *qn = (flags & 1) ? reinterpret_cast<const __nv_bfloat16 *>(d.p[3]) : nullptr;
  const __nv_bfloat16 *kn = (flags & 1) ? reinterpret_cast<const __nv_bfloat16 *>(d.p[4]) : nullptr;
  const __nv_bfloat16 *cosT = (flags & 2) ? reinterpret_cast<const __nv_bfloat16 *>(d.p[5]) : nullptr;
  const __nv_bfloat16 *sinT = (flags & 2) ? reinterpret_cast<const __nv_bfloat16 *>(d.p[6]) : nullptr;
  __nv_bfloat16 *out = reinterpret_cast<__nv_bfloat16 *>(d.p[7]);
  const int ldq = d.a[A_LDQKV], ldo = d.a[A_LDO];
  const int rope_rows = d.a[A_ROPE_ROWS];
  const int start = pre.start, end = pre.end, new_start = pre.new_start, n_active = pre.n_active;
  const size_t head_base = (size_t)head * (G + 2) * 128;

  const bool aprof = P.profiler != nullptr && (uint64_t)(task + 1) * 8 <= P.profiler_entries;
  float *q_s = reinterpret_cast<float *>(c.s.xtile);            // [G][128], pre-scaled
  float *w_ml = q_s + G * 128;                                    // [8 warps][G][2]
  float *w_o = w_ml + 8 * G * 2;                                  // [8 warps][G][128]
  uint2 *new_kv = reinterpret_cast<uint2 *>(w_o + 8 * G * 128);   // [nq][k 32 lanes | v 32 lanes] (4 bf16 per lane)

  // ---- append the new keys / values that fall into this chunk (cache + shared-memory copy) ----
  for (int pos = max(start, new_start) + warp; pos < end; pos += 8) {
    const int tok = rv.q0 + (pos - new_start);
    const __nv_bfloat16 *kp = qkv + (size_t)tok * ldq + head_base + (size_t)G * 128 + lane * 4;
    const uint2 kr = __ldcg(reinterpret_cast<const uint2 *>(kp));
    const uint2 vr = __ldcg(reinterpret_cast<const uint2 *>(kp + 128));
    float x[4] = {bf16_lo(kr.x), bf16_hi(kr.x), bf16_lo(kr.y), bf16_hi(kr.y)};
    uint2 cs = pre.cs0, sn = pre.sn0;
    if (pos != new_start) load_rope(cosT, sinT, pos, rope_rows, lane, cs, sn);
    norm_rope_head(x, kn, eps, cosT != nullptr, cs, sn, lane);
    const uint2 kw = make_uint2(pack_bf16(x[0], x[1]), pack_bf16(x[2], x[3]));
    const size_t off = kv_offset(P, d, rv, pos) + lane * 4;
    *reinterpret_cast<uint2 *>(kc + off) = kw;
    *reinterpret_cast<uint2 *>(vc + off) = vr;
    new_kv[(size_t)(pos - new_start) * 64 + lane] = kw;
    new_kv[(size_t)(pos - new_start) * 64 + 32 + lane] = vr;
  }

  const float qscale = 0.08838834764831845f * 1.4426950408889634f;   // 1/sqrt(128) * log2(e)
  const int hw = lane >> 4;          // half-warp
  const int hl = lane & 15;          // lane within the half-warp: dims hl*8 .. hl*8+7
  const unsigned hmask = hw ? 0xffff0000u : 0x0000ffffu;
  const int old_end = min(end, new_start);

  for (int t = 0; t < rv.nq; ++t) {
    const int pq = new_start + t;
    const int tok = rv.q0 + t;
    const int lim = min(end, pq + 1);
    if (warp < G) {
      const __nv_bfloat16 *qp = qkv + (size_t)tok * ldq + head_base + (size_t)warp * 128 + lane * 4;
      const uint2 qr = __ldcg(reinterpret_cast<const uint2 *>(qp));
      float x[4] = {bf16_lo(qr.x), bf16_hi(qr.x), bf16_lo(qr.y), bf16_hi(qr.y)};
      uint2 cs = pre.cs0, sn = pre.sn0;
      if (t != 0) load_rope(cosT, sinT, pq, rope_rows, lane, cs, sn);
      norm_rope_head(x, qn, eps, cosT != nullptr, cs, sn, lane);
      *reinterpret_cast<float4 *>(&q_s[warp * 128 + lane * 4]) =
          make_float4(x[0] * qscale, x[1] * qscale, x[2] * qscale, x[3] * qscale);
    }
    consumer_sync();   // q_s and new_kv are ready
    if (tid == 0 && aprof && t == 0) P.profiler[(size_t)task * 8 + 4] = globaltimer_ns();
    const int first = start + warp * 2 + hw;
    for (int gb = 0; gb < G; gb += GT) {   // GT query heads at a time keeps the register footprint bounded
      float q[GT][8];
#pragma unroll
      for (int g = 0; g < GT; ++g) {
        const float4 a = *reinterpret_cast<const float4 *>(&q_s[(gb + g) * 128 + hl * 8]);
        const float4 b = *reinterpret_cast<const float4 *>(&q_s[(gb + g) * 128 + hl * 8 + 4]);
        q[g][0] = a.x; q[g][1] = a.y; q[g][2] = a.z; q[g][3] = a.w;
        q[g][4] = b.x; q[g][5] = b.y; q[g][6] = b.z; q[g][7] = b.w;
      }
      AttnState<GT> s;
#pragma unroll
      for (int g = 0; g < GT; ++g) {
        s.m[g] = -INFINITY;
        s.l[g] = 0.f;
#pragma unroll
        for (int i = 0; i < 8; ++i) s.o[g][i] = 0.f;
      }
      // rows fetched ahead of the dependency (positions first, first + 16, ...: a prefix of them is valid)
      {
        const int bound = min(old_end, lim);
        const int nrows = first < bound ? min((bound - first + 15) >> 4, kAttnPre) : 0;
        if (nrows > 0) attn_rows4<GT>(s, q, pre.k, pre.v, nrows, hmask);   // uniform per half-warp
      }
      if (tid == 0 && aprof && t == 0 && gb == 0) P.profiler[(size_t)task * 8 + 5] = globaltimer_ns();
      // remaining old rows of a long chunk
      for (int pos = first + 16 * kAttnPre; pos < min(old_end, lim); pos += 16) {
        const size_t off = kv_offset(P, d, rv, pos) + hl * 8;
        const uint4 kr = __ldcs(reinterpret_cast<const uint4 *>(kc + off));
        const uint4 vr = __ldcs(reinterpret_cast<const uint4 *>(vc + off));
        attn_row<GT>(s, q, kr, vr, hmask);
      }
      // rows appended by this task: read back from shared memory
      {
        int pos = first;
        if (pos < new_start) pos += ((new_start - pos + 15) / 16) * 16;
        for (; pos < lim; pos += 16) {
          const uint4 kr = *reinterpret_cast<const uint4 *>(&new_kv[(size_t)(pos - new_start) * 64 + hl * 2]);
          const uint4 vr = *reinterpret_cast<const uint4 *>(&new_kv[(size_t)(pos - new_start) * 64 + 32 + hl * 2]);
          attn_row<GT>(s, q, kr, vr, hmask);
        }
      }
      if (tid == 0 && aprof && t == 0 && gb == 0) P.profiler[(size_t)task * 8 + 6] = globaltimer_ns();
      __syncwarp();
      // fold the two half-warps together
#pragma unroll
      for (int g = 0; g < GT; ++g) {
        const float m2 = __shfl_xor_sync(0xffffffffu, s.m[g], 16);
        const float l2 = __shfl_xor_sync(0xffffffffu, s.l[g], 16);
        const float mn = fmaxf(s.m[g], m2);
        const float c1 = (s.m[g] == -INFINITY) ? 0.f : exp2f(s.m[g] - mn);
        const float c2 = (m2 == -INFINITY) ? 0.f : exp2f(m2 - mn);
        s.l[g] = s.l[g] * c1 + l2 * c2;
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          const float o2 = __shfl_xor_sync(0xffffffffu, s.o[g][i], 16);
          s.o[g][i] = s.o[g][i] * c1 + o2 * c2;
        }
        s.m[g] = mn;
        if (hw == 0) {
          float4 *wo = reinterpret_cast<float4 *>(&w_o[((size_t)warp * G + gb + g) * 128 + hl * 8]);
          wo[0] = make_float4(s.o[g][0], s.o[g][1], s.o[g][2], s.o[g][3]);
          wo[1] = make_float4(s.o[g][4], s.o[g][5], s.o[g][6], s.o[g][7]);
          if (hl == 0) {
            w_ml[(warp * G + gb + g) * 2 + 0] = s.m[g];
            w_ml[(warp * G + gb + g) * 2 + 1] = s.l[g];
          }
        }
      }
    }
    if (tid == 0 && aprof && t == 0) P.profiler[(size_t)task * 8 + 7] = globaltimer_ns();
    consumer_sync();
    // combine the 8 warps; thread -> (g, dim) pairs
    for (int idx = tid; idx < G * 128; idx += kConsumerThreads) {
      const int g = idx >> 7, dd = idx & 127;
      float M = -INFINITY;
#pragma unroll
      for (int w = 0; w < 8; ++w) M = fmaxf(M, w_ml[(w * G + g) * 2]);
      float Ls = 0.f, O = 0.f;
#pragma unroll
      for (int w = 0; w < 8; ++w) {
        const float mw = w_ml[(w * G + g) * 2];
        const float sc = (mw == -INFINITY) ? 0.f : exp2f(mw - M);
        Ls += w_ml[(w * G + g) * 2 + 1] * sc;
        O += w_o[((size_t)w * G + g) * 128 + dd] * sc;
      }
      const int hq_idx = head * G + g;
      if (NC == 1) {
        out[(size_t)tok * ldo + (size_t)hq_idx * 128 + dd] = __float2bfloat16_rn(Ls > 0.f ? O / Ls : 0.f);
      } else {
        const size_t base = ((size_t)tok * hq + hq_idx) * NC + chunk;
        __stcg(&P.attn_scratch[base * 130 + 2 + dd], O);
        if (dd == 0) {
          __stcg(&P.attn_scratch[base * 130 + 0], M);
          __stcg(&P.attn_scratch[base * 130 + 1], Ls);
        }
      }
    }
    if (t + 1 < rv.nq) consumer_sync();   // q_s / w_o are rewritten for the next query token
  }
  if (NC == 1) return;
  // ---- split-KV merge by the last chunk task to arrive ---------------------------
  consumer_sync();
  if (tid == 0) {
    unsigned int old;
    asm volatile("atom.acq_rel.gpu.global.add.u32 %0, [%1], 1;"
                 : "=r"(old)
                 : "l"(&P.attn_tickets[d.a[A_TICKET] + d.a[A_SLOT] * d.a[A_HKV] + head])
                 : "memory");
    c.s.flags[1] = ((old + 1u) % (unsigned)NC == 0u) ? 1 : 0;
  }
  consumer_sync();
  if (c.s.flags[1] == 0) return;
  // Merge: one warp per 32 consecutive output dims of a (token, head).  Lane c fetches chunk c's (max, sum)
  // while every lane fetches its dim of all chunks; all loads are in flight together (a single round trip to
  // L2), then the weights are formed with shuffles.  NC <= 32.
  for (int item = warp; item < rv.nq * G * 4; item += 8) {
    const int row = item >> 2, dd = ((item & 3) << 5) + lane;
    const int t = row / G, g = row - t * G;
    const int tok = rv.q0 + t;
    const int hq_idx = head * G + g;
    const size_t base = ((size_t)tok * hq + hq_idx) * NC;
    const bool v = lane < n_active;
    const float m = v ? __ldcg(&P.attn_scratch[(base + lane) * 130]) : -INFINITY;
    const float l = v ? __ldcg(&P.attn_scratch[(base + lane) * 130 + 1]) : 0.f;
    float ow[16], ow2[16];
#pragma unroll
    for (int u = 0; u < 16; ++u)
      ow[u] = (u < n_active) ? __ldcg(&P.attn_scratch[(base + u) * 130 + 2 + dd]) : 0.f;
    if (n_active > 16) {
#pragma unroll
      for (int u = 0; u < 16; ++u)
        ow2[u] = (16 + u < n_active) ? __ldcg(&P.attn_scratch[(base + 16 + u) * 130 + 2 + dd]) : 0.f;
    }
    float M = m;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) M = fmaxf(M, __shfl_xor_sync(0xffffffffu, M, o));
    const float w = (m == -INFINITY) ? 0.f : exp2f(m - M);
    const float Ls = warp_sum(l * w);
    float O = 0.f;
#pragma unroll
    for (int u = 0; u < 16; ++u) O = fmaf(ow[u], __shfl_sync(0xffffffffu, w, u), O);
    if (n_active > 16) {
#pragma unroll
      for (int u = 0; u < 16; ++u) O = fmaf(ow2[u], __shfl_sync(0xffffffffu, w, 16 + u), O);
    }
    out[(size_t)tok * ldo + (size_t)hq_idx * 128 + dd] = __float2bfloat16_rn(Ls > 0.f ? O / Ls : 0.f);
  }
}

__device__ __forceinline__ void run_attention(const Ctx &c, const TaskDesc &d, const AttnPre &pre, int task) {
  const int G = d.a[A_HQ] / d.a[A_HKV];
  switch (G) {
    case 1: attention_body<1>(c, d, pre, 1, task); break;
    case 2: attention_body<2>(c, d, pre, 2, task); break;
    default: attention_body<4>(c, d, pre, G, task); break;   // 4 or 8 heads per kv head, four at a time
  }
}

// ---------------------------------------------------------------------------
// TASK_ATTENTION, general instantiation (many tokens): every warp takes an equal share of all key steps
// ---------------------------------------------------------------------------
// The unit of work is a step: 8 positions of one (request, kv head) for one tile of 16 query rows (16 / G tokens x the G heads of the
// group; a decoding request has one tile).  Eight kv heads go together, one per warp of a worker (with fewer, the warps share out
// ranges), so that a cached position is read whole, 2 KB at a time: with a range per (head, warp) the same bytes came at 1.3 TB/s.  The
// steps of the whole layer, in the order request, head group, tile, position, are cut into equal ranges by arithmetic on the batch
// description alone: 16 requests of 512 to 4000 positions keep all workers busy to the end, where a task per (request, head, chunk)
// left the last ones 38 us behind.  A warp walks its range without any block barrier: its
// own ring of stages, filled by two tensor-map copies a step, runs on across the borders of heads and requests, and starts before the task waits for this layer's
// qkv projection, because rows already in the cache do not depend on it.  Rows that this launch appends are normed and rotated by
// the warp that meets them (the first tile's warp writes them to the cache), so no warp waits for another's append.
// A tile that lies in one range is written out at once; otherwise every range leaves its part in a scratch record and the last of them
// to arrive (a ticket per tile) merges.  Per step: S = Q K^T on mma.sync m16n8k16, online softmax (fp32, base 2), P rounded to bf16 as the
// reference does (tasks/blackwell/attention_sm100.cuh:558; in graphs of few tokens the sum of two), O += P V on m16n8k8 with V through ldmatrix.trans.
// Where that leaves a range fewer than kAfMinSteps steps, the latency of a few steps in a row and of merging many parts through L2 is what
// counts.  Then a worker takes a tile of one kv head, or one of the parts of a tile whose steps exceed a worker's average (af_parts), its eight
// warps share the positions and combine in shared memory.
// Measured, us per layer, before (one task per request, head and chunk) and now: 16 requests of 512 to 4000 positions 76 -> 56,
// 64 of 512 to 1536 109 -> 75 (3.6 TB/s), 32 + 32 prompt tokens behind 1000 and 343 positions 235 -> 39, 24 requests of 60 positions 14.8 -> 11.8, 41 of
// 94 to 214 positions with 4 kv heads 14.4 -> 12.4.  The two ways are instantiations of their own and rows are prepared two at a time:
// what one body of both spilled cost a tenth.  What bounds it now is the latency of the steps of a warp (two in flight) and, for short contexts, the fixed part.
constexpr int kAfRows = 8;                       // positions of a step
constexpr int kAfTile = kAfRows * 256;           // K or V rows of a step: two blocks of 64 columns in the 128-byte swizzle of the tensor map
constexpr int kAfStage = 2 * kAfTile;            // K rows, then V rows; also the 16 query rows of a tile
constexpr uint32_t kAfWild = 1u << 31;           // bit of a warp's stage parities: values that are not finite have been set aside (af_put_back)
constexpr int kAfMinSteps = 16;                  // ranges of fewer steps: the warps of a worker share a tile instead (see below)
constexpr int kAfRecord = 16 * 132;              // floats of a record: 16 rows x {max, sum, -, -, 128 outputs}

__device__ __forceinline__ uint32_t af_piece(int row, int piece) { return (uint32_t)((piece >> 3) * 1024 + row * 128 + (((piece & 7) ^ row) << 4)); }
__device__ __forceinline__ uint32_t af_qpiece(int row, int piece) { return (uint32_t)((piece >> 3) * 2048 + row * 128 + (((piece & 7) ^ (row & 7)) << 4)); }

__device__ __forceinline__ void mma_bf16_1688(float (&d)[4], uint32_t a0, uint32_t a1, uint32_t b0) {
  asm volatile("mma.sync.aligned.m16n8k8.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5}, {%6}, {%0,%1,%2,%3};"
               : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
               : "r"(a0), "r"(a1), "r"(b0));
}

__device__ __forceinline__ void ldmatrix_x2(uint32_t (&r)[2], uint32_t smem_addr) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x2.shared.b16 {%0,%1}, [%2];" : "=r"(r[0]), "=r"(r[1]) : "r"(smem_addr));
}

// Table of the requests that have tokens, behind the other small areas of shared memory: two vectors in front, [0] what it was built for
// (slots, kv heads, query heads of one, page | contiguous) and [1] the number of entries, the steps, the items of shared tiles (0: ranges), the first slot; then two
// vectors an entry, {first token, tokens, kv0 (contiguous caches: slot), length} and {first step (shared tiles: item), first tile,
// first record (ranges: of the pass), parts of a tile}.  The order is that of the batch slots, the same in every worker.  Warp 0
// builds it in the first attention task of a launch (three round trips to L2); it holds for every layer with the same geometry.  More than kAttnTableCap
// requests (graphs without linears) are gone through in passes of so many slots, each a task with a table of its own.
// One pointer and counts that are read where they are used: held in registers they were spilled in the loop over the steps.
struct AfTable {
  int4 *at;
  __device__ __forceinline__ int n() const { return at[1].x; }
  __device__ __forceinline__ int total() const { return at[1].y; }
  __device__ __forceinline__ int items() const { return at[1].z; }
  __device__ __forceinline__ int4 &req(int e) const { return at[2 * e + 2]; }
  __device__ __forceinline__ int4 &pos(int e) const { return at[2 * e + 3]; }
};
// kv heads that go together: the largest power of two, eight at most, that divides their number.
__device__ __forceinline__ int af_heads(int hkv) { return min(hkv & -hkv, 8); }
// Shared tiles: parts of a tile of S steps, of `tile_steps` in all.  As many whole shares of a worker as it holds, so that a long request
// among short ones is cut however many tiles there are; every part leaves the last one to arrive a record, so no more than 16 and one for
// each 96 steps, and 64 in all.  The parts of cut tiles, each with a record, are no more than the workers.
// Measured, every tile cut into workers / tiles parts and now: 6 layers, 8 kv heads, one request of 16000 positions and 15 of 64 2163 -> 1022 us; one layer alone,
// one request, 1 kv head, 1000 positions 80 -> 35 us, 16000 84 -> 50, 100000 94 -> 76.  Caps tried there: 16, 24 and 32 parts 35, 39 and 41 us at
// 1000 positions, 53, 51 and 51 at 16000, 121, 98 and 88 at 100000 (64: 76); in a model of 4 kv heads, 16000 positions, 23, 31, 36 and 37 parts 19.2, 18.3, 17.3 and 15.0.
__device__ __forceinline__ int af_parts(int S, int workers, int tile_steps) { return max(1, min(S * workers / tile_steps, min(16 + S / 96, 64))); }
// Whole shares leave a tile of just under two of them in one part.  Where all tiles get a worker at once (tiles <= workers), the smallest
// limit of steps that keeps the parts no more than the workers is taken if its longest part is shorter (returns the limit, 0: whole shares).
// Limits are the average share times 1, 9/8, 10/8 .. 39/8, one per lane.  FP8, 12 layers of width 2048, 8 requests of 700 to 1400 positions
// 1201 -> 1180 us (every tile in workers / tiles parts: 1166), 6 layers of width 4096 1067 -> 1061 us; one long request among short ones keeps whole shares.
__device__ __forceinline__ int af_limit(const AfTable &t, int n, int hkv, int G, int workers, int tile_steps) {
  const int lane = threadIdx.x & 31, limit = ((tile_steps + workers - 1) / workers * (8 + lane) + 7) / 8;
  int parts = 0, longest = 0, shares = 0;
  for (int e = 0; e < n; ++e) {
    const int S = (t.req(e).w + kAfRows - 1) / kAfRows, k = min((S + limit - 1) / limit, min(16 + S / 96, 64)), f = af_parts(S, workers, tile_steps);
    parts += hkv * ((t.req(e).y * G + 15) / 16) * k;
    longest = max(longest, (S + k - 1) / k);
    shares = max(shares, (S + f - 1) / f);
  }
  const unsigned fits = __ballot_sync(0xffffffffu, parts <= workers && longest < shares);
  return fits ? __shfl_sync(0xffffffffu, limit, __ffs(fits) - 1) : 0;
}
static __device__ __noinline__ void af_build_table(const KernelParams &P, const TaskDesc &d, const AfTable t) {
  const int lane = threadIdx.x & 31, slot0 = d.a[A_SLOT0], slots = min(d.a[A_SLOT], slot0 + d.a[A_PASS]), G = d.a[A_HQ] / d.a[A_HKV], hkv = d.a[A_HKV], page = d.a[A_PAGE], hh = af_heads(hkv);
  // records and tickets of a pass are its own: the tiles of earlier slots are no more than one a slot and kv head and one for each 16 rows
  const int record0 = slot0 / d.a[A_PASS] * P.num_workers * 16;
  int n = 0, steps = 0, tiles = hkv * (slot0 + (slot0 && !(d.a[A_FLAGS] & 4) ? __ldcg(&P.meta.qo_indptr[slot0]) * G / 16 : 0));
  for (int s0 = slot0; s0 < slots; s0 += 32) {
    const int slot = s0 + lane;
    int4 r = make_int4(0, 0, 0, 0);
    if (slot < slots) {
      if (d.a[A_FLAGS] & 4) {   // contiguous cache: one token per slot, length = step + 1
        r = make_int4(slot, slot < active_tokens(P) ? 1 : 0, slot, P.meta.step ? __ldcg(&P.meta.step[slot]) + 1 : 1);
      } else {
        r.x = __ldcg(&P.meta.qo_indptr[slot]);
        r.y = __ldcg(&P.meta.qo_indptr[slot + 1]) - r.x;
        r.z = __ldcg(&P.meta.paged_kv_indptr[slot]);
        const int pages = __ldcg(&P.meta.paged_kv_indptr[slot + 1]) - r.z;
        r.w = (pages - 1) * page + __ldcg(&P.meta.paged_kv_last_page_len[slot]);
      }
    }
    const bool on = r.y > 0 && r.w >= r.y;
    const unsigned bal = __ballot_sync(0xffffffffu, on);
    const int at = n + __popc(bal & ((1u << lane) - 1u));
    const int nt = on ? hkv * ((r.y * G + 15) / 16) : 0, ns = nt / hh * ((r.w + kAfRows - 1) / kAfRows);
    int it = nt, is = ns;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int a = __shfl_up_sync(0xffffffffu, it, o), b = __shfl_up_sync(0xffffffffu, is, o);
      if (lane >= o) { it += a; is += b; }
    }
    if (on && at < d.a[A_CAP]) {
      t.req(at) = r;
      t.pos(at) = make_int4(steps + is - ns, tiles + it - nt, record0, 1);
    }
    steps += __shfl_sync(0xffffffffu, is, 31);
    tiles += __shfl_sync(0xffffffffu, it, 31);
    n += __popc(bal);
  }
  n = min(n, d.a[A_CAP]);
  int items = 0;
  if (steps < P.num_workers * (8 / hh) * kAfMinSteps) {   // few steps to a range: the warps share tiles
    int recs = 0;
    __syncwarp();
    const int limit = n > 0 && n * hkv <= P.num_workers ? af_limit(t, n, hkv, G, P.num_workers, steps * hh) : 0;
    for (int e0 = 0; e0 < n; e0 += 32) {
      const int e = e0 + lane;
      int parts = 0, nt = 0;
      if (e < n) {
        nt = hkv * ((t.req(e).y * G + 15) / 16);
        const int S = (t.req(e).w + kAfRows - 1) / kAfRows;
        parts = limit ? min((S + limit - 1) / limit, min(16 + S / 96, 64)) : af_parts(S, P.num_workers, steps * hh);
      }
      int it = nt * parts, ir = parts > 1 ? it : 0;
      const int own = it, rec = ir;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const int a = __shfl_up_sync(0xffffffffu, it, o), b = __shfl_up_sync(0xffffffffu, ir, o);
        if (lane >= o) { it += a; ir += b; }
      }
      if (e < n) {
        t.pos(e).x = items + it - own;
        t.pos(e).z = record0 + recs + ir - rec;
        t.pos(e).w = parts;
      }
      items += __shfl_sync(0xffffffffu, it, 31);
      recs += __shfl_sync(0xffffffffu, ir, 31);
    }
  }
  if (lane == 0) {
    t.at[0] = make_int4(d.a[A_SLOT], hkv, G, (d.a[A_FLAGS] & 4) ? -page : page);
    t.at[1] = make_int4(n, steps, items, slot0);
  }
}

// Thread 0 acquires the task's events, then the compute warps meet (wait_dependencies, for bodies that take no Ctx).
static __device__ __noinline__ bool af_wait(const KernelParams &P, const TaskDesc &d, unsigned long long iteration, uint64_t deadline, int *flags, int task) {
  if (threadIdx.x == 0) {
    bool good = flags[0] == 0;
    for (int i = 0; i < kMaxDeps && good; ++i) {
      const int ev = d.dep_event[i];
      if (ev < 0) continue;
      const unsigned long long need = (unsigned long long)d.dep_need[i] * iteration;
      const bool remote = (d.flags & (TF_DEP0_REMOTE << i)) != 0;
      uint32_t polls = 0;
      while ((remote ? ld_acquire_sys(&P.counters[ev]) : ld_acquire_gpu(&P.counters[ev])) < need) {
        if ((++polls & 0xff) != 0) continue;
        if (ld_volatile_i32(&P.status->error) != 0) { good = false; break; }
        if (globaltimer_ns() > deadline) {
          report_timeout(P.status, (int)blockIdx.x, 1, task);
          good = false;
          break;
        }
      }
    }
    if (!good) flags[0] = 1;
    *reinterpret_cast<volatile uint64_t *>(flags + 6) = globaltimer_ns();   // (profiler: dependencies satisfied)
  }
  consumer_sync();
  return *reinterpret_cast<volatile int *>(flags) == 0;
}

// Where a warp stands: tile (entry of the table, head group, query tile) and step, and what it needs of the request.
struct AfCursor {
  int e, h, i, s;            // table entry, head group, query tile, step
  int kv0, nq, q0, len, S, I;
  int pg, off;               // page of the step's first position, and the position within it
};
__device__ __forceinline__ void af_load(AfCursor &c, const AfTable &t, int G) {
  const int4 r = t.req(c.e);
  c.q0 = r.x; c.nq = r.y; c.kv0 = r.z; c.len = r.w;
  c.S = (c.len + kAfRows - 1) / kAfRows;
  c.I = (c.nq * G + 15) / 16;
}
__device__ __forceinline__ void af_next_tile(AfCursor &c, const AfTable &t, int G, int groups) {
  c.s = c.pg = c.off = 0;
  if (++c.i < c.I) return;
  c.i = 0;
  if (++c.h < groups) return;
  c.h = 0;
  if (++c.e < t.n()) af_load(c, t, G);
}
// Infinities and NaNs of the value rows of positions pos .. end - 1, which the products took for zeros (0 x infinity is NaN, for every query
// row of a tile): each goes to the rows of the tile that see its position (`first`: of the tile's first token).  Out of line, on parts in
// memory: as code of the segment, on the accumulators, it cost 16 requests of 512 to 4000 positions 2 us a layer.
static __device__ __noinline__ void af_put_back(const __nv_bfloat16 *v, int ldq, int pos, int end, int first, int G, int rows, float *acc, int pitch) {
  __syncwarp();
  for (; pos < end; ++pos, v += ldq)
    for (int col = threadIdx.x & 31; col < 128; col += 32) {
      const float x = bf16_to_f(__ldcg(v + col));
      if (fabsf(x) < INFINITY) continue;
      for (int row = max(pos - first, 0) * G; row < rows; ++row) {
        volatile float *to = acc + row * pitch + col;
        *to = *to + x;
      }
    }
  __syncwarp();
}

template <bool shared, bool EXACT>
__device__ __forceinline__ bool run_attention_steps(const KernelParams &P, const TaskDesc &d, uint8_t *xtile, int *sflags, const AfTable &tab,
                                                    unsigned long long iteration, uint64_t deadline, int task) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, q = lane & 3;
  const int hkv = d.a[A_HKV], G = d.a[A_HQ] / hkv, flags = d.a[A_FLAGS], page = (flags & 4) ? 1 << 30 : d.a[A_PAGE];
  const int nstg = d.a[A_NSTAGE];
  const uint32_t tile = (smem_u32(xtile) + 1023u) & ~1023u;
  const int hh = af_heads(hkv), hw = warp & (hh - 1), groups = hkv / hh;   // this warp's head of every head group
  const int ranges = P.num_workers * (8 / hh);
  const int total = tab.total(), per = max((total + ranges - 1) / ranges, kAfMinSteps);
  const int range = warp / hh * P.num_workers + d.a[A_CHUNK];
  int item = d.a[A_CHUNK];                                      // (tile, part) of this worker, then the one num_workers on
  const int u0 = min(range * per, total);
  int left = shared ? 0 : min(per, total - u0);                 // steps to consume
  int flying = 0;                                               // requested steps that have not been consumed
  const uint32_t qbuf = tile + (uint32_t)(warp * (nstg + 1) * kAfStage), ring = qbuf + kAfStage;
  const uint32_t bars = smem_u32(sflags + 16) + (uint32_t)(warp * kAttnStages * 8);
  const uint8_t *maps = reinterpret_cast<const uint8_t *>(P.tmaps) + (size_t)d.a[A_TMAP] * 128;
  int *place = sflags + 16 + 16 * kAttnStages + warp;           // where this warp's ring stood after its last task: parities of the stages
  uint32_t parity = *reinterpret_cast<volatile int *>(place);

  AfCursor cur;
  cur.e = cur.h = cur.i = cur.s = cur.pg = cur.off = 0;
  cur.kv0 = cur.nq = cur.q0 = cur.len = 0;
  cur.S = cur.I = 1;
  int head = 0;                                                 // kv head
  // this warp's steps of the worker's item
  const auto take_item = [&]() {
    cur.e = -1;
    for (int b = 0, n = tab.n(); b < n; b += 32) cur.e += __popc(__ballot_sync(0xffffffffu, b + lane < n && tab.pos(b + lane).x <= item));
    af_load(cur, tab, G);
    const int4 at = tab.pos(cur.e);
    const int NC = at.w, k = (item - at.x) / NC, part = item - at.x - k * NC;
    head = k / cur.I;
    cur.i = k - head * cur.I;
    const int a = cur.S * part / NC, b = cur.S * (part + 1) / NC, first = a + (b - a) * warp / 8;
    left = a + (b - a) * (warp + 1) / 8 - first;
    cur.s = first;
    cur.pg = first * kAfRows / page;
    cur.off = first * kAfRows - cur.pg * page;
  };
  if (shared) {
    if (item < tab.items()) take_item();
  } else if (left > 0) {
    // entry whose steps contain u0: the last one that begins at or before it
    for (int k = 0, n = tab.n(); k < n; k += 32) cur.e += __popc(__ballot_sync(0xffffffffu, k + lane < n && tab.pos(k + lane).x <= u0));
    --cur.e;
    af_load(cur, tab, G);
    int u = u0 - tab.pos(cur.e).x;
    cur.s = u % cur.S;
    u /= cur.S;
    cur.i = u % cur.I;
    cur.h = u / cur.I;
    cur.pg = cur.s * kAfRows / page;
    cur.off = cur.s * kAfRows - cur.pg * page;
    head = cur.h * hh + hw;
  }
  AfCursor req = cur;                                           // the requesting cursor runs ahead
  int togo = left;                                              // steps to request
  int pg0 = 0, pages = 0;                                       // lane l holds the id of page pg0 + l of the requesting cursor's request
  bool have = false;
  int in_slot = 0;                                              // ring stage of the next request
  bool ok = true;
  const auto request = [&]() {
    if (togo > 0 && ok) {
      --togo;
      ++flying;
      const uint32_t bar = bars + (uint32_t)(in_slot * 8);
      if (req.s * kAfRows < req.len - req.nq) {                 // some of its positions lie in the cache
        int row;
        if (flags & 4) {
          row = req.kv0 * d.a[A_CSEQ] + req.off;
        } else {
          if (!have || req.pg < pg0 || req.pg >= pg0 + 32) {
            pg0 = req.pg;
            pages = req.pg + lane < (req.len + page - 1) / page ? __ldcg(&P.meta.paged_kv_indices[req.kv0 + req.pg + lane]) : 0;
            have = true;
          }
          row = __shfl_sync(0xffffffffu, pages, req.pg - pg0) * page + req.off;
        }
        if (lane == 0) {
          const uint32_t dst = ring + (uint32_t)(in_slot * kAfStage);
          const int at = shared ? head : req.h * hh + hw;
          bar_arrive_expect_tx(bar, kAfStage);
          tma_load_3d_shared(dst, maps, 0, row, 2 * at, bar);
          tma_load_3d_shared(dst + kAfTile, maps + 128, 0, row, 2 * at, bar);
        }
      } else if (lane == 0) {
        bar_arrive(bar);
      }
      if (++in_slot == nstg) in_slot = 0;
      req.off += kAfRows;
      if (req.off >= page) { req.off = 0; ++req.pg; }
      if (++req.s == req.S && !shared) {
        const int e = req.e;
        af_next_tile(req, tab, G, groups);
        if (req.e != e) have = false;
      }
    }
  };
  for (int j = 0; j < nstg - 1; ++j) request();
  ok = af_wait(P, d, iteration, deadline, sflags, task);
  const bool run = ok;                                          // (the same in all warps)

  // (pointers are read from the descriptor where they are used: registers)
  const auto ptr = [&](int k, bool on) { return on ? reinterpret_cast<const __nv_bfloat16 *>(d.p[k]) : nullptr; };
  const int ldq = d.a[A_LDQKV], ldo = d.a[A_LDO], rope_rows = d.a[A_ROPE_ROWS];
  const float eps = __int_as_float(d.a[A_EPS]);
  const int TP = 16 / G;                                        // tokens of a query tile
  int out_slot = 0, unit = u0;
  // (a warp whose wait was abandoned still takes part in the barriers of shared tiles)
  while (run && (shared ? item < tab.items() : ok && left > 0)) {
    // ---- query tile of this segment: rows (token, head), normed and rotated ----
    const int t0 = cur.i * TP, rows = min(16, (cur.nq - t0) * G), new_start = cur.len - cur.nq;
    if (!shared) head = cur.h * hh + hw;
    const size_t head0 = (size_t)head * (G + 2) * 128 + lane * 4;
    // (warps that share a tile share it out, two rows each)
    const uint32_t qtile = shared ? tile : qbuf;
    const int rend = shared ? 2 : 16;
    for (int r = 0; r < rend; r += 2) {
      const __nv_bfloat16 *qkv = ptr(0, true), *qn = ptr(3, flags & 1), *cosT = ptr(5, flags & 2), *sinT = ptr(6, flags & 2);
      uint2 x2[2], cs[2], sn[2];
#pragma unroll
      for (int k = 0; k < 2; ++k) {
        const int row = shared ? warp + 8 * k : r + k;
        x2[k] = make_uint2(0, 0);
        if (r + k < rend && row < rows) {
          load_rope(cosT, sinT, new_start + t0 + row / G, rope_rows, lane, cs[k], sn[k]);
          x2[k] = __ldcg(reinterpret_cast<const uint2 *>(qkv + (size_t)(cur.q0 + t0 + row / G) * ldq + head0 + (size_t)(row % G) * 128));
        }
      }
#pragma unroll
      for (int k = 0; k < 2; ++k) {
        const int row = shared ? warp + 8 * k : r + k;
        if (r + k >= rend) continue;
        if (row < rows) {
          float x[4] = {bf16_lo(x2[k].x), bf16_hi(x2[k].x), bf16_lo(x2[k].y), bf16_hi(x2[k].y)};
          norm_rope_head(x, qn, eps, cosT != nullptr, cs[k], sn[k], lane);
          x2[k] = make_uint2(pack_bf16(x[0], x[1]), pack_bf16(x[2], x[3]));
        }
        asm volatile("st.shared.v2.b32 [%0], {%1, %2};" ::"r"(qtile + af_qpiece(row, lane >> 1) + (lane & 1) * 8), "r"(x2[k].x), "r"(x2[k].y) : "memory");
      }
    }
    if (shared) consumer_sync();
    __syncwarp();
    const int lim0 = new_start + t0 + g / G, lim1 = new_start + t0 + (g + 8) / G;   // last position that row g / row g + 8 sees
    float m0 = -INFINITY, m1 = -INFINITY, l0 = 0.f, l1 = 0.f, o[16][4];
#pragma unroll
    for (int nt = 0; nt < 16; ++nt) o[nt][0] = o[nt][1] = o[nt][2] = o[nt][3] = 0.f;

    const int seg = shared ? left : min(left, cur.S - cur.s), first_s = cur.s;
    for (int j = 0; j < seg && ok; ++j) {
      ok = wait_bar(P, bars + (uint32_t)(out_slot * 8), (parity >> out_slot) & 1u, deadline, task);
      ok = __all_sync(0xffffffffu, ok);
      if (!ok) break;
      --flying;
      request();                                                // (into the stage before this one, which the whole warp has left)
      const uint32_t kt = ring + (uint32_t)(out_slot * kAfStage), vt = kt + kAfTile;
      parity ^= 1u << out_slot;
      if (++out_slot == nstg) out_slot = 0;
      const int pos0 = (first_s + j) * kAfRows;
      if (pos0 + kAfRows > new_start) {
        // rows that this launch appends; behind them zeros (a masked position has weight 0, and 0 x NaN would still be NaN)
        const int end = min(pos0 + kAfRows, cur.len);
        for (int r = end - pos0; r < kAfRows; ++r) {
          const uint32_t to = af_piece(r, lane >> 1) + (lane & 1) * 8;
          asm volatile("st.shared.v2.b32 [%0], {%1, %1};" ::"r"(kt + to), "r"(0u) : "memory");
          asm volatile("st.shared.v2.b32 [%0], {%1, %1};" ::"r"(vt + to), "r"(0u) : "memory");
        }
        for (int p0 = max(pos0, new_start); p0 < end; p0 += 2) {   // two rows' loads in flight
          const __nv_bfloat16 *qkv = ptr(0, true), *kn = ptr(4, flags & 1), *cosT = ptr(5, flags & 2), *sinT = ptr(6, flags & 2);
          uint2 kr[2], vr[2], cs[2], sn[2];
#pragma unroll
          for (int k = 0; k < 2; ++k) {
            const int pos = min(p0 + k, end - 1);
            const __nv_bfloat16 *kp = qkv + (size_t)(cur.q0 + pos - new_start) * ldq + head0 + (size_t)G * 128;
            kr[k] = __ldcg(reinterpret_cast<const uint2 *>(kp));
            vr[k] = __ldcg(reinterpret_cast<const uint2 *>(kp + 128));
            load_rope(cosT, sinT, pos, rope_rows, lane, cs[k], sn[k]);
          }
#pragma unroll
          for (int k = 0; k < 2; ++k) {
            const int pos = p0 + k;
            if (pos >= end) continue;
            float x[4] = {bf16_lo(kr[k].x), bf16_hi(kr[k].x), bf16_lo(kr[k].y), bf16_hi(kr[k].y)};
            norm_rope_head(x, kn, eps, cosT != nullptr, cs[k], sn[k], lane);
            const uint2 kw = make_uint2(pack_bf16(x[0], x[1]), pack_bf16(x[2], x[3]));
            const uint32_t to = af_piece(pos - pos0, lane >> 1) + (lane & 1) * 8;
            asm volatile("st.shared.v2.b32 [%0], {%1, %2};" ::"r"(kt + to), "r"(kw.x), "r"(kw.y) : "memory");
            // (0 x infinity is NaN, for every query row of the tile: such values are zero here and are put back later)
            uint2 vs = vr[k];
            if (__builtin_expect(__any_sync(0xffffffffu, !finite_bf16x2(vs.x) || !finite_bf16x2(vs.y)), 0)) {
              parity |= kAfWild;
              vs = make_uint2(finite_or_zero_bf16x2(vs.x), finite_or_zero_bf16x2(vs.y));
            }
            asm volatile("st.shared.v2.b32 [%0], {%1, %2};" ::"r"(vt + to), "r"(vs.x), "r"(vs.y) : "memory");
            if (cur.i == 0) {   // the first tile's warp writes the cache
              size_t row;
              if (flags & 4) row = (size_t)cur.kv0 * d.a[A_CSEQ] + pos;
              else row = (size_t)__ldcg(&P.meta.paged_kv_indices[cur.kv0 + pos / page]) * page + pos % page;
              const size_t off = (row * hkv + head) * 128 + lane * 4;
              *reinterpret_cast<uint2 *>(reinterpret_cast<__nv_bfloat16 *>(d.p[1]) + off) = kw;
              *reinterpret_cast<uint2 *>(reinterpret_cast<__nv_bfloat16 *>(d.p[2]) + off) = vr[k];
            }
          }
        }
        fence_proxy_async_smem();                               // these stores come before the copy that refills the stage
        __syncwarp();
      }
      // ---- scores, online softmax, P V ----
      float sc[4] = {0.f, 0.f, 0.f, 0.f}, sd[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
      for (int kk = 0; kk < 4; ++kk) {
        uint32_t a[4], b[4];                                    // (the query fragments are read again each step: registers)
        ldmatrix_x4(b, kt + af_piece(lane & 7, 4 * kk + (lane >> 3)));
        ldmatrix_x4(a, qtile + af_qpiece(lane & 15, 4 * kk + (lane >> 4)));
        mma_bf16_16816(sc, a, b[0], b[1]);
        ldmatrix_x4(a, qtile + af_qpiece(lane & 15, 4 * kk + 2 + (lane >> 4)));
        mma_bf16_16816(sd, a, b[2], b[3]);
      }
      const float qscale = 0.08838834764831845f * 1.4426950408889634f;   // 1/sqrt(128) * log2(e)
      const int p = pos0 + 2 * q;
      const float s0 = p <= lim0 ? (sc[0] + sd[0]) * qscale : -INFINITY, s1 = p + 1 <= lim0 ? (sc[1] + sd[1]) * qscale : -INFINITY;
      const float s2 = p <= lim1 ? (sc[2] + sd[2]) * qscale : -INFINITY, s3 = p + 1 <= lim1 ? (sc[3] + sd[3]) * qscale : -INFINITY;
      float x0 = fmaxf(s0, s1), x1 = fmaxf(s2, s3);
      x0 = fmaxf(x0, __shfl_xor_sync(0xffffffffu, x0, 1));
      x1 = fmaxf(x1, __shfl_xor_sync(0xffffffffu, x1, 1));
      x0 = fmaxf(x0, __shfl_xor_sync(0xffffffffu, x0, 2));
      x1 = fmaxf(x1, __shfl_xor_sync(0xffffffffu, x1, 2));
      const float n0 = fmaxf(m0, x0), n1 = fmaxf(m1, x1);
      const float z0 = n0 == -INFINITY ? 0.f : n0, z1 = n1 == -INFINITY ? 0.f : n1;   // (a row that sees nothing yet)
      const float c0 = exp2f(m0 - z0), c1 = exp2f(m1 - z1);                            // 0 on the first step (m = -inf)
      const float p0 = exp2f(s0 - z0), p1 = exp2f(s1 - z0), p2 = exp2f(s2 - z1), p3 = exp2f(s3 - z1);
      l0 = l0 * c0 + p0 + p1;                                                           // (this lane's columns; summed over the quad at the end)
      l1 = l1 * c1 + p2 + p3;
      m0 = n0;
      m1 = n1;
      if (__any_sync(0xffffffffu, c0 != 1.f || c1 != 1.f)) {
#pragma unroll
        for (int nt = 0; nt < 16; ++nt) { o[nt][0] *= c0; o[nt][1] *= c0; o[nt][2] *= c1; o[nt][3] *= c1; }
      }
      uint32_t pw[4] = {pack_bf16(p0, p1), pack_bf16(p2, p3), 0u, 0u};
      if (EXACT) {
        // P as the sum of two bf16, side by side along k, and V twice: less than 2^-17 of a weight is lost.  Graphs of few tokens, whose batch-1 form
        // holds the weights in fp32 (for all graphs: 16 requests 6.51 -> 6.62 ms, 64 requests 7.79 -> 7.97)
        pw[2] = pack_bf16(p0 - bf16_lo(pw[0]), p1 - bf16_hi(pw[0]));
        pw[3] = pack_bf16(p2 - bf16_lo(pw[1]), p3 - bf16_hi(pw[1]));
      }
#pragma unroll
      for (int vq = 0; vq < 4; ++vq) {
        uint32_t b[4];
        ldmatrix_x4_trans(b, vt + af_piece(lane & 7, 4 * vq + (lane >> 3)));
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          if (EXACT) mma_bf16_16816(o[4 * vq + k], pw, b[k], b[k]);
          else mma_bf16_1688(o[4 * vq + k], pw[0], pw[1], b[k]);
        }
      }
      __syncwarp();                                             // every lane is done with the stage before it is refilled
    }
    if (!ok && !shared) break;
    l0 += __shfl_xor_sync(0xffffffffu, l0, 1);
    l1 += __shfl_xor_sync(0xffffffffu, l1, 1);
    l0 += __shfl_xor_sync(0xffffffffu, l0, 2);
    l1 += __shfl_xor_sync(0xffffffffu, l1, 2);

    // ---- results of the segment ----
    __nv_bfloat16 *out = reinterpret_cast<__nv_bfloat16 *>(d.p[7]);
    const size_t row_out = (size_t)(cur.q0 + t0) * ldo + (size_t)head * G * 128;
    const auto put_back = [&](float *acc, int pitch) {
      parity &= ~kAfWild;
      const int pos = max(first_s * kAfRows, new_start);
      af_put_back(ptr(0, true) + (size_t)(cur.q0 + pos - new_start) * ldq + (size_t)(head * (G + 2) + G + 1) * 128, ldq, pos,
                  min((first_s + seg) * kAfRows, cur.len), new_start + t0, G, rows, acc, pitch);
    };
    if (shared) {
      // the eight warps' parts meet in shared memory: sums and maxima where the query tiles were, outputs in the rings (idle now)
      consumer_sync();                                          // (the query tile has been read by all)
      float *mine = reinterpret_cast<float *>(xtile + (ring - smem_u32(xtile))), *ml = reinterpret_cast<float *>(xtile + (qbuf - smem_u32(xtile)));
#pragma unroll
      for (int half = 0; half < 2; ++half) {
        const int row = g + 8 * half;
        if (row < rows) {
          if (q == 0) { ml[2 * row] = half ? m1 : m0; ml[2 * row + 1] = half ? l1 : l0; }
#pragma unroll
          for (int nt = 0; nt < 16; ++nt) *reinterpret_cast<float2 *>(mine + row * 128 + nt * 8 + 2 * q) = make_float2(o[nt][2 * half], o[nt][2 * half + 1]);
        }
      }
      if (__builtin_expect((parity & kAfWild) != 0u, 0)) put_back(mine, 128);
      consumer_sync();
      const int4 at = tab.pos(cur.e);
      const int NC = at.w, pitch = (nstg + 1) * kAfStage / 4;               // floats between two warps' areas
      const float *ml0 = reinterpret_cast<const float *>(xtile + (tile - smem_u32(xtile)));
      for (int idx = threadIdx.x; idx < rows * 128; idx += kConsumerThreads) {
        const int row = idx >> 7, dim = idx & 127;
        float M = -INFINITY, L = 0.f, O = 0.f;
#pragma unroll
        for (int w = 0; w < 8; ++w) M = fmaxf(M, ml0[w * pitch + 2 * row]);
        const float z = M == -INFINITY ? 0.f : M;
#pragma unroll
        for (int w = 0; w < 8; ++w) {
          const float e = exp2f(ml0[w * pitch + 2 * row] - z);
          L += ml0[w * pitch + 2 * row + 1] * e;
          O += ml0[w * pitch + kAfStage / 4 + row * 128 + dim] * e;
        }
        if (NC == 1) {
          out[row_out + (size_t)(row / G) * ldo + (size_t)(row % G) * 128 + dim] = __float2bfloat16_rn(L > 0.f ? O / L : 0.f);
        } else {
          float *rec = P.attn_scratch + (size_t)(d.a[A_BANK] + at.z + item - at.x) * kAfRecord + row * 132;
          if (dim == 0) __stcg(reinterpret_cast<float2 *>(rec), make_float2(M, L));
          __stcg(rec + 4 + dim, O);
        }
      }
      if (NC > 1) {
        consumer_sync();
        const int k = head * cur.I + cur.i;
        if (threadIdx.x == 0) {
          unsigned int old, *ticket = &P.attn_tickets[d.a[A_TICKET] + at.y + k];
          asm volatile("atom.acq_rel.gpu.global.add.u32 %0, [%1], 1;" : "=r"(old) : "l"(ticket) : "memory");
          const bool last = old + 1u == (unsigned)NC;
          if (last) *ticket = 0u;                                // for the next launch
          sflags[4] = last ? 1 : 0;
        }
        consumer_sync();
        for (int idx = threadIdx.x; sflags[4] && idx < rows * 128; idx += kConsumerThreads) {
          const int row = idx >> 7, dim = idx & 127;
          const float *rec = P.attn_scratch + (size_t)(d.a[A_BANK] + at.z + k * NC) * kAfRecord + row * 132;
          float M = -INFINITY, L = 0.f, O = 0.f;
          for (int c0 = 0; c0 < NC; c0 += 8) {
            float2 pm[8];
            float po[8];
#pragma unroll
            for (int c = 0; c < 8; ++c) {
              const bool on = c0 + c < NC;
              pm[c] = on ? __ldcg(reinterpret_cast<const float2 *>(rec + (size_t)(c0 + c) * kAfRecord)) : make_float2(-INFINITY, 0.f);
              po[c] = on ? __ldcg(rec + (size_t)(c0 + c) * kAfRecord + 4 + dim) : 0.f;
            }
            float N = M;
#pragma unroll
            for (int c = 0; c < 8; ++c) N = fmaxf(N, pm[c].x);
            const float z = N == -INFINITY ? 0.f : N, w = exp2f(M - z);
            L *= w;
            O *= w;
#pragma unroll
            for (int c = 0; c < 8; ++c) {
              const float e = exp2f(pm[c].x - z);
              L += pm[c].y * e;
              O += po[c] * e;
            }
            M = N;
          }
          out[row_out + (size_t)(row / G) * ldo + (size_t)(row % G) * 128 + dim] = __float2bfloat16_rn(L > 0.f ? O / L : 0.f);
        }
      }
      item += P.num_workers;
      left = 0;
      if (item < tab.items()) {
        fence_proxy_async_smem();                               // the rings were written and read through the generic proxy
        consumer_sync();
        take_item();
        req = cur;
        togo = left;
        have = false;
        for (int j = 0; j < nstg - 1; ++j) request();
      }
      continue;
    }
    if (seg == cur.S && __builtin_expect((parity & kAfWild) == 0u && !(flags & 8), 1)) {
      // (a row whose sum is not positive, or NaN, is zero in every form)
      if (__builtin_expect(!(l0 > 0.f && l1 > 0.f), 0)) {
#pragma unroll
        for (int nt = 0; nt < 16; ++nt) {
          if (!(l0 > 0.f)) o[nt][0] = o[nt][1] = 0.f;
          if (!(l1 > 0.f)) o[nt][2] = o[nt][3] = 0.f;
        }
      }
      const float i0 = l0 > 0.f ? 1.f / l0 : 0.f, i1 = l1 > 0.f ? 1.f / l1 : 0.f;
#pragma unroll
      for (int half = 0; half < 2; ++half) {
        const int row = g + 8 * half;
        if (row < rows) {
          __nv_bfloat16 *dst = out + row_out + (size_t)(row / G) * ldo + (size_t)(row % G) * 128 + 2 * q;
#pragma unroll
          for (int nt = 0; nt < 16; ++nt)
            *reinterpret_cast<uint32_t *>(dst + nt * 8) = pack_bf16(o[nt][2 * half] * (half ? i1 : i0), o[nt][2 * half + 1] * (half ? i1 : i0));
        }
      }
    } else {
      // a range has at most two records: of the tile it begins in (0) and of the one it ends in (1; whole tiles with values to put back
      // pass through it, and all tiles where the output allows no wide stores)
      float *rec = P.attn_scratch + (size_t)(d.a[A_BANK] + tab.pos(cur.e).z + (2 * range + (unit == u0 ? 0 : 1)) * hh + hw) * kAfRecord;
#pragma unroll
      for (int half = 0; half < 2; ++half) {
        const int row = g + 8 * half;
        if (row < rows) {
          float *dst = rec + row * 132;
          if (q == 0) __stcg(reinterpret_cast<float2 *>(dst), half ? make_float2(m1, l1) : make_float2(m0, l0));
#pragma unroll
          for (int nt = 0; nt < 16; ++nt) __stcg(reinterpret_cast<float2 *>(dst + 4 + nt * 8 + 2 * q), make_float2(o[nt][2 * half], o[nt][2 * half + 1]));
        }
      }
      if (__builtin_expect((parity & kAfWild) != 0u, 0)) put_back(rec + 4, 132);
      __threadfence();
      __syncwarp();
      const int begin = unit - first_s, end = begin + cur.S;     // the tile's steps
      const int r0 = begin / per, parts = (end - 1) / per - r0 + 1;
      unsigned int *ticket = &P.attn_tickets[d.a[A_TICKET] + tab.pos(cur.e).y + head * cur.I + cur.i];
      unsigned int old = 0;
      if (lane == 0) asm volatile("atom.acq_rel.gpu.global.add.u32 %0, [%1], 1;" : "=r"(old) : "l"(ticket) : "memory");
      old = __shfl_sync(0xffffffffu, old, 0);
      if (old + 1u == (unsigned)parts) {
        __syncwarp();                                           // lane 0's acquire holds for all of them: a shuffle orders no memory
        if (lane == 0) *ticket = 0u;                            // for the next launch
        const int record0 = d.a[A_BANK] + tab.pos(cur.e).z;
        for (int row = 0; row < rows; ++row) {
          float M = -INFINITY, L = 0.f;
          float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
          for (int k0 = 0; k0 < parts; k0 += 8) {
            float2 ml[8];
            float4 ov[8];
#pragma unroll
            for (int k = 0; k < 8; ++k) {
              ml[k] = make_float2(-INFINITY, 0.f);
              ov[k] = make_float4(0.f, 0.f, 0.f, 0.f);
              if (k0 + k < parts) {
                const int r = r0 + k0 + k;
                const float *src = P.attn_scratch + (size_t)(record0 + (2 * r + (begin <= r * per ? 0 : 1)) * hh + hw) * kAfRecord + row * 132;
                ml[k] = __ldcg(reinterpret_cast<const float2 *>(src));
                ov[k] = __ldcg(reinterpret_cast<const float4 *>(src + 4) + lane);
              }
            }
            float N = M;
#pragma unroll
            for (int k = 0; k < 8; ++k) N = fmaxf(N, ml[k].x);
            const float z = N == -INFINITY ? 0.f : N, w = exp2f(M - z);
            L *= w; acc.x *= w; acc.y *= w; acc.z *= w; acc.w *= w;
#pragma unroll
            for (int k = 0; k < 8; ++k) {
              const float e = exp2f(ml[k].x - z);
              L += ml[k].y * e;
              acc.x += ov[k].x * e; acc.y += ov[k].y * e; acc.z += ov[k].z * e; acc.w += ov[k].w * e;
            }
            M = N;
          }
          if (__builtin_expect(!(L > 0.f), 0)) acc = make_float4(0.f, 0.f, 0.f, 0.f);
          const float inv = L > 0.f ? 1.f / L : 0.f;
          __nv_bfloat16 *dst = out + row_out + (size_t)(row / G) * ldo + (size_t)(row % G) * 128 + lane * 4;
          const uint2 y = make_uint2(pack_bf16(acc.x * inv, acc.y * inv), pack_bf16(acc.z * inv, acc.w * inv));
          if (__builtin_expect((flags & 8) != 0, 0)) {
            const uint32_t h[2] = {y.x, y.y};
#pragma unroll
            for (int k = 0; k < 4; ++k) reinterpret_cast<uint16_t *>(dst)[k] = (uint16_t)(h[k >> 1] >> (16 * (k & 1)));
          } else {
            *reinterpret_cast<uint2 *>(dst) = y;
          }
        }
      }
    }
    left -= seg;
    unit += seg;
    cur.s += seg;
    if (cur.s == cur.S) af_next_tile(cur, tab, G, groups);
  }
  if (!ok) {
    // abandoned: what is in flight always arrives; wait for it, a bounded number of polls each
    for (; flying > 0; --flying) {
      uint32_t polls = 0;
      while (!bar_try_wait(bars + (uint32_t)(out_slot * 8), (parity >> out_slot) & 1u) && ++polls < (1u << 22)) {}
      parity ^= 1u << out_slot;
      if (++out_slot == nstg) out_slot = 0;
    }
    sflags[0] = 1;
    return false;
  }
  if (lane == 0) *place = (int)parity;
  __syncwarp();
  return true;
}

template <bool EXACT>
__device__ __forceinline__ bool run_attention_flat(const KernelParams &P, const TaskDesc &d, uint8_t *xtile, int *sflags, unsigned long long iteration,
                                                          uint64_t deadline, int task) {
  const int warp = threadIdx.x >> 5;
  const int hkv = d.a[A_HKV], G = d.a[A_HQ] / hkv, flags = d.a[A_FLAGS];
  const AfTable tab{reinterpret_cast<int4 *>(reinterpret_cast<uint8_t *>(sflags) - kFlagsOffset + kMiscBytes)};
  fence_proxy_async_smem();                                     // earlier generic accesses to the area come before its copies
  if (warp == 0) {
    const int4 k = tab.at[0];
    if (k.x != d.a[A_SLOT] || k.y != hkv || k.z != G || k.w != ((flags & 4) ? -d.a[A_PAGE] : d.a[A_PAGE]) || tab.at[1].w != d.a[A_SLOT0])
      af_build_table(P, d, tab);
  }
  consumer_sync();
  if (tab.total() == 0 || tab.items() > 0) return run_attention_steps<true, EXACT>(P, d, xtile, sflags, tab, iteration, deadline, task);
  return run_attention_steps<false, EXACT>(P, d, xtile, sflags, tab, iteration, deadline, task);
}

static __device__ void run_embed(const Ctx &c, const TaskDesc &d) {
  const int B = active_tokens(c.P);
  const int t0 = d.a[E_T0], t1 = min(d.a[E_T1], B), width = d.a[E_WIDTH];
  const int64_t *ids = reinterpret_cast<const int64_t *>(d.p[0]);
  const __nv_bfloat16 *tab = reinterpret_cast<const __nv_bfloat16 *>(d.p[1]);
  __nv_bfloat16 *out = reinterpret_cast<__nv_bfloat16 *>(d.p[2]);
  const int vecs = width / 8;
  for (int t = t0; t < t1; ++t) {
    const long long id = __ldcg(reinterpret_cast<const long long *>(&ids[t]));
    for (int v = threadIdx.x; v < vecs; v += kConsumerThreads) {
      uint4 val = make_uint4(0, 0, 0, 0);
      // ids outside the table (e.g. the argmax of a row of NaNs) read as a zero row instead of a wild address
      if (id >= 0 && id < (long long)d.a[E_AUX]) val = __ldg(reinterpret_cast<const uint4 *>(tab + (size_t)id * d.a[E_LDI]) + v);
      reinterpret_cast<uint4 *>(out + (size_t)t * d.a[E_LDO])[v] = val;
    }
  }
}

static __device__ void run_rmsnorm(const Ctx &c, const TaskDesc &d) {
  const int B = active_tokens(c.P);
  const int t0 = d.a[E_T0], t1 = min(d.a[E_T1], B), width = d.a[E_WIDTH];
  const __nv_bfloat16 *in = reinterpret_cast<const __nv_bfloat16 *>(d.p[0]);
  const __nv_bfloat16 *gam = reinterpret_cast<const __nv_bfloat16 *>(d.p[1]);
  __nv_bfloat16 *out = reinterpret_cast<__nv_bfloat16 *>(d.p[2]);
  const float eps = __int_as_float(d.a[E_AUX]);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int vecs = width / 8;
  for (int t = t0; t < t1; ++t) {
    const uint4 *row = reinterpret_cast<const uint4 *>(in + (size_t)t * d.a[E_LDI]);
    float ss = 0.f;
    for (int v = tid; v < vecs; v += kConsumerThreads) {
      const uint4 x = __ldcg(row + v);
      const uint32_t w[4] = {x.x, x.y, x.z, x.w};
#pragma unroll
      for (int q = 0; q < 4; ++q) ss += bf16_lo(w[q]) * bf16_lo(w[q]) + bf16_hi(w[q]) * bf16_hi(w[q]);
    }
    ss = warp_sum(ss);
    if (lane == 0) c.s.red[warp] = ss;
    consumer_sync();
    float tot = 0.f;
#pragma unroll
    for (int w = 0; w < 8; ++w) tot += c.s.red[w];
    const float inv = rsqrtf(tot / (float)width + eps);
    for (int v = tid; v < vecs; v += kConsumerThreads) {
      const uint4 x = __ldcg(row + v);
      const uint4 g = __ldg(reinterpret_cast<const uint4 *>(gam) + v);
      const uint32_t xw[4] = {x.x, x.y, x.z, x.w}, gw[4] = {g.x, g.y, g.z, g.w};
      uint32_t ow[4];
#pragma unroll
      for (int q = 0; q < 4; ++q)
        ow[q] = pack_bf16(bf16_lo(xw[q]) * inv * bf16_lo(gw[q]), bf16_hi(xw[q]) * inv * bf16_hi(gw[q]));
      reinterpret_cast<uint4 *>(out + (size_t)t * d.a[E_LDO])[v] = make_uint4(ow[0], ow[1], ow[2], ow[3]);
    }
    consumer_sync();
  }
}

// silu_mul over columns [a[7], a[8]) of the activation (width a[2] = I), group-interleaved input
static __device__ void run_silu_mul(const Ctx &c, const TaskDesc &d) {
  const int B = active_tokens(c.P);
  const int t0 = d.a[E_T0], t1 = min(d.a[E_T1], B), I = d.a[E_WIDTH];
  const int groups = d.a[E_AUX];
  const int per = I / groups;
  const __nv_bfloat16 *in = reinterpret_cast<const __nv_bfloat16 *>(d.p[0]);
  __nv_bfloat16 *out = reinterpret_cast<__nv_bfloat16 *>(d.p[2]);
  const int c0 = d.a[7], c1 = d.a[8];
  if (((per | c0 | c1 | d.a[E_LDI] | d.a[E_LDO]) & 7) == 0 && ((d.p[0] | d.p[2]) & 15) == 0 && t1 > t0) {
    // 16-byte vectors (eight columns of one interleave group), tokens and columns flattened over the threads so that
    // every thread has several independent loads in flight
    const int nv = (c1 - c0) >> 3, total = nv * (t1 - t0);
    for (int i = threadIdx.x; i < total; i += kConsumerThreads) {
      const int t = t0 + i / nv, j = c0 + ((i - (i / nv) * nv) << 3);
      const int g = j / per, off = j - g * per;
      const __nv_bfloat16 *gp = in + (size_t)t * d.a[E_LDI] + (size_t)g * 2 * per + off;
      const uint4 gv = __ldcg(reinterpret_cast<const uint4 *>(gp));
      const uint4 uv = __ldcg(reinterpret_cast<const uint4 *>(gp + per));
      const uint32_t gw[4] = {gv.x, gv.y, gv.z, gv.w}, uw[4] = {uv.x, uv.y, uv.z, uv.w};
      uint32_t ow[4];
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        const float g0 = bf16_lo(gw[q]), g1 = bf16_hi(gw[q]);
        const float a0 = round_bf16(g0 / (1.0f + expf(-g0))), a1 = round_bf16(g1 / (1.0f + expf(-g1)));
        ow[q] = pack_bf16(a0 * bf16_lo(uw[q]), a1 * bf16_hi(uw[q]));
      }
      *reinterpret_cast<uint4 *>(out + (size_t)t * d.a[E_LDO] + j) = make_uint4(ow[0], ow[1], ow[2], ow[3]);
    }
    return;
  }
  for (int t = t0; t < t1; ++t)
    for (int j = c0 + threadIdx.x; j < c1; j += kConsumerThreads) {
      const int g = j / per, off = j - g * per;
      const float gv = bf16_to_f(__ldcg(&in[(size_t)t * d.a[E_LDI] + (size_t)g * 2 * per + off]));
      const float uv = bf16_to_f(__ldcg(&in[(size_t)t * d.a[E_LDI] + (size_t)g * 2 * per + per + off]));
      const float a = round_bf16(gv / (1.0f + expf(-gv)));
      out[(size_t)t * d.a[E_LDO] + j] = __float2bfloat16_rn(a * uv);
    }
}

static __device__ void run_elementwise_add(const Ctx &c, const TaskDesc &d) {
  const int B = active_tokens(c.P);
  const int t0 = d.a[E_T0], t1 = min(d.a[E_T1], B), width = d.a[E_WIDTH];
  const __nv_bfloat16 *a = reinterpret_cast<const __nv_bfloat16 *>(d.p[0]);
  const __nv_bfloat16 *b = reinterpret_cast<const __nv_bfloat16 *>(d.p[1]);
  __nv_bfloat16 *out = reinterpret_cast<__nv_bfloat16 *>(d.p[2]);
  for (int t = t0; t < t1; ++t)
    for (int j = threadIdx.x; j < width; j += kConsumerThreads)
      out[(size_t)t * d.a[E_LDO] + j] = __float2bfloat16_rn(bf16_to_f(__ldcg(&a[(size_t)t * d.a[E_LDI] + j])) +
                                                           bf16_to_f(__ldcg(&b[(size_t)t * d.a[E_LDI2] + j])));
}

static __device__ void run_tensor_init(const Ctx &c, const TaskDesc &d) {
  // zero rows [t0,t1) of width a[2] BYTES
  uint8_t *out = reinterpret_cast<uint8_t *>(d.p[2]);
  const size_t row_bytes = (size_t)d.a[E_WIDTH];
  for (int t = d.a[E_T0]; t < d.a[E_T1]; ++t)
    for (size_t j = threadIdx.x * 4; j < row_bytes; j += kConsumerThreads * 4)
      *reinterpret_cast<uint32_t *>(out + (size_t)t * d.a[E_LDO] + j) = 0u;
}

// (value, index) argmax with lowest-index tie-break
__device__ __forceinline__ void argmax_merge(float &v, long long &i, float v2, long long i2) {
  if (v2 > v || (v2 == v && i2 < i)) {
    v = v2;
    i = i2;
  }
}

static __device__ void block_argmax(const Ctx &c, float &v, long long &i) {
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    const float v2 = __shfl_xor_sync(0xffffffffu, v, o);
    const long long i2 = __shfl_xor_sync(0xffffffffu, i, o);
    argmax_merge(v, i, v2, i2);
  }
  long long *ri = reinterpret_cast<long long *>(c.s.red + 16);
  if (lane == 0) {
    c.s.red[warp] = v;
    ri[warp] = i;
  }
  consumer_sync();
  v = c.s.red[0];
  i = ri[0];
#pragma unroll
  for (int w = 1; w < 8; ++w) argmax_merge(v, i, c.s.red[w], ri[w]);
  consumer_sync();
}

// ---- Gumbel-max sampling (the reference's sampling task, tasks/common/sampling.cuh:100-226) --------------------
// Philox4x32-10 as cuRAND's curand_init(seed, subsequence, offset 0) followed by one curand_uniform4 uses it: the
// counter is (0, 0, subsequence low, subsequence high), the key is the seed, and the four outputs map to
// (0, 1] by x * 2^-32 + 2^-33.
__device__ __forceinline__ uint4 philox4x32_10(uint4 ctr, uint2 key) {
#pragma unroll
  for (int r = 0; r < 10; ++r) {
    const uint32_t hi0 = __umulhi(0xD2511F53u, ctr.x), lo0 = 0xD2511F53u * ctr.x;
    const uint32_t hi1 = __umulhi(0xCD9E8D57u, ctr.z), lo1 = 0xCD9E8D57u * ctr.z;
    ctr = make_uint4(hi1 ^ ctr.y ^ key.x, lo1, hi0 ^ ctr.w ^ key.y, lo0);
    key.x += 0x9E3779B9u;
    key.y += 0xBB67AE85u;
  }
  return ctr;
}

__device__ __forceinline__ float gumbel_noise(uint32_t r) {
  const float u = fmaf(__uint2float_rn(r), 2.3283064e-10f, 1.1641532e-10f);
  return -0.6931471806f * __log2f(-__log2f(u + 1e-20f) + 1e-20f);
}

// (value, index) maximum where equal values go to the highest index: the order the reference's block reduction
// resolves ties in (later element, higher lane, later warp, later pass).
__device__ __forceinline__ void sample_merge(float &v, long long &i, float v2, long long i2) {
  if (v2 > v || (v2 == v && i2 > i)) {
    v = v2;
    i = i2;
  }
}

// One column range of the vocabulary: key = bf16(logit + bf16(noise)), noise by groups of four columns from one
// Philox block whose subsequence is (row within the reference task) * V + first column of the group.
__device__ __forceinline__ float logit_value(const __nv_bfloat16 *p) { return bf16_to_f(__ldcg(p)); }
__device__ __forceinline__ float logit_value(const float *p) { return round_bf16(__ldcg(p)); }
template <typename LOGIT>
__device__ void run_sampling_partial(const Ctx &c, const TaskDesc &d) {
  const int B = active_tokens(c.P);
  const LOGIT *logits = reinterpret_cast<const LOGIT *>(d.p[0]);
  __nv_bfloat16 *pv = reinterpret_cast<__nv_bfloat16 *>(d.p[1]);
  long long *pi = reinterpret_cast<long long *>(d.p[2]);
  const int c0 = d.a[0], c1 = d.a[1], cid = d.a[2], ldl = d.a[3], ldp = d.a[4];
  const uint2 key = make_uint2((uint32_t)d.a[6], (uint32_t)d.a[7]);
  const int rows_per_task = max(d.a[8], 1);
  const uint32_t V = (uint32_t)d.a[9];
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  long long *ri = reinterpret_cast<long long *>(c.s.red + 16);
  for (int b = 0; b < B; ++b) {
    float v = -INFINITY;
    long long i = -1;
    const uint32_t row_base = (uint32_t)(b % rows_per_task) * V;
    for (int q = (c0 >> 2) + tid; q * 4 < c1; q += kConsumerThreads) {
      const uint4 r = philox4x32_10(make_uint4(0u, 0u, row_base + (uint32_t)q * 4u, 0u), key);
      const uint32_t rr[4] = {r.x, r.y, r.z, r.w};
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const int j = q * 4 + e;
        if (j >= c0 && j < c1) {
          const float noise = bf16_to_f(__float2bfloat16_rn(gumbel_noise(rr[e])));
          const float k = bf16_to_f(__float2bfloat16_rn(logit_value(&logits[(size_t)b * ldl + j]) + noise));
          sample_merge(v, i, k, (long long)j);
        }
      }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      const float v2 = __shfl_xor_sync(0xffffffffu, v, o);
      const long long i2 = __shfl_xor_sync(0xffffffffu, i, o);
      sample_merge(v, i, v2, i2);
    }
    if (lane == 0) {
      c.s.red[warp] = v;
      ri[warp] = i;
    }
    consumer_sync();
    if (tid == 0) {
      for (int w = 1; w < 8; ++w) sample_merge(v, i, c.s.red[w], ri[w]);
      pv[(size_t)b * ldp + cid] = __float2bfloat16_rn(v);
      pi[(size_t)b * ldp + cid] = i;
    }
    consumer_sync();
  }
}

static __device__ void run_sampling_reduce(const Ctx &c, const TaskDesc &d) {
  const int B = active_tokens(c.P);
  const __nv_bfloat16 *pv = reinterpret_cast<const __nv_bfloat16 *>(d.p[0]);
  const long long *pi = reinterpret_cast<const long long *>(d.p[1]);
  long long *out = reinterpret_cast<long long *>(d.p[2]);
  const int n = d.a[0], ldp = d.a[1];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  for (int b = warp; b < B; b += 8) {
    float v = -INFINITY;
    long long i = -1;
    for (int j = lane; j < n; j += 32)
      sample_merge(v, i, bf16_to_f(__ldcg(&pv[(size_t)b * ldp + j])), __ldcg(&pi[(size_t)b * ldp + j]));
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      const float v2 = __shfl_xor_sync(0xffffffffu, v, o);
      const long long i2 = __shfl_xor_sync(0xffffffffu, i, o);
      sample_merge(v, i, v2, i2);
    }
    if (lane == 0) out[b] = i < 0 ? 0 : i;
  }
}

static __device__ void run_argmax_partial(const Ctx &c, const TaskDesc &d) {
  const int B = active_tokens(c.P);
  const __nv_bfloat16 *logits = reinterpret_cast<const __nv_bfloat16 *>(d.p[0]);
  __nv_bfloat16 *pv = reinterpret_cast<__nv_bfloat16 *>(d.p[1]);
  long long *pi = reinterpret_cast<long long *>(d.p[2]);
  const int c0 = d.a[0], c1 = d.a[1], cid = d.a[2], ldl = d.a[3], ldp = d.a[4];
  // A warp per token, no barrier; eight columns a load where the row allows it.  What bounds it is the latency of a few loads in a
  // row: the form with one block-wide pass and two barriers per token took 116 us for 64 tokens x 1027 columns.
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  for (int b = warp; b < B; b += 8) {
    const __nv_bfloat16 *row = logits + (size_t)b * ldl;
    float v = -INFINITY;
    int i = 0x7fffffff;
    const auto take = [&](float x, int j) {
      if (x > v || (x == v && j < i)) { v = x; i = j; }
    };
    const int head = min(c1, c0 + (int)(((16u - (uint32_t)(reinterpret_cast<uintptr_t>(row + c0) & 15u)) & 15u) >> 1));
    const int vecs = (c1 - head) >> 3, tail = head + 8 * vecs;
    if (c0 + lane < head) take(bf16_to_f(__ldcg(row + c0 + lane)), c0 + lane);
    const uint4 *src = reinterpret_cast<const uint4 *>(row + head);
#pragma unroll 4
    for (int k = lane; k < vecs; k += 32) {
      const uint4 x = __ldcg(src + k);
      const uint32_t w[4] = {x.x, x.y, x.z, x.w};
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        take(bf16_lo(w[q]), head + 8 * k + 2 * q);
        take(bf16_hi(w[q]), head + 8 * k + 2 * q + 1);
      }
    }
    if (tail + lane < c1) take(bf16_to_f(__ldcg(row + tail + lane)), tail + lane);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      const float v2 = __shfl_xor_sync(0xffffffffu, v, o);
      const int i2 = __shfl_xor_sync(0xffffffffu, i, o);
      take(v2, i2);
    }
    if (lane == 0) {
      pv[(size_t)b * ldp + cid] = __float2bfloat16_rn(v);
      pi[(size_t)b * ldp + cid] = i == 0x7fffffff ? 0x7fffffffffffffffLL : (long long)i;
    }
  }
}

static __device__ void run_argmax_reduce(const Ctx &c, const TaskDesc &d) {
  const int B = active_tokens(c.P);
  const __nv_bfloat16 *pv = reinterpret_cast<const __nv_bfloat16 *>(d.p[0]);
  const long long *pi = reinterpret_cast<const long long *>(d.p[1]);
  long long *out = reinterpret_cast<long long *>(d.p[2]);
  const int n = d.a[0], ldp = d.a[1];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  for (int b = warp; b < B; b += 8) {
    float v = -INFINITY;
    long long i = 0x7fffffffffffffffLL;
    for (int j = lane; j < n; j += 32)
      argmax_merge(v, i, bf16_to_f(__ldcg(&pv[(size_t)b * ldp + j])), __ldcg(&pi[(size_t)b * ldp + j]));
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      const float v2 = __shfl_xor_sync(0xffffffffu, v, o);
      const long long i2 = __shfl_xor_sync(0xffffffffu, i, o);
      argmax_merge(v, i, v2, i2);
    }
    if (lane == 0) out[b] = i;
  }
}

// Argmax over a vocabulary sharded across the ranks.  Warp b merges this rank's partials of token b, then lane r
// exchanges with rank r: it stores this rank's {value | seq} and {index | seq} 64-bit words into rank r's inbox and
// polls, in its own inbox, for the pair rank r pushed; the warp then takes the best pair (largest value, lowest index).
// Every rank sees the same pairs and writes the same id.
__device__ __forceinline__ void run_argmax_exchange(const Ctx &c, const TaskDesc &d) {
  const KernelParams &P = c.P;
  const int B = active_tokens(P);
  const __nv_bfloat16 *pv = reinterpret_cast<const __nv_bfloat16 *>(d.p[0]);
  const long long *pi = reinterpret_cast<const long long *>(d.p[1]);
  long long *out = reinterpret_cast<long long *>(d.p[2]);
  const int n = d.a[0], ldp = d.a[1], W = P.world_size, mbt = P.max_num_batched_tokens;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const unsigned long long inst = c.iteration * (unsigned)d.a[L_NAR] + (unsigned)d.a[L_ARIDX];
  const unsigned long long seq = (unsigned long long)ll_seq(c.iteration, d.a[L_NAR], d.a[L_ARIDX]);
  const size_t area = (size_t)d.p[5] + (size_t)(inst & 1ull) * (size_t)d.a[L_PARSTRIDE];   // in 32-bit words
  for (int b = warp; b < B; b += 8) {
    float v = -INFINITY;
    long long i = 0x7fffffffffffffffLL;
    for (int j = lane; j < n; j += 32)
      argmax_merge(v, i, bf16_to_f(__ldcg(&pv[(size_t)b * ldp + j])), __ldcg(&pi[(size_t)b * ldp + j]));
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      const float v2 = __shfl_xor_sync(0xffffffffu, v, o);
      const long long i2 = __shfl_xor_sync(0xffffffffu, i, o);
      argmax_merge(v, i, v2, i2);
    }
    i += (long long)d.a[2];   // column of the whole vocabulary (all lanes hold the merged pair)
    float rv = -INFINITY;
    long long ri = 0x7fffffffffffffffLL;
    if (lane < W) {
      const size_t slot = ((size_t)P.rank * mbt + b) * 4;
      unsigned long long *dst = reinterpret_cast<unsigned long long *>(reinterpret_cast<uint32_t *>(P.peer_inbox[lane]) + area + slot);
      const unsigned long long w0 = (unsigned long long)__float_as_uint(v) | (seq << 32);
      const unsigned long long w1 = ((unsigned long long)i & 0xffffffffull) | (seq << 32);
      asm volatile("st.relaxed.sys.global.v2.u64 [%0], {%1, %2};" ::"l"(dst), "l"(w0), "l"(w1) : "memory");
      const unsigned long long *src = reinterpret_cast<const unsigned long long *>(
          reinterpret_cast<const uint32_t *>(P.peer_inbox[P.rank]) + area + ((size_t)lane * mbt + b) * 4);
      uint32_t polls = 0;
      while (true) {
        unsigned long long a0, a1;
        asm volatile("ld.relaxed.sys.global.v2.u64 {%0, %1}, [%2];" : "=l"(a0), "=l"(a1) : "l"(src) : "memory");
        if ((a0 >> 32) == seq && (a1 >> 32) == seq) {
          rv = __uint_as_float((uint32_t)a0);
          ri = (long long)(a1 & 0xffffffffull);
          break;
        }
        if ((++polls & 0xff) == 0) {
          if (ld_volatile_i32(&P.status->error) != 0) break;
          if (globaltimer_ns() > c.deadline_ns) {
            report_timeout(P.status, c.worker, 3, lane);
            break;
          }
        }
      }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      const float v2 = __shfl_xor_sync(0xffffffffu, rv, o);
      const long long i2 = __shfl_xor_sync(0xffffffffu, ri, o);
      argmax_merge(rv, ri, v2, i2);
    }
    if (lane == 0) out[b] = ri;
  }
}

// Sum the per-rank fp32 inbox slots in rank order (+ residual) -> bf16.
static __device__ void run_allreduce(const Ctx &c, const TaskDesc &d) {
  const KernelParams &P = c.P;
  const int B = active_tokens(P);
  const int c0 = d.a[0], c1 = d.a[1], world = d.a[2], slot = d.a[3], ldo = d.a[4], ldr = d.a[5], N = d.a[6];
  const size_t parity = (size_t)((c.iteration * (unsigned)d.a[8] + (unsigned)d.a[7]) & 1ull);
  const float *inbox = P.peer_inbox[P.rank] + (size_t)d.p[0] + parity * (size_t)d.a[9];
  const __nv_bfloat16 *res = reinterpret_cast<const __nv_bfloat16 *>(d.p[1]);
  __nv_bfloat16 *out = reinterpret_cast<__nv_bfloat16 *>(d.p[2]);
  const int w = c1 - c0;
  for (int idx = threadIdx.x; idx < B * w; idx += kConsumerThreads) {
    const int b = idx / w, j = c0 + (idx - b * w);
    float v = 0.f;
    for (int r = 0; r < world; ++r) v += __ldcg(&inbox[(size_t)r * slot + (size_t)b * N + j]);
    if (res) v += bf16_to_f(__ldcg(&res[(size_t)b * ldr + j]));
    out[(size_t)b * ldo + j] = __float2bfloat16_rn(v);
  }
}

// Push stage of an unfused allreduce: columns [c0, c1) of a local bf16 tensor go, as fp32, into this rank's slot of
// every rank's inbox; the task's event is incremented on every rank once the stores are ordered (TF_REMOTE_TRIGGER).
static __device__ void run_ar_push(const Ctx &c, const TaskDesc &d) {
  const KernelParams &P = c.P;
  const int B = active_tokens(P);
  const int c0 = d.a[0], c1 = d.a[1], ldx = d.a[2], slot = d.a[3], N = d.a[6];
  const size_t parity = (size_t)((c.iteration * (unsigned)d.a[8] + (unsigned)d.a[7]) & 1ull);
  const size_t base = (size_t)d.p[5] + parity * (size_t)d.a[9] + (size_t)P.rank * (size_t)slot;
  const __nv_bfloat16 *x = reinterpret_cast<const __nv_bfloat16 *>(d.p[0]);
  const int w = c1 - c0;
  for (int idx = threadIdx.x; idx < B * w; idx += kConsumerThreads) {
    const int b = idx / w, j = c0 + (idx - b * w);
    const float v = bf16_to_f(__ldcg(&x[(size_t)b * ldx + j]));
    for (int peer = 0; peer < P.world_size; ++peer) P.peer_inbox[peer][base + (size_t)b * N + j] = v;
  }
}

// ---------------------------------------------------------------------------
// TASK_BATCH: device-side continuous batching, block-parallel.
// Same result, array by array, as the reference's single-threaded
// prepare_next_batch (include/mirage/persistent_kernel/persistent_kernel.cuh:206-368).
// Two additions:
//   * every live request owns a recurrent-state slot (M.state_slots[batch slot]): the lowest free one when it is
//     admitted, kept while the batch is compacted around it, free again when it retires;
//   * online mode (M.request_ctl given): rows of the token table are requests the host posts, extends and closes
//     while the loop runs (REQ_* in runtime_types.h), admitted in row order; a request advances no further than the
//     tokens the host has supplied (REQ_HOLD) or decodes on its own (REQ_RUN), and never further than the free pages.
// ---------------------------------------------------------------------------
static __device__ __noinline__ void run_batch(const Ctx c) {
  if (c.tmem_base & 0x80000000u) {   // called for TASK_ARGMAX_EXCHANGE (see task_other)
    run_argmax_exchange(c, c.s.desc[c.tmem_base & 1u]);
    return;
  }
  const KernelParams &P = c.P;
  const BatchMeta &M = P.meta;
  const int tid = threadIdx.x;
  const int mbr = P.max_num_batched_requests, mbt = P.max_num_batched_tokens;
  const int PS = P.page_size, S = P.max_seq_length, MP = P.max_num_pages;
  int *sm = reinterpret_cast<int *>(c.s.xtile);
  int *s_rid = sm;                 // [mbr]  request id per old slot (-1 when empty or retired)
  int *s_kv = s_rid + mbr;         // [mbr+1] old kv indptr
  int *s_step = s_kv + mbr + 1;    // [mbr]  updated step
  int *s_plen = s_step + mbr;      // [mbr]
  int *s_free = s_plen + mbr;      // [mbr+1] pages freed (then exclusive prefix)
  int *n_rid = s_free + mbr + 1;   // [mbr]  new slot -> request id
  int *n_tok = n_rid + mbr;        // [mbr+1] new qo indptr
  int *n_pg = n_tok + mbr + 1;     // [mbr+1] new kv indptr
  int *n_old = n_pg + mbr + 1;     // [mbr]  pages carried over
  int *n_src = n_old + mbr;        // [mbr]  old kv offset of carried pages
  int *n_newoff = n_src + mbr;     // [mbr]  offset into freshly allocated pages
  int *n_step = n_newoff + mbr;    // [mbr]  token read offset in `tokens`
  int *s_slot = n_step + mbr;      // [mbr]  state slot per old batch slot
  int *n_slot = s_slot + mbr;      // [mbr]  state slot per new batch slot
  int *s_used = n_slot + mbr;      // [mbr]  state slot taken
  int *sc = s_used + mbr;          // scalars: [0] head [1] tail [2] next_req [3] num_reqs [4] num_tokens [5] num_pages
  int *s_ctl = sc + 16;            // [total_num_requests] online mode: control word | live << 8
  const bool online = M.request_ctl != nullptr;
  const int R = P.total_num_requests;

  const int prev_tokens = M.qo_indptr[mbr];   // active tokens of the previous iteration (0 after a reset)
  if (tid < 3) sc[tid] = M.sched_scalars[tid];
  for (int i = tid; i <= mbr; i += kConsumerThreads) s_kv[i] = M.paged_kv_indptr[i];
  for (int i = tid; i < mbr; i += kConsumerThreads) {
    s_slot[i] = M.state_slots[i];
    s_used[i] = 0;
  }
  if (online)
    for (int r = tid; r < R; r += kConsumerThreads) s_ctl[r] = (M.request_ctl[r] & 0xff) | (M.request_ctl[R + r] ? 0x100 : 0);
  consumer_sync();
  // Step 1: commit outputs, advance steps, retire finished requests.
  // s_rid: request id, -1 for an empty slot, -2 for a request retired in this step.
  for (int i = tid; i < mbr; i += kConsumerThreads) {
    int rid = M.request_ids[i];
    int freed = 0, step_new = 0, plen = 0;
    if (rid != -1) {
      const int step = M.step[rid];
      const int qo = M.qo_indptr[i];
      const int n = M.qo_indptr[i + 1] - qo;
      plen = M.prompt_lengths[rid];
      for (int j = 0; j < n; ++j)
        if (step + j + 1 >= plen && step + j + 1 < S)
          M.tokens[(size_t)rid * S + step + j + 1] = M.output_tokens[qo + j];
      step_new = step + n;
      M.step[rid] = step_new;
      bool done = (step_new + 1 >= S) ||
                  (M.tokens[(size_t)rid * S + step_new] == P.eos_token_id && step_new >= plen);
      if (online) {
        const int ctl = s_ctl[rid] & 0xff;
        if (ctl == REQ_HOLD) done = false;
        else if (ctl == REQ_CLOSE) done = step_new >= plen;
        if (done) {
          s_ctl[rid] = 0;
          M.request_ctl[rid] = REQ_FREE;
          M.request_ctl[R + rid] = 0;
        }
      }
      if (done) {
        freed = s_kv[i + 1] - s_kv[i];
        rid = -2;
      }
    }
    s_free[i] = freed;
    s_rid[i] = rid;
    s_step[i] = step_new;
    s_plen[i] = plen;
  }
  consumer_sync();
  if (tid == 0) {
    int acc = 0;
    for (int i = 0; i < mbr; ++i) {
      const int f = s_free[i];
      s_free[i] = acc;
      acc += f;
    }
    s_free[mbr] = acc;
  }
  consumer_sync();
  for (int i = 0; i < mbr; ++i) {
    if (s_rid[i] != -2) continue;
    const int cnt = s_free[i + 1] - s_free[i];
    for (int j = tid; j < cnt; j += kConsumerThreads)
      M.page_queue[(unsigned)(sc[1] + s_free[i] + j) % (unsigned)MP] = M.paged_kv_indices[s_kv[i] + j];
  }
  // Step 2: snapshot of the page table (compaction below may overlap its source).
  for (int i = tid; i < s_kv[mbr]; i += kConsumerThreads) M.paged_kv_indices_snapshot[i] = M.paged_kv_indices[i];
  consumer_sync();
  // Step 3: lay out the next batch (serial over slots, all operands in shared memory).
  if (tid == 0) {
    int num_reqs = 0, num_tokens = 0, num_pages = 0, new_pages = 0;
    int head = sc[0];
    const int avail = sc[1] + s_free[mbr] - head;   // free pages
    for (int i = 0; i < mbr; ++i) {
      const int rid = s_rid[i];
      if (rid < 0) continue;
      const int step = s_step[i];
      int nn = s_plen[i] - step;
      nn = (nn > 0) ? min(nn, mbt - num_tokens) : min(1, mbt - num_tokens);
      const int n_old_pages = s_kv[i + 1] - s_kv[i];
      if (online) {
        if (s_plen[i] <= step && (s_ctl[rid] & 0xff) != REQ_RUN) nn = 0;
        nn = max(0, min(nn, (n_old_pages + avail - new_pages) * PS - step));
      }
      n_slot[num_reqs] = s_slot[i];
      if ((unsigned)s_slot[i] < (unsigned)mbr) s_used[s_slot[i]] = 1;
      const int np = (step + nn + PS - 1) / PS;
      n_rid[num_reqs] = rid;
      n_tok[num_reqs] = num_tokens;
      n_pg[num_reqs] = num_pages;
      n_old[num_reqs] = n_old_pages;
      n_src[num_reqs] = s_kv[i];
      n_newoff[num_reqs] = new_pages;
      n_step[num_reqs] = step;
      new_pages += max(np - n_old_pages, 0);
      num_pages += np;
      num_tokens += nn;
      ++num_reqs;
    }
    int next = online ? 0 : sc[2], slot = 0;
    while (num_reqs < mbr && num_tokens < mbt && next < P.total_num_requests) {
      int nn = mbt - num_tokens;
      if (online) {
        const int ctl = s_ctl[next];
        if (ctl != REQ_RUN && ctl != REQ_HOLD && ctl != REQ_CLOSE) { ++next; continue; }   // free row, or live already
        nn = min(nn, (avail - new_pages) * PS);
        if (nn <= 0) break;
        M.step[next] = 0;
        M.request_ctl[R + next] = 1;
      }
      nn = min(M.prompt_lengths[next], nn);
      const int np = (nn + PS - 1) / PS;
      while (slot < mbr - 1 && s_used[slot]) ++slot;
      s_used[slot] = 1;
      n_slot[num_reqs] = slot;
      n_rid[num_reqs] = next;
      n_tok[num_reqs] = num_tokens;
      n_pg[num_reqs] = num_pages;
      n_old[num_reqs] = 0;
      n_src[num_reqs] = 0;
      n_newoff[num_reqs] = new_pages;
      n_step[num_reqs] = 0;
      new_pages += np;
      num_pages += np;
      num_tokens += nn;
      ++num_reqs;
      ++next;
    }
    n_tok[num_reqs] = num_tokens;
    n_pg[num_reqs] = num_pages;
    sc[3] = num_reqs;
    sc[4] = num_tokens;
    sc[5] = num_pages;
    sc[6] = head;              // ring position of the first fresh page
    sc[0] = head + new_pages;
    sc[1] = sc[1] + s_free[mbr];
    sc[2] = online ? 0 : next;
  }
  consumer_sync();
  const int num_reqs = sc[3], num_tokens = sc[4], num_pages = sc[5], head0 = sc[6];
  // Step 4: write the batch description.
  for (int k = 0; k < num_reqs; ++k) {
    const int rid = n_rid[k];
    const int nn = n_tok[k + 1] - n_tok[k];
    const int np = n_pg[k + 1] - n_pg[k];
    for (int j = tid; j < nn; j += kConsumerThreads)
      M.input_tokens[n_tok[k] + j] = M.tokens[(size_t)rid * S + n_step[k] + j];
    for (int j = tid; j < np; j += kConsumerThreads) {
      int pg;
      if (j < n_old[k]) pg = M.paged_kv_indices_snapshot[n_src[k] + j];
      else pg = M.page_queue[(unsigned)(head0 + n_newoff[k] + (j - n_old[k])) % (unsigned)MP];
      M.paged_kv_indices[n_pg[k] + j] = pg;
    }
  }
  for (int k = tid; k < mbr; k += kConsumerThreads) {
    if (k < num_reqs) {
      M.request_ids[k] = n_rid[k];
      M.state_slots[k] = n_slot[k];
      M.qo_indptr[k] = n_tok[k];
      M.paged_kv_indptr[k] = n_pg[k];
      const int tot = n_step[k] + (n_tok[k + 1] - n_tok[k]);
      const int lpl = tot % PS;
      M.paged_kv_last_page_len[k] = (lpl == 0) ? PS : lpl;
    } else {
      M.request_ids[k] = -1;
      M.qo_indptr[k] = num_tokens;
      M.paged_kv_indptr[k] = num_pages;
    }
  }
  if (P.world_size > 1 && P.ll_row_words > 0 && num_tokens < prev_tokens) {
    // token rows that go idle: no sequence number may survive in them (see ll_seq)
    uint32_t *inbox = reinterpret_cast<uint32_t *>(P.peer_inbox[P.rank]);
    const size_t N = (size_t)P.ll_row_words, span = (size_t)(prev_tokens - num_tokens) * N;
    for (int buf = 0; buf < 2; ++buf)
      for (int r = 0; r < P.world_size; ++r) {
        uint32_t *rows = inbox + (size_t)buf * (size_t)P.ll_buffer_words + ((size_t)r * mbt + (size_t)num_tokens) * N;
        for (size_t i = tid; i < span; i += kConsumerThreads) rows[i] = 0u;
      }
  }
  if (tid == 0) {
    M.qo_indptr[mbr] = num_tokens;
    M.paged_kv_indptr[mbr] = num_pages;
    M.sched_scalars[0] = sc[0];
    M.sched_scalars[1] = sc[1];
    M.sched_scalars[2] = sc[2];
    P.status->active_tokens = num_tokens;
    P.status->all_done = (num_tokens == 0) ? 1 : 0;
  }
}

}  // namespace mpk

#include "hybrid_tasks.cuh"

namespace mpk {

// ---------------------------------------------------------------------------
// compute warps: walk the task list
// ---------------------------------------------------------------------------
struct TaskTimes {   // profiler timestamps of the running task (thread 0 only)
  uint64_t begin_ns, ready_ns;
  bool on;
};

// Thread 0 acquire-polls the task's event counters, then the compute warps meet.  Returns false when
// the launch is being abandoned.
__device__ __forceinline__ bool wait_dependencies(const Ctx &c, const TaskDesc &d, int t, bool ok, TaskTimes &tt) {
  const KernelParams &P = c.P;
  if (threadIdx.x == 0) {
    if (tt.on) tt.begin_ns = globaltimer_ns();
    bool good = ok;
    for (int i = 0; i < kMaxDeps && good; ++i) {
      const int ev = d.dep_event[i];
      if (ev < 0) continue;
      good = wait_counter(c, &P.counters[ev], (unsigned long long)d.dep_need[i] * c.iteration,
                          (d.flags & (TF_DEP0_REMOTE << i)) != 0, 1, t);
    }
    if (!good) c.s.flags[0] = 1;
    if (tt.on) tt.ready_ns = globaltimer_ns();
  }
  consumer_sync();
  return c.s.flags[0] == 0;
}

// Each task kind has its own non-inlined runner so that register allocation of the heavy bodies
// (attention) does not leak into the weight-streaming loop.
template <bool GENERAL, bool TPX, int HYB>
__device__ __forceinline__ bool task_linear(const Ctx &c, const TaskDesc &d, int t, bool ok, TaskTimes &tt,
                                         LinearState &ls) {
  const int tid = threadIdx.x;
  // constants the prologue needs are fetched before the dependency wait
  uint4 gpre[2] = {make_uint4(0, 0, 0, 0), make_uint4(0, 0, 0, 0)};
  if (GENERAL && (d.flags & TF_TC) && !(d.flags & TF_FP8)) {
    fence_proxy_async_smem();   // the tile area was used by generic accesses; what comes next writes it by tensor-map copies
    ok = wait_dependencies(c, d, t, ok, tt);
    ls = run_linear_tc<HYB>(c, d, ls, t, ok);
    return ok;
  }
  if (d.a[L_PRO] == PRO_RMSNORM) {
    const uint4 *gam = reinterpret_cast<const uint4 *>(d.p[4]);
    const int vecs = d.a[L_KT] / 8;
    if (tid < vecs) gpre[0] = __ldg(gam + tid);
    if (tid + kConsumerThreads < vecs) gpre[1] = __ldg(gam + tid + kConsumerThreads);
  }
  ok = wait_dependencies(c, d, t, ok, tt);
  // the weight chunks must be consumed even when the launch is being abandoned or no token is active
  if (GENERAL && !HYB && (d.flags & TF_TC) && (d.flags & TF_FP8)) run_linear_fp8_tc(c, d, ls, t, ok);
  else if (GENERAL && !HYB && (d.flags & TF_FP8)) run_linear_fp8(c, d, ls, t, ok);
  else run_linear<GENERAL, TPX, HYB>(c, d, ls, t, gpre, ok);
  return ok;
}

template <bool GENERAL, bool EXACT>
__device__ __forceinline__ bool task_attention(const Ctx &c, const TaskDesc &d, int t, bool ok, TaskTimes &tt) {
  const KernelParams &P = c.P;
  // the batch description must be final before the page table is read; that event fired long ago
  if (d.a[A_EARLY_EV] >= 0) {
    if (threadIdx.x == 0 && ok &&
        !wait_counter(c, &P.counters[d.a[A_EARLY_EV]], (unsigned long long)d.a[A_EARLY_NEED] * c.iteration,
                      false, 1, t))
      c.s.flags[0] = 1;
    consumer_sync();
    ok = ok && (c.s.flags[0] == 0);
  }
  if (GENERAL) {
    if (tt.on && threadIdx.x == 0) tt.begin_ns = globaltimer_ns();
    if (!ok) return false;
    ok = run_attention_flat<EXACT>(P, d, c.s.xtile, c.s.flags, c.iteration, c.deadline_ns, t);
    if (tt.on && threadIdx.x == 0) tt.ready_ns = *reinterpret_cast<volatile uint64_t *>(c.s.flags + 6);
    return ok;
  }
  AttnPre pre;
  pre.rv.nq = 0;
  if (ok) attention_prefetch(c, d, pre, t);
  if (threadIdx.x == 0) *reinterpret_cast<volatile int *>(&c.s.flags[2]) = 1;   // quiet the weight stream
  ok = wait_dependencies(c, d, t, ok, tt);
  if (ok) run_attention(c, d, pre, t);
  if (threadIdx.x == 0) *reinterpret_cast<volatile int *>(&c.s.flags[2]) = 0;
  return ok;
}

template <bool GENERAL, bool TPX, int HYB>
__device__ __forceinline__ bool task_other(const Ctx &c, const TaskDesc &d, int t, bool ok, TaskTimes &tt) {
  ok = wait_dependencies(c, d, t, ok, tt);
  if (!ok) return false;
  if (HYB) {
    run_hybrid_task<HYB>(c, d, t);
    return true;
  }
  switch (d.type) {
    // (the argmax exchange of multi-rank graphs shares the batching task's out-of-line function and its call site: a
    // second call in this switch moved the register allocation of the linear loop; bit 31 of the tensor-memory field,
    // never set in an address, says which body is meant and which descriptor slot holds the task)
    case TASK_ARGMAX_EXCHANGE: if (!TPX) break; [[fallthrough]];
    case TASK_BATCH: {
      Ctx cc = c;
      if (TPX && d.type == TASK_ARGMAX_EXCHANGE) cc.tmem_base = 0x80000000u | (&d == &c.s.desc[1] ? 1u : 0u);
      run_batch(cc);
      break;
    }
    case TASK_EMBED: run_embed(c, d); break;
    case TASK_RMSNORM: run_rmsnorm(c, d); break;
    case TASK_SILU_MUL: run_silu_mul(c, d); break;
    case TASK_ARGMAX_PARTIAL: run_argmax_partial(c, d); break;
    case TASK_ARGMAX_REDUCE: run_argmax_reduce(c, d); break;
    case TASK_ALLREDUCE: run_allreduce(c, d); break;
    case TASK_ELEMENTWISE_ADD: run_elementwise_add(c, d); break;
    case TASK_TENSOR_INIT: run_tensor_init(c, d); break;
    case TASK_QUANTIZE_FP8: if (GENERAL) run_quantize_fp8(c, d); break;
    case TASK_MOE_ROUTING: if (GENERAL) run_moe_routing(c, d); break;
    case TASK_MOE_SILU_MUL: if (GENERAL) run_moe_silu_mul(c, d); break;
    case TASK_MOE_MUL_SUM_ADD: if (GENERAL) run_moe_mul_sum_add(c, d); break;
    case TASK_MLA_APPEND: if (GENERAL) run_mla_append(c, d); break;
    case TASK_MLA_DECODE: if (GENERAL) run_mla_decode(c, d); break;
    case TASK_MLA_REDUCE: if (GENERAL) run_mla_reduce(c, d); break;
    case TASK_SAMPLING_PARTIAL: if (GENERAL) run_sampling_partial<__nv_bfloat16>(c, d); break;
    case TASK_SAMPLING_REDUCE: if (GENERAL) run_sampling_reduce(c, d); break;
    case TASK_AR_PUSH: if (GENERAL && TPX) run_ar_push(c, d); break;
    default: break;
  }
  return true;
}

template <bool GENERAL, bool TPX, int HYB, bool EXACT>
__device__ void consumer_loop(const Ctx &c, int t_begin, int t_end) {
  const KernelParams &P = c.P;
  const int tid = threadIdx.x;
  LinearState ls{0, 0u, 0u};
  if (t_begin < t_end && tid < kDescVecs)
    reinterpret_cast<uint4 *>(&c.s.desc[0])[tid] = __ldg(reinterpret_cast<const uint4 *>(&P.tasks[t_begin]) + tid);
  consumer_sync();
  bool ok = true;
  for (int t = t_begin; t < t_end; ++t) {
    const TaskDesc &d = c.s.desc[(t - t_begin) & 1];
    uint4 nxt = make_uint4(0, 0, 0, 0);
    const bool fetch = (t + 1 < t_end) && tid >= 224 && tid < 224 + kDescVecs;
    if (fetch) nxt = __ldg(reinterpret_cast<const uint4 *>(&P.tasks[t + 1]) + (tid - 224));
    TaskTimes tt{0, 0, (P.profiler != nullptr) && (uint64_t)(t + 1) * 8 <= P.profiler_entries};
    const uint32_t type = d.type;
    if (HYB != HYB_F32 && type == TASK_LINEAR) ok = task_linear<GENERAL, TPX, HYB>(c, d, t, ok, tt, ls);
    else if (HYB == HYB_BF16 && type == TASK_MOE_GEMM) {
      ok = wait_dependencies(c, d, t, ok, tt);
      ls = run_moe_gemm_hybrid<GENERAL>(c, d, ls, t, ok);
    } else if (GENERAL && !HYB && type == TASK_MOE_GEMM) {
      ok = wait_dependencies(c, d, t, ok, tt);
      ls = run_moe_gemm_decoder(c, d, ls, t, ok);
    } else if (!HYB && type == TASK_ATTENTION) ok = task_attention<GENERAL, EXACT>(c, d, t, ok, tt);
    else ok = task_other<GENERAL, TPX, HYB>(c, d, t, ok, tt);
    if (fetch) reinterpret_cast<uint4 *>(&c.s.desc[(t + 1 - t_begin) & 1])[tid - 224] = nxt;
    const int trig = d.trig_event;
    const uint32_t tflags = d.flags;
    consumer_sync();
    ok = ok && (c.s.flags[0] == 0);
    if (!ok) break;
    if (tid == 0 && tt.on) {
      // per task: [wait begin, dependencies satisfied, body end, worker << 40 | event << 8 | type]  (globaltimer ns)
      uint64_t *rec = P.profiler + (size_t)t * 8;
      rec[0] = tt.begin_ns;
      rec[1] = tt.ready_ns;
      rec[2] = globaltimer_ns();
      rec[3] = ((uint64_t)c.worker << 40) | ((uint64_t)(uint32_t)trig << 8) | (uint64_t)type;
    }
    if (tid == 0 && trig >= 0) {
      // red.release orders this CTA's writes (observed through the barrier above) before the increment
      if (tflags & TF_REMOTE_TRIGGER) {
        // one system-scope fence orders the pushed partial sums before the counter increments; the increments
        // themselves are relaxed so that they travel to all peers concurrently instead of one round trip each
        __threadfence_system();
        for (int r = 0; r < P.world_size; ++r) red_relaxed_sys(&P.peer_counters[r][trig], 1ull);
      } else {
        red_release_gpu(&P.counters[trig], 1ull);
      }
    }
  }
}

// Two instantiations: GENERAL = false is the batch-1 product path (bf16 weights, at most 8 batched tokens),
// kept free of every other task body so that its register allocation at the 168-register cap stays as tuned;
// GENERAL = true adds FP8 tasks and linear tasks for up to 64 tokens.  The host picks by graph content.
// TPX marks the instantiations that graphs of more than one rank run.  Code written for tensor parallelism after the
// single-GPU paths had been tuned sits behind it -- the allreduce prologue with all ranks' loads in flight (batch-1
// kernel), the argmax exchange of a sharded lm_head -- so that the single-GPU instantiations <*, false> stay exactly
// the code that was measured: both run at the register cap, where unrelated code moves their allocation.
// HYB marks the instantiations of graphs with recurrent or extended-attention layers (hybrid_tasks.cuh): they hold the
// linear bodies and the hybrid tasks only.  HYB_BF16 serves in bf16; HYB_F32 computes everything in 32-bit floats and has
// no tensor-core code at all.
// EXACT marks the general instantiation of graphs of up to 8 tokens that the batch-1 one would run too: its attention keeps the softmax weights as two bf16.
// (A flag in the loop instead cost the graphs without it 290 bytes of spills: 64 requests 7.79 -> 8.42 ms.)
template <bool GENERAL, bool TPX = false, int HYB = 0, bool EXACT = false>
__global__ void __launch_bounds__(block_threads(GENERAL), 1) mpk_megakernel(const __grid_constant__ KernelParams P) {
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  Smem s = carve(smem_raw, P);
  const int tid = threadIdx.x;
  const unsigned long long iteration = *reinterpret_cast<volatile unsigned long long *>(&P.status->iteration) + 1ull;
  if (tid == 0) {
    if (blockIdx.x == 0) P.status->t_start[iteration & 7] = globaltimer_ns();
    for (int i = 0; i < P.num_stages; ++i) {
      mbar_init(&s.full[i], 1);
      mbar_init(&s.empty[i], 8);
    }
    s.flags[0] = 0;
    s.flags[1] = 0;
    s.flags[2] = 0;
    s.flags[3] = 0;   // (run_linear_tc)
    if (!GENERAL) *reinterpret_cast<volatile int *>(&s.full[8]) = -1;   // attention stash: empty
    if (GENERAL) {
      mbar_init(s.acc_bar, 8);   // one tcgen05.commit per compute warp
      for (int i = 0; i < 8; ++i) s.flags[16 + 16 * kAttnStages + i] = 0;
      if (P.attn_table_bytes) *reinterpret_cast<int *>(reinterpret_cast<uint8_t *>(s.flags) - kFlagsOffset + kMiscBytes) = -1;   // the request table: not built
    }
    mbar_fence_init();
  }
  if (GENERAL && tid >= 64 && tid < 128) {   // (one thread for all of them: 1 us of every launch)
    const int i = tid - 64;
    if (i < 8 * kAttnStages) mbar_init(reinterpret_cast<uint64_t *>(s.flags + 16) + i, 1);
    if (i < 33) mbar_init(s.full + kXBarsOffset / 8 + i, i < 8 ? 1 : i < 16 ? kXIssuers : i >= 24 && i < 32 ? 8 : 1);
    mbar_fence_init();
  }
  // graphs with tcgen05 tasks: warp 0 takes all 512 tensor-memory columns (one CTA per SM, so nothing else asks)
  const bool use_tmem = GENERAL && P.use_tmem != 0;
  if (use_tmem && tid < 32) tmem_alloc(s.tmem_holder, kTmemCols);
  if (use_tmem) tc_fence_before_sync();
  __syncthreads();
  if (use_tmem) tc_fence_after_sync();
  Ctx c{P, s, iteration, globaltimer_ns() + (uint64_t)P.spin_limit * 1000000ull, (int)blockIdx.x,
        use_tmem ? *reinterpret_cast<volatile uint32_t *>(s.tmem_holder) : 0u};
  const int t_begin = P.worker_begin[blockIdx.x], t_end = P.worker_begin[blockIdx.x + 1];
  if (tid >= kConsumerThreads) {
    if (GENERAL) asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(kStreamerRegs));
    if (GENERAL && P.borrow) {
      if ((tid & 31) == 0) stream_borrowing(c, t_begin, t_end);
      __syncwarp();
    } else if (tid < kConsumerThreads + 32) {
      streamer_loop<GENERAL, HYB>(c, t_begin, t_end);
    }
  } else {
    if (GENERAL) asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(kConsumerRegs));
    consumer_loop<GENERAL, TPX, HYB, EXACT>(c, t_begin, t_end);
  }
  if (use_tmem) tc_fence_before_sync();
  __syncthreads();
  if (use_tmem && tid < 32) {
    // Every exit path of both loops ends here.  MMAs still in flight after an abandoned launch must finish before
    // the columns are freed: one more commit, awaited with a bounded number of polls.
    tc_fence_after_sync();
    if (tid == 0 && s.flags[0] != 0) {
      // parity is unknown after an abort: a fresh barrier in the (now idle) full-barrier array
      mbar_init(&s.full[15], 1);
      mbar_fence_init();
      umma_commit(&s.full[15]);
      uint32_t polls = 0;
      while (!mbar_try_wait(&s.full[15], 0u) && ++polls < (1u << 22)) {}
    }
    __syncwarp();
    tmem_dealloc(c.tmem_base, kTmemCols);
  }
  if (tid == 0) {
    __threadfence();
    const unsigned int ticket = atomicAdd(&P.status->exit_ticket, 1u);
    if (ticket == gridDim.x - 1) {
      P.status->exit_ticket = 0;
      P.status->t_end[iteration & 7] = globaltimer_ns();
      P.status->iteration = iteration;
      __threadfence();
    }
  }
}

}  // namespace mpk

