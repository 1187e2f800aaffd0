// Triangular solve of one level of ILU factors by dataflow inside a CTA: one
// CTA per subdomain, warps that work on several dependency levels at once.
//
//   lower:  y_r = rhs_r - sum_j L_rj y_j               (unit diagonal)
//   upper:  x_r = (y_r - sum_j U_rj x_j) * dinv_r     (dinv = inverse diagonal)
// as IluClass::SolveHost (ParGeMSLR SRC/preconditioners/ilu.cpp:3677-3790),
// rows in the level-set order of IluClass::BuildLevels (ilu.cpp:832-1062).
//
// What bounds it is the chain of dependency levels (2015 at 64^3, some 20
// rows wide), not the factor's bytes.  In these factors only 7-8% of a row's
// entries (a third in 2D) have their source in the level before, so most of
// a row's sum need not wait for the chain:
//   - a task is at most 32 rows of one level, one row a lane, no shuffles;
//     task t belongs to warp t % W, so W tasks of successive levels are in
//     hand at once, each summing its old entries while the chain runs below;
//   - entries are laid out oldest first, four to a quad (two loads), right-
//     aligned, so that only a row's last quads can touch tasks in flight;
//   - results sit in a shared-memory ring by schedule position.  A slot not
//     solved yet holds a signalling NaN, so a consumer polls the value itself:
//     one store and one load a level.  (A progress counter beside the value
//     took 270 ns a level where this takes 130 to 160, with or without its
//     fences; a CTA barrier a level took 600-900.)
//   - one more warp streams the factor into shared memory by bulk copies.
// On a B200, level 0 of the 7-point Laplacian at 64^3 (ILUT 1e-3), lower /
// upper pass: 0.32 / 0.30 ms mixed and 0.50 / 0.47 ms FP64, one lane (one
// barrier a level: 1.30 / 1.19 and 1.64 / 1.52 ms); 0.51 / 0.46 ms for four
// lanes mixed.  At 128^3, mixed: 2.1 / 1.9 ms one lane (6.04 / 5.76), 4.7 /
// 4.1 ms four lanes.
#pragma once

#include "pgx_device.cuh"
#include "pgx_flow_pack.h"

namespace pgx {

constexpr int kFlowPolls = 1 << 23;      // bound of a wait, in polls

struct FlowArgs {
  int n;                    // rows; also the length of the slot vector
  const int4* chunk;        // {first 16-byte unit, 16-byte units, tasks, 0}
  const int* comp_chunk0;   // ncomp + 1
  const int2* first;        // ncomp x W: chunk (within the subdomain) and header offset of each warp's first task
  const unsigned char* blob;
};

__device__ __forceinline__ unsigned flow_ld(const unsigned* p) {
  unsigned v;
  asm volatile("ld.acquire.cta.shared::cta.u32 %0, [%1];" : "=r"(v) : "r"(smem_u32(p)) : "memory");
  return v;
}
__device__ __forceinline__ void flow_st(unsigned* p, unsigned v) {
  asm volatile("st.release.cta.shared::cta.u32 [%0], %1;" ::"r"(smem_u32(p)), "r"(v) : "memory");
}
__device__ __forceinline__ void flow_add(unsigned* p) {
  asm volatile("red.release.cta.shared::cta.add.u32 [%0], 1;" ::"r"(smem_u32(p)) : "memory");
}
// until every task below `lim` is done (bounded); task t belongs to warp t % W, prog[w] counts warp w's done tasks.
// A warp gives up as a whole: its lanes meet in votes and warp barriers again.  Returns prog[W] (0 if it gave up).
template <int W>
__device__ __forceinline__ unsigned flow_wait(unsigned* prog, int lim, int lane, int* err, unsigned* abort) {
  const unsigned need = lane < W && lim > lane ? (unsigned)(lim - lane + W - 1) / W : 0u;
  for (int k = 0;; k++) {
    const unsigned v = lane <= W ? flow_ld(&prog[lane]) : 0u;
    if (__all_sync(0xffffffffu, v >= need)) {
      __syncwarp();  // a vote orders no memory: the lanes that acquired hand over to the others here
      return __shfl_sync(0xffffffffu, v, W);
    }
    if ((k & 255) == 255) {
      if (k >= kFlowPolls) {
        atomicOr(err, kErrStage);
        *(volatile unsigned*)abort = 1u;
      }
      if (__any_sync(0xffffffffu, *(volatile unsigned*)abort != 0)) return 0u;
    }
  }
}

// Ring entries as 32-bit words; a slot not solved yet holds the sentinel in
// every word (4-byte types) or in the high word of every double.
template <typename T, int R>
union FlowVal {
  VecR<T, R> v;
  unsigned u[sizeof(T) * R / 4];
  __device__ FlowVal() {}
};
template <typename T>
constexpr bool kFlowWide = sizeof(typename Sc<T>::real) == 8;
constexpr unsigned kFlowS32 = 0xFFA0BEEFu, kFlowS64 = 0xFFF4DEADu;  // signalling NaNs: no operation returns them
template <typename T, int R>
__device__ __forceinline__ void flow_ring_load(FlowVal<T, R>& o, unsigned at) {
  constexpr int NW = sizeof(T) * R / 4;
  if constexpr (NW == 1) {
    asm volatile("ld.volatile.shared.b32 %0, [%1];" : "=r"(o.u[0]) : "r"(at) : "memory");
  } else if constexpr (NW == 2 && kFlowWide<T>) {
    unsigned long long q;
    asm volatile("ld.volatile.shared.b64 %0, [%1];" : "=l"(q) : "r"(at) : "memory");
    o.u[0] = (unsigned)q;
    o.u[1] = (unsigned)(q >> 32);
  } else if constexpr (NW == 2) {
    asm volatile("ld.volatile.shared.v2.b32 {%0, %1}, [%2];" : "=r"(o.u[0]), "=r"(o.u[1]) : "r"(at) : "memory");
  } else {
#pragma unroll
    for (int w = 0; w < NW; w += 4) {
      if constexpr (kFlowWide<T>) {
        unsigned long long q0, q1;
        asm volatile("ld.volatile.shared.v2.b64 {%0, %1}, [%2];" : "=l"(q0), "=l"(q1) : "r"(at + 4 * w) : "memory");
        o.u[w] = (unsigned)q0;
        o.u[w + 1] = (unsigned)(q0 >> 32);
        o.u[w + 2] = (unsigned)q1;
        o.u[w + 3] = (unsigned)(q1 >> 32);
      } else {
        asm volatile("ld.volatile.shared.v4.b32 {%0, %1, %2, %3}, [%4];"
                     : "=r"(o.u[w]), "=r"(o.u[w + 1]), "=r"(o.u[w + 2]), "=r"(o.u[w + 3])
                     : "r"(at + 4 * w)
                     : "memory");
      }
    }
  }
}
template <typename T, int R>
__device__ __forceinline__ void flow_ring_store(unsigned at, const FlowVal<T, R>& o) {
  constexpr int NW = sizeof(T) * R / 4;
  if constexpr (NW == 1) {
    asm volatile("st.volatile.shared.b32 [%0], %1;" ::"r"(at), "r"(o.u[0]) : "memory");
  } else if constexpr (NW == 2 && kFlowWide<T>) {
    asm volatile("st.volatile.shared.b64 [%0], %1;" ::"r"(at),
                 "l"((unsigned long long)o.u[0] | ((unsigned long long)o.u[1] << 32))
                 : "memory");
  } else if constexpr (NW == 2) {
    asm volatile("st.volatile.shared.v2.b32 [%0], {%1, %2};" ::"r"(at), "r"(o.u[0]), "r"(o.u[1]) : "memory");
  } else {
#pragma unroll
    for (int w = 0; w < NW; w += 4) {
      if constexpr (kFlowWide<T>)
        asm volatile("st.volatile.shared.v2.b64 [%0], {%1, %2};" ::"r"(at + 4 * w),
                     "l"((unsigned long long)o.u[w] | ((unsigned long long)o.u[w + 1] << 32)),
                     "l"((unsigned long long)o.u[w + 2] | ((unsigned long long)o.u[w + 3] << 32))
                     : "memory");
      else
        asm volatile("st.volatile.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(at + 4 * w), "r"(o.u[w]),
                     "r"(o.u[w + 1]), "r"(o.u[w + 2]), "r"(o.u[w + 3])
                     : "memory");
    }
  }
}
template <typename T, int R>
__device__ __forceinline__ bool flow_missing(const FlowVal<T, R>& o) {
  constexpr int NW = sizeof(T) * R / 4;
  bool m = false;
#pragma unroll
  for (int w = kFlowWide<T> ? 1 : 0; w < NW; w += kFlowWide<T> ? 2 : 1) m |= o.u[w] == (kFlowWide<T> ? kFlowS64 : kFlowS32);
  return m;
}

template <typename T>
struct FlowQuad {  // four entries of a row: ring positions and values
  uint2 c;
  T v[4];
};
template <typename T>
__device__ __forceinline__ FlowQuad<T> flow_load_quad(const unsigned char* cols, const unsigned char* vals, int k) {
  FlowQuad<T> q;
  q.c = *(const uint2*)(cols + (size_t)k * 8);
  if constexpr (sizeof(T) == 4) {
    const float4 f = *(const float4*)(vals + (size_t)k * 16);
    q.v[0] = f.x;
    q.v[1] = f.y;
    q.v[2] = f.z;
    q.v[3] = f.w;
  } else {
    const T* p = (const T*)(vals + (size_t)k * 4 * sizeof(T));
#pragma unroll
    for (int u = 0; u < 4; u++) q.v[u] = p[u];
  }
  return q;
}

// What the warps of a pass share beside the ring and the stages.
template <typename C>
struct FlowShared {
  unsigned long long full[C::stages];  // a chunk has landed
  unsigned prog[C::W + 1];  // tasks each warp has done; chunks whose copies are issued
  unsigned freed[C::stages], abort;
};

// Until chunk `ch` has landed (bounded); `issued`: the number of chunks that
// the warp knows to be issued.  The abort flag is looked at only where a wait
// does not end at once, and the count of issued chunks comes with the progress
// (flow_wait): both lie between a warp's tasks, which wait for little else
// where rows are short.  With a look at each once a task, B200: a 61x55x64
// imported application (FP64) 544 us, now 509; 256^2 FP64 solve 98.5 and 95.0
// ms; 64^3 mixed 84.0 and 82.9 ms.  Returns false, to every lane, when a wait gave up.
template <typename C>
__device__ __forceinline__ bool flow_chunk(FlowShared<C>& sh, int ch, unsigned& issued, int* err) {
  unsigned long long* const bar = &sh.full[ch % C::stages];
  const unsigned parity = (unsigned)((ch / C::stages) & 1);
  if (flow_issued(issued, ch) && __all_sync(0xffffffffu, mbar_try_wait(bar, parity))) return true;
  const long long t0 = clock64();
  for (;;) {
    if (!flow_issued(issued, ch)) {
      if (__all_sync(0xffffffffu, flow_issued(flow_ld(&sh.prog[C::W]), ch))) issued = (unsigned)ch + 1u;
    } else if (__all_sync(0xffffffffu, mbar_try_wait(bar, parity))) {
      return true;
    }
    const bool late = clock64() - t0 >= kMbarWaitCycles;
    if (late) atomicOr(err, kErrStage);
    if (__any_sync(0xffffffffu, late || *(volatile unsigned*)&sh.abort != 0)) {
      *(volatile unsigned*)&sh.abort = 1u;
      return false;
    }
  }
}

// One pass over subdomain `comp`, whose chunks are a.chunk[c0 .. c0 + nch):
// called by every thread of a CTA of at least C::threads threads; the caller
// synchronises the CTA before it uses sh or smem again (and after
// flow_end, if it makes another pass).
template <typename T, bool UPPER, int R, typename C>
__device__ __forceinline__ void flow_pass(FlowShared<C>& sh, unsigned char* smem_raw, const FlowArgs& a, int comp,
                                          int c0, int nch, const PtrR<T, R>& yslot, const PtrR<T, R>& rhs,
                                          const PtrR<T, R>& x, int* err) {
  using V = VecR<T, R>;
  constexpr int D = C::stages;
  unsigned long long* const s_full = sh.full;
  unsigned *const s_prog = sh.prog, *const s_freed = sh.freed;
  unsigned& s_abort = sh.abort;
  V* ring = (V*)smem_raw;
  unsigned char* stage0 = smem_raw + C::ring_bytes;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  if (tid == 0) {
    // a wait of an earlier pass gave up: the solve reports the timeout, and the passes after it do no work
    s_abort = (*(volatile int*)err & (kErrTimeout | kErrStage)) != 0;
    for (int s = 0; s < D; s++) {
      mbar_init(&s_full[s], 1);
      s_freed[s] = 0;
    }
    mbar_fence_init();
  }
  if (tid <= C::W) s_prog[tid] = 0;
  {
    unsigned* w = (unsigned*)smem_raw;
    constexpr int words = C::ring * (int)sizeof(V) / 4;
    for (int i = tid; i < words + (int)sizeof(V) / 4; i += blockDim.x)
      w[i] = i >= words ? 0u : kFlowWide<T> ? kFlowS64 : kFlowS32;
  }
  // the stages may hold what this thread wrote before the pass (the systems
  // kernel's packed passes use the same buffer); a CTA barrier alone does not
  // order that before the bulk copies
  proxy_fence_smem();
  __syncthreads();
  if (s_abort || warp > C::W) return;
  if (warp == C::W) {
    if (lane == 0) {
      unsigned tot[D];
#pragma unroll
      for (int s = 0; s < D; s++) tot[s] = 0;
      int c = 0;
      bool ok = true;
      int4 nx = __ldg(&a.chunk[c0]);
      while (c < nch && ok) {
#pragma unroll
        for (int s = 0; s < D; s++) {
          if (c < nch && ok) {
            const int4 m = nx;
            if (c + 1 < nch) nx = __ldg(&a.chunk[c0 + c + 1]);
            if (c >= D) {
              int k = 0;
              while (flow_ld(&s_freed[s]) < tot[s]) {
                if (++k > kFlowPolls || *(volatile unsigned*)&s_abort) {
                  if (k > kFlowPolls) atomicOr(err, kErrStage);
                  s_abort = 1;
                  ok = false;
                  break;
                }
                __nanosleep(32);
              }
              proxy_fence_smem();  // the reads of the stage's last use, acquired above, before the copy over them
            }
            if (ok) {
              tot[s] += m.z;
              mbar_arrive_expect_tx(&s_full[s], (unsigned)m.y * 16u);
              bulk_g2s(stage0 + (size_t)s * C::stage_bytes, a.blob + (size_t)m.x * 16, (unsigned)m.y * 16u, &s_full[s]);
              c++;
              flow_st(&s_prog[C::W], (unsigned)c);
            }
          }
        }
      }
      // every copy lands before the CTA's shared memory is released
      for (int k = max(c - D, 0); k < c; k++) mbar_wait(&s_full[k % D], (unsigned)((k / D) & 1), err);
    }
    return;
  }
  const int2 f = __ldg(&a.first[comp * C::W + warp]);
  int ch = f.x, off = f.y;
  bool have_b = false;
  T b[R];
#pragma unroll
  for (int r = 0; r < R; r++) b[r] = T(0);
  const unsigned ring_at = smem_u32(smem_raw);
  unsigned mine = 0;    // tasks this warp has done
  unsigned issued = 0;  // chunks this warp knows to be issued
  while (ch >= 0) {
    const int st = ch % D;
    if (!flow_chunk<C>(sh, ch, issued, err)) break;
    const unsigned char* base = stage0 + (size_t)st * C::stage_bytes;
    const int4 h0 = *(const int4*)(base + off), h1 = *(const int4*)(base + off + 16),
               h2 = *(const int4*)(base + off + 32), h3 = *(const int4*)(base + off + 48);
    const int nrows = h0.w & 0xff, stride = h0.w >> 8;
    const bool on = lane < nrows;
    const int l = on ? lane : 0;
    const int id = *(const int*)(base + h0.x + 4 * l);       // natural row
    if (!have_b) {
#pragma unroll
      for (int r = 0; r < R; r++) b[r] = UPPER ? ldcg(&yslot.p[r][h3.w + l]) : ldcg(&rhs.p[r][id]);
    }
    T acc[kFlowSets<T>][4][R], last[2][R];  // the last quad's sums: entries 0 and 1, entries 2 and 3
#pragma unroll
    for (int r = 0; r < R; r++) last[0][r] = last[1][r] = T(0);
#pragma unroll
    for (int e = 0; e < kFlowSets<T>; e++)
#pragma unroll
      for (int u = 0; u < 4; u++)
#pragma unroll
        for (int r = 0; r < R; r++) acc[e][u][r] = T(0);
    T old[R];  // the sum of all but the last quad; one set of sums: of the blocks that are complete
#pragma unroll
    for (int r = 0; r < R; r++) old[r] = T(0);
    auto fold = [&]() {
#pragma unroll
      for (int r = 0; r < R; r++) {
        old[r] += (acc[0][0][r] + acc[0][2][r]) + (acc[0][1][r] + acc[0][3][r]);
#pragma unroll
        for (int u = 0; u < 4; u++) acc[0][u][r] = T(0);
      }
    };
    // far operands: solved so long ago that they left the ring.  Their tasks
    // are 3 W back: this warp's last wait covers the release after their stores.
    constexpr int FQ = R == 1 ? 2 : 1;  // far quads whose loads are in flight together
    for (int q0 = 0; q0 < h3.x; q0 += FQ) {
      int cc[FQ][4];
      T fv[FQ][4], w[FQ][4][R];
#pragma unroll
      for (int e = 0; e < FQ; e++) {
        const bool have = q0 + e < h3.x;
        const size_t at = (size_t)((have ? q0 + e : q0) * stride + l);
        const int4 fc = *(const int4*)(base + h3.y + at * 16);
        const T* vp = (const T*)(base + h3.y + (size_t)h3.x * stride * 16 + at * 4 * sizeof(T));
        cc[e][0] = have ? fc.x : -1;
        cc[e][1] = have ? fc.y : -1;
        cc[e][2] = have ? fc.z : -1;
        cc[e][3] = have ? fc.w : -1;
#pragma unroll
        for (int u = 0; u < 4; u++) {
          const int j = cc[e][u] & kFlowIndex;
          const bool in = cc[e][u] >= 0 && j < a.n;
          fv[e][u] = in ? vp[u] : T(0);
#pragma unroll
          for (int r = 0; r < R; r++) w[e][u][r] = in ? ldcg(UPPER ? &x.p[r][j] : &yslot.p[r][j]) : T(0);
        }
      }
#pragma unroll
      for (int e = 0; e < FQ; e++) {
        if constexpr (kFlowSets<T> == 1) {
          bool next = false;
#pragma unroll
          for (int u = 0; u < 4; u++) next |= cc[e][u] >= 0 && (cc[e][u] & kFlowOther);
          if (next) fold();
        }
#pragma unroll
        for (int u = 0; u < 4; u++) {
          const bool newest = (cc[e][u] & kFlowLast) != 0;
          const bool other = kFlowSets<T> == 2 && (cc[e][u] & kFlowOther);
#pragma unroll
          for (int r = 0; r < R; r++) {
            T t = newest ? last[u / 2][r] : other ? acc[kFlowSets<T> - 1][u][r] : acc[0][u][r];
            mac(t, fv[e][u], w[e][u][r]);
            if (newest)
              last[u / 2][r] = t;
            else if (other)
              acc[kFlowSets<T> - 1][u][r] = t;
            else
              acc[0][u][r] = t;
          }
        }
      }
    }
    // with the progress comes the number of chunks issued, in time for the look ahead at the end of the task
    issued = max(issued, flow_wait<C::W>(s_prog, h1.y, lane, err, &s_abort));
    // the slots of the rows half a ring ahead: their old values are read no more
    if (on) {
      FlowVal<T, R> none;
#pragma unroll
      for (int w = 0; w < (int)sizeof(V) / 4; w++) none.u[w] = kFlowWide<T> ? kFlowS64 : kFlowS32;
      flow_ring_store<T, R>(ring_at + (unsigned)((h2.y + C::ahead + lane) & (C::ring - 1)) * (unsigned)sizeof(V), none);
    }
    const unsigned char* cols = base + h0.y;
    const unsigned char* vals = base + h0.z;
    const int g1 = h1.x & 0xff, g2 = (h1.x >> 8) & 0xff, g4 = (h1.x >> 16) & 0xff;
    int k = 0;
    FlowQuad<T> cur;
    if (g4 > 0) cur = flow_load_quad<T>(cols, vals, l);
    // before the oldest quad of a block, unless the far operands began it (or the row has nothing in it)
    auto next_block = [&]() {
      if constexpr (kFlowSets<T> == 1)
        if ((g4 - k) % kFlowBlock == 0 && (cur.c.x & 0xffffu) != (unsigned)C::ring) fold();
    };
    auto use = [&](T (&s)[4][R]) {
      next_block();
      FlowQuad<T> nxt = cur;
      if (k + 1 < g4) nxt = flow_load_quad<T>(cols, vals, (k + 1) * stride + l);
      const unsigned i0 = cur.c.x & 0xffffu, i1 = cur.c.x >> 16, i2 = cur.c.y & 0xffffu, i3 = cur.c.y >> 16;
      const V w0 = ring[i0], w1 = ring[i1], w2 = ring[i2], w3 = ring[i3];
#pragma unroll
      for (int r = 0; r < R; r++) {
        mac(s[0][r], cur.v[0], w0.v[r]);
        mac(s[1][r], cur.v[1], w1.v[r]);
        mac(s[2][r], cur.v[2], w2.v[r]);
        mac(s[3][r], cur.v[3], w3.v[r]);
      }
      cur = nxt;
      k++;
    };
    auto run = [&](int end) {
      if constexpr (kFlowSets<T> == 2) {
        while (k + 1 < end) {
          use(acc[0]);
          use(acc[1]);
        }
        if (k < end) {  // the sets change places: they are added up alike in the end
          use(acc[0]);
#pragma unroll
          for (int u = 0; u < 4; u++)
#pragma unroll
            for (int r = 0; r < R; r++) {
              const T t = acc[0][u][r];
              acc[0][u][r] = acc[1][u][r];
              acc[1][u][r] = t;
            }
        }
      } else {
        while (k < end) use(acc[0]);
      }
    };
    run(min(g1, g4 - 1));
    if (g2 > g1) {
      issued = max(issued, flow_wait<C::W>(s_prog, h1.z, lane, err, &s_abort));
      run(min(g2, g4 - 1));
    }
    // what the end of the task needs, and the right-hand side of this warp's next task
    const int nch_ = h2.z, noff = h2.w;
    const int us = UPPER ? 0 : *(const int*)(base + h0.x + 4 * stride + 4 * l);
    T dg = T(1);
    if (UPPER) dg = *(const T*)(base + h0.x + 4 * ((stride + 3) & ~3) + (size_t)l * sizeof(T));
    // operands of the tasks in flight: each is its own flag
    FlowVal<T, R> w0, w1, w2, w3;
    auto poll = [&](const FlowQuad<T>& q) {
      const unsigned sz = (unsigned)sizeof(V);
      const unsigned i0 = ring_at + (q.c.x & 0xffffu) * sz, i1 = ring_at + (q.c.x >> 16) * sz,
                     i2 = ring_at + (q.c.y & 0xffffu) * sz, i3 = ring_at + (q.c.y >> 16) * sz;
      for (int p = 0;; p++) {
        flow_ring_load<T, R>(w0, i0);
        flow_ring_load<T, R>(w1, i1);
        flow_ring_load<T, R>(w2, i2);
        flow_ring_load<T, R>(w3, i3);
        if (!(flow_missing<T, R>(w0) | flow_missing<T, R>(w1) | flow_missing<T, R>(w2) | flow_missing<T, R>(w3))) break;
        if ((p & 255) == 255) {
          if (p >= kFlowPolls) {
            atomicOr(err, kErrStage);
            *(volatile unsigned*)&s_abort = 1u;
          }
          if (*(volatile unsigned*)&s_abort) break;
        }
      }
    };
    auto fresh = [&](T (&s)[4][R]) {
      next_block();
      const FlowQuad<T> nxt = flow_load_quad<T>(cols, vals, (k + 1) * stride + l);
      poll(cur);
#pragma unroll
      for (int r = 0; r < R; r++) {
        mac(s[0][r], cur.v[0], w0.v.v[r]);
        mac(s[1][r], cur.v[1], w1.v.v[r]);
        mac(s[2][r], cur.v[2], w2.v.v[r]);
        mac(s[3][r], cur.v[3], w3.v.v[r]);
      }
      cur = nxt;
      k++;
    };
    while (k + 1 < g4) {
      fresh(acc[0]);
      if (kFlowSets<T> == 2 && k + 1 < g4) fresh(acc[kFlowSets<T> - 1]);
    }
    // the sum of all but the last quad is formed before that is waited for
#pragma unroll
    for (int r = 0; r < R; r++) {
      T part[4];
#pragma unroll
      for (int u = 0; u < 4; u++) part[u] = kFlowSets<T> == 2 ? acc[0][u][r] + acc[kFlowSets<T> - 1][u][r] : acc[0][u][r];
      const T sum = (part[0] + part[2]) + (part[1] + part[3]);
      old[r] = kFlowSets<T> == 2 ? sum : old[r] + sum;
    }
    if (g4 > 0) {
      poll(cur);
#pragma unroll
      for (int r = 0; r < R; r++) {
        mac(last[0][r], cur.v[0], w0.v.v[r]);
        mac(last[1][r], cur.v[2], w2.v.v[r]);
        mac(last[0][r], cur.v[1], w1.v.v[r]);
        mac(last[1][r], cur.v[3], w3.v.v[r]);
      }
    }
    FlowVal<T, R> res;
#pragma unroll
    for (int r = 0; r < R; r++) {
      const T t = b[r] - (old[r] + (last[0][r] + last[1][r]));
      res.v.v[r] = UPPER ? t * dg : t;
    }
    if (on) flow_ring_store<T, R>(ring_at + (unsigned)((h2.y + lane) & (C::ring - 1)) * (unsigned)sizeof(V), res);
    __syncwarp();
    mine++;
    if (lane == 0) flow_st(&s_prog[warp], mine);
    // off the chain: the result to global memory, the stage, the next right-hand side
    if (on) {
#pragma unroll
      for (int r = 0; r < R; r++) {
        if (UPPER)
          x.p[r][id] = res.v.v[r];
        else
          yslot.p[r][us] = res.v.v[r];
      }
    }
    if (lane == 0) flow_add(&s_freed[st]);
    bool nb = false;
    T bn[R];
#pragma unroll
    for (int r = 0; r < R; r++) bn[r] = T(0);
    if (nch_ >= 0 && flow_issued(issued, nch_) && mbar_try_wait(&s_full[nch_ % D], (unsigned)((nch_ / D) & 1))) {
      const unsigned char* nbase = stage0 + (size_t)(nch_ % D) * C::stage_bytes;
      const int nr2 = *(const int*)(nbase + noff + 12) & 0xff;
      const int l2 = lane < nr2 ? lane : 0;
      if (UPPER) {
        const int s2 = *(const int*)(nbase + noff + 60);
#pragma unroll
        for (int r = 0; r < R; r++) bn[r] = ldcg(&yslot.p[r][s2 + l2]);
      } else {
        const int id2 = *(const int*)(nbase + *(const int*)(nbase + noff) + 4 * l2);
#pragma unroll
        for (int r = 0; r < R; r++) bn[r] = ldcg(&rhs.p[r][id2]);
      }
      nb = true;
    }
#pragma unroll
    for (int r = 0; r < R; r++) b[r] = bn[r];
    have_b = nb;
    ch = nch_;
    off = noff;
  }
}


template <typename T, bool UPPER, int R, typename C = FlowCfg<T, R>>
__global__ void __launch_bounds__(C::threads, 1) trsv_flow_kernel(FlowArgs a, PtrR<T, R> yslot, PtrR<T, R> rhs,
                                                                  PtrR<T, R> x, int* err, SkipR<R> skip) {
  if (skip.on()) return;
  extern __shared__ __align__(16) unsigned char flow_smem[];
  __shared__ __align__(8) FlowShared<C> sh;
  const int c0 = a.comp_chunk0[blockIdx.x], nch = a.comp_chunk0[blockIdx.x + 1] - c0;
  if (nch > 0) flow_pass<T, UPPER, R, C>(sh, flow_smem, a, blockIdx.x, c0, nch, yslot, rhs, x, err);
}

// the barriers of a finished pass, before the CTA makes another one (after a __syncthreads)
template <typename C>
__device__ __forceinline__ void flow_end(FlowShared<C>& sh) {
  if (threadIdx.x == 0)
    for (int s = 0; s < C::stages; s++)
      asm volatile("mbarrier.inval.shared::cta.b64 [%0];" ::"r"(smem_u32(&sh.full[s])) : "memory");
  __syncthreads();
}

}  // namespace pgx
