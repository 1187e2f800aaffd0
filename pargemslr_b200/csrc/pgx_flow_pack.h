// Host layout of the per-subdomain triangular solve (trsv_flow_kernel in
// pgx_flow.cuh): shared-memory plan and task images.  No CUDA in this file, so
// that the layout can be checked on the host alone.
#pragma once

#include <algorithm>
#include <climits>
#include <cstddef>
#include <new>
#include <utility>
#include <vector>

namespace pgx {

constexpr int kFlowHead = 16;                  // ints of a task header
constexpr int kFlowMaxQuads = 250;             // quads of one row (a byte each in the header)
constexpr int kFlowOther = 1 << 30;            // far operand: the second set of sums; with one set, see kFlowBlock
constexpr int kFlowLast = 1 << 29;             // far operand: one of the row's four newest entries
constexpr int kFlowIndex = kFlowLast - 1;
// A row's four newest entries are summed by themselves, the others in
// kFlowSets sets of four accumulators, successive quads on alternate sets: as
// many partial sums as the eight lanes that summed a row before (sixteen where
// a factor has more than 32 entries a row), and no more rounding up to that length (the
// lower pass at 48^3 in FP32 against FP64: 4.1e-8 with eight, 4.4e-8 with
// four, 4.9e-8 with two; in a CPU model of 67 / 201 entries a row sixteen sums
// round 0 to 8% / 12 to 17% less than eight).
template <typename T>
constexpr int kFlowSets = sizeof(T) <= 8 ? 2 : 1;
// Two sets of 16-byte values do not fit the registers (four lanes spilled, and
// took twice the time).  There the one set is added up after every kFlowBlock
// quads, counted from the row's end, and starts again from zero.  Error of a
// pass against 80 bits in a CPU model (ILUT factors of shifted 3D Laplacians),
// as a multiple of eight lanes' error, 35 / 67 / 201 entries a row: 1.00 to
// 1.02 / 0.96 to 0.97 / 0.94; with the set running through 1.03 to 1.05 /
// 1.08 / 1.23 to 1.24.
constexpr int kFlowBlock = 8;

// Whether a warp may test the barrier of chunk `chunk`, with `issued` chunks
// issued so far.  Chunk c uses the stage and the barrier of chunk c - stages
// again, and the test is by parity: while that older chunk is on its way the
// barrier looks as if c had landed, and copies land in any order.  A chunk
// is issued only after the older one is consumed, so once it is issued the
// parity says what it should.
#ifdef __CUDACC__
__host__ __device__
#endif
inline bool flow_issued(unsigned issued, int chunk) { return issued > (unsigned)chunk; }

// Shared-memory plan of the solve: a ring of the last results (one value per
// right-hand side and schedule position), then `stages` staging buffers for
// the factor.
template <int VEC, int RING, int STAGE_BYTES, int SMEM, int MAXW>
struct FlowPlan {
  static constexpr int vec = VEC;                    // bytes of one ring entry
  static constexpr int ring = RING;
  static constexpr int stage_bytes = STAGE_BYTES;
  static constexpr size_t ring_bytes = (size_t)vec * ring + 64;  // one more entry, zero, for padding
  static constexpr int stages = (int)((SMEM - ring_bytes) / stage_bytes);
  static constexpr int W = stages < MAXW ? stages : MAXW;  // solving warps; one more stages the factor
  static constexpr int threads = 32 * (W + 1);
  static constexpr int ahead = 32 * (W + 2);           // a task clears the ring slots of the rows this far ahead
  static constexpr int reach = ring - ahead - 32 * W;  // operands at most this old are in the ring
  static constexpr size_t bytes = ring_bytes + (size_t)stages * stage_bytes;
  // a warp looks one task of its own ahead, at most W chunks: with at least W
  // stages that chunk can be on its way while the warp is still in its own
  static_assert(stages >= W && W >= 2 && ring >= ahead + 32 * (4 * W + 1), "flow solve: shared memory");
  static_assert((ring & (ring - 1)) == 0 && vec <= 64, "flow solve: ring");
};
constexpr int flow_ring(int vec, bool lng) {
  return (vec <= 4 ? 8192 : vec <= 16 ? 4096 : 2048) << (lng && vec < 64 ? 1 : 0);
}
// The CTA owns an SM's shared memory.  Twelve warps: with eight the sums of
// the tasks ahead fall behind the chain (64^3, one lane mixed: 0.39 against
// 0.30 ms a pass).  16 KB stages: a task's image is 3-10 KB, and 12 KB stages
// leave too few bytes on their way (0.34 ms).  LONG: twice the ring and fewer warps,
// for factors whose rows reach far back.
template <typename T, int R, bool LONG = false>
struct FlowCfg
    : FlowPlan<(int)sizeof(T) * R, flow_ring((int)sizeof(T) * R, LONG), 16 * 1024, 226 * 1024, 12> {
  static constexpr bool has_long = flow_ring((int)sizeof(T) * R, true) > flow_ring((int)sizeof(T) * R, false);
  static constexpr int task_bytes = 16 * 1024;  // image of one task at most, the same under every lane count
  static constexpr int task_reach() {           // the shortest reach of any lane count
    int r = FlowCfg<T, 1>::reach;
    r = FlowCfg<T, 2>::reach < r ? FlowCfg<T, 2>::reach : r;
    return FlowCfg<T, 4>::reach < r ? FlowCfg<T, 4>::reach : r;
  }
};
// A CTA that shares the SM with others (the systems kernel, one right-hand side).
template <typename T>
struct SysFlowCfg : FlowPlan<(int)sizeof(T), 2048, 8 * 1024, 8 * 8 * 1024 + (int)sizeof(T) * 2048 + 64, 7> {
  static constexpr int task_bytes = 8 * 1024;
  static constexpr int task_reach() { return SysFlowCfg::reach; }
};

// ------------------------------------------------------------------ packing
// The factor as the kernel reads it: per subdomain a list of chunks, each the
// images of consecutive tasks (header, row ids, quads), laid out on the host.
template <typename T>
struct FlowPack {
  int ncomp = 0, nlevels = 0;
  long long ntasks = 0, nfar = 0, padded = 0;
  std::vector<int> chunk;  // int4 per chunk
  std::vector<int> comp_chunk0, first;
  std::vector<unsigned char> blob;
  std::vector<int> slot_of_row;  // position of every row in the schedule, subdomain after subdomain
};

// one subdomain, rows [r0, r1)
template <typename T, typename C, typename Val, typename Diag>
static bool flow_pack_comp(int r0, int r1, const int* rp, const int* cj, const Val& val, bool upper, const Diag* dinv,
                           const std::vector<int>* up_slot, int* lev, int* pos, int* task_of, long long most_far,
                           FlowPack<T>& o) {
  const int m = r1 - r0;
  auto align16 = [](size_t v) { return (v + 15) & ~(size_t)15; };
  // dependency levels and the schedule: rows by level, then by index
  int nlev = 0;
  for (int t = 0; t < m; t++) {
    const int i = upper ? r1 - 1 - t : r0 + t;
    int v = 0;
    for (int k = rp[i]; k < rp[i + 1]; k++) {
      if (cj[k] < r0 || cj[k] >= r1) return false;  // the factor couples two subdomains
      v = std::max(v, lev[cj[k]] + 1);
    }
    lev[i] = v;
    nlev = std::max(nlev, v + 1);
  }
  o.nlevels = nlev;
  std::vector<int> lp(nlev + 1, 0), order(m);
  for (int i = r0; i < r1; i++) lp[lev[i] + 1]++;
  for (int l = 0; l < nlev; l++) lp[l + 1] += lp[l];
  {
    std::vector<int> cur(lp.begin(), lp.end() - 1);
    for (int i = r0; i < r1; i++) order[cur[lev[i]]++] = i;
  }
  for (int p = 0; p < m; p++) pos[order[p]] = p;
  long long far = 0;
  for (int i = r0; i < r1; i++)
    for (int k = rp[i]; k < rp[i + 1]; k++) far += pos[i] - pos[cj[k]] > C::reach;
  if (far > most_far && 2 * far > rp[r1] - rp[r0]) return false;
  // tasks: at most 32 rows of one level.  The bound of a task's image holds
  // under every lane count, so all of them cut the same tasks (and sum every
  // row in the same order).
  const int reach = C::task_reach();
  std::vector<int> len(m), flen(m);
  for (int p = 0; p < m; p++) {
    const int i = order[p];
    int f = 0;
    for (int k = rp[i]; k < rp[i + 1]; k++) f += p - pos[cj[k]] > reach;
    len[p] = rp[i + 1] - rp[i];
    flen[p] = f ? f + 3 : 0;
  }
  auto bytes_of = [&](int a, int e) {
    int mx = 0, mxf = 0;
    for (int p = a; p < e; p++) {
      mx = std::max(mx, len[p]);
      mxf = std::max(mxf, flen[p]);
    }
    const int quads = (mx + 3) / 4, fq = (mxf + 3) / 4, stride = (e - a + 1) & ~1;
    return (size_t)kFlowHead * 4 + align16((size_t)stride * 4) + align16((size_t)stride * std::max<size_t>(4, sizeof(T))) +
           (size_t)quads * stride * (8 + 4 * sizeof(T)) + (size_t)fq * stride * (16 + 4 * sizeof(T)) + 64;
  };
  std::vector<int> ta;  // first position of every task, and m
  for (int l = 0; l < nlev; l++) {
    const int w = lp[l + 1] - lp[l];
    auto cut = [&](int q, int parts) { return lp[l] + (int)((long long)w * q / parts); };
    int parts = (w + 31) / 32;
    for (;;) {
      bool ok = true;
      for (int q = 0; q < parts && ok; q++) ok = bytes_of(cut(q, parts), cut(q + 1, parts)) <= (size_t)C::task_bytes;
      if (ok) break;
      if (parts >= w) return false;  // a single row is too long
      parts = std::min(w, parts * 2);
    }
    for (int q = 0; q < parts; q++) ta.push_back(cut(q, parts));
  }
  const int nt = (int)ta.size();
  ta.push_back(m);
  for (int t = 0; t < nt; t++)
    for (int p = ta[t]; p < ta[t + 1]; p++) task_of[order[p]] = t;
  o.ntasks = nt;
  // images, appended to chunks of at most stage_bytes and W tasks
  std::vector<int> tch(nt);
  std::vector<size_t> tat(nt);  // where the image starts in the blob
  std::vector<size_t> chunk_at;
  std::vector<int> chunk_tasks;
  std::vector<std::pair<int, int>> ent[32];  // (source position, entry) of each row, oldest first
  int nnear[32], nfar[32];
  for (int t = 0; t < nt; t++) {
    const int a = ta[t], nr = ta[t + 1] - a, stride = (nr + 1) & ~1;
    int mx = 0, mxf = 0;
    for (int q = 0; q < nr; q++) {
      const int i = order[a + q];
      auto& e = ent[q];
      e.clear();
      for (int k = rp[i]; k < rp[i + 1]; k++) e.push_back({pos[cj[k]], k});
      std::sort(e.begin(), e.end());
      // near: its slot is cleared by the task that holds position pos + ring -
      // ahead, which starts after this task is done; else far, read back from
      // global memory, where its warp's next task has published it
      int f = 0;
      for (auto& x : e) {
        const int pr = x.first + C::ring - C::ahead;
        if (pr >= m || task_of[order[pr]] >= t + C::W) break;
        if (task_of[cj[x.second]] + 3 * C::W > t) return false;
        f++;
      }
      nfar[q] = f;
      nnear[q] = (int)e.size() - f;
      o.nfar += f;
      mx = std::max(mx, nnear[q]);
      // some places more keep every entry on the accumulator that its distance
      // from the row's last entry names
      mxf = std::max(mxf, f ? f + nnear[q] % 4 : 0);
    }
    const int quads = (mx + 3) / 4, fq = (mxf + 3) / 4;
    if (quads > kFlowMaxQuads || fq > kFlowMaxQuads) return false;
    o.padded += (long long)(quads + fq) * 4 * stride;
    const size_t idb = upper ? align16((size_t)stride * 4) + (size_t)stride * sizeof(T) : (size_t)stride * 8;
    const size_t off_ids = kFlowHead * 4, off_cols = align16(off_ids + idb);
    const size_t off_vals = align16(off_cols + (size_t)quads * stride * 8);
    const size_t off_far = align16(off_vals + (size_t)quads * stride * 4 * sizeof(T));
    const size_t total = align16(off_far + (size_t)fq * stride * (16 + 4 * sizeof(T)));
    if (total > (size_t)C::stage_bytes) return false;
    if (chunk_at.empty() || chunk_tasks.back() >= C::W ||
        o.blob.size() - chunk_at.back() + total > (size_t)C::stage_bytes) {
      chunk_at.push_back(o.blob.size());
      chunk_tasks.push_back(0);
    }
    const size_t base = chunk_at.back();
    tch[t] = (int)chunk_at.size() - 1;
    tat[t] = o.blob.size();
    chunk_tasks.back()++;
    o.blob.resize(tat[t] + total, 0);
    unsigned char* b = o.blob.data() + tat[t];
    int need[kFlowMaxQuads + 1] = {0};  // highest source task of each quad, plus one
    for (int q = 0; q < stride; q++) {
      const bool real = q < nr;
      const int i = real ? order[a + q] : order[a];
      ((int*)(b + off_ids))[q] = i;
      if (upper)
        ((T*)(b + off_ids + align16((size_t)stride * 4)))[q] = (*dinv)(i);
      else
        ((int*)(b + off_ids))[stride + q] = (*up_slot)[i];
      const int nn = real ? nnear[q] : 0, nf = real ? nfar[q] : 0;
      for (int u = 0; u < quads * 4; u++) {
        const size_t slot = (size_t)(u / 4) * stride + q;
        unsigned short* cp = (unsigned short*)(b + off_cols) + slot * 4 + (u & 3);
        T* vp = (T*)(b + off_vals) + slot * 4 + (u & 3);
        const int e = u - (quads * 4 - nn);  // right-aligned: the newest entries share the last quad
        if (e < 0) {
          *cp = (unsigned short)C::ring;  // the zero slot
          *vp = T(0);
        } else {
          const std::pair<int, int>& x = ent[q][nf + e];
          *cp = (unsigned short)(x.first & (C::ring - 1));
          *vp = val(x.second);
          need[u / 4] = std::max(need[u / 4], task_of[cj[x.second]] + 1);
        }
      }
      for (int u = 0; u < fq * 4; u++) {
        const size_t slot = (size_t)(u / 4) * stride + q;
        int* cp = (int*)(b + off_far) + slot * 4 + (u & 3);
        T* vp = (T*)(b + off_far + (size_t)fq * stride * 16) + slot * 4 + (u & 3);
        const int e = nf ? u - (fq * 4 - nf - nn % 4) : -1;
        if (e >= 0 && e < nf) {
          const int k = ent[q][e].second;
          const int back = nn + nf - 1 - e;  // entries of the row after this one
          *cp = upper ? cj[k] : (*up_slot)[cj[k]];
          if (back < 4)
            *cp |= kFlowLast;
          else if (kFlowSets<T> == 2 ? (back / 4 + quads + 1) % 2 : back / 4 % kFlowBlock == kFlowBlock - 1)
            *cp |= kFlowOther;
          *vp = val(k);
        } else {
          *cp = -1;
          *vp = T(0);
        }
      }
    }
    // quads whose sources are W tasks back, W / 2 tasks back, and the rest
    const int lim1 = std::max(0, t - C::W + 1), lim2 = std::max(0, t - C::W / 2 + 1);
    int g1 = 0;
    while (g1 < quads && need[g1] <= lim1) g1++;
    int g2 = g1;
    while (g2 < quads && need[g2] <= lim2) g2++;
    const int in_chunk = (int)(tat[t] - base);
    int* h = (int*)b;
    h[0] = in_chunk + (int)off_ids;
    h[1] = in_chunk + (int)off_cols;
    h[2] = in_chunk + (int)off_vals;
    h[3] = nr | (stride << 8);
    h[4] = g1 | (g2 << 8) | (quads << 16);
    h[5] = lim1;
    h[6] = lim2;
    h[9] = a;
    h[10] = -1;
    h[12] = fq;
    h[13] = in_chunk + (int)off_far;
    h[15] = r0 + a;
    if (t >= C::W) {
      int* before = (int*)(o.blob.data() + tat[t - C::W]);
      before[10] = tch[t];
      before[11] = in_chunk;
    }
  }
  for (size_t c = 0; c < chunk_at.size(); c++) {
    const size_t end = c + 1 < chunk_at.size() ? chunk_at[c + 1] : o.blob.size();
    o.chunk.insert(o.chunk.end(), {(int)(chunk_at[c] / 16), (int)((end - chunk_at[c]) / 16), chunk_tasks[c], 0});
  }
  for (int w = 0; w < C::W; w++) {
    o.first.push_back(w < nt ? tch[w] : -1);
    o.first.push_back(w < nt ? (int)(tat[w] - chunk_at[tch[w]]) : 0);
  }
  return true;
}

// Returns false when the factor does not suit the kernel: it couples two
// subdomains, a row is too long, an operand is too old for the ring yet too
// new to be read back, or most operands of a subdomain, and more than
// `most_far`, are that old.
template <typename T, typename C, typename Val, typename Diag>
static bool flow_pack(int n, const int* rp, const int* cj, const Val& val, bool upper, const std::vector<int>& dom,
                      const Diag* dinv, const std::vector<int>* up_slot, FlowPack<T>& o,
                      long long most_far = LLONG_MAX) {
  const int ncomp = (int)dom.size() - 1;
  o = FlowPack<T>();
  o.ncomp = ncomp;
  std::vector<int> lev(n, 0), pos(n, 0), task_of(n, 0);
  std::vector<FlowPack<T>> part(ncomp);
  std::vector<char> ok(ncomp, 0);
  // in parallel where that pays: 33,000 entries take 2.6 ms on one thread, and
  // a team takes 10 ms and more to wake up
#pragma omp parallel for schedule(dynamic, 1) if (rp[n] > 300000)
  for (int c = 0; c < ncomp; c++) {
    try {
      ok[c] = flow_pack_comp<T, C>(dom[c], dom[c + 1], rp, cj, val, upper, dinv, up_slot, lev.data(), pos.data(),
                                   task_of.data(), most_far, part[c]);
    } catch (const std::bad_alloc&) {
      ok[c] = 2;  // no exception may leave the parallel region
    }
  }
  for (int c = 0; c < ncomp; c++)
    if (ok[c] == 2) throw std::bad_alloc();
  size_t bytes = 0;
  for (int c = 0; c < ncomp; c++) {
    if (!ok[c]) return false;
    bytes += part[c].blob.size();
  }
  if (bytes / 16 > (size_t)INT_MAX || n > kFlowIndex) return false;
  o.blob.reserve(bytes);
  o.comp_chunk0.assign(1, 0);
  for (int c = 0; c < ncomp; c++) {
    FlowPack<T>& q = part[c];
    const int unit0 = (int)(o.blob.size() / 16);
    for (size_t k = 0; k < q.chunk.size(); k += 4) q.chunk[k] += unit0;
    o.chunk.insert(o.chunk.end(), q.chunk.begin(), q.chunk.end());
    o.first.insert(o.first.end(), q.first.begin(), q.first.end());
    o.blob.insert(o.blob.end(), q.blob.begin(), q.blob.end());
    o.comp_chunk0.push_back((int)o.chunk.size() / 4);
    o.nlevels = std::max(o.nlevels, q.nlevels);
    o.ntasks += q.ntasks;
    o.nfar += q.nfar;
    o.padded += q.padded;
    q = FlowPack<T>();
  }
  o.slot_of_row.resize(n);
  for (int c = 0; c < ncomp; c++)
    for (int i = dom[c]; i < dom[c + 1]; i++) o.slot_of_row[i] = dom[c] + pos[i];
  return true;
}

}  // namespace pgx
