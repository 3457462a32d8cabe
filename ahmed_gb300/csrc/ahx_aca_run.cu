// Host side of an assembly's ACA: order of the leaves, workspace slots, retries.
#include <algorithm>
#include <cmath>

#include "ahx_aca.cuh"
#include "ahx_hmat.hpp"

namespace ahx {
namespace {

// A leaf goes to a CTA instead of a warp when its rows and columns are more than half of
// what a resident warp gets on average (a warp that takes longer ends after the others),
// or when half the workspace budget would not hold a slot for every resident warp; but
// never below 512, where the work on the k x k arrays (one warp, the others wait)
// outweighs the rows.  A leaf's k x k work counts as 256 rows.  Where the budget does not
// hold slots for half of the resident CTAs either, the leaves too large for that run first,
// alone and in all of the budget.  (1,048,576 points, 440,940 leaves: with the first rule
// only, 130 warps at a time, the assembly took 7.6 s; so 0.90 s; 262,144 points 0.35 -> 0.12 s.)
constexpr uint64_t kLeafRows = 256, kLargeMin = 512;

uint64_t class_bytes(uint32_t c) {  // an upper bound of the class, a multiple of 256
  const uint64_t top = (uint64_t)(16 + (c & 15) + 1) << (c / 16 - 4);
  return (top + 255) & ~255ull;
}

// A set of tasks in descending class of their workspace, with the classes' bytes
struct Sorted {
  std::vector<AcaTask> t;
  std::vector<uint64_t> bytes;
  Sorted() = default;
  Sorted(const std::vector<AcaTask>& in, size_t elem) : t(in.size()), bytes(in.size()) {
    std::vector<uint64_t> size(in.size());
    for (size_t i = 0; i < in.size(); ++i) size[i] = aca_ws_bytes(in[i].n1, in[i].n2, in[i].kcap, elem);
    std::vector<uint32_t> ord;
    order_by_size(size, ord, 4);
    for (size_t i = 0; i < in.size(); ++i) {
      t[i] = in[ord[i]];
      bytes[i] = class_bytes(size_class(size[ord[i]]));
    }
  }
  // slots for the first tasks from `at` on: at most n, one at least, within `room` bytes
  uint32_t slots(size_t at, uint64_t n, uint64_t room) const {
    n = std::min<uint64_t>(n, t.size() - at);
    uint64_t part = 0;
    uint32_t k = 0;
    for (; k < n; ++k) {
      part += bytes[at + k];
      if (k && part > room) break;
    }
    return k;
  }
  // the first task from which on n slots (or as many as tasks are left) fit into `room` bytes
  size_t fits(uint64_t n, uint64_t room) const {
    uint64_t part = 0;
    size_t i = 0, j = 0;
    for (; i < t.size(); ++i) {
      for (; j < t.size() && j < i + n; ++j) part += bytes[j];
      if (part <= room) break;
      part -= bytes[i];
    }
    return i;
  }
};

}  // namespace

uint32_t size_class(uint64_t size) {
  const int m = 63 - __builtin_clzll(size | 16);
  return (uint32_t)(m * 16) + (uint32_t)((size >> (m - 4)) & 15);
}

void order_by_size(const std::vector<uint64_t>& size, std::vector<uint32_t>& order, int bits) {
  // sizes below 2^bits as they are, from there on 2^bits steps an octave
  auto key = [bits](uint64_t s) -> uint32_t {
    if (s >> bits == 0) return (uint32_t)s;
    const int m = 63 - __builtin_clzll(s);
    return ((uint32_t)(m - bits) << bits) + (uint32_t)(s >> (m - bits));
  };
  const uint32_t n = (uint32_t)(65 - bits) << bits;
  std::vector<uint32_t> at(n + 1, 0);
  for (uint64_t s : size) ++at[n - key(s)];
  for (uint32_t c = 0; c < n; ++c) at[c + 1] += at[c];
  order.resize(size.size());
  for (size_t i = 0; i < size.size(); ++i) order[at[n - 1 - key(size[i])]++] = (uint32_t)i;
}

std::vector<DenseTask> dense_tasks(const std::vector<Leaf>& Ls, uint32_t n, const std::vector<uint32_t>& leaves,
                                   const std::vector<uint64_t>& off) {
  // lists of the tasks by first row (their leaf has b1 < b2), for the mirror images
  std::vector<DenseTask> t;
  std::vector<uint32_t> head(n, 0u), next;
  t.reserve(leaves.size());
  next.reserve(leaves.size());
  for (int pass = 0; pass < 2; ++pass)
    for (uint32_t l : leaves) {
      const Leaf& L = Ls[l];
      if ((L.b1 > L.b2) != (pass == 1)) continue;
      if (pass == 1) {
        uint32_t q = head[L.b2];
        while (q && (t[q - 1].b2 != L.b1 || t[q - 1].n1 != L.n2 || t[q - 1].n2 != L.n1)) q = next[q - 1];
        if (q) {
          t[q - 1].mirror = off[l];
          continue;
        }
      }
      t.push_back(DenseTask{L.b1, L.n1, L.b2, L.n2, off[l], kNoMirror});
      next.push_back(0u);
      if (L.b1 < L.b2) {
        next.back() = head[L.b1];
        head[L.b1] = (uint32_t)t.size();
      }
    }
  return t;
}

int run_aca(ahx_hmat* H, bool cplx, std::vector<AcaTask>& tasks, AcaParams p, std::vector<uint32_t>& dense) {
  const size_t elem = cplx ? 16 : 8;
  DevBuf& arena = cplx ? H->z.arena : H->arena64;
  uint64_t& elems = cplx ? H->z.elems : H->arena64_elems;
  std::vector<int32_t>& rank = cplx ? H->z.rank : H->rank;
  std::vector<int32_t>& aca_rank = cplx ? H->z.aca_rank : H->aca_rank;
  std::vector<uint64_t>& offs = cplx ? H->z.off : H->off;
  const uint64_t budget = aca_ws_budget();
  p.variant = H->tree.sym ? kAcaVariantSym : kAcaVariantGeneral;
  uint32_t ctas = 0;
  AHX_CUDA(cplx ? resident_zaca(H->device, ctas) : resident_aca(H->device, ctas));
  constexpr uint32_t kWarps = kAcaThreads / 32;
  ScopedBuf ws, dtasks, dres, dslots, dctl;
  int rc;
  while (!tasks.empty()) {
    uint64_t rows = 0;
    for (const AcaTask& t : tasks) rows += (uint64_t)t.n1 + t.n2 + kLeafRows;
    const uint64_t lim = std::max<uint64_t>(kLargeMin, rows / ((uint64_t)ctas * kWarps * 2));
    const Sorted all_tasks(tasks, elem);
    const size_t cut = all_tasks.fits((uint64_t)ctas * kWarps, budget / 2);
    Sorted large, small;
    small.t.reserve(tasks.size());
    small.bytes.reserve(tasks.size());
    for (size_t i = 0; i < all_tasks.t.size(); ++i) {
      const uint64_t n = (uint64_t)all_tasks.t[i].n1 + all_tasks.t[i].n2;
      Sorted& to = n > kLargeMin && (n > lim || i < cut) ? large : small;
      to.t.push_back(all_tasks.t[i]);
      to.bytes.push_back(all_tasks.bytes[i]);
    }
    // the largest leaves in a launch of their own?
    std::vector<AcaTask> later;
    const uint32_t ns = large.slots(0, ctas, budget / 2);
    uint64_t room = budget / 2;
    if (2 * (uint64_t)ns < std::min<uint64_t>(ctas, large.t.size())) {
      const size_t first = large.fits(ctas, budget / 2);
      if (first >= 2 * (size_t)ns) {
        later.assign(large.t.begin() + (std::ptrdiff_t)first, large.t.end());
        later.insert(later.end(), small.t.begin(), small.t.end());
        large.t.resize(first);
        large.bytes.resize(first);
        small = Sorted();
        room = budget;
      }
    }
    // slots: each phase takes at most half the budget, and at least one team runs
    p.nlarge = (uint32_t)large.t.size();
    p.nsmall = (uint32_t)small.t.size();
    p.nslot_l = large.slots(0, ctas, room);
    p.nslot_s = small.slots(0, (uint64_t)ctas * kWarps, budget / 2);
    std::vector<uint64_t> slots;
    uint64_t bytes = 0;
    for (uint32_t i = 0; i < p.nslot_l + p.nslot_s; ++i) {
      slots.push_back(bytes);
      bytes += i < p.nslot_l ? large.bytes[i] : small.bytes[i - p.nslot_l];
    }
    H->stat_ws_bytes = std::max<uint64_t>(H->stat_ws_bytes, bytes);
    H->stat_batches++;
    std::vector<AcaTask> all(std::move(large.t));
    all.insert(all.end(), small.t.begin(), small.t.end());
    struct Ctl {
      unsigned long long used;
      uint32_t ctr[2];
    };
    const std::vector<Ctl> ctl{{elems, {0u, 0u}}};
    if ((rc = ws.reserve(bytes)) || (rc = upload(dtasks, all, H->stream)) || (rc = upload(dslots, slots, H->stream)) ||
        (rc = upload(dctl, ctl, H->stream)) || (rc = dres.reserve(all.size() * sizeof(AcaResult))))
      return rc;
    p.tasks = dtasks.as<AcaTask>();
    p.res = dres.as<AcaResult>();
    p.slots = dslots.as<uint64_t>();
    p.ws = ws.as<unsigned char>();
    p.arena = arena.p;
    p.cap = arena.bytes / elem;
    p.used = &dctl.as<Ctl>()->used;
    p.ctr = dctl.as<Ctl>()->ctr;
    const uint32_t grid = std::max(p.nslot_l, (p.nslot_s + kWarps - 1) / kWarps);
    AHX_CUDA(cplx ? launch_zaca(p, grid, H->stream) : launch_aca(p, grid, H->stream));
    std::vector<AcaResult> res(all.size());
    AHX_CUDA(cudaMemcpyAsync(res.data(), dres.p, res.size() * sizeof(AcaResult), cudaMemcpyDeviceToHost, H->stream));
    AHX_CUDA(cudaStreamSynchronize(H->stream));
    std::vector<AcaTask> retry;
    uint64_t end = elems, more = 0;
    for (size_t q = 0; q < all.size(); ++q) {
      const AcaTask& t = all[q];
      const AcaResult& r = res[q];
      const uint64_t size = (uint64_t)r.kt * ((uint64_t)t.n1 + t.n2);
      // an overflow at the full capacity cannot happen (kcap_limit); were it
      // to, the leaf is treated as an ACA failure so that the loop ends
      if (r.status == kAcaOverflow && t.kcap < kcap_limit(t.kmax)) {
        AcaTask u = t;
        u.kcap = std::min(kcap_limit(t.kmax), std::max(t.kcap * 4, 16u));
        retry.push_back(u);
        H->stat_retries++;
      } else if (r.status == kAcaNoSpace) {  // the arena was estimated too small
        retry.push_back(t);
        more += size;
      } else if (r.status != kAcaOk) {
        dense.push_back(t.leaf);
      } else {
        aca_rank[t.leaf] = (int32_t)r.k_aca;
        rank[t.leaf] = (int32_t)r.kt;
        if (r.kt == 0) continue;
        offs[t.leaf] = r.off;
        end = std::max(end, r.off + size);
      }
    }
    elems = end;
    if (!retry.empty()) {
      // room for the retried leaves: what they needed, or twice the estimate's 16 columns
      for (const AcaTask& t : retry) more += (uint64_t)(t.n1 + t.n2) * std::min(t.kmax, 32u);
      uint64_t off = 0;
      if ((rc = cplx ? zarena_append(H, more, off) : arena_append(H, more, off))) return rc;
      elems = off;
    }
    retry.insert(retry.end(), later.begin(), later.end());
    tasks.swap(retry);
  }
  return AHX_OK;
}

}  // namespace ahx
