// Host plan of the gather kernels (gather.h) and the launches of commutator_122 by pair groups.
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstring>

#include "engine.h"
#include "kernels.h"
#include "pair_groups.h"

using namespace imsrg;

// The FP64 commutator's use of the plan: wanted by the size of the basis, and left for good where the device has no room
// for its tables (the kernels that take a thread per element need none).
imsrg_status Ctx::gather_prepare_fp64(bool& groups) {
  groups = L.slab >= kGatherMinSlab && !gather_no_room;
  if (!groups) return IMSRG_OK;
  const imsrg_status s = gather_prepare(true);
  if (s != IMSRG_ERR_OUT_OF_MEMORY) return s;
  cudaGetLastError();
  gather_release();
  gather_no_room = true;
  groups = false;
  return IMSRG_OK;
}

imsrg_status Ctx::gather_prepare(bool optional) {
  if (gp.state) return IMSRG_OK;
  gather_release();  // what a failed preparation left
  const Layout& l = L;
  if (l.JM + 1 > 26) {
    gp.why = "mixed recoupling supports 2j <= 25 (eMax <= 12)";
    gp.state = -1;
    return IMSRG_OK;
  }
  if (l.wcc_size >= (int64_t)1 << 31) {
    gp.why = "cross-coupled matrices too large for 32-bit positions";
    gp.state = -1;
    return IMSRG_OK;
  }
  PairGroups pg;
  build_pair_groups(pg, l);
  gp.why = build_g122_plan(l, pg, gp.g122);
  if (!gp.why.empty()) {
    gp.state = -1;
    return IMSRG_OK;
  }
  gp.nspb = pg.nspb;
  // ---- recoupling quadruples: bra (i<=j) of class c1, ket (k<=l) of class c2, with
  //      c1 < c2, or c1 == c2 and (i,j) <= (k,l) (the unique stored elements), matching
  //      2Tz and parity and sharing at least one J
  {
    const int N = l.N;
    std::vector<std::vector<int>> by_tp(4);  // orbits grouped by (tz, l parity)
    for (int o = 0; o < N; ++o) by_tp[((l.tz[o] + 1) / 2) * 2 + (l.ll[o] & 1)].push_back(o);
    for (int i = 0; i < N; ++i)
      for (int k = 0; k < N; ++k)
        for (int ll2 = k; ll2 < N; ++ll2) {
          const int tzj = l.tz[k] + l.tz[ll2] - l.tz[i];
          if (tzj != -1 && tzj != 1) continue;
          const int par = ((l.ll[k] + l.ll[ll2] - l.ll[i]) % 2 + 2) % 2;
          const int c2 = l.con[k] + l.con[ll2];
          const int kl_lo = std::abs(l.jj[k] - l.jj[ll2]), kl_hi = l.jj[k] + l.jj[ll2];
          for (int j : by_tp[((tzj + 1) / 2) * 2 + par]) {
            if (j < i) continue;
            const int c1 = l.con[i] + l.con[j];
            if (c1 > c2) continue;
            if (c1 == c2 && (i > k || (i == k && j > ll2))) continue;
            const int lo = std::max(std::abs(l.jj[i] - l.jj[j]), kl_lo), hi = std::min(l.jj[i] + l.jj[j], kl_hi);
            if (lo > hi) continue;
            gp.quads.push_back((uint64_t)i | ((uint64_t)j << 16) | ((uint64_t)k << 32) | ((uint64_t)ll2 << 48));
          }
        }
    // within the quadruples of one orbit i, by (jj, jk, jl): neighbouring threads then share their J and J' ranges and
    // 6j rows, so a warp's loops run with its lanes in step (the X rows read for one i are the same in any order)
    auto shape = [&](uint64_t qd) {
      return (l.jj[(qd >> 16) & 0xFFFF] * 64 + l.jj[(qd >> 32) & 0xFFFF]) * 64 + l.jj[(qd >> 48) & 0xFFFF];
    };
    for (size_t a = 0; a < gp.quads.size();) {
      size_t b = a;
      while (b < gp.quads.size() && (gp.quads[b] & 0xFFFF) == (gp.quads[a] & 0xFFFF)) ++b;
      std::stable_sort(gp.quads.begin() + a, gp.quads.begin() + b,
                       [&](uint64_t x, uint64_t y) { return shape(x) < shape(y); });
      a = b;
    }
  }
  cudaDeviceGetAttribute(&gp.num_sms, cudaDevAttrMultiProcessorCount, device);
  const std::vector<int> xcol = build_xcol(l);
  struct Piece {
    const void* src;
    size_t bytes;
    const void** dst;
  };
  const Piece pieces[] = {
      {pg.spb_start.data(), sizeof(int) * pg.spb_start.size(), (const void**)&gp.groups.spb_start},
      {pg.spb_n.data(), sizeof(int) * pg.spb_n.size(), (const void**)&gp.groups.spb_n},
      {pg.spb_orb.data(), sizeof(int) * pg.spb_orb.size(), (const void**)&gp.groups.spb_orb},
      {pg.grp_b1.data(), sizeof(int) * pg.grp_b1.size(), (const void**)&gp.groups.grp_b1},
      {pg.grp_b2.data(), sizeof(int) * pg.grp_b2.size(), (const void**)&gp.groups.grp_b2},
      {pg.blk_off.data(), sizeof(int) * pg.blk_off.size(), (const void**)&gp.groups.blk_off},
      {gp.g122.codes.data(), sizeof(unsigned) * gp.g122.codes.size(), (const void**)&gp.d_codes},
      {gp.quads.data(), sizeof(uint64_t) * gp.quads.size(), (const void**)&gp.d_quads},
      {xcol.data(), sizeof(int) * xcol.size(), (const void**)&gp.d_xcol},
      {nullptr, sizeof(G122Task) * gp.g122.all.size(), (const void**)&gp.d_tasks},
      {nullptr, sizeof(int2) * gp.g122.all.size(), (const void**)&gp.d_items},
      {nullptr, sizeof(int) * 2, (const void**)&gp.d_counter},
      {nullptr, sizeof(double2) * (size_t)std::max(pg.nblk2, 1), (const void**)&gp.fb}};
  size_t total = 0;
  for (const Piece& p : pieces) total += (p.bytes + 255) & ~size_t(255);
  if (optional && !room_for(total)) return IMSRG_ERR_OUT_OF_MEMORY;
  CK_TC(alloc(&gp.d_mem, std::max<size_t>(total, 256), "cudaMalloc(gather plan)"));
  char* at = static_cast<char*>(gp.d_mem);
  for (const Piece& p : pieces) {
    *p.dst = at;
    if (p.src && p.bytes)
      CK_TC(cuda(cudaMemcpyAsync(at, p.src, p.bytes, cudaMemcpyHostToDevice, stream), "cudaMemcpyAsync(gather plan)"));
    at += (p.bytes + 255) & ~size_t(255);
  }
  CK_TC(cuda(cudaMemsetAsync(gp.d_counter, 0, sizeof(int) * 2, stream), "memset(122 counter)"));
  CK_TC(cuda(cudaStreamSynchronize(stream), "cudaStreamSynchronize(gather plan)"));
  // 8 lanes for a task of up to 32 elements while the warps are not all busy, up to 64 in larger bases (FP32: eMax 4 25 ->
  // 20 us, eMax 7 53 -> 50, eMax 8 91 either way, eMax 10 385 against 399)
  CK_TC(g122_upload(l.slab < (int64_t)1 << 23 ? 32 : 64, 256));
  gp.state = 1;
  return IMSRG_OK;
}

void Ctx::gather_release() {
  if (gp.d_mem) cudaFree(gp.d_mem);
  gp = GatherPlan();
}

// Splits the 122 tasks into [tiny | warp | cta] runs by size, keeping channel order inside
// each run, and uploads the list.  The caps must keep the per-CTA shared memory of the
// 8-lane and warp kernels within the 48 KiB default.
imsrg_status Ctx::g122_upload(int tiny_cap, int small_cap) {
  G122Plan& P = gp.g122;
  const int bt = P.tiny_cap, bw = P.warp_cap;
  const std::string e = g122_partition(P, tiny_cap, small_cap);
  if (!e.empty()) {
    g122_partition(P, bt, bw);  // keep the previous caps
    return fail(IMSRG_ERR_INVALID_ARGUMENT, e);
  }
  if (!P.tasks.empty()) {
    CK_TC(cuda(cudaMemcpyAsync(gp.d_tasks, P.tasks.data(), sizeof(G122Task) * P.tasks.size(),
                               cudaMemcpyHostToDevice, stream), "cudaMemcpyAsync(122 tasks)"));
    if (!P.items.empty())
      CK_TC(cuda(cudaMemcpyAsync(gp.d_items, P.items.data(), sizeof(int2) * P.items.size(),
                                 cudaMemcpyHostToDevice, stream), "cudaMemcpyAsync(122 runs)"));
    CK_TC(cuda(cudaStreamSynchronize(stream), "cudaStreamSynchronize(122 tasks)"));
  }
  CK_TC(cuda(g122_occupancy(P.smem_bytes, gp.per_sm), "occupancy (122)"));
  return IMSRG_OK;
}

// Other caps for a plan in use.  A captured step holds the counts, the grid and the shared memory of the list that is rewritten
// here, in whatever precision it was captured: it goes first.
imsrg_status Ctx::g122_set_caps(int tiny_cap, int small_cap) {
  graph_drop();
  return g122_upload(tiny_cap, small_cap);
}

// commutator_122 on pair-group sub-blocks: RES's rectangular arrays and the upper triangles of its square ones.  In FP64 it
// does nothing unless k_check_mirror finds both operators' lower triangles in line with the upper ones.
template <typename T>
imsrg_status Ctx::c122_groups(const double* Lp, int hL, const double* Rp, int hR, double* RES, int hRES) {
  const G122Plan& P = gp.g122;
  launch_comm122_fb<T>(gp.nspb, stream, D, gp.groups, Lp, hL, Rp, hR, gp.fb, gp.d_counter);
  CK_TC(launched("k_comm122_fb2"));
  const bool f64 = sizeof(T) == sizeof(double);
  if (f64) {  // operators whose lower triangles are not herm times the upper ones are left to k_comm122
    k_check_mirror<<<(int)std::max<size_t>(upd_tiles.size(), 1), 256, 0, stream>>>(D, d_upd_tiles, (int)upd_tiles.size(), Lp, hL,
                                                                                  Rp, hR, gp.d_counter + 1);
    CK_TC(launched("k_check_mirror"));
  }
  // the big tasks, then enough eight-warp CTAs to fill the GPU at the occupancy the shared
  // memory allows (the warps take the runs from the counter)
  const int grid = P.nbig + gp.num_sms * std::max(1, gp.per_sm[f64 ? 1 : 0]);
  launch_comm122<T>(grid, P.smem_bytes * (f64 ? 2 : 1), stream, D, gp.d_tasks, gp.d_items, (int)P.items.size(), P.nbig,
                    gp.d_counter, gp.d_codes, std::max(P.warp_cap, 4 * P.tiny_cap), P.tiny_cap, Lp, hL, Rp, hR, RES, hRES,
                    gp.fb, f64 ? gp.d_counter + 1 : nullptr);
  return launched("k_comm122_sub");
}
template imsrg_status Ctx::c122_groups<float>(const double*, int, const double*, int, double*, int);
template imsrg_status Ctx::c122_groups<double>(const double*, int, const double*, int, double*, int);
