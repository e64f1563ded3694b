// Tiling and device numbering of the tiled fused step (host side).
//
// Per domain:
//   1. elements of each block are grown into compact tiles of <= TE elements
//      (breadth-first over elements that share a global point);
//   2. a point is "complete" when every contribution to it is an
//      unconstrained slot of one tile and it carries no boundary, coupling,
//      source, receiver, Dirichlet or axis term; all other points are halo
//      points;
//   3. device numbering: complete points tile by tile (the inner points of
//      its direct elements column by column across the elements, then the
//      others in ascending reference order), then halo points in ascending
//      reference order;
//   4. slot descriptors give each slot its tile point; edge complete points
//      list the places of their contributions in ascending slot order (the
//      order of DofMap::assemble, dof_map.hpp:123-141);
//   5. halo slots write to a halo buffer whose entries each halo point sums
//      through a CSR in ascending slot order (weights of constrained maps kept).
#include <algorithm>
#include <cstring>
#include <map>
#include <mutex>
#include <numeric>

#include "tiled_path.cuh"

namespace insem_b200 {

void set_constant_basis_ng2(const float*, const float*, const float*);
void set_constant_basis_ng3(const float*, const float*, const float*);
void set_constant_basis_ng4(const float*, const float*, const float*);
void set_constant_basis_ng5(const float*, const float*, const float*);
void set_constant_basis_ng6(const float*, const float*, const float*);
void set_constant_basis_ng7(const float*, const float*, const float*);
void set_constant_basis_ng8(const float*, const float*, const float*);
void set_constant_basis_ng9(const float*, const float*, const float*);

namespace {
// What each device's constant basis holds per ngll.  Solves of one ngll share
// the bank: D and w2 are written by the first solve and must agree after; the
// GLJ matrix is written by the first solve that has axial elements and never
// cleared (a solve without it does not read it).  So a bank is written at most
// once per part, never while kernels of that ngll that read the part run.
struct BasisBank {
  std::vector<float> D, Dj, w2;
};
std::mutex g_basis_mutex;
std::map<std::pair<int, int>, BasisBank> g_basis;  // (device, ngll)

void write_basis(int ngll, const float* D, const float* Dj, const float* w2) {
  switch (ngll) {
    case 2: set_constant_basis_ng2(D, Dj, w2); break;
    case 3: set_constant_basis_ng3(D, Dj, w2); break;
    case 4: set_constant_basis_ng4(D, Dj, w2); break;
    case 5: set_constant_basis_ng5(D, Dj, w2); break;
    case 6: set_constant_basis_ng6(D, Dj, w2); break;
    case 7: set_constant_basis_ng7(D, Dj, w2); break;
    case 8: set_constant_basis_ng8(D, Dj, w2); break;
    case 9: set_constant_basis_ng9(D, Dj, w2); break;
    default: check_ngll(ngll);
  }
}
}  // namespace

void set_constant_basis(int ngll, const std::vector<float>& D, const std::vector<float>& Dj,
                        const std::vector<float>& w2) {
  check_ngll(ngll);
  int device = 0;
  CUDA_CHECK(cudaGetDevice(&device));
  std::lock_guard<std::mutex> lk(g_basis_mutex);
  BasisBank& bank = g_basis[{device, ngll}];
  if (bank.D.empty()) {
    write_basis(ngll, D.data(), nullptr, w2.data());
    bank.D = D;
    bank.w2 = w2;
  } else {
    INSEM_REQUIRE(bank.D == D && bank.w2 == w2, INSEM_CUDA_ERR_INVALID,
                  "solves of one ngll must share the GLL basis (D, w_i w_j)");
  }
  if (!Dj.empty()) {
    if (bank.Dj.empty()) {
      write_basis(ngll, nullptr, Dj.data(), nullptr);
      bank.Dj = Dj;
    } else {
      INSEM_REQUIRE(bank.Dj == Dj, INSEM_CUDA_ERR_INVALID, "solves of one ngll must share the GLJ derivative matrix");
    }
  }
}

void launch_tiles(int ngll, const TileLaunch& a) {
  switch (ngll) {
    case 2: launch_tiles_ng2(a); break;
    case 3: launch_tiles_ng3(a); break;
    case 4: launch_tiles_ng4(a); break;
    case 5: launch_tiles_ng5(a); break;
    case 6: launch_tiles_ng6(a); break;
    case 7: launch_tiles_ng7(a); break;
    case 8: launch_tiles_ng8(a); break;
    case 9: launch_tiles_ng9(a); break;
    default: check_ngll(ngll);
  }
}

namespace {
std::mutex g_tile_mutex;
std::map<int, int> g_tile_table;  // key (ngll, kind, elastic, m) -> elements per tile
int tile_key(int ngll, int kind, bool elastic, int m) { return ((ngll * 4 + kind) * 2 + (elastic ? 1 : 0)) * 2 + m; }
}  // namespace

void set_tile_elements(int ngll, int kind, bool elastic, int m, int te) {
  check_ngll(ngll);
  INSEM_REQUIRE(te <= 64, INSEM_CUDA_ERR_INVALID, "more tile elements than a tile may have");
  std::lock_guard<std::mutex> lk(g_tile_mutex);
  if (te <= 0) g_tile_table.erase(tile_key(ngll, kind, elastic, m));
  else g_tile_table[tile_key(ngll, kind, elastic, m)] = te;
}

int choose_tile_elements(int ngll, int kind, bool elastic, int m, int requested) {
  check_ngll(ngll);
  if (requested <= 0) {
    std::lock_guard<std::mutex> lk(g_tile_mutex);
    const auto it = g_tile_table.find(tile_key(ngll, kind, elastic, m));
    if (it != g_tile_table.end()) requested = it->second;
  }
  return requested > 0 ? std::min(requested, kTileLanes) : kTileLanes;
}

void tile_batch(int ngll, const TileBatchLaunch& a, bool launch) {
  switch (ngll) {
    case 2: tile_batch_ng2(a, launch); break;
    case 3: tile_batch_ng3(a, launch); break;
    case 4: tile_batch_ng4(a, launch); break;
    case 5: tile_batch_ng5(a, launch); break;
    case 6: tile_batch_ng6(a, launch); break;
    case 7: tile_batch_ng7(a, launch); break;
    case 8: tile_batch_ng8(a, launch); break;
    case 9: tile_batch_ng9(a, launch); break;
    default: check_ngll(ngll);
  }
}

namespace {
uint32_t bits_of(float v) {
  uint32_t b;
  std::memcpy(&b, &v, sizeof b);
  return b;
}
}  // namespace

BlockDev TiledDomain::BlockTiles::view() const {
  BlockDev v;
  v.kind = kind;
  v.m = m;
  v.n = n;
  v.metric = data.get();
  v.coef0 = coef0.get();
  v.coef1 = coef1.get();
  v.axial = axial.get();
  return v;
}

TiledDev TiledDomain::view(int parity) const {
  TiledDev t;
  t.ng = ng;
  t.n_complete = n_complete;
  t.n_hbuf = n_hbuf;
  t.inv_mass = inv_mass.get();
  t.mass = mass.get();
  t.u_cur = parity ? u1.get() : u0.get();
  t.u_nxt = const_cast<float*>(parity ? u0.get() : u1.get());
  t.v = const_cast<float*>(v.get());
  t.a = const_cast<float*>(a.get());
  t.vn = const_cast<float*>(vn.get());
  t.rs = (rank_cap + 3) & ~3;
  t.sdesc = sdesc.get();
  t.plist = plist.get();
  t.tiles = tiles.get();
  t.halo_tp = halo_tp.get();
  t.hs_slot = hs_slot.get();
  t.hs_dst = hs_dst.get();
  t.mdst_off = mdst_off.get();
  t.mdst = mdst.get();
  t.cs_slot = cs_slot.get();
  t.cs_row = cs_row.get();
  t.row_dofs = rows_dofs.get();
  t.row_w = rows_w.get();
  t.hbuf = const_cast<float*>(hbuf.get());
  return t;
}

HaloDev TiledDomain::halo_view() const {
  HaloDev h;
  h.n = n_halo;
  h.off = h_off.get();
  h.w = weighted ? h_w.get() : nullptr;
  h.spec = h_spec.get();
  h.rec = h_rec.get();
  h.src_which = src_which.get();
  h.src_coef = src_coef.get();
  h.cpl = h_cpl.get();
  h.abs_coef = abs_coef_d.get();
  return h;
}

// The coupling entries' partner points (device numbering of the other domain)
// and coefficients, by entry of the interface.
void TiledDomain::set_partners(const std::vector<int32_t>& partner, const std::vector<float>& cx,
                               const std::vector<float>& cz) {
  std::vector<CouplingEntry> e(std::max<std::size_t>(cpl_entry.size(), 1), CouplingEntry{0, 0.0f, 0.0f, 0});
  for (std::size_t q = 0; q < cpl_entry.size(); ++q)
    e[q] = CouplingEntry{partner[cpl_entry[q]], cx[cpl_entry[q]], cz[cpl_entry[q]], 0};
  h_cpl.upload(e);
}

void TiledDomain::build(const insem_cuda_domain& d, int ngll, int te, const SpecialTerms& sp,
                        const std::vector<float>& abs_coef_host) {
  medium = d.medium;
  ncomp = d.ncomp;
  m = d.azimuthal_order;
  this->te = te;
  ng = d.dofs.n_global;  // reference count while building; the padded stride at the end
  ng_ref = ng;
  npe = ngll * ngll;
  n_elements = d.dofs.n_elements;
  const std::size_t n_slots = static_cast<std::size_t>(n_elements) * npe;
  // the maps are read where they are: the domain's upload has checked them
  const int32_t *l2g = d.dofs.l2g, *t_off = d.dofs.t_offsets, *t_slots = d.dofs.t_slots;
  weighted = d.dofs.n_rows > 0 && d.dofs.t_weights != nullptr;
  const double* t_w = d.dofs.t_weights;

  // special points
  std::vector<char> special(ng, 0);
  for (const auto& kv : sp.sources) special[kv.first] = 1;
  for (const auto& kv : sp.coupling) special[kv.first] = 1;
  for (const auto& kv : sp.absorbing) special[kv.first] = 1;
  for (const auto& kv : sp.zero) special[kv.first] = 1;
  for (int32_t g : sp.receivers) special[g] = 1;

  // 1. tiles per block
  std::vector<int32_t> eblock(n_elements, -1), epos(n_elements, -1);
  for (int b = 0; b < d.n_blocks; ++b)
    for (int q = 0; q < d.blocks[b].n_elements; ++q) {
      const int32_t e = d.blocks[b].elements[q];
      INSEM_REQUIRE(e >= 0 && e < n_elements && eblock[e] < 0, INSEM_CUDA_ERR_INVALID, "block elements overlap");
      eblock[e] = b;
      epos[e] = q;
    }
  std::vector<int32_t> tile_of(n_elements, -1), stamp(n_elements, -1);
  std::vector<std::vector<int32_t>> tile_elems;
  std::vector<int32_t> tile_block;
  blocks.clear();
  blocks.resize(d.n_blocks);
  std::vector<int32_t> queue;
  for (int b = 0; b < d.n_blocks; ++b) {
    blocks[b].kind = d.blocks[b].kind;
    blocks[b].m = d.blocks[b].azimuthal_order;
    blocks[b].n = d.blocks[b].n_elements;
    blocks[b].tile0 = static_cast<int>(tile_elems.size());
    for (int q = 0; q < d.blocks[b].n_elements; ++q) {
      const int32_t seed = d.blocks[b].elements[q];
      if (tile_of[seed] >= 0) continue;
      const int32_t t = static_cast<int32_t>(tile_elems.size());
      tile_elems.emplace_back();
      tile_block.push_back(b);
      auto& te_list = tile_elems.back();
      te_list.reserve(te);
      queue.clear();
      queue.push_back(seed);
      stamp[seed] = t;
      std::size_t head = 0;
      while (head < queue.size() && static_cast<int>(te_list.size()) < te) {
        const int32_t e = queue[head++];
        tile_of[e] = t;
        te_list.push_back(e);
        for (int k = 0; k < npe; ++k) {
          const int32_t g = l2g[static_cast<std::size_t>(e) * npe + k];
          if (g < 0) continue;
          for (int32_t s = t_off[g]; s < t_off[g + 1]; ++s) {
            const int32_t e2 = t_slots[s] / npe;
            if (eblock[e2] == b && tile_of[e2] < 0 && stamp[e2] != t) {
              stamp[e2] = t;
              queue.push_back(e2);
            }
          }
        }
      }
      std::sort(te_list.begin(), te_list.end());
    }
    blocks[b].ntiles = static_cast<int>(tile_elems.size()) - blocks[b].tile0;
  }
  n_tiles = static_cast<int>(tile_elems.size());

  // 2. point classification
  std::vector<int32_t> owner(ng, -1);
  for (int32_t g = 0; g < ng; ++g) {
    if (special[g]) continue;
    int32_t t = -2;
    bool ok = true;
    for (int32_t s = t_off[g]; s < t_off[g + 1] && ok; ++s) {
      const int32_t slot = t_slots[s];
      if (l2g[slot] != g) ok = false;
      const int32_t tt = tile_of[slot / npe];
      if (t == -2) t = tt;
      else if (tt != t) ok = false;
    }
    if (ok && t >= 0) owner[g] = t;
  }
  // 3. device numbering.  A direct element's inner points each belong to it
  // alone and are complete: the tile's direct elements come first (its first
  // lanes), and their inner points are numbered column by column across them.
  const int ni = ngll > 2 ? ngll - 2 : 0;
  std::vector<int32_t> lane_of(n_elements, -1), n_direct(n_tiles, 0);
  std::vector<char> inner(ng, 0);
  auto inner_slot = [&](int q) { return (q % ni + 1) * ngll + q / ni + 1; };  // q = (i - 1) ni + j - 1
  for (int t = 0; t < n_tiles; ++t) {
    auto direct = [&](int32_t e) {
      for (int q = 0; q < ni * ni; ++q) {
        const int32_t g = l2g[static_cast<std::size_t>(e) * npe + inner_slot(q)];
        if (g < 0 || owner[g] != t || t_off[g + 1] - t_off[g] != 1) return false;
      }
      return true;
    };
    auto& list = tile_elems[t];
    n_direct[t] = static_cast<int32_t>(std::stable_partition(list.begin(), list.end(), direct) - list.begin());
    for (std::size_t q = 0; q < list.size(); ++q) lane_of[list[q]] = static_cast<int32_t>(q);
    for (int32_t l = 0; l < n_direct[t]; ++l)
      for (int q = 0; q < ni * ni; ++q) inner[l2g[static_cast<std::size_t>(list[l]) * npe + inner_slot(q)]] = 1;
  }
  std::vector<int32_t> count(n_tiles, 0);  // edge complete points
  for (int32_t g = 0; g < ng; ++g)
    if (owner[g] >= 0 && !inner[g]) ++count[owner[g]];
  n_halo = ng;
  for (int t = 0; t < n_tiles; ++t) n_halo -= n_direct[t] * ni * ni + count[t];
  auto up4 = [](int32_t x) { return (x + 3) & ~3; };
  const TileNumbers numbers = number_tiles(count, ni, n_halo);
  const auto &cbeg = numbers.cbeg, &ebeg = numbers.ebeg;
  n_complete = numbers.n_complete;
  perm.assign(ng, -1);
  {
    for (int t = 0; t < n_tiles; ++t)
      for (int q = 0; q < ni * ni; ++q)
        for (int32_t l = 0; l < n_direct[t]; ++l)
          perm[l2g[static_cast<std::size_t>(tile_elems[t][l]) * npe + inner_slot(q)]] = cbeg[t] + q * kTileLanes + l;
    std::vector<int32_t> fill(ebeg);
    std::vector<char> last(ng, 0);
    for (int32_t g : sp.coupled) last[g] = 1;
    int32_t h = n_complete;
    for (int32_t g = 0; g < ng; ++g) {
      if (inner[g] || last[g]) continue;
      perm[g] = owner[g] >= 0 ? fill[owner[g]]++ : h++;
    }
    for (int32_t g : sp.coupled) perm[g] = h++;
  }
  const int32_t ng_dev = numbers.stride;
  const int W = kTileLanes;

  // 4. per tile: tile points, descriptors, halo and constrained slots.  The
  // place of slot k of the element in lane l is k * 32 + l.
  std::vector<TileHdr> hdr(n_tiles);
  std::vector<uint16_t> desc(static_cast<std::size_t>(std::max(n_tiles, 1)) * npe * W, 0);
  std::vector<int32_t> htp, hslot, cslot, crow;
  std::vector<int32_t> hpos_of_slot(n_slots, -1);
  std::vector<int32_t> tpi(ng_dev, -1), tpi_stamp(ng, -1);
  int32_t hb = 0, pl_running = 0;
  std::vector<int32_t> hp;
  for (int b = 0; b < d.n_blocks; ++b) {
    for (int t = blocks[b].tile0; t < blocks[b].tile0 + blocks[b].ntiles; ++t) {
      TileHdr& th = hdr[t];
      th.tb = t - blocks[b].tile0;
      th.ne = static_cast<int32_t>(tile_elems[t].size());
      th.nd = n_direct[t];
      th.cbeg = cbeg[t];
      th.ebeg = ebeg[t];
      th.nc = count[t];  // [ebeg + nc, cbeg of the next tile) is padding
      th.hl_off = static_cast<int32_t>(htp.size());
      th.hs_off = static_cast<int32_t>(hslot.size());
      th.cs_off = static_cast<int32_t>(cslot.size());
      th.pl_off = pl_running;
      pl_running += up4(th.nc);
      // halo points read by the tile; they follow the edge points' padded range
      hp.clear();
      for (int32_t e : tile_elems[t])
        for (int k = 0; k < npe; ++k) {
          const int32_t g = l2g[static_cast<std::size_t>(e) * npe + k];
          if (g >= 0 && owner[g] != t && tpi_stamp[g] != t) {
            tpi_stamp[g] = t;
            hp.push_back(perm[g]);
          }
        }
      std::sort(hp.begin(), hp.end());
      htp.insert(htp.end(), hp.begin(), hp.end());
      th.ntp = th.nc + static_cast<int32_t>(hp.size());
      for (std::size_t q = 0; q < hp.size(); ++q) tpi[hp[q]] = up4(th.nc) + static_cast<int32_t>(q);
      int32_t nh = 0;
      for (int el = 0; el < th.ne; ++el) {
        const int32_t e = tile_elems[t][el];
        for (int k = 0; k < npe; ++k) {
          const std::size_t s = static_cast<std::size_t>(e) * npe + k;
          const int32_t g = l2g[s];
          const int32_t place = k * W + el;
          uint32_t dsc = 0;
          if (g >= 0) {
            if (!inner[g]) {
              const int32_t pg = perm[g];
              const int32_t p = owner[g] == t ? pg - th.ebeg : tpi[pg];
              INSEM_REQUIRE(p >= 0 && p < static_cast<int32_t>(kSlotConstrained), INSEM_CUDA_ERR_UNSUPPORTED,
                            "tile has too many points");
              dsc = static_cast<uint32_t>(p);
              if (owner[g] != t) {
                hpos_of_slot[s] = hb + nh++;
                hslot.push_back(place);
              }
            }
          } else {
            dsc = kSlotConstrained;
            cslot.push_back(place);
            crow.push_back(-1 - g);
            hpos_of_slot[s] = hb + nh++;
            hslot.push_back(place);
          }
          desc[static_cast<std::size_t>(t) * npe * W + place] = static_cast<uint16_t>(dsc);
        }
      }
      th.nhs = nh;
      th.ncs = static_cast<int32_t>(cslot.size()) - th.cs_off;
      hb += nh;
    }
  }
  const int32_t n_entries = hb;
  tp_cap = 4;
  nc_cap = 4;
  for (const auto& th : hdr) {
    tp_cap = std::max(tp_cap, up4(th.nc) + th.ntp - th.nc);
    nc_cap = std::max(nc_cap, up4(th.nc));
  }
  tp_cap = up4(tp_cap);  // keeps every component row of the staged u 16-byte aligned

  // 5. place lists of the edge complete points, in ascending slot order
  rank_cap = 1;
  for (int32_t g = 0; g < ng; ++g)
    if (owner[g] >= 0 && !inner[g]) rank_cap = std::max<int32_t>(rank_cap, t_off[g + 1] - t_off[g]);
  const int rs = (rank_cap + 3) & ~3;
  std::vector<uint16_t> lists(static_cast<std::size_t>(std::max(pl_running, 4)) * rs, static_cast<uint16_t>(kLastPlace));
  for (int32_t g = 0; g < ng; ++g) {
    if (owner[g] < 0 || inner[g]) continue;
    const TileHdr& th = hdr[owner[g]];
    const std::size_t at = static_cast<std::size_t>(th.pl_off + perm[g] - th.ebeg) * rs;
    for (int32_t s = t_off[g]; s < t_off[g + 1]; ++s) {
      const int32_t slot = t_slots[s], e = slot / npe;
      uint32_t place = static_cast<uint32_t>((slot - e * npe) * W + lane_of[e]);
      if (s + 1 == t_off[g + 1]) place |= kLastPlace;
      lists[at + (s - t_off[g])] = static_cast<uint16_t>(place);
    }
  }

  // 6. halo CSR and special records (device order of halo points)
  std::vector<int32_t> hoff{0}, hpos, hspec(n_halo, -1), swhich;
  std::vector<HaloRec> recs;
  std::vector<float> hw, scoef;
  cpl_entry.clear();
  hoff.reserve(static_cast<std::size_t>(n_halo) + 1);
  hpos.reserve(n_entries);
  std::vector<int32_t> halo_orig(n_halo);
  for (int32_t g = 0; g < ng; ++g)
    if (owner[g] < 0) halo_orig[perm[g] - n_complete] = g;
  for (int32_t h = 0; h < n_halo; ++h) {
    const int32_t g = halo_orig[h];
    for (int32_t s = t_off[g]; s < t_off[g + 1]; ++s) {
      const int32_t pos = hpos_of_slot[t_slots[s]];
      INSEM_REQUIRE(pos >= 0, INSEM_CUDA_ERR_INVALID, "halo contribution without a halo-buffer entry");
      hpos.push_back(pos);
      if (weighted) hw.push_back(static_cast<float>(t_w[s]));
    }
    hoff.push_back(static_cast<int32_t>(hpos.size()));
    if (!special[g]) continue;
    hspec[h] = static_cast<int32_t>(recs.size());
    HaloRec r{static_cast<int32_t>(swhich.size()), 0, static_cast<int32_t>(cpl_entry.size()), 0, -1, 0};
    if (auto it = sp.sources.find(g); it != sp.sources.end())
      for (const auto& [s, cs] : it->second) {
        swhich.push_back(s);
        scoef.insert(scoef.end(), cs.begin(), cs.end());
      }
    r.src1 = static_cast<int32_t>(swhich.size());
    if (auto it = sp.coupling.find(g); it != sp.coupling.end())
      cpl_entry.insert(cpl_entry.end(), it->second.begin(), it->second.end());
    r.cpl1 = static_cast<int32_t>(cpl_entry.size());
    if (auto ia = sp.absorbing.find(g); ia != sp.absorbing.end()) r.abs = ia->second;
    if (auto iz = sp.zero.find(g); iz != sp.zero.end()) r.zero = iz->second;
    recs.push_back(r);
  }

  // Places of the halo-buffer entries in hbuf: hbuf holds each halo point's
  // contributions in its ascending slot order, point after point (the list
  // hoff indexes), so the halo kernel reads them contiguously.  An entry has
  // one place, unless it is a constrained slot feeding several parent
  // points; those entries keep a list of places.
  n_hbuf = static_cast<int32_t>(hpos.size());
  std::vector<int32_t> ecount(n_entries, 0);
  for (int32_t e : hpos) ++ecount[e];
  std::vector<int32_t> hdst(n_entries, 0), moff{0}, mlist;
  {
    for (int32_t e = 0; e < n_entries; ++e) {
      if (ecount[e] == 1) continue;
      hdst[e] = -1 - (static_cast<int32_t>(moff.size()) - 1);
      moff.push_back(moff.back() + ecount[e]);
    }
    mlist.resize(moff.back());
    std::vector<int32_t> fill(moff.begin(), moff.end() - 1);
    for (int32_t q = 0; q < n_hbuf; ++q) {
      const int32_t e = hpos[q];
      if (ecount[e] == 1) hdst[e] = q;
      else mlist[fill[-1 - hdst[e]]++] = q;
    }
  }

  // 7. uploads
  sdesc.upload(desc);
  plist.upload(lists);
  tiles.upload(hdr);
  host_tiles = std::move(hdr);
  halo_tp.upload(htp.empty() ? std::vector<int32_t>{0} : htp);
  hs_slot.upload(hslot.empty() ? std::vector<int32_t>{0} : hslot);
  hs_dst.upload(hdst.empty() ? std::vector<int32_t>{0} : hdst);
  mdst_off.upload(moff);
  mdst.upload(mlist.empty() ? std::vector<int32_t>{0} : mlist);
  cs_slot.upload(cslot.empty() ? std::vector<int32_t>{0} : cslot);
  hbuf.resize(static_cast<std::size_t>(ncomp) * std::max(n_hbuf, 1));
  h_off.upload(hoff);
  if (weighted) h_w.upload(hw.empty() ? std::vector<float>{0.0f} : hw);
  h_spec.upload(hspec.empty() ? std::vector<int32_t>{0} : hspec);
  src_which.upload(swhich.empty() ? std::vector<int32_t>{0} : swhich);
  src_coef.upload(scoef.empty() ? std::vector<float>{0.0f} : scoef);
  h_rec.upload(recs.empty() ? std::vector<HaloRec>(1, HaloRec{0, 0, 0, 0, -1, 0}) : recs);
  abs_coef_d.upload(abs_coef_host.empty() ? std::vector<float>{0.0f} : abs_coef_host);
  // constraint rows with device-numbered dofs (weights rounded as the gather does)
  {
    const auto ro = host_vec(d.dofs.row_offsets, static_cast<std::size_t>(d.dofs.n_rows) + 1);
    const std::size_t nrd = ro.empty() ? 0 : static_cast<std::size_t>(ro.back());
    auto rd = host_vec(d.dofs.row_dofs, nrd);
    const auto rw = host_vec(d.dofs.row_weights, nrd);
    for (auto& g : rd) g = perm[g];
    std::vector<int2> crange;
    crange.reserve(crow.size());
    for (int32_t r : crow) crange.push_back(int2{ro[r], ro[r + 1]});
    cs_row.upload(crange.empty() ? std::vector<int2>{int2{0, 0}} : crange);
    rows_off.upload(ro.empty() ? std::vector<int32_t>{0} : ro);
    rows_dofs.upload(rd.empty() ? std::vector<int32_t>{0} : rd);
    rows_w.upload(rw.empty() ? std::vector<float>{0.0f} : std::vector<float>(rw.begin(), rw.end()));
  }
  // mass in device numbering
  host_mass.assign(ng_dev, 0.0f);
  std::vector<float> im(ng_dev, 0.0f);
  for (int32_t g = 0; g < ng; ++g) {
    host_mass[perm[g]] = d.mass[g];
    im[perm[g]] = d.inv_mass[g];
  }
  mass.upload(host_mass);
  inv_mass.upload(im);
  const std::size_t nf = static_cast<std::size_t>(ncomp) * ng_dev;
  for (auto* buf : {&u0, &u1, &v, &a, &vn}) {
    buf->resize(nf);
    buf->zero();
  }
  // element data of every block, element-minor by tile; one material per
  // element: the tile kernels read one coefficient pair per element
  auto separable = [&](const insem_cuda_block& in) {
    if (in.kind != INSEM_AXISYM) return false;
    for (std::size_t e = 0; e < static_cast<std::size_t>(in.n_elements); ++e) {
      const float *m = in.metric + e * npe * 5, *r = in.r + e * npe;
      for (int k = 1; k < npe; ++k) {
        for (int c : {0, 2, 3})
          if (bits_of(m[k * 5 + c]) != bits_of(m[c])) return false;
        if (bits_of(r[k]) != bits_of(r[k % ngll])) return false;
      }
    }
    return true;
  };
  for (int b = 0; b < d.n_blocks; ++b) {
    BlockTiles& bt = blocks[b];
    const insem_cuda_block& in = d.blocks[b];
    const bool sep = separable(in), axi = in.kind == INSEM_AXISYM;
    bool off_axis = sep && medium == INSEM_ELASTIC;
    for (std::size_t q = 0; off_axis && q < static_cast<std::size_t>(in.n_elements) * npe; ++q)
      off_axis = in.r[q] != 0.0f && !in.axial[q / npe];
    const int kind = off_axis ? kAxisymOffAxis : sep ? kAxisymSeparable : in.kind, na = tile_arrays(kind);
    bt.kind = kind;
    const bool el = medium == INSEM_ELASTIC, staged = tile_data_staged(kind);
    const std::size_t per_tile = static_cast<std::size_t>(tile_data_floats(kind, ngll));
    std::vector<float> data(per_tile * bt.ntiles, 0.0f), c0(static_cast<std::size_t>(W) * bt.ntiles, 0.0f);
    std::vector<float> c1(el ? c0.size() : 0, 0.0f);
    std::vector<uint8_t> axial(axi ? c0.size() : 0, 0);
    for (int tb = 0; tb < bt.ntiles; ++tb) {
      const auto& list = tile_elems[bt.tile0 + tb];
      for (std::size_t l = 0; l < list.size(); ++l) {
        const std::size_t o = static_cast<std::size_t>(epos[list[l]]), p0 = o * npe, at = static_cast<std::size_t>(tb) * W + l;
        float* out = data.data() + per_tile * tb;
        if (sep) {
          for (int k = 0; k < npe; ++k) {
            const int p = k * W + static_cast<int>(l);
            out[tile_data_at(kind, npe, 0, p)] = in.wr[p0 + k];
            out[tile_data_at(kind, npe, 1, p)] = in.hoop[p0 + k];
            out[tile_data_at(kind, npe, 2, p)] = in.metric[(p0 + k) * 5 + 1];
          }
          float* lane = out + tile_staged_floats(kind, ngll) + l;
          for (int c = 0; c < 3; ++c) lane[static_cast<std::size_t>(c) * W] = in.metric[p0 * 5 + (c == 0 ? 0 : c + 1)];
          for (int i = 0; i < ngll; ++i) lane[static_cast<std::size_t>(3 + i) * W] = in.r[p0 + i];
        } else if (staged) {
          for (int k = 0; k < npe; ++k) {
            auto put = [&](int c, float v) { out[tile_data_at(kind, npe, c, k * W + static_cast<int>(l))] = v; };
            for (int c = 0; c < (axi ? 4 : 5); ++c) put(c, in.metric[(p0 + k) * 5 + c]);
            if (axi) {
              put(4, in.wr[p0 + k]);
              put(5, in.hoop[p0 + k]);
              put(6, in.r[p0 + k]);
            }
          }
        } else {
          for (int c = 0; c < na; ++c) out[static_cast<std::size_t>(c) * W + l] = in.metric[o * na + c];
        }
        c0[at] = in.coef0[p0];
        if (el) c1[at] = in.coef1[p0];
        if (axi) {
          axial[at] = in.axial[o];
          bt.any_axial |= in.axial[o] != 0;
        }
        for (int k = 1; k < npe; ++k) {
          const bool same = bits_of(in.coef0[p0 + k]) == bits_of(c0[at]) && (!el || bits_of(in.coef1[p0 + k]) == bits_of(c1[at]));
          INSEM_REQUIRE(same, INSEM_CUDA_ERR_UNSUPPORTED,
                        "material coefficients vary inside an element; the tiled path takes one material per "
                        "element (options.path = 1 takes per-point coefficients)");
        }
      }
    }
    bt.data.upload(data);
    bt.coef0.upload(c0);
    bt.coef1.upload(c1);
    bt.axial.upload(axial);
  }
  ng = ng_dev;  // from here on the component stride of the device arrays
}

}  // namespace insem_b200
