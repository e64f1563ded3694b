// Host-side check of the tile kernels' shared memory against the addresses the
// kernel forms: every kind of the tile kernels (axisymmetric ones with a
// metric kept once and off the axis too), every ngll, component count and
// list length, with capacities of compact, scattered and smallest tiles.
//
// The regions are those of tile_step_body, for the 32 lanes that every tile
// has whatever it holds.  They are followed through its phases:
//   copies    element data, u (and, not late: v, 1/M, place lists) land
//   fluxes    a point's f_xi replace element data of that point only
//   late      v, 1/M and place lists land while f_xi, field rows and axis terms live
//   finish    contributions (over the field rows), lists, v, 1/M, u
// Prints "ok" and exits 0, or prints the first violation and exits 1.
#include <cstdio>
#include <string>
#include <vector>

#include "tiled.cuh"

using namespace insem_b200;

namespace {

struct Region {
  const char* name;
  uint32_t beg, end;
};

int fail(const std::string& what) {
  std::printf("FAIL %s\n", what.c_str());
  return 1;
}

// Byte range [first, last) of the plane or pairs a component's f_xi take, by
// the offsets of Rows<NC, NPE, AT>: pairs [place][2] from 0, the only or third
// component from AT floats on.
struct FluxRows {
  Region pairs, one;
};
FluxRows flux_rows(const TileLayout& L, int kind, int npe, int nc) {
  const uint32_t plane = 4u * kTileLanes * npe;
  const bool staged = tile_data_staged(kind);
  const uint32_t at = staged ? 4u * (tile_arrays(kind) - 1) * npe * kTileLanes : nc >= 2 ? 2 * plane : 0u;
  FluxRows f{{"paired xi fluxes", 0, 0}, {"single xi fluxes", 0, 0}};
  if (nc >= 2) f.pairs = {"paired xi fluxes", L.sfx, L.sfx + 2 * plane};
  if (nc != 2) f.one = {"single xi fluxes", L.sfx + at, L.sfx + at + plane};
  return f;
}

int check(int ng, int kind, int nc, int tp_cap, int nc_cap, int rs, const std::string& id) {
  const int npe = ng * ng;
  const uint32_t plane = 4u * kTileLanes * npe;
  const TileLayout L = TileLayout::make(ng, nc, kind, nc > 1, kTileLanes, tp_cap, nc_cap, rs);
  const uint32_t staged = 4u * tile_staged_floats(kind, ng);
  const uint32_t lists = 2u * ((rs + 3) & ~3) * nc_cap;
  const Region bar{"barriers", L.bar, L.bar + 16};
  const Region elem{"element data", L.metric, L.metric + staged};
  const Region u{"u", L.u, L.u + 4u * nc * tp_cap};
  const Region rows{"field rows", L.su, L.su + plane * nc};
  const Region v{"v", L.v, L.v + 4u * nc * nc_cap};
  const Region im{"1/M", L.im, L.im + 4u * nc_cap};
  const Region pl{"place lists", L.pl, L.pl + lists};
  const Region ax{"axis terms", L.ax, L.ax + (is_axisym(kind) ? 4u * 4u * ng * kTileLanes : 0u)};
  const FluxRows f = flux_rows(L, kind, npe, nc);
  // bulk copies: 16-byte destinations, components at multiples of 16 bytes
  for (const Region* r : {&bar, &elem, &u, &rows, &v, &im, &pl, &ax, &f.pairs, &f.one})
    if (r->end > r->beg && r->beg % 16) return fail(id + ": " + r->name + " not on 16 bytes");
  if (tp_cap % 4 || nc_cap % 4) return fail(id + ": component rows not on 16 bytes");
  std::vector<Region> copies = {bar, elem, u, rows, ax}, late = {bar, u, rows, ax, f.pairs, f.one, v, im, pl},
                      finish = {bar, u, rows, v, im, pl};
  if (!L.late)
    for (const Region& r : {v, im, pl}) copies.push_back(r);
  if (!tile_data_staged(kind)) {  // the fluxes have rows of their own
    copies.push_back(f.pairs);
    copies.push_back(f.one);
  }
  for (const auto* set : {&copies, &late, &finish})
    for (std::size_t a = 0; a < set->size(); ++a) {
      const Region& x = (*set)[a];
      if (x.end > L.total) return fail(id + ": " + x.name + " ends past the total");
      // launches without axial elements allocate up to L.ax only
      if (x.name != ax.name && x.end > L.ax) return fail(id + ": " + x.name + " lies behind the axis terms");
      for (std::size_t b = a + 1; b < set->size(); ++b) {
        const Region& y = (*set)[b];
        if (x.end > x.beg && y.end > y.beg && x.beg < y.end && y.beg < x.end)
          return fail(id + ": " + x.name + " overlaps " + y.name);
      }
    }
  if (!tile_data_staged(kind)) return L.late ? fail(id + ": late copies without staged element data") : 0;
  // staged data: every element value lies inside, each at a place of its own;
  // the f_xi of a point and lane lie inside and on data of that point and lane
  std::vector<int> owner(staged / 4, -1);
  for (int a = 0; a < tile_arrays(kind); ++a)
    for (int p = 0; p < npe * kTileLanes; ++p) {
      const int at = tile_data_at(kind, npe, a, p);
      if (at < 0 || at >= static_cast<int>(owner.size()) || owner[at] >= 0) return fail(id + ": element value misplaced");
      owner[at] = p;
    }
  for (int p = 0; p < npe * kTileLanes; ++p) {
    std::vector<uint32_t> at;
    if (nc >= 2) at = {f.pairs.beg + 8u * p, f.pairs.beg + 8u * p + 4u};
    if (nc != 2) at.push_back(f.one.beg + 4u * p);
    for (uint32_t o : at)
      if (o < elem.beg || o >= elem.end || owner[(o - elem.beg) / 4] != p)
        return fail(id + ": xi flux over another point's element data");
  }
  if (L.late)
    for (const Region& r : {v, im, pl})
      if (r.beg < elem.beg || r.end > elem.end) return fail(id + ": " + r.name + " overruns the element data");
  return 0;
}

}  // namespace

int main() {
  long cases = 0, late = 0;
  for (int ng = 2; ng <= 9; ++ng)
    for (int kind = INSEM_RECT; kind <= kAxisymOffAxis; ++kind)
      for (int nc = 1; nc <= (is_axisym(kind) ? 3 : 2); ++nc) {
        if (kind == kAxisymOffAxis && nc == 1) continue;  // elastic only
        const int npe = ng * ng, edge = 4 * (ng - 1), q = ng - 1;
        if (npe * kTileLanes > static_cast<int>(kLastPlace)) return fail("staging places do not fit the lists' 15 bits");
        // edge complete points: none, of a compact 8 x 4 tile, and every edge
        // point of 32 scattered elements; halo points likewise
        const int complete[] = {0, 11 * q + 3 * 8 * q, kTileLanes * edge};
        const int halo[] = {0, 24 * q, kTileLanes * npe};
        for (int c : complete)
          for (int h : halo)
            for (int rs = 1; rs <= 33; rs += 4) {
              const int nc_cap = std::max(4, (c + 3) & ~3), tp_cap = std::max(4, (nc_cap + h + 3) & ~3);
              const std::string id = "ng " + std::to_string(ng) + " kind " + std::to_string(kind) + " components " +
                                     std::to_string(nc) + " edge points " + std::to_string(c) + " halo points " +
                                     std::to_string(h) + " list " + std::to_string(rs);
              if (const int rc = check(ng, kind, nc, tp_cap, nc_cap, rs, id)) return rc;
              ++cases;
              late += TileLayout::make(ng, nc, kind, nc > 1, kTileLanes, tp_cap, nc_cap, rs).late;
            }
      }
  if (late == 0 || late == cases) return fail("one of the two arrivals of v, 1/M and lists was never checked");
  std::printf("ok %ld layouts, %ld with late copies\n", cases, late);
  return 0;
}
