// Host layout of the packed element list of an AMR hierarchy: elements
// (valid cells of every level, then the ghost elements the predictor needs at
// coarse-fine boundaries), their faces, and the tables the kernels index
// (faces, coarse-fine flux corrections, average-down, ghost fill).  Replaces
// the box / MultiFab / iMultiFab bookkeeping AMReX does for the reference
// (Source/Core/Mesh.h, Source/NumericalMethod/AmrDG/AmrDG_Level.tpp:240-414).
#pragma once

#include <cstdint>
#include <string>
#include <vector>

#include "adg.h"
#include "amr_grids.hpp"

namespace adg {

struct Hierarchy {
  int D = 2;
  int nlev = 0;
  int n_cell0[3] = {1, 1, 1};
  int periodic[3] = {1, 1, 1};
  std::vector<std::vector<amr::IBox>> grids;

  // elements: valid cells of level 0, 1, ... (x-fastest per level), then ghosts
  std::vector<int> elem_cell;      // [elem][3]
  std::vector<int8_t> elem_level;  // [elem]
  std::vector<size_t> lev_valid_off, lev_valid_cnt;
  size_t n_valid_ = 0, n_elem_ = 0;
  std::vector<std::vector<int>> cellmap;   // per level: cell -> element (valid or ghost), -1
  std::vector<std::vector<int>> cellbox;   // per level: cell -> box index (valid cells), -1

  // neighbours of the valid elements, [elem][2D] (low, high per direction):
  // valid or ghost element, -1 outside the domain
  std::vector<int> nbr;
  // valid elements covered by the next level
  std::vector<uint8_t> cov;

  // faces, grouped by direction
  std::vector<int> face_left, face_right;
  int face_off[4] = {0, 0, 0, 0};
  std::vector<int> elem_face;  // [valid elem][2D]

  // coarse-fine corrections (reflux): one record per coarse cell with entries
  std::vector<int> rf_elem;       // [rec] coarse element
  std::vector<int> rf_off;        // [rec+1] entry range
  std::vector<int> rf_face;       // [ent] coarse face id
  std::vector<int8_t> rf_dside;   // [ent] 2*d + side (side 1: the coarse cell's high face)
  std::vector<int> rf_fine;       // [ent][2^(D-1)] fine face ids, child order
  // average down: per fine level lf (1..nlev-1), records (coarse, 2^D fine)
  std::vector<std::vector<int>> ad_rec;   // [lf] flat: coarse, fine_0 .. fine_{2^D-1}
  // ghost fill: ghost element, coarse parent element, child index
  std::vector<int> gf_elem, gf_parent;
  std::vector<int8_t> gf_child;

  int nlevels() const { return nlev; }
  size_t n_valid() const { return n_valid_; }
  size_t n_elem() const { return n_elem_; }
  size_t level_valid_offset(int l) const { return lev_valid_off[l]; }
  size_t level_valid_count(int l) const { return lev_valid_cnt[l]; }

  void dims(int l, int* n) const {
    for (int d = 0; d < 3; ++d) n[d] = d < D ? n_cell0[d] << l : 1;
  }
  size_t cidx(int l, const int* c) const {
    int n[3];
    dims(l, n);
    return ((size_t)c[2] * n[1] + c[1]) * n[0] + c[0];
  }
  // wrap periodically; false if outside a non-periodic domain
  bool wrap(int l, int* c) const {
    int n[3];
    dims(l, n);
    for (int d = 0; d < D; ++d) {
      if (c[d] >= 0 && c[d] < n[d]) continue;
      if (!periodic[d]) return false;
      c[d] = ((c[d] % n[d]) + n[d]) % n[d];
    }
    return true;
  }
  int elem_at(int l, const int* cin) const {
    int c[3] = {cin[0], cin[1], cin[2]};
    if (!wrap(l, c)) return -1;
    return cellmap[l][cidx(l, c)];
  }
  bool is_valid_elem(int e) const { return e >= 0 && (size_t)e < n_valid_; }

  bool build_single_level(const adg_config& c, std::string* msg) {
    amr::GridParams gp = params(c);
    std::vector<std::vector<amr::IBox>> g;
    amr::IBox dom;
    for (int d = 0; d < 3; ++d) {
      dom.lo[d] = 0;
      dom.hi[d] = d < gp.D ? gp.n_cell0[d] - 1 : 0;
    }
    g.push_back({dom});
    return build(gp, g, 0, msg);
  }

  static amr::GridParams params(const adg_config& c) {
    amr::GridParams gp;
    gp.D = c.D;
    for (int d = 0; d < 3; ++d) {
      gp.n_cell0[d] = d < c.D ? c.n_cell[d] : 1;
      gp.periodic[d] = d < c.D ? c.periodic[d] : 1;
    }
    gp.max_level = c.max_level;
    gp.blocking_factor = c.blocking_factor > 0 ? c.blocking_factor : 8;
    gp.max_grid = c.max_grid > 0 ? c.max_grid : 32;
    gp.grid_eff = c.grid_eff > 0 ? c.grid_eff : 0.7;
    gp.n_error_buf = c.n_error_buf >= 0 ? c.n_error_buf : 1;
    return gp;
  }

  // Build every table for the given boxes.  reflux_quirk reproduces the
  // reference's per-box reflux mask (AmrDG_Interpolater.tpp:41-56 with the
  // face ownership rule of AmrDG_Level.tpp:316-330): a coarse cell is
  // corrected only if one of its coarse-fine faces is flagged in its own
  // box's face array, where a box never flags its own low face.
  // reflux = false leaves out every coarse-fine flux correction (the
  // reference's runs without AMR_flux_correction).
  //
  // A regrid waits for this.  Cells are looked up once, into nbr and cov; the
  // other tables read those in element order, sized beforehand, and a rebuilt
  // hierarchy reuses its memory (95,000 elements in 3D: 20 ms with a wrapped
  // lookup per use and growing vectors, 3.6 ms now).
  bool build(const amr::GridParams& gp, const std::vector<std::vector<amr::IBox>>& g, int reflux_quirk,
             std::string* msg, bool reflux = true) {
    auto no = [&](const std::string& m) {
      if (msg) *msg = m;
      return false;
    };
    D = gp.D;
    for (int d = 0; d < 3; ++d) {
      n_cell0[d] = gp.n_cell0[d];
      periodic[d] = gp.periodic[d];
    }
    grids = g;
    nlev = (int)g.size();
    cellmap.resize(nlev);
    cellbox.resize(nlev);
    elem_cell.clear();
    elem_level.clear();
    lev_valid_off.assign(nlev, 0);
    lev_valid_cnt.assign(nlev, 0);
    // ---- valid elements
    for (int l = 0; l < nlev; ++l) {
      int n[3];
      dims(l, n);
      const size_t nc = (size_t)n[0] * n[1] * n[2];
      if (nc > (size_t)1 << 31) return no("level too large");
      cellmap[l].assign(nc, -1);
      cellbox[l].assign(nc, -1);
      size_t cells = 0;
      for (size_t b = 0; b < g[l].size(); ++b) {
        const amr::IBox& bx = g[l][b];
        bool empty = false;
        for (int d = 0; d < 3; ++d) empty = empty || bx.hi[d] < bx.lo[d];
        if (empty) continue;
        for (int d = 0; d < D; ++d)
          if (bx.lo[d] < 0 || bx.hi[d] >= n[d]) return no("box outside the domain");
        for (int k = bx.lo[2]; k <= bx.hi[2]; ++k)
          for (int j = bx.lo[1]; j <= bx.hi[1]; ++j) {
            int* row = cellbox[l].data() + ((size_t)k * n[1] + j) * n[0];
            for (int i = bx.lo[0]; i <= bx.hi[0]; ++i) {
              if (row[i] >= 0) return no("overlapping boxes");
              row[i] = (int)b;
            }
            cells += bx.hi[0] - bx.lo[0] + 1;
          }
      }
      const size_t e0 = elem_level.size();
      lev_valid_off[l] = e0;
      lev_valid_cnt[l] = cells;
      elem_level.resize(e0 + cells, (int8_t)l);
      elem_cell.resize(3 * (e0 + cells));
      int* at = elem_cell.data() + 3 * e0;
      int e = (int)e0;
      const int* box = cellbox[l].data();
      int* map = cellmap[l].data();
      for (int k = 0; k < n[2]; ++k)
        for (int j = 0; j < n[1]; ++j, box += n[0], map += n[0])
          for (int i = 0; i < n[0]; ++i) {
            if (box[i] < 0) continue;
            map[i] = e++;
            at[0] = i, at[1] = j, at[2] = k;
            at += 3;
          }
    }
    n_valid_ = elem_level.size();
    if (n_valid_ == 0 || lev_valid_cnt[0] != (size_t)n_cell0[0] * n_cell0[1] * n_cell0[2])
      return no("level 0 must cover the domain");
    // ---- neighbours, and the ghost elements at coarse-fine boundaries (face
    // neighbours only)
    gf_elem.clear();
    gf_parent.clear();
    gf_child.clear();
    const int F = 2 * D;
    nbr.resize(n_valid_ * F);
    cov.assign(n_valid_, 0);
    size_t nface_hi[3] = {0, 0, 0};  // high faces without a valid element beyond
    for (int l = 0; l < nlev; ++l) {
      const size_t e0 = lev_valid_off[l], e1 = e0 + lev_valid_cnt[l];
      int n[3];
      dims(l, n);
      const size_t st[3] = {1, (size_t)n[0], (size_t)n[0] * n[1]};
      int* map = cellmap[l].data();
      for (size_t e = e0; e < e1; ++e) {
        const int c[3] = {elem_cell[3 * e], elem_cell[3 * e + 1], elem_cell[3 * e + 2]};
        const size_t id = c[0] + c[1] * st[1] + c[2] * st[2];
        if (l > 0) {
          bool first = true;  // of its parent's children
          size_t pid = 0;
          for (int d = D - 1; d >= 0; --d) {
            first = first && !(c[d] & 1);
            pid = pid * (n[d] >> 1) + (c[d] >> 1);
          }
          if (first) {
            const int pe = cellmap[l - 1][pid];
            if (is_valid_elem(pe)) cov[pe] = 1;
          }
        }
        for (int d = 0; d < D; ++d)
          for (int s = 0; s < 2; ++s) {
            int& out = nbr[e * F + 2 * d + s];
            int x = c[d] + (s ? 1 : -1);
            size_t nid = s ? id + st[d] : id - st[d];
            if (x < 0 || x >= n[d]) {
              if (!periodic[d]) {
                out = -1;
                nface_hi[d] += s;
                continue;
              }
              nid = s ? id - (n[d] - 1) * st[d] : id + (n[d] - 1) * st[d];
              x = s ? 0 : n[d] - 1;
            }
            out = map[nid];
            if (out >= 0) {
              if (s && !is_valid_elem(out)) ++nface_hi[d];
              continue;
            }
            if (l == 0) return no("missing neighbour element");
            nface_hi[d] += s;
            out = map[nid] = (int)elem_level.size();
            elem_level.push_back((int8_t)l);
            int nb[3] = {c[0], c[1], c[2]};
            nb[d] = x;
            elem_cell.insert(elem_cell.end(), nb, nb + 3);
            int par[3] = {0, 0, 0}, child = 0;
            for (int a = 0; a < D; ++a) {
              par[a] = nb[a] >> 1;
              child += (nb[a] & 1) << (D - 1 - a);
            }
            const int pe = cellmap[l - 1][cidx(l - 1, par)];
            if (!is_valid_elem(pe))
              return no("level " + std::to_string(l) + " is not properly nested in level " + std::to_string(l - 1));
            gf_elem.push_back(out);
            gf_parent.push_back(pe);
            gf_child.push_back((int8_t)child);
          }
      }
    }
    n_elem_ = elem_level.size();
    // ---- faces: per direction and level the low faces of all elements, then
    // the high faces without a valid element beyond
    size_t nf = 0;
    for (int d = 0; d < D; ++d) {
      face_off[d] = (int)nf;
      nf += n_valid_ + nface_hi[d];
    }
    for (int d = D; d < 4; ++d) face_off[d] = (int)nf;
    face_left.resize(nf);
    face_right.resize(nf);
    elem_face.resize(n_valid_ * F);
    for (int d = 0; d < D; ++d) {
      int f = face_off[d];
      for (int l = 0; l < nlev; ++l) {
        const size_t e0 = lev_valid_off[l], e1 = e0 + lev_valid_cnt[l];
        for (size_t e = e0; e < e1; ++e) {
          const int left = nbr[e * F + 2 * d];
          elem_face[e * F + 2 * d] = f;
          face_left[f] = left < 0 ? (int)e : left;  // outflow: zero-gradient mirror
          face_right[f++] = (int)e;
        }
        for (size_t e = e0; e < e1; ++e) {
          const int right = nbr[e * F + 2 * d + 1];
          if (is_valid_elem(right)) {
            elem_face[e * F + 2 * d + 1] = elem_face[(size_t)right * F + 2 * d];
          } else {
            elem_face[e * F + 2 * d + 1] = f;
            face_left[f] = (int)e;
            face_right[f++] = right < 0 ? (int)e : right;
          }
        }
      }
    }
    // ---- coarse-fine flux corrections
    rf_elem.clear();
    rf_off.assign(1, 0);
    rf_face.clear();
    rf_dside.clear();
    rf_fine.clear();
    const int nfc = 1 << (D - 1);
    for (int l = 0; reflux && l + 1 < nlev; ++l) {
      const size_t e0 = lev_valid_off[l], e1 = e0 + lev_valid_cnt[l];
      for (size_t e = e0; e < e1; ++e) {
        if (cov[e]) continue;
        const int* c = &elem_cell[3 * e];
        const int nent0 = (int)rf_face.size();
        bool apply = !reflux_quirk;
        for (int i = 0; i < F; ++i) {
          const int d = i / 2, side = i % 2, ne = nbr[e * F + i];
          if (!is_valid_elem(ne) || !cov[ne]) continue;
          rf_face.push_back(elem_face[e * F + i]);
          rf_dside.push_back((int8_t)i);
          const int nbd = elem_cell[3 * (size_t)ne + d];
          for (int k = 0; k < nfc; ++k) {
            int f[3] = {0, 0, 0}, bit = 0;
            for (int a = 0; a < D; ++a) {
              if (a == d) {
                f[a] = side ? 2 * nbd : 2 * nbd + 1;
              } else {
                f[a] = 2 * c[a] + ((k >> bit) & 1);
                bit++;
              }
            }
            const int fe = cellmap[l + 1][cidx(l + 1, f)];
            if (!is_valid_elem(fe)) return no("coarse-fine face without fine cells");
            rf_fine.push_back(elem_face[(size_t)fe * F + 2 * d + (side ? 0 : 1)]);
          }
          if (side == 1 || c[d] > grids[l][cellbox[l][cidx(l, c)]].lo[d]) apply = true;
        }
        if ((int)rf_face.size() == nent0) continue;
        if (!apply) {  // the reference never applies these corrections
          rf_face.resize(nent0);
          rf_dside.resize(nent0);
          rf_fine.resize((size_t)nent0 * nfc);
          continue;
        }
        rf_elem.push_back((int)e);
        rf_off.push_back((int)rf_face.size());
      }
    }
    // ---- average down
    ad_rec.resize(nlev);
    for (auto& r : ad_rec) r.clear();
    for (int lf = 1; lf < nlev; ++lf) {
      const int l = lf - 1, nov = 1 << D;
      int n[3];
      dims(lf, n);
      size_t kid[8];
      for (int k = 0; k < nov; ++k) {
        int f[3] = {0, 0, 0};
        for (int a = 0; a < D; ++a) f[a] = (k >> (D - 1 - a)) & 1;
        kid[k] = cidx(lf, f);
      }
      const int* map = cellmap[lf].data();
      const size_t e0 = lev_valid_off[l], e1 = e0 + lev_valid_cnt[l];
      size_t count = 0;
      for (size_t e = e0; e < e1; ++e) count += cov[e];
      ad_rec[lf].resize(count * (nov + 1));
      int* at = ad_rec[lf].data();
      for (size_t e = e0; e < e1; ++e) {
        if (!cov[e]) continue;
        const int* c = &elem_cell[3 * e];
        const int f[3] = {2 * c[0], 2 * c[1], D == 3 ? 2 * c[2] : 0};
        const size_t id = cidx(lf, f);
        *at++ = (int)e;
        for (int k = 0; k < nov; ++k) *at++ = map[id + kid[k]];
      }
    }
    return true;
  }
};

}  // namespace adg
