// Host-side mesh construction and device-layout preparation for libxcal.
#pragma once
#include <cstdint>
#include <string>
#include <vector>

#include "../../include/xcal.h"

namespace xcal {

// Reference-layout mesh held on the host, 0-based.
struct HostMesh {
  int64_t nc = 0, nf = 0, nbf = 0, nnodes = 0;
  int dim = 2;
  std::vector<double> cc, cvol;                      // cc [3*nc]
  std::vector<int64_t> cf_ptr, cf_face, cf_nbr, cf_sign;
  std::vector<int64_t> o1, o2;
  std::vector<double> fc, fn, fe, farea, fdelta, fweight;   // fc/fn/fe [3*nf]
  std::vector<std::string> pname;
  std::vector<int64_t> pptr, pfaces, pcells;       // concatenated patches
  std::vector<double> nodes;                       // [3*nnodes] (optional: VTK output)
  std::vector<int64_t> cn_ptr, cn;                 // cell node lists, 0-based (optional)
  // 1-based export copies (xcal_hmesh_desc)
  std::vector<int64_t> x_cfp, x_cf, x_cn, x_own, x_pf, x_pc, x_cnp, x_cnode;
  std::string names;
  void prepare_export();
};

int build_unv(const char *path, double scale, HostMesh &M, std::string &err);
int mesh_from_desc(const xcal_mesh_desc *d, HostMesh &M, std::string &err);

// Cell renumbering: perm[old] = new.
void renumber_perm(const HostMesh &M, int mode, std::vector<int64_t> &perm);
// Apply a permutation (cells) and, for a non-identity mode, sort internal faces
// by (min owner, max owner, old id); per-cell face lists re-sorted by face id.
void apply_perm(const HostMesh &in, const std::vector<int64_t> &perm, bool reorder_faces,
                HostMesh &out);

// Lists of the sweeps by one CTA (KParams::frow, brow, items, lptr): rows by
// forward and by backward level, items of up to 32 rows of a level, the first
// item of each level.  Empty where the grid sweeps level by level: two levels,
// levels of more than SWEEP_WIDTH rows on average, or any level of more than
// SWEEP_WIDEST (64 rounds of the CTA's 256 threads, about 0.1 ms: the other CTAs
// wait meanwhile, and their wait is limited).
// (ms per SIMPLE iteration, grid / one CTA, by average rows per level: BFS 5k 16:
// 185 / 104; cavity 80^2 40: 65.7 / 36.3; BFS 47k 49: 599 / 532; hex 12^3 51: 4.9 /
// 3.3; cavity 110^2 55: 106 / 85.7; 120^2 60: 99.8 / 64.7; hex 14^3 69: 4.06 / 3.82;
// cavity 160^2 80: 166 / 118; hex 16^3 89: 4.65 / 5.93; 20^3 138: 7.49 / 9.17.  In 2D
// one CTA is still faster somewhat above the line.)
constexpr int SWEEP_WIDTH = 56, SWEEP_WIDEST = 16384;
struct LevelLists {
  std::vector<int> frow, brow, items, ptr;
};
LevelLists level_lists(const std::vector<int> &flev, const std::vector<int> &blev, int n, int nfl, int nbl);

// Device-ready integer structures built from a (renumbered) mesh.  Matrix and
// per-cell face lists use an ELL layout padded to np = 256*ceil(n/256) rows:
// entry k of row i sits at k*np + i (coalesced across a warp); unused entries
// hold column -1.  Entries of a row are in ascending column order.
struct Prep {
  int n = 0, nf = 0, nbf = 0, nnz = 0, np = 0, W = 0, Wf = 0;
  std::vector<int> row_ptr, col, diag, tslot;   // CSR view (export, tests)
  std::vector<int> e_col, e_tpos, dpos, csr2ell;
  std::vector<int> f_face, f_nbr, f_pos;
  std::vector<signed char> f_sign;
  std::vector<unsigned char> f_first;
  std::vector<int> cb_ptr, cb_face;          // boundary faces per cell, face-id order
  std::vector<int> flev, blev;
  int nfl = 0, nbl = 0;
  int n0 = 0;                                // two_level_rows
  LevelLists lists;
  std::vector<int> o1, o2;
};
int prepare(const HostMesh &M, Prep &P, std::string &err);

// n0 > 0 when the rows [0, n0) are of level 0 and the rows [n0, n) of level 1
// and there are no other levels in either sweep (the two-colour numbering),
// else 0.
int two_level_rows(const std::vector<int> &flev, int n, int nfl, int nbl);

}  // namespace xcal
