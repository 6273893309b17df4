// Batches of molecules evaluated together: one screening pass over all their quartets and one
// launch of each evaluation kernel for all their grid points. No counterpart in the reference,
// which runs calculate_intracule (src/mod_intracule.f90:18-572) once per molecule and
// process; a batch runs its radial_plot job (lines 512-533) for every molecule at once.
//
// Layout: the molecules' primitives are concatenated (each primitive carries its molecule and
// that molecule's screening scale 1/(nprim(nprim+1)/2)); their DM2 records are generated into
// one quartet list with global primitive indices; the survivors are sorted by (molecule, angular
// class), so each molecule owns a contiguous range of work chunks; the scan grids are
// concatenated (shell tags offset per molecule), sorted by (molecule, Morton key), and cut into
// tiles that never straddle two molecules. Every evaluation kernel then pairs each tile with
// its own molecule's chunk range.
#include <algorithm>
#include <cmath>
#include <string>
#include <type_traits>
#include <vector>

#include "inca_internal.h"

namespace inca {

int prepare_device(inca_ctx* c, double thresh, int normalize);
int radial_plot_device(inca_ctx* c, double* rintra);

int batch_prepare(inca_ctx* c, double thresh, inca_counts* counts) {
  const int nmol = static_cast<int>(c->batch.size());
  if (nmol == 0) return set_error(c, INCA_E_STATE, "inca_batch_prepare: no molecules added");
  if (!(thresh > 0.0)) return set_error(c, INCA_E_ARG, "inca_batch_prepare: thresh must be > 0");
  // primitives: the context's own, its quartets and its grid's molecules are gone from here on
  c->source_kept = false;
  c->nprim = 0;
  c->nq = 0;
  c->batch_grid_version = -1;
  int np = 0;
  for (const BatchMol& m : c->batch) np += m.nprim;
  std::vector<PrimD> h(np);
  c->h_alpha.clear(); c->h_x.clear(); c->h_y.clear(); c->h_z.clear();
  c->h_tmn.assign(3 * static_cast<size_t>(np), 0);
  std::vector<int> base(nmol);
  int o = 0;
  for (int mi = 0; mi < nmol; ++mi) {
    const BatchMol& m = c->batch[mi];
    base[mi] = o;
    for (int p = 0; p < m.nprim; ++p) {
      const int t[3] = {m.tmn[3 * p], m.tmn[3 * p + 1], m.tmn[3 * p + 2]};
      h[o + p] = make_prim(m.alpha[p], t, m.x[p], m.y[p], m.z[p], m.nprim, mi);
      for (int d = 0; d < 3; ++d) c->h_tmn[3 * (o + p) + d] = t[d];
      c->h_alpha.push_back(m.alpha[p]);
      c->h_x.push_back(m.x[p]);
      c->h_y.push_back(m.y[p]);
      c->h_z.push_back(m.z[p]);
    }
    o += m.nprim;
  }
  assign_shells(h, &c->group_keys);
  if (c->d_prims.reserve(np)) return set_error(c, INCA_E_NOMEM, "batch primitives");
  INCA_CUDA(c, cudaMemcpyAsync(c->d_prims.p, h.data(), sizeof(PrimD) * np, cudaMemcpyHostToDevice, c->stream));
  c->nprim = np;
  // DM2 records, one molecule after the other
  int64_t nrec = 0;
  for (const BatchMol& m : c->batch) nrec += closed_shell_records(m.nprim, m.unique);
  if (c->d_ijkl.reserve(nrec) || c->d_v.reserve(nrec)) return set_error(c, INCA_E_NOMEM, "batch quartet records");
  int64_t at = 0;
  for (int mi = 0; mi < nmol; ++mi) {
    const BatchMol& m = c->batch[mi];
    const int st = gen_closed_shell_into(c, m.nprim, m.D.data(), m.unique, base[mi], at);
    if (st) return st;
    at += closed_shell_records(m.nprim, m.unique);
  }
  c->nq = nrec;
  c->batch_molecules = nmol;
  int st = prepare_device(c, thresh, 1);
  if (st) return st;
  if (counts) *counts = c->counts;
  // grids: the molecules' scan grids one after the other, in one build (a build, its copies and their
  // allocations per molecule: 1.4 of 2.9 ms for six molecules)
  std::vector<ScanSpec> specs;
  for (const BatchMol& m : c->batch)
    specs.push_back(ScanSpec{static_cast<int>(m.start.size()), m.start.data(), m.end.data(), m.step.data(),
                             m.nang.data(), m.nosym});
  std::vector<int> shoff;
  st = grid_scan_device(c, specs, &shoff);
  if (st) return st;
  std::vector<int64_t> moff(nmol + 1, 0);
  for (int mi = 0; mi < nmol; ++mi) {
    moff[mi + 1] = moff[mi];
    for (int s = shoff[mi]; s < shoff[mi + 1]; ++s) moff[mi + 1] += c->h_smn[s];
  }
  c->rgrid = c->ngrid;
  c->maxgrid = c->ngrid;
  c->h_mol_off = moff;
  c->h_mol_shell_off = shoff;
  ++c->grid_version;
  c->batch_grid_version = c->grid_version;
  c->evaluated = false;
  return INCA_OK;
}

}  // namespace inca

using namespace inca;

#define CTX_CHECK(c)             \
  do {                           \
    if (!(c)) return INCA_E_ARG; \
    cudaSetDevice((c)->device);  \
  } while (0)

extern "C" {

int inca_batch_clear(inca_ctx* c) {
  CTX_CHECK(c);
  c->batch.clear();
  return INCA_OK;
}

int inca_batch_add_closed_shell(inca_ctx* c, int32_t nprim, const double* alpha, const int32_t* tmn,
                                const double* xn, const double* yn, const double* zn, const double* D, int unique,
                                int32_t nblock, const double* start, const double* end, const double* step,
                                const int32_t* nang, int nosym, int32_t* nradi) {
  CTX_CHECK(c);
  if (nprim <= 0 || !alpha || !tmn || !xn || !yn || !zn || !D || nblock < 1 || !start || !end || !step || !nang)
    return set_error(c, INCA_E_ARG, "inca_batch_add_closed_shell: bad arguments");
  if (static_cast<int>(c->batch.size()) >= INCA_MAX_BATCH)
    return set_error(c, INCA_E_LIMIT, "inca_batch_add_closed_shell: more than INCA_MAX_BATCH molecules");
  BatchMol m;
  m.nprim = nprim;
  m.alpha.assign(alpha, alpha + nprim);
  m.x.assign(xn, xn + nprim);
  m.y.assign(yn, yn + nprim);
  m.z.assign(zn, zn + nprim);
  m.tmn.assign(3 * static_cast<size_t>(nprim), 0);
  for (int p = 0; p < nprim; ++p) {
    if (!(alpha[p] > 0.0)) return set_error(c, INCA_E_ARG, "inca_batch_add_closed_shell: exponent <= 0");
    for (int d = 0; d < 3; ++d) {
      const int t = tmn[p + static_cast<size_t>(nprim) * d];  // TMN(nprim,3), column-major
      if (t < 0 || t > 4) return set_error(c, INCA_E_LIMIT, "inca_batch_add_closed_shell: Cartesian power outside 0..4");
      m.tmn[3 * p + d] = t;
    }
  }
  m.D.assign(D, D + static_cast<size_t>(nprim) * nprim);
  m.unique = unique ? 1 : 0;
  m.nradi = 0;
  for (int b = 0; b < nblock; ++b) {
    if (!(step[b] > 0.0) || !(end[b] >= start[b]))
      return set_error(c, INCA_E_ARG, "inca_batch_add_closed_shell: bad scan block");
    m.nradi += static_cast<int>((end[b] - start[b]) / step[b]) + 1;
  }
  m.start.assign(start, start + nblock);
  m.end.assign(end, end + nblock);
  m.step.assign(step, step + nblock);
  m.nang.assign(nang, nang + nblock);
  m.nosym = nosym ? 1 : 0;
  if (nradi) *nradi = m.nradi;
  c->batch.push_back(std::move(m));
  return INCA_OK;
}

int inca_batch_prepare(inca_ctx* c, double thresh, inca_counts* counts, int64_t* ngrid) {
  CTX_CHECK(c);
  const int st = batch_prepare(c, thresh, counts);
  if (st == INCA_OK && ngrid) *ngrid = c->ngrid;
  return st;
}

int inca_batch_eval(inca_ctx* c, int mode, double tol, double* rintra) {
  CTX_CHECK(c);
  if (c->batch_molecules == 0 || c->batch_grid_version != c->grid_version)
    return set_error(c, INCA_E_STATE, "inca_batch_eval: prepare the batch first");
  int st = eval_device(c, mode, tol);
  if (st) return st;
  return rintra ? radial_plot_device(c, rintra) : INCA_OK;
}

}  // extern "C"
